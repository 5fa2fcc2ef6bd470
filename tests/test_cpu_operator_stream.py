"""The stream that operator calls take (qwen_inference_engine_b200/layers.py): torch's raw handle, and the public way where torch does not have it."""
import types

import pytest

torch = pytest.importorskip("torch")


class Stream:
    cuda_stream = 77


def test_raw_handle_of_the_current_device(monkeypatch):
    from qwen_inference_engine_b200 import layers as L
    monkeypatch.setattr(torch, "_C", types.SimpleNamespace(_cuda_getDevice=lambda: 3, _cuda_getCurrentRawStream=lambda dev: 40 + dev))
    assert L._st() == 43


@pytest.mark.parametrize("names", [{}, {"_cuda_getDevice": lambda: 3}, {"_cuda_getCurrentRawStream": lambda dev: 40 + dev}])
def test_without_the_private_names(monkeypatch, names):
    from qwen_inference_engine_b200 import layers as L
    monkeypatch.setattr(torch, "_C", types.SimpleNamespace(**names))
    monkeypatch.setattr(torch.cuda, "current_stream", Stream)
    assert L._st() == 77
