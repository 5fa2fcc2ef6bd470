"""The reference-order norm at the edges of its row and width variants (csrc/ops_ref_order.cu), bit for bit against the CPU restatement."""
import numpy as np
import pytest

from util import rand_bf16, to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_tok", [1, 3, 887, 888, 889, 891])
@pytest.mark.parametrize("hidden", [8, 24, 33, 250, 896, 1000, 5112, 5120, 12288])
def test_rows_and_widths(oracle, hidden, n_tok):
    from qwen_inference_engine_b200 import layers as L
    rng = np.random.default_rng(hidden * 7 + n_tok)
    x, w = rand_bf16(rng, (n_tok, hidden), 1.5), rand_bf16(rng, (hidden,), 1.0)
    want = oracle.rmsnorm(x, w)
    xd, wd = to_dev(x), to_dev(w)
    y = torch.full_like(xd, 3.0)
    L.launch_rms(xd, wd, y, hidden, n_tok)
    assert np.array_equal(to_host(y), want)
    L.launch_rms(xd, wd, xd, hidden, n_tok)  # in place
    assert np.array_equal(to_host(xd), want)


@pytest.mark.parametrize("n_tok", [5, 900])
@pytest.mark.parametrize("off", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (8, 8, 8)])
def test_operands_off_a_16_byte_boundary(oracle, n_tok, off):
    from qwen_inference_engine_b200 import layers as L
    hidden = 896
    rng = np.random.default_rng(n_tok + sum(off))
    x, w = rand_bf16(rng, (n_tok, hidden), 1.0), rand_bf16(rng, (hidden,), 1.0)

    def placed(a, o):
        buf = torch.zeros(a.size + 16, dtype=torch.bfloat16, device="cuda")
        t = buf[o:o + a.size].view(a.shape)
        t.copy_(to_dev(a))
        return t
    xd, wd, y = placed(x, off[0]), placed(w, off[1]), placed(np.zeros_like(x), off[2])
    L.launch_rms(xd, wd, y, hidden, n_tok)
    assert np.array_equal(to_host(y), oracle.rmsnorm(x, w))


@pytest.mark.parametrize("n_tok", [1, 889, 1775, 1776, 1777])
@pytest.mark.parametrize("hidden", [8, 15, 16, 17, 31, 40, 250, 632, 640, 1001, 12287, 12288])
def test_remainders_of_the_chain(oracle, hidden, n_tok):
    """the last pieces of a row, whole and cut short; widths around the rule for four rows a block, at 6 and 12 rows an SM; the widest row in fp32"""
    from qwen_inference_engine_b200 import layers as L
    rng = np.random.default_rng(hidden * 3 + n_tok)
    x, w = rand_bf16(rng, (n_tok, hidden), 1.5), rand_bf16(rng, (hidden,), 1.0)
    want = oracle.rmsnorm(x, w)
    for off in (0, 1):  # off 1: element by element at any width
        buf = torch.zeros(x.size + 16, dtype=torch.bfloat16, device="cuda")
        xd = buf[off:off + x.size].view(x.shape)
        xd.copy_(to_dev(x))
        y = torch.full_like(to_dev(x), 3.0)
        L.launch_rms(xd, to_dev(w), y, hidden, n_tok)
        assert np.array_equal(to_host(y), want), off
