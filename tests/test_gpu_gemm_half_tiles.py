"""Tiles of 64 weight rows and four k-blocks a stage (csrc/gemm_tcgen05.cu) against float64, at edges of the tiles, the stages and the rule that takes them:
outputs around multiples of 64, rows around multiples of 16 to 64, inner sizes whose last stage is short.  Exact products of small whole numbers, so
that the results are the same whatever the order of the sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner", [512, 576, 640, 704, 896, 1280, 4096 + 64])
@pytest.mark.parametrize("outer", [8, 56, 64, 72, 130, 896, 1000])
@pytest.mark.parametrize("rows", [1, 16, 17, 33, 64, 65, 200, 520])
def test_whole_numbers(inner, outer, rows):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    g = torch.Generator("cuda").manual_seed(inner + outer + rows)
    a = torch.randint(-1, 2, (rows, inner), generator=g, device="cuda").bfloat16()
    b = torch.randint(-1, 2, (outer, inner), generator=g, device="cuda").bfloat16()
    want = (a.double() @ b.double().T).float().bfloat16()  # (sums below 2^24 are exact; one rounding to bf16)
    for f in (L.launch_matmul, L.launch_matmul_fast):
        out = torch.full((rows + 1, outer), 7.0, dtype=torch.bfloat16, device="cuda")
        f(a, b, out, rows, inner, outer)
        torch.cuda.synchronize()
        assert torch.equal(out[:rows], want)
        assert (out[rows:] == 7).all()
