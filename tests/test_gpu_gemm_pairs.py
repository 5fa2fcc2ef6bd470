"""Pairs of CTAs on one tile, and token tiles first (csrc/gemm_tcgen05.cu: pick_pair, tokens_first): an odd number of weight tiles, segments and tiles that end inside a
pair, ragged rows.  Exact products of small whole numbers against float64, in both numerics, plain, with the residual and with SiLU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def numbers(g, *shape):
    return torch.randint(-1, 2, shape, generator=g, device="cuda").bfloat16()


@pytest.mark.parametrize("rows,inner,outer", [(4096, 1536, 8960), (4000, 1536, 8960 + 128), (2050, 1536, 8960 - 56), (4096, 8960, 1536), (4096, 3584, 3584), (1500, 3584, 3584),
                                              (3000, 1280, 4736), (4096, 1344, 6000), (2100, 1984, 4001), (300, 896, 40000), (1000, 3584, 18944), (129, 2048, 20000 + 8)])
def test_whole_numbers(rows, inner, outer):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    g = torch.Generator("cuda").manual_seed(rows + inner + outer)
    a, b = numbers(g, rows, inner), numbers(g, outer, inner)
    want = (a.float() @ b.float().T).bfloat16()  # (sums below 2^24 are exact in fp32; one rounding to bf16)
    for f in (L.launch_matmul, L.launch_matmul_fast):
        out = torch.full((rows + 1, outer), 7.0, dtype=torch.bfloat16, device="cuda")
        f(a, b, out, rows, inner, outer)
        torch.cuda.synchronize()
        assert torch.equal(out[:rows], want)
        assert (out[rows:] == 7).all()


@pytest.mark.parametrize("tokens", [2300, 4096])
def test_layer_of_pairs(tokens):
    """gate/up, segments of q, k and v and the residual in a model whose projections take pairs, against the same prompt in portions that do not"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import numpy as np
    import qwen_inference_engine_b200 as q
    arch = dict(hidden=1536, inter=8960, layers=1, n_q=12, n_kv=2, head_dim=128, vocab=4096, context=8192)
    ids = np.random.default_rng(tokens).integers(0, 4096, size=tokens, dtype=np.int32)
    got = []
    for most in (4096, 256):
        e = q.Engine(synthetic=q.make_config(arch), seed=3, context=8192, max_seqs=1, max_batch_tokens=most, max_pages=300)
        s = e.new_sequence()
        token = e.prefill(s, ids)
        got.append((token, e.read_activation("logits", 4096)))
        e.close()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
