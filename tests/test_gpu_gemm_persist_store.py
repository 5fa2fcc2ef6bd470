"""How the persistent GEMM's results leave the chip (csrc/gemm_tcgen05.cu): bulk copies for plain results, residual and SiLU * up from the
staging tiles.  Against the kernel with one tile per CTA, in the reference order, so there is no tolerance."""
import numpy as np
import pytest
import torch

from util import prompt_ids

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def device():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("rows", [257, 320, 1000, 1023])
@pytest.mark.parametrize("outer", [19976, 20096])
def test_plain_results(rows, outer):
    """tiles cut at both ends (8 of 128 outputs, 1 row of a step); what lies behind the last row stays"""
    from qwen_inference_engine_b200 import layers as L
    g = torch.Generator("cuda").manual_seed(rows)
    a = torch.randn(rows, 72, generator=g, device="cuda").bfloat16()
    b = torch.randn(outer, 72, generator=g, device="cuda").bfloat16()
    out = torch.full((rows + 2, outer), 7.0, dtype=torch.bfloat16, device="cuda")
    L.launch_matmul(a, b, out[:rows], rows, 72, outer)
    for r in range(0, rows, 16):  # 16 rows: one tile per CTA
        n = min(16, rows - r)
        part = torch.empty(n, 5000, dtype=torch.bfloat16, device="cuda")
        for c in (0, outer - 5000):
            L.launch_matmul(a[r:r + n].clone(), b[c:c + 5000].clone(), part, n, 72, 5000)
            assert torch.equal(out[r:r + n, c:c + 5000].view(torch.int16), part.view(torch.int16))
    assert (out[rows:] == 7).all()


def test_residual_and_gate_up():
    """a prompt of 1003 rows at once (all projections persistent) and in portions of 100 rows"""
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(hidden=2560, inter=1320, layers=2, n_q=40, n_kv=8, head_dim=64, vocab=4096), context=2048)
    got = []
    for most in (1024, 100):
        e = q.Engine(synthetic=cfg, seed=5, context=2048, max_seqs=1, max_batch_tokens=most, max_pages=70)
        token = e.prefill(e.new_sequence(), prompt_ids(1003, 4096, seed=1))
        got.append((token, e.read_activation("logits", 4096)))
        e.close()
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])
