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


@pytest.mark.parametrize("rows", [9, 64, 128])
def test_few_rows_keep_the_reference_silu(rows):
    """gate/up of 7B widths (more tiles than SMs at any row count) in fast numerics: the sums are the reference order's, since nothing splits them, and
    so are silu and the product, bit for bit"""
    import ctypes as C
    import qwen_inference_engine_b200 as q
    from qwen_inference_engine_b200 import _lib
    from qwen_inference_engine_b200 import layers as L
    hidden, inter = 3584, 18944
    cfg = q.make_config(dict(hidden=hidden, inter=inter, layers=1, n_q=28, n_kv=4, head_dim=128, vocab=4096), context=256)
    e = q.Engine(synthetic=cfg, seed=5, context=256, max_seqs=1, max_batch_tokens=rows, max_pages=16, numerics="fast")
    e.set_int("layer_count", 1)  # the layer alone: its operand stays in place
    e.prefill(e.new_sequence(), prompt_ids(rows, 4096, seed=rows))
    xn, h = (torch.from_numpy(e.read_activation(n, rows * w).view(np.int16)).cuda().view(torch.bfloat16) for n, w in (("xn", hidden), ("h", inter)))
    gate, up = (torch.empty(rows, inter, dtype=torch.bfloat16, device="cuda") for _ in "gu")
    torch.cuda.synchronize()
    for name, out in (("gate", gate), ("up", up)):
        _lib.check(_lib.lib().qie_matmul(C.c_void_p(xn.data_ptr()), C.c_void_p(e.weight_ptr("mlp.%s_proj.weight" % name, 0)[0]), C.c_void_p(out.data_ptr()), rows, hidden, inter,
                                         torch.cuda.current_stream().cuda_stream))
    L.launch_act(gate, gate.numel())
    L.launch_elem(gate, up, gate, gate.numel())
    torch.cuda.synchronize()
    assert torch.equal(gate.view(torch.int16).view(rows, inter), h.view(torch.int16).view(rows, inter))
    e.close()
