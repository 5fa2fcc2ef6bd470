"""Gate/up tiles that take both matrices by one request, two k-blocks a stage (csrc/gemm_tcgen05.cu), at edges of the tiles and of the stages: outputs that are
no multiple of 64, an odd number of k-blocks, rows around the tile widths of 16, 32 and 64, two CTAs an SM, clusters that split the inner dimension."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter", [(896, 4864), (448, 200), (512, 64), (896, 9536), (2560, 512)])
@pytest.mark.parametrize("rows", [9, 16, 17, 33, 64])
def test_against_single_operators(hidden, inter, rows):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    from qwen_inference_engine_b200 import _lib
    from qwen_inference_engine_b200 import layers as L
    cfg = q.make_config(dict(hidden=hidden, inter=inter, layers=1, n_q=4, n_kv=2, head_dim=64, vocab=4096), context=256)
    for numerics in ("reference_order", "fast"):
        if numerics == "fast" and inter % 64:
            continue  # (refused)
        e = q.Engine(synthetic=cfg, seed=5, context=256, max_seqs=1, max_batch_tokens=rows, max_pages=16, numerics=numerics)
        e.set_int("layer_count", 1)  # the layer alone: its operand stays in place
        e.prefill(e.new_sequence(), np.random.default_rng(rows).integers(0, 4096, size=rows, dtype=np.int32))
        xn, h = (torch.from_numpy(e.read_activation(n, rows * w).view(np.int16)).cuda().view(torch.bfloat16) for n, w in (("xn", hidden), ("h", inter)))
        gate, up = (torch.empty(rows, inter, dtype=torch.bfloat16, device="cuda") for _ in "gu")
        torch.cuda.synchronize()
        for name, out in (("gate", gate), ("up", up)):
            _lib.check(_lib.lib().qie_matmul(C.c_void_p(xn.data_ptr()), C.c_void_p(e.weight_ptr("mlp.%s_proj.weight" % name, 0)[0]), C.c_void_p(out.data_ptr()), rows, hidden,
                                             inter, torch.cuda.current_stream().cuda_stream))
        L.launch_act(gate, gate.numel())
        L.launch_elem(gate, up, gate, gate.numel())
        torch.cuda.synchronize()
        want, got = gate.flatten(), h.flatten()
        if numerics == "fast":
            # another order of the sums: gate, up, SiLU and the product may each round the other way, a bf16 step (2^-8) of at most the largest result
            assert (want.float() - got.float()).abs().max() <= 4 * 2.0 ** -8 * want.float().abs().max()
        else:
            assert torch.equal(want.view(torch.int16), got.view(torch.int16))
        e.close()
