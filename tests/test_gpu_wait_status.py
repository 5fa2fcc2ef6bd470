"""A wait inside a kernel that runs out (csrc/tc_ptx.cuh) is an error of the call that learns of it, once, and the context stays usable.  The
self-test's wait is on a barrier that nothing completes, through the limit and the report that the tcgen05 kernels use.  It is a pair of CTAs as the GEMM's are: the
first one waits and the other one, which waits for nothing, reports what it was told (tell_other_tc)."""
import numpy as np
import pytest
import torch

from util import prompt_ids

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import _lib
    return _lib


def test_an_operator_learns_of_it(lib):
    from qwen_inference_engine_b200 import layers
    L = lib.lib()
    a, b, out = (torch.ones(s, dtype=torch.bfloat16, device="cuda") for s in ((4, 64), (8, 64), (4, 8)))
    assert L.qie_kernel_status() == 0
    assert L.qie_wait_selftest(None, None) == 0
    torch.cuda.synchronize()
    assert L.qie_kernel_status() < 0 and b"ran out" in L.qie_last_error()
    assert L.qie_kernel_status() == 0
    for f in (layers.launch_matmul, layers.launch_matmul_fast):
        assert L.qie_wait_selftest(None, None) == 0
        torch.cuda.synchronize()
        with pytest.raises(lib.QieError, match="ran out"):
            f(a, b, out, 4, 64, 8)
        f(a, b, out, 4, 64, 8)
        torch.cuda.synchronize()
        assert (out == 64).all() and L.qie_kernel_status() == 0


def test_an_engine_learns_of_its_own(lib):
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(hidden=896, inter=4864, layers=1, n_q=14, n_kv=2, head_dim=64, vocab=4096), context=256)
    one, other = (q.Engine(synthetic=cfg, seed=5, context=256, max_seqs=2, max_batch_tokens=64, max_pages=16) for _ in range(2))
    ids = prompt_ids(20, 4096, seed=1)
    want = one.prefill(one.new_sequence(), ids)
    assert lib.lib().qie_wait_selftest(one._h, None) < 0 and b"this engine" in lib.lib().qie_last_error()
    assert lib.lib().qie_kernel_status() == 0
    for e in (other, one):
        s = e.new_sequence()
        assert e.prefill(s, ids) == want
        assert np.asarray(e.decode_step([s], [want])).size == 1
        e.close()
