"""Reference-order attention of several rows per CTA (csrc/attn_ref_rows.cu) where its fused products would round differently from products and sums, and
over a pool off a 16-byte boundary, against one block per row and head (attention_ref_kernel), bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
WIDE = 6000  # positions of a table that leaves every row to attention_ref_kernel


def ints(v):
    return torch.as_tensor(v, dtype=torch.int32, device="cuda")


def both(nq, nkv, hd, n, q, k, v, off=0):
    """outputs of the two kernels for n rows of one sequence"""
    from qwen_inference_engine_b200 import layers as L
    got = []
    for most in (n, WIDE):
        pool = L.KvPool((most + 15) // 16, 16, 1, nkv, hd, max_seqs=1)
        if most == n and off:
            pool.store_at = torch.zeros(pool.pool.numel() + 8, dtype=torch.bfloat16, device="cuda")
            pool.view.pool = pool.store_at.data_ptr() + 2 * off
        pool.store(0, k, v, torch.arange(n, dtype=torch.int32, device="cuda"), ints([0] * n))
        out = torch.full_like(q, 3.0)
        L.launch_attn(q, out, pool, 0, ints(range(n)), ints([0] * n), nq)
        torch.cuda.synchronize()
        got.append(out.view(torch.int16))
    return got


def inputs(nq, nkv, hd, n, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    return [torch.randn(n, w * hd, generator=g, device="cuda") for w in (nq, nkv, nkv)]


@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (12, 2, 128), (16, 2, 256)])
@pytest.mark.parametrize("scale_q,scale_k,first", [(2.0 ** -70, 2.0 ** -70, 0), (2.0 ** -60, 2.0 ** -75, 150), (2.0 ** 66, 2.0 ** 62, 150), (1.0, 2.0 ** 100, 150), (1.0, 0.0, 70)])
def test_products_beyond_the_fused_range(nq, nkv, hd, scale_q, scale_k, first):
    """keys from `first` on are scaled: tiles in front of them still take the fused products"""
    q, k, v = inputs(nq, nkv, hd, 200, hd + first)
    q *= scale_q
    k[first:] *= scale_k
    k[first::5, ::7] = 0.0
    a, b = both(nq, nkv, hd, 200, q.bfloat16(), k.bfloat16(), v.bfloat16())
    assert torch.equal(a, b)


@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (12, 2, 128), (16, 2, 256)])
@pytest.mark.parametrize("n", [17, 63, 65, 130])
def test_pool_off_a_16_byte_boundary(nq, nkv, hd, n):
    q, k, v = (x.bfloat16() for x in inputs(nq, nkv, hd, n, n))
    a, b = both(nq, nkv, hd, n, q, k, v, off=2)
    assert torch.equal(a, b)
