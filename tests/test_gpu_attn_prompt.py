"""Prompt attention on tcgen05 with 64-key tiles (csrc/attn_prompt_tc.cu) against the reference-order attention, over the edges of tiles, the
split of the keys over a cluster and the border between the two forms of the weights.  Pool rows that no position owns hold NaN.

Bounds: a rounding to bf16 (8 significant bits) is off by at most 2^-8 of the value, and both results are rounded: 2^-7 of the value.  Weights as
bf16 hi + lo pairs are good to 2^-16, the exponentials to 2^-20: 2^-14 of the largest value covers their sum.  Single bf16 weights are off by 2^-8 of
themselves and add up to one: 2^-8 of the largest value."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TWO_TERM = 1024


@pytest.fixture(scope="module")
def layers():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    return L


def check(layers, entry, nq, nkv, hd, first, n, spare=0, scale=1.0):
    g = torch.Generator("cuda").manual_seed(1000 * first + n + hd)
    total = first + n

    def rand(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    pool = layers.KvPool((total + 15) // 16 + spare, 16, 2, nkv, hd, max_seqs=1)
    pool.pool.fill_(float("nan"))
    q, k, v = (scale * rand(n, nq * hd)).bfloat16(), rand(total, nkv * hd).bfloat16(), rand(total, nkv * hd).bfloat16()
    at = torch.arange(total, dtype=torch.int32, device="cuda")
    pool.store(1, k, v, at, torch.zeros_like(at))
    pos, slot = at[first:].contiguous(), torch.zeros(n, dtype=torch.int32, device="cuda")
    want, got = torch.zeros_like(q), torch.full_like(q, float("nan"))
    layers.launch_attn(q, want, pool, 1, pos, slot, nq)
    getattr(layers, entry)(q, got, pool, 1, pos, slot, nq)
    torch.cuda.synchronize()
    top = v.abs().max().double()
    d = (got.double() - want.double()).abs() - 2.0 ** -7 * want.double().abs()
    pairs = entry.endswith("fast") * (torch.arange(n, device="cuda") + first < TWO_TERM)
    assert torch.isfinite(got).all()
    assert (d <= torch.where(pairs, 2.0 ** -14, 2.0 ** -8)[:, None] * top).all(), float(d.max() / top)


@pytest.mark.parametrize("entry,nq,nkv,hd", [("launch_attn_prefill_fast", 14, 2, 64), ("launch_attn_prefill_fast", 3, 3, 64),
                                             ("launch_attn_prefill_fast", 12, 2, 128), ("launch_attn_prefill_tc", 28, 4, 128)])
@pytest.mark.parametrize("first,n", [(0, 1), (0, 63), (0, 64), (0, 65), (0, 129), (127, 1), (128, 130), (300, 100), (950, 200), (1500, 17), (0, 1100), (2050, 300)])
def test_against_reference_order(layers, entry, nq, nkv, hd, first, n):
    check(layers, entry, nq, nkv, hd, first, n)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("spare", [0, 4, 30, 200])
@pytest.mark.parametrize("first,n", [(70, 90), (200, 100), (0, 300)])
def test_more_parts_than_keys(layers, hd, spare, first, n):
    """a block table for more positions than the sequence has: parts of the cluster without a key, parts that a row does not see, query tiles
    that the cluster's first CTA does alone beside others"""
    check(layers, "launch_attn_prefill_fast", 4, 2, hd, first, n, spare)


def test_growing_maxima(layers):
    """scores of a few hundred: the reference maximum moves by more than an exponent's range between tiles"""
    check(layers, "launch_attn_prefill_fast", 2, 1, 64, 0, 700, scale=40.0)


@pytest.mark.parametrize("entry,nq,nkv,hd", [("launch_attn_prefill_fast", 14, 2, 64), ("launch_attn_prefill_fast", 12, 2, 128), ("launch_attn_prefill_tc", 12, 2, 128)])
@pytest.mark.parametrize("first,n", [(0, 1500), (1200, 128)])
def test_same_bits_every_time(layers, entry, nq, nkv, hd, first, n):
    """scores two tiles ahead take the columns of the weights in front: whatever the products' timing, beside other work and on an idle chip, the same
    bits (one query tile with its keys split over a cluster, and many tiles)"""
    g = torch.Generator("cuda").manual_seed(hd + n)
    total = first + n
    pool = layers.KvPool((total + 15) // 16, 16, 1, nkv, hd, max_seqs=1)
    pool.pool.normal_(generator=g)
    q = torch.randn(n, nq * hd, generator=g, device="cuda").bfloat16()
    pos, slot = torch.arange(first, total, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    a = torch.randn(2048, 2048, generator=g, device="cuda").bfloat16()
    side, outs = torch.cuda.Stream(), []
    torch.cuda.synchronize()
    for i in range(40):
        if i % 2:
            with torch.cuda.stream(side):
                a @ a
        outs.append(torch.empty_like(q))
        getattr(layers, entry)(q, outs[-1], pool, 0, pos, slot, nq)
        if i % 4 == 0:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    assert all(torch.equal(o.view(torch.int16), outs[0].view(torch.int16)) for o in outs[1:])


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("lo,hi", [(1000, 1500), (0, 200), (700, 704)])
def test_keys_that_are_not_numbers(layers, hd, lo, hi):
    """parts of the cluster that see nothing else: the row is not a number, as in the reference's order, and does not go on without them"""
    g = torch.Generator("cuda").manual_seed(hd)
    nq, nkv, total, n = 4, 2, 1516, 16
    pool = layers.KvPool((total + 15) // 16, 16, 1, nkv, hd, max_seqs=1)
    k, v = (torch.randn(total, nkv * hd, generator=g, device="cuda").bfloat16() for _ in "kv")
    k[lo:hi, :hd] = float("nan")  # the first kv head
    at = torch.arange(total, dtype=torch.int32, device="cuda")
    pool.store(0, k, v, at, torch.zeros_like(at))
    q = torch.randn(n, nq * hd, generator=g, device="cuda").bfloat16()
    pos, slot = at[total - n:].contiguous(), torch.zeros(n, dtype=torch.int32, device="cuda")
    want, got = torch.zeros_like(q), torch.zeros_like(q)
    layers.launch_attn(q, want, pool, 0, pos, slot, nq)
    layers.launch_attn_prefill_fast(q, got, pool, 0, pos, slot, nq)
    torch.cuda.synchronize()
    assert torch.equal(got.isnan(), want.isnan()) and got.isnan().sum() == n * 2 * hd
