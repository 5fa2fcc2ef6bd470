"""Reference-order attention of few rows (csrc/attn_ref_decode.cu) against one block per row and head (attention_ref_kernel), bit for bit.  The same
cache in pages of 4 positions behind a block table for more positions than other kernels take runs the latter kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu
WIDE = 6000


@pytest.fixture(scope="module")
def layers():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    return L


def ints(v):
    return torch.as_tensor(v, dtype=torch.int32, device="cuda")


def both(layers, nq, nkv, hd, page, lens, rows, spoil=None):
    """rows: (sequence, position); the outputs of the two kernels as integers"""
    g = torch.Generator("cuda").manual_seed(sum(lens) + hd + page)
    q = torch.randn(len(rows), nq * hd, generator=g, device="cuda")
    kv = [[torch.randn(n, nkv * hd, generator=g, device="cuda") for _ in "kv"] for n in lens]
    if spoil:
        spoil(q, kv)
    q, kv = q.bfloat16(), [[x.bfloat16() for x in p] for p in kv]
    got = []
    for psz, most in ((page, max(lens)), (4, WIDE)):
        pages = (most + psz - 1) // psz
        pool = layers.KvPool(pages * len(lens), psz, 2, nkv, hd, max_seqs=len(lens))
        pool.pool.fill_(float("nan"))  # what no sequence wrote is not read
        pool.max_pages, pool.block_table = pages, pool.block_table[:, :pages].contiguous()
        for b, (k, v) in enumerate(kv):
            pool.store(1, k, v, torch.arange(len(k), dtype=torch.int32, device="cuda"), ints([b] * len(k)))
        out = torch.full_like(q, 3.0)
        layers.launch_attn(q, out, pool, 1, ints([p for _, p in rows]), ints([s for s, _ in rows]), nq)
        torch.cuda.synchronize()
        got.append(out.view(torch.int16))
    return got


HEADS = [(14, 2, 64), (12, 2, 128), (3, 3, 64), (5, 1, 128), (18, 2, 64), (28, 4, 128)]


@pytest.mark.parametrize("nq,nkv,hd", HEADS)
@pytest.mark.parametrize("page", [8, 16, 48, 64])
def test_sequences_of_all_lengths(layers, nq, nkv, hd, page):
    """edges of groups of keys (64 or 32), stages of values (128 or 64) and turns of the softmax (128); a row that sees nothing"""
    lens = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 192, 255, 256, 257, 700]
    rows = [(b, n - 1) for b, n in enumerate(lens)] + [(15, -1), (15, 300)]
    a, b = both(layers, nq, nkv, hd, page, lens, rows)
    assert torch.equal(a, b)


@pytest.mark.parametrize("nq,nkv,hd,n", [(14, 2, 64, 1), (14, 2, 64, 5), (14, 2, 64, 20), (14, 2, 64, 70), (14, 2, 64, 100), (12, 2, 128, 9), (16, 1, 64, 30), (28, 4, 128, 40)])
def test_heads_of_a_cta(layers, nq, nkv, hd, n):
    """one to eight heads a CTA, one or two a warp, by the number of rows; the longest ring of values and more than one wave"""
    lens = [1100 + 13 * (i % 7) for i in range(n)]
    a, b = both(layers, nq, nkv, hd, 16, lens, [(i, m - 1) for i, m in enumerate(lens)])
    assert torch.equal(a, b)


def small(q, kv):  # products below the smallest normal number
    for k, _ in kv:
        k *= 2.0 ** -130


def large(q, kv):  # products that overflow, sums that come back
    q[:, ::2] *= 2.0 ** 70
    for k, _ in kv:
        k[::3] *= 2.0 ** 66


def zeros(q, kv):
    q[0] = 0
    for k, v in kv:
        k[::5] = 0
        v[:, ::4] = -0.0


def peaked(q, kv):  # exponentials of zero and of few bits
    q *= 40


def no_numbers(q, kv):
    kv[0][0][10, 3] = float("nan")
    kv[1][1][20, 7] = float("inf")
    kv[2][0][5, ::9] = float("-inf")


@pytest.mark.parametrize("spoil", [small, large, zeros, peaked, no_numbers])
@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (12, 2, 128)])
def test_values_at_the_edges(layers, nq, nkv, hd, spoil):
    lens = [90, 150, 300]
    a, b = both(layers, nq, nkv, hd, 16, lens, [(i, m - 1) for i, m in enumerate(lens)], spoil)
    nan = [(x.view(torch.bfloat16).isnan()) for x in (a, b)]  # (a NaN's payload is not defined)
    assert torch.equal(nan[0], nan[1]) and torch.equal(a[~nan[0]], b[~nan[1]])
