"""Reference-order attention of several rows per CTA (csrc/attn_ref_rows.cu) against one block per row and head (attention_ref_kernel), bit
for bit.  The same cache behind a block table for more positions than the tiles take runs the latter kernel."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
WIDE = 6000  # positions of a table that leaves every row to attention_ref_kernel


@pytest.fixture(scope="module")
def layers():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    return L


def ints(v):
    return torch.as_tensor(v, dtype=torch.int32, device="cuda")


def both(layers, nq, nkv, hd, page, lens, rows, seed, spoil=None):
    """rows: (sequence, position); the outputs of the two kernels as integers, and the queries, keys, values"""
    g = torch.Generator("cuda").manual_seed(seed)
    kv = [[torch.randn(n, nkv * hd, generator=g, device="cuda") for _ in "kv"] for n in lens]
    if spoil:
        spoil(kv)
    kv = [[x.bfloat16() for x in p] for p in kv]
    q = torch.randn(len(rows), nq * hd, generator=g, device="cuda").bfloat16()
    got = []
    for most in (max(lens), WIDE):
        pool = layers.KvPool((most + page - 1) // page * len(lens), page, 2, nkv, hd, max_seqs=len(lens))
        if most != WIDE:
            pool.max_pages = (most + page - 1) // page
            pool.block_table = pool.block_table[:, :pool.max_pages].contiguous()
        for b, (k, v) in enumerate(kv):
            pool.store(1, k, v, torch.arange(len(k), dtype=torch.int32, device="cuda"), ints([b] * len(k)))
        out = torch.full_like(q, 3.0)
        layers.launch_attn(q, out, pool, 1, ints([p for _, p in rows]), ints([s for s, _ in rows]), nq)
        torch.cuda.synchronize()
        got.append(out.view(torch.int16))
    return got, q, kv


@pytest.mark.parametrize("nq,nkv,hd,page", [(14, 2, 64, 16), (4, 4, 64, 16), (16, 1, 64, 4), (32, 1, 64, 16), (12, 2, 128, 16), (28, 4, 128, 3), (16, 2, 256, 16)])
@pytest.mark.parametrize("first,n", [(0, 1), (0, 2), (63, 3), (0, 65), (300, 33), (0, 400), (1000, 9)])
def test_rows_of_one_sequence(layers, nq, nkv, hd, page, first, n):
    got, _, _ = both(layers, nq, nkv, hd, page, [first + n], [(0, first + i) for i in range(n)], 7 * first + n + hd)
    assert torch.equal(got[0], got[1])


def infinite_later(kv):  # values behind a row's own positions may be anything
    for k, v in kv:
        v[len(v) // 2:] = float("inf")
        k[-2:, ::3] = float("nan")


def tiny(kv):
    for k, _ in kv:
        k *= 2.0 ** -130


@pytest.mark.parametrize("spoil", [None, infinite_later, tiny])
@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (8, 4, 128)])
def test_rows_of_several_sequences(layers, nq, nkv, hd, spoil):
    """tiles with rows of one sequence beside tiles that several share, positions in any order"""
    rows = [(0, i) for i in range(40, 100)] + [(1, 36), (2, 255), (3, 199), (1, 5)] + [(2, i) for i in range(250, 180, -1)] + [(3, 37 * i % 200) for i in range(41)]
    got, _, _ = both(layers, nq, nkv, hd, 16, [100, 37, 256, 200], rows, hd, spoil)
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (12, 2, 128), (8, 2, 256)])
def test_rows_that_see_nothing(layers, nq, nkv, hd):
    """rows at position -1 (nothing to attend to) give zeros, in tiles of their own and beside others"""
    rows = [(0, -1)] * 40 + [(0, i) for i in range(17)] + [(0, -1), (0, 30), (0, -1)] + [(0, -1)] * 33
    got, _, _ = both(layers, nq, nkv, hd, 16, [40], rows, hd)
    assert torch.equal(got[0], got[1])
    assert not got[0][torch.tensor([p < 0 for _, p in rows], device="cuda")].any()


@pytest.mark.parametrize("offset", [0, 2])
@pytest.mark.parametrize("hd,n", [(64, 50), (128, 21)])
def test_page_list(layers, hd, n, offset):
    """the reference's page layout [slot][layer][kv_dim], pages on and off a 16-byte boundary"""
    from qwen_inference_engine_b200 import _lib
    nq, nkv, page, n_layers, layer = 6, 2, 4, 3, 1
    got, q, kv = both(layers, nq, nkv, hd, 16, [n], [(0, i) for i in range(n)], n)
    dkv, n_pages = nkv * hd, (n + page - 1) // page
    lists, keep = [], []
    for x in kv[0]:
        whole = torch.zeros(n_pages, page * n_layers * dkv + 8, dtype=torch.bfloat16, device="cuda")
        for p in range(n):
            at = offset + (p % page * n_layers + layer) * dkv
            whole[p // page, at:at + dkv] = x[p]
        keep.append(whole)
        lists.append(torch.tensor([whole[i].data_ptr() + 2 * offset for i in range(n_pages)], dtype=torch.int64, device="cuda"))
    out = torch.zeros_like(q)
    pos = torch.arange(n, dtype=torch.int32, device="cuda")
    lib = _lib.lib()
    _lib.check(lib.qie_attention_pagelist(C.c_void_p(lists[0].data_ptr()), C.c_void_p(lists[1].data_ptr()), n_pages, page, n_layers, layer, nkv, hd,
                                          C.c_void_p(q.data_ptr()), C.c_void_p(out.data_ptr()), C.c_void_p(pos.data_ptr()), n, nq,
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert np.array_equal(out.view(torch.int16).cpu().numpy(), got[1].cpu().numpy())


@pytest.mark.parametrize("nq,nkv,hd,n", [(14, 2, 64, 400), (14, 2, 64, 3), (12, 2, 128, 5), (16, 2, 256, 7)])
@pytest.mark.parametrize("end", [17, 63, 64, 65, 127, 128, 129, 255, 257, 300])
def test_softmax_where_the_last_turn_is_short(layers, nq, nkv, hd, n, end):
    """a thread's eight positions of a turn reach behind the end, by one to all but one"""
    n = min(n, end)
    got, _, _ = both(layers, nq, nkv, hd, 16, [end], [(0, end - n + i) for i in range(n)], end + hd)
    assert torch.equal(got[0], got[1])
