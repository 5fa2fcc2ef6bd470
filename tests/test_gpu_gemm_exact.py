"""Reference-order products on the tcgen05 kernels (csrc/gemm_tcgen05.cu, launch_gemm_ref_rows): the bits of the mma.sync chain at every
row count, tile width and output alignment.  No tolerance: the order is defined."""
import numpy as np
import pytest
import torch

from util import prompt_ids

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layers():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    return L


def draw(shape, kind, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    r = torch.randn(shape, generator=g, device="cuda")
    if kind == "wide":  # magnitudes over 2^+-40 or so
        r = r * torch.exp2(12 * torch.randn(shape, generator=g, device="cuda"))
    if kind == "small":  # subnormal products and sums
        r = r * 2.0 ** -66
    if kind == "special":
        r[::3, 5] = float("inf")
        r[::5, 7] = float("nan")
        r[:, 9] = -0.0
    return r.bfloat16()


def matmul(layers, a, b):
    out = torch.full((a.shape[0], b.shape[0]), 7.0, dtype=torch.bfloat16, device="cuda")
    layers.launch_matmul(a, b, out, a.shape[0], a.shape[1], b.shape[0])
    torch.cuda.synchronize()
    return out.view(torch.int16)


@pytest.mark.parametrize("kind", ["normal", "wide", "small", "special"])
@pytest.mark.parametrize("rows", [1, 8, 17, 64, 200])
def test_same_bits_as_the_mma_sync_kernel(layers, rows, kind):
    """An inner dimension below one k-block takes the mma.sync kernel; with zeros appended up to a k-block (two for up to 8 rows) the same sums take tcgen05
    (a product with zeros leaves an accumulator as it is; infinities stay out of the zero columns)."""
    a, b = draw((rows, 56), kind, 3 + rows), draw((520, 56), "normal" if kind == "special" else kind, 4)
    pad, more = torch.nn.functional.pad, 8 if rows > 8 else 72
    assert torch.equal(matmul(layers, a, b), matmul(layers, pad(a, (0, more)), pad(b, (0, more))))


@pytest.mark.parametrize("kind", ["normal", "wide", "small"])
@pytest.mark.parametrize("rows", [1, 5, 8])
def test_same_bits_over_more_than_one_block(layers, rows, kind):
    """up to 8 rows of less than two k-blocks take the mma.sync kernel too: chains of 5 to 7 products against two blocks of a tcgen05 tile"""
    pad = torch.nn.functional.pad
    for inner in (72, 104, 120):
        a, b = draw((rows, inner), kind, inner + rows), draw((1000, inner), kind, inner)
        assert torch.equal(matmul(layers, a, b), matmul(layers, pad(a, (0, 136 - inner)), pad(b, (0, 136 - inner))))


@pytest.mark.parametrize("inner,outer", [(896, 4864), (4864, 896), (72, 20000), (1536, 264)])
@pytest.mark.parametrize("rows", [2, 16, 33, 129, 300, 1000])
def test_rows_and_tiles_do_not_matter(layers, rows, inner, outer):
    """every tile width, the persistent kernel and one tile per CTA: a row's result is that of the row alone; an odd number of outputs
    (2-byte stores) gives the first columns of the aligned result"""
    a, b = draw((rows, inner), "normal", rows), draw((outer, inner), "normal", 1)
    whole = matmul(layers, a, b)
    for r in {0, rows // 2, rows - 1}:
        assert torch.equal(matmul(layers, a[r:r + 1].clone(), b)[0], whole[r])
    cut = rows // 3 + 1
    assert torch.equal(matmul(layers, a[:cut].clone(), b), whole[:cut])
    assert torch.equal(matmul(layers, a, b[:outer - 3].clone()), whole[:, :outer - 3])


@pytest.mark.parametrize("batch", [1, 8, 9, 33, 64])
def test_operators_equal_the_persistent_kernel(layers, batch):
    """one decode step, projections of every kind (three segments, residual, gate and up): operators on tcgen05 against the persistent
    kernel's mma.sync chains; logits and tokens bit for bit"""
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(hidden=896, inter=4864, layers=1, n_q=14, n_kv=2, head_dim=64, vocab=4096), context=256)
    got = []
    for mega in (1, 0):
        e = q.Engine(synthetic=cfg, seed=5, context=256, max_seqs=batch, max_batch_tokens=max(batch, 64), max_pages=batch * 4)
        e.set_int("mega", mega)
        seqs = [e.new_sequence() for _ in range(batch)]
        first = [e.prefill(s, prompt_ids(3 + i % 7, 4096, seed=i)) for i, s in enumerate(seqs)]
        assert e.uses_mega(batch, 16) == bool(mega)
        tokens = e.decode_step(seqs, first)
        got.append((first, tokens.tolist(), e.read_activation("logits", batch * 4096)))
        e.close()
    assert got[0][:2] == got[1][:2]
    assert np.array_equal(got[0][2], got[1][2])
