"""Sampling with a cluster of CTAs per row (csrc/ops_ref_order.cu, sample_topk_cluster_kernel) against the C restatement of the reference's
sampler: rows on and off a 16-byte boundary, ties, rows that overflow the candidate lists, rows with fewer candidates than k."""
import numpy as np
import pytest
import torch

from util import bf16_to_f32, f32_to_bf16, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layers():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    return L


def row(kind, vocab, rng, ctas=8):
    x = rng.standard_normal(vocab).astype(np.float32) * 2.5
    if kind == "ties":
        x = np.round(x)
    if kind == "equal":  # every value is a candidate: more than a slice's list holds
        x[:] = 1.5
    if kind == "few":
        x[:] = -np.inf
        x[rng.integers(0, vocab, size=7)] = rng.standard_normal(7)
    if kind == "one slice":  # all large values side by side
        x[vocab // 2:vocab // 2 + 300] += 40
    if kind == "zeros":
        x = np.where(x > 3, 0.0, -0.0) - (x < 0)
    if kind == "two values":  # ties at the top over all slices, fewer than k above them
        x = np.where(rng.random(vocab) < 0.5, 2.0, np.minimum(x, 1.0)).astype(np.float32)
        x[rng.integers(0, vocab, size=3)] = 5.0
    if kind == "few threads":  # more large values than a list holds, in the 16-byte pieces of 30 threads of a slice
        piece = np.arange(vocab) // 8
        x[piece % max(1, (vocab // 8 + ctas - 1) // ctas) % 512 < 30] += 25
    return f32_to_bf16(x)


@pytest.mark.parametrize("kind", ["normal", "ties", "equal", "few", "one slice", "zeros", "two values", "few threads"])
@pytest.mark.parametrize("vocab,rows", [(151936, 3), (32001, 5), (8200, 2), (6001, 20), (1000, 2), (519, 9)])
@pytest.mark.parametrize("k", [1, 2, 50, 128])
def test_rows_against_the_restatement(layers, oracle, vocab, rows, kind, k):
    rng = np.random.default_rng(vocab + k)
    lg = np.stack([row(kind, vocab, rng) for _ in range(rows)])
    for seed in (1234, 77):
        got = layers.sample_topk_bf16(to_dev(lg), vocab, 0.7, k, seed)
        for r in range(rows):
            want = oracle.argmax_tiebreak(lg[r]) if k == 1 else oracle.sample_topk(lg[r], 0.7, k, seed)
            assert got[r] == want, (r, seed)


def test_nothing_to_choose(layers):
    x = np.full((2, 4099), -np.inf, np.float32)
    x[1, 4098] = 3
    assert layers.sample_topk_bf16(to_dev(f32_to_bf16(x)), 4099, 1.0, 50, 1).tolist() == [-1, 4098]
    assert np.isinf(bf16_to_f32(f32_to_bf16(x))[0]).all()


def some_rows(layers, oracle, lg, vocab, k, seed, check):
    """rows against the restatement; the others are copies, and the same row gives the same token wherever it stands"""
    got = layers.sample_topk_bf16(to_dev(lg), vocab, 0.7, k, seed)
    for r in check:
        want = oracle.argmax_tiebreak(lg[r]) if k == 1 else oracle.sample_topk(lg[r], 0.7, k, seed)
        assert got[r] == want, (r, seed)
    assert np.array_equal(got, np.tile(got[:len(check)], len(got) // len(check) + 1)[:len(got)])


@pytest.mark.parametrize("kind", ["normal", "ties", "few"])
@pytest.mark.parametrize("rows", [17, 33, 70])
@pytest.mark.parametrize("vocab,k", [(1023, 128), (1040, 64), (2056, 128), (2064, 128), (2303, 128), (2304, 128), (4095, 120)])
def test_slices_of_hardly_more_pieces_than_k(layers, oracle, vocab, k, rows, kind):
    rng = np.random.default_rng(vocab + rows)
    lg = np.stack([row(kind, vocab, rng) for _ in range(5)])
    some_rows(layers, oracle, np.tile(lg, (rows // 5 + 1, 1))[:rows], vocab, k, 1234, range(5))


@pytest.mark.parametrize("k", [1, 2, 50, 128])
@pytest.mark.parametrize("vocab,rows,ctas", [(151936, 4, 8), (151936, 5, 8), (151936, 8, 8), (151936, 9, 4), (151936, 16, 4), (151936, 17, 4), (151936, 32, 4), (151936, 33, 2),
                                             (151936, 64, 2), (155655, 9, 4), (155655, 33, 2), (155656, 2, 8), (155656, 17, 8), (262144, 3, 8), (262144, 17, 8), (65536, 16, 4),
                                             (32001, 12, 4), (32001, 40, 2)])
def test_every_cluster_size_and_both_sides_of_its_rules(layers, oracle, vocab, rows, ctas, k):
    """slices of two, four and eight CTAs with and without the copy in shared memory, on and off a 16-byte boundary, lists that overflow, hardly any candidates;
    greedy rows in 64, 32 and 8 slices (k = 1, whole pieces)"""
    rng = np.random.default_rng(vocab + rows + k)
    lg = np.stack([row(kind, vocab, rng, ctas) for kind in ("few threads", "ties", "normal", "equal", "few")])
    for at in range(0, 5, rows):
        part = lg[at:at + rows]
        some_rows(layers, oracle, np.tile(part, (rows // len(part) + 1, 1))[:rows], vocab, k, 77, range(len(part)))
