"""CUDA graphs of decode steps (capi.cu, decode_launch): taken over by longer contexts, given up where there are too many, made anew; tokens and logits are those of
launches without graphs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MOST = 16384  # GRAPH_KERNELS


def engines(q, arch, seqs, positions, **kw):
    for graph in (True, False):
        e = q.Engine(synthetic=q.make_config(arch, context=4096), seed=5, context=4096, max_seqs=seqs, max_batch_tokens=64, use_graph=graph, max_pages=seqs * (positions // 16 + 2), **kw)
        yield graph, e
        e.close()


@pytest.mark.parametrize("numerics", ["reference_order", "fast"])
def test_contexts_that_grow_and_batches_in_turn(numerics):
    """three batches: one of 12 that grows over three multiples of 128, one as large at shorter contexts in turn with it (its graph is taken over and comes back), one of
    changing size"""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    got = []
    for graph, e in engines(q, "small", 24, 900, numerics=numerics):
        a, b = ([e.new_sequence() for _ in range(12)] for _ in "ab")
        for i, s in enumerate(a + b):
            e.fill_synthetic(s, 230 + i if i < 12 else 20 + i, seed=i)
        ta, tb, out = np.arange(12, dtype=np.int32), np.arange(12, dtype=np.int32) + 40, []
        for step in range(300):
            ta = e.decode_step(a, ta)
            out.append((np.array(ta), e.read_activation("logits", 12 * e.config.vocab)))
            if step >= 40:
                tb = e.decode_step(b, tb)
                out.append((np.array(tb), e.read_activation("logits", 12 * e.config.vocab)))
            if step >= 200 and step % 7 == 0:
                n = 1 + step % 11
                out.append((np.array(e.decode_step(b[:n], tb[:n])), e.read_activation("logits", n * e.config.vocab)))
        assert (e.decode_graph_kernels() > 0) == graph
        if graph and numerics == "reference_order":
            assert e.decode_graph_kernels() <= 6 * e.launch_count()  # two that change hands, and the sizes that came often enough
        e.set_int("mega", -1)
        assert e.decode_graph_kernels() == 0
        got.append(out)
    assert all(np.array_equal(t0, t1) and np.array_equal(l0, l1) for (t0, l0), (t1, l1) in zip(*got))


def test_a_bounded_number_of_graphs():
    """more shapes in turn than graphs are kept: 64 batch sizes at eleven lengths"""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    got = []
    for graph, e in engines(q, "small", 64 * 11, 1500):
        groups, out, most = [], [], 0
        for k in range(11):
            groups.append([e.new_sequence() for _ in range(64)])
            for i, s in enumerate(groups[-1]):
                e.fill_synthetic(s, 10 + 128 * k + (i & 1), seed=i)
        for rounds in range(14):
            for n in range(1, 65):
                for seqs in groups:
                    out.append(np.array(e.decode_step(seqs[64 - n:], np.arange(n, dtype=np.int32) + rounds)))
                most = max(most, e.decode_graph_kernels())
        assert most <= MOST
        assert not graph or most > MOST // 2
        got.append(out)
    assert all(np.array_equal(t0, t1) for t0, t1 in zip(*got))


@pytest.mark.parametrize("batch", [1, 20])
def test_runs_without_waits_between_steps(batch):
    """decode_run over several multiples of 128 positions: graphs are taken over while earlier launches of them are on their way"""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    got = []
    for graph, e in engines(q, "small", batch, 800):
        seqs = [e.new_sequence() for _ in range(batch)]
        for i, s in enumerate(seqs):
            e.fill_synthetic(s, 100 - i, seed=i)
        got.append(np.array(e.decode_run(seqs, np.arange(batch, dtype=np.int32), 600)))
        assert graph == (e.decode_graph_kernels() > 0)
        assert not graph or e.decode_graph_kernels() < 100  # one graph, which five lengths had in turn
    assert np.array_equal(*got)
