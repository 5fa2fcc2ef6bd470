"""-m gpu: the GEMV decode kernel (csrc/decode_gemv.cu: fast numerics, <= 4 rows, one persistent launch per step)
against the reference-order persistent kernel, which tests/test_gpu_mega.py pins bit for bit to the reference's own
kernels.  Both engines are fed the SAME input tokens every step (the reference-order engine's samples), so a
rounding flip in one sampled token cannot turn into a different continuation.  Tolerance: 1e-2
relative error in bf16 on the logits (||a-b|| / ||b||) for models of <= 3 layers, and the KV rows the kernel stores."""
import numpy as np
import pytest

from util import prompt_ids, rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def qie():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    return q


def _engine(qie, arch, numerics, gemv, context=4096, page_size=16):
    eng = qie.Engine(synthetic=arch, seed=1234, context=context, max_batch_tokens=64, max_seqs=8, use_graph=False,
                     kv_bytes=96 << 20, numerics=numerics, page_size=page_size)
    eng.set_int("mega", 1)
    eng.set_int("gemv", int(gemv))
    return eng


def _run(eng, n_seq, ctxs, n_steps, feed=None, prompts=None):
    seqs = []
    first = []
    for i in range(n_seq):
        s = eng.new_sequence()
        seqs.append(s)
        if prompts is not None:
            first.append(eng.prefill(s, prompts[i]))
        else:
            eng.fill_synthetic(s, ctxs[i], seed=i)
            first.append((37 * i + 11) % eng.config.vocab)
    cur = np.asarray(first, np.int32) if feed is None else feed[0]
    toks, logits = [cur.copy()], []
    for st in range(n_steps):
        out = eng.decode_step(seqs, cur)
        logits.append(eng.read_activation("logits", n_seq * eng.config.vocab))
        toks.append(out.copy())
        cur = out if feed is None else feed[st + 1]
    kv = [eng.kv_read(s, ctxs[i] if prompts is None else len(prompts[i]), n_steps) for i, s in enumerate(seqs)]
    return toks, logits, kv


@pytest.mark.parametrize("arch,n_seq,page_size", [("tiny", 1, 16), ("small", 1, 16), ("small", 2, 8), ("small", 3, 16),
                                                   ("small128", 4, 16), ("small128", 1, 4), ("small", 4, 1)])
def test_gemv_decode_steps_vs_reference_order(qie, arch, n_seq, page_size):
    n_steps = 12
    vocab = qie.make_config(arch).vocab
    prompts = [prompt_ids(5 + 3 * i, vocab, seed=21 + i) for i in range(n_seq)]
    ref = _engine(qie, arch, "reference_order", 0, page_size=page_size)
    want_t, want_l, want_kv = _run(ref, n_seq, None, n_steps, prompts=prompts)
    ref.close()
    eng = _engine(qie, arch, "fast", 1, page_size=page_size)
    assert eng.uses_mega(n_seq, 64)
    # the prefill of the fast engine differs from the reference-order one within tolerance; the decode steps are what
    # this test compares, so they start from the same first token and are fed the reference-order samples
    got_t, got_l, got_kv = _run(eng, n_seq, None, n_steps, feed=want_t, prompts=prompts)
    launches_per_step = eng.launch_count()
    eng.close()
    assert launches_per_step > 0
    for i in range(n_steps):
        assert rel_l2(got_l[i], want_l[i]) < 1e-2, f"logits step {i}"
    for s in range(n_seq):
        assert rel_l2(got_kv[s][0], want_kv[s][0]) < 1e-2 and rel_l2(got_kv[s][1], want_kv[s][1]) < 1e-2
    # greedy samples agree wherever the reference-order top-2 logits are not within a bf16 rounding step of each other
    agree = np.mean([np.mean(g == w) for g, w in zip(got_t[1:], want_t[1:])])
    assert agree > 0.8


@pytest.mark.parametrize("arch,ctxs,page_size", [("small", [122], 16), ("small", [250, 60], 16), ("small128", [60, 125, 251], 8),
                                                 ("small128", [254], 1), ("small", [383, 2], 4)])
def test_gemv_staged_kv_rows_and_bucket_boundaries(qie, arch, ctxs, page_size):
    """contexts up to a KV bucket of 256 run the kernel build that stages the task's first 128 (head_dim 128: 64) cached K / V
    rows in shared memory a phase ahead; the steps below cross the end of the staged rows (the rest is loaded in the
    task), the bucket boundaries 128 -> 256 -> 384 (switch to the build without staging, then to split KV) and ragged rows
    with fewer positions than lanes -- logits of every step against the reference-order kernel"""
    n_seq, n_steps = len(ctxs), 10
    ref = _engine(qie, arch, "reference_order", 0, page_size=page_size)
    want_t, want_l, want_kv = _run(ref, n_seq, ctxs, n_steps)
    ref.close()
    eng = _engine(qie, arch, "fast", 1, page_size=page_size)
    assert eng.uses_mega(n_seq, 64)
    got_t, got_l, got_kv = _run(eng, n_seq, ctxs, n_steps, feed=want_t)
    eng.close()
    for i in range(n_steps):
        assert rel_l2(got_l[i], want_l[i]) < 1e-2, f"logits step {i}"
    for s in range(n_seq):
        assert rel_l2(got_kv[s][0], want_kv[s][0]) < 1e-2 and rel_l2(got_kv[s][1], want_kv[s][1]) < 1e-2


@pytest.mark.parametrize("arch,ctxs", [("small", [700]), ("small", [1500, 33]), ("small128", [2000, 1, 513, 300]),
                                       ("qwen2.5-0.5b", [2048])])
def test_gemv_split_kv_long_context(qie, arch, ctxs):
    """contexts above 256 positions split a (row, head) into several tasks whose partial soft-max results the o_proj
    phase combines; ragged rows leave some splits empty"""
    n_seq, n_steps = len(ctxs), 3
    ref = _engine(qie, arch, "reference_order", 0)
    want_t, want_l, _ = _run(ref, n_seq, ctxs, n_steps)
    ref.close()
    eng = _engine(qie, arch, "fast", 1)
    got_t, got_l, _ = _run(eng, n_seq, ctxs, n_steps, feed=want_t)
    eng.close()
    tol = 1e-2 if qie.make_config(arch).layers <= 3 else 5e-2  # (24 layers: see test_mega_fast_numerics_tolerance)
    for i in range(n_steps):
        assert rel_l2(got_l[i], want_l[i]) < tol, f"logits step {i}"


def test_gemv_equals_itself_under_graph_replay_and_decode_run(qie):
    """the kernel is deterministic: eager steps, CUDA-graph replay and the device-side token feedback of qie_decode_run
    give the same tokens"""
    outs = []
    for use_graph in (False, True):
        eng = qie.Engine(synthetic="small", seed=1234, context=512, max_batch_tokens=64, max_seqs=8, use_graph=use_graph,
                         kv_bytes=64 << 20, numerics="fast")
        seqs = []
        for i in range(2):
            s = eng.new_sequence()
            eng.fill_synthetic(s, 40 + 7 * i, seed=i)
            seqs.append(s)
        outs.append(eng.decode_run(seqs, np.asarray([5, 6], np.int32), 24))
        eng.close()
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.gpu
@pytest.mark.parametrize("arch,n_seq,ctx", [("small", 1, 40), ("small", 3, 300), ("qwen2.5-0.5b", 1, 33), ("qwen2.5-0.5b", 2, 700)])
def test_gemv_polled_buffers_equal_grid_barriers(qie, arch, n_seq, ctx):
    """the phases of the GEMV kernel are chained through polled per-layer buffers (no grid barrier); the same kernel with
    grid barriers between the phases does the same arithmetic, so tokens AND logits must be bit-identical -- over several
    steps (the kernel has to leave the not-stored-yet pattern behind for the next launch) and with split KV partials"""
    res = []
    for dataflow in (1, 0):
        eng = qie.Engine(synthetic=arch, seed=77, context=1024, max_batch_tokens=64, max_seqs=8, use_graph=False,
                         kv_bytes=256 << 20, numerics="fast")
        eng.set_int("gemv_dataflow", dataflow)
        seqs = []
        for i in range(n_seq):
            s = eng.new_sequence()
            eng.fill_synthetic(s, ctx + 5 * i, seed=10 + i)
            seqs.append(s)
        tok = np.arange(n_seq, dtype=np.int32) + 11
        toks, logits = [], []
        for _ in range(6):
            tok = eng.decode_step(seqs, tok)
            toks.append(np.array(tok))
            logits.append(eng.read_activation("logits", n_seq * eng.config.vocab).copy())
        res.append((np.stack(toks), np.stack(logits)))
        eng.close()
    assert np.array_equal(res[0][0], res[1][0])
    assert np.array_equal(res[0][1], res[1][1])
