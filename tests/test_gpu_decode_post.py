"""Decode steps whose attention kernel does the head norms, the positions and the store (csrc/attn_ref_decode.cu) against steps that launch qkv_post_kernel in
front of it (the engine's captures of q and v): logits and tokens bit for bit, at edges of the groups of keys and of the stages of values, over steps that read
what earlier ones stored.  Heads of 128 have two launches either way, by graphs and by launches."""
import numpy as np
import pytest

from hf_util import make_hf_checkpoint

pytestmark = pytest.mark.gpu

LENS = [1, 2, 30, 31, 32, 62, 63, 64, 65, 126, 127, 128, 254, 255, 256, 300]


@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (12, 2, 128), (4, 4, 64), (9, 1, 64)])
@pytest.mark.parametrize("batch", [1, 5, 16, 70])
@pytest.mark.parametrize("page", [8, 16, 48])
def test_against_two_kernels(nq, nkv, hd, batch, page):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(hidden=256, inter=512, layers=2, n_q=nq, n_kv=nkv, head_dim=hd, vocab=2048), context=512)
    got, launches = [], []
    for capture in (False, True):
        e = q.Engine(synthetic=cfg, seed=3, context=512, max_seqs=batch, max_batch_tokens=batch, max_pages=batch * (320 // page + 2), page_size=page)
        e.set_int("mega", 0)
        e.capture(capture)
        seqs = [e.new_sequence() for _ in range(batch)]
        for i, s in enumerate(seqs):
            e.fill_synthetic(s, LENS[(i + batch) % len(LENS)], seed=100 + i)
        tokens, out = np.arange(batch, dtype=np.int32) + 7, []
        for _ in range(4):
            tokens = e.decode_step(seqs, tokens)
            out.append((np.array(tokens), e.read_activation("logits", batch * 2048)))
        launches.append(e.launch_count())
        e.close()
        got.append(out)
    assert launches[1] - launches[0] == (2 if hd == 64 else 0)  # a launch a layer
    for (t0, l0), (t1, l1) in zip(*got):
        assert np.array_equal(t0, t1)
        assert np.array_equal(l0.view(np.uint16), l1.view(np.uint16))


@pytest.mark.parametrize("kind", ["qwen2", "qwen3"])
def test_biases_and_halves(tmp_path, kind):
    """projection biases without head norms, and the half rotation"""
    torch = pytest.importorskip("torch")
    pytest.importorskip("transformers")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    _, meta, wts = make_hf_checkpoint(kind, str(tmp_path))
    got = []
    for capture in (False, True):
        e = q.Engine(meta, wts, head_dim_hint=64, context=512, max_batch_tokens=64, kv_bytes=64 << 20, semantics="hf")
        e.capture(capture)
        seqs = [e.new_sequence() for _ in range(3)]
        tokens = [e.prefill(s, np.arange(1, n + 1, dtype=np.int32)) for s, n in zip(seqs, (1, 31, 63))]
        out = []
        for _ in range(4):
            tokens = e.decode_step(seqs, tokens)
            out.append((np.array(tokens), e.read_activation("logits", 3 * 1024)))
        e.close()
        got.append(out)
    for (t0, l0), (t1, l1) in zip(*got):
        assert np.array_equal(t0, t1)
        assert np.array_equal(l0.view(np.uint16), l1.view(np.uint16))


@pytest.mark.parametrize("nq,nkv,hd,batch", [(16, 16, 64, 90), (8, 8, 128, 170), (16, 1, 64, 200), (9, 1, 64, 230), (16, 1, 128, 256)])
@pytest.mark.parametrize("first", [1, 120])
def test_many_rows_of_short_contexts(nq, nkv, hd, batch, first):
    """several waves of CTAs at contexts where the steps go to other kernels (attention_ref_decode_step), and over the end of that range, against steps of a few rows: tokens and logits
    bit for bit"""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(hidden=256, inter=512, layers=2, n_q=nq, n_kv=nkv, head_dim=hd, vocab=2048), context=512)
    got = []
    for portion in (batch, 8):
        e = q.Engine(synthetic=cfg, seed=3, context=512, max_seqs=batch, max_batch_tokens=batch, max_pages=batch * 12)
        e.set_int("mega", 0)
        seqs = [e.new_sequence() for _ in range(batch)]
        for i, s in enumerate(seqs):
            e.fill_synthetic(s, first + i % 7, seed=100 + i)
        tokens, out = np.arange(batch, dtype=np.int32) + 7, []
        for _ in range(8):
            step = [(np.array(e.decode_step(seqs[b:b + portion], tokens[b:b + portion])), e.read_activation("logits", len(seqs[b:b + portion]) * 2048)) for b in range(0, batch, portion)]
            tokens = np.concatenate([t for t, _ in step])
            out.append((tokens, np.concatenate([x for _, x in step])))
        e.close()
        got.append(out)
    for (t0, l0), (t1, l1) in zip(*got):
        assert np.array_equal(t0, t1)
        assert np.array_equal(l0.view(np.uint16), l1.view(np.uint16))
