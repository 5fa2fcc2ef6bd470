"""-m gpu: the FAST-numerics kernels (tcgen05/TMEM/TMA GEMM with split-K, split-KV
flash-decoding, parallel RMSNorm) against the reference's own kernels and the
reference-order path.  These kernels change the fp32 summation order, so the bar is a
tolerance -- 1e-2 relative error in bf16 -- and it is written here."""
import numpy as np
import pytest

from util import bf16_to_f32, prompt_ids, rand_bf16, rel_err, rel_l2, to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL_BF16 = 1e-2      # relative error in bf16 (||a-b||/||b|| for a tensor; max-norm for one op)
TOL_MAXNORM = 3.2e-2  # whole-forward sanity bound: max|a-b|/max|b| <= 4 bf16 ulps of the largest value
                      # (two pipelines that round to bf16 ~20 times per layer differ by an ulp or two per element)


def close(a, b):
    return rel_l2(a, b) < TOL_BF16 and rel_err(a, b) < TOL_MAXNORM


@pytest.fixture(scope="module")
def layers():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from qwen_inference_engine_b200 import layers as L
    return L


def p(t):
    return t.data_ptr()


@pytest.mark.parametrize("M,N,K", [(64, 896, 896), (64, 896, 128), (64, 896, 4864), (64, 4864, 896), (9, 896, 1152),
                                   (16, 1536, 256), (17, 128, 384), (32, 896, 9728), (33, 256, 640), (128, 896, 896),
                                   (130, 512, 264), (256, 1536, 1536), (300, 896, 896), (64, 896, 15104), (40, 64, 128),
                                   (64, 3584, 3584), (600, 1536, 8960), (1000, 512, 2568)])
def test_tcgen05_gemm_vs_reference_kernel(layers, ref, M, N, K):
    """C[M,K] = A[M,N] @ B[K,N]^T : tcgen05 path vs the reference's wmma kernel."""
    rng = np.random.default_rng(M * 7919 + N * 13 + K)
    A = rand_bf16(rng, (M, N), 1.0)
    B = rand_bf16(rng, (K, N), 0.05)
    Ad, Bd = to_dev(A), to_dev(B)
    c_ref = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    c_new = torch.full((M, K), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert ref.L.ref_matmul(p(Ad), p(Bd), p(c_ref), M, N, K) == 0
    layers.launch_matmul_fast(Ad, Bd, c_new, M, N, K)
    torch.cuda.synchronize()
    got, want = to_host(c_new), to_host(c_ref)
    assert not np.isnan(bf16_to_f32(got)).any()
    assert rel_err(got, want) < TOL_BF16
    # most elements are even bit-identical to the reference (the sum order only moves values that sit
    # on a bf16 rounding boundary)
    assert np.mean(got == want) > 0.9


@pytest.mark.parametrize("hd,n_q,n_kv,B,t,splits", [(64, 14, 2, 4, 300, 1), (64, 14, 2, 3, 1000, 4), (64, 14, 2, 2, 64, 0),
                                                     (64, 14, 2, 5, 1, 2), (128, 12, 2, 3, 515, 3), (128, 28, 4, 2, 130, 0),
                                                     (64, 4, 4, 2, 77, 5), (64, 16, 1, 2, 200, 2),
                                                     # clusters of every size, more splits than tiles, the combining kernel, what `0` picks at length
                                                     (64, 14, 2, 2, 100, 6), (128, 12, 2, 2, 700, 7), (64, 14, 2, 3, 700, 8), (64, 4, 2, 2, 1000, 12),
                                                     (128, 12, 2, 1, 1500, 16), (64, 14, 2, 2, 300, 16), (64, 14, 2, 2, 2300, 24), (128, 4, 2, 2, 900, 40),
                                                     (64, 14, 2, 2, 4200, 0), (128, 28, 4, 1, 4100, 0), (64, 14, 2, 40, 600, 16),
                                                     # as many splits as find room at once: 8, 7, 6, 5, 4, 3, 2 of them, three CTAs an SM, and 4 that
                                                     # find none as clusters
                                                     (64, 14, 2, 20, 260, 0), (64, 14, 2, 36, 500, 0), (64, 14, 2, 40, 600, 0), (64, 14, 2, 60, 700, 0),
                                                     (64, 14, 2, 70, 600, 0), (128, 12, 2, 16, 220, 0), (128, 12, 2, 17, 300, 0), (128, 12, 2, 20, 300, 0),
                                                     (128, 12, 2, 24, 330, 0), (128, 12, 2, 36, 480, 0), (128, 12, 2, 48, 640, 0), (128, 12, 2, 36, 480, 4)])
def test_flash_decoding_vs_reference_order_attention(layers, hd, n_q, n_kv, B, t, splits):
    """ragged batch: sequence b has t - 13*b (>=1) cached positions."""
    rng = np.random.default_rng(hd + n_q + t)
    Dq, Dkv = n_q * hd, n_kv * hd
    n_layers, layer = 2, 1
    ps = 16
    lens = [max(1, t - 13 * b) for b in range(B)]
    pool = layers.KvPool(n_pages=B * ((t + ps - 1) // ps + 1), page_size=ps, n_layers=n_layers, n_kv_heads=n_kv,
                         head_dim=hd, max_seqs=B)
    for b in range(B):
        K = rand_bf16(rng, (lens[b], Dkv), 1.0)
        V = rand_bf16(rng, (lens[b], Dkv), 1.0)
        pos = torch.arange(lens[b], dtype=torch.int32, device="cuda")
        slot = torch.full((lens[b],), b, dtype=torch.int32, device="cuda")
        pool.store(layer, to_dev(K), to_dev(V), pos, slot)
    Q = to_dev(rand_bf16(rng, (B, Dq), 1.0))
    pos = torch.tensor([l - 1 for l in lens], dtype=torch.int32, device="cuda")
    slot = torch.arange(B, dtype=torch.int32, device="cuda")
    o_ref = torch.zeros_like(Q)
    o_new = torch.full_like(Q, float("nan"))
    layers.launch_attn(Q, o_ref, pool, layer, pos, slot, n_q)  # reference-order kernel (bit-exact vs reference)
    layers.launch_attn_decode_fast(Q, o_new, pool, layer, pos, slot, n_q, splits)
    torch.cuda.synchronize()
    got, want = to_host(o_new), to_host(o_ref)
    assert not np.isnan(bf16_to_f32(got)).any()
    assert rel_err(got, want) < TOL_BF16


def test_flash_decoding_workspace_of_several_streams(layers):
    """more splits than a cluster has write partial results: calls on two streams of one thread, and a captured one, each have memory of their own"""
    rng = np.random.default_rng(1)
    n_q, n_kv, hd, t, n = 14, 2, 64, 3000, 2
    pool = layers.KvPool(n_pages=n * ((t + 15) // 16), page_size=16, n_layers=1, n_kv_heads=n_kv, head_dim=hd, max_seqs=n)
    pool.pool.normal_(generator=torch.Generator("cuda").manual_seed(2))
    pos, slot = torch.full((n,), t - 1, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda")
    qs = [to_dev(rand_bf16(rng, (n, n_q * hd), 1.0)) for _ in range(2)]
    outs = [[torch.empty_like(x) for _ in range(20)] for x in qs]
    want = [torch.empty_like(x) for x in qs]
    for x, o in zip(qs, want):
        layers.launch_attn_decode_fast(x, o, pool, 0, pos, slot, n_q, 40)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in qs]
    for i in range(20):
        for x, o, st in zip(qs, outs, streams):
            with torch.cuda.stream(st):
                layers.launch_attn_decode_fast(x, o[i], pool, 0, pos, slot, n_q, 40)
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        assert all(torch.equal(x.view(torch.int16), w.view(torch.int16)) for x in o)
    g, x, o = torch.cuda.CUDAGraph(), qs[0].clone(), torch.empty_like(qs[0])
    with torch.cuda.graph(g, stream=streams[0]):
        layers.launch_attn_decode_fast(x, o, pool, 0, pos, slot, n_q, 40)
    for src, w in ((1, want[1]), (0, want[0])):
        x.copy_(qs[src])
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(o.view(torch.int16), w.view(torch.int16))
    del g


# pages of other than 16 positions: the mma.sync kernel at every length
@pytest.mark.parametrize("hd,n_q,n_kv,prefix,T,ps", [(64, 14, 2, 0, 64, 16), (64, 14, 2, 0, 1, 16), (64, 14, 2, 0, 200, 16), (64, 14, 2, 37, 91, 16),
                                                      (128, 12, 2, 0, 257, 16), (128, 28, 4, 130, 70, 16), (64, 4, 4, 15, 17, 16),
                                                      (128, 2, 1, 64, 128, 16), (64, 14, 2, 37, 700, 8), (128, 12, 2, 0, 257, 32), (128, 4, 2, 77, 1100, 4),
                                                      (64, 4, 2, 900, 300, 3)])
def test_prefill_attention_vs_reference_order_attention(layers, hd, n_q, n_kv, prefix, T, ps):
    """prefill chunk of T rows at positions prefix..prefix+T-1 of sequence 1 (sequence 0 holds other
    data); the cache already contains the prefix (chunked prefill) and the chunk's own K/V."""
    rng = np.random.default_rng(hd * 3 + n_q + prefix + T)
    Dq, Dkv = n_q * hd, n_kv * hd
    n_layers, layer = 2, 1
    total = prefix + T
    pool = layers.KvPool(n_pages=2 * ((total + ps - 1) // ps + 1), page_size=ps, n_layers=n_layers, n_kv_heads=n_kv,
                         head_dim=hd, max_seqs=2)
    for b, n in ((0, 9), (1, total)):
        K, V = rand_bf16(rng, (n, Dkv), 1.0), rand_bf16(rng, (n, Dkv), 1.0)
        pos = torch.arange(n, dtype=torch.int32, device="cuda")
        pool.store(layer, to_dev(K), to_dev(V), pos, torch.full((n,), b, dtype=torch.int32, device="cuda"))
    Q = to_dev(rand_bf16(rng, (T, Dq), 1.0))
    pos = torch.arange(prefix, total, dtype=torch.int32, device="cuda")
    slot = torch.full((T,), 1, dtype=torch.int32, device="cuda")
    o_ref = torch.zeros_like(Q)
    o_new = torch.full_like(Q, float("nan"))
    layers.launch_attn(Q, o_ref, pool, layer, pos, slot, n_q)  # reference-order kernel (bit-exact vs reference)
    layers.launch_attn_prefill_fast(Q, o_new, pool, layer, pos, slot, n_q)
    torch.cuda.synchronize()
    got, want = to_host(o_new), to_host(o_ref)
    assert not np.isnan(bf16_to_f32(got)).any()
    assert rel_err(got, want) < TOL_BF16


@pytest.mark.parametrize("ps", [16, 8, 32, 3])
@pytest.mark.parametrize("n_q,n_kv,prefix,T", [(12, 2, 0, 257), (28, 4, 130, 70), (2, 1, 64, 128), (4, 2, 77, 1000),
                                                (2, 2, 0, 1), (6, 1, 300, 129)])
def test_prefill_attention_tcgen05_vs_reference_order_attention(layers, n_q, n_kv, prefix, T, ps):
    """the tcgen05 / TMEM prefill attention (head_dim 128: S and P V on the 5th-gen tensor cores, softmax over
    tcgen05.ld) against the reference-order kernel: ragged last tile, cache prefix, GQA groups, one-row chunk.  Pages of 16
    positions are attn_prompt_tc.cu, others attn_prefill_tc.cu."""
    hd = 128
    rng = np.random.default_rng(n_q * 31 + prefix + T)
    Dq, Dkv = n_q * hd, n_kv * hd
    n_layers, layer = 2, 1
    total = prefix + T
    pool = layers.KvPool(n_pages=2 * ((total + ps - 1) // ps + 1), page_size=ps, n_layers=n_layers, n_kv_heads=n_kv,
                         head_dim=hd, max_seqs=2)
    for b, n in ((0, 9), (1, total)):
        K, V = rand_bf16(rng, (n, Dkv), 1.0), rand_bf16(rng, (n, Dkv), 1.0)
        pos = torch.arange(n, dtype=torch.int32, device="cuda")
        pool.store(layer, to_dev(K), to_dev(V), pos, torch.full((n,), b, dtype=torch.int32, device="cuda"))
    Q = to_dev(rand_bf16(rng, (T, Dq), 1.0))
    pos = torch.arange(prefix, total, dtype=torch.int32, device="cuda")
    slot = torch.full((T,), 1, dtype=torch.int32, device="cuda")
    o_ref = torch.zeros_like(Q)
    o_new = torch.full_like(Q, float("nan"))
    layers.launch_attn(Q, o_ref, pool, layer, pos, slot, n_q)
    layers.launch_attn_prefill_tc(Q, o_new, pool, layer, pos, slot, n_q)
    torch.cuda.synchronize()
    got, want = to_host(o_new), to_host(o_ref)
    assert not np.isnan(bf16_to_f32(got)).any()
    assert rel_err(got, want) < TOL_BF16


def test_fast_prefill_engine_long_prompt():
    """whole prefill, 300-token prompt in chunks of 128 rows (tcgen05 GEMMs + tiled causal attention):
    logits and per-layer activations of the last chunk within tolerance of the reference-order engine."""
    import qwen_inference_engine_b200 as q
    kw = dict(synthetic="small128", seed=3, context=1024, max_batch_tokens=128, max_seqs=4)
    e_ref = q.Engine(numerics="reference_order", **kw)
    e_fast = q.Engine(numerics="fast", **kw)
    ids = prompt_ids(300, e_ref.config.vocab, seed=11)
    for eng in (e_ref, e_fast):
        eng.capture(True)
    ta, tb = e_ref.prefill(e_ref.new_sequence(), ids), e_fast.prefill(e_fast.new_sequence(), ids)
    assert close(e_fast.read_capture("logits", -1), e_ref.read_capture("logits", -1))
    for l in range(e_ref.config.layers):
        for tag in ("attn", "x_out"):
            assert close(e_fast.read_capture(tag, l), e_ref.read_capture(tag, l)), (tag, l)
    print("fast prefill token", tb, "reference-order token", ta)
    e_ref.close()
    e_fast.close()


def test_fast_prefill_persistent_gemm_whole_prompt():
    """3000-token prompt in ONE forward on a 2-layer model with the 0.5B layer shape: every projection is
    large enough for the persistent tcgen05 GEMM (tile loop, double-buffered TMEM accumulator, overlapped
    store / residual / SiLU*up epilogues); logits and layer outputs against the reference-order engine."""
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(q.ARCHS["qwen2.5-0.5b"], layers=2, vocab=8192), context=4096)
    kw = dict(synthetic=cfg, seed=9, context=4096, max_batch_tokens=3072, max_seqs=2, kv_bytes=256 << 20)
    e_ref = q.Engine(numerics="reference_order", **kw)
    e_fast = q.Engine(numerics="fast", **kw)
    ids = prompt_ids(3000, cfg.vocab, seed=17)
    for eng in (e_ref, e_fast):
        eng.capture(True)
    ta, tb = e_ref.prefill(e_ref.new_sequence(), ids), e_fast.prefill(e_fast.new_sequence(), ids)
    assert close(e_fast.read_capture("logits", -1), e_ref.read_capture("logits", -1))
    for l in range(cfg.layers):
        for tag in ("attn", "x_attn", "mlp_h", "x_out"):
            a, b = e_fast.read_capture(tag, l), e_ref.read_capture(tag, l)
            assert close(a, b), (tag, l, rel_l2(a, b), rel_err(a, b))
    print("fast prefill token", tb, "reference-order token", ta)
    e_ref.close()
    e_fast.close()


def test_fast_prefill_chunking():
    """the same 700-token prompt prefilled in one forward, in chunks of 256 and in chunks of 100 rows (different
    GEMM variants: persistent / one tile per CTA / cluster split-K, attention with a cache prefix).  Rows are
    independent, only the split-K summation order depends on the chunk size, so logits agree within the fast-path
    tolerance and the reference-order engine -- where chunking must be invisible bit for bit -- is checked too."""
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(q.ARCHS["qwen2.5-0.5b"], layers=3, vocab=4096), context=2048)
    ids = prompt_ids(700, cfg.vocab, seed=23)
    for numerics, chunks in (("fast", (1024, 256, 100)), ("reference_order", (256, 64))):
        outs, logits = [], []
        for chunk in chunks:
            eng = q.Engine(synthetic=cfg, seed=4, context=2048, max_batch_tokens=chunk, max_seqs=2, kv_bytes=128 << 20,
                           numerics=numerics)
            eng.capture(True)
            s = eng.new_sequence()
            t = eng.prefill(s, ids)
            logits.append(eng.read_capture("logits", -1).copy())
            eng.capture(False)
            outs.append([t] + [int(x) for x in eng.decode_run([s], [t], 12)[:, 0]])
            eng.close()
        for lg, o in zip(logits[1:], outs[1:]):
            if numerics == "fast":
                assert close(lg, logits[0]), (rel_l2(lg, logits[0]), rel_err(lg, logits[0]))
            else:
                assert np.array_equal(lg, logits[0]) and o == outs[0]


def test_fast_engine_vs_reference_order_engine():
    """whole forward, batch 16 decode: FAST numerics vs REFERENCE_ORDER numerics on the same
    weights: logits within tolerance at every step; token agreement reported."""
    import qwen_inference_engine_b200 as q
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    kw = dict(synthetic="small", seed=21, context=512, max_batch_tokens=64, max_seqs=32)
    e_ref = q.Engine(numerics="reference_order", **kw)
    e_fast = q.Engine(numerics="fast", **kw)
    prompts = [prompt_ids(5 + 3 * i, e_ref.config.vocab, seed=i) for i in range(16)]
    agree = total = 0
    for eng in (e_ref, e_fast):
        eng.capture(True)
    s_ref = [e_ref.new_sequence() for _ in prompts]
    s_fast = [e_fast.new_sequence() for _ in prompts]
    cur = []
    for a, b, ids in zip(s_ref, s_fast, prompts):
        ta, tb = e_ref.prefill(a, ids), e_fast.prefill(b, ids)
        assert close(e_fast.read_capture("logits", -1), e_ref.read_capture("logits", -1))
        cur.append(ta)  # teacher-force the reference-order tokens so both engines see the same inputs
        agree += ta == tb
        total += 1
    for step in range(12):
        na = e_ref.decode_step(s_ref, cur)
        nb = e_fast.decode_step(s_fast, cur)
        la, lb = e_ref.read_capture("logits", -1), e_fast.read_capture("logits", -1)
        assert close(lb, la), f"step {step}: l2 {rel_l2(lb, la):.2e} max {rel_err(lb, la):.2e}"
        for l in range(e_ref.config.layers):
            for tag in ("attn", "x_out", "mlp_h"):
                assert close(e_fast.read_capture(tag, l), e_ref.read_capture(tag, l)), (step, tag, l)
        agree += int((na == nb).sum())
        total += len(na)
        cur = list(na)
    print(f"fast vs reference-order greedy token agreement: {agree}/{total}")
    assert agree / total > 0.9
    # graph replay of the fast path == eager fast path
    e_fast.capture(False)
    out = e_fast.decode_run(s_fast, cur, 6)
    assert out.shape == (6, 16)
    e_ref.close()
    e_fast.close()
