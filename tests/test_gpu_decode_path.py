"""Which way a decode step goes: by default the operators where their attention takes it, "mega" 1 the persistent kernel, -1 the default again, 0 never.  Engine.runs_mega says
it, and the launches of the steps are those of that way; the tokens are the same."""
import numpy as np
import pytest

from util import prompt_ids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("page,default", [(16, False), (4, True)])  # (pages of 4 positions: the operators' attention does not take them)
@pytest.mark.parametrize("graph", [False, True])
def test_ways(page, default, graph):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    e = q.Engine(synthetic="small", seed=7, context=256, max_batch_tokens=64, max_seqs=4, page_size=page, use_graph=graph, kv_bytes=32 << 20)
    layers, got = e.config.layers, []
    for mega, way in ((None, default), (0, False), (1, True), (-1, default), (0, False), (-1, default)):
        if mega is not None:
            e.set_int("mega", mega)
        seqs = [e.new_sequence() for _ in range(3)]
        tokens = [e.prefill(s, prompt_ids(5 + i, e.config.vocab, seed=i)) for i, s in enumerate(seqs)]
        out = []
        for _ in range(4):
            assert e.uses_mega(3, 12) == (mega != 0) and e.runs_mega(3, 12) == way
            tokens = e.decode_step(seqs, tokens)
            assert (e.launch_count() < layers) == way
            out.append(np.array(tokens))
        got.append(np.stack(out))
        for s in seqs:
            e.free_sequence(s)
    e.close()
    assert all(np.array_equal(got[0], g) for g in got)


@pytest.mark.parametrize("hd,kinds", [(64, ("attention",)), (128, ("qkv_post", "attention"))])
def test_a_profile_times_the_launches_of_the_step(hd, kinds):
    """heads of 64: one launch does the head norms, the positions, the store and the attention, in a profiled step as in others"""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qwen_inference_engine_b200 as q
    cfg = q.make_config(dict(hidden=256, inter=512, layers=3, n_q=4, n_kv=2, head_dim=hd, vocab=2048), context=256)
    e = q.Engine(synthetic=cfg, seed=7, context=256, max_batch_tokens=64, max_seqs=4, max_pages=64)
    seqs = [e.new_sequence() for _ in range(3)]
    tokens = [e.prefill(s, prompt_ids(5 + i, 2048, seed=i)) for i, s in enumerate(seqs)]
    tokens = e.decode_step(seqs, tokens)
    launches = e.launch_count()
    prof = e.decode_step_profile(seqs, tokens)
    e.close()
    assert [k for k in ("qkv_post", "attention") if prof.get(k, (0, 0))[1]] == list(kinds) and prof["attention"][1] == 3
    assert sum(n for _, n in prof.values()) == launches
