"""The float32 decoder on the operator surface (nn_b200.gpt_f32.GptF32 over NsB200Backend) against the oracle's
float32 decoder (the reference's CPU backend restated), restating the reference's decoding tests:
CachedDecodingMatchesFull (DecodingTests.cs:69-98: TinyGpt vocab 11, dim 16, 4 heads, ffDim 32, 2 layers, ctx 12,
prefill 4 then 6 single steps == full forward, 1e-4), BatchedDecoding (:100-142, B=3 == each sequence alone),
GraphReplay (:144-189, graph == direct over 8 steps), and benchmark configuration 1 (char-level GPT: vocab 96, d_model 128,
4 layers, 4 heads, FFN 512, context 128, prompt 32, greedy 128 tokens: logits <= 1e-4, token ids equal, one context
reset at the 97th token).
"""
import ctypes as C

import numpy as np
import pytest

from nn_b200 import native as N
from nn_b200.backend import NsB200Backend
from nn_b200.gpt import GptConfig
from nn_b200.gpt_f32 import GptF32
from oracle import model as om

pytestmark = pytest.mark.gpu
TINY = GptConfig(vocab=11, dim=16, heads=4, layers=2, ff_dim=32, context=12)
TINY12 = GptConfig(vocab=12, dim=16, heads=4, layers=2, ff_dim=32, context=12)     # a vocabulary the step kernels take


@pytest.mark.parametrize("TINY", [TINY, TINY12], ids=["operators", "step kernels"])
def test_cached_decoding_matches_full(dev, orc, TINY):
    w = om.make_weights(TINY, seed=7, std=0.3, sinusoid=True)
    ids = orc.token_ids((1, 10), 70, TINY.vocab).astype(np.int64)
    m = GptF32(dev, TINY, w, 1, max_steps=10)
    assert m.step_kernels == (TINY.vocab == 12)
    # full forward over 10 positions
    m.prefill(ids)
    dev.synchronize()
    full = m.logits.download((10, TINY.vocab), count=10 * TINY.vocab).copy()
    ref = om.F32Decoder(TINY, w, 1)
    assert orc.close(ref.forward(ids), full[-1:], 1e-4)
    # prefill 4, then 6 single steps, teacher-forced with the same ids
    m.prefill(ids[:, :4])
    rows = [m.logits.download((4, TINY.vocab), count=4 * TINY.vocab).copy()]
    for s in range(4, 10):
        m.be.Upload(np.pad(ids[0, s:s + 1].astype(np.float32), (0, m.ids.count - 1)), m.ids)
        m.step(use_graph=False)
        dev.synchronize()
        rows.append(m.logits.download((1, TINY.vocab), count=TINY.vocab).copy())
    assert orc.close(full, np.concatenate(rows), 1e-4)


@pytest.mark.parametrize("TINY", [TINY, TINY12], ids=["operators", "step kernels"])
def test_batched_decoding_and_graph_replay(dev, orc, TINY):
    w = om.make_weights(TINY, seed=8, std=0.3, sinusoid=True)
    prompts = orc.token_ids((3, 3), 71, TINY.vocab).astype(np.int64)
    together = GptF32(dev, TINY, w, 3, max_steps=6)
    tok_b, _, trace_b = together.generate(prompts, 8, use_graph=True)
    tok_d, _, trace_d = together.generate(prompts, 8, use_graph=False)
    assert np.array_equal(tok_b, tok_d)                                   # GraphReplay
    for a, b in zip(trace_b, trace_d):
        assert np.array_equal(a, b)
    for i in range(3):                                                     # BatchedDecoding
        alone = GptF32(dev, TINY, w, 1, max_steps=6)
        tok_1, _, trace_1 = alone.generate(prompts[i:i + 1], 8, use_graph=False)
        for s in range(8):
            assert orc.close(trace_1[s], trace_b[s][i:i + 1], 1e-4)
    ref = om.F32Decoder(TINY, w, 3)
    exp, _ = ref.generate(prompts, 8)
    for s in range(8):
        assert orc.close(ref.logit_trace[s], trace_b[s], 1e-4)


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("batch", [1, 3, 9])
def test_steps_have_the_operators_bits(dev, orc, batch, use_graph):
    """The same model with and without the step kernels, across a context reset: tokens, logits and caches."""
    cfg = GptConfig(vocab=40, dim=48, heads=3, layers=2, ff_dim=100, context=20)
    w = om.make_weights(cfg, seed=9, std=0.3)
    prompts = orc.token_ids((batch, 5), 72, cfg.vocab).astype(np.int64)
    models = [GptF32(dev, cfg, w, batch, max_steps=10) for _ in range(2)]
    assert models[0].step_kernels
    models[1].step_kernels = False
    (tok, resets, trace), (tok_o, resets_o, trace_o) = (m.generate(prompts, 24, use_graph) for m in models)
    assert resets == resets_o == 1 and np.array_equal(tok, tok_o)
    for a, b in zip(trace, trace_o):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for a, b in zip(models[0].keys + models[0].values, models[1].keys + models[1].values):
        assert np.array_equal(a.download().view(np.uint32), b.download().view(np.uint32))


@pytest.mark.parametrize("dim,ff,batch,kernels", [(8, 2048, 600, True), (8, 2052, 512, True), (8, 2052, 513, False), (776, 2052, 96, True), (776, 2052, 97, False),
                                                  (1032, 8, 96, True), (1032, 8, 97, False), (1032, 2052, 32, True), (1032, 2052, 33, False), (8, 4100, 1, False)])
def test_step_kernels_are_taken_where_they_are_faster(dev, orc, dim, ff, batch, kernels):
    cfg = GptConfig(vocab=8, dim=dim, heads=2, layers=1, ff_dim=ff, context=4)
    assert GptF32(dev, cfg, om.make_weights(cfg, seed=1), batch, max_steps=1).step_kernels == kernels


@pytest.mark.parametrize("batch,steps,position", [(1, 1, 0), (3, 1, 6), (2, 4, 4), (2, 3, 9)])
def test_step_embedding_has_the_operators_bits(dev, orc, batch, steps, position):
    """Ids and positions past their tables, fractions and negative ids are taken as Gather takes them."""
    be, D, V, cap, n = NsB200Backend(dev), 20, 11, 7, batch * steps
    up = lambda a: dev.from_numpy(np.ascontiguousarray(a, dtype=np.float32))
    table, places = up(orc.normal((V, D), 95)), up(orc.normal((cap, D), 96))
    ids = up(np.resize([3.0, 10.0, 11.0, 1e9, -2.0, 0.0, 4.7, 9.0], n))
    where, pos = up(np.resize(position + np.arange(steps), n)), up([position])
    x, t, e = dev.empty(n * D), dev.empty(n * D), dev.empty(n * D)
    N.call("ns_f32_embed_positions", dev.handle, ids.ptr, table.ptr, places.ptr, pos.ptr, x.ptr, batch, steps, D, V, cap)
    be.Gather(table, ids, t, n, D, V)
    be.Gather(places, where, e, n, D, cap)
    be.Add(t, e, t, n * D)
    dev.synchronize()
    assert np.array_equal(x.download().view(np.uint32), t.download().view(np.uint32))


@pytest.mark.parametrize("sinusoid", [False, True])
def test_baseline_config_1(dev, orc, sinusoid):
    cfg = GptConfig(vocab=96, dim=128, heads=4, layers=4, ff_dim=512, context=128)
    w = om.make_weights(cfg, seed=0, std=0.02, sinusoid=sinusoid)
    for k in w:
        if k.endswith("_b") and "ln" not in k:
            w[k] = np.zeros_like(w[k])                                     # biases 0, as Linear initialises them
    prompt = orc.token_ids((1, 32), 1, cfg.vocab).astype(np.int64)
    ref = om.F32Decoder(cfg, w, 1)
    exp, exp_resets = ref.generate(prompt, 128)
    assert exp_resets == 1
    m = GptF32(dev, cfg, w, 1, max_steps=64)
    got, resets, trace = m.generate(prompt, 128, use_graph=True)
    assert resets == 1
    worst, first_div = 0.0, None
    for s in range(128):
        if first_div is None and got[0, s] != exp[0, s]:
            first_div = s
        if first_div is None or s <= first_div:                            # identical histories up to the first divergence
            worst = max(worst, orc.max_err(ref.logit_trace[s], trace[s]))
    assert worst <= 1e-4, f"max logit error {worst:.2e}"
    if first_div is not None:
        top2 = np.sort(ref.logit_trace[first_div][0])[-2:]
        assert top2[1] - top2[0] <= 2e-4 * max(1.0, abs(top2[1])), f"tokens diverge at step {first_div} without a near-tie"


# around a warp's rows (1, 2 and 4 of tiles of 8, 16 and 32), a tile's 32 columns, the ring's 64-step slices (8 of them), the longest row of each form
@pytest.mark.parametrize("m,n,k", [(1, 4, 4), (1, 128, 512), (3, 36, 60), (8, 32, 64), (9, 28, 452), (17, 100, 516), (33, 64, 1024), (17, 32, 1028), (9, 8, 2052), (2, 8, 4096), (2097153, 4, 4)])
def test_step_linear_has_the_operators_bits(dev, orc, m, n, k):
    be = NsB200Backend(dev)
    up = lambda a: dev.from_numpy(np.ascontiguousarray(a, dtype=np.float32))
    x, w, g, b, bias, res = (up(orc.normal(s, 80 + i)) for i, s in enumerate([(m, k), (k, n), (k,), (k,), (n,), (m, n)]))
    y, t, u = dev.empty(m * n), dev.empty(m * k), dev.empty(m * n)
    bits = lambda s: s.download(count=m * n).view(np.uint32)
    for norm, with_bias, gelu, residual in [(0, 0, 0, 0), (1, 1, 0, 0), (1, 1, 1, 0), (0, 1, 0, 1), (1, 0, 0, 1)]:
        N.call("ns_f32_linear", dev.handle, x.ptr, g.ptr if norm else 0, b.ptr if norm else 0, C.c_float(1e-5), w.ptr, bias.ptr if with_bias else 0,
               res.ptr if residual else 0, gelu, y.ptr, m, n, k)
        if norm:
            be.LayerNormFused(x, g, b, t, m, k, 1e-5)
        be.MatMul(t if norm else x, w, u, m, n, k, False, False, 0.0)
        if gelu:
            be.BiasGelu(u, bias, u, m * n, n)
        elif with_bias:
            be.AddRowVector(u, bias, u, m, n)
        if residual:
            be.Add(res, u, u, m * n)
        dev.synchronize()
        assert np.array_equal(bits(y), bits(u)), (norm, with_bias, gelu, residual)


@pytest.mark.parametrize("batch,heads,cap,dim,pos", [(1, 4, 128, 32, 0), (2, 3, 128, 32, 127), (1, 2, 5, 4, 3), (3, 2, 300, 36, 129), (1, 2, 257, 132, 256), (1, 1, 12, 8, 12)])
def test_step_attention_has_the_operators_bits(dev, orc, batch, heads, cap, dim, pos):
    be, D = NsB200Backend(dev), heads * dim
    up = lambda a: dev.from_numpy(np.ascontiguousarray(a, dtype=np.float32))
    qkv_h, k_h, v_h = orc.normal((batch, 3 * D), 90), orc.normal((batch * heads, cap, dim), 91), orc.normal((batch * heads, cap, dim), 92)
    qkv, position = up(qkv_h), up([float(pos)])
    got, exp = [up(k_h), up(v_h), dev.empty(batch * D)], [up(k_h), up(v_h), dev.empty(batch * D)]
    scale = float(np.float32(dim) ** np.float32(-0.5))
    N.call("ns_f32_attention_step", dev.handle, qkv.ptr, got[0].ptr, got[1].ptr, position.ptr, got[2].ptr, batch, heads, cap, dim, C.c_float(scale))
    part = [up(qkv_h[:, i * D:(i + 1) * D]) for i in range(3)]           # one position: [batch, heads, 1, dim] as it lies
    mask, scores, probs = dev.empty(cap), dev.empty(batch * heads * cap), dev.empty(batch * heads * cap)
    be.DecoderMask(position, mask, 1, cap)
    be.KeyValueWrite(part[1], exp[0], position, batch * heads, 1, cap, dim)
    be.KeyValueWrite(part[2], exp[1], position, batch * heads, 1, cap, dim)
    be.BatchedMatMul(part[0], exp[0], scores, batch * heads, 1, cap, dim, False, True, 0.0)
    be.ScaleMaskSoftmax(scores, mask, probs, batch * heads, cap, 1, scale)
    be.BatchedMatMul(probs, exp[1], exp[2], batch * heads, 1, dim, cap, False, False, 0.0)
    dev.synchronize()
    for a, b in zip(got, exp):
        assert np.array_equal(a.download().view(np.uint32), b.download().view(np.uint32))
