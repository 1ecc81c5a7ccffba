"""Causal attention over a whole sequence (ns_attention_prefill, tcgen05) against the oracle's reference-order
attention: scale, additive mask, row maximum, exp, float sum, normalise, . V (Layers/Attention.cs:54-90,
CpuBackend.Decoding.cs:9-41) on the same bf16-rounded inputs.  Tolerance 1e-2 relative on bf16 outputs.
benchmark configuration 4: [batch 8, heads 32, seq, 128], seq in {512, 2048, 8192}, scale 1/sqrt(128), seed 3.
"""
import ctypes as C

import numpy as np
import pytest

from nn_b200 import native as N

pytestmark = pytest.mark.gpu
TOL = 1e-2
DH = 128


def _strides(*v):
    return (C.c_int64 * 3)(*v)


def _run_bhsd(dev, q, k, v, B, H, S, scale, causal=True):
    dq, dk, dv = dev.from_numpy(q), dev.from_numpy(k), dev.from_numpy(v)
    do = dev.zeros(B * H * S * DH, N.NS_BF16)
    st = _strides(H * S * DH, S * DH, DH)
    N.call("ns_attention_prefill", dev.handle, dq.ptr, dk.ptr, dv.ptr, do.ptr, B, H, S, DH, st, st, st, st, C.c_float(scale), int(causal))
    dev.synchronize()
    return do.download((B, H, S, DH))


@pytest.mark.parametrize("S", [1, 37, 128, 129, 300, 640])
@pytest.mark.parametrize("causal", [True, False])
def test_small_sequences(dev, orc, S, causal):
    B, H = 2, 3
    scale = 1.0 / np.sqrt(DH)
    q = orc.round_bf16(orc.normal((B, H, S, DH), 1))
    k = orc.round_bf16(orc.normal((B, H, S, DH), 2))
    v = orc.round_bf16(orc.normal((B, H, S, DH), 3))
    got = orc.widen_bf16(_run_bhsd(dev, q, k, v, B, H, S, scale, causal))
    for b in range(B):
        for h in range(H):
            exp = orc.attention_slice(orc.widen_bf16(q[b, h]), orc.widen_bf16(k[b, h]), orc.widen_bf16(v[b, h]), 0, scale, causal)
            assert orc.close(orc.bf16_round_trip(exp), got[b, h], TOL), (b, h, orc.max_err(exp, got[b, h]))


def test_large_scores_and_growing_maximum(dev, orc):
    """Scores that keep growing along the sequence force the running maximum (and the rescale of O) to move."""
    B, H, S = 1, 2, 512
    q = orc.normal((B, H, S, DH), 4)
    k = orc.normal((B, H, S, DH), 5)
    k *= np.linspace(0.2, 6.0, S, dtype=np.float32)[None, None, :, None]
    v = orc.normal((B, H, S, DH), 6)
    qb, kb, vb = orc.round_bf16(q), orc.round_bf16(k), orc.round_bf16(v)
    scale = 0.5
    got = orc.widen_bf16(_run_bhsd(dev, qb, kb, vb, B, H, S, scale))
    for h in range(H):
        exp = orc.attention_slice(orc.widen_bf16(qb[0, h]), orc.widen_bf16(kb[0, h]), orc.widen_bf16(vb[0, h]), 0, scale)
        assert orc.close(orc.bf16_round_trip(exp), got[0, h], TOL), orc.max_err(exp, got[0, h])


def test_fused_qkv_layout(dev, orc):
    """q, k, v read in place from a [batch * seq, 3 * D] buffer (the output of the fused QKV product), o written
    as [batch * seq, D]: the reference's narrow + permute copies (Attention.cs:54-58) are not needed."""
    B, H, S = 2, 4, 200
    D = H * DH
    scale = 1.0 / np.sqrt(DH)
    qkv = orc.round_bf16(orc.normal((B, S, 3 * D), 7))
    dqkv = dev.from_numpy(qkv)
    do = dev.zeros(B * S * D, N.NS_BF16)
    st_in = _strides(S * 3 * D, DH, 3 * D)
    st_out = _strides(S * D, DH, D)
    N.call("ns_attention_prefill", dev.handle, dqkv.ptr, dqkv.ptr + 2 * D, dqkv.ptr + 4 * D, do.ptr, B, H, S, DH, st_in, st_in, st_in, st_out,
           C.c_float(scale), 1)
    dev.synchronize()
    got = orc.widen_bf16(do.download((B, S, H, DH)))
    f = orc.widen_bf16(qkv).reshape(B, S, 3, H, DH)
    for b in range(B):
        for h in range(H):
            exp = orc.attention_slice(f[b, :, 0, h], f[b, :, 1, h], f[b, :, 2, h], 0, scale)
            assert orc.close(orc.bf16_round_trip(exp), got[b, :, h], TOL), (b, h, orc.max_err(exp, got[b, :, h]))


@pytest.mark.parametrize("S", [512, 2048, 8192])
def test_baseline_shapes(dev, orc, S):
    B, H = 8, 32
    scale = 1.0 / np.sqrt(DH)
    n = B * H * S * DH
    dq, dk, dv, do = (dev.empty(n, N.NS_BF16) for _ in range(4))
    for t, seed in ((dq, 31), (dk, 32), (dv, 33)):
        N.call("ns_fill_normal", dev.handle, t.ptr, N.NS_BF16, C.c_int64(n), seed, C.c_float(0.0), C.c_float(1.0))
    st = _strides(H * S * DH, S * DH, DH)
    N.call("ns_attention_prefill", dev.handle, dq.ptr, dk.ptr, dv.ptr, do.ptr, B, H, S, DH, st, st, st, st, C.c_float(scale), 1)
    dev.synchronize()
    rng = np.random.default_rng(S)
    for (b, h) in [(0, 0), (7, 31), (3, 17)]:
        off = (b * H + h) * S * DH
        qs, ks, vs, os_ = (orc.widen_bf16(t.download((S, DH), offset=off, count=S * DH)) for t in (dq, dk, dv, do))
        starts = sorted(set([0, S - 64, S // 2 - 32] + [int(x) for x in rng.integers(0, S - 64, 2)]))
        for r0 in starts:
            exp = orc.attention_slice(qs[r0:r0 + 64], ks, vs, r0, scale)
            assert orc.close(orc.bf16_round_trip(exp), os_[r0:r0 + 64], TOL), (b, h, r0, orc.max_err(exp, os_[r0:r0 + 64]))
    # size-independent property: row 0 attends to key 0 only, so o[:, :, 0, :] == v[:, :, 0, :] exactly
    o0 = do.download((B * H, S * DH))[:, :DH]
    v0 = dv.download((B * H, S * DH))[:, :DH]
    assert np.array_equal(o0, v0)


def test_results_do_not_depend_on_the_tile_schedule(dev, orc):
    """The kernel's CTAs draw their (batch, head, query tile) work from a counter at run time, so which CTA -- and which of
    its two softmax groups -- handles a tile's even and odd key blocks changes from run to run.  The output must not:
    three runs on the same inputs are bit-identical (a greedy decoder downstream turns a last-bit difference into
    another token at a near-tie)."""
    import ctypes as C
    B, H, S = 16, 16, 640
    n = B * H * S * 128
    q, k, v = (dev.empty(n, N.NS_BF16) for _ in range(3))
    for t, seed in ((q, 11), (k, 12), (v, 13)):
        N.call("ns_fill_normal", dev.handle, t.ptr, N.NS_BF16, C.c_int64(n), seed, C.c_float(0.0), C.c_float(1.0))
    st = (C.c_int64 * 3)(H * S * 128, S * 128, 128)
    outs = []
    for rep in range(3):
        o = dev.zeros(n, N.NS_BF16)
        N.call("ns_attention_prefill", dev.handle, q.ptr, k.ptr, v.ptr, o.ptr, B, H, S, 128, st, st, st, st, C.c_float(0.0884), 1)
        dev.synchronize()
        outs.append(o.download())
        o.release()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


@pytest.mark.parametrize("S", [1, 127, 128, 129, 255, 256, 257, 384, 511, 513, 1000])
@pytest.mark.parametrize("causal", [True, False])
def test_tiles_of_one_group_and_of_two(dev, orc, S, causal):
    """Where every 128 query rows get an SM of their own a tile is one group's, else two groups' (one without rows where S leaves fewer than 129):
    a row's result is the same to the bit, and within bf16 of the oracle.  Scores grow along the sequence, so the reference maximum moves."""
    heads, scale = 2, 0.2
    many = 200 // heads                                              # 200 tiles of 128 rows are more than a B200 has SMs
    grow = np.linspace(0.3, 2.0, S, dtype=np.float32)[:, None]
    q, k, v = (orc.round_bf16(orc.normal((1, heads, S, DH), 20 + i) * (grow if i == 1 else 1)) for i in range(3))
    one = _run_bhsd(dev, q, k, v, 1, heads, S, scale, causal)
    all_ = _run_bhsd(dev, *(np.repeat(x, many, 0) for x in (q, k, v)), many, heads, S, scale, causal)
    assert np.array_equal(all_, np.repeat(one, many, 0))
    for h in range(heads):
        exp = orc.attention_slice(*(orc.widen_bf16(x[0, h]) for x in (q, k, v)), 0, scale, causal)
        got = orc.widen_bf16(one[0, h])
        assert orc.close(orc.bf16_round_trip(exp), got, TOL), (h, orc.max_err(exp, got))


@pytest.mark.parametrize("S,batch", [(300, 1), (300, 100)])      # tiles of one group, of two
@pytest.mark.parametrize("causal", [True, False])
def test_scores_that_are_no_numbers(dev, S, batch, causal):
    """A NaN in a key makes every row that sees it NaN, whichever key it is (one exponential in eight is a polynomial); so does a score of +infinity.  A score of
    -infinity weighs nothing.  Other rows keep their bits."""
    rng = np.random.default_rng(9)
    heads, scale = 2, 0.1
    q, k, v = (rng.standard_normal((heads, S, DH)).astype(np.float32) for _ in range(3))
    q[:, ::2, 0], q[:, 1::2, 0] = 1, -1
    bits = lambda a: (np.ascontiguousarray(a, np.float32).view(np.uint32) >> 16).astype(np.uint16)
    wide = lambda b: (b.astype(np.uint32) << 16).view(np.float32).astype(np.float64)

    def run(key):
        many = [np.repeat(bits(x)[None], batch, 0) for x in (q, key, v)]
        out = _run_bhsd(dev, *many, batch, heads, S, scale, causal)
        assert np.array_equal(out, np.repeat(out[:1], batch, 0))
        return out[0]

    clean = run(k)
    rows = np.arange(S)
    for j in [*range(16), 62, 63, 127, 128, 142, 143, 255, 256, 270, 298, 299]:
        sees = rows >= j if causal else rows >= 0
        for value in (np.nan, np.inf):
            key = k.copy()
            key[:, j, 0] = value
            got = run(key)
            lost = sees & (np.isnan(value) | (rows % 2 == 0))
            assert np.isnan(wide(got[:, lost])).all(), (j, value)
            assert np.array_equal(got[:, ~sees], clean[:, ~sees]), (j, value)
            rest = np.nonzero(sees & ~lost)[0][:: 7]
            if len(rest):
                for h in range(heads):
                    s = wide(bits(q[h, rest])) @ wide(bits(k[h])).T * scale
                    s[:, j] = -np.inf
                    if causal:
                        s[rows[None, :] > rest[:, None]] = -np.inf
                    p = np.exp(s - s.max(1, keepdims=True))
                    p /= p.sum(1, keepdims=True)
                    value_rows = wide(bits(v[h]))
                    # weights and results are rounded to bf16, whose numbers are 2^-7 apart: 2^-8 of each term, and of the sum
                    assert np.all(np.abs(wide(got[h, rest]) - p @ value_rows) <= 2.0 ** -7 * (p @ np.abs(value_rows)))
