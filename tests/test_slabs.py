"""Operators that read partial sums: whatever the number of slabs and however they are read, the bits are those of one slab that holds their
sum in order.  Widths with and without vectors, few rows and many, up to one group of slabs read together (8) and past it."""
import ctypes as C

import numpy as np
import pytest

from nn_b200 import native as N
from tests.test_fabezen_ops import rng_for

pytestmark = pytest.mark.gpu
u, i64, fl = C.c_uint64, C.c_int64, C.c_float


def slabs_and_sum(dev, rows, ld, splits):
    parts = rng_for(splits, rows, ld).standard_normal((splits, rows, ld)).astype(np.float32)
    total = parts[0].copy()
    for p in parts[1:]:
        total += p
    return dev.from_numpy(parts), dev.from_numpy(total)


def same(dev, run, source, total, splits):
    """run(source, splits) returns what the operator wrote."""
    got, want = run(source, splits), run(total, 1)
    dev.synchronize()
    for g, w in zip(got, want):
        a, b = g.download(), w.download()
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
        assert np.any(a)


SPLITS = [2, 3, 7, 8, 9, 16]


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("rows,cols", [(3, 64), (2, 61), (5, 1028), (300, 2048), (300, 2047), (3, 4096), (2, 8000), (2, 9001)])
@pytest.mark.parametrize("out", [N.NS_F32, N.NS_BF16])
def test_rows(dev, rows, cols, splits, out):
    ld = (cols + 7) // 8 * 8
    source, total = slabs_and_sum(dev, rows, ld, splits)
    rng = rng_for(1, rows, cols)
    x, w, post = (dev.from_numpy(rng.standard_normal(s).astype(np.float32)) for s in ((rows, cols), cols, cols))

    def norm(src, n):
        y, xo = dev.zeros(rows * ld, out), dev.zeros(rows * cols)
        N.call("ns_rms_rows", dev.handle, u(x.ptr), u(src.ptr), n, N.NS_F32, ld, fl(0.3), u(xo.ptr), u(w.ptr), fl(1e-3), u(0), i64(rows), i64(rows), cols, out, u(y.ptr), ld)
        return xo, y

    def both_norms(src, n):
        y, xo = dev.zeros(rows * ld, out), dev.zeros(rows * cols)
        N.call("ns_rms_post_rows", dev.handle, u(x.ptr), u(src.ptr), n, N.NS_F32, ld, u(post.ptr), u(0), u(xo.ptr), u(w.ptr), fl(1e-3), i64(rows), cols, out, u(y.ptr), ld)
        return xo, y

    def columns(src, n):
        y = dev.zeros(rows * ld, out)
        N.call("ns_copy_cols", dev.handle, u(src.ptr), n, N.NS_F32, ld, 1, i64(rows), cols - 1, out, u(y.ptr), ld)
        return (y,)

    for run in (norm, both_norms, columns):
        same(dev, run, source, total, splits)


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("rows,ff", [(1, 8), (3, 37), (3, 1000), (120, 5632), (60, 2047)])
def test_gated_unit(dev, rows, ff, splits):
    ld, y_ld = (2 * ff + 7) // 8 * 8, (ff + 7) // 8 * 8
    source, total = slabs_and_sum(dev, rows, ld, splits)
    for act in (N.ACT_GELU, N.ACT_RELU):
        for out in (N.NS_F32, N.NS_BF16):
            def unit(src, n):
                y = dev.zeros(rows * y_ld, out)
                N.call("ns_glu_rows", dev.handle, u(src.ptr), n, N.NS_F32, ld, i64(rows), ff, act, out, u(y.ptr), y_ld)
                return (y,)

            same(dev, unit, source, total, splits)


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("H,G,dim,vdim,steps", [(4, 2, 32, 24, 3), (3, 1, 33, 27, 2), (16, 4, 128, 128, 70)])
def test_window_append(dev, H, G, dim, vdim, steps, splits):
    nq, nk, nv, ring = H * dim, G * dim, G * vdim, 128
    k_ld, v_ld, rows = (dim + 7) // 8 * 8, (vdim + 7) // 8 * 8, 2 * steps
    ld = (nq + nk + nv + H + 7) // 8 * 8
    source, total = slabs_and_sum(dev, rows, ld, splits)
    wq, wk = (dev.from_numpy(rng_for(3, n).standard_normal(n).astype(np.float32)) for n in (nq, nk))
    slots, pos = dev.from_numpy(np.array([1, 0], np.int32)), dev.from_numpy(np.array([5, 90], np.int32))
    for dtype in (N.NS_F32, N.NS_BF16):
        def append(src, n):
            q, gate, kr, vr = dev.zeros(rows * H * k_ld, dtype), dev.zeros(rows * H), dev.zeros(2 * G * ring * k_ld, dtype), dev.zeros(2 * G * ring * v_ld, dtype)
            N.call("ns_window_append", dev.handle, u(src.ptr), n, N.NS_F32, ld, 0, nq, nq + nk, nq + nk + nv, H, G, dim, vdim, u(wq.ptr), u(wk.ptr), fl(1e-5), u(slots.ptr),
                   u(pos.ptr), 2, steps, dtype, u(q.ptr), u(gate.ptr), u(kr.ptr), u(vr.ptr), i64(G * ring * k_ld), i64(G * ring * v_ld), ring, k_ld, v_ld)
            return q, gate, kr, vr

        same(dev, append, source, total, splits)


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("heads,hd,taps", [(3, 32, 4), (5, 64, 4), (4, 128, 4), (2, 128, 7), (2, 60, 6), (2, 256, 3), (1, 500, 4), (2, 33, 10)])
@pytest.mark.parametrize("batch,steps", [(2, 1), (70, 2), (2, 40)])
def test_short_convolution(dev, heads, hd, taps, batch, steps, splits):
    channels = heads * hd
    source, total = slabs_and_sum(dev, batch * steps, channels + 4, splits)
    w, before = (rng_for(4, channels, k).standard_normal(n).astype(np.float32) for k, n in enumerate((channels * taps, batch * taps * channels)))
    w, slots, pos = dev.from_numpy(w), dev.from_numpy(np.arange(batch, dtype=np.int32)), dev.from_numpy(np.full(batch, 9, np.int32))

    def conv(src, n):
        hist, out = dev.from_numpy(before), dev.zeros(batch * steps * channels)
        fields = (C.c_int64 * 9)(4, heads, hd, taps, 1, w.ptr, hist.ptr, out.ptr, channels)
        N.call("ns_short_conv", dev.handle, u(src.ptr), n, N.NS_F32, channels + 4, 1, fields, (C.c_float * 1)(0.25), i64(taps * channels), u(slots.ptr), u(pos.ptr), batch,
               steps, N.NS_F32)
        dev.synchronize()
        return out, hist

    same(dev, conv, source, total, splits)


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("H,dim,vdim", [(3, 20, 28), (2, 60, 64), (2, 64, 128), (2, 128, 40), (4, 96, 130), (2, 200, 72)])
@pytest.mark.parametrize("batch,steps", [(2, 3), (170, 1)])
def test_linear_attention(dev, H, dim, vdim, batch, steps, splits):
    cols = H * (2 * dim + vdim)
    source, total = slabs_and_sum(dev, batch * steps, (cols + 7) // 8 * 8, splits)
    decay = np.linspace(0.5, 1.0, H).astype(np.float32)
    dec, log2, slots = dev.from_numpy(decay), dev.from_numpy(np.log2(decay)), dev.from_numpy(np.arange(batch, dtype=np.int32))
    before = rng_for(5, H, dim, vdim, batch).standard_normal(batch * H * dim * vdim).astype(np.float32)
    for name, extra in (("ns_lightning_recurrent", ()), ("ns_lightning_chunked", (0,))):
        if name == "ns_lightning_chunked" and dim > 128:
            continue

        def run(src, n):
            state, o = dev.from_numpy(before), dev.zeros(batch * steps * H * vdim)
            N.call(name, dev.handle, u(src.ptr), n, N.NS_F32, (cols + 7) // 8 * 8, 0, H * dim, 2 * H * dim, u(dec.ptr), u(log2.ptr), u(state.ptr), i64(H * dim * vdim),
                   u(slots.ptr), batch, steps, H, dim, vdim, u(o.ptr), H * vdim, *extra)
            return o, state

        same(dev, run, source, total, splits)


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("H,kv,dim,vdim", [(4, 2, 20, 28), (2, 1, 64, 128), (3, 3, 100, 130), (2, 2, 128, 64), (2, 2, 200, 96)])
@pytest.mark.parametrize("batch,steps", [(2, 3), (170, 1)])
@pytest.mark.parametrize("channelwise", [0, 1])
def test_delta_rule(dev, H, kv, dim, vdim, batch, steps, channelwise, splits):
    rows, ac = batch * steps, H * dim if channelwise else H
    ld = (ac + H + 7) // 8 * 8
    source, total = slabs_and_sum(dev, rows, ld, splits)
    rng = rng_for(6, H, dim, vdim, rows)
    q, k, v, a_log, dt, before = (rng.standard_normal(s).astype(np.float32) for s in ((rows, kv, dim), (rows, kv, dim), (rows, H * vdim), H, ac, batch * H * dim * vdim))
    q, k, v, a_log, dt = (dev.from_numpy(a) for a in (q / np.float32(dim ** 0.5), k / np.linalg.norm(k, axis=-1, keepdims=True), v, a_log, dt))
    slots = dev.from_numpy(np.arange(batch, dtype=np.int32))
    for name in ("ns_delta_recurrent", "ns_delta_chunked"):
        if name == "ns_delta_chunked" and dim > 128:
            continue

        def run(src, n):
            state, o = dev.from_numpy(before), dev.zeros(rows * H * vdim)
            N.call(name, dev.handle, u(q.ptr), kv * dim, u(k.ptr), kv * dim, u(v.ptr), H * vdim, u(src.ptr), n, ld, 0, u(src.ptr), n, ld, ac, u(a_log.ptr), u(dt.ptr), channelwise,
                   u(state.ptr), i64(H * dim * vdim), u(slots.ptr), batch, steps, H, kv, dim, vdim, u(o.ptr), H * vdim)
            return o, state

        same(dev, run, source, total, splits)


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("rows,heads,vdim", [(3, 2, 64), (3, 2, 61), (300, 16, 128), (5, 1, 1028), (2, 1, 4100), (2, 1, 601)])
def test_gated_norm(dev, rows, heads, vdim, splits):
    n = heads * vdim
    ld = (n + 7) // 8 * 8
    source, total = slabs_and_sum(dev, rows, ld, splits)
    o, w = (dev.from_numpy(rng_for(7, k, n).standard_normal(k).astype(np.float32)) for k in (rows * ld, vdim))
    for out in (N.NS_F32, N.NS_BF16):
        def norm(src, k):
            y = dev.zeros(rows * ld, out)
            N.call("ns_gated_norm", dev.handle, u(o.ptr), ld, u(src.ptr), k, N.NS_F32, ld, 0, N.ACT_SILU, u(w.ptr), fl(1e-4), i64(rows), heads, vdim, out, u(y.ptr), ld)
            return (y,)

        same(dev, norm, source, total, splits)


@pytest.mark.parametrize("splits", SPLITS)
@pytest.mark.parametrize("q_rank,kv_rank,rot", [(64, 32, 16), (61, 31, 14), (1024, 512, 64)])
def test_latent_rows(dev, q_rank, kv_rank, rot, splits):
    batch, steps, ring, n = 2, 5, 16, q_rank + kv_rank + rot
    ld, q_ld, r_ld, heads = (n + 7) // 8 * 8, (q_rank + 7) // 8 * 8, (kv_rank + rot + 7) // 8 * 8, 2
    source, total = slabs_and_sum(dev, batch * steps, ld, splits)
    wq, wk, freq = (dev.from_numpy(rng_for(8, k).standard_normal(k).astype(np.float32)) for k in (q_rank, kv_rank, rot // 2))
    slots, pos = dev.from_numpy(np.array([1, 0], np.int32)), dev.from_numpy(np.array([3, 14], np.int32))
    for dtype in (N.NS_F32, N.NS_BF16):
        def append(src, k):
            cq, rows = dev.zeros(batch * steps * q_ld, dtype), dev.zeros(2 * ring * r_ld, dtype)
            N.call("ns_latent_append", dev.handle, u(src.ptr), k, N.NS_F32, ld, q_rank, kv_rank, rot, rot, u(wq.ptr), u(wk.ptr), fl(1e-4), u(freq.ptr), u(slots.ptr), u(pos.ptr),
                   batch, steps, dtype, u(cq.ptr), q_ld, u(rows.ptr), i64(ring * r_ld), ring, r_ld)
            return cq, rows

        def rotate(src, k):
            dim = n // heads - rot
            plain, turned = dev.zeros(batch * steps * heads * dim, dtype), dev.zeros(batch * steps * heads * rot, dtype)
            N.call("ns_rotate_heads", dev.handle, u(src.ptr), k, N.NS_F32, ld, heads, dim, rot, rot, u(freq.ptr), u(slots.ptr), u(pos.ptr), batch, steps, dtype, u(plain.ptr),
                   i64(heads * dim), dim, dtype, u(turned.ptr), i64(heads * rot), rot)
            return plain, turned

        for run in (append, rotate):
            same(dev, run, source, total, splits)
