"""The streaming bf16 product of few rows: edges of its tiles (16 columns), units (128 elements of K), shares of warps and CTAs, and of the
sizes it is chosen for, against float64."""
import ctypes as C

import numpy as np
import pytest

from nn_b200 import native as N

pytestmark = pytest.mark.gpu
u64 = C.c_uint64


def _bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


def _wide(b):
    return (b.astype(np.uint32) << 16).view(np.float32).astype(np.float64)


@pytest.mark.parametrize("n,k", [(8, 8), (16, 128), (24, 72), (40, 1032), (1000, 264), (2368, 2048), (2376, 136), (4096, 2048), (4104, 2048), (2048, 5632),
                                 (4800, 5120), (32000, 256), (768, 8192), (2400, 8192), (2048, 9216), (2048, 10240), (42624, 264), (42640, 264), (42640, 256)])
def test_products(dev, n, k):
    rng = np.random.default_rng(n * 7 + k)
    w = _bf16(rng.standard_normal((n, k)))
    h = C.c_void_p()
    N.call("ns_linear_create_bf16", dev.handle, n, k, w.ctypes.data_as(C.c_void_p), C.byref(h))
    wide = _wide(w)
    rows = {}
    for m in (1, 5, 8, 9, 16, 17, 64, 128):
        x = _bf16(np.random.default_rng(3).standard_normal((128, k))[:m])
        d_x, d_y = dev.from_numpy(x), dev.from_numpy(np.full((m + 1, n), 7.0, np.float32))
        N.call("ns_linear_forward", dev.handle, h, u64(d_x.ptr), u64(0), m, N.EPI_NONE, u64(0), N.NS_F32, N.NS_F32, u64(d_y.ptr))
        dev.synchronize()
        y = d_y.download((m + 1, n))
        assert np.all(y[m] == 7.0)                               # nothing behind the matrix
        # K products of bf16 are exact in float; each of at most K + 16 sums is off by less than 2^-22 of the sum of magnitudes (the tensor
        # cores' sums drop bits below the largest term's last one)
        a = _wide(x)
        assert np.all(np.abs(y[:m] - a @ wide.T) <= (k + 16) * 2.0 ** -22 * (np.abs(a) @ np.abs(wide).T))
        ptr, splits = u64(), C.c_int()
        N.call("ns_linear_forward_partial", dev.handle, h, u64(d_x.ptr), m, C.byref(ptr), C.byref(splits))
        slabs = dev.empty(splits.value * m * n, N.NS_F32)
        N.call("ns_d2d_async", dev.handle, u64(slabs.ptr), ptr, u64(4 * splits.value * m * n))
        dev.synchronize()
        slabs = slabs.download((splits.value, m, n))
        # tiles that divide badly and rows that are too long are split for the row kernel, and from some length on for a finished matrix too
        if m <= 8 and (n, k) not in ((4800, 5120), (768, 8192), (2400, 8192), (2048, 10240), (42640, 264)):
            assert splits.value == 1 and np.array_equal(slabs[0], y[:m])
        assert np.all(np.abs(slabs.astype(np.float64).sum(0) - a @ wide.T) <= (k + 16) * 2.0 ** -22 * (np.abs(a) @ np.abs(wide).T))
        rows[m] = y[0]
        d_b = dev.empty(m * n, N.NS_BF16)
        N.call("ns_linear_forward", dev.handle, h, u64(d_x.ptr), u64(0), m, N.EPI_NONE, u64(0), N.NS_F32, N.NS_BF16, u64(d_b.ptr))
        dev.synchronize()
        assert np.array_equal(d_b.download((m, n)), _bf16(y[:m]))
    # a row does not depend on the others, nor on how many there are, within what one kernel takes: one to eight rows (to sixteen of narrow products), and
    # up to 128
    few = [m for m in rows if m <= (16 if k <= 2048 and n <= 4096 else 8)] if (n, k) not in ((2400, 8192), (2048, 10240), (42640, 264)) else []
    for of in (few, [m for m in rows if m not in few]):
        assert all(np.array_equal(rows[of[0]], rows[m]) for m in of)
    N.call("ns_linear_destroy", h)


@pytest.mark.parametrize("m", [3, 11])
@pytest.mark.parametrize("epilogue", [N.EPI_BIAS, N.EPI_BIAS_GELU, N.EPI_BIAS_RESIDUAL])
def test_epilogues(dev, orc, m, epilogue):
    n, k = 300, 392
    a, b = orc.round_bf16(orc.normal((m, k), 41)), orc.round_bf16(orc.normal((n, k), 42))
    bias, res = orc.normal((n,), 43), orc.normal((m, n), 44)
    d_a, d_b, d_bias, d_res, d_c = dev.from_numpy(a), dev.from_numpy(b), dev.from_numpy(bias), dev.from_numpy(res), dev.empty(m * n, N.NS_F32)
    N.call("ns_matmul_bf16", dev.handle, d_a.ptr, d_b.ptr, d_c.ptr, 1, m, n, k, 1, d_bias.ptr, d_res.ptr if epilogue == N.EPI_BIAS_RESIDUAL else 0, N.NS_F32,
           epilogue, N.NS_F32)
    dev.synchronize()
    exp = orc.matmul_bf16(a, b, b_is_nk=True).astype(np.float64) + bias
    if epilogue == N.EPI_BIAS_GELU:
        exp = 0.5 * exp * (1 + np.tanh(0.7978845608 * (exp + 0.044715 * exp ** 3)))
    if epilogue == N.EPI_BIAS_RESIDUAL:
        exp = exp + res
    assert orc.close(exp.astype(np.float32), d_c.download((m, n)), 1e-4)      # as test_gemm_bf16: sums of 392 terms in another order
