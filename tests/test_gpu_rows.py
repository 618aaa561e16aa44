"""Element-wise rows in their wide and narrow forms: gated SiLU and RMS norm at sizes around the pieces a thread handles, aligned and not, in place."""
import ctypes as C

import numpy as np
import pytest

import koboldcpp_b200.host as H
from koboldcpp_b200.lib import F32, Tensor, check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 2044, 2048, 2052, 4100, 11008 * 3])
@pytest.mark.parametrize("offset,act", [(0, True), (0, False), (4, False)])
def test_silu_mul(n, offset, act):
    rng = np.random.default_rng(n)
    g, u = (rng.standard_normal(n).astype(np.float32) * 4 for _ in range(2))
    want = g.astype(np.float64) / (1 + np.exp(-g.astype(np.float64)))
    pad = np.zeros(offset // 4, np.float32)
    dg, du = H.DeviceBuffer.from_numpy(np.concatenate([pad, g])), H.DeviceBuffer.from_numpy(np.concatenate([pad, u]))
    da = H.DeviceBuffer(4 * n + 16) if act else None
    check(lib().b200_op_silu_mul(dg.ptr + offset, du.ptr + offset, da.ptr if act else None, dg.ptr + offset, n, None))  # in place over gate
    got = dg.to_numpy(np.float32, (n + offset // 4,))[offset // 4:]
    np.testing.assert_allclose(got, want * u, rtol=1e-6, atol=1e-6)  # a few roundings in f32 behind expf's two ulp
    if act:
        np.testing.assert_allclose(da.to_numpy(np.float32, (n,)), want, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("n", [4, 100, 252, 256, 260, 1020, 1024, 1028, 4096, 5120, 16384, 16388])
@pytest.mark.parametrize("gap,keep", [(0, True), (4, False), (3, False)])
def test_rms_norm_mul(n, gap, keep):
    rows, eps = 5, 1e-5
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((rows, n + gap)) * 3).astype(np.float32)
    w = rng.standard_normal(n).astype(np.float32)
    z = x[:, :n].astype(np.float64)
    z = z / np.sqrt((z * z).mean(1, keepdims=True) + eps)
    dx, dw, dn = H.DeviceBuffer.from_numpy(x), H.DeviceBuffer.from_numpy(w), H.DeviceBuffer(4 * rows * n)
    t = Tensor.contiguous(dx.ptr, F32, (n, rows))
    for i in (1, 2, 3):
        t.nb[i] = 4 * (n + gap) * (1 if i == 1 else rows)
    check(lib().b200_op_rms_norm_mul(C.byref(t), dw.ptr, dn.ptr if keep else None, C.byref(t), eps, None))  # in place
    got = dx.to_numpy(np.float32, (rows, n + gap))
    np.testing.assert_allclose(got[:, :n], z * w, rtol=2e-6, atol=2e-6)  # f32 sums of up to 16388 squares, rsqrt of two ulp
    np.testing.assert_array_equal(got[:, n:], x[:, n:])
    if keep:
        np.testing.assert_allclose(dn.to_numpy(np.float32, (rows, n)), z, rtol=2e-6, atol=2e-6)
