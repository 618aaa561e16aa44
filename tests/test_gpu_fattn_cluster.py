"""Decoding over short caches: splits that are one thread-block cluster merge in shared memory.  Lengths around one tile a warp and 2, 4 and 8 splits, every number
of columns, both cache types of that kernel, against float64 over the rows as they are stored."""
import ctypes as C

import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import F16, Q8_0, FattnArgs, check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("heads,kv_heads,kind", [(1, 1, F16), (4, 2, F16), (8, 1, F16), (32, 4, F16), (2, 2, Q8_0), (5, 5, Q8_0)])
@pytest.mark.parametrize("n_kv", [16, 64, 127, 128, 129, 250, 256, 511, 520, 1024, 1100, 2048])
def test_short_caches(D, heads, kv_heads, kind, n_kv):
    rng = np.random.default_rng(n_kv + heads + D)
    q, k, v = rng.standard_normal((heads, 1, D)).astype(np.float32), rng.standard_normal((kv_heads, n_kv, D)), rng.standard_normal((kv_heads, n_kv, D))
    mask = np.zeros((32, n_kv), np.float16)
    mask[:, (3 * n_kv + 3) // 4:] = -np.inf      # (a split of the cluster may see nothing)
    pk, pv = O.pack_kv(kind, k), O.pack_kv(kind, v)
    exact = O.flash_attn_f64(q, pk, pv, mask, kind, D ** -0.5)
    # queries rounded to f16 (a score off by about 2^-12), or to q8_0 (a score off by about 1/250 of its deviation of 1, results of size up to 1 .. 4 by that)
    assert np.abs(H.flash_attn_ext(q, pk, pv, mask, kind, D ** -0.5) - exact).max() <= (2.5e-3 if kind == F16 else 2.5e-2)


@pytest.mark.parametrize("n_kv", [40, 100, 200])
def test_short_caches_without_a_workspace(n_kv):
    """What needs no workspace, because it was never split, is served without one."""
    rng = np.random.default_rng(n_kv)
    D, heads = 64, 4
    q, k, v = rng.standard_normal((heads, 1, D)).astype(np.float32), rng.standard_normal((heads, n_kv, D)), rng.standard_normal((heads, n_kv, D))
    pk, pv = O.pack_kv(F16, k), O.pack_kv(F16, v)
    dq, dk, dv, dd = H.DeviceBuffer.from_numpy(q), H.DeviceBuffer.from_numpy(pk, pad=64), H.DeviceBuffer.from_numpy(pv, pad=64), H.DeviceBuffer(4 * heads * D)
    a = FattnArgs(dq.ptr, dk.ptr, dv.ptr, None, dd.ptr, D, 1, heads, heads, n_kv, F16, F16, 4 * D, 4 * D, 2 * D, 2 * D * n_kv, 2 * D, 2 * D * n_kv, 0, 0.125, 0.0, 0.0)
    check(lib().b200_flash_attn_ext(C.byref(a), None, 0, None))
    assert np.abs(dd.to_numpy(np.float32, (1, heads, D)) - O.flash_attn_f64(q, pk, pv, None, F16, 0.125)).max() <= 2.5e-3
