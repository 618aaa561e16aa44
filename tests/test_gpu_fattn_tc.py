"""Prompt attention over an f16 cache on tcgen05: edges of its tiles (128 columns, 64 keys, four buffers), masks read ahead or from the table in the
workspace, cells that hold no finite values.  Against float64 over the rows as they are stored, with the bound of tests/test_gpu_fattn_prefill.py."""
import ctypes as C

import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import F16, FattnArgs, check, lib

pytestmark = pytest.mark.gpu

BOUND = 2.5e-3


def causal(N, n_kv, n_past, window=0):
    mask = np.full(((N + 31) // 32 * 32, n_kv), -np.inf, np.float16)
    for i in range(N):
        mask[i, max(0, n_past + i + 1 - window) if window else 0:min(n_kv, n_past + i + 1)] = 0
    return mask


def run(q, k, v, mask, scale, scratch=True, interleaved=False):
    """b200_flash_attn_ext with or without a workspace; interleaved: a cache row holds all kv-heads of a token."""
    heads, N, D = q.shape
    kv_heads, n_kv, _ = k.shape
    k16, v16 = k.astype(np.float16), v.astype(np.float16)
    if interleaved:
        k16, v16 = np.ascontiguousarray(k16.transpose(1, 0, 2)), np.ascontiguousarray(v16.transpose(1, 0, 2))
        nb1, nb2 = 2 * D * kv_heads, 2 * D
    else:
        nb1, nb2 = 2 * D, 2 * D * n_kv
    dq, dk, dv = H.DeviceBuffer.from_numpy(q.astype(np.float32)), H.DeviceBuffer.from_numpy(k16.view(np.uint8), pad=64), H.DeviceBuffer.from_numpy(v16.view(np.uint8), pad=64)
    dm = None if mask is None else H.DeviceBuffer.from_numpy(mask)
    dd = H.DeviceBuffer(4 * N * heads * D)
    a = FattnArgs(dq.ptr, dk.ptr, dv.ptr, dm.ptr if dm else None, dd.ptr, D, N, heads, kv_heads, n_kv, F16, F16, 4 * D, 4 * D * N, nb1, nb2, nb1, nb2, 2 * n_kv if dm else 0, scale, 0.0, 0.0)
    ws = H.DeviceBuffer(max(int(lib().b200_flash_attn_workspace_bytes(C.byref(a))), 256), zero=True) if scratch else None
    check(lib().b200_flash_attn_ext(C.byref(a), ws.ptr if ws else None, ws.nbytes if ws else 0, None))
    out = dd.to_numpy(np.float32, (N, heads, D))
    assert lib().b200_gemm_status() == 0
    return out


def inputs(heads, kv_heads, N, n_kv, D, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((heads, N, D)).astype(np.float32), rng.standard_normal((kv_heads, n_kv, D)), rng.standard_normal((kv_heads, n_kv, D))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("heads,kv_heads,N,n_kv,window", [
    (1, 1, 33, 64, 0), (2, 2, 127, 128, 0), (1, 1, 128, 136, 0), (2, 1, 129, 192, 0), (3, 1, 100, 200, 0), (4, 4, 257, 320, 0), (4, 4, 64, 448, 0),
    (8, 2, 40, 1600, 0), (2, 2, 130, 1024, 100), (6, 1, 50, 832, 64), (5, 5, 40, 2048, 300),
])
def test_edges_of_tiles(D, heads, kv_heads, N, n_kv, window):
    q, k, v = inputs(heads, kv_heads, N, n_kv, D, N + n_kv)
    mask = causal(N, n_kv, n_kv - N if n_kv > N else 0, window)
    exact = O.flash_attn_f64(q, O.pack_kv(F16, k), O.pack_kv(F16, v), mask, F16, D ** -0.5)
    got = run(q, k, v, mask, D ** -0.5)
    assert np.abs(got - exact).max() <= BOUND
    assert np.array_equal(run(q, k, v, mask, D ** -0.5, scratch=False), got)      # the mask from L2 instead of the table
    assert np.array_equal(run(q, k, v, mask, D ** -0.5, interleaved=True), got)


def test_sequences_side_by_side_and_growing_scores():
    """Tokens of three sequences in one batch, cells in stretches; scores that grow along the keys move the running maximum again and again."""
    N, n_kv, D = 150, 768, 128
    q, k, v = inputs(4, 4, N, n_kv, D, 1)
    q = q.astype(np.float16).astype(np.float32)  # (scores of 30 and more: an f16 rounding of the queries would be the larger part of the difference)
    k *= np.linspace(0.2, 6.0, n_kv)[None, :, None]
    mask = np.full((160, n_kv), -np.inf, np.float16)
    for i in range(N):
        s = i // 50
        mask[i, 256 * s:256 * s + 60 + 3 * (i % 50)] = 0
    exact = O.flash_attn_f64(q, O.pack_kv(F16, k), O.pack_kv(F16, v), mask, F16, 0.2)
    assert np.abs(run(q, k, v, mask, 0.2) - exact).max() <= BOUND


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("what", ["v nan", "v inf", "k nan"])
def test_a_cell_without_finite_values_stays_with_those_that_see_it(D, what):
    N, n_kv, cell = 140, 320, 250
    q, k, v = inputs(2, 1, N, n_kv, D, D)
    mask = causal(N, n_kv, n_kv - N)
    exact = O.flash_attn_f64(q, O.pack_kv(F16, k), O.pack_kv(F16, v), mask, F16, D ** -0.5)
    (k if what[0] == "k" else v)[0, cell] = np.inf if what[2:] == "inf" else np.nan
    got = run(q, k, v, mask, D ** -0.5)
    sees = mask[:N, cell] == 0
    assert np.isfinite(got[~sees]).all() and np.abs(got[~sees] - exact[~sees]).max() <= BOUND
    assert not np.isfinite(got[sees]).any()
