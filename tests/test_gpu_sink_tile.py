"""Prompt attention over rounded cache rows (with a workspace) against the kernel that converts tile by tile (without one, itself tested against
float64): every form the call takes, over shuffled cells of two sequences with NaN in the free ones.  Both round queries, rows and weights to bf16;
the weights' roundings differ where the running maxima do: 2^-9 / sqrt(3) each, so 2^-9 sqrt(2 / 3) = 1.6e-3 in the 2-norm, bound 3e-3."""
import ctypes as C

import numpy as np
import pytest

import koboldcpp_b200.host as H
from koboldcpp_b200.lib import SinkAttnArgs, check, lib

pytestmark = pytest.mark.gpu

FORMS = [
    dict(), dict(window=40), dict(window=40, keep_first=3), dict(chunk=64), dict(sink=True), dict(softcap=5.0), dict(weights=1), dict(weights=1, table=50),
    dict(table=30), dict(linear=True), dict(gate="head", out_scale=0.5), dict(gate="value", sink=True), dict(scale=-0.1), dict(one=True), dict(one=True, window=100),
]


@pytest.mark.parametrize("form", range(len(FORMS)))
@pytest.mark.parametrize("D,V,G,R,T", [(128, 128, 24, 2, 64), (64, 64, 48, 1, 33), (20, 100, 8, 7, 70), (96, 30, 48, 1, 64), (70, 128, 16, 3, 70)])
def test_with_and_without_workspace(form, D, V, G, R, T):
    f = FORMS[form]
    Hh, cells = G * R, 300
    rng = np.random.default_rng(form * 7 + D)
    order = rng.permutation(cells)
    used = 270
    n1 = used if f.get("one") else 180
    cell_seq, cell_pos = np.full(cells, -1, np.int32), np.zeros(cells, np.int32)
    cell_seq[order[:n1]], cell_pos[order[:n1]] = 0, np.arange(n1)
    cell_seq[order[n1:used]], cell_pos[order[n1:used]] = 1, np.arange(used - n1)
    if f.get("one"):  # cells in order: tiles that are seen wholly
        cell_seq[:], cell_pos[:] = -1, 0
        cell_seq[:used], cell_pos[:used] = 0, np.arange(used)
    k, v = (rng.standard_normal((cells, G * d)).astype(np.float32) for d in (D, V))
    k[cell_seq < 0], v[cell_seq < 0] = np.nan, np.nan
    half = T if f.get("one") else T // 2
    tok_seq = np.where(np.arange(T) < half, 0, 1).astype(np.int32)
    tok_pos = np.where(np.arange(T) < half, n1 - half + np.arange(T), (used - n1) - T + np.arange(T)).astype(np.int32)
    q = rng.standard_normal((T, Hh * D)).astype(np.float32)
    keep = [H.DeviceBuffer.from_numpy(x) for x in (q, k, v, cell_seq, cell_pos, tok_seq, tok_pos)]
    extra = {}
    if f.get("sink"):
        keep.append(H.DeviceBuffer.from_numpy(rng.standard_normal(Hh).astype(np.float32)))
        extra["sink"] = keep[-1].ptr
    if f.get("table") or f.get("linear"):
        n = f.get("table", 1)
        keep.append(H.DeviceBuffer.from_numpy((rng.standard_normal((Hh, n)) * (0.02 if f.get("linear") else 1)).astype(np.float32)))
        extra.update(dist_bias=keep[-1].ptr, n_dist=n, dist_linear=1 if f.get("linear") else 0)
    if f.get("gate"):
        w = Hh * (V if f["gate"] == "value" else 1)
        keep.append(H.DeviceBuffer.from_numpy(rng.standard_normal((T, w)).astype(np.float32)))
        extra.update(gate=keep[-1].ptr, gate_stride=w, gate_per_value=1 if f["gate"] == "value" else 0)
    out = H.DeviceBuffer(4 * T * Hh * V)
    a = SinkAttnArgs(q=keep[0].ptr, q_stride=Hh * D, k_cache=keep[1].ptr, k_cache_stride=G * D, v_cache=keep[2].ptr, v_cache_stride=G * V, cell_seq=keep[3].ptr,
                     cell_pos=keep[4].ptr, tok_seq=keep[5].ptr, tok_pos=keep[6].ptr, dst=out.ptr, dst_stride=Hh * V, n_head=Hh, n_head_kv=G, dim=D, vdim=V, n_tokens=T, n_kv=cells,
                     window=f.get("window", 0), keep_first=f.get("keep_first", 0), scale=f.get("scale", D ** -0.5), bf16_products=1, chunk=f.get("chunk", 0),
                     weights=f.get("weights", 0), out_scale=f.get("out_scale", 0.0), softcap=f.get("softcap", 0.0), **extra)
    need = lib().b200_sink_attn_workspace_bytes(C.byref(a))
    if T * R * G >= 48 * 64:
        assert need > 0
    ws = H.DeviceBuffer(need + 16)
    check(lib().b200_op_sink_attn_ws(C.byref(a), ws.ptr, need, None))
    got = out.to_numpy(np.float32, (T, Hh * V)).astype(np.float64)
    check(lib().b200_op_sink_attn(C.byref(a), None))
    want = out.to_numpy(np.float32, (T, Hh * V)).astype(np.float64)
    assert np.isfinite(got).all()
    assert np.linalg.norm(got - want) < 3e-3 * np.linalg.norm(want)
