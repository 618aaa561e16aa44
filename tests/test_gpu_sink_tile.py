"""Prompt attention over rounded cache rows (with a workspace) against the kernel that converts tile by tile (without one): every form the call
takes, over shuffled cells of two sequences with NaN in the free ones.  Both round queries, rows and weights to bf16; the weights' roundings
differ where the running maxima do: 2^-9 / sqrt(3) each, so 2^-9 sqrt(2 / 3) = 1.6e-3 in the 2-norm, bound 3e-3.  And against float64 over the
rounded queries, keys and values: then only the rounding of the weights is left, 2^-9 / sqrt(3) = 1.13e-3 of every product in the 2-norm where
the products of a sum are independent; they are not all of one size, so twice that, 2.3e-3."""
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


def bf16(x):
    b = np.ascontiguousarray(x, np.float32).view(np.uint32).astype(np.uint64)
    return (((b + 0x7fff + ((b >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32).astype(np.float64)


def seen_by(f, cell_seq, cell_pos, tok_seq, tok_pos):
    """[token, cell]: which cells a token sees, by the words of include/b200_ggml_ops.h."""
    far = tok_pos[:, None].astype(np.int64) - cell_pos[None, :]
    seen = (cell_seq[None, :] >= 0) & (cell_seq[None, :] == tok_seq[:, None]) & (far >= 0)
    if f.get("window"):
        seen &= (far < f["window"]) | (cell_pos[None, :] < f.get("keep_first", 0))
    if f.get("chunk"):
        seen &= tok_pos[:, None] // f["chunk"] == cell_pos[None, :] // f["chunk"]
    return seen


def oracle(f, q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D, V, host):
    T, R = q.shape[0], Hh // G
    seen = seen_by(f, cell_seq, cell_pos, tok_seq, tok_pos)
    far = tok_pos[:, None].astype(np.int64) - cell_pos[None, :]
    used = cell_seq >= 0
    kk, vv = np.where(used[:, None], bf16(k), 0.0).reshape(-1, G, D), np.where(used[:, None], bf16(v), 0.0).reshape(-1, G, V)
    qq, out = bf16(q).reshape(T, Hh, D), np.zeros((T, Hh, V))
    for h in range(Hh):
        s = qq[:, h] @ kk[:, h // R].T * f.get("scale", D ** -0.5)
        if f.get("softcap"):
            s = f["softcap"] * np.tanh(s / f["softcap"])
        if "bias" in host:
            b = host["bias"][h].astype(np.float64)
            s = s + (b[0] * far if f.get("linear") else b[np.clip(far, 0, len(b) - 1)])
        if f.get("weights"):
            p = np.where(seen, 1.0 / (1.0 + np.exp(-s)), 0.0)
        else:
            s = np.where(seen, s, -np.inf)
            sink = host["sink"][h] if "sink" in host else -np.inf
            m = np.maximum(s.max(axis=1), sink)
            p = np.exp(s - m[:, None])
            p = p / (p.sum(axis=1) + np.exp(sink - m))[:, None]
        out[:, h] = p @ vv[:, h // R]
        if "gate" in host:
            g = host["gate"][:, h * V:(h + 1) * V] if f["gate"] == "value" else host["gate"][:, h:h + 1]
            out[:, h] /= 1.0 + np.exp(-g.astype(np.float64))
    return out.reshape(T, Hh * V) * (f.get("out_scale") or 1.0)


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
    extra, host = {}, {}
    if f.get("sink"):
        host["sink"] = rng.standard_normal(Hh).astype(np.float32)
        keep.append(H.DeviceBuffer.from_numpy(host["sink"]))
        extra["sink"] = keep[-1].ptr
    if f.get("table") or f.get("linear"):
        n = f.get("table", 1)
        host["bias"] = (rng.standard_normal((Hh, n)) * (0.02 if f.get("linear") else 1)).astype(np.float32)
        keep.append(H.DeviceBuffer.from_numpy(host["bias"]))
        extra.update(dist_bias=keep[-1].ptr, n_dist=n, dist_linear=1 if f.get("linear") else 0)
    if f.get("gate"):
        w = Hh * (V if f["gate"] == "value" else 1)
        host["gate"] = rng.standard_normal((T, w)).astype(np.float32)
        keep.append(H.DeviceBuffer.from_numpy(host["gate"]))
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
    exact = oracle(f, q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D, V, host)
    assert np.linalg.norm(got - exact) < 2.3e-3 * np.linalg.norm(exact)


def run_plain(q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D, window=0, workspace=True, chunk=0):
    T, cells = q.shape[0], k.shape[0]
    keep = [H.DeviceBuffer.from_numpy(x) for x in (q, k, v, cell_seq, cell_pos, tok_seq, tok_pos)]
    out = H.DeviceBuffer(4 * T * Hh * D)
    a = SinkAttnArgs(q=keep[0].ptr, q_stride=Hh * D, k_cache=keep[1].ptr, k_cache_stride=G * D, v_cache=keep[2].ptr, v_cache_stride=G * D, cell_seq=keep[3].ptr, cell_pos=keep[4].ptr,
                     tok_seq=keep[5].ptr, tok_pos=keep[6].ptr, dst=out.ptr, dst_stride=Hh * D, n_head=Hh, n_head_kv=G, dim=D, vdim=D, n_tokens=T, n_kv=cells, window=window,
                     scale=D ** -0.5, bf16_products=1, chunk=chunk)
    need = lib().b200_sink_attn_workspace_bytes(C.byref(a)) if workspace else 0
    assert need > 0 or not workspace
    ws = H.DeviceBuffer.from_numpy(np.full(need + 16, 0xff, np.uint8))  # (rows that are not written are NaN)
    check(lib().b200_op_sink_attn_ws(C.byref(a), ws.ptr if workspace else None, need, None))
    return out.to_numpy(np.float32, (T, Hh * D)).astype(np.float64)


def test_weights_are_rounded_as_without_workspace():
    """Both kernels take the running maximum over 32 cells at a time, so the roundings of the weights to bf16 agree but where the f32 values in front of them
    straddle a rounding border: scores up to about 5 differ by some 2^-21, relative to a bf16 step of 2^-8 that turns one weight in 2^12 by a step.
    A result of n such weights differs by 2^-8 sqrt(2^-12 / 3) = 3.5e-5 of its size; bound 1.5e-4 (roundings at different maxima gave 1.2e-3)."""
    T, Hh, G, D, past = 256, 16, 4, 128, 700
    rng = np.random.default_rng(5)
    cells = past + T + 12
    q, k, v = (rng.standard_normal((n, w * D)).astype(np.float32) for n, w in ((T, Hh), (cells, G), (cells, G)))
    at = np.arange(cells, dtype=np.int32)
    args = (q, k, v, np.where(at < past + T, 0, -1).astype(np.int32), at, np.zeros(T, np.int32), np.arange(past, past + T, dtype=np.int32), Hh, G, D)
    got, want = run_plain(*args), run_plain(*args, workspace=False)
    assert np.linalg.norm(got - want) < 1.5e-4 * np.linalg.norm(want)


def test_hidden_group_of_32_cells_beside_a_visible_one():
    """Cells 32 .. 63 of each tile of 64 belong to a sequence of which the batch has no token and hold infinities: they stay out of the products."""
    T, Hh, G, D, cells = 128, 24, 24, 64, 256
    rng = np.random.default_rng(3)
    q, k, v = (rng.standard_normal((n, w * D)).astype(np.float32) for n, w in ((T, Hh), (cells, G), (cells, G)))
    other = np.arange(cells) % 64 >= 32
    k[other], v[other] = np.inf, np.nan
    cell_seq, cell_pos = np.where(other, 1, 0).astype(np.int32), np.arange(cells, dtype=np.int32)
    tok_seq, tok_pos = np.zeros(T, np.int32), np.arange(cells, cells + T, dtype=np.int32)
    got = run_plain(q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D)
    assert np.isfinite(got).all()
    k[other], v[other] = 0.0, 0.0
    exact = oracle({}, q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D, D, {})
    assert np.linalg.norm(got - exact) < 2.3e-3 * np.linalg.norm(exact)


def test_tokens_of_many_sequences_in_turn():
    """Columns of one warp that belong to several sequences: what it sees of a half tile follows from its own tokens, not from whether cells are in use."""
    T, Hh, G, D, n_seq, each = 192, 16, 16, 64, 6, 128
    rng = np.random.default_rng(21)
    cells = n_seq * each
    q, k, v = (rng.standard_normal((n, w * D)).astype(np.float32) for n, w in ((T, Hh), (cells, G), (cells, G)))
    cell_seq, cell_pos = (np.arange(cells) // each).astype(np.int32), (np.arange(cells) % each).astype(np.int32)
    # tokens 0 .. 95: sequences 0 and 1 in turn; 96 .. 191: 2 to 5 in turn
    tok_seq = np.where(np.arange(T) < 96, np.arange(T) % 2, 2 + np.arange(T) % 4).astype(np.int32)
    tok_pos = np.where(np.arange(T) < 96, np.arange(T) // 2 + each - 48, (np.arange(T) - 96) // 4 + each - 24).astype(np.int32)
    for f in ({}, {"window": 30}, {"chunk": 64}):
        got = run_plain(q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D, window=f.get("window", 0), chunk=f.get("chunk", 0))
        exact = oracle(f, q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D, D, {})
        assert np.linalg.norm(got - exact) < 2.3e-3 * np.linalg.norm(exact)
    # what sequences 2 to 5 hold does not reach the first tokens' results
    other = cell_seq >= 2
    k[other], v[other] = np.inf, np.nan
    got = run_plain(q, k, v, cell_seq, cell_pos, tok_seq, tok_pos, Hh, G, D)
    assert np.isfinite(got[:96]).all()
