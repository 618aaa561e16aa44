"""The gated delta rule scan takes four tokens at a time: lengths around whole groups and whole chunks, every width of the state, one decay a head and one a
channel, and more CTAs than SMs."""
import ctypes as C
import math

import numpy as np
import pytest

from koboldcpp_b200 import host as H
from koboldcpp_b200.lib import DeltaRuleArgs, check, lib

pytestmark = pytest.mark.gpu


def dev(x, dtype=np.float32):
    return H.DeviceBuffer.from_numpy(np.ascontiguousarray(x, dtype), pad=256)


def run(lengths, heads, kv, D, V, channel, seed, poison=None):
    """Sequences of these lengths behind one another, every second one fresh, in slots in reverse order; the result and the states, and both in 64 bits.
    poison: (token, value) for all of that token's v."""
    rng = np.random.default_rng(seed)
    T, n = sum(lengths), len(lengths)
    gates = heads * (D if channel else 1)
    q, k, v = rng.standard_normal((T, kv, D)), rng.standard_normal((T, kv, D)), rng.standard_normal((T, heads, V))
    a, b, a_log, dt = rng.standard_normal((T, gates)), rng.standard_normal((T, heads)), rng.uniform(-2, 1, heads), rng.standard_normal(gates)
    q, k, v, a, b, a_log, dt = (x.astype(np.float32).astype(np.float64) for x in (q, k, v, a, b, a_log, dt))
    if poison:
        v[poison[0]] = poison[1]
    slot = heads * D * V + (0 if seed % 2 else 3)  # (columns of the state on 16 bytes, or not)
    start = rng.standard_normal((n, slot)).astype(np.float32)
    first = np.concatenate([[0], np.cumsum(lengths)[:-1]])
    info = np.stack([first, lengths, np.arange(n)[::-1], np.arange(n) % 2]).astype(np.int32)
    bufs = [dev(x) for x in (q, k, v, a, b, a_log, dt, start)]
    dq, dk, dv, da, db, dl, dd, ds = bufs
    dinfo, dy = dev(info, np.int32), H.DeviceBuffer(4 * T * heads * V + 256)
    args = DeltaRuleArgs(q=dq.ptr, k=dk.ptr, v=dv.ptr, q_stride=kv * D, k_stride=kv * D, v_stride=heads * V, a=da.ptr, b=db.ptr, a_stride=gates, b_stride=heads, a_log=dl.ptr,
                         dt_bias=dd.ptr, seq_info=dinfo.ptr, n_seq=n, state=ds.ptr, slot_stride=slot, dst=dy.ptr, dst_stride=heads * V, heads=heads, kv_heads=kv, dim=D, vdim=V, unit_qk=1,
                         unit_eps=1e-6, q_scale=D ** -0.5, channel_decay=1 if channel else 0)
    check(lib().b200_op_delta_rule_scan(C.byref(args), None))
    got, states = dy.to_numpy(np.float32, (T, heads, V)), ds.to_numpy(np.float32, (n, slot))
    qn = np.repeat(q / np.sqrt((q * q).sum(-1, keepdims=True) + 1e-6), heads // kv, 1) * D ** -0.5
    kn = np.repeat(k / np.sqrt((k * k).sum(-1, keepdims=True) + 1e-6), heads // kv, 1)
    soft = np.logaddexp(0, a + dt).reshape(T, heads, -1)
    g, beta = np.exp(-np.exp(a_log)[:, None] * soft)[:, :, None, :], 1 / (1 + np.exp(-b))
    want, ends = np.zeros((T, heads, V)), start.astype(np.float64)
    for i, (t0, m) in enumerate(zip(first, lengths)):
        at = n - 1 - i
        S = ends[at, :heads * D * V].reshape(heads, V, D) * (0 if i % 2 else 1)
        for t in range(t0, t0 + m):
            S = S * g[t]
            u = beta[t][:, None] * (v[t] - np.einsum("hvd,hd->hv", S, kn[t]))
            S = S + u[:, :, None] * kn[t][:, None, :]
            want[t] = np.einsum("hvd,hd->hv", S, qn[t])
        if m:
            ends[at, :heads * D * V] = S.reshape(-1)
    return got, want, states, ends


def rel(x, y):
    return float(np.linalg.norm(x - y) / np.linalg.norm(y))


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("lengths,heads,kv,D,V", [([3, 4, 5, 0, 1], 2, 1, 32, 8), ([7, 8, 9], 4, 2, 33, 40), ([15, 16, 17], 2, 2, 64, 33), ([31, 2, 32], 2, 1, 65, 16), ([35, 18], 3, 3, 128, 64),
                                                  ([19, 20, 21, 22], 2, 1, 129, 7), ([37], 1, 1, 256, 35), ([23, 1, 6], 28, 14, 128, 64)])
def test_delta_scan_around_groups_and_chunks(lengths, heads, kv, D, V, channel):
    # f32 sums over dim values and over the tokens that still count (a few tens): about sqrt(256 + 37) roundings of 6e-8 each way, so 2e-6 with room
    got, want, states, ends = run(lengths, heads, kv, D, V, channel, seed=D + V)
    assert rel(got, want) < 2e-6 and rel(states, ends) < 2e-6


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("at", [16, 17, 18, 19])
def test_what_is_not_finite_stays_behind_its_token(at, channel):
    """Tokens of one group go through shared sums; an infinity must not reach the tokens in front of it."""
    got, want, _, _ = run([24], 2, 1, 64, 32, channel, seed=at, poison=(at, math.inf))
    assert np.isfinite(got[:at]).all() and rel(got[:at], want[:at]) < 2e-6
    assert not np.isfinite(got[at:]).any()
