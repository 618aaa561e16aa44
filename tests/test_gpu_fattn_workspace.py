"""One workspace, zeroed once, serves prompts, batches of a few tokens and single tokens in turn: what one plan leaves in its scratch must not be another
one's arrival counters.  40 heads of 128 without groups: 20 tokens are 80 (kv-head, column tile) pairs, more counters than fit 256 bytes."""
import ctypes as C

import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import F16, Q8_0, FattnArgs, check, lib

pytestmark = pytest.mark.gpu


class Call:
    def __init__(self, tokens, cells, heads=40, D=128, kind=F16):
        rng = np.random.default_rng(tokens + cells)
        q, k, v = rng.standard_normal((heads, tokens, D)).astype(np.float32), rng.standard_normal((heads, cells, D)), rng.standard_normal((heads, cells, D))
        mask = np.zeros(((tokens + 31) // 32 * 32, cells), np.float16)
        for i in range(tokens):
            mask[i, cells - tokens + 1 + i:] = -np.inf
        pk, pv = O.pack_kv(kind, k), O.pack_kv(kind, v)
        row = pk.shape[2]
        self.keep = [H.DeviceBuffer.from_numpy(x, pad=64) for x in (q, pk, pv, mask)]
        self.nan, self.shape = np.full((tokens, heads, D), np.nan, np.float32), (tokens, heads, D)
        self.dst = H.DeviceBuffer.from_numpy(self.nan)
        dq, dk, dv, dm = (b.ptr for b in self.keep)
        self.args = FattnArgs(dq, dk, dv, dm, self.dst.ptr, D, tokens, heads, heads, cells, kind, kind, 4 * D, 4 * D * tokens, row, row * cells, row, row * cells, 2 * cells, D ** -0.5, 0.0, 0.0)
        self.bytes = int(lib().b200_flash_attn_workspace_bytes(C.byref(self.args)))

    def run(self, ws):
        check(lib().b200_memcpy_h2d(self.dst.ptr, self.nan.ctypes.data, self.nan.nbytes, None))
        check(lib().b200_flash_attn_ext(C.byref(self.args), ws.ptr, ws.nbytes, None))
        return self.dst.to_numpy(np.float32, self.shape)


def test_one_workspace_for_all_shapes():
    calls = [Call(64, 512), Call(20, 2816), Call(1, 2816), Call(20, 4096), Call(200, 1024, 32, 64), Call(40, 1024, 40, 128, Q8_0)]
    alone = [c.run(H.DeviceBuffer(max(c.bytes, 256), zero=True)) for c in calls]
    assert all(np.isfinite(x).all() for x in alone)
    shared = H.DeviceBuffer(max(c.bytes for c in calls), zero=True)
    for order in ([0, 1, 2, 1, 0, 3], [2, 1, 3, 0, 2, 3], [4, 1, 5, 3, 5, 2, 4, 1]):
        for i in order:
            assert np.array_equal(calls[i].run(shared), alone[i]), (order, i)
