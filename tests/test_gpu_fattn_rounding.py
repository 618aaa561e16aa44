"""Roundings of prompt attention on tcgen05: queries and weights go through f16, and the running maximum may lag.  Wherever the energy of the queries lies among
the dims, the result is no further from 64 bits than with weights rounded beside a maximum that never lags."""
import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import F16

pytestmark = pytest.mark.gpu


def f16(x):
    return x.astype(np.float16).astype(np.float64)


def rounded(q, k, v, scale):
    """Queries and weights as f16, tiles of 64 keys, each tile's weights beside the maximum so far."""
    out = np.empty(q.shape)
    for h in range(len(q)):
        s = f16(q[h]) @ k[h].T * scale
        m, l, o = np.full((len(s), 1), -np.inf), 0.0, 0.0
        for t in range(0, s.shape[1], 64):
            x = s[:, t:t + 64]
            top = np.maximum(m, x.max(1, keepdims=True))
            w, a = np.exp(x - top), np.exp(m - top)
            m, l, o = top, l * a + w.sum(1, keepdims=True), o * a + f16(w) @ v[h, t:t + 64]
        out[h] = o / l
    return out


DIMS = {"all": slice(0, None), "last three quarters": slice(32, None), "last quarter": slice(96, None), "one block": slice(48, 64), "odd ones": slice(1, None, 2)}


@pytest.mark.parametrize("sharp", [1.0, 3.0])
@pytest.mark.parametrize("where", list(DIMS))
@pytest.mark.parametrize("D", [64, 128])
def test_no_further_from_64_bits_than_without_the_lag(D, where, sharp):
    rng = np.random.default_rng(D + len(where))
    heads, N, cells = 4, 256, 1024
    at = np.zeros(128)
    at[DIMS[where]] = 1
    at = at.reshape(-1, 128 // D).max(1)
    q = (rng.standard_normal((heads, N, D)) * at * np.sqrt(D / at.sum())).astype(np.float32)
    k, v = f16(sharp * rng.standard_normal((heads, cells, D))), f16(rng.standard_normal((heads, cells, D)))
    s = q.astype(np.float64) @ k.transpose(0, 2, 1) * D ** -0.5
    w = np.exp(s - s.max(2, keepdims=True))
    exact = w @ v / w.sum(2, keepdims=True)  # (queries as they are, not as f16)
    got = H.flash_attn_ext(q, O.pack_kv(F16, k), O.pack_kv(F16, v), None, F16, D ** -0.5).transpose(1, 0, 2)
    err = lambda x: np.linalg.norm(x - exact) / np.linalg.norm(exact)
    # 0.5 % for the noise of the comparison itself: 131072 (65536) errors a side, of which the larger part is the same in both
    assert err(got) <= 1.005 * err(rounded(q, k, v, D ** -0.5))
