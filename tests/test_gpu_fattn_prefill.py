"""Attention of prompt batches over an f16 cache, tiles of 64 keys (32 for heads wider than 128): masks at any place, cells that nobody sees, ragged
ends.  Against float64 over the rows as they are stored; the bound is that of tests/test_gpu_kernels.py for outputs of size 0.3 (P rounded to f16, at most
2^-11 of the largest value, some 4, beside f16 roundings of the queries)."""
import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import F16

pytestmark = pytest.mark.gpu

BOUND = 2.5e-3


def causal(N, n_kv, n_past):
    mask = np.full(((N + 31) // 32 * 32, n_kv), -np.inf, np.float16)
    for i in range(N):
        mask[i, :min(n_kv, n_past + i + 1)] = 0
    return mask


def poisoned_run(q, k, v, mask, hidden, scale, **kw):
    """The result with sane and with poisoned hidden cells: the same bits; returns it and the float64 one."""
    kf, vf = k.copy(), v.copy()
    exact = O.flash_attn_f64(q, O.pack_kv(F16, k), O.pack_kv(F16, v), mask, F16, scale, **kw)
    got = H.flash_attn_ext(q, O.pack_kv(F16, k), O.pack_kv(F16, v), mask, F16, scale, **kw)
    kf[:, hidden], vf[:, hidden] = np.inf, np.nan
    again = H.flash_attn_ext(q, O.pack_kv(F16, kf), O.pack_kv(F16, vf), mask, F16, scale, **kw)
    assert np.isfinite(again).all() and np.array_equal(again, got)
    return got, exact


@pytest.mark.parametrize("D", [64, 80, 128, 256])
@pytest.mark.parametrize("n_kv,N,n_past", [
    (512, 250, 200),   # seen: 450 cells; hidden from 464 on, inside a tile of 64 that has visible keys
    (336, 250, 6),     # 256 cells seen, the last 80 not: a whole hidden tile and a ragged one behind it
    (333, 250, 50),    # mask rows at odd places, ragged end behind the diagonal
    (1001, 300, 20),   # many hidden cells, rows at odd places
    (300, 300, 0),     # the ragged tile is the diagonal's
])
def test_hidden_groups_of_16_stay_out(D, n_kv, N, n_past):
    rng = np.random.default_rng(D + n_kv)
    q, k, v = rng.standard_normal((8, N, D)).astype(np.float32), rng.standard_normal((4, n_kv, D)), rng.standard_normal((4, n_kv, D))
    hidden = np.arange(n_kv) >= (n_past + N + 15) // 16 * 16
    got, exact = poisoned_run(q, k, v, causal(N, n_kv, n_past), hidden, D ** -0.5)
    assert np.abs(got - exact).max() <= BOUND


@pytest.mark.parametrize("n_kv", [640, 637])
@pytest.mark.parametrize("first,last", [(128, 256), (80, 96), (64, 400), (0, 144)])
def test_hidden_cells_between_visible_ones(n_kv, first, last):
    """Cells [first, last) belong to something else: whole tiles, one group of 16 inside a tile, several tiles and a part of one, the first ones."""
    N, D = 200, 128
    rng = np.random.default_rng(first + n_kv)
    q, k, v = rng.standard_normal((8, N, D)).astype(np.float32), rng.standard_normal((8, n_kv, D)), rng.standard_normal((8, n_kv, D))
    mask = causal(N, n_kv, n_kv - N)
    mask[:, first:last] = -np.inf
    got, exact = poisoned_run(q, k, v, mask, (np.arange(n_kv) >= first) & (np.arange(n_kv) < last), D ** -0.5)
    assert np.abs(got - exact).max() <= BOUND


@pytest.mark.parametrize("n_kv", [256, 250])
@pytest.mark.parametrize("kw", [dict(scale=-0.1), dict(scale=0.1, softcap=4.0), dict(scale=0.1, max_bias=8.0), dict(scale=0.1, plain=True), dict(scale=-0.1, plain=True)])
def test_scores_of_every_form(n_kv, kw):
    """A negative scale, a soft cap, a slope of the mask, no mask at all; the mask holds values other than 0 and -inf."""
    N, D = 130, 128
    kw = dict(kw)
    scale, plain = kw.pop("scale"), kw.pop("plain", False)
    rng = np.random.default_rng(n_kv)
    q, k, v = rng.standard_normal((8, N, D)).astype(np.float32), rng.standard_normal((2, n_kv, D)), rng.standard_normal((2, n_kv, D))
    mask = causal(N, n_kv, n_kv - N)
    mask[:N] += rng.uniform(-2, 0, (N, n_kv)).astype(np.float16)
    mask = None if plain else mask
    exact = O.flash_attn_f64(q, O.pack_kv(F16, k), O.pack_kv(F16, v), mask, F16, scale, **kw)
    got = H.flash_attn_ext(q, O.pack_kv(F16, k), O.pack_kv(F16, v), mask, F16, scale, **kw)
    assert np.abs(got - exact).max() <= BOUND
