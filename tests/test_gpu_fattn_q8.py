"""Attention over a q8_0 cache on the tensor cores: the narrow form (up to 8 query columns) and the wide one, last tiles of 1 to 16 keys, odd key
counts (mask rows at any even byte), all-masked keys and ALiBi.  Against 64 bits: Q, d * q and P are each rounded to f16 (2^-11 of values whose
weighted mean is O(0.3), with scores of O(1): 3 roundings of at most 2^-11 x 4 sigma), bound 5e-3 as for the other caches."""
import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import Q8_0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("heads,kv,N,n_kv", [(2, 1, 1, 1), (8, 1, 1, 17), (9, 1, 1, 31), (4, 2, 4, 33), (4, 2, 5, 160), (32, 8, 1, 1023), (16, 1, 2, 255), (4, 4, 2, 640)])
def test_columns_and_remainders(D, heads, kv, N, n_kv):
    rng = np.random.default_rng(D + heads + N + n_kv)
    q = rng.standard_normal((heads, N, D)).astype(np.float32)
    k, v = (O.pack_kv(Q8_0, rng.standard_normal((kv, n_kv, D)).astype(np.float32)) for _ in range(2))
    mask = np.zeros((max(32, N), n_kv), np.float16)
    mask[:, rng.random(n_kv) < 0.2] = -np.inf
    mask[:, 0] = 0
    for bias in (0.0, 8.0):
        got = H.flash_attn_ext(q, k, v, mask, Q8_0, D ** -0.5, bias)
        want = O.flash_attn_f64(q, k, v, mask, Q8_0, D ** -0.5, bias)
        assert np.abs(got - want).max() < 5e-3
