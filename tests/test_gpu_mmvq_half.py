"""Rows of at most 2048 values, which the decode GEMV takes two at a time, one in each half of a warp: every format, rows that end inside a slice, odd numbers of rows,
a pair whose rows are of two formats, gate and up rows, experts that do not exist.  Against the oracle's q8_1 arithmetic with the bound of the other GEMV tests: sums
of K / 32 exact products in f32."""
import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import IQ4_NL, IQ4_XS, Q2_K, Q3_K, Q4_0, Q4_1, Q4_K, Q5_0, Q5_1, Q5_K, Q6_K, Q8_0
from koboldcpp_b200.llama import random_blocks

pytestmark = pytest.mark.gpu
BLOCKS_OF_32 = (Q4_0, Q4_1, Q5_0, Q5_1, Q8_0, IQ4_NL)


def close(got, want):
    return float(np.abs(got - want).max() / np.abs(want).max()) < 3e-5


@pytest.mark.parametrize("t", [Q4_0, Q4_1, Q5_0, Q5_1, Q8_0, IQ4_NL, IQ4_XS, Q2_K, Q3_K, Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,M", [(32, 5), (256, 1), (288, 40), (1024, 149), (1792, 2371), (2016, 33), (2048, 300), (2048, 4740), (2080, 40), (2304, 33)])
def test_one_column(t, K, M):
    if K % 256 and t not in BLOCKS_OF_32:
        pytest.skip("rows are whole blocks of 256")
    rng = np.random.default_rng(K + M + t)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((1, K)).astype(np.float32)
    assert close(H.mul_mat_vec_q(t, w, x, K, M), O.mul_mat_q8_1(t, w, x, K, M))


@pytest.mark.parametrize("ta,tb", [(Q4_K, Q6_K), (Q5_K, Q6_K), (Q4_K, Q5_K)])
@pytest.mark.parametrize("Ms", [(2048, 256, 256), (301, 33, 77), (1, 2, 1)])
def test_rows_of_two_formats(ta, tb, Ms):
    K = 2048
    rng = np.random.default_rng(sum(Ms) + ta)
    types = (ta, ta, tb)
    ws, x = [random_blocks(rng, t, M, K) for t, M in zip(types, Ms)], rng.standard_normal((1, K)).astype(np.float32)
    for got, t, w, M in zip(H.mul_mat_vec_q_multi(ta, ws, x, K, types=types), types, ws, Ms):
        assert close(got, O.mul_mat_q8_1(t, w, x, K, M))


@pytest.mark.parametrize("t", [Q4_0, Q4_K, Q6_K])
def test_experts_that_do_not_exist(t):
    K, M, n_expert = 1024, 301, 4
    rng = np.random.default_rng(t)
    w, b = random_blocks(rng, t, n_expert * M, K), rng.standard_normal((1, 1, K)).astype(np.float32)
    ids = np.array([[2, 7, 0, -1]], np.int32)
    got = H.mul_mat_id_vec_q(t, w, ids, b, K, M, n_expert)
    assert np.isnan(got[0, 1]).all() and np.isnan(got[0, 3]).all()
    for s in (0, 2):
        e = ids[0, s]
        assert close(got[0, s], O.mul_mat_q8_1(t, w[e * M:(e + 1) * M], b[0], K, M)[0])
