"""The GEMV of several columns on the integer tensor cores: row tiles of 16 and their remainders, K parts for 1 to 16 warps and for two CTAs, odd and even column counts,
rows at any even byte, jobs of different sizes, norm prologue, residual and raw results.  Against the oracle's q8_1 arithmetic: sums of K / 32 exact
products in f32, 2^-24 sqrt(K / 32) of their size, bound 3e-5 as for the other GEMV kernels."""
import ctypes as C

import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import Q4_0, Q4_1, Q4_K, Q5_K, Q6_K, Q8_0, GemvFuse, GemvJob, check, lib, row_size
from koboldcpp_b200.llama import random_blocks

pytestmark = pytest.mark.gpu


def close(got, want):
    return float(np.abs(got - want).max() / np.abs(want).max()) < 3e-5


@pytest.mark.parametrize("t", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,M,N", [(256, 511, 8), (256, 512, 8), (256, 513, 7), (512, 527, 5), (1024, 700, 8), (2816, 545, 7), (4096, 2500, 4), (5120, 530, 6), (11008, 512, 5), (13824, 560, 4)])
def test_columns(t, K, M, N):
    rng = np.random.default_rng(K + M + N + t)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    assert close(H.mul_mat_vec_q(t, w, x, K, M), O.mul_mat_q8_1(t, w, x, K, M))


@pytest.mark.parametrize("t", [Q4_0, Q8_0, Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,M", [(256, 1), (256, 17), (512, 640), (1280, 33), (2304, 527), (4096, 300), (8192, 64), (13824, 130)])
@pytest.mark.parametrize("N", [2, 3, 4, 5, 6, 7, 8])
def test_packed_columns(t, K, M, N):
    """Two, four or eight columns to a tile; columns of very different size, one of zeros, and one with a single value that is not."""
    rng = np.random.default_rng(K + M + N + t)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    x *= np.float32(10.0) ** rng.integers(-3, 4, (N, 1))
    x[N // 2] = 0
    if N > 3:
        x[1] = 0
        x[1, K - 1] = 3
    got, want = H.mul_mat_vec_q(t, w, x, K, M), O.mul_mat_q8_1(t, w, x, K, M)
    for n in range(N):
        if not want[n].any():
            assert (got[n] == 0).all()
        else:
            assert close(got[n], want[n]), n


@pytest.mark.parametrize("t,N", [(Q6_K, 6), (Q6_K, 2), (Q6_K, 3), (Q4_0, 2), (Q4_0, 4), (Q4_0, 7), (Q8_0, 2), (Q8_0, 3), (Q8_0, 8)])
@pytest.mark.parametrize("offset,pad", [(2, 0), (6, 2), (14, 10), (8, 4)])
def test_rows_at_any_even_byte(t, N, offset, pad):
    K, M = 1024, 515
    rng = np.random.default_rng(offset)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    rs = row_size(t, K)
    raw = np.zeros(offset + M * (rs + pad) + 64, np.uint8)
    for m in range(M):
        raw[offset + m * (rs + pad):offset + m * (rs + pad) + rs] = w[m]
    dw, dx, dd = H.DeviceBuffer.from_numpy(raw), H.DeviceBuffer.from_numpy(x), H.DeviceBuffer(4 * N * M)
    check(lib().b200_mul_mat_vec_q(t, dw.ptr + offset, rs + pad, dx.ptr, K, dd.ptr, M, K, M, N, None))
    assert close(dd.to_numpy(np.float32, (N, M)), O.mul_mat_q8_1(t, w, x, K, M))


@pytest.mark.parametrize("t", [Q4_0, Q8_0, Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,N", [(1280, 4), (1280, 3), (1280, 2), (11008, 3)])
def test_jobs_with_norm_and_residual(t, K, N):
    Ms, eps = [100, 16, 433], 1e-5
    rng = np.random.default_rng(N + t)
    ws = [random_blocks(rng, t, M, K) for M in Ms]
    x, nw = rng.standard_normal((N, K)).astype(np.float32), rng.standard_normal(K).astype(np.float32)
    total = sum(Ms)
    res = rng.standard_normal((N, total)).astype(np.float32)
    scale = (1.0 / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + eps)).astype(np.float32)
    xn = x * scale * nw
    dx, dn, dr = H.DeviceBuffer.from_numpy(x), H.DeviceBuffer.from_numpy(nw), H.DeviceBuffer.from_numpy(res)
    dws = [H.DeviceBuffer.from_numpy(w, pad=16) for w in ws]
    dd, draw, dnorm, dmul = (H.DeviceBuffer(4 * N * n) for n in (total, total, K, K))
    jobs, fuse, at = (GemvJob * len(Ms))(), GemvFuse(), 0
    fuse.norm_weight, fuse.norm_eps, fuse.norm_out, fuse.norm_mul_out = dn.ptr, eps, dnorm.ptr, dmul.ptr
    for i, (w, M) in enumerate(zip(dws, Ms)):
        jobs[i].W, jobs[i].X, jobs[i].dst, jobs[i].M, jobs[i].id_index = w.ptr, dx.ptr, dd.ptr + 4 * at, M, -1
        if i != 1:
            fuse.residual[i], fuse.raw_dst[i] = dr.ptr + 4 * at, draw.ptr + 4 * at
        at += M
    check(lib().b200_mul_mat_vec_q_fused(t, jobs, len(Ms), row_size(t, K), K, total, K, N, C.byref(fuse), None))
    got, raw = dd.to_numpy(np.float32, (N, total)), draw.to_numpy(np.float32, (N, total))
    np.testing.assert_allclose(dnorm.to_numpy(np.float32, (N, K)), x * scale, rtol=3e-6, atol=3e-6)
    np.testing.assert_allclose(dmul.to_numpy(np.float32, (N, K)), xn, rtol=3e-6, atol=3e-6)
    at = 0
    for i, (w, M) in enumerate(zip(ws, Ms)):
        want = O.mul_mat_q8_1(t, w, xn, K, M)
        sl = slice(at, at + M)
        # (a value on the edge between two quants may fall to the other side with the norm's last bit: one step of 2^-7 of a block)
        tol = 2e-3 * np.abs(want).max()
        assert np.abs(got[:, sl] - (want + (res[:, sl] if i != 1 else 0))).max() < tol
        if i != 1:
            assert np.abs(raw[:, sl] - want).max() < tol
        at += M


def test_five_columns_of_several_jobs_stay_refused():
    K, M = 256, 272
    w = H.DeviceBuffer(row_size(Q4_K, K) * M + 16, zero=True)
    x, d = H.DeviceBuffer(4 * 5 * K, zero=True), H.DeviceBuffer(4 * 5 * 2 * M)
    jobs = (GemvJob * 2)()
    for i in range(2):
        jobs[i].W, jobs[i].X, jobs[i].dst, jobs[i].M, jobs[i].id_index = w.ptr, x.ptr, d.ptr + 4 * M * i, M, -1
    assert lib().b200_mul_mat_vec_q_multi(Q4_K, jobs, 2, row_size(Q4_K, K), K, 2 * M, K, 5, None, 0, 0, None) == 1


@pytest.mark.parametrize("t", [Q4_K, Q5_K, Q6_K, Q4_0, Q8_0])
@pytest.mark.parametrize("K,N", [(13824, 7), (13824, 8), (20480, 5), (20480, 8)])
def test_columns_of_long_rows(t, K, N):
    """Where shared memory does not hold all columns' activations for the dp4a form: the tensor form holds more, else half of the columns at a time."""
    M = 530
    rng = np.random.default_rng(K + N + t)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    assert close(H.mul_mat_vec_q(t, w, x, K, M), O.mul_mat_q8_1(t, w, x, K, M))


def test_columns_of_long_rows_with_norm_and_residual():
    t, K, M, N, eps = Q4_0, 13824, 300, 8, 1e-5
    rng = np.random.default_rng(3)
    w, x, nw = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32), rng.standard_normal(K).astype(np.float32)
    res = rng.standard_normal((N, M)).astype(np.float32)
    scale = (1.0 / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + eps)).astype(np.float32)
    xn = x * scale * nw
    dw, dx, dn, dr = H.DeviceBuffer.from_numpy(w, pad=16), H.DeviceBuffer.from_numpy(x), H.DeviceBuffer.from_numpy(nw), H.DeviceBuffer.from_numpy(res)
    dd, draw, dnorm, dmul = (H.DeviceBuffer(4 * N * n) for n in (M, M, K, K))
    jobs, fuse = (GemvJob * 1)(), GemvFuse()
    fuse.norm_weight, fuse.norm_eps, fuse.norm_out, fuse.norm_mul_out = dn.ptr, eps, dnorm.ptr, dmul.ptr
    fuse.residual[0], fuse.raw_dst[0] = dr.ptr, draw.ptr
    jobs[0].W, jobs[0].X, jobs[0].dst, jobs[0].M, jobs[0].id_index = dw.ptr, dx.ptr, dd.ptr, M, -1
    check(lib().b200_mul_mat_vec_q_fused(t, jobs, 1, row_size(t, K), K, M, K, N, C.byref(fuse), None))
    want = O.mul_mat_q8_1(t, w, xn, K, M)
    tol = 2e-3 * np.abs(want).max()  # (as in test_jobs_with_norm_and_residual)
    assert np.abs(dd.to_numpy(np.float32, (N, M)) - (want + res)).max() < tol and np.abs(draw.to_numpy(np.float32, (N, M)) - want).max() < tol
    np.testing.assert_allclose(dnorm.to_numpy(np.float32, (N, K)), x * scale, rtol=3e-6, atol=3e-6)
    np.testing.assert_allclose(dmul.to_numpy(np.float32, (N, K)), xn, rtol=3e-6, atol=3e-6)


@pytest.mark.parametrize("t", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,M,N", [(256, 1, 7), (2048, 64, 8), (1024, 300, 7), (4096, 511, 8)])
def test_many_columns_of_few_rows(t, K, M, N):
    rng = np.random.default_rng(K + M + t)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    assert close(H.mul_mat_vec_q(t, w, x, K, M), O.mul_mat_q8_1(t, w, x, K, M))


@pytest.mark.parametrize("t", [Q4_0, Q8_0, Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,N", [(256, 8), (1280, 3), (2048, 2), (5120, 4), (4352, 8), (8192, 4), (11008, 3), (8448, 8)])
def test_norm_is_that_of_the_other_kernel(t, K, N):
    """A column's norm to the bit (q4_1 has no tensor form): a last bit of it moves values to another quant."""
    M, eps = 80, 1e-5
    rng = np.random.default_rng(K + N)
    x = (rng.standard_normal((N, K)) * np.exp(rng.standard_normal((N, 1)))).astype(np.float32)
    nw = (1 + 0.3 * rng.standard_normal(K)).astype(np.float32)
    dx, dn = H.DeviceBuffer.from_numpy(x), H.DeviceBuffer.from_numpy(nw)

    def norm(kind):
        dw, dd, dnorm, dmul = H.DeviceBuffer.from_numpy(random_blocks(rng, kind, M, K), pad=16), *(H.DeviceBuffer(4 * N * n) for n in (M, K, K))
        jobs, fuse = (GemvJob * 1)(), GemvFuse()
        fuse.norm_weight, fuse.norm_eps, fuse.norm_out, fuse.norm_mul_out = dn.ptr, eps, dnorm.ptr, dmul.ptr
        jobs[0].W, jobs[0].X, jobs[0].dst, jobs[0].M, jobs[0].id_index = dw.ptr, dx.ptr, dd.ptr, M, -1
        check(lib().b200_mul_mat_vec_q_fused(kind, jobs, 1, row_size(kind, K), K, M, K, N, C.byref(fuse), None))
        return dnorm.to_numpy(np.float32, (N, K)), dmul.to_numpy(np.float32, (N, K))

    for got, want in zip(norm(t), norm(Q4_1)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("t", [Q4_K, Q5_K])
@pytest.mark.parametrize("K,N", [(7936, 2), (7936, 3), (6144, 4), (5120, 5), (3072, 8), (13824, 4)])
def test_activations_of_one_sign(t, K, N):
    """The minima take away most of what the quants add up to, block by block: a row's error is that of its blocks' sums.  A block of 256 rounds 8 partial sums of its
    quants, of 1/8 .. 8/8 of what they add up to (A), as many of its minima and the difference: about 2^-24 A (0.43 sqrt(2 * 3.2 + 1) = 1.2 for roundings at all places of a
    binade); bound 2.  (Two sums of whole rows, subtracted at the end, are 2.5 to 4 off.)"""
    M = 512
    rng = np.random.default_rng(K + N + t)
    w = random_blocks(rng, t, M, K)
    q = rng.integers(1, 33, (N, K // 32, 32))
    q[:, :, 5] = 127  # scale 2^-7 and sums below 2048: exact in f16, so that quantised activations are the activations
    x = (q.reshape(N, K) / 128).astype(np.float32)
    rows = np.stack([O.dequantize(t, r, K) for r in w]).astype(np.float64)
    blocks = w.reshape(M, K // 256, -1)
    low = blocks[:, :, 2:4].copy().view(np.float16).astype(np.float64)[:, :, 0]
    s = blocks[:, :, 4:16].astype(np.int64)
    mins = np.concatenate([s[:, :, 4:8] & 63, (s[:, :, 8:] >> 4) | (s[:, :, 4:8] >> 6 << 4)], axis=2) * low[:, :, None]  # [row][block][8]
    quants = rows.reshape(M, K // 256, 8, 32) + mins[..., None]
    A = np.einsum("mbsi,nbsi->nmb", quants, x.reshape(N, K // 256, 8, 32).astype(np.float64))
    err = H.mul_mat_vec_q(t, w, x, K, M) - x.astype(np.float64) @ rows.T
    c = np.sqrt((err ** 2).mean() / (A ** 2).sum(2).mean()) * 2 ** 24
    print("error", c)
    assert c < 2


@pytest.mark.parametrize("t", [Q4_0, Q8_0, Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,N", [(512, 2), (2048, 3), (4096, 2), (4096, 3), (13824, 2), (13824, 3)])
def test_bits_of_two_and_three_columns_do_not_follow_from_the_rows(t, K, N):
    """One and two CTAs a row tile: rows of a large launch, of a small one, of a single one, and in a launch of several matrices."""
    M = 5000
    rng = np.random.default_rng(K + N + t)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    whole = H.mul_mat_vec_q(t, w, x, K, M)
    for part in (slice(0, 1000), slice(4321, 4322), slice(100, 2500)):
        assert np.array_equal(H.mul_mat_vec_q(t, w[part], x, K, part.stop - part.start), whole[:, part])
    parts = [slice(0, 300), slice(300, 301), slice(301, 1400)]
    for got, part in zip(H.mul_mat_vec_q_multi(t, [w[p] for p in parts], x, K), parts):
        assert np.array_equal(got, whole[:, part])


@pytest.mark.parametrize("t,K,N,M", [(Q4_K, 4096, 7, 2500), (Q6_K, 4096, 8, 20000), (Q4_0, 4096, 7, 76800), (Q8_0, 8192, 8, 40000), (Q5_K, 13824, 3, 5000), (Q4_K, 2048, 3, 50000),
                                     (Q6_K, 5120, 4, 1184), (Q8_0, 4096, 3, 1200), (Q5_K, 7168, 2, 1201)])
def test_many_row_tiles(t, K, N, M):
    """Several row tiles a cluster and several batches of them (64 and, where shared memory holds no more, fewer), one tile a cluster with all warps: 1000 rows again and again,
    which are to come out the same wherever they lie, and twice the same."""
    each = min(M, 1000)
    rng = np.random.default_rng(K + M + N + t)
    w, x = random_blocks(rng, t, each, K), rng.standard_normal((N, K)).astype(np.float32)
    dw, dx, dd = H.DeviceBuffer.from_numpy(np.tile(w, (-(-M // each), 1))[:M], pad=16), H.DeviceBuffer.from_numpy(x), H.DeviceBuffer(4 * N * M)
    got = []
    for _ in range(2):
        check(lib().b200_mul_mat_vec_q(t, dw.ptr, row_size(t, K), dx.ptr, K, dd.ptr, M, K, M, N, None))
        got.append(dd.to_numpy(np.float32, (N, M)))
    assert np.array_equal(*got)
    assert close(got[0][:, :each], O.mul_mat_q8_1(t, w, x, K, each))
    assert np.array_equal(got[0], np.tile(got[0][:, :each], (1, -(-M // each)))[:, :M])


@pytest.mark.parametrize("scale", ["any", "halves", "edges"])
@pytest.mark.parametrize("N", [2, 4, 8])
def test_quants_of_the_columns(N, scale):
    """What b200_quantize_q8_1 makes of the columns, seen through q8_0 rows with a single 1: scale times quant, exact in f32.  Values of every size, values halfway between two
    quants, and blocks whose largest value lies around the limits of the shortcut for its quotient."""
    K = 1024
    rng = np.random.default_rng(N)
    w = np.zeros((K, K // 32, 34), np.uint8)
    w[:, :, :2] = np.array([1], np.float16).view(np.uint8)
    w[np.arange(K), np.arange(K) // 32, 2 + np.arange(K) % 32] = 1
    dw, dd = H.DeviceBuffer.from_numpy(w.reshape(K, -1), pad=16), H.DeviceBuffer(4 * N * K)
    for _ in range(20):
        x = rng.standard_normal((N, K // 32, 32)).astype(np.float32)
        if scale == "any":
            x *= (np.float32(10) ** rng.uniform(-9, 5, (N, K // 32, 1))).astype(np.float32)
        elif scale == "halves":
            x = (rng.integers(-127, 127, x.shape) + np.float32(0.5)).astype(np.float32)
            x[:, :, 7] = 127
            x *= np.float32(2) ** rng.integers(-12, 8, (N, K // 32, 1)).astype(np.float32)
        else:
            x *= (np.float32(1e-25) * np.float32(2) ** rng.integers(-60, 4, (N, K // 32, 1)).astype(np.float32)).astype(np.float32)
            x[:, ::5] = 0
        x = x.reshape(N, K)
        packed = H.quantize_q8_1(x).reshape(N, K // 32, 36)
        want = packed[:, :, :2].copy().view(np.float16).astype(np.float32) * packed[:, :, 4:].view(np.int8).astype(np.float32)
        dx = H.DeviceBuffer.from_numpy(x)
        check(lib().b200_mul_mat_vec_q(Q8_0, dw.ptr, row_size(Q8_0, K), dx.ptr, K, dd.ptr, K, K, K, N, None))
        assert np.array_equal(dd.to_numpy(np.float32, (N, K)), want.reshape(N, K))
