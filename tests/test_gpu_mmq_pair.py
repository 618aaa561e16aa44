"""The paired-SM prompt GEMM where it can go wrong: weight rows and columns around the tile edges, rows that start at any even byte, two halves
of K, results inside wider rows, batches of products and experts of uneven size.  Against float64 over the dequantised weights; the bound is
that of tests/test_gpu_mmq.py (both operands rounded to bf16: 2^-9 / sqrt(3) each, relative to the product)."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import koboldcpp_b200.host as H
import orc as O
from koboldcpp_b200.lib import BF16, Q2_K, Q3_K, Q4_0, Q4_K, Q5_0, Q5_1, Q5_K, Q6_K, Q8_0, IQ4_XS, check, lib, row_size
from koboldcpp_b200.llama import random_blocks

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def product(t, w, x, K, M, offset=0, row_bytes=None, dst_stride=None):
    """b200_mul_mat_q with the weight rows `row_bytes` apart, the first one `offset` bytes into its allocation."""
    N, rs = x.shape[0], row_size(t, K)
    row_bytes, dst_stride = row_bytes or rs, dst_stride or M
    raw = np.zeros(offset + M * row_bytes + 64, np.uint8)
    for m in range(M):
        raw[offset + m * row_bytes:offset + m * row_bytes + rs] = w[m]
    dw, dx, dd = H.DeviceBuffer.from_numpy(raw), H.DeviceBuffer.from_numpy(x), H.DeviceBuffer.from_numpy(np.full((N, dst_stride), np.nan, np.float32))
    need = lib().b200_mul_mat_q_workspace_bytes(t, K, M, N)
    ws = H.DeviceBuffer(need + 16)
    check(lib().b200_mul_mat_q(t, dw.ptr + offset, row_bytes, dx.ptr, K, dd.ptr, dst_stride, K, M, N, ws.ptr, need, None))
    return dd.to_numpy(np.float32, (N, dst_stride))


def expected(t, w, x, K):
    return x.astype(np.float64) @ np.stack([O.dequantize(t, r, K) for r in w]).astype(np.float64).T


@pytest.mark.parametrize("t", [Q4_K, Q5_K, Q6_K, Q4_0, Q8_0])
@pytest.mark.parametrize("K,M,N", [(256, 1, 9), (256, 255, 31), (512, 257, 33), (2304, 129, 177), (2048, 513, 16), (768, 700, 257)])
def test_edges_of_tiles(t, K, M, N):
    rng = np.random.default_rng(K + M + N + t)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    got = product(t, w, x, K, M, dst_stride=M + 5)
    assert np.isnan(got[:, M:]).all()
    assert rel(got[:, :M], expected(t, w, x, K)) < 4e-3


@pytest.mark.parametrize("t", [Q4_K, Q5_K, Q6_K, Q4_0, Q8_0, BF16])
@pytest.mark.parametrize("K,M,N", [(2048, 1, 9), (2560, 257, 70), (1280, 515, 31), (5120, 1000, 199), (11008, 300, 17), (4096, 4096, 40), (4096, 2048, 300)])
def test_parts_of_k(t, K, M, N):
    """Few tiles and many K steps: a tile's parts, of unequal size, are added in one order whatever the run; ragged rows, and a result whose rows start at odd places."""
    if M == 1 and t in (Q5_K, Q8_0):
        pytest.skip("nine values of one row: the bound is relative to their size, which is chance")
    rng = np.random.default_rng(K + M + N + t)
    x = rng.standard_normal((N, K)).astype(np.float32)
    if t == BF16:
        bits = (rng.standard_normal((M, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        w, want = bits.view(np.uint8), x.astype(np.float64) @ (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64).T
    else:
        w = random_blocks(rng, t, M, K)
        want = expected(t, w, x, K)
    got = product(t, w, x, K, M, dst_stride=M + 5)
    assert np.isnan(got[:, M:]).all()
    assert rel(got[:, :M], want) < 4e-3
    for _ in range(3):
        assert np.array_equal(product(t, w, x, K, M), got[:, :M])


@pytest.mark.parametrize("K,M,N,batch,pad", [(8192, 40, 12, 3, 0), (8192, 300, 33, 2, 3), (4096, 257, 100, 3, 4), (8192, 515, 9, 2, 1)])
def test_parts_of_k_of_a_batch(K, M, N, batch, pad):
    """Dense products of a batch that are split: each product's weights, activations and result lie behind the last one's, result rows at odd places among them."""
    rng = np.random.default_rng(K + M + N)
    bits = (rng.standard_normal((batch, M, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    W = (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    x, row = rng.standard_normal((batch, N, K)).astype(np.float32), M + pad
    dw, dx, dd = H.DeviceBuffer.from_numpy(bits), H.DeviceBuffer.from_numpy(x), H.DeviceBuffer.from_numpy(np.full((batch, N, row), np.nan, np.float32))
    need = batch * lib().b200_mul_mat_q_workspace_bytes(BF16, K, M, N)
    ws, got = H.DeviceBuffer(need + 16), []
    for _ in range(2):
        check(lib().b200_mul_mat_bf16_batched(dw.ptr, 2 * K, 2 * M * K, dx.ptr, K, N * K, dd.ptr, row, N * row, K, M, N, batch, ws.ptr, need, None))
        got.append(dd.to_numpy(np.float32, (batch, N, row)))
    assert np.isnan(got[0][:, :, M:]).all() and np.array_equal(got[0], got[1], equal_nan=True)
    for b in range(batch):
        assert rel(got[0][b, :, :M], x[b].astype(np.float64) @ W[b].T) < 4e-3, b


FIRST = """
import sys, threading
sys.path[:0] = [{root!r}, {tests!r}]
import numpy as np
from test_gpu_mmq_pair import BF16, Q4_K, Q6_K, expected, product, random_blocks, rel
rng = np.random.default_rng(0)
K, M, N = 5120, 600, 60
work = []
for t in (Q4_K, Q6_K):
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    work += [(t, w, x, expected(t, w, x, K))] * 4
start, wrong = threading.Barrier(len(work)), []
def run(t, w, x, want):
    start.wait()
    got = product(t, w, x, K, M)
    if not rel(got, want) < 4e-3:
        wrong.append(t)
threads = [threading.Thread(target=run, args=a) for a in work]
[t.start() for t in threads]
[t.join() for t in threads]
assert not wrong, wrong
"""


def test_first_products_of_several_threads():
    """What a device holds at once is found out by the first of them, in a process of its own."""
    tests = Path(__file__).resolve().parent
    r = subprocess.run([sys.executable, "-c", FIRST.format(root=str(tests.parent), tests=str(tests))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


@pytest.mark.parametrize("K", [64, 960, 1088, 4032, 4096, 4160, 8256])
def test_rows_of_activations_of_any_length(K):
    """The conversion of the activations takes 4096 values of a row at a time."""
    M, N = 70, 19
    rng = np.random.default_rng(K)
    x = rng.standard_normal((N, K)).astype(np.float32)
    bits = (rng.standard_normal((M, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    want = x.astype(np.float64) @ (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64).T
    assert rel(product(BF16, bits.view(np.uint8), x, K, M), want) < 4e-3


@pytest.mark.parametrize("t,K,M,N,whole", [(Q6_K, 2560, 20483, 40, 18944), (Q8_0, 2560, 20000, 100, 18944), (Q4_K, 2560, 19300, 200, 18944), (Q6_K, 4096, 11008, 280, 9472), (BF16, 4096, 19300, 40, 18944)])
def test_rows_behind_whole_waves(t, K, M, N, whole):
    """A little more than a wave of tiles (74 pairs): the rows behind row `whole` are a launch of their own, in parts of K.  Rows at its edge and a sample of the others, and
    nothing beyond the last row."""
    rng = np.random.default_rng(K + M + N + t)
    each, x = 500, rng.standard_normal((N, K)).astype(np.float32)
    if t == BF16:
        bits = (rng.standard_normal((each, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        w, W = bits.view(np.uint8), (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    else:
        w = random_blocks(rng, t, each, K).reshape(each, -1)
        W = np.stack([O.dequantize(t, r, K) for r in w]).astype(np.float64)
    at = rng.integers(0, each, M)  # which of the rows each is
    got = product(t, w[at], x, K, M, dst_stride=M + 3)
    assert np.isnan(got[:, M:]).all()
    want = (x.astype(np.float64) @ W.T)[:, at]
    for rows in (slice(0, M), slice(whole - 256, whole), slice(whole, whole + 256), slice(M - 30, M)):
        assert rel(got[:, rows], want[:, rows]) < 6e-3, rows
    assert np.array_equal(got, product(t, w[at], x, K, M, dst_stride=M + 3), equal_nan=True)


@pytest.mark.parametrize("T", [40, 150])
def test_experts_without_a_valid_pair(T):
    """No tile at all: nothing is stored, and the launch ends.  (Up to 32 pairs an expert on average, and more: a kernel each.)"""
    K, M, used, n_expert = 512, 300, 2, 4
    rng = np.random.default_rng(1)
    w, b = random_blocks(rng, Q4_K, n_expert * M, K), rng.standard_normal((T, 1, K)).astype(np.float32)
    need = lib().b200_mul_mat_id_q_workspace_bytes(Q4_K, K, M, used, T, n_expert)
    dw, db, di = H.DeviceBuffer.from_numpy(w.reshape(-1)), H.DeviceBuffer.from_numpy(b), H.DeviceBuffer.from_numpy(np.full((T, used), -1, np.int32))
    dd, ws, rs = H.DeviceBuffer.from_numpy(np.full((T, used, M), 7.0, np.float32)), H.DeviceBuffer(need + 512), row_size(Q4_K, K)
    check(lib().b200_mul_mat_id_q(Q4_K, dw.ptr, rs, rs * M, n_expert, di.ptr, used, db.ptr, K, K, dd.ptr, M, used * M, K, M, used, 1, T, (ws.ptr + 255) // 256 * 256, need, None))
    assert (dd.to_numpy(np.float32, (T, used, M)) == 7.0).all()


@pytest.mark.parametrize("t", [Q6_K, Q8_0, Q4_0, Q2_K, Q3_K, Q5_0, Q5_1, IQ4_XS])
@pytest.mark.parametrize("offset,pad", [(0, 0), (2, 0), (6, 2), (14, 10), (4, 6), (8, 12)])
def test_rows_at_any_even_byte(t, offset, pad):
    K, M, N = 1024, 40, 20
    rng = np.random.default_rng(t + offset)
    w, x = random_blocks(rng, t, M, K), rng.standard_normal((N, K)).astype(np.float32)
    assert rel(product(t, w, x, K, M, offset, row_size(t, K) + pad), expected(t, w, x, K)) < 4e-3


@pytest.mark.parametrize("K,M,N,batch", [(64, 130, 20, 3), (320, 256, 100, 5), (128, 300, 300, 2)])
def test_batches_of_dense_products(K, M, N, batch):
    rng = np.random.default_rng(K + M)
    w = rng.standard_normal((batch, M, K)).astype(np.float32)
    bits = (w.view(np.uint32) >> 16).astype(np.uint16)
    w = (bits.astype(np.uint32) << 16).view(np.float32)
    x = rng.standard_normal((batch, N, K)).astype(np.float32)
    for gap in (0, 8):  # values between two products: with 8 the stride is no multiple of a row
        stack = np.zeros((batch, M * K + gap), np.uint16)
        stack[:, :M * K] = bits.reshape(batch, -1)
        dw, dx, dd = H.DeviceBuffer.from_numpy(stack), H.DeviceBuffer.from_numpy(x), H.DeviceBuffer(4 * batch * N * M)
        need = batch * lib().b200_mul_mat_q_workspace_bytes(BF16, K, M, N)
        ws = H.DeviceBuffer(need + 16)
        check(lib().b200_mul_mat_bf16_batched(dw.ptr, 2 * K, 2 * (M * K + gap), dx.ptr, K, N * K, dd.ptr, M, N * M, K, M, N, batch, ws.ptr, need, None))
        assert rel(dd.to_numpy(np.float32, (batch, N, M)), np.einsum("bnk,bmk->bnm", x.astype(np.float64), w.astype(np.float64))) < 4e-3


@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("T,n_expert,hot", [(9, 4, 0.5), (300, 4, 0.9), (520, 8, 0.6)])
def test_experts_of_uneven_size(t, T, n_expert, hot):
    """One expert takes most pairs (several full tiles and a remainder), another none."""
    K, M, used = 512, 300, 2
    rng = np.random.default_rng(T + t)
    w, b = random_blocks(rng, t, n_expert * M, K), rng.standard_normal((T, 1, K)).astype(np.float32)
    ids = np.where(rng.random((T, used)) < hot, 1, rng.integers(0, n_expert - 1, (T, used))).astype(np.int32)
    got = H.mul_mat_id_q(t, w, ids, b, K, M, n_expert)
    W = [np.stack([O.dequantize(t, r, K) for r in w[e * M:(e + 1) * M]]).astype(np.float64) for e in range(n_expert)]
    exp = np.stack([[W[ids[i, s]] @ b[i, 0].astype(np.float64) for s in range(used)] for i in range(T)])
    assert rel(got, exp) < 4e-3


GIVE_UP = """
import sys, numpy as np
sys.path[:0] = [{root!r}, {tests!r}]
import koboldcpp_b200.host as H, orc as O
from koboldcpp_b200.lib import Q4_K, check, lib, row_size
from koboldcpp_b200.llama import random_blocks
K, M, N = {shape}
rng = np.random.default_rng(0)
w, x = random_blocks(rng, Q4_K, M, K), rng.standard_normal((N, K)).astype(np.float32)
want = x.astype(np.float64) @ np.stack([O.dequantize(Q4_K, r, K) for r in w]).astype(np.float64).T
dw, dx = H.DeviceBuffer.from_numpy(w.reshape(-1)), H.DeviceBuffer.from_numpy(x)
need = lib().b200_mul_mat_q_workspace_bytes(Q4_K, K, M, N)
ws = H.DeviceBuffer(need + 16)
def run(limit):
    dd = H.DeviceBuffer.from_numpy(np.full((N, M), np.nan, np.float32))
    check(lib().b200_mul_mat_q_wait(Q4_K, dw.ptr, row_size(Q4_K, K), dx.ptr, K, dd.ptr, M, K, M, N, ws.ptr, need, limit, None))
    return dd.to_numpy(np.float32, (N, M))
whole = run(4_000_000_000)
assert np.isfinite(whole).all() and np.linalg.norm(whole - want) < 4e-3 * np.linalg.norm(want)
assert lib().b200_gemm_status() == 0
for limit in {limits}:
    got = run(limit)
    stored = ~np.isnan(got)
    print(limit, stored.mean())
    assert np.array_equal(got[stored], whole[stored]), limit
assert not stored.all()
{more}
"""


def give_up(more="", limits=(0,), shape=(1792, 19500, 200)):
    """The statements above in a process of their own (that a product gave up is remembered for the life of a process), then `more`."""
    tests = Path(__file__).resolve().parent
    r = subprocess.run([sys.executable, "-c", GIVE_UP.format(root=str(tests.parent), tests=str(tests), more=more, limits=limits, shape=shape)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_what_is_stored_is_right_when_waits_run_out():
    """With a limit of some cycles the pipeline gives up at its start, in its middle or not at all, in either CTA of a pair: every value is the right one, to
    the bit, or was never written."""
    give_up(limits=(100_000, 20_000, 6_000, 2_000, 700, 200, 0))


def test_parts_of_k_are_stored_together_or_not_at_all():
    """The same where the pairs of a cluster take parts of K: two tiles of 256 rows, long rows (the wait for an accumulator is one of 20 us)."""
    give_up(limits=(100_000, 50_000, 20_000, 9_000, 6_000, 2_000, 200, 0), shape=(32768, 300, 100))


def test_status_is_set_for_a_caller_without_a_backend():
    give_up("assert lib().b200_gemm_status() == 1")


STEP = """
import koboldcpp_b200.llama as L
from koboldcpp_b200.lib import F16
def failing(call):
    try:
        call()
    except Exception as e:
        assert "gave up waiting" in str(e), e
        return
    raise AssertionError("a step behind a product that gave up was reported as done")
m = L.LlamaModel(L.SHAPES["test-dense"], 512, F16)
m.init_random(1)
m.finalize(64)
failing(lambda: m.decode(list(range(40)), 0))
m.decode_async(list(range(40)), 0)
failing(m.synchronize)
"""


def test_decoder_reports_a_step_behind_a_product_that_gave_up():
    give_up(STEP)


@pytest.mark.parametrize("t", [Q4_K, Q6_K, Q8_0, Q4_0, Q5_1, IQ4_XS, BF16])
@pytest.mark.parametrize("K,N", [(256, 300), (768, 177)])
def test_several_tiles_a_pair(t, K, N):
    """More than twice as many tiles as pairs of SMs: the second accumulator and its parity, stages and weight copies that run on into the next tile."""
    M = 20000
    rng = np.random.default_rng(K + t)
    x = rng.standard_normal((N, K)).astype(np.float32)
    if t == BF16:
        bits = (rng.standard_normal((M, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        w, W = bits.view(np.uint8), (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    else:
        w = random_blocks(rng, t, M, K).reshape(M, -1)
        W = np.stack([O.dequantize(t, r, K) for r in w]).astype(np.float64)
    got, want = product(t, w, x, K, M), x.astype(np.float64) @ W.T
    assert rel(got, want) < 4e-3
    # every tile by itself: 256 rows of the result each
    for m in range(0, M, 256):
        assert rel(got[:, m:m + 256], want[:, m:m + 256]) < 6e-3, m


def test_several_tiles_a_pair_of_a_batch():
    K, M, N, batch = 128, 3000, 300, 8
    rng = np.random.default_rng(8)
    bits = (rng.standard_normal((batch, M, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    W = (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    x = rng.standard_normal((batch, N, K)).astype(np.float32)
    dw, dx, dd = H.DeviceBuffer.from_numpy(bits), H.DeviceBuffer.from_numpy(x), H.DeviceBuffer(4 * batch * N * M)
    need = batch * lib().b200_mul_mat_q_workspace_bytes(BF16, K, M, N)
    ws = H.DeviceBuffer(need + 16)
    check(lib().b200_mul_mat_bf16_batched(dw.ptr, 2 * K, 2 * M * K, dx.ptr, K, N * K, dd.ptr, M, N * M, K, M, N, batch, ws.ptr, need, None))
    got = dd.to_numpy(np.float32, (batch, N, M))
    for b in range(batch):
        assert rel(got[b], x[b].astype(np.float64) @ W[b].T) < 4e-3, b


@pytest.mark.parametrize("t", [Q4_K, Q6_K, Q8_0])
def test_several_tiles_a_pair_of_experts(t):
    """Tiles of different widths follow one another on a pair: experts with 1 to 256 pairs and one with none."""
    K, M, used, n_expert, T = 256, 5000, 2, 8, 300
    rng = np.random.default_rng(t)
    w, b = random_blocks(rng, t, n_expert * M, K).reshape(n_expert * M, -1), rng.standard_normal((T, 1, K)).astype(np.float32)
    odds = np.array([0.45, 0.2, 0.15, 0.1, 0.06, 0.035, 0.005, 0.0])
    ids = rng.choice(n_expert, (T, used), p=odds / odds.sum()).astype(np.int32)
    ids[0] = 6
    got = H.mul_mat_id_q(t, w, ids, b, K, M, n_expert)
    for e in range(n_expert):
        tok, slot = np.nonzero(ids == e)
        if len(tok):
            W = np.stack([O.dequantize(t, r, K) for r in w[e * M:(e + 1) * M]]).astype(np.float64)
            assert rel(got[tok, slot], b[tok, 0].astype(np.float64) @ W.T) < 4e-3, e


@pytest.mark.parametrize("gap", [0, 8])
def test_dense_experts_at_odd_strides(gap):
    """Values between two experts: with 8 their stride is no multiple of a row, which one tensor map cannot cover."""
    K, M, used, n_expert, T = 192, 300, 2, 5, 120
    rng = np.random.default_rng(gap)
    bits = (rng.standard_normal((n_expert, M, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    W = (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    stack = np.zeros((n_expert, M * K + gap), np.uint16)
    stack[:, :M * K] = bits.reshape(n_expert, -1)
    b, ids = rng.standard_normal((T, 1, K)).astype(np.float32), rng.integers(0, n_expert, (T, used)).astype(np.int32)
    need = lib().b200_mul_mat_id_q_workspace_bytes(BF16, K, M, used, T, n_expert)
    dw, db, di, dd, ws = H.DeviceBuffer.from_numpy(stack), H.DeviceBuffer.from_numpy(b), H.DeviceBuffer.from_numpy(ids), H.DeviceBuffer(4 * T * used * M), H.DeviceBuffer(need + 512)
    check(lib().b200_mul_mat_id_q(BF16, dw.ptr, 2 * K, 2 * (M * K + gap), n_expert, di.ptr, used, db.ptr, K, K, dd.ptr, M, used * M, K, M, used, 1, T, (ws.ptr + 255) // 256 * 256, need, None))
    want = np.einsum("tsmk,tk->tsm", W[ids], b[:, 0].astype(np.float64))
    assert rel(dd.to_numpy(np.float32, (T, used, M)), want) < 4e-3
