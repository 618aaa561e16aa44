"""Kernels whose CTAs may be placed while the kernel in front of them drains see what it wrote: weights and activations that change from launch to launch."""
import ctypes as C

import pytest

from koboldcpp_b200.lib import F16, F32, Q4_0, Q4_K, Q6_K, FattnArgs, RopeParams, Tensor, check, lib

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BLOCK = {Q4_0: (32, 18, (0,)), Q4_K: (256, 144, (0, 2)), Q6_K: (256, 210, (208,))}


def weights(g, kind, rows, k):
    values, size, scales = BLOCK[kind]
    raw = torch.randint(0, 256, (rows, k // values, size), generator=g, device="cuda", dtype=torch.uint8)
    for at in scales:
        raw[:, :, at:at + 2] = (torch.rand(rows, k // values, generator=g, device="cuda") * 1e-3 + 1e-4).half().view(torch.uint8).reshape(rows, k // values, 2)
    return torch.cat([raw.reshape(-1), torch.zeros(256, dtype=torch.uint8, device="cuda")])


@pytest.mark.parametrize("kind,k,rows,n", [(Q4_0, 512, 96, 1), (Q4_K, 4096, 1024, 1), (Q6_K, 8192, 600, 1), (Q4_K, 2048, 2048, 4), (Q6_K, 1024, 700, 3), (Q4_K, 1024, 512, 64), (Q6_K, 2048, 512, 200)])
def test_a_product_reads_what_the_launch_in_front_wrote(kind, k, rows, n):
    g = torch.Generator(device="cuda").manual_seed(k + rows + n)
    values, size, _ = BLOCK[kind]
    rb = k // values * size
    ws = [weights(g, kind, rows, k) for _ in range(6)]
    xs = [torch.randn(n, k, generator=g, device="cuda") for _ in range(6)]
    norm = torch.ones(k, device="cuda")
    w, x, h = torch.zeros_like(ws[0]), torch.zeros_like(xs[0]), torch.zeros_like(xs[0])
    dst = torch.zeros(6, n, rows, device="cuda")
    scratch = torch.zeros(int(lib().b200_mul_mat_q_workspace_bytes(kind, k, rows, n)) + 256, dtype=torch.uint8, device="cuda")

    def step(i, wait):
        x.copy_(xs[i])
        check(lib().b200_op_rms_norm_mul(C.byref(Tensor.contiguous(x.data_ptr(), F32, (k, n))), norm.data_ptr(), None, C.byref(Tensor.contiguous(h.data_ptr(), F32, (k, n))), 1e-5, None))
        wait()
        w.copy_(ws[i])
        wait()
        if n <= 8:
            check(lib().b200_mul_mat_vec_q(kind, w.data_ptr(), rb, h.data_ptr(), k, dst[i].data_ptr(), rows, k, rows, n, None))
        else:
            check(lib().b200_mul_mat_q(kind, w.data_ptr(), rb, h.data_ptr(), k, dst[i].data_ptr(), rows, k, rows, n, scratch.data_ptr(), scratch.numel(), None))
        wait()

    for i in range(6):
        step(i, torch.cuda.synchronize)
    want = dst.clone()
    assert (want.abs().sum((1, 2)) > 0).all()
    for _ in range(5):
        dst.zero_()
        for i in range(6):
            step(i, lambda: None)
        torch.cuda.synchronize()
        assert torch.equal(dst, want)


@pytest.mark.parametrize("D,n", [(64, 64), (96, 64), (128, 4), (64, 1)])
def test_a_row_of_launches_that_read_one_another(D, n):
    """Gate -> router logits -> expert ids as positions -> rotation and cache store -> the stored rows as the mask of an attention: prompts on both kernels,
    a few tokens, one token.  Each launch's input changes from step to step and is written by the launch in front."""
    heads, experts = 8, 256
    n_kv = D * heads
    g = torch.Generator(device="cuda").manual_seed(D + n)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    gates, qs, masks = [rand(n, experts) * 4 for _ in range(6)], [rand(n, heads, D) for _ in range(6)], []
    for i in range(6):
        m = torch.where(torch.rand(n, n_kv, generator=g, device="cuda") < 0.5, 0.0, -torch.inf)
        m[:, 100 * i // 2:][:, :5] = 0
        masks.append(m)
    up, gate, logits, q, qo, k, ko = torch.ones(n, experts, device="cuda"), rand(n, experts), rand(n, experts), rand(n, heads, D), rand(n, heads, D), rand(n, heads, D), rand(n, heads, D)
    probs, ids, w3 = torch.zeros(n, experts, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda"), [torch.zeros(n, device="cuda") for _ in range(3)]
    rows, krows, v = torch.zeros(32 * ((n + 31) // 32), n_kv, dtype=torch.float16, device="cuda"), torch.zeros(n, n_kv, dtype=torch.float16, device="cuda"), torch.zeros(n, n_kv, device="cuda")
    kc, vc = rand(heads, n_kv, D).half(), rand(heads, n_kv, D).half()
    dst = torch.zeros(6, n, heads, D, device="cuda")
    rp = RopeParams(D, 0, 4096, 10000.0, 1.0, 0.0, 1.0, 32.0, 1.0)
    t = lambda x, *s: C.byref(Tensor.contiguous(x.data_ptr(), F32, s))

    def step(i, wait):
        gate.copy_(gates[i])
        q.copy_(qs[i])
        v.copy_(masks[i])
        for call in (lambda: lib().b200_op_silu_mul(gate.data_ptr(), up.data_ptr(), None, logits.data_ptr(), n * experts, None),
                     lambda: lib().b200_op_moe_router(logits.data_ptr(), experts, probs.data_ptr(), experts, ids.data_ptr(), 1, w3[0].data_ptr(), w3[1].data_ptr(), w3[2].data_ptr(), experts, 1, n, None),
                     lambda: lib().b200_op_rope_kv_store(t(q, D, heads, n), t(qo, D, heads, n), t(k, D, heads, n), t(ko, D, heads, n), t(v, n_kv, n), ids.data_ptr(), None, C.byref(rp), F16,
                                                         krows.data_ptr(), rows.data_ptr(), None, None, None),
                     lambda: lib().b200_flash_attn_ext(C.byref(args[i]), ws.data_ptr(), ws.numel(), None)):
            wait()
            check(call())

    args = [FattnArgs(qo.data_ptr(), kc.data_ptr(), vc.data_ptr(), rows.data_ptr(), dst[i].data_ptr(), D, n, heads, heads, n_kv, F16, F16, 4 * D * heads, 4 * D, 2 * D, 2 * D * n_kv, 2 * D,
                      2 * D * n_kv, 2 * n_kv, D ** -0.5, 0.0, 0.0) for i in range(6)]
    ws = torch.zeros(max(int(lib().b200_flash_attn_workspace_bytes(C.byref(args[0]))), 256), dtype=torch.uint8, device="cuda")
    for i in range(6):
        step(i, torch.cuda.synchronize)
    torch.cuda.synchronize()
    want = dst.clone()
    assert torch.isfinite(want).all() and all((want[i] != want[i - 1]).any() for i in range(6))
    for _ in range(5):
        dst.zero_()
        for i in range(6):
            step(i, lambda: None)
        torch.cuda.synchronize()
        assert torch.equal(dst, want)
