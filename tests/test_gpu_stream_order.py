"""Kernels whose CTAs may be placed while the kernel in front of them drains see what it wrote: weights and activations that change from launch to launch."""
import ctypes as C

import pytest

from koboldcpp_b200.lib import F32, Q4_0, Q4_K, Q6_K, Tensor, check, lib

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
