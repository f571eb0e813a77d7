"""Tensor-core GEMM on each tile of its dispatch (CTA pairs, 128 x 256, 128 x
128; for HGEMM by K and the columns), at ragged edges and K blocks, against an
FP64 product of the same inputs.

Bars: the split modes' (relative Frobenius 2e-3 TF32, 3e-5 3xBF16, 2e-6
6xBF16); HGEMM 5e-4 (one half-precision rounding is at most 4.9e-4)."""
import pytest

from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu
BARS = {B.MATH_TF32: 2e-3, B.MATH_BF16X3: 3e-5, B.MATH_BF16X6: 2e-6}


def check(handle, fn, m, n, k, bar, dtype, torch):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = (torch.rand(k, m, generator=gen, device="cuda") * 2 - 1).to(dtype)
    Bm = (torch.rand(n, k, generator=gen, device="cuda") * 2 - 1).to(dtype)
    C0 = (torch.rand(n, m, generator=gen, device="cuda") * 2 - 1).to(dtype)
    handle.set_stream(torch.cuda.current_stream())
    for beta in (0.0, 0.5):
        C = C0.clone()
        assert fn(handle, 0, 0, m, n, k, 1.5, A, m, Bm, k, beta, C, m) == B.SUCCESS
        assert handle.synchronize() == B.SUCCESS
        want = 1.5 * (Bm.double() @ A.double()) + beta * C0.double()
        assert ((C.double() - want).norm() / want.norm()).item() <= bar


@pytest.mark.parametrize("mode", list(BARS))
@pytest.mark.parametrize("m,n,k", [(1900, 2050, 130), (2050, 1100, 65), (130, 129, 700), (5000, 128, 257),
                                   (1300, 1500, 64), (300, 2000, 193)])
def test_split_modes(handle, cuda, mode, m, n, k):
    import torch
    handle.set_math_mode(mode)
    check(handle, B.iclblasSgemm, m, n, k, BARS[mode], torch.float32, torch)


@pytest.mark.parametrize("m,n,k", [(20000, 128, 72), (20000, 64, 320), (9000, 300, 136), (1600, 2000, 512),
                                   (4096, 3000, 1024), (40, 16, 8)])
def test_hgemm(handle, cuda, m, n, k):
    import torch
    check(handle, B.iclblasHgemm, m, n, k, 5e-4, torch.float16, torch)
