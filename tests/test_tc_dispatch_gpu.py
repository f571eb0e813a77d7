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


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("mode", list(BARS))
@pytest.mark.parametrize("n", [192, 640, 1664])
def test_back_to_back_products(handle, cuda, mode, n, captured):
    """Each product reads what the launch before it wrote, with no host
    synchronisation between them, live and replayed: the same bits as with one
    after every call (the kernels overlap their prologues, not their reads)."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    X0, W = ((torch.rand(n, n, generator=gen, device="cuda") * 2 - 1) / 16 for _ in range(2))
    steps = 6
    X = [X0.clone()] + [torch.empty_like(X0) for _ in range(steps)]
    want = [X0.clone()] + [torch.empty_like(X0) for _ in range(steps)]
    handle.set_math_mode(mode)

    def chain(bufs, sync):
        for i in range(steps):
            assert B.iclblasSgemm(handle, 0, 0, n, n, n, 1.0, W, n, bufs[i], n, 0.0, bufs[i + 1], n) == B.SUCCESS
            if sync:
                assert handle.synchronize() == B.SUCCESS

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    handle.set_stream(s)
    with torch.cuda.stream(s):
        chain(want, True)
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                chain(X, False)
            for _ in range(3):
                for t in X[1:]:
                    t.fill_(float("nan"))
                g.replay()
        else:
            chain(X, False)
    s.synchronize()
    assert handle.synchronize() == B.SUCCESS
    for got, ref in zip(X, want):
        assert torch.equal(got, ref)
