"""Complex device operands at 4 modulo 8: a complex number is two floats, so
every multiple of 4 is a legal address.  Every kernel that moves whole complex
elements otherwise, against the oracle: relative Frobenius error <= 1e-5, the
bar of the other complex tests (TF32 2e-3, 3xBF16 3e-5, as in the GEMM tests)."""
import numpy as np
import pytest

import oracle_lib as O
from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu
TOL = {0: 1e-5, 1: 2e-3, 2: 3e-5, 3: 1e-5}


def shifted(a, cuda, floats=1):
    """The complex array `a` on the device, `floats` floats past an aligned address."""
    import torch
    t = torch.zeros(2 * a.size + floats, device=cuda)
    t[floats:] = torch.from_numpy(a.view(np.float32)).to(cuda)
    return t[floats:]


def back(t):
    return t.cpu().numpy().view(np.complex64)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("m,n,k", [(5, 3, 7), (100, 90, 65), (700, 900, 33)])
def test_cgemm(handle, cuda, mode, m, n, k):
    import torch
    handle.set_stream(torch.cuda.current_stream())
    handle.set_math_mode(mode)
    rng = np.random.default_rng(m)
    for ta, tb in ((0, 0), (2, 1), (1, 2)):
        ra, ca = (m, k) if ta == 0 else (k, m)
        rb, cb = (k, n) if tb == 0 else (n, k)
        A, Bm, C = (O.colmajor(r, c, r, rng, np.complex64) for r, c in ((ra, ca), (rb, cb), (m, n)))
        want = C.copy()
        O.cgemm(ta, tb, m, n, k, 1.25 - 0.5j, A, ra, Bm, rb, 0.5j, want, m)
        for sa, sb, sc in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1)):
            Cd = shifted(C, cuda, sc)
            assert B.iclblasCgemm(handle, ta, tb, m, n, k, 1.25 - 0.5j, shifted(A, cuda, sa), ra, shifted(Bm, cuda, sb),
                                  rb, 0.5j, Cd, m) == B.SUCCESS
            assert O.rel_fro(back(Cd), want) <= TOL[mode]
    handle.set_math_mode(0)


# op N with four column groups and with one, op T/C by blocks and by warps
@pytest.mark.parametrize("m,n", [(1, 1), (300, 70), (2500, 40), (305000, 9), (60, 6500)])
def test_cgemv(handle, cuda, m, n):
    import torch
    handle.set_stream(torch.cuda.current_stream())
    rng = np.random.default_rng(n)
    for trans in (0, 1, 2):
        for pad, sa, sx, sy in ((0, 1, 0, 0), (1, 1, 1, 1), (1, 0, 1, 0)):
            lda = m + pad
            xl, yl = (n, m) if trans == 0 else (m, n)
            A, x, y = (O.colmajor(r, c, r, rng, np.complex64) for r, c in ((lda, n), (xl, 1), (yl, 1)))
            want = y.copy()
            O.cgemv(trans, m, n, 1.25, A, lda, x, 1, 0.5, want, 1)
            yd = shifted(y, cuda, sy)
            assert B.iclblasCgemv(handle, trans, m, n, 1.25, shifted(A, cuda, sa), lda, shifted(x, cuda, sx), 1, 0.5, yd,
                                  1) == B.SUCCESS
            assert O.rel_fro(back(yd), want) <= 1e-5


def lower(n, rng):
    A = (O.colmajor(n, n, n, rng, np.complex64) / np.float32(np.sqrt(n))).astype(np.complex64)
    A[::n + 1] = rng.uniform(1, 2, n)
    return A


@pytest.mark.parametrize("n", [1, 64, 200, 1100])
def test_ctrsv(handle, cuda, n):
    import torch
    handle.set_stream(torch.cuda.current_stream())
    rng = np.random.default_rng(n)
    A, b = lower(n, rng), O.colmajor(n, 1, n, rng, np.complex64)
    for trans in (0, 1, 2):
        want = b.copy()
        O.ctrsv(1, trans, 0, n, A, n, want, 1)
        for sa, sx in ((1, 0), (0, 1), (1, 1)):
            x = shifted(b, cuda, sx)
            assert B.iclblasCtrsv(handle, 1, trans, 0, n, shifted(A, cuda, sa), n, x, 1) == B.SUCCESS
            assert O.rel_fro(back(x), want) <= 1e-5


@pytest.mark.parametrize("mode", [0, 2])
def test_ctrsm(handle, cuda, mode):
    import torch
    handle.set_stream(torch.cuda.current_stream())
    handle.set_math_mode(mode)
    m, n = 300, 40
    rng = np.random.default_rng(7)
    A, Bm = lower(m, rng), O.colmajor(m, n, m, rng, np.complex64)
    want = Bm.copy()
    O.ctrsm(0, 1, 0, 0, m, n, 1.0, A, m, want, m)
    Bd = shifted(Bm, cuda)
    assert B.iclblasCtrsm(handle, 0, 1, 0, 0, m, n, 1.0, shifted(A, cuda), m, Bd, m) == B.SUCCESS
    assert O.rel_fro(back(Bd), want) <= TOL[mode]
    handle.set_math_mode(0)
