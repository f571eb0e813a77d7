"""GEMV on operands without 16-byte alignment (odd leading dimensions, shifted
bases, strides), at the edges of its 8-column and 8 x 32-row steps and of its
row tiles, against the oracle: relative Frobenius error <= 1e-5, the bar of
the other GEMV tests."""
import numpy as np
import pytest

import oracle_lib as O
from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (31, 8), (255, 7), (256, 9), (257, 65), (511, 1023), (513, 130), (3001, 177),
                                 (77, 3001), (64, 2049), (416, 6001), (417, 6001), (1025, 2050),
                                 (1025, 2051), (2049, 2400), (2049, 2401), (16385, 65)])
@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
def test_unaligned(handle, cuda, m, n, dtype):
    import torch
    cplx = dtype == np.complex64
    rng = np.random.default_rng(m * 7 + n)
    f, want = (B.iclblasCgemv, O.cgemv) if cplx else (B.iclblasSgemv, O.sgemv)
    handle.set_stream(torch.cuda.current_stream())
    for trans in (0, 1, 2):
        for pad, shift, inc, beta in ((1, 0, 1, 0.0), (2, 1, 1, 0.5), (0, 1, 2, 0.0)):
            lda = m + pad
            A = O.colmajor(m, n, lda, rng, dtype)
            xl, yl = (n, m) if trans == 0 else (m, n)
            x = O.colmajor(xl * inc, 1, xl * inc, rng, dtype)
            y = O.colmajor(yl * inc, 1, yl * inc, rng, dtype)
            y_ref = y.copy()
            want(trans, m, n, 1.25, A, lda, x, inc, beta, y_ref, inc)
            Ad = torch.empty(A.size + 1, dtype=torch.complex64 if cplx else torch.float32, device=cuda)
            Ad[shift:shift + A.size] = torch.from_numpy(A).to(cuda)
            xd, yd = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
            assert f(handle, trans, m, n, 1.25, Ad[shift:], lda, xd, inc, beta, yd, inc) == B.SUCCESS
            assert O.rel_fro(yd.cpu().numpy(), y_ref) <= 1e-5


# (the widest single slice, and unaligned columns below two slices)
@pytest.mark.parametrize("trans,m,n,lda", [(0, 700, 127, 700), (0, 2001, 127, 2001), (1, 2047, 6100, 2047)])
def test_first_call_captured(cuda, trans, m, n, lda):
    """Calls that need no scratch may be a handle's first, and captured."""
    import torch
    rng = np.random.default_rng(n)
    xl, yl = (n, m) if trans == 0 else (m, n)
    A, x, y = (O.colmajor(r, c, r, rng) for r, c in ((lda, n), (xl, 1), (yl, 1)))
    want = y.copy()
    O.sgemv(trans, m, n, 1.25, A, lda, x, 1, 0.5, want, 1)
    Ad, xd, yd = (torch.from_numpy(v).to(cuda) for v in (A, x, y))
    h = B.Handle()
    s = torch.cuda.Stream()
    h.set_stream(s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        status = B.iclblasSgemv(h, trans, m, n, 1.25, Ad, lda, xd, 1, 0.5, yd, 1)
    assert status == B.SUCCESS
    g.replay()
    torch.cuda.synchronize()
    assert O.rel_fro(yd.cpu().numpy(), want) <= 1e-5
    del g
    h.destroy()
