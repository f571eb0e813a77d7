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
                                 (77, 3001)])
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
