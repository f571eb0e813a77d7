"""TRSV's 64-row block kernel (complex data, and real data that TMA cannot
address) at the edges of its blocks and clusters, against the oracle.

Tolerance: relative Frobenius error <= 1e-5 against the FP64-accumulating
oracle, the bar of the other TRSV tests."""
import numpy as np
import pytest

import oracle_lib as O
from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu
TOL = 1e-5


def tri(n, lda, lower, rng, dtype):
    A = O.colmajor(n, n, lda, rng, dtype)
    M = A.reshape(n, lda).T[:n]
    off = (O.colmajor(n, n, n, rng, dtype).reshape(n, n) / np.sqrt(n)).astype(dtype)
    mask = np.tril(np.ones((n, n), bool), -1) if lower else np.triu(np.ones((n, n), bool), 1)
    M[mask] = off[mask]
    M[np.arange(n), np.arange(n)] = rng.uniform(1, 2, n)
    return A


def solve(handle, dtype, *args):
    return (B.iclblasCtrsv if dtype == np.complex64 else B.iclblasStrsv)(handle, *args)


def want(dtype, *args):
    (O.ctrsv if dtype == np.complex64 else O.strsv)(*args)


# one block, its edges, two blocks, a cluster's 8 blocks and the first of the next, several clusters
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 511, 512, 513, 577, 1333])
@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
def test_block_edges(handle, n, dtype):
    rng = np.random.default_rng(n)
    for uplo in (0, 1):
        for trans in (0, 1, 2):
            for diag, lda, inc in ((0, n, 1), (1, n + 1, 2)):
                lda += 1 if dtype == np.float32 and lda % 4 == 0 else 0  # a leading dimension TMA cannot take
                A = tri(n, lda, uplo == 1, rng, dtype)
                x = O.colmajor(n * inc, 1, n * inc, rng, dtype)
                x_ref = x.copy()
                want(dtype, uplo, trans, diag, n, A, lda, x_ref, inc)
                assert solve(handle, dtype, uplo, trans, diag, n, A, lda, x, inc) == B.SUCCESS
                assert O.rel_fro(x, x_ref) <= TOL
                if inc == 2:
                    assert np.array_equal(x[1::2], x_ref[1::2])


@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
@pytest.mark.parametrize("uplo", [0, 1])
def test_non_finite(handle, dtype, uplo):
    """A NaN or an infinity in b and a zero on the diagonal make exactly the
    entries non-finite that substitution makes so."""
    n = 201
    rng = np.random.default_rng(5 + uplo)
    for what in ("nan", "inf", "zero"):
        A = tri(n, n, uplo == 1, rng, dtype)
        x = O.colmajor(n, 1, n, rng, dtype)
        if what == "zero":
            A[100 * n + 100] = 0
        else:
            x[100] = np.nan if what == "nan" else np.inf
        x_ref = x.copy()
        with np.errstate(all="ignore"):
            want(dtype, uplo, 0, 0, n, A, n, x_ref, 1)
        assert solve(handle, dtype, uplo, 0, 0, n, A, n, x, 1) == B.SUCCESS
        fin = np.isfinite(x_ref)
        assert np.array_equal(np.isfinite(x), fin)
        assert fin.any() and not fin.all()
        assert O.rel_fro(x[fin], x_ref[fin]) <= TOL


def test_first_call_captured_and_replayed(handle, cuda):
    """The handle's first solve may be a captured one; replays give the eager result."""
    import torch
    n = 1000
    rng = np.random.default_rng(3)
    A = tri(n, n, True, rng, np.complex64)
    b = O.colmajor(n, 1, n, rng, np.complex64)
    x_ref = b.copy()
    O.ctrsv(1, 0, 0, n, A, n, x_ref, 1)
    Ad, bd = torch.from_numpy(A).to(cuda), torch.from_numpy(b).to(cuda)
    x = torch.empty_like(bd)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    handle.set_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        x.copy_(bd)
        st = B.iclblasCtrsv(handle, 1, 0, 0, n, Ad, n, x, 1)
    assert st == B.SUCCESS
    for _ in range(3):
        x.fill_(7)
        g.replay()
        torch.cuda.synchronize()
        assert O.rel_fro(x.cpu().numpy(), x_ref) <= TOL
    handle.set_stream(torch.cuda.current_stream())
    del g
