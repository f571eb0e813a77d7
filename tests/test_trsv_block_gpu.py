"""TRSV's 64-row block kernel (complex data, short solves, and real data that
TMA cannot address) at the edges of its blocks and clusters, and the one-CTA
substitution of up to 128 rows at the edges of its warps' rows, against the
oracle.

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


# one CTA with one, two and four rows a lane; then blocks and their edges, a cluster's 8 blocks and the first of
# the next, several clusters
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 97, 127, 128, 129, 511, 512, 513, 577, 1333])
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


# more than 48 blocks: clusters of at most 8
@pytest.mark.parametrize("n", [3072, 3073, 4100])
@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
def test_long_solves(handle, n, dtype):
    rng = np.random.default_rng(n)
    lda = n | 1
    for uplo in (0, 1):
        A = tri(n, lda, uplo == 1, rng, dtype)
        for trans in (0, 1, 2):
            x = O.colmajor(n, 1, n, rng, dtype)
            x_ref = x.copy()
            want(dtype, uplo, trans, 0, n, A, lda, x_ref, 1)
            assert solve(handle, dtype, uplo, trans, 0, n, A, lda, x, 1) == B.SUCCESS
            assert O.rel_fro(x, x_ref) <= TOL


@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
@pytest.mark.parametrize("uplo", [0, 1])
def test_non_finite(handle, dtype, uplo):
    """A NaN or an infinity in b and a zero on the diagonal make exactly the
    entries non-finite that substitution makes so."""
    rng = np.random.default_rng(5 + uplo)
    for n, what in ((n, what) for n in (201, 50) for what in ("nan", "inf", "zero")):
        A = tri(n, n, uplo == 1, rng, dtype)
        x = O.colmajor(n, 1, n, rng, dtype)
        if what == "zero":
            A[n // 2 * n + n // 2] = 0
        else:
            x[n // 2] = np.nan if what == "nan" else np.inf
        x_ref = x.copy()
        with np.errstate(all="ignore"):
            want(dtype, uplo, 0, 0, n, A, n, x_ref, 1)
        assert solve(handle, dtype, uplo, 0, 0, n, A, n, x, 1) == B.SUCCESS
        fin = np.isfinite(x_ref)
        assert np.array_equal(np.isfinite(x), fin)
        if dtype == np.float32:  # infinities and NaNs where substitution has them
            assert np.array_equal(x[~fin], x_ref[~fin], equal_nan=True)
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


def forms(dtype):
    """(n, lda): complex, real that TMA cannot address, and short aligned real solves."""
    return ((100, 101), (130, 131), (200, 200)) + (() if dtype == np.complex64 else ((512, 512),))


@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
@pytest.mark.parametrize("uplo", [0, 1])
def test_growth(handle, dtype, uplo):
    """Unit triangles with entries of size 1, whose diagonal blocks have large
    inverses: substitution leaves a residual of about sqrt(n) roundings of
    |T| |x|, a product with an FP32 inverse hundreds of them."""
    for n, lda in ((130, 131), (200, 200)) + (() if dtype == np.complex64 else ((256, 256),)):
        rng = np.random.default_rng(n)
        A = O.colmajor(n, n, lda, rng, dtype)
        T = A.reshape(n, lda).T[:n].astype(np.complex128 if dtype == np.complex64 else np.float64)
        T = (np.tril(T, -1) if uplo == 1 else np.triu(T, 1)) + np.eye(n)
        b = (T @ rng.uniform(-1, 1, n)).astype(dtype)
        x = b.copy()
        assert solve(handle, dtype, uplo, 0, 1, n, A, lda, x, 1) == B.SUCCESS
        assert np.isfinite(x).all()
        res = np.abs(T @ x - b).max() / (np.abs(T) @ np.abs(x)).max()
        assert res <= 2 * np.sqrt(n) * 2.0 ** -24


@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
@pytest.mark.parametrize("uplo", [0, 1])
def test_inverse_below_normal_range(handle, dtype, uplo):
    """Diagonals so large that the inverse's other entries vanish in FP32: each
    entry of x is still right to a few roundings."""
    mid = (3e18, 1e-3, 1e18) if dtype == np.complex64 else (1e23, 1.0, 1e23)
    # (70: diagonals whose reciprocals the one-CTA substitution does not form either)
    for n, lda, (d, e, f) in [(n, lda, mid) for n, lda in forms(dtype)] + [(70, 71, (1e32, 1.0, 1e32))]:
        rng = np.random.default_rng(n)
        A = (O.colmajor(n, n, lda, rng, dtype) * dtype(e)).astype(dtype)
        M = A.reshape(n, lda).T[:n]
        M[np.arange(n), np.arange(n)] = d
        b = np.zeros(n, dtype)
        b[::64] = f
        if uplo == 0:
            b = b[::-1].copy()
        wide = np.complex128 if dtype == np.complex64 else np.float64
        want = b.astype(wide)
        T = M.astype(wide)
        for i in range(n) if uplo == 1 else range(n - 1, -1, -1):
            want[i] /= T[i, i]
            rest = slice(i + 1, n) if uplo == 1 else slice(0, i)
            want[rest] -= T[rest, i] * want[i]
        assert (np.abs(want) > 1e-36).all()
        x = b.copy()
        assert solve(handle, dtype, uplo, 0, 0, n, A, lda, x, 1) == B.SUCCESS
        assert (np.abs(x - want) <= 1e-4 * np.abs(want)).all()


@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
def test_narrow_band(handle, dtype):
    """An inverse that falls off below FP32's range, harmlessly."""
    for n, lda in forms(dtype):
        rng = np.random.default_rng(n)
        A = np.zeros(lda * n, dtype)
        M = A.reshape(n, lda).T[:n]
        M[np.arange(n), np.arange(n)] = 4096
        M[np.arange(1, n), np.arange(n - 1)] = 1
        x = O.colmajor(n, 1, n, rng, dtype)
        x_ref = x.copy()
        want(dtype, 1, 0, 0, n, A, lda, x_ref, 1)
        assert solve(handle, dtype, 1, 0, 0, n, A, lda, x, 1) == B.SUCCESS
        assert O.rel_fro(x, x_ref) <= TOL
