"""Plain GEMM on every tile of its dispatch, at the tile's edges, real and
complex, against the oracle.

Real: bit-identical (each output sums k in order by FP32 FMAs).  Complex:
relative Frobenius error <= 1e-5, the bar of the other CGEMM tests."""
import numpy as np
import pytest

import oracle_lib as O
from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu

# one row / column below, at and above a tile edge, for shapes that take the
# 16, 32, 64 x 64, 128 x 64 and 128 x 128 tiles; k at and around a K tile
SHAPES = [(1, 1, 1), (15, 17, 33), (100, 90, 31), (129, 255, 65), (512, 500, 17), (700, 900, 16), (897, 1025, 15),
          (1290, 1410, 40), (2047, 2049, 9)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_sgemm_tiles(handle, m, n, k):
    rng = np.random.default_rng(m + n + k)
    for ta, tb in ((0, 0), (0, 1), (1, 0), (2, 2)):
        for pad, beta in ((0, 0.5), (1, 0.0)):
            ra, ca = (m, k) if ta == 0 else (k, m)
            rb, cb = (k, n) if tb == 0 else (n, k)
            A = O.colmajor(ra, ca, ra + pad, rng)
            Bm = O.colmajor(rb, cb, rb + pad, rng)
            C = O.colmajor(m, n, m + pad, rng)
            want = C.copy()
            O.sgemm(ta, tb, m, n, k, 1.25, A, ra + pad, Bm, rb + pad, beta, want, m + pad)
            assert B.iclblasSgemm(handle, ta, tb, m, n, k, 1.25, A, ra + pad, Bm, rb + pad, beta, C, m + pad) == B.SUCCESS
            assert np.array_equal(C, want)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (15, 17, 33), (100, 90, 31), (333, 400, 17), (513, 700, 9), (3140, 3200, 7)])
def test_cgemm_tiles(handle, m, n, k):
    rng = np.random.default_rng(m + n + k)
    for ta, tb in ((0, 0), (2, 1), (1, 2)):
        pad = ta
        ra, ca = (m, k) if ta == 0 else (k, m)
        rb, cb = (k, n) if tb == 0 else (n, k)
        A = O.colmajor(ra, ca, ra + pad, rng, np.complex64)
        Bm = O.colmajor(rb, cb, rb + pad, rng, np.complex64)
        C = O.colmajor(m, n, m + pad, rng, np.complex64)
        want = C.copy()
        O.cgemm(ta, tb, m, n, k, 1.25 - 0.5j, A, ra + pad, Bm, rb + pad, 0.5j, want, m + pad)
        assert B.iclblasCgemm(handle, ta, tb, m, n, k, 1.25 - 0.5j, A, ra + pad, Bm, rb + pad, 0.5j, C, m + pad) == B.SUCCESS
        assert O.rel_fro(C, want) <= 1e-5


# flat products of millions of columns: more column tiles of the small sizes
# than a grid has in y
def test_sgemm_flat(handle):
    m, n, k = 4, 2_100_000, 4
    rng = np.random.default_rng(1)
    A, Bm, C = (O.colmajor(r, c, r, rng) for r, c in ((m, k), (k, n), (m, n)))
    want = C.copy()
    O.sgemm(0, 0, m, n, k, 1.25, A, m, Bm, k, 0.5, want, m)
    assert B.iclblasSgemm(handle, 0, 0, m, n, k, 1.25, A, m, Bm, k, 0.5, C, m) == B.SUCCESS
    assert np.array_equal(C, want)


@pytest.mark.parametrize("m,n", [(4, 1_100_000), (20, 2_100_000)])
def test_cgemm_flat(handle, m, n):
    k = 3
    rng = np.random.default_rng(m)
    A, Bm, C = (O.colmajor(r, c, r, rng, np.complex64) for r, c in ((m, k), (k, n), (m, n)))
    want = C.copy()
    O.cgemm(0, 0, m, n, k, 1.25, A, m, Bm, k, 0.5j, want, m)
    assert B.iclblasCgemm(handle, 0, 0, m, n, k, 1.25, A, m, Bm, k, 0.5j, C, m) == B.SUCCESS
    assert O.rel_fro(C, want) <= 1e-5
