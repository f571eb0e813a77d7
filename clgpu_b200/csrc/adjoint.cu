// Adjoints (reverse-mode derivatives) of TRSM and GEMM.  No reference
// counterpart.
//
// TRSM, left side, X = alpha * M^-1 * B with M = op(A):
//     W = M^-T G                      (TRSM with the transposed operator)
//     dB = alpha * W
//     dM = -W X^T,   dA = dM (op N) or dM^T (op T/C), kept on the stored
//                    triangle (and off the diagonal for a unit diagonal).
// Right side, X = alpha * B * M^-1:
//     W = G M^-T,  dB = alpha * W,  dM = -X^T W.
// GEMM, C = alpha*op(A)*op(B) + beta*C:
//     d op(A) = alpha * G op(B)^T,  d op(B) = alpha * op(A)^T G,  dC = beta * G.
// The products run through the library's GEMM and TRSM (and so follow the
// handle's math mode).  dA is formed by the triangular-output GEMM, which
// computes only the tiles meeting the stored triangle; one small kernel then
// zeroes the other triangle (and a unit diagonal).
#include "common.cuh"

namespace iclb {

namespace {

// Zero the entries of the n x n block that are not on the stored triangle
// (the triangular-output GEMM leaves them untouched); with a unit diagonal
// the diagonal is not an input either.  One warp a column (grid-stride), its
// run of zeros only, 16 bytes a store past the first aligned entry: bound by
// the 2 n^2 bytes it writes (n = 8192: 22 us; an element a thread, with a
// division each, 108 us)
__global__ void __launch_bounds__(256) mask_triangle_kernel(int n, int lower, int unit, float* __restrict__ D, long ldd)
{
    const int lane = threadIdx.x & 31, nw = gridDim.x * 8;
    for (int j = blockIdx.x * 8 + (threadIdx.x >> 5); j < n; j += nw) {
        // rows [b, e) of column j
        const int b = lower ? 0 : j + (unit ? 0 : 1), e = lower ? j + (unit ? 1 : 0) : n;
        float* const c = D + (long)j * ldd;
        const int a = min(e, b + (int)((4 - (((uintptr_t)(c + b) >> 2) & 3)) & 3));  // first 16-byte aligned row
        if (b + lane < a) c[b + lane] = 0.f;
        const int q = a + (max(0, e - a) & ~3);
        for (int i = a + 4 * lane; i < q; i += 128) *reinterpret_cast<float4*>(c + i) = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q + lane < e) c[q + lane] = 0.f;
    }
}

// D = s * S (m x n blocks, column-major)
__global__ void scale_copy_kernel(int m, int n, float s, const float* __restrict__ S, long lds, float* __restrict__ D,
                                  long ldd)
{
    const long total = (long)m * n;
    for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        const long j = e / m, i = e % m;
        D[j * ldd + i] = s * S[j * lds + i];
    }
}

int grid_for(iclblasHandle_t h, long total)
{
    long g = (total + 255) / 256;
    long cap = (long)h->sm_count * 8;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

cudaError_t strsm_backward(iclblasHandle_t h, int side, int uplo, int trans, int diag, int m, int n, float alpha,
                           const float* A, int lda, const float* X, int ldx, float* G, int ldg, float* dA, int ldda)
{
    const bool left = side == ICLBLAS_SIDE_LEFT;
    const bool t = trans != ICLBLAS_OP_N;
    const int flipped = t ? ICLBLAS_OP_N : ICLBLAS_OP_T;
    // W in place of G
    cudaError_t e = strsm(h, side, uplo, flipped, diag, m, n, 1.f, A, lda, G, ldg);
    if (e != cudaSuccess) return e;
    if (dA) {
        const int na = left ? m : n;
        // only the stored triangle of dA is formed (1: row >= col, 2: row <= col)
        const int tri = uplo == ICLBLAS_FILL_MODE_LOWER ? 1 : 2;
        if (left) {
            // dM = -W X^T (m x m, inner n); dA = dM or dM^T = -X W^T
            e = t ? sgemm_tri(h, tri, ICLBLAS_OP_N, ICLBLAS_OP_T, m, m, n, -1.f, X, ldx, G, ldg, 0.f, dA, ldda)
                  : sgemm_tri(h, tri, ICLBLAS_OP_N, ICLBLAS_OP_T, m, m, n, -1.f, G, ldg, X, ldx, 0.f, dA, ldda);
        } else {
            // dM = -X^T W (n x n, inner m); dA = dM or dM^T = -W^T X
            e = t ? sgemm_tri(h, tri, ICLBLAS_OP_T, ICLBLAS_OP_N, n, n, m, -1.f, G, ldg, X, ldx, 0.f, dA, ldda)
                  : sgemm_tri(h, tri, ICLBLAS_OP_T, ICLBLAS_OP_N, n, n, m, -1.f, X, ldx, G, ldg, 0.f, dA, ldda);
        }
        if (e != cudaSuccess) return e;
        mask_triangle_kernel<<<grid_for(h, (long)na * 32), 256, 0, h->stream>>>(
            na, uplo == ICLBLAS_FILL_MODE_LOWER, diag == ICLBLAS_DIAG_UNIT, dA, ldda);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (alpha != 1.f) {
        scale_copy_kernel<<<grid_for(h, (long)m * n), 256, 0, h->stream>>>(m, n, alpha, G, ldg, G, ldg);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t sgemm_backward(iclblasHandle_t h, int ta, int tb, int m, int n, int k, float alpha, const float* A, int lda,
                           const float* B, int ldb, float beta, const float* G, int ldg, float* dA, int ldda,
                           float* dB, int lddb, float* dC, int lddc)
{
    const bool at = ta != ICLBLAS_OP_N, bt = tb != ICLBLAS_OP_N;
    cudaError_t e = cudaSuccess;
    if (dA) {
        // d op(A) = alpha G op(B)^T (m x k); stored A is op(A) or its transpose
        if (!at)
            e = bt ? sgemm(h, ICLBLAS_OP_N, ICLBLAS_OP_N, m, k, n, alpha, G, ldg, B, ldb, 0.f, dA, ldda)
                   : sgemm(h, ICLBLAS_OP_N, ICLBLAS_OP_T, m, k, n, alpha, G, ldg, B, ldb, 0.f, dA, ldda);
        else
            e = bt ? sgemm(h, ICLBLAS_OP_T, ICLBLAS_OP_T, k, m, n, alpha, B, ldb, G, ldg, 0.f, dA, ldda)
                   : sgemm(h, ICLBLAS_OP_N, ICLBLAS_OP_T, k, m, n, alpha, B, ldb, G, ldg, 0.f, dA, ldda);
        if (e != cudaSuccess) return e;
    }
    if (dB) {
        // d op(B) = alpha op(A)^T G (k x n)
        if (!bt)
            e = at ? sgemm(h, ICLBLAS_OP_N, ICLBLAS_OP_N, k, n, m, alpha, A, lda, G, ldg, 0.f, dB, lddb)
                   : sgemm(h, ICLBLAS_OP_T, ICLBLAS_OP_N, k, n, m, alpha, A, lda, G, ldg, 0.f, dB, lddb);
        else
            e = at ? sgemm(h, ICLBLAS_OP_T, ICLBLAS_OP_T, n, k, m, alpha, G, ldg, A, lda, 0.f, dB, lddb)
                   : sgemm(h, ICLBLAS_OP_T, ICLBLAS_OP_N, n, k, m, alpha, G, ldg, A, lda, 0.f, dB, lddb);
        if (e != cudaSuccess) return e;
    }
    if (dC) {
        scale_copy_kernel<<<grid_for(h, (long)m * n), 256, 0, h->stream>>>(m, n, beta, G, ldg, dC, lddc);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace iclb
