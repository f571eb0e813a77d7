// GEMV: y = alpha*op(A)*x + beta*y for float and complex float.
//
// Replaces the reference's Sgemv_opt_simd16 / Sgemv_opt_simd16_TC /
// Cgemv_naive kernels (libs/blas/funcs/Sgemv/*, Cgemv/*), whose lanes stride
// across columns of a column-major matrix.  Here A is read once, coalesced:
//   op N: each thread owns 16 bytes of consecutive rows (4 floats or 2
//         complex) and walks a slice of columns; slices of columns run in
//         different blocks, their per-row partial sums go to scratch, and the
//         last block of each row tile adds them in slice order (deterministic)
//         and applies alpha/beta;
//   op T/C: one warp per column (a column is contiguous), 128-bit loads down
//         the column, shuffle-tree sum; one block per column where tall
//         columns allow only scalar loads.
// Operands without 16-byte alignment are read by scalar loads, a warp's rows
// consecutive, several columns' loads issued together.
// beta == 0 means y is written without being read (Sgemv_naive.cl:34,54).
#include "common.cuh"
#include "pdl.cuh"

namespace iclb {
namespace {

constexpr int kNThreads = 128;  // op N block
constexpr int kTThreads = 256;  // op T block (8 warps = 8 columns)

// ---- element arithmetic
__device__ __forceinline__ float zero_of(float) { return 0.f; }
__device__ __forceinline__ cfloat zero_of(cfloat) { return cfloat{0.f, 0.f}; }

template <bool CONJ>
__device__ __forceinline__ void madd(float& acc, float a, float x) { acc = fmaf(a, x, acc); }
template <bool CONJ>
__device__ __forceinline__ void madd(cfloat& acc, cfloat a, cfloat x)
{
    const float ai = CONJ ? -a.im : a.im;
    acc.re = fmaf(a.re, x.re, acc.re);
    acc.re = fmaf(-ai, x.im, acc.re);
    acc.im = fmaf(a.re, x.im, acc.im);
    acc.im = fmaf(ai, x.re, acc.im);
}
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ cfloat add(cfloat a, cfloat b) { return cfloat{a.re + b.re, a.im + b.im}; }

// y_out = alpha*s + beta*y (beta == 0: y not read)
__device__ __forceinline__ float axpby(float alpha, float s, float beta, const float* y)
{
    return beta == 0.f ? alpha * s : fmaf(alpha, s, beta * *y);
}
__device__ __forceinline__ cfloat cmulf(cfloat a, cfloat b)
{
    return cfloat{fmaf(a.re, b.re, -a.im * b.im), fmaf(a.re, b.im, a.im * b.re)};
}
__device__ __forceinline__ cfloat axpby(cfloat alpha, cfloat s, cfloat beta, const cfloat* y)
{
    cfloat r = cmulf(alpha, s);
    if (beta.re != 0.f || beta.im != 0.f) r = add(r, cmulf(beta, *y));
    return r;
}

// for kernels whose launch may start before the one ahead of it has ended:
// their inputs aren't constant data.  HALF: complex data at 4 modulo 8.
template <bool HALF = false>
__device__ __forceinline__ float ld_of(const float* p)
{
    return *p;
}
template <bool HALF = false>
__device__ __forceinline__ cfloat ld_of(const cfloat* p)
{
    if (HALF) return cfloat{((const float*)p)[0], ((const float*)p)[1]};
    const float2 v = *(const float2*)p;
    return cfloat{v.x, v.y};
}
// another block's partial sum, past this SM's L1
__device__ __forceinline__ float ldcg_of(const float* p) { return __ldcg(p); }
__device__ __forceinline__ cfloat ldcg_of(const cfloat* p)
{
    const float2 v = __ldcg((const float2*)p);
    return cfloat{v.x, v.y};
}

template <class T>
__device__ __forceinline__ T warp_sum_t(T v);
template <>
__device__ __forceinline__ float warp_sum_t<float>(float v) { return warp_sum(v); }
template <>
__device__ __forceinline__ cfloat warp_sum_t<cfloat>(cfloat v)
{
    return cfloat{warp_sum(v.re), warp_sum(v.im)};
}

// ------------------------------------------------------------------ op N
// Large aligned matrices: block (rt, s) owns rows [rt*R*128, +R*128) and
// columns [s*cps, min(n, (s+1)*cps)); a thread's R rows of a column are one
// 128-bit load.  (The kernel below with G = 1 measured 4 % slower here:
// complex 8192 x 8192 87 us against 83.)
template <class T>
__global__ void __launch_bounds__(kNThreads) gemv_n_stream_kernel(int m, int n, T alpha, const T* __restrict__ A, long lda,
                                                                  const T* __restrict__ x, long incx, T beta,
                                                                  T* __restrict__ y, long incy, int cps,
                                                                  T* __restrict__ partial, unsigned* counters)
{
    constexpr int R = 16 / sizeof(T);
    constexpr int XC = 256;  // x values staged per chunk
    __shared__ T xs[XC];
    const int splits = gridDim.y;
    const int s = blockIdx.y;
    const long row0 = ((long)blockIdx.x * kNThreads + threadIdx.x) * R;
    const int c0 = s * cps;
    const int c1 = min(n, c0 + cps);

    T acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = zero_of(T());

    for (int cb = c0; cb < c1; cb += XC) {
        const int cn = min(XC, c1 - cb);
        __syncthreads();
        for (int i = threadIdx.x; i < cn; i += kNThreads) xs[i] = x[(long)(cb + i) * incx];
        __syncthreads();
        if (row0 < m) {
            const T* Ac = A + (long)cb * lda + row0;
            if (row0 + R <= m) {
                int c = 0;
                for (; c + 8 <= cn; c += 8) {
                    float4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = ld_stream4((const float4*)(Ac + (long)(c + u) * lda));
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const T* e = (const T*)&v[u];
#pragma unroll
                        for (int r = 0; r < R; ++r) madd<false>(acc[r], e[r], xs[c + u]);
                    }
                }
                for (; c < cn; ++c) {
                    float4 v = ld_stream4((const float4*)(Ac + (long)c * lda));
                    const T* e = (const T*)&v;
#pragma unroll
                    for (int r = 0; r < R; ++r) madd<false>(acc[r], e[r], xs[c]);
                }
            } else {
                for (int c = 0; c < cn; ++c) {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (row0 + r < m) madd<false>(acc[r], Ac[(long)c * lda + r], xs[c]);
                }
            }
        }
    }

    if (splits == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (row0 + r < m) {
                T* yp = y + (row0 + r) * incy;
                *yp = axpby(alpha, acc[r], beta, yp);
            }
        return;
    }
    // publish this slice's partial sums; the last slice of the row tile adds them
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (row0 + r < m) partial[(long)s * m + row0 + r] = acc[r];
    if (!last_block_of(counters + blockIdx.x, splits)) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const long row = row0 + r;
        if (row >= m) continue;
        T sum = zero_of(T());
        for (int k = 0; k < splits; ++k) sum = add(sum, ((volatile T*)partial)[(long)k * m + row]);
        T* yp = y + row * incy;
        *yp = axpby(alpha, sum, beta, yp);
    }
    if (threadIdx.x == 0) counters[blockIdx.x] = 0u;
}

// Block (rt, s): rows [rt*R*128, +R*128), columns [s*cps, min(n, (s+1)*cps)),
// in G groups of 128 threads that take turns of 8 columns.
// VEC: lda*sizeof(T) and A are 16-byte aligned, so each thread's R rows of a
// column are one 128-bit load.  Otherwise its rows are 128 apart: every load
// of a warp is one run of 32 elements, and a block still reads whole runs of
// 128 * R elements of a column (runs of 128 alone measured 3 times slower on
// 9001 x 9000).
// G = 1 when the matrix fills the GPU with bandwidth-bound blocks.  Smaller
// ones are bound by the time of a few dependent steps: a batch of 8 columns
// per load latency, then the last block's sum over the slices.  G = 4 does
// four batches at once, adds the groups in shared memory and splits that
// last sum over the groups as well.
// Measured (us, before and after, operands in L2): real 256 x 256 10.7, 4.2;
// 423 x 9911, lda 425, 41, 9.1; 4096 x 4096 19.0, 12.3; 5000 x 5001 42, 15.8;
// 9001 x 9000 (G = 1) 78, 61; complex 3001 x 1777, lda 3003, 18.2, 9.1.
template <class T, bool VEC, int G, bool HALF = false>
__global__ void __launch_bounds__(kNThreads * G) gemv_n_kernel(int m, int n, T alpha, const T* __restrict__ A, long lda,
                                                               const T* __restrict__ x, long incx, T beta,
                                                               T* __restrict__ y, long incy, int cps,
                                                               T* __restrict__ partial, unsigned* counters)
{
    pdl_wait();
    PDL_FRESH(A);
    PDL_FRESH(x);
    PDL_FRESH(y);
    PDL_FRESH(partial);
    pdl_trigger();
    constexpr int R = 16 / sizeof(T);
    constexpr int RS = VEC ? 1 : kNThreads;  // rows of a thread: row0 + r * RS
    constexpr int XC = 256;  // x values staged per chunk
    __shared__ T xs[XC];
    __shared__ T red[G > 1 ? G - 1 : 1][G > 1 ? R * kNThreads : 1];
    const int tid = threadIdx.x % kNThreads, g = G > 1 ? threadIdx.x / kNThreads : 0;
    const int splits = gridDim.y;
    const int s = blockIdx.y;
    const long row0 = VEC ? ((long)blockIdx.x * kNThreads + tid) * R : (long)blockIdx.x * kNThreads * R + tid;
    const int c0 = s * cps;
    const int c1 = min(n, c0 + cps);

    T acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = zero_of(T());
    // acc of group 0 += those of the other groups, in order
    auto add_groups = [&]() {
        if constexpr (G > 1) {
            if (g > 0)
#pragma unroll
                for (int r = 0; r < R; ++r) red[g - 1][r * kNThreads + tid] = acc[r];
            __syncthreads();
            if (g == 0)
#pragma unroll
                for (int q = 0; q < G - 1; ++q)
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[r] = add(acc[r], red[q][r * kNThreads + tid]);
        }
    };

    for (int cb = c0; cb < c1; cb += XC) {
        const int cn = min(XC, c1 - cb);
        __syncthreads();
        for (int i = threadIdx.x; i < cn; i += kNThreads * G) xs[i] = x[(long)(cb + i) * incx];
        __syncthreads();
        if (row0 < m) {
            const T* Ac = A + (long)cb * lda + row0;
            if (VEC && row0 + R <= m) {
                int c = 8 * g;
                for (; c + 8 <= cn; c += 8 * G) {
                    float4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = ld_stream4((const float4*)(Ac + (long)(c + u) * lda));
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const T* e = (const T*)&v[u];
#pragma unroll
                        for (int r = 0; r < R; ++r) madd<false>(acc[r], e[r], xs[c + u]);
                    }
                }
                for (const int ce = min(c + 8, cn); c < ce; ++c) {
                    float4 v = ld_stream4((const float4*)(Ac + (long)c * lda));
                    const T* e = (const T*)&v;
#pragma unroll
                    for (int r = 0; r < R; ++r) madd<false>(acc[r], e[r], xs[c]);
                }
            } else {
                int c = 8 * g;
                // (VEC: the few rows past the last whole vector)
                for (; c + 8 <= cn; c += 8 * G) {
                    T v[8][R];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            v[u][r] = row0 + r * RS < m ? ld_of<HALF>(Ac + (long)(c + u) * lda + r * RS) : zero_of(T());
#pragma unroll
                    for (int u = 0; u < 8; ++u)
#pragma unroll
                        for (int r = 0; r < R; ++r) madd<false>(acc[r], v[u][r], xs[c + u]);
                }
                for (; c < cn; c += VEC ? 8 * G : cn) {
                    for (int u = c; u < min(c + 8, cn); ++u) {
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            if (row0 + r * RS < m) madd<false>(acc[r], Ac[(long)u * lda + r * RS], xs[u]);
                    }
                }
            }
        }
    }
    add_groups();

    if (splits == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (g == 0 && row0 + r * RS < m) {
                T* yp = y + (row0 + r * RS) * incy;
                *yp = axpby(alpha, acc[r], beta, yp);
            }
        return;
    }
    // publish this slice's partial sums; the last slice of the row tile adds
    // them, each group a run of consecutive slices
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (g == 0 && row0 + r * RS < m) partial[(long)s * m + row0 + r * RS] = acc[r];
    if (!last_block_of(counters + blockIdx.x, splits)) return;
    const int per = (splits + G - 1) / G, k1 = min(splits, (g + 1) * per);
    constexpr int KU = 32 / R;  // slices in flight
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = zero_of(T());
    for (int k = g * per; k < k1; k += KU) {
        T t[KU][R];
#pragma unroll
        for (int u = 0; u < KU; ++u)
#pragma unroll
            for (int r = 0; r < R; ++r)
                t[u][r] = (k + u < k1 && row0 + r * RS < m) ? ldcg_of(partial + (long)(k + u) * m + row0 + r * RS)
                                                            : zero_of(T());
#pragma unroll
        for (int u = 0; u < KU; ++u)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = add(acc[r], t[u][r]);
    }
    add_groups();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const long row = row0 + r * RS;
        if (g != 0 || row >= m) continue;
        T* yp = y + row * incy;
        *yp = axpby(alpha, acc[r], beta, yp);
    }
    if (threadIdx.x == 0) counters[blockIdx.x] = 0u;
}

// ------------------------------------------------------------------ op T / C
// Warp w of the grid handles column col = w / S, row slice w % S of S.
template <class T, bool CONJ, bool VEC, int U>
__global__ void __launch_bounds__(kTThreads) gemv_t_kernel(int m, int n, T alpha, const T* __restrict__ A, long lda,
                                                           const T* __restrict__ x, long incx, T beta,
                                                           T* __restrict__ y, long incy, int S, int rps,
                                                           T* __restrict__ partial, unsigned* counters)
{
    constexpr int R = 16 / sizeof(T);
    const int lane = threadIdx.x & 31;
    const long gw = ((long)blockIdx.x * kTThreads + threadIdx.x) >> 5;
    const long col = gw / S;
    const int s = (int)(gw % S);
    if (col >= n) return;
    const int r0 = s * rps, r1 = min(m, r0 + rps);
    const T* Ac = A + col * lda;
    T acc = zero_of(T());
    if (VEC) {
        // r0 is a multiple of 32*R: every load is one aligned 128-bit vector.
        // Real data: two partial sums (even and odd vectors of the unrolled
        // step) halve the dependent FMA chain and are added in a fixed order
        // after it (complex data keeps one: its four-FMA updates already
        // interleave, and a second sum measured slower).
        T acc2 = zero_of(T());
        int r = r0 + lane * R;
        for (; r + 3 * 32 * R + R <= r1; r += 4 * 32 * R) {
            float4 v[4], xv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[u] = ld_stream4((const float4*)(Ac + r + u * 32 * R));
                xv[u] = __ldg((const float4*)(x + r + u * 32 * R));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const T* e = (const T*)&v[u];
                const T* xe = (const T*)&xv[u];
#pragma unroll
                for (int k = 0; k < R; ++k) madd<CONJ>((sizeof(T) == sizeof(float) && (u & 1)) ? acc2 : acc, e[k], xe[k]);
            }
        }
        acc = add(acc, acc2);
        for (; r + R <= r1; r += 32 * R) {
            float4 v = ld_stream4((const float4*)(Ac + r));
            float4 xv = __ldg((const float4*)(x + r));
            const T* e = (const T*)&v;
            const T* xe = (const T*)&xv;
#pragma unroll
            for (int k = 0; k < R; ++k) madd<CONJ>(acc, e[k], xe[k]);
        }
        for (int k = 0; k < R; ++k)
            if (r + k < r1) madd<CONJ>(acc, Ac[r + k], x[r + k]);
    } else {
        // U > 1 (real data): U loads of each operand in flight, the last ones
        // predicated
        if constexpr (U > 1) {
            for (int r = r0 + lane; r < r1; r += U * 32) {
                T v[U], xv[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool in = r + u * 32 < r1;
                    v[u] = in ? __ldg(Ac + r + u * 32) : zero_of(T());
                    xv[u] = in ? __ldg(x + (long)(r + u * 32) * incx) : zero_of(T());
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (r + u * 32 < r1) madd<CONJ>(acc, v[u], xv[u]);
            }
        } else {
            for (int r = r0 + lane; r < r1; r += 32) madd<CONJ>(acc, Ac[r], x[(long)r * incx]);
        }
    }
    acc = warp_sum_t(acc);
    if (S == 1) {
        if (lane == 0) {
            T* yp = y + col * incy;
            *yp = axpby(alpha, acc, beta, yp);
        }
        return;
    }
    if (lane == 0) {
        partial[(long)s * n + col] = acc;
        __threadfence();
        unsigned t = atomicAdd(counters + col, 1u);
        if (t == (unsigned)S - 1) {
            __threadfence();
            T sum = zero_of(T());
            for (int k = 0; k < S; ++k) sum = add(sum, ((volatile T*)partial)[(long)k * n + col]);
            T* yp = y + col * incy;
            *yp = axpby(alpha, sum, beta, yp);
            counters[col] = 0u;
        }
    }
}

// Tall columns without 16-byte alignment: a block a column, its rows in eight
// runs, one a warp, 8 loads of each operand in flight, the warps' sums added
// in shared memory.  Against warps that each take a slice of a column, whose
// sums go through global memory and an atomic, see block_columns().
template <class T, bool CONJ>
__global__ void __launch_bounds__(kTThreads) gemv_t_block_kernel(int m, T alpha, const T* __restrict__ A, long lda,
                                                                 const T* __restrict__ x, long incx, T beta,
                                                                 T* __restrict__ y, long incy, int seg)
{
    pdl_wait();
    PDL_FRESH(A);
    PDL_FRESH(x);
    PDL_FRESH(y);
    pdl_trigger();
    constexpr int W = kTThreads / 32, U = 8;
    __shared__ T part[W];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long col = blockIdx.x;
    const T* Ac = A + col * lda;
    const int r1 = min(m, (w + 1) * seg);
    T acc = zero_of(T());
    for (int r = w * seg + lane; r < r1; r += U * 32) {
        T v[U], xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = r + u * 32 < r1;
            v[u] = in ? ld_of(Ac + r + u * 32) : zero_of(T());
            xv[u] = in ? ld_of(x + (long)(r + u * 32) * incx) : zero_of(T());
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (r + u * 32 < r1) madd<CONJ>(acc, v[u], xv[u]);
    }
    acc = warp_sum_t(acc);
    if (lane == 0) part[w] = acc;
    __syncthreads();
    if (threadIdx.x != 0) return;
    T sum = part[0];
#pragma unroll
    for (int k = 1; k < W; ++k) sum = add(sum, part[k]);
    T* yp = y + col * incy;
    *yp = axpby(alpha, sum, beta, yp);
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// Whether op T / C of an unaligned m x n matrix takes a block a column.  The
// slices have a warp per 1024 rows of a column, so few columns leave the SMs
// idle, all the more below 2048 rows, where a column is one slice; many columns
// fill them, and then the blocks' reductions and partly empty last wave cost
// more than the slices' sums.  Very long columns keep a block's eight warps
// reading for longer than the slices' sums take, unless there are columns for
// all SMs.  Complex columns of two slices lose to the blocks only up to twice
// as many columns as the SMs hold blocks.
// Time in blocks over time in slices, several sets of operands in turn (one
// set, in L2): real 1297 x 800 0.58 (0.65), 1297 x 3500 1.24 (1.15), 2047 x
// 2600 0.84 (0.86), 4001 x 4500 0.80 (0.82), 12001 x 500 1.13 (0.96), 30001 x
// 100 2.05 (1.09), 1000001 x 33 13 (13); complex 2047 x 1700 0.50 (0.68), 1297
// x 3500 1.03 (1.34), 3001 x 1700 0.88 (0.92), 3001 x 4500 1.41 (1.48), 4001 x
// 3500 0.79 (0.80), 30001 x 300 1.42 (1.02), 30001 x 1200 0.81 (0.81).
bool block_columns(bool cplx, int m, int n)
{
    if (m < 1024 || n > 6000) return false;
    if (m < 2048) return n <= 2 * m;
    if (!cplx) return m <= 16384;
    if (m < 3072) return n <= 2400;
    return m <= 12288 || (m <= 65536 && n >= 500);
}

template <class T>
cudaError_t gemv_impl(iclblasHandle_t h, int trans, int m, int n, T alpha, const T* A, int lda, const T* x, int incx,
                      T beta, T* y, int incy)
{
    constexpr int R = 16 / sizeof(T);
    const int target = h->sm_count * 8;
    if (trans == ICLBLAS_OP_N) {
        const bool vec = aligned16(A) && ((long)lda * sizeof(T)) % 16 == 0;
        const int rows_per_block = kNThreads * R;
        const int rt = ceil_div(m, rows_per_block);
        // bandwidth-bound: enough blocks of 64 columns and more to fill the
        // GPU (one group a block); else four groups a block and as many
        // slices as the SMs hold blocks, at least one batch of columns a
        // group (16384 x 16384 with four groups: 297 us against 159).  Up to
        // 128 columns are one slice: adding slices costs more than a few
        // batches (3000 x 33 4.1 us with two, 2.4), and so they are where the
        // row tiles nearly fill the GPU (100000 x 200 12.5, 8.9); with a batch
        // or two of columns three groups would be idle (complex 1000000 x 4
        // 17 us with four groups, 5.8 with one; 100000 x 4 3.3, 2.4).  The other
        // side: at 100 to 128 columns and a dozen to 40 row tiles two slices are
        // faster on operands in HBM (complex 6001 x 128, lda 6001, 9.3 us in one,
        // 6.1), but then a handle's first call would need scratch; over 200 to
        // 1000000 rows and 1 to 2000 columns, in L2 and in HBM, this rule is 2.5 %
        // above the best of the three on average, slices throughout 12 %
        const bool wide = rt >= 96, few = n <= 16 && (!vec || rt > 2 * h->sm_count);
        const bool small = (long)rt * max(1, n / 64) < target && !few && !(wide && n > 320);
        int splits = 1, unit = 8;
        if (small) {
            unit = 32;
            if (n > 128 && !wide) splits = min(ceil_div(2 * h->sm_count, rt), ceil_div(n, unit));
        } else if (rt < target && rt <= kCounterWords) {
            splits = ceil_div(target, rt);
            splits = min(splits, max(1, n / 64));
        }
        int cps = ceil_div(n, splits);
        cps = (cps + unit - 1) / unit * unit;
        splits = ceil_div(n, cps);
        T* partial = nullptr;
        if (splits > 1) {
            partial = (T*)scratch(h, sizeof(T) * (size_t)splits * (size_t)m);
            if (!partial) return cudaErrorMemoryAllocation;
        }
        dim3 grid(rt, splits);
#define LAUNCH(V, G, HALF)                                                                                       \
    return pdl_launch(gemv_n_kernel<T, V, G, HALF>, dim3(grid), kNThreads * G, 0, h->stream, dependent((long)m * n), \
                      m, n, alpha, A, lda, x, incx, beta, y, incy, cps, partial, h->ws.counters)
        if constexpr (sizeof(T) == sizeof(cfloat)) {
            if (!aligned8(A)) { if (small) LAUNCH(false, 4, true); else LAUNCH(false, 1, true); }
        }
        if (small) { if (vec) LAUNCH(true, 4, false); else LAUNCH(false, 4, false); }
        else if (!vec) LAUNCH(false, 1, false);
        else
            gemv_n_stream_kernel<T><<<grid, kNThreads, 0, h->stream>>>(m, n, alpha, A, lda, x, incx, beta, y, incy, cps,
                                                                       partial, h->ws.counters);
#undef LAUNCH
        return cudaGetLastError();
    }
    // op T / C: columns of A are dot products with x
    const bool vec = aligned16(A) && ((long)lda * sizeof(T)) % 16 == 0 && incx == 1 && aligned16(x);
    const bool conj = (trans == ICLBLAS_OP_C) && sizeof(T) == sizeof(cfloat);
    const bool elems = sizeof(T) == sizeof(float) || (aligned8(A) && aligned8(x));  // else only a float at a time
    if (!vec && elems && block_columns(sizeof(T) == sizeof(cfloat), m, n)) {
        const int seg = ceil_div(ceil_div(m, kTThreads / 32), 32) * 32;
        if (conj)
            return pdl_launch(gemv_t_block_kernel<T, true>, dim3(n), kTThreads, 0, h->stream, dependent((long)m * n),
                              m, alpha, A, lda, x, incx, beta, y, incy, seg);
        else
            return pdl_launch(gemv_t_block_kernel<T, false>, dim3(n), kTThreads, 0, h->stream, dependent((long)m * n),
                              m, alpha, A, lda, x, incx, beta, y, incy, seg);
    }
    const int warps_target = target * (kTThreads / 32);
    int S = 1;
    if (n < warps_target && n <= kCounterWords) S = min(ceil_div(warps_target, n), max(1, m / 1024));
    int rps = ceil_div(m, S);
    rps = (rps + 32 * R - 1) / (32 * R) * (32 * R);
    S = ceil_div(m, rps);
    T* partial = nullptr;
    if (S > 1) {
        partial = (T*)scratch(h, sizeof(T) * (size_t)S * (size_t)n);
        if (!partial) return cudaErrorMemoryAllocation;
    }
    const long warps = (long)n * S;
    const int grid = (int)((warps * 32 + kTThreads - 1) / kTThreads);
#define LAUNCH(C, V, U)                                                                                         \
    gemv_t_kernel<T, C, V, U><<<grid, kTThreads, 0, h->stream>>>(m, n, alpha, A, lda, x, incx, beta, y, incy, S, \
                                                                 rps, partial, h->ws.counters)
    if (conj) { if (vec) LAUNCH(true, true, 1); else LAUNCH(true, false, 1); return cudaGetLastError(); }
    if constexpr (sizeof(T) == sizeof(float)) {
        // batches of loads, unless other columns' warps hide the latency and
        // most of a column's loads would be predicated off: columns of one or
        // two loads a lane, and, with still more columns, those whose second
        // batch is at least 3/8 empty.  Time in batches over time with one load
        // at a time, several sets of operands in turn (one set, in L2): 33 x 2600
        // 1.08 (1.06), 33 x 30000 1.34 (1.35); 300 x 3500 0.91 (1.09), 300 x 30000
        // 1.21 (1.36), 416 x 8000 1.14 (1.13), 440 x 12000 0.94 (1.13), 480 x
        // 12000 0.83 (1.06), 508 x 5036 0.43 (0.62), 1000 x 30000 0.37 (0.37)
        const int rows = min(m, rps);
        const bool single = rows <= 64 ? n > 2048 : rows > 256 && rows <= 416 && n > 6000;
        if (!vec && !single) { LAUNCH(false, false, 8); return cudaGetLastError(); }
    }
    if (vec) LAUNCH(false, true, 1); else LAUNCH(false, false, 1);
#undef LAUNCH
    return cudaGetLastError();
}

}  // namespace

cudaError_t sgemv(iclblasHandle_t h, int trans, int m, int n, float alpha, const float* A, int lda, const float* x,
                  int incx, float beta, float* y, int incy)
{
    return gemv_impl<float>(h, trans, m, n, alpha, A, lda, x, incx, beta, y, incy);
}

cudaError_t cgemv(iclblasHandle_t h, int trans, int m, int n, cfloat alpha, const cfloat* A, int lda, const cfloat* x,
                  int incx, cfloat beta, cfloat* y, int incy)
{
    return gemv_impl<cfloat>(h, trans, m, n, alpha, A, lda, x, incx, beta, y, incy);
}

}  // namespace iclb
