// Plain FP32 GEMM on the CUDA cores (the drop-in default math mode):
// C = alpha*op(A)*op(B) + beta*C for float and complex float, every
// combination of op in {N, T, C}, any lda/ldb/ldc.
//
// Arithmetic is the reference's (Sgemm_ntransAB.cl:16-40 and the epilogue of
// gemm_n3_template.h.cl:493-511): each output accumulates its k terms in
// increasing k with fused multiply-adds in FP32, then
// C = fma(alpha, acc, beta*C), or alpha*acc without reading C when beta == 0.
// Because every thread keeps whole outputs and walks k in order, a result is
// bit-identical to the serial oracle for the same inputs.
//
// Structure: register-tiled CTA tiles (BM x BN) whose operands arrive by
// cp.async, one element per copy, in a ring of shared-memory stages, always
// k-major: the copies of an operand that is contiguous along k (A of op T/C,
// B of op N) scatter into that layout, so neither the layout nor the
// alignment of an operand changes the main loop, no register holds data in
// flight, and K tiles are under way while earlier ones are multiplied.
//
// What bounds it: large products the FMA pipe (ncu at 4096^3: 75 % busy, warps
// waiting for it) together with shared-memory reads (47 % with 16 x 8 outputs
// a thread, 69 % with 8 x 8: a 16-byte read costs four passes however many
// lanes share the address, so 8 x 8 spend as many cycles reading as
// multiplying); small ones
// the latency of one k step times k, since each output sums k in order.
// Against register-staged tiles of the same shapes (us before, after):
// 8192 x 8192 x 4096 NN 11981, 11112, TN 11978, 10524; 2000 x 1500 x 3001 TN
// with odd leading dimensions 670, 463; 1000^3 98.4, 68.6; 512^3 34.9, 18.5;
// 256^3 18.5, 8.3; 128 x 100 x 3000 171, 41.  Complex: 4096 x 4096 x 2048 NN
// 6185, 5430, TN 6456, 5195; 500 x 10000 x 2000 NN 1959, 1734; 2048^2 x 2000
// NN 1551, 1527; (re, im) pairs updated by fma.rn.f32x2 measured 10 % slower than scalar
// FMAs there.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "pdl.cuh"

namespace iclb {
namespace {

__device__ __forceinline__ float conj_if(float v, bool) { return v; }
__device__ __forceinline__ cfloat conj_if(cfloat v, bool c) { return c ? cfloat{v.re, -v.im} : v; }
__device__ __forceinline__ float zero_v(float) { return 0.f; }
__device__ __forceinline__ cfloat zero_v(cfloat) { return cfloat{0.f, 0.f}; }

__device__ __forceinline__ void mac(cfloat& acc, cfloat a, cfloat b)
{
    acc.re = fmaf(a.re, b.re, acc.re);
    acc.re = fmaf(-a.im, b.im, acc.re);
    acc.im = fmaf(a.re, b.im, acc.im);
    acc.im = fmaf(a.im, b.re, acc.im);
}

// Two FP32 fused multiply-adds in one instruction (fma.rn.f32x2): each lane
// of the pair is rounded exactly as fmaf, so a result keeps its bits; the
// float kernel issues half as many FMA instructions (it is issue-bound)
__device__ __forceinline__ unsigned long long pack2(float lo, float hi)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float half2f(unsigned long long v, int hi)
{
    float lo_v, hi_v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo_v), "=f"(hi_v) : "l"(v));
    return hi ? hi_v : lo_v;
}
__device__ __forceinline__ void mac2(unsigned long long& acc, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__host__ __device__ __forceinline__ bool is_zero(float v) { return v == 0.f; }
__host__ __device__ __forceinline__ bool is_zero(cfloat v) { return v.re == 0.f && v.im == 0.f; }

__device__ __forceinline__ float epilogue(float alpha, float acc, float beta, const float* c)
{
    return beta == 0.f ? __fmul_rn(alpha, acc) : fmaf(alpha, acc, __fmul_rn(beta, *c));
}
__device__ __forceinline__ cfloat cmul(cfloat a, cfloat b)
{
    return cfloat{fmaf(a.re, b.re, -a.im * b.im), fmaf(a.re, b.im, a.im * b.re)};
}
__device__ __forceinline__ cfloat epilogue(cfloat alpha, cfloat acc, cfloat beta, const cfloat* c)
{
    cfloat r = cmul(acc, alpha);
    if (beta.re != 0.f || beta.im != 0.f) {
        cfloat t = cmul(*c, beta);
        r.re += t.re;
        r.im += t.im;
    }
    return r;
}

// N consecutive elements from shared memory in 16- or 8-byte vector loads
// (the caller guarantees the alignment).
template <class T, int N>
__device__ __forceinline__ void lds_vec(T* dst, const T* src)
{
    constexpr int bytes = N * (int)sizeof(T);
    if constexpr (bytes == 16) {
        union { float4 v; T t[N]; } u;
        u.v = *reinterpret_cast<const float4*>(src);
#pragma unroll
        for (int i = 0; i < N; ++i) dst[i] = u.t[i];
    } else if constexpr (bytes == 8) {
        union { float2 v; T t[N]; } u;
        u.v = *reinterpret_cast<const float2*>(src);
#pragma unroll
        for (int i = 0; i < N; ++i) dst[i] = u.t[i];
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) dst[i] = src[i];
    }
}

__device__ __forceinline__ void cp_async_elem(float* dst, const float* src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_elem(cfloat* dst, const cfloat* src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 8 : 0)
                 : "memory");
}
// HALF: a complex element as its two floats (operands at 4 modulo 8)
template <bool HALF, class T>
__device__ __forceinline__ void cp_async_from(T* dst, const T* src, bool in)
{
    if constexpr (HALF) {
        cp_async_elem(&dst->re, &src->re, in);
        cp_async_elem(&dst->im, &src->im, in);
    } else {
        cp_async_elem(dst, src, in);
    }
}

// Threads: (BM/TM) x (BN/TN).  Each thread owns TM x TN outputs in runs of VA
// rows and VB columns (16 bytes, or all it has) spread evenly over the tile,
// so its shared-memory reads are conflict-free vectors.
// The warp covers 4 thread rows x 8 thread columns: a fragment read then
// touches 4 or 8 distinct vectors, one shared-memory pass each.
// ST: stages of the ring.  MB: CTAs per SM the registers are bounded for.
template <class T, int BM, int BN, int BK, int TM, int TN, int ST>
struct Cfg {
    static constexpr int TX = BN / TN, TY = BM / TM, NT = TX * TY;
    static constexpr int A_PER = BM * BK / NT, B_PER = BN * BK / NT;
    // rows apart: copies that scatter (8 consecutive k of 2 or 4 rows a
    // warp) fall in different banks, and fragment reads stay 16-byte aligned
    static constexpr int VA = TM < 16 / (int)sizeof(T) ? TM : 16 / (int)sizeof(T), NA = TM / VA;
    static constexpr int VB = TN < 16 / (int)sizeof(T) ? TN : 16 / (int)sizeof(T), NB = TN / VB;
    static constexpr int PAD = 16 / (int)sizeof(T);
    static constexpr int A_EL = BK * (BM + PAD), B_EL = BK * (BN + PAD);
    static constexpr int SMEM = ST * (A_EL + B_EL) * (int)sizeof(T);
    static_assert(A_PER * NT == BM * BK && B_PER * NT == BN * BK, "tile/thread mismatch");
    static_assert(TX % 8 == 0 && TY % 4 == 0 && BK % 8 == 0 && NT % 32 == 0, "warp layout");
    static_assert(NT % BM == 0 || BM % NT == 0, "copy layout");
    static_assert(NT % BN == 0 || BN % NT == 0, "copy layout");
};

// Copies of one operand's BX x BK tile into [kk][i] (pitch PX).  CONTIG_K:
// element (i, kk) at p[i*ld + kk], else at p[kk*ld + i].
template <class T, int BX, int BK, int NT, int PX, bool HALF>
struct TileCopy {
    static constexpr int PER = BX * BK / NT;
    const T* base;   // first element this thread copies, at k = 0
    long ld;
    bool contig_k;
    int i0, kk0;     // its row and k
    int rows;        // rows of the operand from the tile's first
    __device__ TileCopy(const T* p, long ld_, bool ck, int x0, int nx) : ld(ld_), contig_k(ck), rows(nx - x0)
    {
        const int t = threadIdx.x;
        if (ck) { kk0 = t % 8; i0 = t / 8; } else { i0 = t % BX; kk0 = t / BX; }
        base = p + (ck ? (long)(x0 + i0) * ld + kk0 : (long)kk0 * ld + x0 + i0);
    }
    __device__ void copy(T* dst, int k0, int k) const
    {
        if (contig_k) {
            constexpr int KH = BK / 8, RS = NT / 8;   // k octets; rows per pass
            const T* src = base + k0;
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int kk = 8 * (q % KH), i = (q / KH) * RS;
                const bool in = i0 + i < rows && k0 + kk0 + kk < k;
                cp_async_from<HALF>(dst + (kk0 + kk) * PX + i0 + i, in ? src + (long)i * ld + kk : base, in);
            }
        } else {
            constexpr int KS = NT >= BX ? NT / BX : 1, IP = NT >= BX ? 1 : BX / NT;   // k per pass; row passes
            const T* src = base + (long)k0 * ld;
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int kk = (q / IP) * KS, i = (q % IP) * NT;
                const bool in = i0 + i < rows && k0 + kk0 + kk < k;
                cp_async_from<HALF>(dst + (kk0 + kk) * PX + i0 + i, in ? src + (long)kk * ld + i : base, in);
            }
        }
    }
};

// Tiles of tile column bn that meet the lower (tri 1) or upper (2) triangle of
// a square matrix of tm tile rows: those from row tile bn * BN / BM on, or up to
// the one of the column's last row.
template <int BM, int BN>
__host__ __device__ constexpr int tri_tiles(int tri, int tm, int bn)
{
    const int last = (bn * BN + BN - 1) / BM + 1;
    return tri == 1 ? tm - bn * BN / BM : (last < tm ? last : tm);
}

// HALF: complex operands at 4 modulo 8.  CONJ: an operand may be conjugated
// (choosing inside the k loop costs 12 selects per 32 complex products, and a
// fifth of the time: 4096 x 4096 x 2048 NN 6656 us with, 5430 without).
// TRI: triangular output (finding the tile at run time cost every product:
// 512^3 18.4 us without, 21.1 with).
template <class T, int BM, int BN, int BK, int TM, int TN, int ST, int MB, bool HALF, bool CONJ, bool TRI>
__global__ void __launch_bounds__(Cfg<T, BM, BN, BK, TM, TN, ST>::NT, MB)
    gemm_simt_kernel(int ta, int tb, int m, int n, int k, T alpha, const T* __restrict__ A, long lda,
                     const T* __restrict__ B, long ldb, T beta, T* __restrict__ C, long ldc, int tri)
{
    using CF = Cfg<T, BM, BN, BK, TM, TN, ST>;
    constexpr int NT = CF::NT, TX = CF::TX, PA = BM + CF::PAD, PB = BN + CF::PAD;
    extern __shared__ __align__(16) unsigned char simt_smem[];
    T* As = reinterpret_cast<T*>(simt_smem);  // [stage][kk][i]
    T* Bs = As + ST * CF::A_EL;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int WX = TX / 8;  // warps along n
    const int ty = (warp / WX) * 4 + lane / 8, tx = (warp % WX) * 8 + lane % 8;
    int bm = blockIdx.x, bn = blockIdx.y;
    if constexpr (TRI) {
        // tri 1 / 2: only C's lower (row >= col) / upper triangle is formed, by
        // a row of blocks for the tiles that meet it, column after column
        // (blocks of the others took places on the SMs too, and the rest lay
        // unevenly: ssyrk of 2000 x 3000, 136 tiles of 128 x 128, 583 to 647 us with
        // them, 314 to 348 without)
        const int tm = (m + BM - 1) / BM;
        for (bn = 0;; ++bn) {
            const int c = tri_tiles<BM, BN>(tri, tm, bn);
            if (bm < c) break;
            bm -= c;
        }
        if (tri == 1) bm += bn * BN / BM;
    }
    const int m0 = bm * BM, n0 = bn * BN;
    pdl_wait();
    PDL_FRESH(A);
    PDL_FRESH(B);
    PDL_FRESH(C);
    // no pdl_trigger(): blocks of the next launch would take the free places of
    // an SM before this one's end, so that an even grid of that launch came to
    // lie unevenly (1000 x 2000 x 2000, two 128 x 64 tiles an SM: 328 us in a
    // chain of such calls, 229 without; 512^3 the same either way)
    // (a triangle's launch is TRI; with this test and the masks at the end left
    // to run time the other instantiations come out faster: 512^3 18.8 us
    // without, 18.4 so)
    if (!TRI && tri != 0) return;
    const bool a_conj = ta == ICLBLAS_OP_C, b_conj = tb == ICLBLAS_OP_C;
    const TileCopy<T, BM, BK, NT, PA, HALF> ca(A, lda, ta != ICLBLAS_OP_N, m0, m);
    const TileCopy<T, BN, BK, NT, PB, HALF> cb(B, ldb, tb == ICLBLAS_OP_N, n0, n);

    // float: accumulators in pairs along the longer dimension of the thread's
    // outputs (fewer values of the other operand to duplicate)
    constexpr bool kPair = std::is_same<T, float>::value, kPairI = kPair && TM > TN;
    using AccT = std::conditional_t<kPair, unsigned long long, T>;
    constexpr int TMA = kPairI ? TM / 2 : TM, TNA = kPair && !kPairI ? TN / 2 : TN;
    AccT acc[TMA][TNA];
#pragma unroll
    for (int i = 0; i < TMA; ++i)
#pragma unroll
        for (int j = 0; j < TNA; ++j) {
            if constexpr (kPair) acc[i][j] = 0ull;  // (+0.f, +0.f)
            else acc[i][j] = zero_v(T());
        }
    auto acc_at = [&](int i, int j) -> T {
        if constexpr (kPairI) return half2f(acc[i >> 1][j], i & 1);
        else if constexpr (kPair) return half2f(acc[i][j >> 1], j & 1);
        else return acc[i][j];
    };

    const int ktiles = (k + BK - 1) / BK;
    auto fetch = [&](int t) {
        if (t < ktiles) {
            ca.copy(As + (t % ST) * CF::A_EL, t * BK, k);
            cb.copy(Bs + (t % ST) * CF::B_EL, t * BK, k);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int t = 0; t < ST - 1; ++t) fetch(t);
    for (int t = 0; t < ktiles; ++t) {
        // tile t has arrived, and every thread is done with tile t - 1,
        // whose stage the next copies overwrite
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();
        fetch(t + ST - 1);
        const T* at = As + (t % ST) * CF::A_EL + ty * CF::VA;
        const T* bt = Bs + (t % ST) * CF::B_EL + tx * CF::VB;
        // fragments of k kk + 1 are read while those of kk are multiplied
        T a[2][TM], b[2][TN];
        auto read = [&](int kk) {
            T* fa = a[kk & 1];
            T* fb = b[kk & 1];
#pragma unroll
            for (int q = 0; q < CF::NA; ++q) lds_vec<T, CF::VA>(fa + q * CF::VA, at + kk * PA + q * (BM / CF::NA));
#pragma unroll
            for (int q = 0; q < CF::NB; ++q) lds_vec<T, CF::VB>(fb + q * CF::VB, bt + kk * PB + q * (BN / CF::NB));
        };
        read(0);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            if (kk + 1 < BK) read(kk + 1);
            T* fa = a[kk & 1];
            T* fb = b[kk & 1];
            if constexpr (CONJ) {
#pragma unroll
                for (int i = 0; i < TM; ++i) fa[i] = conj_if(fa[i], a_conj);
#pragma unroll
                for (int j = 0; j < TN; ++j) fb[j] = conj_if(fb[j], b_conj);
            }
            if constexpr (kPairI) {
                unsigned long long ap[TMA];
#pragma unroll
                for (int i = 0; i < TMA; ++i) ap[i] = pack2(fa[2 * i], fa[2 * i + 1]);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const unsigned long long bp = pack2(fb[j], fb[j]);
#pragma unroll
                    for (int i = 0; i < TMA; ++i) mac2(acc[i][j], ap[i], bp);
                }
            } else if constexpr (kPair) {
                unsigned long long bp[TNA];
#pragma unroll
                for (int j = 0; j < TNA; ++j) bp[j] = pack2(fb[2 * j], fb[2 * j + 1]);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const unsigned long long ap = pack2(fa[i], fa[i]);
#pragma unroll
                    for (int j = 0; j < TNA; ++j) mac2(acc[i][j], ap, bp[j]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) mac(acc[i][j], fa[i], fb[j]);
            }
        }
    }

    // the row's C values are all loaded before any is stored, so the loads
    // overlap (C is read only when beta != 0)
    const bool read_c = !is_zero(beta);
    auto col = [&](int j) { return n0 + (j / CF::VB) * (BN / CF::NB) + tx * CF::VB + j % CF::VB; };
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gi = m0 + (i / CF::VA) * (BM / CF::NA) + ty * CF::VA + i % CF::VA;
        if (gi >= m) continue;
        T cv[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gj = col(j);
            const bool in = tri == 0 || (tri == 1 ? gi >= gj : gi <= gj);
            cv[j] = (read_c && gj < n && in) ? C[(long)gj * ldc + gi] : zero_v(T());
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gj = col(j);
            if (gj >= n) continue;
            if (tri != 0 && (tri == 1 ? gi < gj : gi > gj)) continue;
            C[(long)gj * ldc + gi] = epilogue(alpha, acc_at(i, j), beta, &cv[j]);
        }
    }
}

template <class T, int BM, int BN, int BK, int TM, int TN, int ST, int MB, bool HALF = false, bool CONJ = false, bool TRI = false>
cudaError_t launch(iclblasHandle_t h, int ta, int tb, int m, int n, int k, T alpha, const T* A, int lda, const T* B,
                   int ldb, T beta, T* C, int ldc, int tri)
{
    using CF = Cfg<T, BM, BN, BK, TM, TN, ST>;
    auto kern = gemm_simt_kernel<T, BM, BN, BK, TM, TN, ST, MB, HALF, CONJ, TRI>;
    if (CF::SMEM > 48 * 1024) {
        // the attribute belongs to the current device's copy of the kernel
        static std::atomic<unsigned long long> smem_set{0};
        const unsigned long long bit = 1ull << (h->device & 63);
        if (!(smem_set.load() & bit)) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CF::SMEM);
            if (e != cudaSuccess) return e;
            smem_set.fetch_or(bit);
        }
    }
    dim3 grid(ceil_div(m, BM), ceil_div(n, BN));
    if (TRI) {
        unsigned tiles = 0;
        for (unsigned j = 0; j < grid.y; ++j) tiles += (unsigned)tri_tiles<BM, BN>(tri, (int)grid.x, (int)j);
        grid = dim3(tiles);
    }
    return pdl_launch(kern, grid, CF::NT, CF::SMEM, h->stream, 1,
                      ta, tb, m, n, k, alpha, A, (long)lda, B, (long)ldb, beta, C, (long)ldc, tri);
}

}  // namespace

namespace {
// Estimated SM cycles of a product: a lone tile on an SM takes alone0 (its
// first copies and its stores) + alone * k, bound by latency; several take
// each0 + full * (the part of the tiles inside C) + each * k apiece, bound by
// throughput.  Fitted, near the figures of grids of one to 500 full tiles an
// SM, to the times of every tile at 1481 real and 1478 complex shapes of 1 to a
// million rows or columns and k of 2 to 4000: the tile so picked costs 0.24 %
// (complex 0.34 %) more than the fastest one on average, without the constant
// terms and `full` it was 3.0 % (1.1 %), and 60 % at 1000000 x 1 x 4 or 30 % at
// 1000 x 2000 x 4.
struct TileCost {
    int bm, bn;
    double alone0, alone, each0, full, each;
};
constexpr TileCost kRealTiles[] = {{128, 128, 15100, 193, 523, 11900, 200},
                                   {128, 64, 9000, 128, 709, 6300, 110},
                                   {64, 64, 9320, 124, 296, 4210, 67.3},
                                   {32, 32, 2410, 43.9, 200, 476, 22},
                                   {16, 16, 293, 27.8, 270, 129, 10.2}};
constexpr TileCost kCplxTiles[] = {{64, 64, 7410, 244, 333, 5040, 213},
                                   {32, 32, 1600, 71, 309, 1050, 58.4},
                                   {16, 16, 263, 42.8, 140, 253, 19.1}};

// the tile of the least estimated time, of those whose columns fit the grid's
// 65,535 blocks in y (the largest tile of a table, the first, may not: n above
// 8.3 million real or 4.1 million complex columns)
template <int N>
int pick_tile(const TileCost (&c)[N], int sms, int m, int n, int k, bool tri)
{
    int best = 0;
    double best_t = 0;
    for (int q = 0; q < N; ++q) {
        const long tm = ceil_div(m, c[q].bm), tn = ceil_div(n, c[q].bn);
        if (q > 0 && tn > 65535) continue;
        const long tiles = tri ? (tm * tn + std::max(tm, tn)) / 2 : tm * tn;
        const double inside = (double)m * n / ((double)tm * c[q].bm * tn * c[q].bn);
        const double t = std::max(c[q].alone0 + c[q].alone * k,
                                  ceil_div(tiles, sms) * (c[q].each0 + c[q].full * inside + c[q].each * k));
        if (q == 0 || t < best_t) {
            best = q;
            best_t = t;
        }
    }
    return best;
}
}  // namespace

cudaError_t sgemm_simt(iclblasHandle_t h, int ta, int tb, int m, int n, int k, float alpha, const float* A, int lda,
                       const float* B, int ldb, float beta, float* C, int ldc, int tri)
{
#define LAUNCH(...)                                                                                               \
    (tri != 0 ? launch<float, __VA_ARGS__, false, false, true>(h, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, tri) \
              : launch<float, __VA_ARGS__>(h, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, 0))
    switch (pick_tile(kRealTiles, h->sm_count, m, n, k, tri != 0)) {
    case 0:
        // 16 x 8 outputs a thread read less shared memory per product, 8 x 8
        // hide latency with twice the warps: 4000 x 4000 (7 tiles an SM) x
        // 2000 1368 us against 1399, x 1000 712 and 711, x 500 384 and 372,
        // x 48 76 and 54; 3000 x 3000 x 1000 (4 tiles an SM) 39.7 TFLOP/s
        // against 41.8
        if (k >= 1000 && (long)ceil_div(m, 128) * ceil_div(n, 128) >= 6L * h->sm_count) return LAUNCH(128, 128, 16, 16, 8, 3, 2);
        return LAUNCH(128, 128, 16, 8, 8, 3, 2);
    case 1: return LAUNCH(128, 64, 16, 8, 8, 4, 3);
    case 2: return LAUNCH(64, 64, 16, 8, 8, 4, 6);
    case 3: return LAUNCH(32, 32, 16, 4, 4, 4, 4);
    default: return LAUNCH(16, 16, 32, 2, 2, 4, 4);
    }
#undef LAUNCH
}

cudaError_t cgemm_simt(iclblasHandle_t h, int ta, int tb, int m, int n, int k, cfloat alpha, const cfloat* A, int lda,
                       const cfloat* B, int ldb, cfloat beta, cfloat* C, int ldc)
{
#define LAUNCH(...) launch<cfloat, __VA_ARGS__>(h, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, 0)
    const int tile = pick_tile(kCplxTiles, h->sm_count, m, n, k, false);
    if (!aligned8(A) || !aligned8(B)) {
        // two copies an element: the small tile is not worth a third of these
        return tile == 0 ? LAUNCH(64, 64, 8, 8, 4, 4, 3, true, true) : LAUNCH(32, 32, 16, 4, 2, 3, 4, true, true);
    }
    if (ta == ICLBLAS_OP_C || tb == ICLBLAS_OP_C) {
        switch (tile) {
        case 0: return LAUNCH(64, 64, 8, 8, 4, 4, 3, false, true);
        case 1: return LAUNCH(32, 32, 16, 4, 2, 3, 4, false, true);
        default: return LAUNCH(16, 16, 16, 2, 2, 3, 4, false, true);
        }
    }
    switch (tile) {
    case 0: return LAUNCH(64, 64, 8, 8, 4, 4, 3);
    case 1: return LAUNCH(32, 32, 16, 4, 2, 3, 4);
    default: return LAUNCH(16, 16, 16, 2, 2, 3, 4);
    }
#undef LAUNCH
}

}  // namespace iclb
