// TRSV: solve op(A) x = b in place (x holds b on entry), float and complex,
// op in {N, T, C}, upper/lower, unit/non-unit.
//
// Replaces Strsv_simd16x16_* (one work-group of 256 serialising every
// 16-column block with barriers) and the serial Strsv_naive / Ctrsv_naive
// (libs/blas/funcs/Strsv/*, Ctrsv/*).  One launch covers the whole solve: the
// n rows are cut into blocks, one CTA per block; the CTAs draw tickets from
// an atomic counter and own blocks in solve order (forward for a lower
// op(A), backward for an upper one), so a CTA only ever waits for CTAs that
// are already running.  Two kernels share that structure, and solves of up to
// 128 rows are one CTA's substitution (trsv_small_kernel):
//   - strsv_tma_kernel: long real solves that TMA can address, 128-row blocks;
//   - trsv_block_kernel: everything else (complex data, short solves, any
//     base address and leading dimension), 64-row blocks fetched element by
//     element.
// Every wait is bounded: a CTA that gives up records kDevWaitTimeout in the
// device status word and returns, and so do the CTAs that wait for it; the
// host reports EXECUTION_FAILED.
#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cstddef>
#include <type_traits>

#include "common.cuh"
#include "tma.cuh"

namespace iclb {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float zero_v(float) { return 0.f; }
__device__ __forceinline__ cfloat zero_v(cfloat) { return cfloat{0.f, 0.f}; }
__device__ __forceinline__ float conj_v(float v) { return v; }
__device__ __forceinline__ cfloat conj_v(cfloat v) { return cfloat{v.re, -v.im}; }
__device__ __forceinline__ float ldg(const float* p) { return __ldg(p); }
__device__ __forceinline__ cfloat ldg(const cfloat* p)
{
    float2 v = __ldg((const float2*)p);
    return cfloat{v.x, v.y};
}
__device__ __forceinline__ void msub(float& acc, float a, float x) { acc = fmaf(-a, x, acc); }
__device__ __forceinline__ void msub(cfloat& acc, cfloat a, cfloat x)
{
    acc.re = fmaf(-a.re, x.re, acc.re);
    acc.re = fmaf(a.im, x.im, acc.re);
    acc.im = fmaf(-a.re, x.im, acc.im);
    acc.im = fmaf(-a.im, x.re, acc.im);
}
__device__ __forceinline__ float addv(float a, float b) { return a + b; }
__device__ __forceinline__ cfloat addv(cfloat a, cfloat b) { return cfloat{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ float subv(float a, float b) { return a - b; }
__device__ __forceinline__ cfloat subv(cfloat a, cfloat b) { return cfloat{a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ float shfl(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ cfloat shfl(cfloat v, int src)
{
    return cfloat{__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
}

__device__ __forceinline__ int ld_volatile(const int* p) { return *(const volatile int*)p; }

// ---------------------------------------------------------------- substitution
__device__ __forceinline__ float abs_max(float v) { return fabsf(v); }
__device__ __forceinline__ float abs_max(cfloat v) { return fmaxf(fabsf(v.re), fabsf(v.im)); }
__device__ __forceinline__ float quot(float a, float d) { return a / d; }
// complex quotient through |d|^2 (the reference's cdiv, core/src/ocl/complex.h.cl:36),
// in FP64, whose range no square of an FP32 number leaves
__device__ __forceinline__ cfloat quot(cfloat a, cfloat d)
{
    const double re = d.re, im = d.im, q = 1.0 / fma(re, re, im * im);
    return cfloat{(float)(fma((double)a.re, re, a.im * im) * q), (float)(fma((double)a.im, re, -(double)a.re * im) * q)};
}
// 1 / d as hi + lo
__device__ __forceinline__ void recip(float d, float& hi, float& lo)
{
    const double w = 1.0 / d;
    hi = (float)w;
    lo = (float)(w - (double)hi);
}
__device__ __forceinline__ void recip(cfloat d, cfloat& hi, cfloat& lo)
{
    const double re = d.re, im = d.im, q = 1.0 / fma(re, re, im * im);
    hi = cfloat{(float)(re * q), (float)(-im * q)};
    lo = cfloat{(float)(re * q - (double)hi.re), (float)(-im * q - (double)hi.im)};
}
// v / d for 1 / d = hi + lo, right to less than a rounding where nothing
// leaves the normal range; an infinite v as hi alone has it (lo may be zero or
// of the other sign)
__device__ __forceinline__ float finite_or_0(float v) { return isfinite(v) ? v : 0.f; }
__device__ __forceinline__ float times(float v, float hi, float lo) { return fmaf(v, hi, finite_or_0(v * lo)); }
__device__ __forceinline__ cfloat times(cfloat v, cfloat hi, cfloat lo)
{
    const float re = finite_or_0(fmaf(v.re, lo.re, -v.im * lo.im)), im = finite_or_0(fmaf(v.re, lo.im, v.im * lo.re));
    return cfloat{fmaf(v.re, hi.re, fmaf(-v.im, hi.im, re)), fmaf(v.re, hi.im, fmaf(v.im, hi.re, im))};
}

// One warp solves the nr x nr lower triangle with element (r, k) at
// D[r * sr + k * sc] (shared memory, sr odd) in place of v: lane l holds rows
// l + 32 q, those past nr anything.  (An upper triangle is a lower one with rows
// and columns in reverse order.)  Bound by the chain of nr steps, each a
// quotient, a shuffle and an update; so that no division lies in it, the
// diagonal's reciprocals are formed first, as two floats each, wherever they
// are in range.
template <class T, int R, bool FAST>
__device__ __forceinline__ void substitute_steps(const T* D, int sr, int sc, int nr, bool unit, const T (&hi)[R],
                                                 const T (&lo)[R], T (&v)[R])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int steps = min(32, nr - 32 * q);
#pragma unroll 1
        for (int l = 0; l < steps; ++l) {
            T x = v[q];
            if (!unit) x = FAST ? times(x, hi[q], lo[q]) : quot(x, hi[q]);
            x = shfl(x, l);
            if (lane == l) v[q] = x;
#pragma unroll
            for (int p = q; p < R; ++p)
                if ((p > q || lane > l) && lane + 32 * p < nr)
                    msub(v[p], D[(lane + 32 * p) * sr + (l + 32 * q) * sc], x);
        }
    }
}
template <class T, int R>
__device__ __forceinline__ void substitute(const T* D, int sr, int sc, int nr, bool unit, T (&v)[R])
{
    const int lane = threadIdx.x & 31;
    T hi[R], lo[R];
    bool fast = true;
#pragma unroll
    for (int q = 0; q < R; ++q) {
        hi[q] = lo[q] = zero_v(T());
        if (unit || lane + 32 * q >= nr) continue;
        hi[q] = D[(lane + 32 * q) * (sr + sc)];
        fast = fast && abs_max(hi[q]) >= 0x1p-100f && abs_max(hi[q]) <= 0x1p100f;
    }
    if (__all_sync(0xffffffffu, fast)) {
#pragma unroll
        for (int q = 0; q < R; ++q)
            if (!unit) recip(hi[q], hi[q], lo[q]);
        substitute_steps<T, R, true>(D, sr, sc, nr, unit, hi, lo, v);
    } else {
        substitute_steps<T, R, false>(D, sr, sc, nr, unit, hi, lo, v);
    }
}

// Solves of up to kSmall rows, a CTA: the triangle goes to shared memory, the
// first warp substitutes.  R: rows of a lane.
// Measured in one run (us, 64-row block kernel and this one): real n = 1 8.2,
// 2.2, n = 64 12.3, 6.1, n = 96 13.9, 11.6, n = 128 13.9, 14.0; complex n = 1
// 12.5, 2.3, n = 64 17.0, 6.7, n = 128 18.8, 15.9.  The line: at 128 real rows
// the two are level, and the substitution grows by the row, the blocks do not
// (n = 129 14.4 and 19.2 there).
constexpr int kSmall = 128;
template <class T, int R>
__global__ void __launch_bounds__(kThreads) trsv_small_kernel(int n, int lower_op, int op, int unit,
                                                              const T* __restrict__ A, long lda, T* x, long incx)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* const D = reinterpret_cast<T*>(smem_raw);
    const int P = n | 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // consecutive lanes read consecutive addresses, rows of a column of A; a
    // lane's elements of 8 columns are in flight at once (one column at a time
    // n = 65 took 15 us)
    const bool lower_a = (op == 0) == (lower_op != 0);
    for (int c0 = warp; c0 < n; c0 += 8 * (kThreads / 32)) {
        T e[8][R];
        auto in = [&](int r, int c) { return r < n && c < n && (lower_a ? r >= c : r <= c); };
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int r = lane + 32 * q, c = c0 + u * (kThreads / 32);
                e[u][q] = in(r, c) ? A[(long)c * lda + r] : zero_v(T());
            }
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int r = lane + 32 * q, c = c0 + u * (kThreads / 32);  // (r, c) of A, (r, c) or (c, r) of op(A)
                if (in(r, c)) D[op == 0 ? r * P + c : c * P + r] = op == 2 ? conj_v(e[u][q]) : e[u][q];
            }
    }
    T v[R];
    auto row = [&](int q) { return lower_op ? lane + 32 * q : n - 1 - lane - 32 * q; };
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = warp == 0 && lane + 32 * q < n ? x[(long)row(q) * incx] : zero_v(T());
    __syncthreads();
    if (warp != 0) return;
    const int sg = lower_op ? 1 : -1;
    substitute<T, R>(lower_op ? D : D + (n - 1) * (P + 1), sg * P, sg, n, unit != 0, v);
#pragma unroll
    for (int q = 0; q < R; ++q)
        if (lane + 32 * q < n) x[(long)row(q) * incx] = v[q];
}

// ---------------------------------------------------------------- STRSV, TMA path
// Float TRSV when A is 16-byte aligned with lda a multiple of 4 and >= n
// (the usual case).  The ticket-ordered one-launch structure, with
// blocks of RB = 128 rows, one CTA of 256 threads per block (one CTA per SM),
// and changes that shorten the chain of dependent block solves:
//   - tiles arrive by TMA (boxes of 128 rows x 64 columns of op(A), half a
//     block's columns each) into a 6-stage shared-memory ring, so 192 KiB per
//     CTA are in flight while the CTA waits for earlier blocks;
//   - the first two boxes are the diagonal block D, inverted in FP64: both
//     64 x 64 diagonal halves at once (16 x 16 blocks by substitution, then
//     two doubling steps), then the off-diagonal half from those two
//     (-inv(D22) D21 inv(D11) for a lower D), each product register-tiled.
//     The inverse is kept in FP32 in registers: each thread holds 4 rows x
//     16 columns, so a product with a vector takes 4 16-byte shared-memory
//     reads per thread (not 64 broadcast words: 8 warps reading a vector
//     word by word spend the SM's shared-memory bandwidth) and a butterfly
//     over the 8 lanes sharing the rows.  The FP64 workspace overlays the
//     ring before the ring is used;
//   - the next two boxes are the tile T next to D (the block solved just
//     before this one), kept in registers in the same layout; then the
//     remaining tiles in solve order, consumed with 16-byte reads along the
//     stage's contiguous direction into per-thread partial row sums.  Once
//     all but the last earlier block are known, the CTA holds
//     y = b - (sum of those tiles' products), so its own step of the chain,
//     when the last block x_prev is published, is x = inv(D) (y - T x_prev):
//     two register products with one barrier between them, and the
//     publication;
//   - each solved entry is published as one 64-bit word (value, call epoch):
//     a consumer polls the entries it needs directly, with no separate flag.
//     The epoch lives in device memory: each CTA reads the last launch's
//     epoch at its start and uses the next one; the CTA that solves the last
//     block stores it back once everything is published (every other CTA has
//     read it by then), so replays of a captured launch get fresh epochs;
//   - launched as clusters of CL consecutive blocks, a solved block also goes
//     straight into the shared memory of the later CTAs of its cluster
//     (st.async on a transaction barrier), so CL - 1 of every CL steps of the
//     chain skip the global-memory round trip.  CL is the largest size from
//     8 down to 2 for which the GPU holds every cluster of the launch at once
//     (a cluster that can only start when another has finished starts its
//     own setup late and then streams its tiles alone).
// Against 64-row blocks (two CTAs per SM, n = 16384 in 230 us) the chain has
// half the steps and half the hand-offs between clusters.
constexpr int RB = 128;  // rows (and columns) of a block
constexpr int HB = 64;   // columns of op(A) in one stage
constexpr int STAGE_ELEMS = RB * HB;
constexpr int FS = 6;
constexpr int kMaxCluster = 8;
constexpr int XQ = 8 * 20;  // a block's 128 entries in shared memory: 8 groups of 16, 20 floats apart
constexpr unsigned long long kTrsvWaitNs = 2000000000ull;  // a wait gives up after 2 s

// shared-memory index of entry c (0 .. 127) of a block's entries (the
// padding keeps the 16-byte reads of 8 threads with different groups in
// different banks)
__device__ __forceinline__ int qidx(int c) { return (c >> 4) * 20 + (c & 15); }

// FP64 workspace of the diagonal-block inverse, in doubles: the inverses of
// the two 64 x 64 diagonal halves, the off-diagonal half, and two doubling
// temporaries.  It starts at stage 2 of the ring.
constexpr int kY = HB * (HB + 1);
constexpr int kTm = 32 * 33;
constexpr int kInvDoubles = 3 * kY + 2 * kTm;
static_assert(kInvDoubles * 8 <= (FS - 2) * STAGE_ELEMS * 4, "inverse workspace inside the ring");

struct FastSmem {
    float stage[FS][STAGE_ELEMS];
    // cluster launches: the solved blocks of the earlier CTAs of this
    // cluster, delivered into this CTA's shared memory by st.async, one
    // transaction barrier per source rank
    float xin[kMaxCluster][XQ];
    float xs[XQ];  // entries of the block being streamed, from the published words
    float xp[XQ];  // x_prev, from the published words
    float y[XQ];   // b - the products of the tiles of blocks 0 .. s-2
    float y2[XQ];  // y - T x_prev
    float part[16][RB];  // partial row sums of the streamed tiles
    uint64_t xbar[kMaxCluster];
    uint64_t full[FS];
    unsigned s, epoch, cl;
    int failed;  // a wait of the chain step gave up
};
static_assert(sizeof(FastSmem) + 1024 <= 232448, "STRSV shared memory");
static_assert(offsetof(FastSmem, xin) % 16 == 0 && offsetof(FastSmem, xs) % 16 == 0 &&
                  offsetof(FastSmem, xp) % 16 == 0 && offsetof(FastSmem, y) % 16 == 0 &&
                  offsetof(FastSmem, y2) % 16 == 0,
              "16-byte reads of block entries");

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// ---- thread-block-cluster helpers (distributed shared memory)
__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// this CTA's shared address `a` as seen in the shared memory of CTA `rank`
__device__ __forceinline__ uint32_t map_to(const void* a, unsigned rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(tma::smem_u32(a)), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, unsigned v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// 16 bytes into another CTA's shared memory (16-byte aligned), counted as
// transaction bytes on that CTA's barrier
__device__ __forceinline__ void st_async_f32x4(uint32_t addr, float a, float b, float c, float d, uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     addr),
                 "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// bounded wait, acquiring at cluster scope (the bytes come from another CTA)
__device__ __forceinline__ bool xbar_wait_bounded(uint64_t* bar, unsigned long long limit_ns)
{
    auto try_once = [&]() {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(tma::smem_u32(bar))
            : "memory");
        return ok != 0;
    };
    if (try_once()) return true;
    const unsigned long long t0 = tma::global_ns();
    while (!try_once())
        if (tma::global_ns() - t0 > limit_ns) return false;
    return true;
}
// polls a published (value, epoch) word until it carries `epoch`; false when
// the wait gives up or another CTA has recorded a failure
__device__ __forceinline__ bool poll_word(const unsigned long long* src, unsigned epoch, const int* status,
                                          float& v)
{
    unsigned long long w = ld_relaxed_u64(src);
    if ((unsigned)(w >> 32) != epoch) {
        const unsigned long long t0 = tma::global_ns();
        // the status word is read on one poll in 64: its load would double
        // the time between two looks at the entry
        for (unsigned it = 1;; ++it) {
            w = ld_relaxed_u64(src);
            if ((unsigned)(w >> 32) == epoch) break;
            if ((it & 63) == 0 && (ld_volatile(status) != kDevOk || tma::global_ns() - t0 > kTrsvWaitNs)) return false;
        }
    }
    v = __uint_as_float((unsigned)w);
    return true;
}

// FP64 product tile of the diagonal-block inverse: acc(i, j) = sum_k A(r, k)
// B(k, c) for rows r = r0 + i*rs and columns c = c0 + j*cs (interleaved, so
// that a warp reads consecutive columns of B and few rows of A)
template <int TR, int TC, int K, class FA, class FB>
__device__ __forceinline__ void dtile(double (&acc)[TR][TC], int r0, int rs, int c0, int cs, FA A, FB B)
{
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) acc[i][j] = 0.0;
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
        double a[TR], b[TC];
#pragma unroll
        for (int i = 0; i < TR; ++i) a[i] = A(r0 + i * rs, k);
#pragma unroll
        for (int j = 0; j < TC; ++j) b[j] = B(k, c0 + j * cs);
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
}

// CL = 1: one CTA per block, every solved block handed on through global
// memory.  CL > 1 (a cluster launch): the CTAs of a cluster solve CL
// consecutive blocks and hand each solved block to the later CTAs of the
// cluster directly into their shared memory (st.async, completed on a
// transaction barrier), so CL - 1 of every CL steps of the chain skip the
// global-memory round trip; blocks of earlier clusters still come from the
// published words.  Every CTA of a cluster arrives at a final cluster
// barrier before it exits, so no CTA leaves while another may still write
// into its shared memory.
template <int CL>
__global__ void __launch_bounds__(kThreads, 1)
    strsv_tma_kernel(const __grid_constant__ CUtensorMap amap, int n, int lower_op, int op, int unit, float* x,
                     long incx, unsigned long long* pub, unsigned* ticket, unsigned* epoch_word, int* status)
{
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte aligned; an offset from the array (not an integer cast) keeps
    // the accesses in the shared address space
    FastSmem& S = *reinterpret_cast<FastSmem*>(smem_raw + ((1024u - (tma::smem_u32(smem_raw) & 1023u)) & 1023u));
    const int t = threadIdx.x;
    const int nb = (n + RB - 1) / RB;
    const unsigned rank = CL > 1 ? cluster_rank() : 0u;
    if (t == 0) {
        unsigned e = *(volatile unsigned*)epoch_word + 1u;
        S.epoch = e == 0u ? 1u : e;
        if (CL == 1) S.s = atomicAdd(ticket, 1u);
        for (int i = 0; i < FS; ++i) tma::mbar_init(&S.full[i], 1);
        S.failed = 0;
        if constexpr (CL > 1) {
            // one arrival (this one, declaring the bytes) plus RB floats per earlier rank
            for (unsigned r = 0; r < (unsigned)CL; ++r) tma::mbar_init(&S.xbar[r], 1);
            tma::mbar_init_fence();
            for (unsigned r = 0; r < rank; ++r) tma::mbar_expect_tx(&S.xbar[r], RB * 4);
        } else {
            tma::mbar_init_fence();
        }
    }
    if constexpr (CL > 1) {
        // every CTA of the cluster has started and set up its barriers before
        // any shared memory of another CTA is written
        __syncthreads();
        cluster_sync_all();
        if (rank == 0 && t == 0) {
            const unsigned c = atomicAdd(ticket, 1u);
            for (unsigned r = 0; r < (unsigned)CL; ++r) st_cluster_u32(map_to(&S.cl, r), c);
            if (c == gridDim.x / CL - 1) *ticket = 0u;  // every ticket of this launch is taken
        }
        cluster_sync_all();
        if (t == 0) S.s = S.cl * CL + rank;
    }
    __syncthreads();
    const int s = (int)S.s;
    const unsigned epoch = S.epoch;
    const int cfirst = CL > 1 ? (int)S.cl * CL : 0;  // first block (solve order) of this cluster
    if (CL == 1 && s == nb - 1 && t == 0) *ticket = 0u;  // every ticket of this launch is taken
    if (CL > 1 && s >= nb) {  // a cluster's spare CTA past the last block
        cluster_sync_all();
        return;
    }
    auto blk = [&](int p) { return lower_op ? p : nb - 1 - p; };
    const int kb = blk(s), r0 = kb * RB, nr = min(RB, n - r0);
    // loads, numbered: 0 and 1 the two halves of D; 2 and 3 the halves of the
    // tile of block s-1 (s >= 1); then 4 + 2i + h half h of the tile of block
    // i, i = 0 .. s-2 in solve order.  Load L goes to stage L % FS and
    // completes phase L / FS of that stage's barrier; it is issued once load
    // L - FS has been consumed.
    const int nloads = s == 0 ? 2 : 4 + 2 * (s - 1);
    int issued = 0;  // (thread 0)
    auto issue = [&](int L) {
        issued = L + 1;
        const int cb = L < 2 ? kb : (L < 4 ? blk(s - 1) : blk((L - 4) >> 1));
        const int c = cb * RB + (L & 1) * HB;
        uint64_t* bar = &S.full[L % FS];
        tma::mbar_expect_tx(bar, STAGE_ELEMS * 4);
        if (op == 0) tma::load_2d(S.stage[L % FS], &amap, r0, c, bar);  // A[r0 .. +127, c .. +63]
        else tma::load_2d(S.stage[L % FS], &amap, c, r0, bar);          // A[c .. +63, r0 .. +127]
    };
    auto wait_load = [&](int L) { return tma::mbar_wait_bounded(&S.full[L % FS], (L / FS) & 1, kTrsvWaitNs); };
    if (t == 0) {
        issue(0);
        issue(1);
        // the tiles needed first after the inverse (block s-1's, then block
        // 0's) start towards L2 now, while the inverse is formed
        for (int L = 2; L < min(6, nloads); ++L) {
            const int cb = L < 4 ? blk(s - 1) : blk(0);
            const int c = cb * RB + (L & 1) * HB;
            if (op == 0) tma::prefetch_2d(&amap, r0, c);
            else tma::prefetch_2d(&amap, c, r0);
        }
    }
    const float b = (t < nr) ? x[(long)(r0 + t) * incx] : 0.f;  // (threads t < RB)
    // on a failed wait: record it, let this CTA's copies still in flight land
    // (each wait bounded), then leave
    auto bail = [&](int consumed) {
        if (t == 0) {
            atomicOr(status, (int)kDevWaitTimeout);
            for (int L = consumed; L < issued; ++L) wait_load(L);
            // bytes other CTAs of the cluster may still be sending here
            if constexpr (CL > 1)
                for (unsigned r = 0; r < rank; ++r) xbar_wait_bounded(&S.xbar[r], kTrsvWaitNs);
        }
        if constexpr (CL > 1) {
            __syncthreads();
            cluster_sync_all();
        }
    };
    // the solved entries of the block with solve index p: this CTA's own
    // shared memory when an earlier CTA of the cluster solved it (every
    // thread waits on the transaction barrier), else the published words
    // (threads t < RB poll, into `buf`; the caller's barrier publishes them)
    auto fetch_x = [&](int p, float* buf, int& bad) -> const float* {
        if (CL > 1 && p >= cfirst) {
            if (!xbar_wait_bounded(&S.xbar[p - cfirst], kTrsvWaitNs)) {
                atomicOr(status, (int)kDevWaitTimeout);
                bad = 1;
            }
            return S.xin[p - cfirst];
        }
        const int c0 = blk(p) * RB, nc = min(RB, n - c0);
        if (t < RB) {
            float v = 0.f;
            if (t < nc && !poll_word(pub + c0 + t, epoch, status, v)) {
                atomicOr(status, (int)kDevWaitTimeout);
                bad = 1;
            }
            buf[qidx(t)] = v;
        }
        return buf;
    };
    // op(A) element (r, c) of a stage: r < 128, c < 64
    auto el = [&](const float* T, int r, int c) { return op == 0 ? T[c * RB + r] : T[r * HB + c]; };
    // register layout of a 128 x 128 matrix (inv(D), and the tile of block
    // s-1): the thread holds rows R0 .. R0+3, columns cg*16 .. cg*16+15
    const int lane = t & 31, warp = t >> 5;
    const int cg = lane & 7, R0 = warp * 16 + (lane >> 3) * 4;
    // out[k] = row R0+k of M times v (v in the block-entry layout), in every
    // lane of the 8 that share the rows: 4 16-byte reads, 64 FMAs, and a
    // butterfly over the column groups
    auto mv = [&](const float(&m)[4][16], const float* v, float(&out)[4]) {
        const float* vp = v + cg * 20;
        float4 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4*>(vp + 4 * i);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float a0 = 0.f, a1 = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a0 = fmaf(m[k][4 * i], q[i].x, a0);
                a1 = fmaf(m[k][4 * i + 1], q[i].y, a1);
                a0 = fmaf(m[k][4 * i + 2], q[i].z, a0);
                a1 = fmaf(m[k][4 * i + 3], q[i].w, a1);
            }
            out[k] = a0 + a1;
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < 4; ++k) out[k] += __shfl_xor_sync(0xffffffffu, out[k], o);
    };
    auto pick = [](const float(&o)[4], int k) { return k == 0 ? o[0] : (k == 1 ? o[1] : (k == 2 ? o[2] : o[3])); };

    // ---- diagonal block: FP64 inverse, kept in FP32 registers
    int bad = (wait_load(0) && wait_load(1)) ? 0 : 1;
    if (__syncthreads_or(bad)) {
        bail(0);
        return;
    }
    float iv[4][16];  // inv(D)[R0 + k][cg*16 + j]
    {
        double* ws = reinterpret_cast<double*>(&S.stage[2][0]);
        double(*Y)[HB][HB + 1] = reinterpret_cast<double(*)[HB][HB + 1]>(ws);   // inverses of D11, D22
        double(*Yc)[HB + 1] = reinterpret_cast<double(*)[HB + 1]>(ws + 2 * kY);  // the off-diagonal half
        double(*Tm)[32][33] = reinterpret_cast<double(*)[32][33]>(ws + 3 * kY);  // doubling temporaries
        // element (r, c) of D, r, c < 128; rows and columns past nr are zero (box fill)
        auto d = [&](int r, int c) -> double { return (double)el(S.stage[c >> 6], r, c & (HB - 1)); };
        double* rd = &Tm[0][0][0];  // 1 / diagonal, until the doubling steps use Tm
        for (int idx = t; idx < 2 * kY; idx += kThreads) (&Y[0][0][0])[idx] = 0.0;
        if (t < RB) rd[t] = (unit || t >= nr) ? 1.0 : 1.0 / d(t, t);
        __syncthreads();
        if (t < RB) {
            // thread t owns column j of the 16 x 16 diagonal block at b of
            // half hb; the column stays in registers
            const int hb = t >> 6, b = ((t & (HB - 1)) >> 4) * 16, j = t & 15, o = hb * HB + b;
            double y[16];
            if (lower_op) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    double acc = (i == j) ? 1.0 : 0.0;
#pragma unroll
                    for (int k = 0; k < i; ++k) acc = fma(-d(o + i, o + k), y[k], acc);
                    y[i] = (i >= j) ? acc * rd[o + i] : 0.0;
                }
            } else {
#pragma unroll
                for (int i = 15; i >= 0; --i) {
                    double acc = (i == j) ? 1.0 : 0.0;
#pragma unroll
                    for (int k = i + 1; k < 16; ++k) acc = fma(-d(o + i, o + k), y[k], acc);
                    y[i] = (i <= j) ? acc * rd[o + i] : 0.0;
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) Y[hb][b + i][b + j] = y[i];
        }
        __syncthreads();
        // doubling inside both halves at once (h = 16, then 32): the
        // off-diagonal h x h block of each 2h x 2h diagonal block is
        // -Y22 C Y11 (lower: C below Y11) or -Y11 C Y22 (upper: C right of
        // Y11).  64 / h products of h x h at a time, a TR x TC tile per thread
        auto doubling = [&](auto hc) {
            constexpr int h = decltype(hc)::value;
            constexpr int G = 64 / h, TPG = kThreads / G;  // products, threads per product
            constexpr int TR = 2, TC = h / 8, RS = h / TR;  // 8 thread columns, RS thread rows
            const int gid = t / TPG, u = t % TPG, hb = gid / (G / 2), pr = gid % (G / 2);
            const int ob = hb * HB, o = pr * 2 * h, tr = u / 8, tcl = u % 8;
            double acc[TR][TC];
            if (lower_op)
                dtile<TR, TC, h>(
                    acc, tr, RS, tcl, 8, [&](int r, int k) { return d(ob + o + h + r, ob + o + k); },
                    [&](int k, int c) { return Y[hb][o + k][o + c]; });
            else
                dtile<TR, TC, h>(
                    acc, tr, RS, tcl, 8, [&](int r, int k) { return d(ob + o + r, ob + o + h + k); },
                    [&](int k, int c) { return Y[hb][o + h + k][o + h + c]; });
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) Tm[hb][pr * h + tr + i * RS][tcl + 8 * j] = acc[i][j];
            __syncthreads();
            if (lower_op)
                dtile<TR, TC, h>(
                    acc, tr, RS, tcl, 8, [&](int r, int k) { return Y[hb][o + h + r][o + h + k]; },
                    [&](int k, int c) { return Tm[hb][pr * h + k][c]; });
            else
                dtile<TR, TC, h>(
                    acc, tr, RS, tcl, 8, [&](int r, int k) { return Y[hb][o + r][o + k]; },
                    [&](int k, int c) { return Tm[hb][pr * h + k][c]; });
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) {
                    const int r = tr + i * RS, c = tcl + 8 * j;
                    if (lower_op) Y[hb][o + h + r][o + c] = -acc[i][j];
                    else Y[hb][o + r][o + h + c] = -acc[i][j];
                }
            __syncthreads();
        };
        doubling(std::integral_constant<int, 16>{});
        doubling(std::integral_constant<int, 32>{});
        // the off-diagonal half: lower D: -inv(D22) (D21 inv(D11)); upper D:
        // -inv(D11) (D12 inv(D22)); 4 x 4 outputs per thread
        {
            const int tr = t / 16, tcl = t % 16;
            double acc[4][4];
            if (lower_op)
                dtile<4, 4, HB>(
                    acc, tr, 16, tcl, 16, [&](int r, int k) { return d(HB + r, k); },
                    [&](int k, int c) { return Y[0][k][c]; });
            else
                dtile<4, 4, HB>(
                    acc, tr, 16, tcl, 16, [&](int r, int k) { return d(r, HB + k); },
                    [&](int k, int c) { return Y[1][k][c]; });
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) Yc[tr + 16 * i][tcl + 16 * j] = acc[i][j];
            __syncthreads();
            const int yl = lower_op ? 1 : 0;
            dtile<4, 4, HB>(
                acc, tr, 16, tcl, 16, [&](int r, int k) { return Y[yl][r][k]; },
                [&](int k, int c) { return Yc[k][c]; });
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) Yc[tr + 16 * i][tcl + 16 * j] = -acc[i][j];
        }
        __syncthreads();
        // the inverse in FP32, row-major through stages 0 and 1 (16-byte word
        // f of row R at f ^ ((f >> 2) & 7)), then each thread's 4 x 16 block
        // from it: neither pass has bank conflicts (reading the FP64 pieces
        // straight into the register layout had 8-way conflicts and took 3 us).
        // Rows and columns past nr are cut off.
        {
            float4* Iv = reinterpret_cast<float4*>(&S.stage[0][0]);
            for (int idx = t; idx < RB * 32; idx += kThreads) {
                const int R = idx >> 5, f = idx & 31, C = 4 * f, rr = R & (HB - 1);
                const bool right = C >= HB;  // columns 64 .. 127
                const double* src;           // row R of the 64 x 64 piece holding the columns
                if (lower_op) src = R < HB ? (right ? nullptr : Y[0][rr]) : (right ? Y[1][rr] : Yc[rr]);
                else src = R < HB ? (right ? Yc[rr] : Y[0][rr]) : (right ? Y[1][rr] : nullptr);
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    v[e] = (src != nullptr && R < nr && C + e < nr) ? (float)src[(C + e) & (HB - 1)] : 0.f;
                Iv[R * 32 + (f ^ (f >> 2 & 7))] = make_float4(v[0], v[1], v[2], v[3]);
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 v = Iv[(R0 + k) * 32 + ((cg * 4 + q) ^ cg)];
                    iv[k][4 * q] = v.x;
                    iv[k][4 * q + 1] = v.y;
                    iv[k][4 * q + 2] = v.z;
                    iv[k][4 * q + 3] = v.w;
                }
        }
        // D (stages 0, 1) and the FP64 workspace (stages 2 on) are free; the
        // stores to them come before the copies that reuse the stages
        tma::fence_proxy_async_smem();
        __syncthreads();
    }
    if (t == 0)
        for (int L = 2; L < min(2 + FS, nloads); ++L) issue(L);

    // ---- the tile T of block s-1, kept in registers in the same layout
    float tc[4][16];
    if (s >= 1) {
        bad = (wait_load(2) && wait_load(3)) ? 0 : 1;
        if (__syncthreads_or(bad)) {
            bail(2);
            return;
        }
        const float* T = S.stage[2 + (cg >> 2)];
        const int c0 = (cg & 3) * 16;  // first column inside the stage
        if (op == 0) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float4 v = *reinterpret_cast<const float4*>(&T[(c0 + j) * RB + R0]);
                tc[0][j] = v.x;
                tc[1][j] = v.y;
                tc[2][j] = v.z;
                tc[3][j] = v.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 v = *reinterpret_cast<const float4*>(&T[(R0 + k) * HB + c0 + 4 * q]);
                    tc[k][4 * q] = v.x;
                    tc[k][4 * q + 1] = v.y;
                    tc[k][4 * q + 2] = v.z;
                    tc[k][4 * q + 3] = v.w;
                }
        }
        // the registers are not read until the chain step: the reads of
        // stages 2 and 3 must be complete before the copies that reuse them
        tma::fence_proxy_async_smem();
        __syncthreads();
        if (t == 0)
            for (int L = 2 + FS; L < min(4 + FS, nloads); ++L) issue(L);
    }

    // ---- the other earlier blocks, in solve order: y = b - their products.
    // Each thread keeps partial row sums in registers; 16-byte reads run
    // along the stage's contiguous direction.
    //   op N (stage column-major): rows 4*lane .. +3, columns warp*8 .. +7
    //   op T (stage row-major): rows (2*warp + lane/16)*8 .. +7, columns
    //   4*(lane%16) .. +3
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    for (int i = 0; i + 1 < s; ++i) {
        bad = 0;
        const float* xv = fetch_x(i, S.xs, bad);
        for (int hh = 0; hh < 2; ++hh) {
            const int L = 4 + 2 * i + hh;
            if (!wait_load(L)) bad = 1;
            if (__syncthreads_or(bad)) {
                bail(L);
                return;
            }
            const float* T = S.stage[L % FS];
            if (op == 0) {
                const int c0 = warp * 8;
                const float* xq = xv + qidx(hh * HB + c0);
                const float4 xa = *reinterpret_cast<const float4*>(xq);
                const float4 xb = *reinterpret_cast<const float4*>(xq + 4);
                const float xk[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float4 v = *reinterpret_cast<const float4*>(&T[(c0 + k) * RB + 4 * lane]);
                    acc[0] = fmaf(-v.x, xk[k], acc[0]);
                    acc[1] = fmaf(-v.y, xk[k], acc[1]);
                    acc[2] = fmaf(-v.z, xk[k], acc[2]);
                    acc[3] = fmaf(-v.w, xk[k], acc[3]);
                }
            } else {
                const int cq = lane & 15, rb = (2 * warp + (lane >> 4)) * 8;
                const float4 xa = *reinterpret_cast<const float4*>(xv + qidx(hh * HB + 4 * cq));
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float4 v = *reinterpret_cast<const float4*>(&T[(rb + k) * HB + 4 * cq]);
                    acc[k] = fmaf(-v.x, xa.x, acc[k]);
                    acc[k] = fmaf(-v.y, xa.y, acc[k]);
                    acc[k] = fmaf(-v.z, xa.z, acc[k]);
                    acc[k] = fmaf(-v.w, xa.w, acc[k]);
                }
            }
            __syncthreads();
            if (t == 0 && L + FS < nloads) issue(L + FS);
        }
    }
    if (op == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) S.part[warp][4 * lane + k] = acc[k];
    } else {
        const int cq = lane & 15, rb = (2 * warp + (lane >> 4)) * 8;
#pragma unroll
        for (int k = 0; k < 8; ++k) S.part[cq][rb + k] = acc[k];
    }
    __syncthreads();
    if (t < RB) {
        float sum = 0.f;
        const int np = op == 0 ? 8 : 16;
        for (int p = 0; p < np; ++p) sum += S.part[p][t];
        S.y[qidx(t)] = t < nr ? b + sum : 0.f;
    }
    __syncthreads();

    // ---- this block's step of the chain: x = inv(D) (y - T x_prev).  From
    // the arrival of x_prev to the hand-off of x: two register products and
    // one barrier (one more on the global path, after the polls)
    bool ok = true;
    float o[4];
    const int own = cg & 3, row = R0 + own;  // the row this lane publishes
    // hand-off: lane 4 + d sends rows R0 .. R0+3 to the later CTAs rank + 1 + d
    // and rank + 5 + d of the cluster (those that have blocks), 16 bytes
    // each; the remote addresses are formed here, off the critical path
    int ndst = 0;
    uint32_t dx0 = 0, db0 = 0, dx1 = 0, db1 = 0;
    if constexpr (CL > 1) {
        if (cg >= 4) {
            const unsigned d0 = rank + 1u + (unsigned)(cg - 4), d1 = d0 + 4u;
            if (d0 < (unsigned)CL && cfirst + (int)d0 < nb) {
                dx0 = map_to(&S.xin[rank][qidx(R0)], d0);
                db0 = map_to(&S.xbar[rank], d0);
                ndst = 1;
                if (d1 < (unsigned)CL && cfirst + (int)d1 < nb) {
                    dx1 = map_to(&S.xin[rank][qidx(R0)], d1);
                    db1 = map_to(&S.xbar[rank], d1);
                    ndst = 2;
                }
            }
        }
    }
    if (s >= 1) {
        const int p = s - 1;
        const float* xpv;
        if (CL > 1 && p >= cfirst) {
            ok = __all_sync(0xffffffffu, xbar_wait_bounded(&S.xbar[p - cfirst], kTrsvWaitNs));
            xpv = S.xin[p - cfirst];
        } else {
            const int c0 = blk(p) * RB, nc = min(RB, n - c0);
            if (t < RB) {
                float v = 0.f;
                if (t < nc && !poll_word(pub + c0 + t, epoch, status, v)) ok = false;
                S.xp[qidx(t)] = v;
            }
            ok = __syncthreads_and(ok);
            xpv = S.xp;
        }
        mv(tc, xpv, o);
        if (cg < 4) S.y2[qidx(row)] = S.y[qidx(row)] - pick(o, own);
    } else {
        if (cg < 4) S.y2[qidx(row)] = S.y[qidx(row)];
    }
    __syncthreads();
    mv(iv, S.y2, o);
    const float xf = pick(o, own);
    if (ok) {
        // the hand-offs first, then the published words; the output x last
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = R0 + k < nr ? o[k] : 0.f;
        // the next CTA of the cluster, which waits for them, first
        if (ndst > 0 && cg == 4) st_async_f32x4(dx0, v[0], v[1], v[2], v[3], db0);
        __syncwarp();
        if (ndst > 0 && cg != 4) st_async_f32x4(dx0, v[0], v[1], v[2], v[3], db0);
        if (ndst > 1) st_async_f32x4(dx1, v[0], v[1], v[2], v[3], db1);
        if (cg < 4 && row < nr) st_relaxed_u64(pub + r0 + row, ((unsigned long long)epoch << 32) | __float_as_uint(xf));
        if (cg < 4 && row < nr) x[(long)(r0 + row) * incx] = xf;
    } else {
        atomicOr(status, (int)kDevWaitTimeout);
        S.failed = 1;
    }
    __syncthreads();
    if (t == 0) {
        // after a failed wait, let bytes other CTAs of the cluster may still
        // send land before leaving (each wait bounded)
        if constexpr (CL > 1)
            if (S.failed)
                for (unsigned r = 0; r < rank; ++r) xbar_wait_bounded(&S.xbar[r], kTrsvWaitNs);
        if (s == nb - 1) *(volatile unsigned*)epoch_word = epoch;
    }
    if constexpr (CL > 1) cluster_sync_all();
}

// ---------------------------------------------------------------- any layout, float and complex
// 64-row blocks, 256 threads.  What bounds it is the chain of dependent block
// steps, so everything that does not depend on the previous block is done
// before that block arrives:
//   - the diagonal block is inverted in FP64 (16 x 16 blocks by substitution,
//     two doubling steps) and kept in FP32 registers, 2 rows x 8 columns a
//     thread, and so is the tile next to it;
//   - the other tiles are fetched by cp.async, element by element (4 or 8
//     bytes: any base address and leading dimension), into a 3-stage ring and
//     multiplied in the same thread layout: a thread's partial sums of all
//     tiles stay in its registers, and the 8 threads that share rows add them
//     once, together with the product of the last tile;
//   - the chain step is then two register products, x = inv(D) (y - T x_prev),
//     with one barrier between them, and solved entries travel as in
//     strsv_tma_kernel: by st.async inside a cluster, as (value, epoch) words
//     between clusters.  A thread's two rows make one remote store, and those
//     to the next CTA of the cluster, which waits for them, go first.
// A block is solved by substitution instead, as accurate as that is,
//   - when its inverse or right-hand side holds an infinity or a NaN, so that
//     those reach exactly the entries that substitution gives them to;
//   - when the largest row sum of |inv(D)| |D| is above kBGrowth: the residual
//     of a product with the inverse grows with it, substitution's does not.
//     (FP32 blocks of order 64, residual over |D| |x|, product and
//     substitution: factors of random matrices by LU, 300 to 550, 2.5e-7 and
//     9e-8, by Cholesky at condition 1e4, 620, 1.2e-7 and 7e-8; unit triangles
//     of entries up to 0.5, 750, 3.5e-7 and 1.1e-7, up to 1, 5e4 and more,
//     2.1e-5 and 9e-8; the error of x is below substitution's in all but the
//     last.)
//   - when nonzero entries of its inverse lie below FP32's normal range and
//     what they lack could show in an entry of x.
// Measured (us; before: one substitution warp per block and a flag per
// block): complex n = 3001 512, 84 to 89; n = 4096 603, 83; n = 512 78, 23;
// real with an odd leading dimension n = 4096 494, 67, n = 16384 354.  A step of
// the chain takes 0.85 us (real) or 1.15 (complex).  Measured and dropped: W = inv(D) T formed
// beforehand for a one-product step (8 us more before the chain starts, the
// step no shorter: the hand-off, not the products, sets it).
constexpr int NB = 64;
constexpr int kBStages = 3;
// CTAs of a cluster: up to 16 for solves of at most kBWide blocks (fewer
// hand-offs through global memory; us with 8 and with 16: real n = 2048 38.5,
// 37.0, 3072 52.5, 51.0, complex n = 1024 31.5, 30.1, 3072 66.8, 65.5), up to 8
// for longer ones, whose clusters of 16 wait for GPCs with 16 free SMs (real n
// = 3584 58.9, 60.5, complex 74.9, 77.0; equal from 4096 on).
constexpr int kBCluster = 16, kBWide = 48;
constexpr float kBGrowth = 1024.f;

struct alignas(16) dcomplex {
    double re, im;
};
__device__ __forceinline__ double wide(float v) { return (double)v; }
__device__ __forceinline__ dcomplex wide(cfloat v) { return dcomplex{(double)v.re, (double)v.im}; }
__device__ __forceinline__ float narrow(double v) { return (float)v; }
__device__ __forceinline__ cfloat narrow(dcomplex v) { return cfloat{(float)v.re, (float)v.im}; }
__device__ __forceinline__ void dset(double& v, double r) { v = r; }
__device__ __forceinline__ void dset(dcomplex& v, double r) { v = dcomplex{r, 0.0}; }
__device__ __forceinline__ double dneg(double v) { return -v; }
__device__ __forceinline__ dcomplex dneg(dcomplex v) { return dcomplex{-v.re, -v.im}; }
__device__ __forceinline__ void dmac(double& acc, double a, double b) { acc = fma(a, b, acc); }
__device__ __forceinline__ void dmac(dcomplex& acc, dcomplex a, dcomplex b)
{
    acc.re = fma(a.re, b.re, acc.re);
    acc.im = fma(a.re, b.im, acc.im);
    acc.re = fma(-a.im, b.im, acc.re);
    acc.im = fma(a.im, b.re, acc.im);
}
__device__ __forceinline__ double dinv(double v) { return 1.0 / v; }
__device__ __forceinline__ dcomplex dinv(dcomplex v)
{
    const double q = 1.0 / fma(v.re, v.re, v.im * v.im);
    return dcomplex{v.re * q, -v.im * q};
}
__device__ __forceinline__ double dmul(double a, double b) { return a * b; }
__device__ __forceinline__ dcomplex dmul(dcomplex a, dcomplex b)
{
    return dcomplex{fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re)};
}
__device__ __forceinline__ float abs_sum(float v) { return fabsf(v); }
__device__ __forceinline__ float abs_sum(cfloat v) { return fabsf(v.re) + fabsf(v.im); }
__device__ __forceinline__ bool is_zero(double v) { return v == 0.0; }
__device__ __forceinline__ bool is_zero(dcomplex v) { return v.re == 0.0 && v.im == 0.0; }
__device__ __forceinline__ bool finite_v(float v) { return isfinite(v); }
__device__ __forceinline__ bool finite_v(cfloat v) { return isfinite(v.re) && isfinite(v.im); }
__device__ __forceinline__ void madd_v(float& acc, float a, float x) { acc = fmaf(a, x, acc); }
__device__ __forceinline__ void madd_v(cfloat& acc, cfloat a, cfloat x)
{
    acc.re = fmaf(a.re, x.re, acc.re);
    acc.im = fmaf(a.re, x.im, acc.im);
    acc.re = fmaf(-a.im, x.im, acc.re);
    acc.im = fmaf(a.im, x.re, acc.im);
}
__device__ __forceinline__ float xor_add(float v, int o) { return v + __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ cfloat xor_add(cfloat v, int o) { return cfloat{xor_add(v.re, o), xor_add(v.im, o)}; }

template <class T>
using wide_t = decltype(wide(T()));

// A thread's 8 columns of a 64-column tile are cg + 8j (j = 0 .. 7): its
// entries of a block of x are stored next to each other, 16 bytes between the
// 8 groups, so the 16-byte reads of 8 threads fall in different banks.
template <class T>
constexpr int kBGroup = 8 + 16 / (int)sizeof(T);
template <class T>
__device__ __forceinline__ int bidx(int c)
{
    return (c & 7) * kBGroup<T> + (c >> 3);
}
template <class T>
constexpr int kBEntries = 8 * kBGroup<T>;
// elements between the columns (op N) or rows (op T/C) of a staged tile: the
// reads of a warp (8 column groups x 4 rows) fall in different banks
constexpr int kBPitch = 72;
template <class T>
__device__ __forceinline__ int bpitch(int op)
{
    return op != 0 ? kBPitch : (sizeof(T) == 8 ? 66 : 68);
}

template <class T>
struct alignas(16) BlockSmem {
    T stage[kBStages][NB * kBPitch];   // tiles, [column][row] (op N) or [row][column]
    T xin[kBCluster][kBEntries<T>];    // solved blocks of earlier CTAs of this cluster (st.async)
    T xs[2][kBEntries<T>];             // a solved block from the published words
    T y2[kBEntries<T>];                // b - the products of the earlier blocks
    wide_t<T> Y[NB][NB + 1];  // FP64 inverse of the diagonal block (the other triangle: doubling temporaries)
    T D[NB][NB + 1];          // the diagonal block of op(A)
    uint64_t xbar[kBCluster];
    unsigned s, epoch, cl;
};
static_assert(sizeof(BlockSmem<cfloat>) <= 232448 && 2 * (sizeof(BlockSmem<float>) + 1024) <= 233472,
              "block kernel shared memory: one complex or two real CTAs per SM");

__device__ __forceinline__ void cp_async_elem(float* dst, const float* src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tma::smem_u32(dst)), "l"(src), "r"(in ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_elem(cfloat* dst, const cfloat* src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(tma::smem_u32(dst)), "l"(src), "r"(in ? 8 : 0)
                 : "memory");
}
// two neighbouring entries into another CTA's shared memory, counted on its barrier
__device__ __forceinline__ void st_async_pair(uint32_t addr, float a, float b, uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(a), "f"(b), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async_pair(uint32_t addr, cfloat a, cfloat b, uint32_t bar)
{
    st_async_f32x4(addr, a.re, a.im, b.re, b.im, bar);
}

// `cl`: CTAs per cluster (1: no cluster launch attribute).  HALF: complex A at
// 4 modulo 8, fetched a float at a time.  (An instantiation: the choice at run
// time took complex n = 3001 from 89 to 92 us.)
template <class T, bool HALF>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 4 ? 2 : 1)
    trsv_block_kernel(int cl, int n, int lower_op, int op, int unit, const T* __restrict__ A, long lda, T* x,
                      long incx, unsigned long long* pub, unsigned* ticket, unsigned* epoch_word, int* status)
{
    using W = wide_t<T>;
    constexpr int kW = sizeof(T) / 4;  // published words per entry
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BlockSmem<T>& S = *reinterpret_cast<BlockSmem<T>*>(smem_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nb = (n + NB - 1) / NB;
    const unsigned rank = cl > 1 ? cluster_rank() : 0u;
    if (t == 0) {
        const unsigned e = *(volatile unsigned*)epoch_word + 1u;
        S.epoch = e == 0u ? 1u : e;
        if (cl == 1) S.s = atomicAdd(ticket, 1u);
        for (int r = 0; r < cl; ++r) tma::mbar_init(&S.xbar[r], 1);
        tma::mbar_init_fence();
        // one arrival (this one, declaring the bytes) plus a block per earlier rank
        for (unsigned r = 0; r < rank; ++r) tma::mbar_expect_tx(&S.xbar[r], NB * sizeof(T));
    }
    if (cl > 1) {
        // every CTA of the cluster has set up its barriers before any shared
        // memory of another CTA is written
        __syncthreads();
        cluster_sync_all();
        if (rank == 0 && t == 0) {
            const unsigned c = atomicAdd(ticket, 1u);
            for (unsigned r = 0; r < (unsigned)cl; ++r) st_cluster_u32(map_to(&S.cl, r), c);
            if (c == gridDim.x / cl - 1) *ticket = 0u;  // every ticket of this launch is taken
        }
        cluster_sync_all();
        if (t == 0) S.s = S.cl * cl + rank;
    }
    __syncthreads();
    const int s = (int)S.s;
    const unsigned epoch = S.epoch;
    const int cfirst = cl > 1 ? (int)S.cl * cl : nb;  // first block (solve order) delivered by this cluster
    if (cl == 1 && s == nb - 1 && t == 0) *ticket = 0u;
    if (s >= nb) {  // a cluster's spare CTA past the last block
        cluster_sync_all();
        return;
    }
    auto blk = [&](int p) { return lower_op ? p : nb - 1 - p; };
    const int kb = blk(s), r0 = kb * NB, nr = min(NB, n - r0);
    // element (r, c) of op(A), before conjugation
    auto at = [&](int r, int c) -> const T* { return op == 0 ? A + (long)c * lda + r : A + (long)r * lda + c; };
    // thread layout of inv(D) and of every tile: rows R0 and R0 + 8 (next to
    // each other in a stored block of x), columns cg + 8j
    const int cg = lane & 7, R0 = (warp >> 1) * 16 + (warp & 1) * 4 + (lane >> 3);
    // copies of a 64 x 64 tile: op N rows lane and lane + 32 of columns
    // warp*8 .. +7, op T/C columns lane and lane + 32 of rows warp*8 .. +7
    // (consecutive lanes read consecutive addresses)
    const int ntile = max(0, s - 1), P = bpitch<T>(op);
    auto fetch_to = [&](int i, int st) {
        if (i >= 0) {
            const int c0 = blk(i) * NB, nc = min(NB, n - c0);
            T* dst = &S.stage[st][warp * 8 * P + lane];
            const T* src = op == 0 ? at(r0 + lane, c0 + warp * 8) : at(r0 + warp * 8, c0 + lane);
            const int nf = op == 0 ? nr : nc, ng = op == 0 ? nc : nr;
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int f = 32 * (q & 1), g = q >> 1;
                const bool in = lane + f < nf && warp * 8 + g < ng;
                const T* e = in ? src + (long)g * lda + f : A;
                if constexpr (HALF) {
                    cp_async_elem(&dst[g * P + f].re, &e->re, in);
                    cp_async_elem(&dst[g * P + f].im, &e->im, in);
                } else {
                    cp_async_elem(dst + g * P + f, e, in);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto fetch = [&](int i) { fetch_to(i < ntile ? i : -1, i % kBStages); };
    // this thread's share of a staged tile
    auto read_tile = [&](int st, T(&m)[2][8]) {
        const T* src = &S.stage[st][op == 0 ? cg * P + R0 : R0 * P + cg];
        const int rs = op == 0 ? 8 : 8 * P, cs = op == 0 ? 8 * P : 8;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                m[k][j] = src[k * rs + j * cs];
                if (op == 2) m[k][j] = conj_v(m[k][j]);
            }
    };
    // the tile next to D first, in the last stage, which the ring reaches last
    fetch_to(s - 1, kBStages - 1);
    for (int i = 0; i < kBStages - 1; ++i) fetch(i);

    // ---- diagonal block: D, then its FP64 inverse
    float* const rowsum = reinterpret_cast<float*>(S.xs[0]);  // of |D|
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int f = lane + 32 * (q & 1), g = warp * 8 + (q >> 1);
        const int r = op == 0 ? f : g, c = op == 0 ? g : f;
        T v = zero_v(T());
        if (r < nr && c < nr) {
            if constexpr (HALF) v = *at(r0 + r, r0 + c);
            else v = ldg(at(r0 + r, r0 + c));
            if (op == 2) v = conj_v(v);
        }
        S.D[r][c] = v;
    }
    if (t < NB) S.y2[bidx<T>(t)] = t < nr ? x[(long)(r0 + t) * incx] : zero_v(T());  // b
    __syncthreads();
    if (t < NB) {
        // thread t owns column j of the 16 x 16 diagonal block at o; the
        // column stays in registers
        const int o = t & ~15, j = t & 15;
        W y[16];
        auto solve_row = [&](int i, int k0, int k1) {
            W acc;
            dset(acc, i == j ? 1.0 : 0.0);
#pragma unroll
            for (int k = 0; k < 16; ++k)
                if (k >= k0 && k < k1) dmac(acc, dneg(wide(S.D[o + i][o + k])), y[k]);
            return (unit || o + i >= nr) ? acc : dmul(acc, dinv(wide(S.D[o + i][o + i])));
        };
        if (lower_op) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                y[i] = solve_row(i, 0, i);
                if (i < j) dset(y[i], 0.0);
            }
        } else {
#pragma unroll
            for (int i = 15; i >= 0; --i) {
                y[i] = solve_row(i, i + 1, 16);
                if (i > j) dset(y[i], 0.0);
            }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) S.Y[o + i][o + j] = y[i];
    } else if (t < 3 * NB) {
        // meanwhile the row sums of |D|, two threads a row
        const int r = (t - NB) >> 1, h = (t & 1) * 32;
        float v = 0.f;
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
            const int c = h + i;
            v += (lower_op ? c > r : c < r) ? 0.f : c == r && unit ? 1.f : abs_sum(S.D[r][c]);
        }
        v = xor_add(v, 1);
        rowsum[r] = v;
    }
    __syncthreads();
    // the product C Y11 (lower; C Y22 upper) waits in the block's mirror
    // image, which the inverse does not use
    // doubling (h = 16, then 32): the off-diagonal h x h block of each
    // 2h x 2h diagonal block is -Y22 C Y11 (lower) or -Y11 C Y22 (upper);
    // 32 / h products at a time, 2 x TC outputs per thread
    auto doubling = [&](auto hc) {
        constexpr int h = decltype(hc)::value;
        constexpr int TPG = kThreads / (32 / h), TC = h / 16;
        const int pr = t / TPG, u = t % TPG, o = pr * 2 * h;
        const int tr = (u / 16) * 2, tcl = u % 16;
        W acc[2][TC];
        auto prod = [&](auto ea, auto eb) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) dset(acc[i][j], 0.0);
#pragma unroll 4
            for (int k = 0; k < h; ++k) {
                W a[2], bb[TC];
#pragma unroll
                for (int i = 0; i < 2; ++i) a[i] = ea(tr + i, k);
#pragma unroll
                for (int j = 0; j < TC; ++j) bb[j] = eb(k, tcl + 16 * j);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < TC; ++j) dmac(acc[i][j], a[i], bb[j]);
            }
        };
        // rows and columns of the off-diagonal block C and of the two inverses
        const int rl = lower_op ? o + h : o, cl0 = lower_op ? o : o + h;
        prod([&](int r, int k) { return wide(S.D[rl + r][cl0 + k]); },
             [&](int k, int c) { return S.Y[cl0 + k][cl0 + c]; });
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) S.Y[cl0 + tr + i][rl + tcl + 16 * j] = acc[i][j];
        __syncthreads();
        prod([&](int r, int k) { return S.Y[rl + r][rl + k]; },
             [&](int k, int c) { return S.Y[cl0 + k][rl + c]; });
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) S.Y[rl + tr + i][cl0 + tcl + 16 * j] = dneg(acc[i][j]);
        __syncthreads();
        if (h < 32) {  // the next step reads this block with its zeros
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) dset(S.Y[cl0 + tr + i][rl + tcl + 16 * j], 0.0);
            __syncthreads();
        }
    };
    doubling(std::integral_constant<int, 16>{});
    doubling(std::integral_constant<int, 32>{});

    T iv[2][8], tc[2][8];
    bool fin = true, low = false;
    float sum[2] = {0.f, 0.f};  // row sums of |inv(D)| |D|
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = R0 + 8 * k, c = cg + 8 * j;
            const bool in = r < nr && c < nr && (lower_op ? c <= r : c >= r);
            const W w = S.Y[r][c];
            iv[k][j] = in ? narrow(w) : zero_v(T());
            fin = fin && finite_v(iv[k][j]);
            low = low || (in && abs_max(iv[k][j]) < FLT_MIN && !is_zero(w));
            sum[k] = fmaf(abs_sum(iv[k][j]), rowsum[c], sum[k]);
        }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int k = 0; k < 2; ++k) sum[k] = xor_add(sum[k], o);
    fin = fin && sum[0] <= kBGrowth && sum[1] <= kBGrowth;
    asm volatile("cp.async.wait_group %0;" ::"n"(kBStages - 1) : "memory");
    __syncthreads();  // the tile next to D has arrived
    read_tile(kBStages - 1, tc);
    // inv_ok: neither; low: only the last of the three reasons to substitute
    const bool inv_ok = __syncthreads_and(fin && !low);
    if (!inv_ok) low = __syncthreads_and(fin);
    // a[k] += row R0 + 8k of this thread's columns of M times its entries of v
    auto load_x = [&](const T* v, T(&q)[8]) {
        alignas(16) T w[8];
#pragma unroll
        for (int i = 0; i < 2 * kW; ++i)
            reinterpret_cast<float4*>(w)[i] = *reinterpret_cast<const float4*>(&v[cg * kBGroup<T> + i * 4 / kW]);
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = w[j];
    };
    auto mul = [&](const T(&m)[2][8], const T* v, T(&a)[2]) {
        T q[8];
        load_x(v, q);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            T b1 = zero_v(T());
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                madd_v(a[k], m[k][j], q[j]);
                madd_v(b1, m[k][j + 1], q[j + 1]);
            }
            a[k] = addv(a[k], b1);
        }
    };
    // the sums over the 8 threads that share rows, in each of them
    auto share = [&](T(&a)[2]) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < 2; ++k) a[k] = xor_add(a[k], o);
    };

    bool bad = false;
    // the solved entries of the block with solve index p: delivered into this
    // CTA's shared memory by an earlier CTA of the cluster (every thread
    // waits on the transaction barrier), else polled from the published words
    // into `buf` (the caller's barrier makes them visible)
    auto poll_block = [&](int p, T* buf) {
        const int c0 = blk(p) * NB, nc = min(NB, n - c0);
        if (t < NB * kW) {
            float v = 0.f;
            if (t / kW < nc && !poll_word(pub + (long)c0 * kW + t, epoch, status, v)) bad = true;
            reinterpret_cast<float*>(&buf[bidx<T>(t / kW)])[t % kW] = v;
        }
    };
    auto wait_in = [&](int p) {
        if (!xbar_wait_bounded(&S.xbar[p - cfirst], kTrsvWaitNs)) bad = true;
        return (const T*)S.xin[p - cfirst];
    };

    // ---- the earlier blocks but the last, in solve order
    T acc[2] = {zero_v(T()), zero_v(T())};
    for (int i = 0; i < ntile; ++i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kBStages - 2) : "memory");
        // two buffers: a thread that runs ahead writes the other one
        if (i < cfirst) poll_block(i, S.xs[i & 1]);
        // tile i has arrived, and every thread is done with tile i - 1
        if (__syncthreads_or(bad)) { bad = true; break; }
        fetch(i + kBStages - 1);
        const T* xv = i >= cfirst ? wait_in(i) : S.xs[i & 1];
        T m[2][8];
        read_tile(i % kBStages, m);
        mul(m, xv, acc);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    // ---- this block's step of the chain
    // hand-off: lane cg sends this thread's two rows to rank + 1 + cg and rank + 9 + cg
    uint32_t dx[2] = {0, 0}, db[2] = {0, 0};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const unsigned d = rank + 1 + cg + 8 * u;
        if (cl > 1 && d < (unsigned)cl && cfirst + (int)d < nb) {
            dx[u] = map_to(&S.xin[rank][bidx<T>(R0)], d);
            db[u] = map_to(&S.xbar[rank], d);
        }
    }
    // the solved entries of block s-1, once they are known (every thread calls it)
    auto last_x = [&]() -> const T* {
        if (s - 1 >= cfirst) return wait_in(s - 1);
        poll_block(s - 1, S.xs[(s - 1) & 1]);
        bad = __syncthreads_or(bad);
        return S.xs[(s - 1) & 1];
    };
    // the b entry of the row this lane (cg < 2) writes to y2
    const T brow = cg < 2 ? S.y2[bidx<T>(R0 + 8 * cg)] : zero_v(T());
    if (!bad && s >= 1) mul(tc, last_x(), acc);
    share(acc);
    T o[2] = {zero_v(T()), zero_v(T())};
    T yr = zero_v(T());
    if (cg < 2) {
        yr = subv(brow, cg == 0 ? acc[0] : acc[1]);
        S.y2[bidx<T>(R0 + 8 * cg)] = yr;
    }
    // a wait failed, or the inverse may not do
    const int vote = __syncthreads_or(bad || !inv_ok || !finite_v(yr));
    if (vote == 0) {
        mul(iv, S.y2, o);
        share(o);
    } else {
        bad = __syncthreads_or(bad);
        // an inverse with entries below the normal range leaves out at most
        // 64 * 2^-126 max|y| an entry: nothing that shows where |y| <= 2^60 and
        // |x| >= 2^-30
        bool sub = __syncthreads_or(!low || !finite_v(yr) || abs_max(yr) > 0x1p60f);
        if (!sub) {
            mul(iv, S.y2, o);
            share(o);
            sub = __syncthreads_or((R0 < nr && abs_max(o[0]) < 0x1p-30f) || (R0 + 8 < nr && abs_max(o[1]) < 0x1p-30f));
        }
        if (!bad && sub) {
            if (warp == 0) {
                // (rows past nr, lower: 0; upper: the order starts at nr - 1)
                const int sg = lower_op ? 1 : -1, ra = lower_op ? lane : nr - 1 - lane, rb = ra + 32 * sg;
                T v[2] = {ra >= 0 ? S.y2[bidx<T>(ra)] : zero_v(T()), rb >= 0 ? S.y2[bidx<T>(rb)] : zero_v(T())};
                substitute<T, 2>(lower_op ? &S.D[0][0] : &S.D[nr - 1][nr - 1], sg * (NB + 1), sg, nr, unit != 0, v);
                if (ra >= 0) S.y2[bidx<T>(ra)] = v[0];
                if (rb >= 0) S.y2[bidx<T>(rb)] = v[1];
            }
            __syncthreads();
            o[0] = S.y2[bidx<T>(R0)];
            o[1] = S.y2[bidx<T>(R0 + 8)];
        }
    }
    if (!bad) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (R0 + 8 * k >= nr) o[k] = zero_v(T());
        // the hand-offs first, then the published words; the output x last
        if (db[0] != 0 && cg == 0) st_async_pair(dx[0], o[0], o[1], db[0]);
        __syncwarp();
        if (db[0] != 0 && cg != 0) st_async_pair(dx[0], o[0], o[1], db[0]);
        if (db[1] != 0) st_async_pair(dx[1], o[0], o[1], db[1]);
        const int k = cg / kW, row = R0 + 8 * k;
        if (cg < 2 * kW && row < nr) {
            const T v = k == 0 ? o[0] : o[1];
            const float f = reinterpret_cast<const float*>(&v)[cg % kW];
            st_relaxed_u64(pub + (long)(r0 + row) * kW + cg % kW, ((unsigned long long)epoch << 32) | __float_as_uint(f));
            reinterpret_cast<float*>(&x[(long)(r0 + row) * incx])[cg % kW] = f;
        }
    } else {
        atomicOr(status, (int)kDevWaitTimeout);
    }
    // after a failed wait, let bytes that other CTAs of the cluster may still
    // send land before leaving (each wait bounded)
    if (__syncthreads_or(bad) && t == 0)
        for (unsigned r = 0; r < rank; ++r) xbar_wait_bounded(&S.xbar[r], kTrsvWaitNs);
    if (t == 0 && s == nb - 1) *(volatile unsigned*)epoch_word = epoch;
    if (cl > 1) cluster_sync_all();
}

// the number of clusters of CL CTAs of the STRSV kernel the current device
// holds at once (0: none), asked once per device and cluster size
template <int CL>
int strsv_cluster_capacity(int device, int smem)
{
    static std::atomic<int> cap[64];  // capacity + 1; 0: not asked yet
    std::atomic<int>& c = cap[device & 63];
    int v = c.load();
    if (v == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CL;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(CL);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, strsv_tma_kernel<CL>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        v = clusters + 1;
        c.store(v);
    }
    return v - 1;
}

// Published-entry words for a solve of `words` values.  Calls that fit use
// the handle's fixed area, which lives as long as the handle (a captured
// launch may keep its address); only longer solves use the grown buffer.
cudaError_t trsv_pub(iclblasHandle_t h, size_t words, unsigned long long** pub)
{
    if (words <= (size_t)kPubWords) {
        *pub = reinterpret_cast<unsigned long long*>(h->ws.counters + kCounterWords);
        return cudaSuccess;
    }
    if (words > h->ws.pub_elems) {
        if (h->ws.pub) cudaFree(h->ws.pub);
        h->ws.pub = nullptr;
        h->ws.pub_elems = 0;
        cudaError_t e = cudaMalloc(&h->ws.pub, words * sizeof(unsigned long long));
        if (e != cudaSuccess) return e;
        e = cudaMemsetAsync(h->ws.pub, 0, words * sizeof(unsigned long long), h->stream);
        if (e != cudaSuccess) return e;
        h->ws.pub_elems = words;
    }
    *pub = h->ws.pub;
    return cudaSuccess;
}

template <int CL>
cudaError_t strsv_launch(iclblasHandle_t h, int smem, int nb, const CUtensorMap& map, int n, int lower_op, int op,
                         int unit, float* x, int incx, unsigned long long* pub, unsigned* ticket,
                         unsigned* epoch_word)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)((nb + CL - 1) / CL * CL));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = h->stream;
    cfg.attrs = attr;
    cfg.numAttrs = CL > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, strsv_tma_kernel<CL>, map, n, lower_op, op, unit, x, (long)incx,
                                       pub, ticket, epoch_word, h->ws.dev_status);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t strsv_tma(iclblasHandle_t h, int uplo, int trans, int diag, int n, const float* A, int lda, float* x,
                      int incx, bool& used)
{
    used = false;
    const int op = trans == ICLBLAS_OP_N ? 0 : 1;
    CUtensorMap map;
    // op N: boxes of 128 rows x 64 columns of A; op T: 64 rows x 128 columns
    if (lda < n || !tma::map_f32_colmajor(&map, A, n, n, lda, op == 0 ? RB : HB, op == 0 ? HB : RB))
        return cudaSuccess;
    unsigned long long* pub = nullptr;
    cudaError_t e = trsv_pub(h, (size_t)n, &pub);
    if (e != cudaSuccess) return e;
    const int smem = (int)sizeof(FastSmem) + 1024;
    // the attribute belongs to the current device's copy of each kernel
    static std::atomic<unsigned long long> smem_set{0};
    const unsigned long long bit = 1ull << (h->device & 63);
    if (!(smem_set.load() & bit)) {
        const void* kernels[] = {(const void*)strsv_tma_kernel<1>, (const void*)strsv_tma_kernel<2>,
                                 (const void*)strsv_tma_kernel<3>, (const void*)strsv_tma_kernel<4>,
                                 (const void*)strsv_tma_kernel<5>, (const void*)strsv_tma_kernel<6>,
                                 (const void*)strsv_tma_kernel<7>, (const void*)strsv_tma_kernel<8>};
        for (const void* k : kernels) {
            if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess)
                return e;
        }
        smem_set.fetch_or(bit);
    }
    const bool lower = uplo == ICLBLAS_FILL_MODE_LOWER;
    const int lower_op = (op == 0) ? lower : !lower;
    const int nb = (n + RB - 1) / RB;
    const int unit = diag == ICLBLAS_DIAG_UNIT;
    unsigned* ticket = h->ws.counters;
    unsigned* epoch_word = h->ws.counters + kCounterWords - 1;
    used = true;
    // the largest cluster size, 8 down to 2, for which every cluster of
    // the launch is resident at once (sizes need not be powers of two: a
    // GPC that holds two clusters of 8 may hold three of 6); if none is,
    // clusters of 8 (the most DSMEM hand-offs), else one CTA per block
    const int caps[9] = {0,
                         0,
                         strsv_cluster_capacity<2>(h->device, smem),
                         strsv_cluster_capacity<3>(h->device, smem),
                         strsv_cluster_capacity<4>(h->device, smem),
                         strsv_cluster_capacity<5>(h->device, smem),
                         strsv_cluster_capacity<6>(h->device, smem),
                         strsv_cluster_capacity<7>(h->device, smem),
                         strsv_cluster_capacity<8>(h->device, smem)};
    int cl = 0;
    for (int c = 8; c >= 2 && !cl; --c)
        if (caps[c] > 0 && caps[c] * c >= nb) cl = c;
    if (!cl && caps[8] > 0) cl = 8;
    switch (cl) {
    case 8: return strsv_launch<8>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
    case 7: return strsv_launch<7>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
    case 6: return strsv_launch<6>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
    case 5: return strsv_launch<5>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
    case 4: return strsv_launch<4>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
    case 3: return strsv_launch<3>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
    case 2: return strsv_launch<2>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
    default: break;
    }
    return strsv_launch<1>(h, smem, nb, map, n, lower_op, op, unit, x, incx, pub, ticket, epoch_word);
}

// the number of clusters of `cl` CTAs of the block kernel the current device
// holds at once (0: none), asked once per device and cluster size
template <class T, bool HALF>
int trsv_block_capacity(int device, int cl)
{
    static std::atomic<int> cap[64][kBCluster + 1];  // capacity + 1; 0: not asked yet
    std::atomic<int>& c = cap[device & 63][cl];
    int v = c.load();
    if (v == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)cl;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)cl);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = sizeof(BlockSmem<T>);
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, trsv_block_kernel<T, HALF>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        v = clusters + 1;
        c.store(v);
    }
    return v - 1;
}

template <class T, bool HALF>
cudaError_t trsv_block(iclblasHandle_t h, int uplo, int trans, int diag, int n, const T* A, int lda, T* x, int incx)
{
    const int nb = (n + NB - 1) / NB;
    const int op = trans == ICLBLAS_OP_N ? 0 : (trans == ICLBLAS_OP_C && sizeof(T) == sizeof(cfloat)) ? 2 : 1;
    const bool lower = uplo == ICLBLAS_FILL_MODE_LOWER;
    const int lower_op = (op == 0) ? lower : !lower;
    constexpr int kW = sizeof(T) / 4;
    unsigned long long* pub = nullptr;
    cudaError_t e = trsv_pub(h, (size_t)n * kW, &pub);
    if (e != cudaSuccess) return e;
    // the attribute belongs to the current device's copy of the kernel
    static std::atomic<unsigned long long> smem_set{0};
    const unsigned long long bit = 1ull << (h->device & 63);
    if (!(smem_set.load() & bit)) {
        e = cudaFuncSetAttribute(trsv_block_kernel<T, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(BlockSmem<T>));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(trsv_block_kernel<T, HALF>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        smem_set.fetch_or(bit);
    }
    // the cluster size as for strsv_tma_kernel: the largest (up to the number
    // of blocks) for which every cluster of the launch is resident at once,
    // else 8, else none
    int cl = 1;
    if (nb > 1) {
        for (int c = std::min(nb, nb <= kBWide ? kBCluster : kMaxCluster); c >= 2 && cl == 1; --c) {
            const int cap = trsv_block_capacity<T, HALF>(h->device, c);
            if (cap > 0 && cap * c >= nb) cl = c;
        }
        if (cl == 1 && trsv_block_capacity<T, HALF>(h->device, kMaxCluster) > 0) cl = kMaxCluster;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cl;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)((nb + cl - 1) / cl * cl));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = sizeof(BlockSmem<T>);
    cfg.stream = h->stream;
    cfg.attrs = attr;
    cfg.numAttrs = cl > 1 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, trsv_block_kernel<T, HALF>, cl, n, lower_op, op, (int)(diag == ICLBLAS_DIAG_UNIT), A,
                           (long)lda, x, (long)incx, pub, h->ws.counters, h->ws.counters + kCounterWords - 1,
                           h->ws.dev_status);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <class T, int R>
cudaError_t trsv_small_launch(iclblasHandle_t h, int n, int lower_op, int op, int unit, const T* A, int lda, T* x,
                              int incx)
{
    const int smem = n * (n | 1) * (int)sizeof(T);
    if (smem > 48 * 1024) {
        static std::atomic<unsigned long long> smem_set{0};
        const unsigned long long bit = 1ull << (h->device & 63);
        if (!(smem_set.load() & bit)) {
            const cudaError_t e = cudaFuncSetAttribute(trsv_small_kernel<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       kSmall * (kSmall | 1) * (int)sizeof(T));
            if (e != cudaSuccess) return e;
            smem_set.fetch_or(bit);
        }
    }
    trsv_small_kernel<T, R><<<1, kThreads, smem, h->stream>>>(n, lower_op, op, unit, A, lda, x, incx);
    return cudaGetLastError();
}

template <class T>
cudaError_t trsv_small(iclblasHandle_t h, int uplo, int trans, int diag, int n, const T* A, int lda, T* x, int incx)
{
    const int op = trans == ICLBLAS_OP_N ? 0 : (trans == ICLBLAS_OP_C && sizeof(T) == sizeof(cfloat)) ? 2 : 1;
    const bool lower = uplo == ICLBLAS_FILL_MODE_LOWER;
    const int lower_op = (op == 0) ? lower : !lower, unit = diag == ICLBLAS_DIAG_UNIT;
    if (n <= 32) return trsv_small_launch<T, 1>(h, n, lower_op, op, unit, A, lda, x, incx);
    if (n <= 64) return trsv_small_launch<T, 2>(h, n, lower_op, op, unit, A, lda, x, incx);
    return trsv_small_launch<T, 4>(h, n, lower_op, op, unit, A, lda, x, incx);
}

}  // namespace

cudaError_t strsv(iclblasHandle_t h, int uplo, int trans, int diag, int n, const float* A, int lda, float* x, int incx)
{
    if (n <= kSmall) return trsv_small<float>(h, uplo, trans, diag, n, A, lda, x, incx);
    // short solves are bound by the time to the first block's inverse, which
    // 64-row blocks have sooner; 128-row blocks make half the steps (us, 64-
    // and 128-row blocks, op N: n = 512 17.7, 27.4, 1024 22.9, 31.0, 2048 37.0,
    // 39.8, 2560 46.2, 46.0, 3072 51.0, 49.6, 4096 65, 59; op T: 2560 45.0,
    // 47.5, 3072 51.1, 52.5, 3584 60, 58)
    if (n > 2560) {
        bool used = false;
        cudaError_t e = strsv_tma(h, uplo, trans, diag, n, A, lda, x, incx, used);
        if (e != cudaSuccess || used) return e;
    }
    return trsv_block<float, false>(h, uplo, trans, diag, n, A, lda, x, incx);
}

cudaError_t ctrsv(iclblasHandle_t h, int uplo, int trans, int diag, int n, const cfloat* A, int lda, cfloat* x,
                  int incx)
{
    if (n <= kSmall) return trsv_small<cfloat>(h, uplo, trans, diag, n, A, lda, x, incx);
    return aligned8(A) ? trsv_block<cfloat, false>(h, uplo, trans, diag, n, A, lda, x, incx)
                       : trsv_block<cfloat, true>(h, uplo, trans, diag, n, A, lda, x, incx);
}

}  // namespace iclb
