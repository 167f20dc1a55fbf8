// Latency-bound pieces of the plain-precision Cholesky (FP32 and FP64): the
// 64 x 64 diagonal leaf, the panel solve below it and the triangular solves
// with the finished factor.  They replace the vendor calls of the reference
// codelets at examples/cholesky/cholesky_kernels.c:258 (STRSM) and :354
// (SPOTRF), and dpotrs (min-dgels/base/SRC/dpotrs.c).  All matrices are
// column-major with an explicit leading dimension.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace gb300 {

constexpr int CP_W = 64;  // order of a leaf and width of a panel step

// four values of one row, read and written 16 bytes at a time
template <typename T> struct alignas(16) Quad {
    T v[4];
};

// 1 / sqrt(d) for d in the normal range (cp_normal), to 1.5 u relative (u = 2^-24
// or 2^-53, half an ulp of 1): PTX's approximate instruction and one step of an
// iteration for r^-2 - d = 0.  It keeps the pivot chain of the leaf short: the
// square root and the division that it stands for cost several times as much.
// The residual e = 1 - d r^2 takes two FMAs and errs by u, the result's half of
// that and its own rounding are the 1.5 u.
// FP32: Newton's step r (1 + e/2), which leaves 3/8 e^2.
__device__ __forceinline__ bool cp_normal(float d) { return d >= 1.17549435e-38f && d <= 1.7014118e38f; }
__device__ __forceinline__ bool cp_normal(double d) { return d >= 2.3e-308 && d <= 1.7e308; }
__device__ __forceinline__ float cp_rsqrt(float d)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(0.5f * r, fmaf(-d * r, r, 1.0f), r);
}
// FP64: Householder's step of third order, r (1 + e/2 + 3 e^2/8) (Householder, The
// Numerical Treatment of a Single Nonlinear Equation, 1970), which leaves
// (5/16) e^3: nothing while the instruction's error is below 2^-18.  The tests
// hold both against 1 / sqrt over the range.
__device__ __forceinline__ double cp_rsqrt(double d)
{
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d * r, r, 1.0);
    return fma(r * e, fma(0.375, e, 0.5), r);
}
// outside it, and for d <= 0 or NaN: what the unblocked loop gives
template <typename T> __device__ __noinline__ T cp_rsqrt_any(T d) { return T(1) / sqrt(d); }

template <typename T> __device__ __forceinline__ T cp_dot_sub(T c, const Quad<T> &a, const Quad<T> &b)
{
#pragma unroll
    for (int q = 0; q < 4; ++q) c = fma(-a.v[q], b.v[q], c);
    return c;
}

// ---------------------------------------------------------------------------
// The panel of one 64-column step, by one CTA of 8 warps: Cholesky of the n x
// n (n <= 64) block d and, when NX = 2, the solve x <- x L^-T of 64 rows x
// along with it.  Blocks are held in registers: lane = row (two per lane),
// warp w owns columns 4w .. 4w + 3 and 32 + 4w .. 32 + 4w + 3.
//
// The columns go four at a time (16 steps).  The warp that owns a step's
// columns factors their 4 x 4 diagonal block, solves its rows and publishes
// the four columns in shared memory (a buffer and an mbarrier per step, so no
// CTA barrier); the other warps apply the rank-4 update to the columns they
// still have to the right.  The owner of the next step updates those columns
// first, publishes, and catches up on its others afterwards: the chain of one
// step is wait, update of 4 columns, factor, solve, publish.  Bound by that
// chain of 16 steps.  Same operations as the reference codelet loop
// (cholesky_kernels.c:329-342), four columns at a time; a non-positive (or
// NaN) pivot records info_base + its 1-based column in *info, first one wins.
// ---------------------------------------------------------------------------
template <typename T> using CpBlock = T[2][4][2];  // [column group][column][row half]

// the published columns of every step: rows 0 .. 63 of d, then those of x
template <typename T, int NX> using CpPanel = Quad<T>[16][CP_W + 32 * NX];

constexpr int CP_ERR_TIMEOUT = -1000;

// How long a warp waits for what another warp of its CTA publishes, and the
// word that CP_ERR_TIMEOUT goes to when that runs out (never null).  It takes
// the place of a pivot's info: what follows a wait that ran out is garbage, bad
// pivots too.
struct CpWait {
    unsigned us;
    int *err;
    __device__ __forceinline__ void report() const { atomicMin(err, CP_ERR_TIMEOUT); }
};

// Once per kernel, before a CTA barrier.
__device__ __forceinline__ void cp_panel_init(uint64_t (&bar)[16])
{
    if (threadIdx.x < 16) ptx::mbar_init(&bar[threadIdx.x], 32);
    ptx::fence_mbarrier_init();
}

// One thread's elements of a block: f(value, row, column)
template <typename T, typename F> __device__ __forceinline__ void cp_each(CpBlock<T> &v, F f)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h) f(v[g][c][h], 32 * h + lane, 32 * g + 4 * warp + c);
}

// the published columns of step s; bounded (a step takes well below a
// microsecond and the publisher never waits for this warp, but a process may be
// switched out meanwhile)
__device__ __forceinline__ bool cp_wait(uint64_t *bar, uint32_t parity, unsigned us)
{
    // a limit below a microsecond, which the suspended wait alone may exceed: look once
    if (us == 0) return ptx::mbar_test_wait(bar, parity);
    if (ptx::mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = ptx::globaltimer();
    while (!ptx::mbar_try_wait(bar, parity))
        if (ptx::globaltimer() - t0 > 1000ull * us) return false;
    return true;
}

// rank-4 update of the column groups G .. LAST by a published step
template <typename T, int NX, int G, int LAST>
__device__ __forceinline__ void cp_update(CpBlock<T> &d, CpBlock<T> &x, const Quad<T> *p)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Quad<T> ld[2], lx[2];
#pragma unroll
    for (int h = G; h < 2; ++h) ld[h] = p[32 * h + lane];
#pragma unroll
    for (int h = 0; h < NX; ++h) lx[h] = p[CP_W + 32 * h + lane];
#pragma unroll
    for (int g = G; g <= LAST; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const Quad<T> lc = p[32 * g + 4 * warp + c];
#pragma unroll
            for (int h = g; h < 2; ++h) d[g][c][h] = cp_dot_sub(d[g][c][h], ld[h], lc);
#pragma unroll
            for (int h = 0; h < NX; ++h) x[g][c][h] = cp_dot_sub(x[g][c][h], lx[h], lc);
        }
}

// FP32: the four lanes that hold the rows of the 4 x 4 diagonal block pass it
// through shared memory; every lane factors it for itself and solves its
// rows, so nothing is exchanged inside the pivot chain.
template <bool ANY> __device__ __forceinline__ void cp_factor4(float (&l)[4][4], float (&r)[4])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        r[j] = ANY && !cp_normal(l[j][j]) ? cp_rsqrt_any(l[j][j]) : cp_rsqrt(l[j][j]);
#pragma unroll
        for (int i = j + 1; i < 4; ++i) l[i][j] *= r[j];
#pragma unroll
        for (int k = j + 1; k < 4; ++k)
#pragma unroll
            for (int i = k; i < 4; ++i) l[i][k] = fmaf(-l[i][j], l[k][j], l[i][k]);
    }
}

// What a panel's warps keep beside the columns: the pivots, whose roots the
// diagonal holds in the end (a product with the reciprocal root, which the
// columns take, is off by up to an ulp), and whether a bad one was found.
struct CpState {
    Quad<float> piv[16];
    int found;
    // the diagonal: f(column, root), a warp for its own columns
    template <typename F> __device__ __forceinline__ void diagonal(F f) const
    {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = 32 * (lane >> 2) + 4 * warp + (lane & 3);
        if (lane < 8) f(c, sqrtf(((const volatile float *)piv)[c]));
    }
};

// The first pivot of the four that is not positive, or -1.  Of a panel's steps
// only the first that has one says so: it sets st.found before its columns are
// published, so that the steps behind them see it.
template <int NX, int G>
__device__ __forceinline__ int cp_solve4(CpBlock<float> &d, CpBlock<float> &x, Quad<float> *p, CpState &st)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float l[4][4], r[4];
    auto fetch = [&] {
        const int row = 32 * G + 4 * warp;
        if ((lane >> 2) == warp) p[32 * G + lane] = {d[G][0][G], d[G][1][G], d[G][2][G], d[G][3][G]};
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const Quad<float> v = p[row + i];
#pragma unroll
            for (int j = 0; j <= i; ++j) l[i][j] = v.v[j];
        }
        __syncwarp();
    };
    fetch();
    cp_factor4<false>(l, r);
    // pivots outside the normal range (their bits, less those of the smallest
    // normal number, exceed the range's): again, with the plain functions
    int bad = -1;
    unsigned off = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) off = max(off, __float_as_uint(l[j][j]) - 0x00800000u);
    if (off > 0x7E000000u) {
        fetch();
        cp_factor4<true>(l, r);
#pragma unroll
        for (int j = 3; j >= 0; --j)
            if (!(l[j][j] > 0.0f)) bad = j;
        if (bad >= 0) {
            volatile int *found = &st.found;
            if (*found) bad = -1;
            __syncwarp();
            *found = 1;
        }
    }
    if (lane == 0) st.piv[8 * G + warp] = {l[0][0], l[1][1], l[2][2], l[3][3]};
    auto solve = [&](float(&c)[4][2], int h, int row) {
        Quad<float> y;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v = c[j][h];
#pragma unroll
            for (int q = 0; q < j; ++q) v = fmaf(-y.v[q], l[j][q], v);
            y.v[j] = v * r[j];
            c[j][h] = y.v[j];
        }
        p[row] = y;
    };
#pragma unroll
    for (int h = G; h < 2; ++h) solve(d[G], h, 32 * h + lane);
#pragma unroll
    for (int h = 0; h < NX; ++h) solve(x[G], h, CP_W + 32 * h + lane);
    return bad;
}

// The whole panel (but for d's diagonal, CpState::diagonal); `phase` is the parity of the mbarriers (0 for the first
// panel of a kernel, then in turn), with a CTA barrier between two panels;
// st: in shared memory.  False: a wait ran out.
template <typename T, int NX>
__device__ __forceinline__ bool cp_panel(CpBlock<T> &d, CpBlock<T> &x, CpPanel<T, NX> &pan, uint64_t (&bar)[16], uint32_t phase,
                                         CpState &st, int n, int *info, int info_base, bool report,
                                         unsigned us)
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int steps = (n + 3) / 4;
    bool ok = true;
    auto own = [&](int step, int bad) {
        ptx::mbar_arrive(&bar[step]);
        if (bad >= 0 && report && lane == 0 && info && 4 * step + bad < n) atomicCAS(info, 0, info_base + 4 * step + bad + 1);
    };
    if (threadIdx.x == 0) *(volatile int *)&st.found = 0;  // (warp 0 owns step 0, which every other step waits for)
#pragma unroll 1
    for (int i = 0; i < min(w, steps) - 1; ++i) {
        ok = cp_wait(&bar[i], phase, us) && ok;
        cp_update<T, NX, 0, 1>(d, x, pan[i]);
    }
    if (w > 0 && w <= steps) {
        ok = cp_wait(&bar[w - 1], phase, us) && ok;
        cp_update<T, NX, 0, 0>(d, x, pan[w - 1]);
    }
    // (every mbarrier completes in every panel, so that all keep one parity)
    if (w < steps) own(w, cp_solve4<NX, 0>(d, x, pan[w], st));
    else ptx::mbar_arrive(&bar[w]);
    if (8 + w >= steps) ptx::mbar_arrive(&bar[8 + w]);
    __syncwarp();
    if (steps <= 8) return ok;
    if (w > 0) cp_update<T, NX, 1, 1>(d, x, pan[w - 1]);
    cp_update<T, NX, 1, 1>(d, x, pan[w]);
#pragma unroll 1
    for (int i = w + 1; i < min(8 + w, steps); ++i) {
        ok = cp_wait(&bar[i], phase, us) && ok;
        cp_update<T, NX, 1, 1>(d, x, pan[i]);
    }
    if (8 + w < steps) own(8 + w, cp_solve4<NX, 1>(d, x, pan[8 + w], st));
    __syncwarp();  // st.piv
    return ok;
}

// Cholesky of the n x n (n <= 64) lower block A, in place, by one CTA.
static __global__ void __launch_bounds__(256)
potf2_leaf_kernel(int n, float *__restrict__ A, long lda, int *info, int info_base, const CpWait wait)
{
    __shared__ CpPanel<float, 0> pan;
    __shared__ uint64_t bar[16];
    __shared__ CpState st;
    CpBlock<float> a;
    cp_panel_init(bar);
    // rows and columns past n continue the block as the identity
    cp_each<float>(a, [&](float &v, int r, int c) { v = (r < n && c <= r) ? A[r + (long)c * lda] : (r == c ? 1.0f : 0.0f); });
    __syncthreads();
    if (!cp_panel<float, 0>(a, a, pan, bar, 0, st, n, info, info_base, true, wait.us)) wait.report();
    cp_each<float>(a, [&](float &v, int r, int c) {
        if (r < n && c < r) A[r + (long)c * lda] = v;
    });
    st.diagonal([&](int c, float v) {
        if (c < n) A[c * (lda + 1)] = v;
    });
}

// The FP64 leaf.  An instruction holds a sub-partition's FP64 unit for 64 clocks
// whatever its lanes, so what counts is the number of instructions in the pivot
// chain and their spread over the four units: the columns go one by one (lane =
// row, two rows per lane), warp w owns the columns w mod 8, a buffer and an
// mbarrier per column.  The next column's owner updates it first (2
// instructions, 1 in the lower half), takes 1/sqrt (5), scales (2 or 1),
// publishes, and catches up on its other columns afterwards.  Bound by the chain
// and by the 3000 instructions of the block (48000 clocks over four units).
// The products go into sums of their own, which a column takes in where its group
// of 16 begins, so that most roundings are relative to a sum of products: with
// every product rounded into its element (64 times) the factor of a matrix of
// order 1000 was off by 1.6e-16, with a 32-column leaf, as before, by 1.4e-16, and
// is by 1.1e-16 (to 80 bits, on the CPU).
// (Four warps, one per unit, so that nothing shares a unit with the chain, took
// 3 us more: each warp then trails its own backlog.)
template <int H0>  // columns 32 H0 .. 32 H0 + 31, rows 32 H0 .. 63
__device__ __forceinline__ bool cp_leaf64_half(double (&a)[2][4][2], const double (&e)[2][4][2], double (*col)[CP_W],
                                               double2 *pv, uint64_t *bar, int n, int *info, int info_base, unsigned us)
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool ok = true;
    // with published column j: column 32 H0 + 8 q + w, and all right of it
    auto next = [&](int j, int q) {
        const double lc = col[j][32 * H0 + 8 * q + w];
#pragma unroll
        for (int h = H0; h < 2; ++h) a[H0][q][h] = fma(-col[j][32 * h + lane], lc, a[H0][q][h]);
    };
    auto rest = [&](int j, int q0) {
        double l[2];
#pragma unroll
        for (int h = H0; h < 2; ++h) l[h] = col[j][32 * h + lane];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q >= q0) {
                const double lc = col[j][32 * H0 + 8 * q + w];
#pragma unroll
                for (int h = H0; h < 2; ++h) a[H0][q][h] = fma(-l[h], lc, a[H0][q][h]);
            }
        if (H0 == 0)
#pragma unroll
            for (int q = 0; q < 4; ++q) a[1][q][1] = fma(-l[1], col[j][32 + 8 * q + w], a[1][q][1]);
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // this warp's next column: 32 H0 + 8 q + w
        const int j0 = 32 * H0 + 8 * q, mine = j0 + w;
        if (j0 >= n) break;
        if (q % 2 == 0 && H0 + q > 0)  // a group of 16 begins: its elements, less the products so far
#pragma unroll
            for (int u = q; u < q + 2; ++u)
#pragma unroll
                for (int h = H0; h < 2; ++h) a[H0][u][h] += e[H0][u][h];
#pragma unroll 1
        for (int j = j0; j < min(mine, n); ++j) {  // columns of this round before mine
            ok = cp_wait(&bar[j], 0, us) && ok;
            next(j, q);
            if (j + 1 < mine) rest(j, q + 1);
        }
        if (mine < n) {
            const double piv = __shfl_sync(0xffffffffu, a[H0][q][H0], 8 * q + w);
            double r;
            if (cp_normal(piv)) {
                r = cp_rsqrt(piv);
            } else {
                r = cp_rsqrt_any(piv);
                // (before the column is published: the first bad pivot is the first to get there)
                if (!(piv > 0.0) && lane == 0 && info) atomicCAS(info, 0, info_base + mine + 1);
            }
#pragma unroll
            for (int h = H0; h < 2; ++h) {
                a[H0][q][h] *= r;
                col[mine][32 * h + lane] = a[H0][q][h];
            }
            ptx::mbar_arrive(&bar[mine]);
            if (lane == 0) pv[mine] = make_double2(piv, r);
            __syncwarp();
            if (w > 0) rest(mine - 1, q + 1);
            rest(mine, q + 1);
        }
#pragma unroll 1
        for (int j = mine + 1; j < min(j0 + 8, n); ++j) {  // and after it
            ok = cp_wait(&bar[j], 0, us) && ok;
            rest(j, q + 1);
        }
    }
    return ok;
}

static __global__ void __launch_bounds__(256)
potf2_leaf_kernel(int n, double *__restrict__ A, long lda, int *info, int info_base, const CpWait wait)
{
    __shared__ double col[CP_W][CP_W];
    __shared__ double2 pv[CP_W];  // pivots and the factors their columns were scaled with
    __shared__ uint64_t bar[CP_W];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double a[2][4][2], e[2][4][2];  // [half of the columns][q][row half]: column 32 g + 8 q + w
    if (threadIdx.x < CP_W) ptx::mbar_init(&bar[threadIdx.x], 32);
    ptx::fence_mbarrier_init();
    auto each = [&](auto f) {
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) f(a[g][q][h], 32 * h + lane, 32 * g + 8 * q + w);
    };
    each([&](double &v, int r, int c) { v = r < n && c <= r ? A[r + (long)c * lda] : 0.0; });
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                e[g][q][h] = a[g][q][h];
                if (g > 0 || q >= 2) a[g][q][h] = 0.0;
            }
    __syncthreads();
    bool ok = cp_leaf64_half<0>(a, e, col, pv, bar, n, info, info_base, wait.us);
    if (n > 32) ok = cp_leaf64_half<1>(a, e, col, pv, bar, n, info, info_base, wait.us) && ok;
    if (!ok) wait.report();
    each([&](double &v, int r, int c) {
        if (r < n && c < r) A[r + (long)c * lda] = v;
    });
    // the diagonal, sqrt(pivot): the product is off by up to an ulp, one step makes it exact
    __syncthreads();
    if (threadIdx.x < n) {
        const double d = pv[threadIdx.x].x, r = pv[threadIdx.x].y, l = d * r;
        A[threadIdx.x * (lda + 1)] = cp_normal(d) ? fma(fma(-l, l, d), 0.5 * r, l) : sqrt(d);
    }
}

// ---------------------------------------------------------------------------
// X M^T = B for a lower triangular M (n x n), B m x n overwritten by X, with
// M(j, p) at M[j m_js + p m_ps] and B(r, j) at B[r b_rs + j b_js]:
//   B <- B L^{-T}   M = L                    (the Cholesky panel, STRSM R, L, T, N)
//   B <- L^{-1} B   M = L, B transposed      (LU block row, STRSM L, L, N, N)
//   B <- B U^{-1}   M = U^T, unit diagonal   (LU block column, STRSM R, U, N, U)
// Rows are independent, so a CTA takes SR of them through all n columns in one
// launch (left-looking over 64-column blocks, its solved part in shared memory):
//   update  block columns j: B_j -= X_{<j} M_{j,<j}^T, thread = one column
//           and every fourth p, SR accumulators, M from L2 (every CTA reads all
//           of it; FP32 B U^{-1}, where a column of M is contiguous, every fourth
//           four of p by 16-byte loads: 228 us at m = n = 1024, 574 by single
//           elements, 452 in steps of 64 columns with products between them);
//           the next block's diagonal tile and right-hand sides are
//           already on their way;
//   solve   16 lanes per row, 4 columns each, passed on by shuffles (no
//           barrier).  FP32: 4 neighbouring columns per lane, 4 at a time.
//           FP64: every 16th column, one at a time, on M scaled to a unit
//           diagonal: 167 FP64 operations per row pair instead of 416.  Of
//           the columns past the first 16 the products are summed apart until
//           their group of 16 begins, as in the leaf: rounded into the scaled
//           right-hand side they cost the factor 0.15e-16 of 1.6e-16 at order
//           1000.
// SR is 16 where that fills the GPU, else 8 or 4.
// ---------------------------------------------------------------------------
constexpr int CP_TRSM_MAXN = 1024;  // columns of one launch (shared memory: SR n elements)
constexpr int CP_LP = CP_W + 4;     // pitch of the staged diagonal block and rows

template <typename T> struct SlabArgs {
    int m, n;
    const T *M;
    long m_js, m_ps;
    T *B;
    long b_rs, b_js;
    bool unit;
};

template <typename T, int SR> constexpr size_t cp_trsm_smem(int n)
{
    return ((size_t)((n + CP_W - 1) / CP_W * CP_W) * SR + (size_t)CP_W * CP_LP + CP_W + (size_t)SR * CP_LP +
            4 * CP_W * (SR + 1)) * sizeof(T);
}

// 16 lanes per row: the solve of one 64-column block (rows S, block Ls, inverse diagonal inv)
template <int SR> __device__ __forceinline__ void cp_slab_solve(float *S, const float *Ls, const float *inv)
{
    const int r = threadIdx.x >> 4, l = threadIdx.x & 15, src = threadIdx.x & 16;
    Quad<float> x = *reinterpret_cast<const Quad<float> *>(S + r * CP_LP + 4 * l);
#pragma unroll 2
    for (int s = 0; s < 16; ++s) {
        const float *D = Ls + (4 * s) * CP_LP + 4 * s;
        float y[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float v = x.v[c];
#pragma unroll
            for (int q = 0; q < c; ++q) v = fmaf(-y[q], D[q * CP_LP + c], v);
            y[c] = v * inv[4 * s + c];
        }
        if (l == s)
#pragma unroll
            for (int c = 0; c < 4; ++c) x.v[c] = y[c];
#pragma unroll
        for (int c = 0; c < 4; ++c) y[c] = __shfl_sync(0xffffffffu, y[c], src | s);
        if (l > s)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const Quad<float> lv = *reinterpret_cast<const Quad<float> *>(Ls + (4 * s + q) * CP_LP + 4 * l);
#pragma unroll
                for (int c = 0; c < 4; ++c) x.v[c] = fmaf(-y[q], lv.v[c], x.v[c]);
            }
    }
    *reinterpret_cast<Quad<float> *>(S + r * CP_LP + 4 * l) = x;
}
template <int SR> __device__ __forceinline__ void cp_slab_solve(double *S, const double *Ls, const double *inv)
{
    const int r = threadIdx.x >> 4, l = threadIdx.x & 15, src = threadIdx.x & 16;
    double x[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = S[r * CP_LP + 16 * q + l] * inv[16 * q + l], x[q] = 0.0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        x[g] = g ? b[g] + x[g] : b[0];
#pragma unroll 4
        for (int s = 0; s < 16; ++s) {
            const double y = __shfl_sync(0xffffffffu, x[g], src | s);
            const double *D = Ls + (16 * g + s) * CP_LP + l;
#pragma unroll
            for (int q = g; q < 4; ++q)
                if (q > g || l > s) x[q] = fma(-y, D[16 * q], x[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) S[r * CP_LP + 16 * q + l] = x[q];
}

template <typename T, int SR> __global__ void __launch_bounds__(256) trsm_slab_kernel(const SlabArgs<T> a)
{
    extern __shared__ __align__(16) unsigned char cp_smem[];
    constexpr bool SCALED = sizeof(T) == 8;
    const int npad = (a.n + CP_W - 1) / CP_W * CP_W;
    T *Xs = (T *)cp_smem;             // [npad][SR]: solved rows, column by column
    T *Ls = Xs + (size_t)npad * SR;   // [64][CP_LP]: diagonal block, Ls[c * CP_LP + r] = M(r, c), r > c
    T *inv = Ls + CP_W * CP_LP;       // [64]
    T *S = inv + CP_W;                // [SR][CP_LP]: the block's rows
    T *red = S + SR * CP_LP;          // [4][64][SR + 1]
    const int tid = threadIdx.x, col = tid & 63, kg = tid >> 6;
    const int r0 = blockIdx.x * SR;
    const bool b_along = a.b_js == 1;  // neighbouring threads on neighbouring elements of B
    T lreg[16], b[SR / 4], dg = T(1);
    auto bidx = [&](int i, int &r, int &c) {
        const int e = tid + 256 * i;
        r = b_along ? e / CP_W : e % SR;
        c = b_along ? e % CP_W : e / SR;
    };
    auto fetch = [&](int j0) {
        const int w = min(CP_W, a.n - j0);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int r = a.m_js == 1 ? col : 4 * i + kg, c = a.m_js == 1 ? 4 * i + kg : col;
            lreg[i] = (r < w && c < r) ? a.M[(j0 + r) * a.m_js + (j0 + c) * a.m_ps] : T(0);
        }
        if (tid < CP_W) dg = (tid < w && !a.unit) ? a.M[(j0 + tid) * (a.m_js + a.m_ps)] : T(1);
#pragma unroll
        for (int i = 0; i < SR / 4; ++i) {
            int r, c;
            bidx(i, r, c);
            b[i] = (c < w && r0 + r < a.m) ? a.B[(r0 + r) * a.b_rs + (j0 + c) * a.b_js] : T(0);
        }
    };
    fetch(0);
    for (int j0 = 0; j0 < a.n; j0 += CP_W) {
        const int w = min(CP_W, a.n - j0);
        if (tid < CP_W) inv[tid] = T(1) / dg;
        if (SCALED) __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int r = a.m_js == 1 ? col : 4 * i + kg, c = a.m_js == 1 ? 4 * i + kg : col;
            Ls[c * CP_LP + r] = SCALED ? lreg[i] * inv[r] : lreg[i];
        }
        T cur[SR / 4];
#pragma unroll
        for (int i = 0; i < SR / 4; ++i) cur[i] = b[i];
        if (j0 + CP_W < a.n) fetch(j0 + CP_W);
        if (j0 > 0) {
            T acc[SR];
#pragma unroll
            for (int r = 0; r < SR; ++r) acc[r] = T(0);
            const T *Mc = a.M + (j0 + min(col, w - 1)) * a.m_js;
            auto add = [&](T l, int p) {
                const Quad<T> *x = reinterpret_cast<const Quad<T> *>(Xs + (size_t)p * SR);
#pragma unroll
                for (int q = 0; q < SR / 4; ++q) {
                    const Quad<T> xv = x[q];
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[4 * q + i] = fma(l, xv.v[i], acc[4 * q + i]);
                }
            };
            if (sizeof(T) == 4 && a.m_ps == 1) {
                // neighbouring threads are m_js apart: four p at a time
                const bool vec = ((reinterpret_cast<uintptr_t>(a.M) & 15) == 0) && (a.m_js & 3) == 0;
#pragma unroll 4
                for (int p = 4 * kg; p < j0; p += 16) {
                    Quad<T> l;
                    if (vec) l = *reinterpret_cast<const Quad<T> *>(Mc + p);
                    else l = {Mc[p], Mc[p + 1], Mc[p + 2], Mc[p + 3]};
#pragma unroll
                    for (int u = 0; u < 4; ++u) add(l.v[u], p + u);
                }
            } else {
#pragma unroll 8
                for (int p = kg; p < j0; p += 4) add(Mc[p * a.m_ps], p);
            }
#pragma unroll
            for (int r = 0; r < SR; ++r) red[(kg * CP_W + col) * (SR + 1) + r] = acc[r];
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < SR / 4; ++i) {
            int r, c;
            bidx(i, r, c);
            T v = cur[i];
            if (j0 > 0)
                v -= (red[(0 * CP_W + c) * (SR + 1) + r] + red[(1 * CP_W + c) * (SR + 1) + r]) +
                     (red[(2 * CP_W + c) * (SR + 1) + r] + red[(3 * CP_W + c) * (SR + 1) + r]);
            S[r * CP_LP + c] = v;
        }
        __syncthreads();
        if (tid < 16 * SR) cp_slab_solve<SR>(S, Ls, inv);  // whole warps: two rows each
        __syncthreads();
#pragma unroll
        for (int i = 0; i < SR / 4; ++i) {
            int r, c;
            bidx(i, r, c);
            const T v = S[r * CP_LP + c];
            Xs[(size_t)(j0 + c) * SR + r] = v;
            if (c < w && r0 + r < a.m) a.B[(r0 + r) * a.b_rs + (j0 + c) * a.b_js] = v;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Triangular solves with the finished factor (POTRS): per block of CP_SB rows
// one launch that solves the block (trsv_blk_kernel) and one that updates the
// rows still to come (trsv_upd_kernel), forward with L, backward with L^T.
//
// trsv_blk_kernel: one right-hand side per CTA.  Thread = row (forward) or
// column (backward) of the block, warp = 32 of them.  A warp waits for the
// pieces solved before its own (an mbarrier each, no CTA barrier), subtracts
// their products, solves its piece by shuffles and publishes it; its operands
// of the next piece are on their way meanwhile.  Bound by the chain of
// dependent rows: per piece 32 steps of a shuffle and an FMA.  FP32 sums the
// products apart from the right-hand side, so that each rounding is relative to
// their (smaller) sum; FP64 solves a piece scaled to a unit diagonal, one
// operation (64 clocks) per row in the chain instead of three, and sums the
// products apart until a row's group of eight begins (35 operations in the chain
// of 32 rows): rounded into the right-hand side they cost a solution of order 1000
// 0.5e-16 of 4.6e-16.
// ---------------------------------------------------------------------------
constexpr int CP_SB = 256;

template <typename T> constexpr size_t cp_trsv_smem(bool trans)
{
    return ((size_t)CP_SB + (trans ? 8 * 32 * 33 : 0)) * sizeof(T);
}

template <typename T, bool TRANS>
__global__ void __launch_bounds__(256) trsv_blk_kernel(int w, const T *__restrict__ L, long ldl, T *__restrict__ B, long ldb,
                                                       const CpWait wait)
{
    extern __shared__ __align__(16) unsigned char cp_smem[];
    __shared__ uint64_t bar[16];
    constexpr bool SCALED = sizeof(T) == 8;
    T *xs = (T *)cp_smem;  // [CP_SB]: solved pieces
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = 32 * warp + lane;
    T *stage = xs + CP_SB + warp * 32 * 33;
    T *b = B + (long)blockIdx.x * ldb;
    const int np = (w + 31) / 32;
    cp_panel_init(bar);
    __syncthreads();
    if (warp >= np) return;
    // l[j]: this row's elements of piece p, L(r, 32 p + j), or its column's, L(32 p + j, r)
    auto load = [&](T(&l)[32], int p) {
        if (!TRANS) {
#pragma unroll
            for (int j = 0; j < 32; ++j) l[j] = r < w && 32 * p + j < w ? L[r + (long)(32 * p + j) * ldl] : T(0);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {  // column 32 warp + j, lane = row: coalesced, then turned
                const int row = 32 * p + lane, col = 32 * warp + j;
                l[j] = row < w && col < w ? L[row + (long)col * ldl] : T(0);
            }
        }
    };
    auto turn = [&](T(&l)[32]) {
        if (!TRANS) return;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j) stage[j * 33 + lane] = l[j];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j) l[j] = stage[lane * 33 + j];
    };
    const T v = r < w ? b[r] : T(0), d = r < w ? T(1) / L[r + (long)r * ldl] : T(1);
    T m[32], l[32], sum = T(0);
    load(m, warp);  // the piece's own block
    const int n = TRANS ? np - 1 - warp : warp;  // pieces before this one
    if (n > 0) load(l, TRANS ? np - 1 : 0);
    turn(m);
    if (SCALED)
#pragma unroll
        for (int j = 0; j < 32; ++j) m[j] *= d;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
        const int p = TRANS ? np - 1 - i : i;
        turn(l);
        ok = cp_wait(&bar[p], 0, wait.us) && ok;
        const Quad<T> *x = reinterpret_cast<const Quad<T> *>(xs + 32 * p);
        T acc[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const Quad<T> y = x[j / 4];
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] = fma(l[j + q], y.v[q], acc[q]);
        }
        if (i + 1 < n) load(l, TRANS ? p - 1 : p + 1);
        sum += (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
    T y;
    if (SCALED) {
        const T b0 = (v - sum) * d;
        const int at = TRANS ? 31 - lane : lane;
        y = at < 8 ? b0 : T(0);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const int j = TRANS ? 31 - i : i;
            if (i > 0 && i % 8 == 0 && at / 8 == i / 8) y += b0;
            const T xj = __shfl_sync(0xffffffffu, y, j);
            if (TRANS ? lane < j : lane > j) y = fma(-m[j], xj, y);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const int j = TRANS ? 31 - i : i;
            const T xj = __shfl_sync(0xffffffffu, (v - sum) * d, j);
            if (TRANS ? lane < j : lane > j) sum = fma(m[j], xj, sum);
        }
        y = (v - sum) * d;
    }
    xs[r] = y;
    ptx::mbar_arrive(&bar[warp]);
    if (r < w) b[r] = y;
    if (!ok) wait.report();
}

// C right-hand sides of Y[m x nrhs] -= op(L) X[w x nrhs] (w <= CP_SB): op(L) =
// the m x w block at L (forward) or the transpose of the w x m block at L
// (backward).  CTA = 32 rows of Y: lane = row, the 8 warps split the w terms
// and are summed in a fixed order.  L is read once per C right-hand sides,
// along its columns (the transposed block goes through shared memory).  Bound
// by reading L.
template <typename T, int C, bool TRANS>
__global__ void __launch_bounds__(256) trsv_upd_kernel(int m, int w, int nrhs, const T *__restrict__ L, long ldl,
                                                       const T *__restrict__ X, T *__restrict__ Y, long ldb)
{
    extern __shared__ __align__(16) unsigned char cp_smem[];
    T *xs = (T *)cp_smem;     // [CP_SB][C]
    T *Lt = xs + CP_SB * C;   // backward: [CP_SB][33]; then the partial sums [8][32][C + 1]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.y * C, nc = min(C, nrhs - c0);
    const int r = blockIdx.x * 32 + lane;
    for (int e = tid; e < CP_SB * C; e += 256) {
        const int k = e % CP_SB, c = e / CP_SB;
        xs[k * C + c] = (k < w && c < nc) ? X[k + (long)(c0 + c) * ldb] : T(0);
    }
    T l[32];
    if (!TRANS) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const int k = warp + 8 * j;
            l[j] = (r < m && k < w) ? L[r + (long)k * ldl] : T(0);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const int i = 4 * warp + (j >> 3), k = lane + 32 * (j & 7);  // column i of the block, row k
            const int g = blockIdx.x * 32 + i;
            Lt[k * 33 + i] = (g < m && k < w) ? L[k + (long)g * ldl] : T(0);
        }
    }
    __syncthreads();
    if (TRANS) {
#pragma unroll
        for (int j = 0; j < 32; ++j) l[j] = Lt[(warp + 8 * j) * 33 + lane];
        __syncthreads();  // Lt becomes the partial sums
    }
    T acc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = T(0);
#pragma unroll
    for (int j = 0; j < 32; ++j)
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] = fma(l[j], xs[(warp + 8 * j) * C + c], acc[c]);
#pragma unroll
    for (int c = 0; c < C; ++c) Lt[(warp * 32 + lane) * (C + 1) + c] = acc[c];
    __syncthreads();
    for (int e = tid; e < 32 * C; e += 256) {
        const int i = e & 31, c = e >> 5, row = blockIdx.x * 32 + i;
        T s = T(0);
#pragma unroll
        for (int q = 0; q < 8; ++q) s += Lt[(q * 32 + i) * (C + 1) + c];
        if (row < m && c < nc) {
            T *y = Y + row + (long)(c0 + c) * ldb;
            *y -= s;
        }
    }
}

template <typename T, int C> constexpr size_t cp_upd_smem(bool trans)
{
    const size_t part = (size_t)8 * 32 * (C + 1), lt = trans ? (size_t)CP_SB * 33 : 0;
    return ((size_t)CP_SB * C + (part > lt ? part : lt)) * sizeof(T);
}

} // namespace gb300
