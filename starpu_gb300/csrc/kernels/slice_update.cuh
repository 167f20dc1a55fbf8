// FP64 update C[m x n] -= A[m x k] B[n x k]^T (all column-major or strided) on
// the tensor cores, to the accuracy of FP64 FMAs.
//
// GB300 has 2 FP64 FMAs per clock and SM but 4096 FP16 ones on its tensor
// cores.  Row i of an operand is taken as fixed point relative to a power of
// two 2^(e_i) above its largest element,
//     x = 2^(e_i - 55) F,   F = sum_{t=1..7} b_t 2^{8 (7 - t)},
// with balanced digits b_t in [-128, 128]: integers, exact in FP16.  The
// product is sum_d 2^{8 (14 - d)} S_d, S_d = sum_{t+u=d} a_t b_u; every S_d
// over 64 terms is an integer below 2^23 (at most 7 pairs x 2^14 x 64), so
// the tensor cores' FP32 accumulation is exact.  The pairs with t + u <= 8
// are formed (28 products).  The scheme is the error-free splitting of matrix
// products of Ozaki, Ogita, Oishi and Rump (Numerical Algorithms 59, 2012),
// with the operands cut at fixed points.  The epilogue adds the S_d as 64-bit
// integers (units of d = 7) and rounds once to FP64.
//
// Error, in units of 2^(e_i + e_j), per term with two nonzero elements: F
// rounds to half a unit, 2^-56 of either row's power of two, 2^-55 together; a
// dropped diagonal d has 15 - d pairs of at most 2^14 2^{8 (14 - d)} / 2^110:
// d = 9 has 6 2^-56, below 2^-53.4, and the rest 2^-61.7.  Once per 64 terms
// S_8 is rounded: 2^-55.  With random digits the sum over d = 9 is some 2^-56
// a term; with every low digit at -128 it is 2^-53.4.  An FP64 FMA rounds to
// 2^-53 of the running sum at every term.
//
// For the Schur complements of an SPD matrix the running sum is bounded by
// sqrt(A_ii A_jj), and so is 2^(e_i + e_j) within a factor of 4 (a row of L
// never exceeds sqrt(A_ii)): an error of the same order even where every digit
// is at its worst.  Elements of a row that holds Inf or NaN are formed by FP64
// FMAs.
//
// GEMM = false: k <= 64 (the trailing update of a panel), A stays cut over the
// tiles of a row block.  GEMM = true: any k in chunks of 64, a tile's chunks
// summed in registers and C rounded once, as an FMA loop does; A is cut again
// for every tile and chunk.
//
// Products of other matrices (GEMM = true) run guarded: the error of an FP64
// FMA loop is bounded by k 2^-53 G, G = sum_k |a_ik| |b_jk|, which may be far
// below k 2^-53 2^(e_i + e_j) (large elements of a_i that meet small ones of
// b_j).  Here the pairs with t + u = 9 are formed, too (scaled by 2^-8 in the
// accumulator of d = 8, whose roundings weigh 2^-61), so that the error of a
// chunk of c terms, z of them with two nonzero elements, is below
// (z (2^-55 + 2^-61.7) + 2^-55 + 2^-57) 2^(e_i + e_j), and one more product, of
// the top seven bits of |a_ik| 2^-e_i and |b_jk| 2^-e_j cut off, gives 2^14 G
// from below.  Where that is below (4200 z + 5200) / c the error might exceed
// c 2^-53 G, and the element is formed by FP64 FMAs; z = 0 needs none (z: the
// smaller of the two rows' nonzero elements).  An element formed by FMAs costs
// its products twice: with nearly all of them so (columns graded over 14 orders of
// magnitude) 512^3 takes 598 us where FMAs alone took 545 and random operands,
// which need none, take 79; 512 x 512 x 16 44, 35 and 25 us.
//
// The operands are cut in the kernel, so no workspace is needed.  A CTA (one
// per SM, persistent) keeps the slices of 128 rows of A in shared memory and
// goes along the row in tiles of 32 columns:
//   warps 16-19  read B's 32 x 64 tile (FP64), find the row exponents and
//                write its 7 slices (128-byte swizzle), double-buffered
//   warp 20      issues 7 MMAs per 16 k: slice a_t times the slices
//                b_1 .. b_{8-t} stacked as 32 (8 - t) rows, so that the 7
//                scales d land side by side in 224 accumulator columns
//   warps 0-15   cut A's 128 rows when a work item starts (32 rows per four
//                warps), then read the accumulators (two, in turn) and update
//                C, 8 columns per warp
// The exponents live in rings of four: before tile (item) i + 4's are written,
// the MMAs of tile (item) i + 2 (i + 3) are done, which the epilogue of tile
// (item) i has let start.
// Bounds per 128 x 32 tile: 1792 clocks of tensor pipe (2200 measured), 2400 of
// the FP64 pipe (one add per element), about 2000 of issue slots.  The epilogue
// takes 16 warps because its chain of integer operations per element is long
// (with 8 warps a tile took 9000 clocks).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace gb300 {

constexpr int SU_BM = 128, SU_BN = 32, SU_K = 64, SU_S = 7;
constexpr int SU_SLICE_A = SU_BM * SU_K * 2;  // 16 KB: one 128-byte row per matrix row
constexpr int SU_SLICE_B = SU_BN * SU_K * 2;  // 4 KB
constexpr int SU_ABS = SU_S;  // slice of the top bits of the magnitudes (guarded products)
constexpr int SU_A_BYTES = (SU_S + 1) * SU_SLICE_A, SU_B_BYTES = (SU_S + 1) * SU_SLICE_B;
constexpr int SU_EPI = 16 * 32, SU_CONV = 4 * 32, SU_THREADS = SU_EPI + SU_CONV + 32;
constexpr int SU_MMA_WARP = (SU_EPI + SU_CONV) / 32;
constexpr int SU_SMEM = SU_A_BYTES + 2 * SU_B_BYTES + 1024 /*align*/ + 11264 /*exponents, least sums, barriers*/;
constexpr uint32_t SU_TMEM_COLS = 512, SU_ACC_STRIDE = 256;
constexpr int SU_NONFINITE = 1 << 24;  // exponent of a row with Inf or NaN
constexpr int SU_ERR_TIMEOUT = -1000;  // *err when a wait inside the kernel ran out
constexpr uint64_t SU_DRAIN_NS = 2000000000ull;  // limit of the wait for the MMAs in flight

struct SliceUpdateArgs {
    const double *A, *B;
    long a_rs, a_ks, b_rs, b_ks;  // element (i, k) of A at A[i a_rs + k a_ks], of B likewise
    double *C;
    long ldc;
    int m, n, k;
    int lower;     // 1 (m == n): only elements with row >= column
    int col_tiles, total;  // column tiles of a row block, tiles of all row blocks
    int *err;      // gets SU_ERR_TIMEOUT when a wait ran out
    unsigned long long wait_budget_ns;
};

// The column tiles of all row blocks, row block after row block, are cut into
// equal ranges, one per CTA; a work item is the part of a range inside one row
// block.  A CTA cuts A once per item, so hardly more than once.
struct SliceItems {
    int rb;        // row block of the current item
    int next, end; // tiles still to do, counted from the current row block's first
    __device__ __forceinline__ static int tiles(const SliceUpdateArgs &a, int rb)
    {
        return a.lower ? min(a.col_tiles, (SU_BM / SU_BN) * (rb + 1)) : a.col_tiles;
    }
    __device__ __forceinline__ SliceItems(const SliceUpdateArgs &a)
    {
        const long lo = (long)a.total * blockIdx.x / gridDim.x, hi = (long)a.total * (blockIdx.x + 1) / gridDim.x;
        rb = 0;
        next = (int)lo;
        end = (int)hi;
        skip(a);
    }
    __device__ __forceinline__ void skip(const SliceUpdateArgs &a)
    {
        while (next < end) {
            const int nt = tiles(a, rb);
            if (next < nt) break;
            next -= nt;
            end -= nt;
            ++rb;
        }
    }
    // the next item: column tiles [t0, t1) of row block rb; false: no more
    __device__ __forceinline__ bool item(const SliceUpdateArgs &a, int &t0, int &t1)
    {
        skip(a);
        if (next >= end) return false;
        t0 = next;
        t1 = min(end, tiles(a, rb));
        next = t1;
        return true;
    }
};

// The 16 elements v (k = 16 g .. 16 g + 15 of row `row`) as digits relative to
// biased exponent e >= 1 (subnormal numbers have exponent 1 and no leading one),
// written to the 7 slices at `dst` (row pitch 128 bytes,
// 128-byte swizzle: 16-byte chunk c of row r sits at chunk c ^ (r & 7)).
template <bool GEMM>
__device__ __forceinline__ void su_write_digits(const double (&v)[16], int e, uint8_t *dst, int slice_bytes, int row, int g)
{
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t d[SU_S][4], mag[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            uint32_t h[2], l[2], m[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const unsigned long long u = (unsigned long long)__double_as_longlong(v[8 * half + 2 * p + q]);
                const int ex = (int)(u >> 52) & 0x7FF;
                // |x| 2^(55 + 1) / 2^(e - 1022), shifted down and rounded to the last place
                unsigned long long F = ((u & 0xFFFFFFFFFFFFFull) | (ex ? 0x10000000000000ull : 0ull)) << 3;
                F = ((F >> min(e - max(ex, 1), 63)) + 1) >> 1;
                m[q] = (uint32_t)(F >> 32);
                const unsigned long long G =
                    ((long long)u < 0 ? 0ull - F : F) + 0x0080808080808080ull;  // every digit + 128
                h[q] = (uint32_t)(G >> 32);
                l[q] = (uint32_t)G;
            }
            // digit d as the FP16 1024 + 128 + d, minus 1152
            const uint32_t c64 = 0x64646464u;
            const uint32_t h23 = __byte_perm(h[0], h[1], 0x4051);  // bytes: d2 of 0, 1, then d3 of 0, 1
            const uint32_t l45 = __byte_perm(l[0], l[1], 0x6273), l67 = __byte_perm(l[0], l[1], 0x4051);
            const uint32_t w[SU_S] = {__byte_perm(h[0], h[1], 0x7632) | 0x64006400u,
                                      __byte_perm(h23, c64, 0x4140), __byte_perm(h23, c64, 0x4342),
                                      __byte_perm(l45, c64, 0x4140), __byte_perm(l45, c64, 0x4342),
                                      __byte_perm(l67, c64, 0x4140), __byte_perm(l67, c64, 0x4342)};
            const __half2 off = __half2half2(__ushort_as_half((unsigned short)0xE480));  // -1152
#pragma unroll
            for (int t = 0; t < SU_S; ++t) {
                const __half2 x = __hadd2(*reinterpret_cast<const __half2 *>(&w[t]), off);
                d[t][p] = *reinterpret_cast<const uint32_t *>(&x);
            }
            if (GEMM) {  // F >> 48 as the FP16 1024 + it, minus 1024
                const uint32_t w7 = __byte_perm(m[0], m[1], 0x7632) | 0x64006400u;
                const __half2 x = __hadd2(*reinterpret_cast<const __half2 *>(&w7),
                                          __half2half2(__ushort_as_half((unsigned short)0xE400)));
                mag[p] = *reinterpret_cast<const uint32_t *>(&x);
            }
        }
        const int chunk = (2 * g + half) ^ (row & 7);
#pragma unroll
        for (int t = 0; t < SU_S; ++t)
            *reinterpret_cast<uint4 *>(dst + t * slice_bytes + row * 128 + chunk * 16) =
                make_uint4(d[t][0], d[t][1], d[t][2], d[t][3]);
        if (GEMM)
            *reinterpret_cast<uint4 *>(dst + SU_ABS * slice_bytes + row * 128 + chunk * 16) =
                make_uint4(mag[0], mag[1], mag[2], mag[3]);
    }
}

// one element of A B^T by FP64 FMAs
__device__ __noinline__ double su_dot(const SliceUpdateArgs &a, int row, int col)
{
    const double *p = a.A + row * a.a_rs, *q = a.B + col * a.b_rs;
    double v = 0.0;
#pragma unroll 8
    for (int k = 0; k < a.k; ++k) v = fma(p[k * a.a_ks], q[k * a.b_ks], v);
    return v;
}

// Rows row0 .. row0 + 31 of an operand, cut by a group of four warps (member
// cw holds k = k0 + 16 cw ..): this thread's 16 elements of row row0 + lane.
__device__ __forceinline__ void su_load(const double *src, long rs, long ks, int row0, int rows, int k0, int k, int cw, double (&v)[16])
{
    const int lane = threadIdx.x & 31;
    k0 += 16 * cw;
    const double *p = src + (row0 + lane) * rs + k0 * ks;
    const bool in = row0 + lane < rows;
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = in && k0 + i < k ? p[i * ks] : 0.0;
}
// their exponents to ex[0 .. 31], (GEMM) the least sums that their nonzero
// elements of a chunk of `terms` ask for to least[0 .. 31], and their slices to
// dst; rmax: [2][4][32] of the group, rp alternates; bar: the group's named barrier
template <bool GEMM>
__device__ __forceinline__ void su_convert(const double (&v)[16], int *ex, float *least, int terms, uint8_t *dst, int slice_bytes, int row, int cw,
                                           unsigned *rmax, int &rp, int bar)
{
    const int lane = threadIdx.x & 31;
    unsigned mx = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) mx = max(mx, (unsigned)__double2hiint(v[i]) & 0x7FFFFFFFu);
    if (GEMM) {  // the exponent, and the number of nonzero elements below it
        mx &= 0x7FF00000u;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            mx += (((unsigned)__double2hiint(v[i]) << 1) | (unsigned)__double2loint(v[i])) != 0 ? 1u : 0u;
    }
    unsigned *r = rmax + rp * 128;
    rp ^= 1;
    r[cw * 32 + lane] = mx;
    asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
    const int e = max((int)(max(max(r[lane], r[32 + lane]), max(r[64 + lane], r[96 + lane])) >> 20), 1);
    if (cw == 0) {
        ex[lane] = e == 0x7FF ? SU_NONFINITE : e;
        if (GEMM) {
            const unsigned z = (r[lane] + r[32 + lane] + r[64 + lane] + r[96 + lane]) & 0x7FFu;
            least[lane] = z ? (4200.0f * (float)z + 5200.0f) / (float)terms : 0.0f;
        }
    }
    su_write_digits<GEMM>(v, e, dst, slice_bytes, row, cw);
}
// A bounded wait that all four warps of a group pass or none does (they meet
// at barriers afterwards); bar: a named barrier for the vote.  bad: this warp
// has given up on another wait and votes against.
__device__ __forceinline__ bool su_wait_group(uint64_t *mbar, uint32_t parity, volatile int *abort, uint64_t budget_ns, int bar,
                                              bool bad = false)
{
    uint32_t all, mine = !bad && ptx::wait_parity(mbar, parity, abort, budget_ns) ? 1 : 0;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred q, %2, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(all)
                 : "r"(mine), "r"(bar)
                 : "memory");
    return all != 0;
}

// acc 2^(e - 2098) as FP64, rounded to nearest (e: sum of two biased
// exponents, finite)
__device__ __noinline__ double su_to_double_any(long long acc, int e)
{
    if (acc == 0) return 0.0;
    const unsigned long long mag = acc < 0 ? 0ull - (unsigned long long)acc : (unsigned long long)acc;
    const int lz = __clzll((long long)mag);
    const unsigned long long norm = mag << lz;
    const int ex = e - 1012 - lz;  // biased exponent of the result
    const unsigned long long sign = (unsigned long long)acc & 0x8000000000000000ull;
    unsigned long long bits;
    if (ex > 0 && ex < 2047) {  // (rounding up from the largest exponent gives Inf)
        bits = ((unsigned long long)(ex - 1) << 52) + (norm >> 11) + ((norm >> 10) & 1);
    } else if (ex >= 2047) {
        bits = 0x7FF0000000000000ull;
    } else {  // below the normal range
        const int s = 12 - ex;
        bits = s <= 64 ? ((norm >> (s - 1)) + 1) >> 1 : 0ull;
    }
    return __longlong_as_double((long long)(bits | sign));
}
// the same for the usual case: 32 or more significant bits, a normal result
__device__ __forceinline__ double su_to_double(long long acc, int e)
{
    const uint32_t sgn = (uint32_t)((unsigned long long)acc >> 32) & 0x80000000u;
    const unsigned long long mag = (unsigned long long)(acc < 0 ? -acc : acc);
    const uint32_t hi = (uint32_t)(mag >> 32), lo = (uint32_t)mag;
    const int lz = __clz((int)hi), ex = e - 1012 - lz;
    if (hi == 0 || (unsigned)(ex - 1) >= 2046u) return su_to_double_any(acc, e);
    const uint32_t nh = __funnelshift_l(lo, hi, lz), nl = lo << lz;
    const unsigned long long m = ((unsigned long long)(nh >> 11) << 32) | __funnelshift_r(nl, nh, 11);
    const unsigned long long bits = m + ((nl >> 10) & 1u) + ((unsigned long long)(uint32_t)(ex - 1) << 52);
    return __hiloint2double((int)((uint32_t)(bits >> 32) | sgn), (int)(uint32_t)bits);
}

// sum_d S_d 2^{8 (7 - d)}, d = 2 .. 8, the last one rounded.  The integers held
// by floats are taken on the FMA pipe: |S| <= 2^22 (d <= 5) by adding 1.5 2^23,
// S_8 / 256 by adding 1.5 2^31; S_6 and S_7 may reach 2^22.6 and are converted.
__device__ __forceinline__ long long su_combine(const uint32_t (&r)[SU_S][4], int j)
{
    constexpr int K22 = 0x4B400000, K30 = 0x4F400000;  // the bits of those sums for S = 0
    auto f = [&](int d) { return __uint_as_float(r[d][j]); };
    auto raw = [&](int d) { return __float_as_int(f(d) + 12582912.0f); };
    const int t1 = (int)((unsigned)raw(1) * 256u + (unsigned)raw(2) - (unsigned)K22 * 257u);
    const int t2 = __float2int_rn(f(4)) * 256 + __float2int_rn(f(5)) + (__float_as_int(f(6) + 3221225472.0f) - K30);
    const long long lo = (long long)(raw(3) - K22) * 65536 + t2;
    const long long mid = (long long)t1 * 16777216 + lo;
    return mid + ((long long)((raw(0) - K22) * 256) << 32);
}

template <bool GEMM> __global__ void __launch_bounds__(SU_THREADS, 1) slice_update_kernel(const SliceUpdateArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem, *sB = smem + SU_A_BYTES;
    int *ea = (int *)(sB + 2 * SU_B_BYTES);         // [4][128] row exponents of A, by item
    int *eb = ea + 4 * SU_BM;                       // [4][32] of B, by tile
    float *la = (float *)(eb + 4 * SU_BN), *lb = la + 4 * SU_BM;  // GEMM: least sums, like ea and eb
    unsigned *rmax = (unsigned *)(lb + 4 * SU_BN);  // [5 groups][2][4][32]
    uint64_t *bars = (uint64_t *)(rmax + 5 * 2 * 4 * 32);
    uint64_t *b_full = bars, *b_empty = bars + 2, *acc_full = bars + 4, *acc_empty = bars + 6;
    uint64_t *a_full = bars + 8, *a_empty = bars + 9, *drain = bars + 10;
    uint32_t *tmem_slot = (uint32_t *)(bars + 11);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(&b_full[i], SU_CONV);
            ptx::mbar_init(&b_empty[i], 1);
            ptx::mbar_init(&acc_full[i], 1);
            ptx::mbar_init(&acc_empty[i], SU_EPI);
        }
        ptx::mbar_init(a_full, SU_EPI);
        ptx::mbar_init(a_empty, 1);
        ptx::mbar_init(drain, 1);
        *abort_flag = 0;
        ptx::fence_mbarrier_init();
    }
    if (warp == SU_MMA_WARP) {
        ptx::tmem_alloc(tmem_slot, SU_TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;
    const int chunks = GEMM ? (a.k + SU_K - 1) / SU_K : 1;

    if (warp >= SU_EPI / 32 && warp < SU_MMA_WARP) {
        // ---------------------------------------------------- B's slices
        const int cw = warp & 3;
        int tile = 0, rp = 0;  // tile counts accumulators: column tiles times chunks
        SliceItems it(a);
        for (int t0, t1; ok && it.item(a, t0, t1);) {
            double v[16];
            su_load(a.B, a.b_rs, a.b_ks, t0 * SU_BN, a.n, 0, a.k, cw, v);
            for (int t = t0, ch = 0; t < t1; ++tile) {
                const int buf = tile & 1;
                if (!(ok = su_wait_group(&b_empty[buf], ((tile >> 1) & 1) ^ 1, abort_flag, a.wait_budget_ns, 1))) break;
                su_convert<GEMM>(v, eb + (tile & 3) * SU_BN, lb + (tile & 3) * SU_BN, min(SU_K, a.k - ch * SU_K),
                                 sB + buf * SU_B_BYTES, SU_SLICE_B, lane, cw, rmax + 4 * 256, rp, 2);
                ptx::fence_proxy_async_smem();
                ptx::mbar_arrive(&b_full[buf]);
                if (++ch == chunks) ch = 0, ++t;
                if (t < t1) su_load(a.B, a.b_rs, a.b_ks, t * SU_BN, a.n, ch * SU_K, a.k, cw, v);
            }
        }
    } else if (warp == SU_MMA_WARP) {
        // ---------------------------------------------------- MMA issuer
        if (ptx::elect_one()) {
            int tile = 0, item = 0;  // item counts the times A was cut
            SliceItems it(a);
            for (int t0, t1; ok && it.item(a, t0, t1);) {
                if (!GEMM) ok = ptx::wait_parity(a_full, item & 1, abort_flag, a.wait_budget_ns);
                for (int t = t0, ch = 0; t < t1 && ok; ++tile) {
                    const int buf = tile & 1;
                    const uint32_t par = (tile >> 1) & 1;
                    ok = (!GEMM || ptx::wait_parity(a_full, item & 1, abort_flag, a.wait_budget_ns)) &&
                         ptx::wait_parity(&acc_empty[buf], par ^ 1, abort_flag, a.wait_budget_ns) &&
                         ptx::wait_parity(&b_full[buf], par, abort_flag, a.wait_budget_ns);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint32_t d = tmem_base + (uint32_t)buf * SU_ACC_STRIDE;
                    const uint32_t aA = ptx::smem_u32(sA), aB = ptx::smem_u32(sB + buf * SU_B_BYTES);
                    const int ks = (min(SU_K, a.k - ch * SU_K) + 15) / 16;
                    constexpr uint32_t N1 = ptx::make_idesc(SU_BM, SU_BN, ptx::FMT_F16);
                    if (GEMM)  // S_9, where S_8 goes
                        for (int k = 0; k < ks; ++k)
#pragma unroll
                            for (int s = 1; s < SU_S; ++s)
                                ptx::mma_f16_ss(d + (SU_S - 1) * SU_BN, ptx::make_sdesc_k128(aA + s * SU_SLICE_A + k * 32),
                                                ptx::make_sdesc_k128(aB + (SU_S - s) * SU_SLICE_B + k * 32), N1,
                                                (k || s > 1) ? 1u : 0u);
                    for (int k = 0; k < ks; ++k) {
                        const uint64_t bd = ptx::make_sdesc_k128(aB + k * 32);
                        if (GEMM && k == 0) {  // s = 0: a start for S_2 .. S_7, S_9 2^-8 goes on as S_8
                            ptx::mma_f16_ss(d, ptx::make_sdesc_k128(aA), bd,
                                            ptx::make_idesc(SU_BM, SU_BN * (SU_S - 1), ptx::FMT_F16), 0u);
                            ptx::mma_f16_ss_scale8(d + (SU_S - 1) * SU_BN, ptx::make_sdesc_k128(aA),
                                                   ptx::make_sdesc_k128(aB + (SU_S - 1) * SU_SLICE_B), N1);
                        }
#pragma unroll
                        for (int s = 0; s < SU_S; ++s)
                            if (!(GEMM && k == 0 && s == 0))
                                ptx::mma_f16_ss(d + s * SU_BN, ptx::make_sdesc_k128(aA + s * SU_SLICE_A + k * 32), bd,
                                                ptx::make_idesc(SU_BM, SU_BN * (SU_S - s), ptx::FMT_F16), (k | s) ? 1u : 0u);
                        if (GEMM)
                            ptx::mma_f16_ss(d + SU_ABS * SU_BN, ptx::make_sdesc_k128(aA + SU_ABS * SU_SLICE_A + k * 32),
                                            ptx::make_sdesc_k128(aB + SU_ABS * SU_SLICE_B + k * 32), N1, k ? 1u : 0u);
                    }
                    ptx::mma_commit(&b_empty[buf]);
                    ptx::mma_commit(&acc_full[buf]);
                    if (GEMM) ptx::mma_commit(a_empty), ++item;
                    if (++ch == chunks) ch = 0, ++t;
                }
                if (!GEMM && ok) ptx::mma_commit(a_empty), ++item;
            }
            // every MMA issued has read its operands before the CTA ends,
            // whatever the limit of the other waits is
            ptx::mma_commit(drain);
            volatile int never = 0;
            ptx::wait_parity(drain, 0, &never, SU_DRAIN_NS);
        }
    } else {
        // ------------------------------------------ A's slices, epilogue
        const int quarter = warp & 3, group = warp >> 2;  // TMEM lanes; 32 rows of A, 8 columns of a tile
        int tile = 0, item = 0, rp = 0;
        // Set when the wait for an accumulator runs out.  The warps of a group
        // meet at named barriers in cut_a, so this warp goes on to the next of
        // them without touching data and all four leave there together.
        bool bad = false;
        SliceItems it(a);
        auto cut_a = [&](int k0) {
            double v[16];
            su_load(a.A, a.a_rs, a.a_ks, it.rb * SU_BM + 32 * group, a.m, k0, a.k, quarter, v);
            if (!su_wait_group(a_empty, (item & 1) ^ 1, abort_flag, a.wait_budget_ns, 3 + group, bad)) return false;
            su_convert<GEMM>(v, ea + (item & 3) * SU_BM + 32 * group, la + (item & 3) * SU_BM + 32 * group,
                             min(SU_K, a.k - k0), sA, SU_SLICE_A, 32 * group + lane, quarter, rmax + group * 256, rp,
                             7 + group);
            ptx::fence_proxy_async_smem();
            ptx::mbar_arrive(a_full);
            return true;
        };
        for (int t0, t1; ok && it.item(a, t0, t1); ++item) {
            if (!GEMM && !(ok = cut_a(0))) break;
            const int rl = quarter * 32 + lane, row = it.rb * SU_BM + rl;
            for (int t = t0; t < t1 && ok; ++t) {
                const int col0 = t * SU_BN + 8 * group;
                double *crow = a.C + row + (long)col0 * a.ldc;
                // the tile is inside C, on or below the diagonal
                const bool whole = (it.rb + 1) * SU_BM <= a.m && (t + 1) * SU_BN <= a.n &&
                                   (!a.lower || it.rb * SU_BM >= (t + 1) * SU_BN - 1);
                const int jn = whole ? 8 : (row < a.m ? min(8, min(a.n, a.lower ? row + 1 : a.n) - col0) : 0);  // columns of this row
                double c[8];  // GEMM: the sum over the chunks; else C, read before the wait
#pragma unroll
                for (int j = 0; j < 8; ++j) c[j] = !GEMM && j < jn ? crow[(long)j * a.ldc] : 0.0;
                unsigned weak = 0;  // columns that need FMAs
                for (int ch = 0; ch < chunks; ++ch, ++tile) {
                    if (GEMM && !(ok = cut_a(ch * SU_K))) break;
                    const int buf = tile & 1;
                    const uint32_t tb = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * SU_ACC_STRIDE + 8 * group;
                    bad = bad || !ptx::wait_parity(&acc_full[buf], (tile >> 1) & 1, abort_flag, a.wait_budget_ns);
                    bad = __any_sync(0xffffffffu, bad);
                    if (bad) {
                        *abort_flag = 1;
                        if (GEMM) ++item;
                        continue;
                    }
                    ptx::tc_fence_after();
                    const int er = ea[(item & 3) * SU_BM + rl];
                    const int *ec = eb + (tile & 3) * SU_BN + 8 * group;
                    int ev[8], special = 0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) ev[j] = er + ec[j], special |= ev[j];
                    if (__any_sync(0xffffffffu, special >= SU_NONFINITE)) {  // all of the warp's elements by FMAs
                        weak = 0xff;
                        ptx::tc_fence_before();
                        ptx::mbar_arrive(&acc_empty[buf]);
                        if (GEMM) ++item;
                        continue;
                    }
                    const float lr = GEMM ? la[(item & 3) * SU_BM + rl] : 0.0f;
                    const float *lc = lb + (tile & 3) * SU_BN + 8 * group;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t r[SU_S][4], mag[4];
#pragma unroll
                        for (int d = 0; d < SU_S; ++d) ptx::tmem_ld_32x32b_x4(tb + d * SU_BN + 4 * h, r[d]);
                        if (GEMM) ptx::tmem_ld_32x32b_x4(tb + SU_ABS * SU_BN + 4 * h, mag);
                        ptx::tmem_ld_wait();
                        if (h == 1) {
                            ptx::tc_fence_before();
                            ptx::mbar_arrive(&acc_empty[buf]);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const double v = su_to_double(su_combine(r, j), ev[4 * h + j]);
                            if (GEMM) {
                                if (__uint_as_float(mag[j]) < fminf(lr, lc[4 * h + j])) weak |= 1u << (4 * h + j);
                                c[4 * h + j] += v;
                            } else if (4 * h + j < jn) {
                                crow[(long)(4 * h + j) * a.ldc] = c[4 * h + j] - v;
                            }
                        }
                    }
                    if (GEMM) ++item;
                }
                if (!ok || bad) continue;
                if (GEMM) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < jn && !(weak >> j & 1)) crow[(long)j * a.ldc] -= c[j];
                }
                if (jn < 8) weak &= (1u << max(jn, 0)) - 1;
                for (; weak; weak &= weak - 1) {
                    const int j = __ffs((int)weak) - 1;
                    crow[(long)j * a.ldc] -= su_dot(a, row, col0 + j);
                }
            }
            if (GEMM) --item;  // counted per chunk
        }
        ok = ok && !bad;
    }
    if (!ok) {
        atomicMin(a.err, SU_ERR_TIMEOUT);  // (in place of a pivot's info)
        *abort_flag = 1;
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    if (warp == SU_MMA_WARP) ptx::tmem_dealloc(tmem_base, SU_TMEM_COLS);
}

} // namespace gb300
