// FP64 update C[m x n] -= A[m x k] B[n x k]^T (k <= 64, all column-major or
// strided) on the tensor cores, with at least the accuracy of FP64 FMAs.
//
// GB300 has 2 FP64 FMAs per clock and SM but 4096 FP16 ones on its tensor
// cores.  Row i of an operand is taken as fixed point relative to a power of
// two 2^(e_i) above its largest element,
//     x = 2^(e_i - 55) F,   F = sum_{t=1..7} b_t 2^{8 (7 - t)},
// with balanced digits b_t in [-128, 128]: integers, exact in FP16.  The
// product is sum_d 2^{8 (14 - d)} S_d, S_d = sum_{t+u=d} a_t b_u; every S_d
// over 64 terms is an integer below 2^23 (at most 7 pairs x 2^14 x 64), so
// the tensor cores' FP32 accumulation is exact.  The pairs with t + u <= 8
// are formed (28 products).  Error: F resolves a quarter of the last bit of
// the row's largest element, the dropped pairs weigh below 2^-58 of
// 2^(e_i + e_j) per term; an FP64 FMA rounds to 2^-53 of the running sum at
// every term.  The epilogue adds the S_d as 64-bit integers (units of d = 7)
// and rounds once to FP64.
//
// For the Schur complements of an SPD matrix this error is bounded like the
// classical one, by eps sqrt(A_ii A_jj): a row of L never exceeds sqrt(A_ii).
// A row that holds Inf or NaN gives NaN.
//
// The operands are cut in the kernel, so no workspace is needed.  A CTA (one
// per SM, persistent) keeps the slices of 128 rows of A in shared memory and
// goes along the row in tiles of 32 columns:
//   warps 8-11  read B's 32 x 64 tile (FP64), find the row exponents and
//               write its 7 slices (128-byte swizzle), double-buffered; per
//               work item the same for A's 128 rows
//   warp 12     issues 7 MMAs per 16 k: slice a_t times the slices
//               b_1 .. b_{8-t} stacked as 32 (8 - t) rows, so that the 7
//               scales d land side by side in 224 accumulator columns
//   warps 0-7   read the accumulator (two, in turn) and update C
// The exponents live in rings of four: before tile (item) i + 4's are written,
// the MMAs of tile (item) i + 2 (i + 3) are done, which the epilogue of tile
// (item) i has let start.
// Measured bounds per 128 x 32 tile: 1792 clocks of tensor pipe, 2048 of the
// FP64 pipe (one add per element), the rest close below.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace gb300 {

constexpr int SU_BM = 128, SU_BN = 32, SU_K = 64, SU_S = 7;
constexpr int SU_SLICE_A = SU_BM * SU_K * 2;  // 16 KB: one 128-byte row per matrix row
constexpr int SU_SLICE_B = SU_BN * SU_K * 2;  // 4 KB
constexpr int SU_A_BYTES = SU_S * SU_SLICE_A, SU_B_BYTES = SU_S * SU_SLICE_B;
constexpr int SU_THREADS = 13 * 32, SU_EPI = 8 * 32, SU_CONV = 4 * 32;
constexpr int SU_SMEM = SU_A_BYTES + 2 * SU_B_BYTES + 1024 /*align*/ + 4096 /*exponents, barriers*/;
constexpr uint32_t SU_TMEM_COLS = 512, SU_ACC_STRIDE = 256;
constexpr int SU_NONFINITE = 1 << 24;  // exponent of a row with Inf or NaN
constexpr int SU_ERR_TIMEOUT = -1000;  // *err when a wait inside the kernel ran out

struct SliceUpdateArgs {
    const double *A, *B;
    long a_rs, a_ks, b_rs, b_ks;  // element (i, k) of A at A[i a_rs + k a_ks], of B likewise
    double *C;
    long ldc;
    int m, n, k;
    int lower;     // 1 (m == n): only elements with row >= column
    int seg;       // column tiles of one work item
    int row_blocks, col_tiles, items;
    int *err;      // may be null
    unsigned long long wait_budget_ns;
};

// Work items: row blocks from the last (the longest, when lower) to the
// first, each cut into segments of `seg` column tiles.
struct SliceItems {
    int rb, base;  // row block and the index of its first item
    __device__ __forceinline__ SliceItems(const SliceUpdateArgs &a) : rb(a.row_blocks - 1), base(0) {}
    __device__ __forceinline__ static int tiles(const SliceUpdateArgs &a, int rb)
    {
        return a.lower ? min(a.col_tiles, (SU_BM / SU_BN) * (rb + 1)) : a.col_tiles;
    }
    // item id (ascending over calls) -> row block rb, column tiles [t0, t1)
    __device__ __forceinline__ void find(const SliceUpdateArgs &a, int id, int &t0, int &t1)
    {
        int nt = tiles(a, rb), ns = (nt + a.seg - 1) / a.seg;
        while (id >= base + ns) {
            base += ns;
            --rb;
            nt = tiles(a, rb);
            ns = (nt + a.seg - 1) / a.seg;
        }
        t0 = (id - base) * a.seg;
        t1 = min(nt, t0 + a.seg);
    }
};

// The 16 elements v (k = 16 g .. 16 g + 15 of row `row`) as digits relative to
// biased exponent e, written to the 7 slices at `dst` (row pitch 128 bytes,
// 128-byte swizzle: 16-byte chunk c of row r sits at chunk c ^ (r & 7)).
__device__ __forceinline__ void su_write_digits(const double (&v)[16], int e, uint8_t *dst, int slice_bytes, int row, int g)
{
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t d[SU_S][4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            uint32_t h[2], l[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const unsigned long long u = (unsigned long long)__double_as_longlong(v[8 * half + 2 * p + q]);
                const int ex = (int)(u >> 52) & 0x7FF;
                // |x| 2^(55 + 1) / 2^(e - 1022), shifted down and rounded to the last place
                unsigned long long F = ex ? ((u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 3 : 0ull;
                F = ((F >> min(e - ex, 63)) + 1) >> 1;
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
        }
        const int chunk = (2 * g + half) ^ (row & 7);
#pragma unroll
        for (int t = 0; t < SU_S; ++t)
            *reinterpret_cast<uint4 *>(dst + t * slice_bytes + row * 128 + chunk * 16) =
                make_uint4(d[t][0], d[t][1], d[t][2], d[t][3]);
    }
}

// acc 2^(e - 2098) as FP64, rounded to nearest (e: sum of two biased exponents)
__device__ __forceinline__ double su_to_double(long long acc, int e)
{
    if (acc == 0) return 0.0;
    const unsigned long long mag = acc < 0 ? 0ull - (unsigned long long)acc : (unsigned long long)acc;
    const int lz = __clzll((long long)mag);
    const unsigned long long norm = mag << lz;
    const int ex = e - 1012 - lz;  // biased exponent of the result
    const unsigned long long sign = (unsigned long long)acc & 0x8000000000000000ull;
    unsigned long long bits;
    if (ex > 0 && ex < 2046) {
        bits = ((unsigned long long)(ex - 1) << 52) + (norm >> 11) + ((norm >> 10) & 1);
    } else if (ex >= 2046) {
        bits = 0x7FF0000000000000ull;
    } else {  // below the normal range
        const int s = 12 - ex;
        bits = s < 64 ? ((norm >> (s - 1)) + 1) >> 1 : 0ull;
    }
    return __longlong_as_double((long long)(bits | sign));
}

__global__ void __launch_bounds__(SU_THREADS, 1) slice_update_kernel(const SliceUpdateArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem, *sB = smem + SU_A_BYTES;
    int *ea = (int *)(sB + 2 * SU_B_BYTES);       // [4][128] row exponents of A, by item
    int *eb = ea + 4 * SU_BM;                     // [4][32] of B, by tile
    unsigned *rmax = (unsigned *)(eb + 4 * SU_BN);  // [2][4][32]
    uint64_t *bars = (uint64_t *)(rmax + 2 * 4 * 32);
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
        ptx::mbar_init(a_full, SU_CONV);
        ptx::mbar_init(a_empty, 1);
        ptx::mbar_init(drain, 1);
        *abort_flag = 0;
        ptx::fence_mbarrier_init();
    }
    if (warp == 12) {
        ptx::tmem_alloc(tmem_slot, SU_TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;

    if (warp >= 8 && warp < 12) {
        // ------------------------------------------------ operand slices
        const int cw = warp - 8;
        int tile = 0, item = 0, rp = 0;
        SliceItems it(a);
        // 32 rows starting at row0: exponents to ex[0..31], slices to dst
        auto load = [&](const double *src, long rs, long ks, int row0, int rows, double (&v)[16]) {
            const double *p = src + (row0 + lane) * rs + 16 * cw * ks;
            const bool in = row0 + lane < rows;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = in && 16 * cw + i < a.k ? p[i * ks] : 0.0;
        };
        auto convert = [&](const double (&v)[16], int *ex, uint8_t *dst, int slice_bytes, int row) {
            unsigned mx = 0;
#pragma unroll
            for (int i = 0; i < 16; ++i) mx = max(mx, (unsigned)__double2hiint(v[i]) & 0x7FFFFFFFu);
            unsigned *r = rmax + rp * 128;
            rp ^= 1;
            r[cw * 32 + lane] = mx;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const int e = (int)(max(max(r[lane], r[32 + lane]), max(r[64 + lane], r[96 + lane])) >> 20);
            if (cw == 0) ex[lane] = e == 0x7FF ? SU_NONFINITE : e;
            su_write_digits(v, e, dst, slice_bytes, row, cw);
        };
        // all four warps go on or none does: they meet at barriers below
        auto wait_all = [&](uint64_t *bar, uint32_t parity) {
            uint32_t all, mine = ptx::wait_parity(bar, parity, abort_flag, a.wait_budget_ns) ? 1 : 0;
            asm volatile(
                "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred q, 2, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
                : "=r"(all)
                : "r"(mine)
                : "memory");
            return all != 0;
        };
        for (int id = blockIdx.x; id < a.items && ok; id += gridDim.x, ++item) {
            int t0, t1;
            it.find(a, id, t0, t1);
            double v[16];
            load(a.A, a.a_rs, a.a_ks, it.rb * SU_BM, a.m, v);
            if (!(ok = wait_all(a_empty, (item & 1) ^ 1))) break;
#pragma unroll 1
            for (int g = 0; g < 4; ++g) {
                double nx[16];
                if (g < 3) load(a.A, a.a_rs, a.a_ks, it.rb * SU_BM + 32 * (g + 1), a.m, nx);
                else load(a.B, a.b_rs, a.b_ks, t0 * SU_BN, a.n, nx);
                convert(v, ea + (item & 3) * SU_BM + 32 * g, sA, SU_SLICE_A, 32 * g + lane);
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = nx[i];
            }
            ptx::fence_proxy_async_smem();
            ptx::mbar_arrive(a_full);
            for (int t = t0; t < t1; ++t, ++tile) {
                const int buf = tile & 1;
                if (!(ok = wait_all(&b_empty[buf], ((tile >> 1) & 1) ^ 1))) break;
                double nx[16];
                if (t + 1 < t1) load(a.B, a.b_rs, a.b_ks, (t + 1) * SU_BN, a.n, nx);
                convert(v, eb + (tile & 3) * SU_BN, sB + buf * SU_B_BYTES, SU_SLICE_B, lane);
                ptx::fence_proxy_async_smem();
                ptx::mbar_arrive(&b_full[buf]);
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = nx[i];
            }
        }
    } else if (warp == 12) {
        // ---------------------------------------------------- MMA issuer
        if (ptx::elect_one()) {
            int tile = 0, item = 0;
            SliceItems it(a);
            const int ks = (a.k + 15) / 16;
            for (int id = blockIdx.x; id < a.items && ok; id += gridDim.x, ++item) {
                int t0, t1;
                it.find(a, id, t0, t1);
                ok = ptx::wait_parity(a_full, item & 1, abort_flag, a.wait_budget_ns);
                for (int t = t0; t < t1 && ok; ++t, ++tile) {
                    const int buf = tile & 1;
                    const uint32_t par = (tile >> 1) & 1;
                    ok = ptx::wait_parity(&acc_empty[buf], par ^ 1, abort_flag, a.wait_budget_ns) &&
                         ptx::wait_parity(&b_full[buf], par, abort_flag, a.wait_budget_ns);
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint32_t d = tmem_base + (uint32_t)buf * SU_ACC_STRIDE;
                    const uint32_t aA = ptx::smem_u32(sA), aB = ptx::smem_u32(sB + buf * SU_B_BYTES);
                    for (int k = 0; k < ks; ++k) {
                        const uint64_t bd = ptx::make_sdesc_k128(aB + k * 32);
#pragma unroll
                        for (int s = 0; s < SU_S; ++s)
                            ptx::mma_f16_ss(d + s * SU_BN, ptx::make_sdesc_k128(aA + s * SU_SLICE_A + k * 32), bd,
                                            ptx::make_idesc(SU_BM, SU_BN * (SU_S - s), ptx::FMT_F16), (k | s) ? 1u : 0u);
                    }
                    ptx::mma_commit(&b_empty[buf]);
                    ptx::mma_commit(&acc_full[buf]);
                }
                if (ok) ptx::mma_commit(a_empty);
            }
            // every MMA issued has read its operands before the CTA ends
            ptx::mma_commit(drain);
            volatile int never = 0;
            ptx::wait_parity(drain, 0, &never, a.wait_budget_ns);
        }
    } else {
        // ------------------------------------------------------ epilogue
        const int quarter = warp & 3, chalf = warp >> 2;
        int tile = 0, item = 0;
        SliceItems it(a);
        for (int id = blockIdx.x; id < a.items && ok; id += gridDim.x, ++item) {
            int t0, t1;
            it.find(a, id, t0, t1);
            const int rl = quarter * 32 + lane, row = it.rb * SU_BM + rl;
            for (int t = t0; t < t1 && ok; ++t, ++tile) {
                const int buf = tile & 1;
                const uint32_t tb = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * SU_ACC_STRIDE;
                const int col0 = t * SU_BN + 16 * chalf;
                double *crow = a.C + row + (long)col0 * a.ldc;
                auto inside = [&](int j) { return row < a.m && col0 + j < a.n && (!a.lower || row >= col0 + j); };
                double c[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) c[j] = inside(j) ? crow[(long)j * a.ldc] : 0.0;
                ok = ptx::wait_parity(&acc_full[buf], (tile >> 1) & 1, abort_flag, a.wait_budget_ns);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                ptx::tc_fence_after();
                const int er = ea[(item & 3) * SU_BM + rl];
                const int *ec = eb + (tile & 3) * SU_BN + 16 * chalf;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t r[SU_S][8];
#pragma unroll
                    for (int d = 0; d < SU_S; ++d) ptx::tmem_ld_32x32b_x8(tb + d * SU_BN + 16 * chalf + 8 * h, r[d]);
                    int ev[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) ev[j] = er + ec[8 * h + j];
                    ptx::tmem_ld_wait();
                    if (h == 1) {
                        ptx::tc_fence_before();
                        ptx::mbar_arrive(&acc_empty[buf]);
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        int s[SU_S];
#pragma unroll
                        for (int d = 0; d < SU_S; ++d) s[d] = (int)__uint_as_float(r[d][j]);
                        // sum of s[d] 2^{8 (5 - d)}, d = 0 .. 6, the last one rounded off
                        const long long hi = (long long)s[0] * 65536 + (s[1] * 256 + s[2]);
                        const long long lo = (long long)s[3] * 65536 + (s[4] * 256 + s[5] + ((s[6] + 128) >> 8));
                        const int e = ev[j];
                        double val = su_to_double((hi << 24) + lo, e);
                        if (e >= SU_NONFINITE) val = __longlong_as_double(0x7FF8000000000000ll);
                        if (inside(8 * h + j)) crow[(long)(8 * h + j) * a.ldc] = c[8 * h + j] - val;
                    }
                }
            }
        }
    }
    if (!ok) {
        if (!*abort_flag && a.err) atomicCAS(a.err, 0, SU_ERR_TIMEOUT);
        *abort_flag = 1;
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    if (warp == 12) ptx::tmem_dealloc(tmem_base, SU_TMEM_COLS);
}

} // namespace gb300
