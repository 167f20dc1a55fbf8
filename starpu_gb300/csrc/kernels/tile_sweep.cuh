// Single-launch triangular sweeps of the mixed solve's FP32 correction solve
// (POTRS with the factor L: L y = b, then L^T x = y) in tile rows of the
// factorisation's tile order nb, with the explicitly inverted nb x nb
// diagonal tiles the factorisation leaves behind.  The chain of dependent
// steps is n / nb long (32 at n = 32768, nb = 1024) instead of n / 64.
//
// Persistent CTAs take tasks by ticket, in solve order.  Tile row u of the
// solve order (u = T forward, T = ntiles - 1 - u backward) has, for each of
// its 32-row slabs s:
//   u products   P_{u,v,s} = L_{slab, tile v} y_v for the earlier tile rows v
//                (backward: (L_{v, slab})^T x_v), each waiting only for tile
//                row v to be solved, written to its own partial block;
//   one diagonal task: s_s = b_s - sum_{v < u - 1} P_{u,v,s} (v in order:
//                deterministic), published (Z rows, zcount[u]) while tile row
//                u - 1 is still being solved; then, with z = s - P_{u,u-1},
//                y_s = (L_TT^-1)_{slab, 0..slab end} z_T (backward the
//                transposed inverse), stored in place of b (ycount[u]).
// Tickets run over the products of tile row u (v ascending, slabs inner),
// then its diagonal tasks, then tile row u + 1.  The products of a tile row
// therefore spread over all CTAs, and the chain of a tile row is one product
// with the newest tile row, one product with the inverse and the two
// hand-overs between them.  A CTA waits only on tasks with smaller tickets: the
// s of a tile row are claimed one by one, normally one by each diagonal task,
// but a waiting task claims those that nobody works on.  While it works on a
// product a CTA holds the next ticket too, in long tile rows the next two
// (operands are loaded meanwhile); the smallest unfinished ticket is always
// being worked on, so the sweep cannot deadlock however few CTAs run at a time
// and however they are scheduled beside other kernels.  Every wait is bounded by a %globaltimer budget;
// on timeout the CTA records an error and stops waiting, so the launch ends.
//
// The products M (32 x K) V (K x 16), K <= nb, run on the tensor cores with
// warp-level m16n8k8 TF32 MMAs, three per tile on the split x = hi + lo of
// both operands (about 21 significant bits, the FP32 solve's own accuracy).
// (A 32-row slab and 16 right-hand sides are below the smallest tcgen05 tile,
// and the chain of the sweep wants the accumulator in registers: the
// warp-level MMA is the instruction that fits.)  Of every 8 W columns, W the
// warps of a CTA, a warp takes 8; a slab has at most 64 W columns, so that a
// thread holds its whole share of M, 64 floats, in registers, in the layout of
// the MMA's fragment: M does not depend on the flag the task waits for, is
// loaded before the wait (during the previous task's product where that is
// one), and a task's latency behind the flag is one read of V from L2, 8 MMA
// steps a warp and the sum over the warps.  V (16 floats per row, kept
// row-major beside the column-major result) goes through shared memory by
// cp.async, each warp reading back only the rows that it loaded.
//
// Against a 6-stage cp.async ring for both operands, 8 warps, two rounded
// conversions a split and z exchanged on the chain: a product of 32 x 1024 took
// 8 us behind its flag (two CTAs on an SM 13 us) and a sweep 19 us at n =
// 1024, 115 at 4096, 1170 at 32768.  So: 3 us, and 15, 60 and 760 us (a
// sweep's factor is 2.1 GB there: 0.32 ms of DRAM time; what is left is the
// products' own latency with one CTA of 128 registers a thread on an SM).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gb300 {

constexpr int TSW_SLAB = 32;  // rows per task
constexpr int TSW_STEPS = 8;  // MMA steps (8 columns a warp) of a whole task
constexpr int TSW_VP = 20;    // pitch of V's rows: the 64-bit fragment loads of a half-warp hit 32 banks

// Warps of a CTA for tile order nb: the fewest that hold a slab of nb columns,
// so that as many CTAs as the register file allows share an SM (16 warps: one).
inline int tsw_warps(int nb) { return nb <= 256 ? 4 : nb <= 512 ? 8 : 16; }
// Dynamic shared memory: two V buffers and the warps' 32 x 16 blocks.
inline int tsw_dsmem(int warps) { return warps * (2 * 8 * TSW_STEPS * TSW_VP + 512) * 4; }

struct TileSweepArgs {
    int n, nrhs, nb;
    int ntiles, spt;  // tile rows; slabs per tile row (nb / 32)
    unsigned total;   // tasks: spt * ntiles * (ntiles + 1) / 2
    const float *L;
    long ldl;
    const float *Dinv;  // tile T's inverse at Dinv + T * dstride, leading dimension ldd
    long ldd, dstride;
    float *B;  // right-hand sides in, solution out (n x nrhs, ld ldb)
    long ldb;
    float *Zt;  // s of the tile rows, row-major n x 16
    float *Yt;  // solved rows (y forward, x backward), row-major n x 16: the products' right-hand operand
    float *Zp;  // partial products: pair (u, v < u) at Zp + (u (u - 1) / 2 + v) * nb * 16, row-major nb x 16
    const float *DinvT;  // optional: tile T's inverse transposed at DinvT + T * dstride (ld ldd)
    unsigned *ticket;
    // per tile row of the solve order, zero at launch.  pcount: products of the
    // tile rows before the newest in the low half, of the newest in the high;
    // zcount: slabs whose s is there in the low half, slabs claimed in the high
    int *zcount, *ycount, *pcount;
    int *err;
    unsigned long long budget_ns;
    int vec_l, vec_d;  // L, the inverses: columns start 16-byte aligned
    // backward sweep: 1 when the strictly upper part of L's storage holds L^T
    // outside the diagonal tiles (L(j, i) also at (i, j)), so the slab's rows
    // of L^T are read column by column like the forward sweep's operands
    int upper;
};

// Bytes of scratch a sweep pair needs: Zt and Yt (n x 16 each), the partial
// products of every pair of tile rows, and the 3 ntiles + 1 counters.
inline size_t tsw_scratch_bytes(int n, int nb, size_t *yt_off = nullptr, size_t *zp_off = nullptr,
                                size_t *cnt_off = nullptr)
{
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t nt = ((size_t)n + nb - 1) / nb;
    const size_t z = al((size_t)n * 16 * sizeof(float));
    const size_t zp = al(nt * (nt > 0 ? nt - 1 : 0) / 2 * (size_t)nb * 16 * sizeof(float));
    if (yt_off) *yt_off = z;
    if (zp_off) *zp_off = 2 * z;
    if (cnt_off) *cnt_off = 2 * z + zp;
    return 2 * z + zp + al((3 * nt + 1) * sizeof(int));
}

__device__ __forceinline__ void tsw_cp16(float *smem, const float *gmem, int src_bytes)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(gmem), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void tsw_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void tsw_cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ int tsw_ld_acquire(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint64_t tsw_timer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Thread 0 waits until the field (*cnt >> shift) & mask reaches target.  On
// timeout or an error seen elsewhere it stops waiting from then on (skip).
__device__ __forceinline__ void tsw_wait(const TileSweepArgs &a, const int *cnt, int shift, int mask, int target,
                                         bool &skip)
{
    auto there = [&] { return ((tsw_ld_acquire(cnt) >> shift) & mask) >= target; };
    if (skip || there()) return;
    const uint64_t t0 = tsw_timer();
    while (!there()) {
        if (*(volatile int *)a.err || tsw_timer() - t0 > a.budget_ns) {
            atomicCAS(a.err, 0, 1);
            skip = true;
            break;
        }
        __nanosleep(20);
    }
}

// Thread 0 waits until the s of every slab of a tile row is there (low half of
// *cnt; slabs claimed in the high half): -1.  Where some stay unclaimed for 20 us
// -- the CTAs that hold those diagonal tasks are not running yet, because other
// kernels hold their SMs -- it claims one more: its number.
__device__ __forceinline__ int tsw_wait_slabs(const TileSweepArgs &a, int *cnt, bool &skip)
{
    uint64_t t0 = 0;
    while (!skip) {
        const int w = tsw_ld_acquire(cnt);
        if ((w & 0xffff) >= a.spt) break;
        const uint64_t t = tsw_timer();
        if (t0 == 0) t0 = t;
        if (t - t0 > 20000 && (w >> 16) < a.spt) {
            const int slab = atomicAdd(cnt, 0x10000) >> 16;
            if (slab < a.spt) return slab;
        }
        if (*(volatile int *)a.err || t - t0 > a.budget_ns) {
            atomicCAS(a.err, 0, 1);
            skip = true;
        }
        __nanosleep(20);
    }
    return -1;
}

// Every thread's stores become visible with the count (raised by the last
// warp: the first goes on to the next wait).
__device__ __forceinline__ void tsw_publish(int *cnt, int add)
{
    __syncthreads();
    if (threadIdx.x == blockDim.x - 32) {
        __threadfence();
        atomicAdd(cnt, add);
    }
}

// The operand M of a task: rows x K (rows <= 32), element (r, p) at
//   TSW_VEC, TSW_ROWS  M[r + p * ldm]  (rows of L, of L^T's mirror or of an inverse);
//                      VEC: 32 rows and 16-byte aligned columns
//   TSW_TRANS          M[p + r * ldm]  (the transposed operand)
enum { TSW_VEC = 0, TSW_ROWS = 1, TSW_TRANS = 2 };
struct TswOp {
    const float *M;
    long ldm;
    int rows, K, mode;
    bool full;  // VEC and K = 64 W: no guards
};

// A thread's share of M: of step i the columns 2 t and 2 t + 1 of its warp's 8
// (g = lane / 4, t = lane % 4), rows 4 g + j (VEC: one 16-byte load; 8 lanes
// read a column's 128 bytes) or g + 8 j, j = 0 .. 3.  Rows past `rows` and
// columns past K are zero.
template <int W>
__device__ __forceinline__ void tsw_load_step(float (&m)[2][4], const TswOp &op, int i)
{
    const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int p = (i * W + warp) * 8 + 2 * t + h;
        if (op.mode == TSW_VEC) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p < op.K) x = __ldcg(reinterpret_cast<const float4 *>(op.M + 4 * g + (long)p * op.ldm));
            m[h][0] = x.x;
            m[h][1] = x.y;
            m[h][2] = x.z;
            m[h][3] = x.w;
        } else {
            const float *src = op.mode == TSW_ROWS ? op.M + g + (long)p * op.ldm : op.M + p + (long)g * op.ldm;
            const long step = op.mode == TSW_ROWS ? 8 : 8 * op.ldm;
#pragma unroll
            for (int j = 0; j < 4; ++j) m[h][j] = p < op.K && g + 8 * j < op.rows ? __ldcg(src + j * step) : 0.0f;
        }
    }
}
// The same for a full operand, at src = the thread's place in its first column.
template <int W>
__device__ __forceinline__ const float *tsw_full_src(const TswOp &op)
{
    const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    return op.M + 4 * g + (long)(warp * 8 + 2 * t) * op.ldm;
}
__device__ __forceinline__ void tsw_load_full(float (&m)[2][4], const float *src, long ldm)
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float4 x = __ldcg(reinterpret_cast<const float4 *>(src + h * ldm));
        m[h][0] = x.x;
        m[h][1] = x.y;
        m[h][2] = x.z;
        m[h][3] = x.w;
    }
}
template <int W>
__device__ __forceinline__ void tsw_load(float (&m)[TSW_STEPS][2][4], const TswOp &op)
{
    if (op.full) {
        const float *src = tsw_full_src<W>(op);
#pragma unroll
        for (int i = 0; i < TSW_STEPS; ++i, src += 8 * W * op.ldm) tsw_load_full(m[i], src, op.ldm);
    } else {
#pragma unroll
        for (int i = 0; i < TSW_STEPS; ++i) tsw_load_step<W>(m[i], op, i);
    }
}
__device__ __forceinline__ int tsw_row(const TswOp &op, int g, int j) { return op.mode == TSW_VEC ? 4 * g + j : g + 8 * j; }

// The warp's own 8 rows of V (row-major, 16 floats) of every step into buf.
template <int W>
__device__ __forceinline__ void tsw_load_v(float *buf, const float *V, int K)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
#pragma unroll
    for (int i = 0; i < TSW_STEPS; ++i) {
        const int p = (i * W + warp) * 8 + r;
        if (i * W * 8 < K) tsw_cp16(buf + p * TSW_VP + 4 * q, p < K ? V + (long)p * 16 + 4 * q : V, p < K ? 16 : 0);
        tsw_cp_commit();
    }
}

// x = hi + lo for the TF32 product: hi rounded to nearest (half an ulp added
// to the magnitude), lo the rest with its bits below TF32 cut off: an error of
// at most 2^-23 |x|, as rounding it has.  Integer arithmetic: the conversion
// instruction takes a sub-partition's issue 5 clocks a warp.  A NaN whose hi
// overflows to zero stays NaN in lo.
__device__ __forceinline__ void tsw_split_tf32(float x, uint32_t &hi, uint32_t &lo)
{
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi)) & 0xffffe000u;
}

// d += a b for one 16 x 8 x 8 TF32 tile (warp-wide, FP32 accumulation)
__device__ __forceinline__ void tsw_mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                 "{%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// red[warp] (32 x 16, row-major) = the warp's share of M V, with V in vb (DIFF:
// V = sb - vb), M in m; m is refilled with `next` (refill) as it is used up,
// and the warp's rows of the next task's V follow where vnext is given.  The fragments' k slots t and t + 4 hold columns 2 t and 2 t + 1,
// their n = g the right-hand sides 2 g and 2 g + 1 of the two n tiles, so that
// V comes by 64-bit loads and a thread ends with four neighbouring right-hand
// sides of a row.
template <int W, bool DIFF>
__device__ __forceinline__ void tsw_product(float (&m)[TSW_STEPS][2][4], const TswOp &op, float *vb,
                                            const float *sb, float *red, bool refill, const TswOp &next,
                                            const float *vnext)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // All of m is waited for here, by an operation on each register: a refill
    // shares a scoreboard with loads of later steps, and a step that waited for
    // its own operand would wait for the refills of the steps before it (a
    // product 6 us instead of 3).
    unsigned any = 0;
#pragma unroll
    for (int i = 0; i < TSW_STEPS; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) any |= __float_as_uint(m[i][j >> 2][j & 3]);
    if (any == 0xffffffffu) __nanosleep(0);
    const bool full = refill && next.full;
    const float *src = tsw_full_src<W>(next);
    float acc[2][2][4] = {};  // m tile (rows j = 2 mt, 2 mt + 1), n tile
    auto step = [&](int i) {
        if (i * W * 8 < op.K) {
            __syncwarp();
            const int at = ((i * W + warp) * 8 + 2 * t) * TSW_VP + 2 * g;
            uint32_t bh[2][2], bl[2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float2 v = *reinterpret_cast<const float2 *>(vb + at + h * TSW_VP);
                if (DIFF) {
                    const float2 z = *reinterpret_cast<const float2 *>(sb + at + h * TSW_VP);
                    v.x = z.x - v.x;
                    v.y = z.y - v.y;
                }
                tsw_split_tf32(v.x, bh[0][h], bl[0][h]);
                tsw_split_tf32(v.y, bh[1][h], bl[1][h]);
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                uint32_t ah[4], al[4];  // (row, k): (g, t), (g + 8, t), (g, t + 4), (g + 8, t + 4)
#pragma unroll
                for (int q = 0; q < 4; ++q) tsw_split_tf32(m[i][q >> 1][2 * mt + (q & 1)], ah[q], al[q]);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    tsw_mma_tf32(acc[mt][nt], al, bh[nt]);  // the small terms first
                    tsw_mma_tf32(acc[mt][nt], ah, bl[nt]);
                    tsw_mma_tf32(acc[mt][nt], ah, bh[nt]);
                }
            }
        }
        if (full) {
            tsw_load_full(m[i], src, next.ldm);
            src += 8 * W * next.ldm;
        }
    };
    static_assert(TSW_STEPS == 8, "the waits below");
    tsw_cp_wait<7>(), step(0);
    tsw_cp_wait<6>(), step(1);
    tsw_cp_wait<5>(), step(2);
    tsw_cp_wait<4>(), step(3);
    tsw_cp_wait<3>(), step(4);
    tsw_cp_wait<2>(), step(5);
    tsw_cp_wait<1>(), step(6);
    tsw_cp_wait<0>(), step(7);
    if (refill && !full) {
#pragma unroll
        for (int i = 0; i < TSW_STEPS; ++i) tsw_load_step<W>(m[i], next, i);
    }
    if (vnext) {
        __syncwarp();  // the warp has read its rows of vb
        tsw_load_v<W>(vb, vnext, next.K);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(red + warp * 512 + tsw_row(op, g, j) * 16 + 4 * t) =
            make_float4(acc[j >> 1][0][2 * (j & 1)], acc[j >> 1][1][2 * (j & 1)], acc[j >> 1][0][2 * (j & 1) + 1],
                        acc[j >> 1][1][2 * (j & 1) + 1]);
}

// Element e of the 32 x 16 product: the warps' blocks in order.
template <int W>
__device__ __forceinline__ float tsw_sum(const float *red, int e)
{
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < W; ++w) s += red[w * 512 + e];
    return s;
}

// Task of ticket t: tile row u of the solve order (its tickets start at
// spt u (u + 1) / 2: u spt products, then spt diagonal tasks) and the rank r
// within the row (r < u spt: product with earlier tile row r / spt, slab
// r % spt; else diagonal task of slab r - u spt).
__host__ __device__ __forceinline__ void tsw_decode(unsigned t, int spt, int &u, unsigned &r)
{
    const unsigned q = t / (unsigned)spt;
    u = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
    while (u > 0 && (unsigned)u * (u + 1) / 2 > q) --u;
    while ((unsigned)(u + 1) * (u + 2) / 2 <= q) ++u;
    r = t - (unsigned)spt * ((unsigned)u * (u + 1) / 2);
}

struct TswTask {
    int u, v, s;      // tile row, earlier tile row (u: diagonal task), slab
    int r0, t0, kbT;  // first row of the slab, of the tile row; rows of the tile row
    int v0;           // first row of V in the row-major vectors
    TswOp op;
};

// k = the task of ticket `to`; k is that of ticket `from` when near
template <bool TRANS, int W>
__device__ __forceinline__ void tsw_task(const TileSweepArgs &a, unsigned from, unsigned to, bool near, TswTask &k)
{
    if (near && to - from <= 16u * (unsigned)a.spt) {  // a few steps on: no divisions
        for (k.s += (int)(to - from); k.s >= a.spt; k.s -= a.spt)
            if (++k.v > k.u) {
                ++k.u;
                k.v = 0;
            }
    } else {
        unsigned r;
        tsw_decode(to, a.spt, k.u, r);
        k.v = (int)(r / a.spt);
        k.s = (int)(r % a.spt);
    }
    const int T = TRANS ? a.ntiles - 1 - k.u : k.u, c0 = k.s * TSW_SLAB;
    k.t0 = T * a.nb;
    k.kbT = min(a.nb, a.n - k.t0);
    k.r0 = k.t0 + c0;
    k.op.rows = max(0, min(TSW_SLAB, k.kbT - c0));
    bool trans = false, vec;
    if (k.v < k.u) {
        const int j0 = (TRANS ? a.ntiles - 1 - k.v : k.v) * a.nb;
        k.v0 = j0;
        k.op.K = min(a.nb, a.n - j0);
        k.op.ldm = a.ldl;
        vec = a.vec_l != 0;
        trans = TRANS && !a.upper;
        k.op.M = trans ? a.L + j0 + (long)k.r0 * a.ldl : a.L + k.r0 + (long)j0 * a.ldl;
    } else {
        // forward: Dinv(slab rows, 0 .. slab end); backward: Dinv(slab start
        // .. kbT, slab columns)^T, from the transposed tiles where they are kept
        const float *D = a.Dinv + (long)T * a.dstride;
        k.op.ldm = a.ldd;
        vec = a.vec_d != 0;
        if (!TRANS) {
            k.v0 = k.t0;
            k.op.K = c0 + k.op.rows;
            k.op.M = D + c0;
        } else {
            trans = !a.DinvT;
            k.v0 = k.r0;
            k.op.K = k.kbT - c0;
            k.op.M = (trans ? D : a.DinvT + (long)T * a.dstride) + c0 + (long)c0 * a.ldd;
        }
    }
    k.op.mode = trans ? TSW_TRANS : vec && k.op.rows == TSW_SLAB ? TSW_VEC : TSW_ROWS;
    if (k.op.rows == 0) k.op.K = 0;
    k.op.full = k.op.mode == TSW_VEC && k.op.K == 8 * W * TSW_STEPS;
}

template <bool TRANS, int W>
__global__ void __launch_bounds__(32 * W, 16 / W) tile_sweep_kernel(TileSweepArgs a)
{
    constexpr int NT = 32 * W;
    extern __shared__ float4 tsw_dsmem_[];
    float *vb = reinterpret_cast<float *>(tsw_dsmem_);  // 8 W TSW_STEPS rows of TSW_VP floats
    float *sb = vb + 8 * W * TSW_STEPS * TSW_VP, *red = sb + 8 * W * TSW_STEPS * TSW_VP;
    __shared__ unsigned s_ticket;
    const int tid = threadIdx.x;
    bool skip = false;       // thread 0: a wait ran out
    int known = -1;          // the newest tile row known to be solved
    bool loaded = false;     // ticket t is taken, k is its task and m its operand
    bool have_v = false;     // ... and its V is on the way
    bool ahead = false;      // ticket tn is taken, too
    unsigned t = 0, tn = 0;
    float m[TSW_STEPS][2][4];
    TswTask k;
    auto take = [&] {
        __syncthreads();  // s_ticket has been read
        if (tid == 0) s_ticket = atomicAdd(a.ticket, 1u);
        __syncthreads();
        return s_ticket;
    };
    for (;;) {
        if (!loaded) {
            t = take();
            if (t >= a.total) return;
            tsw_task<TRANS, W>(a, 0, t, false, k);
            tsw_load<W>(m, k.op);
            have_v = ahead = false;
        }
        if (k.v < k.u) {
            if (!ahead) tn = take();
            if (known < k.v) {
                if (tid == 0) tsw_wait(a, &a.ycount[k.v], 0, 0x7fffffff, a.spt, skip);
                __syncthreads();
                known = k.v;
            }
            const TswTask c = k;
            if (!have_v) tsw_load_v<W>(vb, a.Yt + (long)c.v0 * 16, c.op.K);
            loaded = tn < a.total;
            if (loaded) tsw_task<TRANS, W>(a, t, tn, true, k);
            t = tn;
            // a further ticket only if the next task is a product of a tile
            // row with two rounds of them or more: it saves the ticket's and V's latency
            // a product (n = 32768: 860 us without, 730 with), but in a short
            // row delays a product the chain waits for (8192: 111 and 122 us)
            ahead = loaded && k.v < k.u && (unsigned)(k.u * a.spt) >= 2 * gridDim.x;
            have_v = ahead && k.v <= known;
            unsigned far = 0;
            if (tid == 0 && ahead) far = atomicAdd(a.ticket, 1u);
            tsw_product<W, false>(m, c.op, vb, sb, red, loaded, k.op, have_v ? a.Yt + (long)k.v0 * 16 : nullptr);
            if (tid == 0) s_ticket = far;
            __syncthreads();
            tn = s_ticket;
            float *P = a.Zp + ((long)c.u * (c.u - 1) / 2 + c.v) * (long)a.nb * 16 + (long)c.s * TSW_SLAB * 16;
#pragma unroll
            for (int e = tid; e < 512; e += NT) P[e] = tsw_sum<W>(red, e);
            tsw_publish(&a.pcount[c.u], c.v == c.u - 1 ? 0x10000 : 1);
            if (!loaded) return;
        } else {
            // s = b - the products of the tile rows before the newest, of the
            // next slab of the tile row that nobody has claimed
            if (tid == 0) {
                s_ticket = (unsigned)atomicAdd(&a.zcount[k.u], 0x10000) >> 16;
                if (k.u > 1) tsw_wait(a, &a.pcount[k.u], 0, 0xffff, (k.u - 1) * a.spt, skip);
            }
            __syncthreads();  // (red has been read, too)
            const float *P = a.Zp + (long)k.u * (k.u - 1) / 2 * (long)a.nb * 16;
            for (int slab = (int)s_ticket; slab >= 0;) {
                if (slab < a.spt) {
                    const int c0 = slab * TSW_SLAB;
#pragma unroll
                    for (int e = tid; e < 512; e += NT) {
                        const int r = c0 + (e >> 4), c = e & 15;
                        if (r < k.kbT && c < a.nrhs) {
                            const float b = __ldcg(&a.B[(long)(k.t0 + r) + (long)c * a.ldb]);
                            const float *Ps = P + (long)c0 * 16 + e;
                            float sum = 0.0f;
#pragma unroll 8
                            for (int v = 0; v < k.u - 1; ++v) sum += __ldcg(Ps + (long)v * a.nb * 16);
                            a.Zt[(long)(k.t0 + r) * 16 + c] = b - sum;
                        }
                    }
                    tsw_publish(&a.zcount[k.u], 1);
                } else {
                    __syncthreads();  // s_ticket has been read
                }
                if (tid == 0) s_ticket = (unsigned)tsw_wait_slabs(a, &a.zcount[k.u], skip);
                __syncthreads();
                slab = (int)s_ticket;
            }
            float *zb = k.u > 0 ? sb : vb;
            tsw_load_v<W>(zb, a.Zt + (long)k.v0 * 16, k.op.K);
            if (k.u > 0) {
                if (tid == 0) tsw_wait(a, &a.pcount[k.u], 16, 0x7fff, a.spt, skip);
                __syncthreads();
                tsw_load_v<W>(vb, P + (long)(k.u - 1) * a.nb * 16 + (long)(k.v0 - k.t0) * 16, k.op.K);
                tsw_product<W, true>(m, k.op, vb, sb, red, false, k.op, nullptr);
            } else {
                tsw_product<W, false>(m, k.op, vb, sb, red, false, k.op, nullptr);
            }
            __syncthreads();
#pragma unroll
            for (int e = tid; e < 512; e += NT) {
                const int r = e >> 4, c = e & 15;
                if (r < k.op.rows && c < a.nrhs) {
                    const float y = tsw_sum<W>(red, e);
                    a.B[(long)(k.r0 + r) + (long)c * a.ldb] = y;
                    a.Yt[(long)(k.r0 + r) * 16 + c] = y;
                }
            }
            tsw_publish(&a.ycount[k.u], 1);
            loaded = false;
        }
    }
}

} // namespace gb300
