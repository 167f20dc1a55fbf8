// Persistent batched SPD solve: one cooperative launch factors and solves
// many independent systems of different sizes (n <= 1024), FP32 blocked
// Cholesky + FP64 iterative refinement.
//
// All systems go through the same phases together, a grid barrier between
// two phases, so that a large system's work is spread over the GPU instead of
// being one CTA's latency (a system of order 1024 took 17 ms alone in its CTA,
// the time of a whole batch of 1024 systems):
//   convert   W = fp32(lower A), row sums of |A|; task = 64 rows of a system
//   step k    panel: the NB columns from k NB on; task = 64 rows below the
//             diagonal block, which every task factors for itself together
//             with its rows (chol_panel.cuh); the factored block goes to a
//             scratch tile, since others still read the unfactored one
//             update: W_ij -= L_i L_j^T; task = 64 x 64 tile of the trailing
//             triangle (or the scratch tile's copy to W)
//   round r   solve: task = one system in one CTA: backward error of the last
//             solution, x += L^-T L^-1 r in shared memory
//             residual: r = b - A x; task = 64 rows of a system
// Systems are sorted by order, largest first, in size buckets with a block
// width NB each (16, 32 or 64, the tuned parameter); a phase's tasks are found
// from the number of systems of a bucket larger than a given order.  Every
// task is a fixed sequence of operations on its system's data, so a system's
// result does not depend on which other systems share the launch.
//
// The residual of a system with n nrhs <= BAT_DF_TERMS runs in double-float
// arithmetic on the FP32 pipe (A split per element, X split once per task into
// shared memory, FP64 flush every 128 terms; ~2^-47 relative per block): the
// FP64 pipe is 64 times slower.  Larger ones, with seven or eight right-hand
// sides, keep FP64 FMAs (64 systems of order 900 to 1024 with eight: 4.99 ms against
// 3.94 in double-float, whose backward error is off by some 40 2^-53 there; with six
// 3.89 ms).
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "chol_panel.cuh"
#include "df_arith.cuh"
#include "tile64.cuh"

namespace gb300 {

constexpr int BAT_THREADS = 256;
constexpr int BAT_MAXN = 1024;
constexpr int BAT_MAXRHS = 8;
constexpr int BAT_DF_TERMS = 6688;        // n nrhs up to which the residual may be double-float
constexpr int BAT_BUCKETS = 6;            // n <= 32, 64, 128, 256, 512, 1024
constexpr int BAT_GRAIN = 16;             // cnt is kept for every multiple of this order
constexpr int BAT_CNT = BAT_MAXN / BAT_GRAIN + 1;

// W's leading dimension: columns start 16-byte aligned
__host__ __device__ __forceinline__ int bat_ldw(int n) { return (n + 3) & ~3; }

struct BatchedSystem {
    int n, index;              // order, position in the caller's arrays
    long long a_off, b_off;    // the caller's offsets (elements of A; of B and X)
    long long w_off, r_off;    // W (floats, n columns of bat_ldw(n)) and R (doubles)
};

// Per-system state, by sorted position.
struct BatchedState {
    unsigned long long anorm;               // ||A||_inf as FP64 bits
    unsigned long long rmax[BAT_MAXRHS];    // max |r| of the last residual, FP64 bits
    double xmax[BAT_MAXRHS], bmax[BAT_MAXRHS];
    int info, done;
};

struct BatchedArgs {
    int nsys, nrhs, max_iter, steps;
    double tol;
    unsigned wait_us;           // limit of a wait inside a panel
    const BatchedSystem *sys;   // [nsys] largest first
    BatchedState *state;        // [nsys], zeroed
    const int *cnt;             // [BAT_BUCKETS][BAT_CNT]: systems of the bucket with n > 16 v
    int first[BAT_BUCKETS];     // sorted position of the bucket's first system
    int nb[BAT_BUCKETS];        // block width
    const double *A, *B;
    double *X;
    float *W;
    float *D;                   // [nsys] 64 x 64 scratch tiles
    double *R;
    int *status;                // [nsys] by caller's index: corrections (>= 0), -(info), -1000 not converged
    double *berr;               // [nsys] final max backward error
    unsigned *active;           // [3] systems still iterating, in turn; zeroed
};

// Task t of a phase as (system, i, j); t is reduced by the tasks passed over.
struct BatTask {
    int pos, i, j, k0, nb;
};

__device__ __forceinline__ int bat_count(const int *cnt, int b, int v)
{
    return v >= BAT_MAXN ? 0 : cnt[b * BAT_CNT + v / BAT_GRAIN];
}

// 64-row blocks of every system: i-th block of the systems with n > 64 i
__device__ __forceinline__ bool bat_find_rows(const BatchedArgs &a, const int *cnt, int t, BatTask &o)
{
    for (int b = BAT_BUCKETS - 1; b >= 0; --b)
        for (int i = 0;; ++i) {
            const int c = bat_count(cnt, b, 64 * i);
            if (c == 0) break;
            if (t < c) {
                o.pos = a.first[b] + t;
                o.i = i;
                return true;
            }
            t -= c;
        }
    return false;
}

// panel of step k: i = 0 the diagonal block alone, i > 0 with the i-th 64 rows below it
__device__ __forceinline__ bool bat_find_panel(const BatchedArgs &a, const int *cnt, int k, int t, BatTask &o)
{
    for (int b = BAT_BUCKETS - 1; b >= 0; --b) {
        const int nb = a.nb[b], k0 = k * nb;
        for (int i = 0;; ++i) {
            const int c = bat_count(cnt, b, i == 0 ? k0 : k0 + nb + 64 * (i - 1));
            if (c == 0) break;
            if (t < c) {
                o.pos = a.first[b] + t;
                o.i = i;
                o.k0 = k0;
                o.nb = nb;
                return true;
            }
            t -= c;
        }
    }
    return false;
}

// update of step k: i = -1 the diagonal block's copy, else tile (i, j) of the trailing triangle
__device__ __forceinline__ bool bat_find_update(const BatchedArgs &a, const int *cnt, int k, int t, BatTask &o)
{
    for (int b = BAT_BUCKETS - 1; b >= 0; --b) {
        const int nb = a.nb[b], k0 = k * nb;
        for (int i = -1;; ++i) {
            const int c = bat_count(cnt, b, i < 0 ? k0 : k0 + nb + 64 * i), tiles = i < 0 ? 1 : i + 1;
            if (c == 0) break;
            if (t < c * tiles) {
                o.pos = a.first[b] + t % c;
                o.i = i;
                o.j = t / c;
                o.k0 = k0;
                o.nb = nb;
                return true;
            }
            t -= c * tiles;
        }
    }
    return false;
}

__device__ __forceinline__ double bat_warp_max(double m)
{
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}

// shared memory of a CTA: the widest phase's
template <int NR> struct BatSmem {
    static constexpr size_t TILES = 2 * DC_B * DC_LD * sizeof(float);
    static constexpr size_t PAN = sizeof(CpPanel<float, 2>);
    // solve: right-hand sides, diagonal block, its inverse pivots, the block's rows
    static constexpr size_t SOLVE = ((size_t)NR * BAT_MAXN + CP_W * CP_LP + CP_W + 8 * CP_LP) * sizeof(float);
    // residual: X split (or X), partial sums
    static constexpr size_t RES = (size_t)NR * BAT_MAXN * sizeof(float2) + 4 * 64 * NR * sizeof(double);
    static constexpr size_t M1 = TILES > PAN ? TILES : PAN, M2 = SOLVE > RES ? SOLVE : RES;
    static constexpr size_t BYTES = M1 > M2 ? M1 : M2;
};

// df_split_scaled for the usual exponents without branches
__device__ __forceinline__ float2 bat_split(double a, int ea)
{
    const uint32_t whi = (uint32_t)__double2hiint(a), wlo = (uint32_t)__double2loint(a);
    const int fe = (int)((whi >> 20) & 0x7FF) - (896 + ea);  // biased FP32 exponent of a 2^-ea
    if ((unsigned)(fe - 53) >= 202u) return df_split_scaled(a, ea);
    const uint32_t sign = whi & 0x80000000u;
    const float r = __uint2float_rn(wlo & 0x1FFFFFFFu);  // the 29 bits below the high part's 24
    return make_float2(__uint_as_float(sign | ((uint32_t)fe << 23) | (__funnelshift_l(wlo, whi, 3) & 0x7FFFFFu)),
                       __uint_as_float(sign | __float_as_uint(__fmul_rn(r, __uint_as_float((uint32_t)(fe - 52) << 23)))));
}

// v as (float)v gives it, by bit operations where the result is a normal number
// (a conversion holds the FP64 pipe)
__device__ __forceinline__ float bat_to_float(double v)
{
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    if (((hi >> 20) & 0x7FF) - 897u > 253u) return (float)v;
    uint32_t f = __funnelshift_l(lo, hi & 0x7FFFFFFFu, 3) - (896u << 23);  // truncated, then to nearest even
    f += (lo & 0x1FFFFFFFu) + (f & 1) > 0x10000000u ? 1u : 0u;
    return __uint_as_float(f | (hi & 0x80000000u));
}

// ---- convert: 64 rows of one system.  A row's sum is taken in 64-bit integers,
// units of 2^-54 of the largest diagonal element's binade, which bounds the
// elements of an SPD matrix: an element's rounding is 2^-55, below that of an
// FP64 addition to a sum of that size, and the largest sum is no smaller.  Rows
// with a larger element (or of a matrix without a finite diagonal) are added in
// FP64.  (FP64 additions and conversions, one each per element, took 530 us for
// 1024 systems: the FP64 pipe's time.)
__device__ void bat_convert(const BatchedArgs &a, const BatTask &t, double *red)
{
    const BatchedSystem s = a.sys[t.pos];
    const int n = s.n, ldw = bat_ldw(n), row = 64 * t.i + (threadIdx.x & 63), cg = threadIdx.x >> 6;
    const double *A0 = a.A + s.a_off, *A = A0 + row;
    float *W = a.W + s.w_off + row;
    unsigned dm = 0;
    for (int i = threadIdx.x & 31; i < n; i += 32) dm = max(dm, (unsigned)__double2hiint(A0[(long)i * (n + 1)]) & 0x7FFFFFFFu);
    dm = __reduce_max_sync(0xffffffffu, dm);
    const int ex = dm >= 0x7FF00000u ? -1 : max((int)(dm >> 20), 1);  // biased; -1: every row in FP64
    unsigned long long F = 0;
    int wide = 0;  // an exponent above ex was met
    if (row < n)
        for (int c0 = cg; c0 < n; c0 += 64) {
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = c0 + 4 * u < n ? A[(long)(c0 + 4 * u) * n] : 0.0;
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const unsigned long long m = (unsigned long long)__double_as_longlong(v[u]);
                const int e = (int)(m >> 52) & 0x7FF, down = ex - max(e, 1);
                wide |= down;
                F += ((((m & 0xFFFFFFFFFFFFFull) | (e ? 0x10000000000000ull : 0ull)) << 3 >> min((unsigned)down, 63u)) + 1) >> 1;
                if (c0 + 4 * u <= row) W[(long)(c0 + 4 * u) * ldw] = bat_to_float(v[u]);
            }
        }
    double sum = ldexp(__ull2double_rn(F), ex - (1023 + 54));
    if (wide < 0) {
        sum = 0.0;
        for (int c = cg; c < n; c += 4) sum += fabs(A[(long)c * n]);
    }
    __syncthreads();
    red[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x < 64) {
        double m = (red[threadIdx.x] + red[64 + threadIdx.x]) + (red[128 + threadIdx.x] + red[192 + threadIdx.x]);
        m = bat_warp_max(isnan(m) ? 0.0 : m);
        if ((threadIdx.x & 31) == 0) atomicMax(&a.state[t.pos].anorm, (unsigned long long)__double_as_longlong(m));
    }
}

// ---- panel: diagonal block and (i > 0) 64 rows below it
__device__ void bat_panel(const BatchedArgs &a, const BatTask &t, CpPanel<float, 2> &pan, uint64_t (&bar)[16], uint32_t phase,
                          CpState &st)
{
    const BatchedSystem s = a.sys[t.pos];
    const int n = s.n, ld = bat_ldw(n), bk = min(t.nb, n - t.k0), r0 = t.k0 + t.nb + 64 * (t.i - 1), rows = t.i > 0 ? min(64, n - r0) : 0;
    float *W = a.W + s.w_off;
    const float *Dg = W + t.k0 + (long)t.k0 * ld;
    float *P = W + r0 + (long)t.k0 * ld;
    CpBlock<float> d, x;
    cp_each<float>(d, [&](float &v, int r, int c) {
        v = (r < bk && c <= r) ? __ldcg(Dg + r + (long)c * ld) : (r == c ? 1.0f : 0.0f);
    });
    cp_each<float>(x, [&](float &v, int r, int c) { v = (r < rows && c < bk) ? __ldcg(P + r + (long)c * ld) : 0.0f; });
    __syncthreads();  // pan of the previous task is free
    if (!cp_panel<float, 2>(d, x, pan, bar, phase, st, bk, &a.state[t.pos].info, t.k0, t.i == 0, a.wait_us))
        atomicMax(&a.state[t.pos].info, BAT_MAXN + 1);  // a wait ran out: the system is reported as failed
    if (t.i > 0) {
        cp_each<float>(x, [&](float &v, int r, int c) {
            if (r < rows && c < bk) P[r + (long)c * ld] = v;
        });
    } else {
        float *D = a.D + (long)t.pos * (DC_B * DC_B);
        cp_each<float>(d, [&](float &v, int r, int c) {
            if (r != c) D[r + DC_B * c] = v;
        });
        st.diagonal([&](int c, float v) { D[c * (DC_B + 1)] = v; });
    }
}

// ---- update: one 64 x 64 tile of the trailing triangle, or the diagonal block's copy
__device__ void bat_update(const BatchedArgs &a, const BatTask &t, float *s0, float *s1)
{
    const BatchedSystem s = a.sys[t.pos];
    const int n = s.n, ld = bat_ldw(n), bk = min(t.nb, n - t.k0);
    float *W = a.W + s.w_off;
    if (t.i < 0) {
        const float *D = a.D + (long)t.pos * (DC_B * DC_B);
        for (int e = threadIdx.x; e < DC_B * DC_B; e += BAT_THREADS) {
            const int r = e & 63, c = e >> 6;
            if (r < bk && c <= r) W[(t.k0 + r) + (long)(t.k0 + c) * ld] = __ldcg(D + e);
        }
        return;
    }
    const int r0 = t.k0 + t.nb, i0 = r0 + 64 * t.i, j0 = r0 + 64 * t.j, ri = min(64, n - i0), rj = min(64, n - j0);
    const bool lower = t.i == t.j, whole = dc_whole(ri, rj, lower, true);
    float *C = W + i0 + (long)j0 * ld;
    const float *P = W + (long)t.k0 * ld;
    DcTile li, lj;
    float c[4][4];
    li.load(P + i0, ld, ri, bk, true);
    lj.load(P + j0, ld, rj, bk, true);
    dc_sub_load(C, ld, ri, rj, lower, whole, c);
    __syncthreads();  // the previous task's operands are free
    li.store(s0);
    lj.store(s1);
    __syncthreads();
    float acc[4][4] = {};
    dc_mma(s0, s1, acc, (bk + 7) & ~7);
    dc_sub_store(C, ld, ri, rj, lower, whole, c, acc);
}

// ---- solve: Y <- L^-T L^-1 Y in shared memory (ys[c * n + i]), 64 rows at a time
template <int NR> __device__ void bat_potrs(const float *W, int n, int ld, float *ys, float *Ls, float *inv, float *S)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nblk = (n + CP_W - 1) / CP_W;
    for (int e = tid; e < 8 * CP_LP; e += BAT_THREADS) S[e] = 0.0f;
    for (int pass = 0; pass < 2; ++pass)
        for (int bb = 0; bb < nblk; ++bb) {
            const bool fwd = pass == 0;
            const int j0 = CP_W * (fwd ? bb : nblk - 1 - bb), w = min(CP_W, n - j0);
            // the diagonal block (backward: reversed, so that the same forward
            // substitution solves with its transpose)
            float l[16], d = 1.0f;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r = tid & 63, c = 4 * i + (tid >> 6);
                l[i] = (r < w && c < r) ? W[(j0 + r) + (long)(j0 + c) * ld] : 0.0f;
            }
            if (tid < w) d = W[(j0 + tid) * (long)(ld + 1)];
            float dot[8][NR];
            if (!fwd) {
                // sums of the rows below over the block's columns, 8 columns per warp
#pragma unroll
                for (int u = 0; u < 8; ++u)
#pragma unroll
                    for (int c = 0; c < NR; ++c) dot[u][c] = 0.0f;
                const float *Wc = W + (long)(j0 + 8 * warp) * ld;
                for (int r = j0 + CP_W + lane; r < n; r += 128) {
                    float v[4][8];  // 32 loads in flight
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int u = 0; u < 8; ++u) v[k][u] = r + 32 * k < n ? Wc[r + 32 * k + (long)u * ld] : 0.0f;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int c = 0; c < NR; ++c) {
                            const float y = r + 32 * k < n ? ys[c * n + r + 32 * k] : 0.0f;
#pragma unroll
                            for (int u = 0; u < 8; ++u) dot[u][c] = fmaf(v[k][u], y, dot[u][c]);
                        }
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
#pragma unroll
                    for (int c = 0; c < NR; ++c)
                        for (int o = 16; o > 0; o >>= 1) dot[u][c] += __shfl_xor_sync(0xffffffffu, dot[u][c], o);
            }
            __syncthreads();  // the first block: ys and S are filled
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r = tid & 63, c = 4 * i + (tid >> 6);
                if (fwd) Ls[c * CP_LP + r] = l[i];
                else if (r < w && c < w) Ls[(w - 1 - r) * CP_LP + (w - 1 - c)] = l[i];
            }
            if (tid < CP_W) inv[fwd || tid >= w ? tid : w - 1 - tid] = 1.0f / d;
            if (fwd) {
                for (int e = tid; e < NR * CP_W; e += BAT_THREADS) {
                    const int c = e / CP_W, i = e % CP_W;
                    S[c * CP_LP + i] = i < w ? ys[c * n + j0 + i] : 0.0f;
                }
            } else {
#pragma unroll
                for (int u = 0; u < 8; ++u)
#pragma unroll
                    for (int c = 0; c < NR; ++c)
                        if (lane == (u * NR + c) % 32) {
                            const int i = 8 * warp + u;
                            if (i < w) S[c * CP_LP + w - 1 - i] = ys[c * n + j0 + i] - dot[u][c];
                            else S[c * CP_LP + i] = 0.0f;
                        }
                // past w the reversed block continues as the identity
                if (w < CP_W)
                    for (int e = tid; e < CP_W * CP_W; e += BAT_THREADS) {
                        const int r = e & 63, c = e >> 6;
                        if (r >= w || c >= w) Ls[c * CP_LP + r] = 0.0f;
                    }
            }
            __syncthreads();
            if (tid < 16 * 8) cp_slab_solve<8>(S, Ls, inv);
            __syncthreads();
            for (int e = tid; e < NR * CP_W; e += BAT_THREADS) {
                const int c = e / CP_W, i = e % CP_W;
                if (i < w) ys[c * n + j0 + i] = S[c * CP_LP + (fwd ? i : w - 1 - i)];
            }
            if (fwd)
                for (int i = j0 + CP_W + tid; i < n; i += BAT_THREADS) {
                    float acc[NR], v[CP_W];  // a row's 64 loads in flight
                    const float *Wi = W + i + (long)j0 * ld;
#pragma unroll
                    for (int q = 0; q < CP_W; ++q) v[q] = Wi[(long)q * ld];
#pragma unroll
                    for (int c = 0; c < NR; ++c) acc[c] = 0.0f;
#pragma unroll
                    for (int q = 0; q < CP_W; q += 4)
#pragma unroll
                        for (int c = 0; c < NR; ++c) {
                            const Quad<float> y = *reinterpret_cast<const Quad<float> *>(S + c * CP_LP + q);
#pragma unroll
                            for (int u = 0; u < 4; ++u) acc[c] = fmaf(v[q + u], y.v[u], acc[c]);
                        }
#pragma unroll
                    for (int c = 0; c < NR; ++c) ys[c * n + i] -= acc[c];
                }
            __syncthreads();
        }
}

// One round of one system: the backward error of its solution (after the
// first round), then the next correction.
template <int NR> __device__ void bat_round(const BatchedArgs &a, int pos, int round, float *smem, double *red)
{
    const BatchedSystem s = a.sys[pos];
    BatchedState &st = a.state[pos];
    const int n = s.n, nrhs = a.nrhs, tid = threadIdx.x;
    if (__ldcg(&st.done)) return;
    const int info = round == 0 ? __ldcg(&st.info) : 0;
    if (info) {
        if (tid == 0) {
            a.status[s.index] = info > BAT_MAXN ? -1000 : -info;
            a.berr[s.index] = INFINITY;
            st.done = 1;
        }
        return;
    }
    if (round > 0) {
        const double anorm = __longlong_as_double((long long)__ldcg(&st.anorm));
        double worst = 0.0;
        for (int c = 0; c < nrhs; ++c) {
            const double rm = __longlong_as_double((long long)__ldcg(&st.rmax[c])), den = anorm * __ldcg(&st.xmax[c]) + __ldcg(&st.bmax[c]);
            worst = fmax(worst, den > 0 ? rm / den : (rm > 0 ? INFINITY : 0.0));
        }
        if (worst <= a.tol || round > a.max_iter) {
            __syncthreads();  // every thread has read done
            if (tid == 0) {
                a.status[s.index] = worst <= a.tol ? round - 1 : -1000;
                a.berr[s.index] = worst;
                st.done = 1;
            }
            return;
        }
    }
    float *ys = smem, *Ls = ys + NR * BAT_MAXN, *inv = Ls + CP_W * CP_LP, *S = inv + CP_W;
    const double *B = a.B + s.b_off, *R = a.R + s.r_off;
    double *X = a.X + s.b_off;
    __syncthreads();  // shared memory of the previous task is free
    for (int e = tid; e < NR * n; e += BAT_THREADS)
        ys[e] = e < nrhs * n ? (float)(round == 0 ? B[e] : __ldcg(R + e)) : 0.0f;
    bat_potrs<NR>(a.W + s.w_off, n, bat_ldw(n), ys, Ls, inv, S);
    for (int c = 0; c < nrhs; ++c) {
        double xm = 0.0, bm = 0.0;
        for (int i = tid; i < n; i += BAT_THREADS) {
            const int e = c * n + i;
            const double x = (round == 0 ? 0.0 : X[e]) + (double)ys[e];
            X[e] = x;
            xm = fmax(xm, fabs(x));
            if (round == 0) bm = fmax(bm, fabs(B[e]));
        }
        xm = bat_warp_max(xm);
        bm = bat_warp_max(bm);
        __syncthreads();
        if ((tid & 31) == 0) red[tid >> 5] = xm, red[8 + (tid >> 5)] = bm;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < BAT_THREADS / 32; ++w) xm = fmax(xm, red[w]), bm = fmax(bm, red[8 + w]);
            st.xmax[c] = xm;
            if (round == 0) st.bmax[c] = bm;
            st.rmax[c] = 0;
        }
    }
    if (tid == 0) atomicAdd(&a.active[round % 3], 1u);
}

// ---- residual: 64 rows of R = B - A X in double-float arithmetic on the
// FP32 pipe (A scaled by the exponent of ||A||_inf and split per element by bit
// operations, each column of X scaled by its own exponent) or by FP64 FMAs,
// thread = row and every fourth column, the four sums added in a fixed order.
template <int NR> __device__ void bat_residual(const BatchedArgs &a, const BatTask &t, float *smem)
{
    const BatchedSystem s = a.sys[t.pos];
    BatchedState &st = a.state[t.pos];
    if (__ldcg(&st.done)) return;
    const int n = s.n, nrhs = a.nrhs, tid = threadIdx.x;
    float2 *Xs = reinterpret_cast<float2 *>(smem);                       // [n][NR]
    double *part = reinterpret_cast<double *>(Xs + (size_t)NR * BAT_MAXN);  // [4][NR][64]
    const double *X = a.X + s.b_off, *B = a.B + s.b_off;
    int ex[NR];
#pragma unroll
    for (int c = 0; c < NR; ++c) ex[c] = c < nrhs ? df_scale_exp(__ldcg(&st.xmax[c])) : 0;
    const int ea = df_scale_exp(__longlong_as_double((long long)__ldcg(&st.anorm)));
    const bool fp64 = NR * BAT_MAXN > BAT_DF_TERMS && n * nrhs > BAT_DF_TERMS;
    double *Xd = reinterpret_cast<double *>(smem);  // fp64: [n][NR]
    __syncthreads();  // shared memory of the previous task is free
#pragma unroll
    for (int c = 0; c < NR; ++c)
        for (int k = tid; k < n; k += BAT_THREADS) {
            const double x = c < nrhs ? __ldcg(X + (long)c * n + k) : 0.0;
            if (fp64) Xd[k * NR + c] = x;
            else Xs[k * NR + c] = df_split_scaled(x, ex[c]);
        }
    __syncthreads();
    const int row = 64 * t.i + (tid & 63), kg = tid >> 6;
    const double *Ai = a.A + s.a_off + min(row, n - 1);
    double acc[NR];
#pragma unroll
    for (int c = 0; c < NR; ++c) acc[c] = 0.0;
    if (fp64)
        for (int j0 = kg; j0 < n; j0 += 32) {
            double av[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) av[u] = j0 + 4 * u < n ? Ai[(long)(j0 + 4 * u) * n] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (j0 + 4 * u >= n) break;
                const double *x = Xd + (j0 + 4 * u) * NR;
#pragma unroll
                for (int c = 0; c < NR; ++c) acc[c] = fma(av[u], x[c], acc[c]);
            }
        }
    for (int j0 = fp64 ? n : kg; j0 < n; j0 += 512) {  // 128 terms of this thread
        float sh[NR], sl[NR];
#pragma unroll
        for (int c = 0; c < NR; ++c) sh[c] = 0.0f, sl[c] = 0.0f;
        const int j1 = min(n, j0 + 512);
        for (int j = j0; j < j1; j += 32) {
            double av[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) av[u] = j + 4 * u < j1 ? Ai[(long)(j + 4 * u) * n] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float2 v = bat_split(av[u], ea);
                const float2 *x = Xs + min(j + 4 * u, n - 1) * NR;
#pragma unroll
                for (int c = 0; c < NR; ++c) df_mac(sh[c], sl[c], v.x, v.y, x[c].x, x[c].y);
            }
        }
#pragma unroll
        for (int c = 0; c < NR; ++c) acc[c] += ldexp((double)sh[c] + (double)sl[c], ea + ex[c]);
    }
#pragma unroll
    for (int c = 0; c < NR; ++c) part[(kg * NR + c) * 64 + (tid & 63)] = acc[c];
    __syncthreads();
    for (int e = tid; e < 64 * NR; e += BAT_THREADS) {
        const int c = e >> 6, i = 64 * t.i + (e & 63);
        double m = 0.0;
        if (c < nrhs && i < n) {
            const double *p = part + c * 64 + (e & 63);
            const double r = B[(long)c * n + i] - ((p[0] + p[64 * NR]) + (p[128 * NR] + p[192 * NR]));
            a.R[s.r_off + (long)c * n + i] = r;
            m = fabs(r);
        }
        m = bat_warp_max(isnan(m) ? 0.0 : m);  // a warp's elements are of one right-hand side
        if ((tid & 31) == 0 && c < nrhs) atomicMax(&st.rmax[c], (unsigned long long)__double_as_longlong(m));
    }
}

template <int NR> __global__ void __launch_bounds__(BAT_THREADS, 2) batched_dposv_kernel(const BatchedArgs a)
{
    extern __shared__ __align__(16) unsigned char bat_smem[];
    __shared__ int cnt[BAT_BUCKETS * BAT_CNT];
    __shared__ uint64_t bar[16];
    __shared__ double red[BAT_THREADS];
    __shared__ CpState st;
    float *smem = (float *)bat_smem;
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    for (int e = threadIdx.x; e < BAT_BUCKETS * BAT_CNT; e += BAT_THREADS) cnt[e] = a.cnt[e];
    cp_panel_init(bar);
    __syncthreads();
    BatTask t;
    for (int q = blockIdx.x; bat_find_rows(a, cnt, q, t); q += gridDim.x) bat_convert(a, t, red);
    grid.sync();
    uint32_t panels = 0;
    for (int k = 0; k < a.steps; ++k) {
        for (int q = blockIdx.x; bat_find_panel(a, cnt, k, q, t); q += gridDim.x)
            bat_panel(a, t, *(CpPanel<float, 2> *)bat_smem, bar, panels++ & 1, st);
        grid.sync();
        for (int q = blockIdx.x; bat_find_update(a, cnt, k, q, t); q += gridDim.x)
            bat_update(a, t, smem, smem + DC_B * DC_LD);
        grid.sync();
    }
    for (int round = 0;; ++round) {
        if (blockIdx.x == 0 && threadIdx.x == 0) a.active[(round + 1) % 3] = 0;  // counted in the next round
        for (int q = blockIdx.x; q < a.nsys; q += gridDim.x) bat_round<NR>(a, q, round, smem, red);
        grid.sync();
        if (__ldcg(&a.active[round % 3]) == 0) break;
        for (int q = blockIdx.x; bat_find_rows(a, cnt, q, t); q += gridDim.x) bat_residual<NR>(a, t, smem);
        grid.sync();
    }
}

} // namespace gb300
