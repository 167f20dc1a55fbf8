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

namespace gb300 {

constexpr int CP_W = 64;  // order of a leaf and width of a panel step

// four values of one row, read and written 16 bytes at a time
template <typename T> struct alignas(16) Quad {
    T v[4];
};

// 1 / sqrt(d) to about one ulp: the hardware approximation and one correction
// step, which keeps the pivot chain of the leaf short (a square root and a
// division cost several times as much).  Outside the normal range, and for
// d <= 0 or NaN, the plain functions give what the unblocked loop gives.
__device__ __forceinline__ float cp_rsqrt(float d)
{
    if (!(d >= 1.17549435e-38f && d <= 3.0e38f)) return 1.0f / sqrtf(d);
    const float r = rsqrtf(d);
    return fmaf(0.5f * r, fmaf(-d * r, r, 1.0f), r);
}
// r from the approximation with relative error below 2^-19, then
// r (1 + e/2 + 3 e^2/8) with e = 1 - d r^2: the next term is (5/16) e^3 < 2^-55
__device__ __forceinline__ double cp_rsqrt(double d)
{
    if (!(d >= 2.3e-308 && d <= 1.7e308)) return 1.0 / sqrt(d);
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d * r, r, 1.0);
    return fma(r * e, fma(0.375, e, 0.5), r);
}

template <typename T> __device__ __forceinline__ T cp_dot_sub(T c, const Quad<T> &a, const Quad<T> &b)
{
#pragma unroll
    for (int q = 0; q < 4; ++q) c = fma(-a.v[q], b.v[q], c);
    return c;
}

// ---------------------------------------------------------------------------
// Cholesky of the n x n (n <= 64) lower block A, in place, by one CTA of 8
// warps.  Lane = row (two rows per lane), warp w owns columns 4w .. 4w+3 and
// 32 + 4w .. 32 + 4w + 3, in registers.  The 64 columns go four at a time
// (16 steps, one barrier each): the warp that owns the step's columns fetches
// their 4 x 4 diagonal block with ten shuffles, every lane factors it for
// itself (no shuffle or barrier inside the pivot chain), solves its own two
// rows and publishes them; then every warp applies the rank-4 update to the
// columns it still has to the right.  Bound by the chain of 64 dependent
// pivots.  Same operations as the reference codelet loop
// (cholesky_kernels.c:329-342), four columns at a time; a non-positive (or
// NaN) pivot records info_base + its 1-based column in *info, first one wins.
// ---------------------------------------------------------------------------
// steps 8 G0 .. 8 G0 + 7 of the leaf (columns 32 G0 .. 32 G0 + 31)
template <typename T, int G0>
__device__ __forceinline__ void cp_leaf_steps(T (&a)[2][4][2], Quad<T> (*pan)[CP_W], int n, int *info, int info_base)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int steps = min(8, (n - 32 * G0 + 3) / 4);
#pragma unroll 1
    for (int ow = 0; ow < steps; ++ow) {
        Quad<T> *p = pan[ow & 1];
        if (warp == ow) {
            T d[4][4], r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) d[i][j] = __shfl_sync(0xffffffffu, a[G0][j][G0], 4 * ow + i);
            int bad = -1;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (!(d[j][j] > T(0)) && bad < 0) bad = j;
                r[j] = cp_rsqrt(d[j][j]);
#pragma unroll
                for (int i = j + 1; i < 4; ++i) d[i][j] *= r[j];
#pragma unroll
                for (int k = j + 1; k < 4; ++k)
#pragma unroll
                    for (int i = k; i < 4; ++i) d[i][k] = fma(-d[i][j], d[k][j], d[i][k]);
            }
            if (bad >= 0 && lane == 0 && info) {
                const int col = 32 * G0 + 4 * ow + bad;
                if (col < n) atomicCAS(info, 0, info_base + col + 1);
            }
#pragma unroll
            for (int h = G0; h < 2; ++h) {
                Quad<T> x;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    T v = a[G0][j][h];
#pragma unroll
                    for (int q = 0; q < j; ++q) v = fma(-x.v[q], d[j][q], v);
                    x.v[j] = v * r[j];
                    a[G0][j][h] = x.v[j];
                }
                p[32 * h + lane] = x;
            }
        }
        __syncthreads();
        Quad<T> li[2];
#pragma unroll
        for (int h = G0; h < 2; ++h) li[h] = p[32 * h + lane];
#pragma unroll
        for (int g = G0; g < 2; ++g) {
            if (g == G0 && warp <= ow) continue;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const Quad<T> lc = p[32 * g + 4 * warp + c];
#pragma unroll
                for (int h = g; h < 2; ++h) a[g][c][h] = cp_dot_sub(a[g][c][h], li[h], lc);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) potf2_leaf_kernel(int n, T *__restrict__ A, long lda, int *info, int info_base)
{
    __shared__ Quad<T> pan[2][CP_W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T a[2][4][2];  // [column group][column][row half]
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = 32 * h + lane, col = 32 * g + 4 * warp + c;
                // rows and columns past n continue the block as the identity
                a[g][c][h] = (h >= g && r < n && col <= r) ? A[r + (long)col * lda] : T(r == col ? 1 : 0);
            }
    cp_leaf_steps<T, 0>(a, pan, n, info, info_base);
    cp_leaf_steps<T, 1>(a, pan, n, info, info_base);
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = g; h < 2; ++h) {
                const int r = 32 * h + lane, col = 32 * g + 4 * warp + c;
                if (r < n && col <= r) A[r + (long)col * lda] = a[g][c][h];
            }
}

// ---------------------------------------------------------------------------
// B[m x n] <- B L^{-T}, L n x n lower non-unit: rows of B are independent, so
// a CTA takes SR rows through all n columns in one launch (left-looking over
// 64-column blocks, the solved part of its rows in shared memory).
//   update  block columns j: B_j -= X_{<j} L_{j,<j}^T, thread = one column
//           and every fourth k, SR accumulators, L read along its columns
//           (coalesced, from L2: every CTA reads all of L);
//   solve   16 lanes per row, 4 columns each: the owner of the next four
//           columns finishes them, shuffles pass them on (no barrier).
// SR: 16 rows, or 4 where 16 would leave most SMs without a CTA.
// ---------------------------------------------------------------------------
constexpr int CP_TRSM_MAXN = 1024;  // columns of one launch (shared memory: SR n elements)
constexpr int CP_LP = CP_W + 4;     // pitch of the staged diagonal block

template <typename T, int SR> constexpr size_t cp_trsm_smem(int n)
{
    return ((size_t)((n + CP_W - 1) / CP_W * CP_W) * SR + (size_t)CP_W * CP_LP + CP_W + 4 * CP_W * (SR + 1)) * sizeof(T);
}

template <typename T, int SR>
__global__ void __launch_bounds__(256) trsm_slab_kernel(int m, int n, const T *__restrict__ L, long ldl,
                                                        T *__restrict__ B, long ldb)
{
    extern __shared__ __align__(16) unsigned char cp_smem[];
    const int npad = (n + CP_W - 1) / CP_W * CP_W;
    T *Xs = (T *)cp_smem;                // [npad][SR]: solved rows, column by column
    T *Ls = Xs + (size_t)npad * SR;      // [64][CP_LP]: diagonal block, Ls[c * CP_LP + r] = L(r, c)
    T *inv = Ls + CP_W * CP_LP;          // [64]
    T *red = inv + CP_W;                 // [4][64][SR + 1]
    const int tid = threadIdx.x, col = tid & 63, kg = tid >> 6;
    const int r0 = blockIdx.x * SR;
    for (int j0 = 0; j0 < n; j0 += CP_W) {
        const int w = min(CP_W, n - j0);
        // the diagonal block (identity past w) and the block's right-hand sides
        for (int e = tid; e < CP_W * CP_W; e += 256) {
            const int r = e & 63, c = e >> 6;
            Ls[c * CP_LP + r] = (r < w && c < r) ? L[(j0 + r) + (long)(j0 + c) * ldl] : T(0);
        }
        if (tid < CP_W) inv[tid] = tid < w ? T(1) / L[(j0 + tid) + (long)(j0 + tid) * ldl] : T(1);
        T b[SR / 4];
#pragma unroll
        for (int i = 0; i < SR / 4; ++i) {
            const int e = tid + 256 * i, r = e % SR, c = e / SR;
            b[i] = (c < w && r0 + r < m) ? B[(r0 + r) + (long)(j0 + c) * ldb] : T(0);
        }
        if (j0 > 0) {
            T acc[SR];
#pragma unroll
            for (int r = 0; r < SR; ++r) acc[r] = T(0);
            const T *Lc = L + j0 + min(col, w - 1);
#pragma unroll 8
            for (int p = kg; p < j0; p += 4) {
                const T l = Lc[(long)p * ldl];
                const Quad<T> *x = reinterpret_cast<const Quad<T> *>(Xs + (size_t)p * SR);
#pragma unroll
                for (int q = 0; q < SR / 4; ++q) {
                    const Quad<T> xv = x[q];
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[4 * q + i] = fma(l, xv.v[i], acc[4 * q + i]);
                }
            }
#pragma unroll
            for (int r = 0; r < SR; ++r) red[(kg * CP_W + col) * (SR + 1) + r] = acc[r];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < SR / 4; ++i) {
            const int e = tid + 256 * i, r = e % SR, c = e / SR;
            T v = b[i];
            if (j0 > 0)
                v -= (red[(0 * CP_W + c) * (SR + 1) + r] + red[(1 * CP_W + c) * (SR + 1) + r]) +
                     (red[(2 * CP_W + c) * (SR + 1) + r] + red[(3 * CP_W + c) * (SR + 1) + r]);
            Xs[(size_t)(j0 + c) * SR + r] = v;
        }
        __syncthreads();
        if (tid < 16 * SR) {
            const int r = tid >> 4, l = tid & 15, src = tid & 16;
            // a warp is two rows of 16 lanes; SR >= 4 keeps whole warps here
            T x[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) x[c] = Xs[(size_t)(j0 + 4 * l + c) * SR + r];
#pragma unroll 2
            for (int s = 0; s < 16; ++s) {
                const T *D = Ls + (4 * s) * CP_LP + 4 * s;
                T y[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    T v = x[c];
#pragma unroll
                    for (int q = 0; q < c; ++q) v = fma(-y[q], D[q * CP_LP + c], v);
                    y[c] = v * inv[4 * s + c];
                }
                if (l == s)
#pragma unroll
                    for (int c = 0; c < 4; ++c) x[c] = y[c];
#pragma unroll
                for (int c = 0; c < 4; ++c) y[c] = __shfl_sync(0xffffffffu, y[c], src | s);
                if (l > s)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const Quad<T> lv = *reinterpret_cast<const Quad<T> *>(Ls + (4 * s + q) * CP_LP + 4 * l);
#pragma unroll
                        for (int c = 0; c < 4; ++c) x[c] = fma(-y[q], lv.v[c], x[c]);
                    }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) Xs[(size_t)(j0 + 4 * l + c) * SR + r] = x[c];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < SR / 4; ++i) {
            const int e = tid + 256 * i, r = e % SR, c = e / SR;
            if (c < w && r0 + r < m) B[(r0 + r) + (long)(j0 + c) * ldb] = Xs[(size_t)(j0 + c) * SR + r];
        }
    }
}

// ---------------------------------------------------------------------------
// Triangular solves with the finished factor (POTRS): per block of CP_SB rows
// one launch that solves the block (trsv_blk_kernel) and one that updates the
// rows still to come (trsv_upd_kernel), forward with L, backward with L^T.
//
// trsv_blk_kernel: C right-hand sides per CTA (8 warps).  The block goes in
// 32-row pieces: warp c solves column c's piece by shuffles (lane = row)
// while the CTA's loads of the piece's off-diagonal part are in flight, then
// thread = row (forward) or column (backward) applies them.  Bound by the
// chain of dependent rows.
// ---------------------------------------------------------------------------
constexpr int CP_SB = 256;

template <typename T, int C> constexpr size_t cp_trsv_smem(bool trans)
{
    return ((size_t)C * CP_SB + 32 * 33 + (trans ? (size_t)CP_SB * 33 : 0)) * sizeof(T);
}

template <typename T, int C, bool TRANS>
__global__ void __launch_bounds__(256) trsv_blk_kernel(int w, int nrhs, const T *__restrict__ L, long ldl,
                                                       T *__restrict__ B, long ldb)
{
    extern __shared__ __align__(16) unsigned char cp_smem[];
    T *xs = (T *)cp_smem;         // [C][CP_SB]
    T *Ld = xs + C * CP_SB;       // [32][33]: forward Ld[j][i] = L(i, j), backward Ld[j][i] = L(j, i)
    T *Lt = Ld + 32 * 33;         // backward: [CP_SB][33], Lt[c][i] = L(piece row i, c)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.x * C, nc = min(C, nrhs - c0);
    for (int e = tid; e < C * CP_SB; e += 256) {
        const int r = e % CP_SB, c = e / CP_SB;
        xs[e] = (r < w && c < nc) ? B[r + (long)(c0 + c) * ldb] : T(0);
    }
    const int np = (w + 31) / 32;
    for (int s = 0; s < np; ++s) {
        const int p0 = 32 * (TRANS ? np - 1 - s : s), pw = min(32, w - p0);
        // the off-diagonal part of this piece, in flight during the solve
        T l[32];
        if (!TRANS) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                l[j] = (tid >= p0 + 32 && tid < w) ? L[tid + (long)(p0 + j) * ldl] : T(0);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const int c = warp + 8 * j;
                l[j] = (c < p0 && lane < pw) ? L[(p0 + lane) + (long)c * ldl] : T(0);
            }
        }
        for (int e = tid; e < 32 * 32; e += 256) {
            const int i = e & 31, j = e >> 5;  // L(i, j) of the piece's diagonal block
            const T v = (i < pw && j <= i) ? L[(p0 + i) + (long)(p0 + j) * ldl] : T(i == j ? 1 : 0);
            Ld[TRANS ? i * 33 + j : j * 33 + i] = v;
        }
        __syncthreads();
        for (int c = warp; c < C; c += 8) {
            // the products are summed apart from the right-hand side, so that
            // each rounding is relative to their (smaller) sum
            const T v = xs[c * CP_SB + p0 + lane], d = T(1) / Ld[lane * 33 + lane];
            T acc = T(0);
            if (!TRANS) {
#pragma unroll 8
                for (int j = 0; j < 32; ++j) {
                    const T xj = __shfl_sync(0xffffffffu, (v - acc) * d, j);
                    if (lane > j) acc = fma(Ld[j * 33 + lane], xj, acc);
                }
            } else {
#pragma unroll 8
                for (int j = 31; j >= 0; --j) {
                    const T xj = __shfl_sync(0xffffffffu, (v - acc) * d, j);
                    if (lane < j) acc = fma(Ld[j * 33 + lane], xj, acc);
                }
            }
            xs[c * CP_SB + p0 + lane] = (v - acc) * d;
        }
        if (TRANS) {
#pragma unroll
            for (int j = 0; j < 32; ++j) Lt[(warp + 8 * j) * 33 + lane] = l[j];
        }
        __syncthreads();
        if (TRANS ? tid < p0 : (tid >= p0 + 32 && tid < w)) {
            if (TRANS) {
#pragma unroll
                for (int j = 0; j < 32; ++j) l[j] = Lt[tid * 33 + j];
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                T acc[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[j & 3] = fma(l[j], xs[c * CP_SB + p0 + j], acc[j & 3]);
                xs[c * CP_SB + tid] -= (acc[0] + acc[1]) + (acc[2] + acc[3]);
            }
        }
        __syncthreads();
    }
    for (int e = tid; e < C * CP_SB; e += 256) {
        const int r = e % CP_SB, c = e / CP_SB;
        if (r < w && c < nc) B[r + (long)(c0 + c) * ldb] = xs[e];
    }
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
