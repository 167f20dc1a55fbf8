// SIMT (CUDA-core) dense kernels for the tiled Cholesky path, FP32 and FP64.
//
// These are the building blocks that the tile codelets and the whole-matrix
// drivers compose.  They replace, for the plain (non-tensor-core) precisions,
// the vendor calls the reference codelets make on the CUDA worker stream:
//   cublasSgemm(N,T)      examples/cholesky/cholesky_kernels.c:98
//   cublasSsyrk(L,N)      examples/cholesky/cholesky_kernels.c:177
//   cublasStrsm(R,L,T,N)  examples/cholesky/cholesky_kernels.c:258
//   cusolverDnSpotrf(L)   examples/cholesky/cholesky_kernels.c:354
// All matrices are column-major with an explicit leading dimension, exactly
// like the StarPU matrix interface (nx rows contiguous, ld >= nx).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

namespace gb300 {

// ---------------------------------------------------------------------------
// GEMM:  C[m x n] = beta*C + alpha * op(A)[m x k] * op(B)[k x n]
//   TA=false: op(A)(i,p) = A[i + p*lda]     TA=true: op(A)(i,p) = A[p + i*lda]
//   TB=false: op(B)(p,j) = B[p + j*ldb]     TB=true: op(B)(p,j) = B[j + p*ldb]
// LOWER (requires m == n, BM == BN): only blocks on/below the diagonal are
// launched (triangular grid) and only elements with i >= j are written.  This
// is the SYRK "L" update and the whole-trailing-matrix update.
// Each thread owns a TM x TN register tile split in two halves along both
// axes (rows h*BM/2 + tr*TM/2 + v) so shared-memory reads are vectorised and
// bank-conflict free, and global C accesses stay coalesced.
// ---------------------------------------------------------------------------
template <typename T> struct vec2_of;
template <> struct vec2_of<float> { typedef float2 type; };
template <> struct vec2_of<double> { typedef double2 type; };

// K split (kchunk > 0): blockIdx.z takes the K range [z*kchunk, (z+1)*kchunk)
// and writes its partial product to C + z*cstride (beta applies to each
// partial); a separate pass reduces the partials in a fixed order, so the
// result does not depend on scheduling.
// Batch (kchunk < 0): blockIdx.z is the problem index; its A, B and C start
// at A + z*astride, B + z*bstride, C + z*cstride.
template <typename T, bool TA, bool TB, int BM, int BN, int BK, int TM, int TN, bool LOWER>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_kernel(int m, int n, int k, T alpha, const T *__restrict__ A, long lda,
                 const T *__restrict__ B, long ldb, T beta, T *__restrict__ C, long ldc, int kchunk = 0,
                 long cstride = 0, long astride = 0, long bstride = 0)
{
    if (kchunk > 0) {
        const int kz = blockIdx.z * kchunk;
        k = min(kchunk, k - kz);
        A += TA ? (long)kz : (long)kz * lda;
        B += TB ? (long)kz * ldb : (long)kz;
        C += (long)blockIdx.z * cstride;
    } else if (kchunk < 0) {
        A += (long)blockIdx.z * astride;
        B += (long)blockIdx.z * bstride;
        C += (long)blockIdx.z * cstride;
    }
    constexpr int RG = BM / TM;            // row groups
    constexpr int CG = BN / TN;            // column groups
    constexpr int NT = RG * CG;
    constexpr int PADA = 16 / sizeof(T);   // keeps rows 16B aligned, breaks bank aliasing
    constexpr int LDA_S = BM + PADA;
    constexpr int LDB_S = BN + PADA;
    constexpr int LA = (BM * BK + NT - 1) / NT;
    constexpr int LB = (BN * BK + NT - 1) / NT;
    static_assert(TM % 2 == 0 || TM == 1, "TM even");
    __shared__ __align__(16) T As[2][BK][LDA_S];
    __shared__ __align__(16) T Bs[2][BK][LDB_S];

    int bi, bj;
    if (LOWER) {
        // triangular block index t -> (bi >= bj)
        long t = blockIdx.x;
        long r = (long)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((r + 1) * (r + 2) / 2 <= t) ++r;
        while (r * (r + 1) / 2 > t) --r;
        bi = (int)r;
        bj = (int)(t - r * (r + 1) / 2);
    } else {
        bi = blockIdx.x;
        bj = blockIdx.y;
    }
    const int m0 = bi * BM, n0 = bj * BN;
    const int tid = threadIdx.x;
    const int tr = tid % RG, tc = tid / RG;

    T acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = T(0);

    T ra[LA], rb[LB];
    auto load_a = [&](int k0) {
#pragma unroll
        for (int l = 0; l < LA; ++l) {
            int idx = tid + l * NT;
            int i, p;
            if (!TA) { i = idx % BM; p = idx / BM; } else { p = idx % BK; i = idx / BK; }
            T v = T(0);
            if (idx < BM * BK && m0 + i < m && k0 + p < k)
                v = TA ? A[(long)(k0 + p) + (long)(m0 + i) * lda] : A[(long)(m0 + i) + (long)(k0 + p) * lda];
            ra[l] = v;
        }
    };
    auto load_b = [&](int k0) {
#pragma unroll
        for (int l = 0; l < LB; ++l) {
            int idx = tid + l * NT;
            int j, p;
            if (TB) { j = idx % BN; p = idx / BN; } else { p = idx % BK; j = idx / BK; }
            T v = T(0);
            if (idx < BN * BK && n0 + j < n && k0 + p < k)
                v = TB ? B[(long)(n0 + j) + (long)(k0 + p) * ldb] : B[(long)(k0 + p) + (long)(n0 + j) * ldb];
            rb[l] = v;
        }
    };
    auto store_ab = [&](int buf) {
#pragma unroll
        for (int l = 0; l < LA; ++l) {
            int idx = tid + l * NT;
            if (idx < BM * BK) {
                int i, p;
                if (!TA) { i = idx % BM; p = idx / BM; } else { p = idx % BK; i = idx / BK; }
                As[buf][p][i] = ra[l];
            }
        }
#pragma unroll
        for (int l = 0; l < LB; ++l) {
            int idx = tid + l * NT;
            if (idx < BN * BK) {
                int j, p;
                if (TB) { j = idx % BN; p = idx / BN; } else { p = idx % BK; j = idx / BK; }
                Bs[buf][p][j] = rb[l];
            }
        }
    };

    const int nk = (k + BK - 1) / BK;
    if (nk > 0) {
        load_a(0);
        load_b(0);
        store_ab(0);
    }
    __syncthreads();
    for (int kt = 0; kt < nk; ++kt) {
        const int cur = kt & 1;
        if (kt + 1 < nk) { load_a((kt + 1) * BK); load_b((kt + 1) * BK); }
#pragma unroll
        for (int p = 0; p < BK; ++p) {
            T a[TM], b[TN];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int v = 0; v < TM / 2; ++v) a[h * (TM / 2) + v] = As[cur][p][h * (BM / 2) + tr * (TM / 2) + v];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int v = 0; v < TN / 2; ++v) b[h * (TN / 2) + v] = Bs[cur][p][h * (BN / 2) + tc * (TN / 2) + v];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        if (kt + 1 < nk) store_ab(cur ^ 1);
        __syncthreads();
    }

#pragma unroll
    for (int jj = 0; jj < TN; ++jj) {
        const int j = n0 + (jj / (TN / 2)) * (BN / 2) + tc * (TN / 2) + (jj % (TN / 2));
        if (j >= n) continue;
#pragma unroll
        for (int ii = 0; ii < TM; ++ii) {
            const int i = m0 + (ii / (TM / 2)) * (BM / 2) + tr * (TM / 2) + (ii % (TM / 2));
            if (i >= m) continue;
            if (LOWER && i < j) continue;
            T *c = &C[(long)i + (long)j * ldc];
            T old = (beta == T(0)) ? T(0) : beta * (*c);
            *c = fma(alpha, acc[ii][jj], old);
        }
    }
}

// ---------------------------------------------------------------------------
// The FP32 products C = beta C + alpha A B^T (TB) and beta C + alpha A B for
// large matrices: the same sums in the same order as gemm_simt_kernel's 128 x
// 128 tile (thread = 8 x 8, k ascending), with the operands read 16 bytes at a
// time, 16 k per barrier and whole tiles stored without per-element tests: the
// scalar form spent a third of its issue slots on addresses and tests (order
// 2048: A B^T 474 -> 362 us, A B 474 -> 411; B's columns are turned on the way
// into shared memory).  A, B and C 16-byte aligned with leading dimensions
// divisible by 4.
// ---------------------------------------------------------------------------
template <bool LOWER, bool TB>
__global__ void __launch_bounds__(256, 2) gemm_f32_kernel(int m, int n, int k, float alpha, const float *__restrict__ A,
                                                          long lda, const float *__restrict__ B, long ldb, float beta,
                                                          float *__restrict__ C, long ldc)
{
    constexpr int BM = 128, BK = 16, LD = BM + 4;
    __shared__ __align__(16) float As[2][BK][LD], Bs[2][BK][LD];
    int bi, bj;
    if (LOWER) {
        const int t = blockIdx.x;
        int r = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
        while ((r + 1) * (r + 2) / 2 <= t) ++r;
        while (r * (r + 1) / 2 > t) --r;
        bi = r;
        bj = t - r * (r + 1) / 2;
    } else {
        bi = blockIdx.x;
        bj = blockIdx.y;
    }
    const int m0 = bi * BM, n0 = bj * BM, tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
    // this thread's loads: 4 rows from 4 (tid % 32), k = tid / 32 and + 8
    const int lr = 4 * (tid & 31), lk = tid >> 5;
    // (B not transposed: 4 k from 4 (tid % 4), columns tid / 4 and + 64)
    const int bk = 4 * (tid & 3), bc = tid >> 2;
    const float *pa = A + m0 + lr + (long)lk * lda;
    const float *pb = TB ? B + n0 + lr + (long)lk * ldb : B + bk + (long)(n0 + bc) * ldb;
    const bool wa = m0 + BM <= m, wb = n0 + BM <= n;
    float4 ra[2], rb[2];
    auto load4 = [](const float *p, bool whole, int rows, bool in) {
        if (whole && in) return *reinterpret_cast<const float4 *>(p);
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (in) {
            if (rows > 0) v.x = p[0];
            if (rows > 1) v.y = p[1];
            if (rows > 2) v.z = p[2];
            if (rows > 3) v.w = p[3];
        }
        return v;
    };
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const bool in = k0 + lk + 8 * q < k;
            ra[q] = load4(pa + (long)(k0 + 8 * q) * lda, wa, m - m0 - lr, in);
            if (TB) rb[q] = load4(pb + (long)(k0 + 8 * q) * ldb, wb, n - n0 - lr, in);
            else rb[q] = load4(pb + k0 + (long)(64 * q) * ldb, k0 + BK <= k, k - k0 - bk, n0 + bc + 64 * q < n);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            *reinterpret_cast<float4 *>(&As[buf][lk + 8 * q][lr]) = ra[q];
            if (TB) {
                *reinterpret_cast<float4 *>(&Bs[buf][lk + 8 * q][lr]) = rb[q];
            } else {
                Bs[buf][bk][bc + 64 * q] = rb[q].x;
                Bs[buf][bk + 1][bc + 64 * q] = rb[q].y;
                Bs[buf][bk + 2][bc + 64 * q] = rb[q].z;
                Bs[buf][bk + 3][bc + 64 * q] = rb[q].w;
            }
        }
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    const int nk = (k + BK - 1) / BK;
    if (nk > 0) {
        load(0);
        store(0);
    }
    __syncthreads();
    for (int kt = 0; kt < nk; ++kt) {
        const int cur = kt & 1;
        if (kt + 1 < nk) load((kt + 1) * BK);
#pragma unroll
        for (int p = 0; p < BK; ++p) {
            float a[8], b[8];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 x = *reinterpret_cast<const float4 *>(&As[cur][p][64 * h + 4 * tr]);
                const float4 y = *reinterpret_cast<const float4 *>(&Bs[cur][p][64 * h + 4 * tc]);
                a[4 * h] = x.x, a[4 * h + 1] = x.y, a[4 * h + 2] = x.z, a[4 * h + 3] = x.w;
                b[4 * h] = y.x, b[4 * h + 1] = y.y, b[4 * h + 2] = y.z, b[4 * h + 3] = y.w;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (kt + 1 < nk) store(cur ^ 1);
        __syncthreads();
    }
    const bool whole = wa && wb && (!LOWER || bi > bj);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int col = n0 + 64 * (j >> 2) + 4 * tc + (j & 3);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = m0 + 64 * h + 4 * tr;
            float *c = C + row + (long)col * ldc;
            if (whole) {
                const float4 o = beta == 0.0f ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : *reinterpret_cast<const float4 *>(c);
                *reinterpret_cast<float4 *>(c) =
                    make_float4(fmaf(alpha, acc[4 * h][j], beta * o.x), fmaf(alpha, acc[4 * h + 1][j], beta * o.y),
                                fmaf(alpha, acc[4 * h + 2][j], beta * o.z), fmaf(alpha, acc[4 * h + 3][j], beta * o.w));
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (col < n && row + i < m && (!LOWER || row + i >= col))
                        c[i] = fmaf(alpha, acc[4 * h + i][j], beta == 0.0f ? 0.0f : beta * c[i]);
            }
        }
    }
}

} // namespace gb300
