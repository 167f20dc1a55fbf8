// SIMT kernels of the tiled LU factorisation (examples/lu): the factor form
// of the reference codelets, A = L U with L lower non-unit and U unit upper
// (the CPU GETRF loop of examples/lu/xlu_kernels.c:369-380 keeps the pivot
// in L and scales the pivot row), and its threshold pivoting: a step whose
// pivot is smaller than the threshold in magnitude takes the largest entry of
// its row and swaps whole columns (xlu_kernels.c:516-545).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "chol_panel.cuh"

namespace gb300 {

// 1 / d rounded to T the way the reference forms its scale factor: in double,
// then converted (the BLAS SCAL takes a T alpha)
template <typename T> __device__ __forceinline__ T lu_recip(T d) { return (T)(1.0 / (double)d); }

// ---------------------------------------------------------------------------
// Unblocked LU of one n x n (n <= NMAX) diagonal block, held in registers:
// 256 threads as NMAX rows x CL column lanes, thread (ti, tc) keeps row ti,
// columns tc, tc + CL, ...  Step z: the owners of column z and of row z
// publish them through double-buffered shared vectors (one barrier per step);
// every thread scales its copy of row z by 1/a_zz and applies the rank-1
// update to its elements.  A zero pivot records info = info_base + z + 1
// (first wins, no trap).  thr > 0: the first step whose pivot has magnitude
// below thr is recorded (atomicMin of info_base + z into *d_first), for the
// caller's pivoting fallback.
// ---------------------------------------------------------------------------
template <typename T, int NMAX>
__global__ void __launch_bounds__(256) getf2_small_kernel(int n, T *__restrict__ A, long lda, T thr, int *d_first,
                                                          int *info, int info_base)
{
    constexpr int CL = 256 / NMAX, NC = NMAX / CL;
    __shared__ T col[2][NMAX], row[2][NMAX];
    const int tid = threadIdx.x;
    const int ti = tid % NMAX, tc = tid / NMAX;
    T a[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) {
        const int c = tc + q * CL;
        a[q] = (ti < n && c < n) ? A[(long)ti + (long)c * lda] : T(0);
    }
    bool flagged = false;
#pragma unroll
    for (int z = 0; z < NMAX; ++z) {
        if (z >= n) break;
        T *cz = col[z & 1], *rz = row[z & 1];
        if (tc == z % CL) cz[ti] = a[z / CL];
        if (ti == z) {
#pragma unroll
            for (int q = 0; q < NC; ++q) rz[tc + q * CL] = a[q];
        }
        __syncthreads();
        const T d = cz[z];
        if (tid == 0) {
            if (d == T(0) && info) atomicCAS(info, 0, info_base + z + 1);
            if (thr > T(0) && !flagged && !(fabs((double)d) >= (double)thr) && d_first) {
                atomicMin(d_first, info_base + z);
                flagged = true;
            }
        }
        const T inv = lu_recip(d);
        if (ti == z) {
#pragma unroll
            for (int q = 0; q < NC; ++q)
                if (tc + q * CL > z) a[q] = a[q] * inv;
        } else if (ti > z) {
            const T l = cz[ti];
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                const int c = tc + q * CL;
                if (c > z) a[q] = fma(-l, rz[c] * inv, a[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NC; ++q) {
        const int c = tc + q * CL;
        if (ti < n && c < n) A[(long)ti + (long)c * lda] = a[q];
    }
}

// ---------------------------------------------------------------------------
// The FP32 leaf: unblocked LU of one n x n (n <= 64) block by one CTA of 8
// warps, the columns four at a time as the Cholesky panel takes them
// (chol_panel.cuh: lane = row, warp w owns columns 4w .. and 32 + 4w .., a
// buffer and an mbarrier per step instead of CTA barriers).  The owner of a
// step factors its 4 x 4 block in every lane, forms its columns of L and
// publishes them with the reciprocal pivots; the others form their elements
// of the four rows of U from the 4 x 4 block (four shuffles per column) and
// apply the rank-4 update to the rows below (the rows above are finished, and
// stay as they are where a zero pivot makes U infinite).  Bound by the chain of 16 steps: 10 us against 36
// for a barrier and a double-precision reciprocal per column.  Same status words
// and threshold as getf2_small_kernel.
// ---------------------------------------------------------------------------
struct GetfPanel {
    Quad<float> pan[16][CP_W];  // L of the step's columns, 0 above its rows
    Quad<float> inv[16];        // 1 / pivots
    uint64_t bar[16];
};

// HS = step / 8: the half of the rows that holds the step's
template <int G, int HS> __device__ __forceinline__ void getf_update(CpBlock<float> &a, const GetfPanel &s, int step)
{
    const int lane = threadIdx.x & 31, blk = step & 7;
    const Quad<float> *p = s.pan[step];
    Quad<float> li[2], l[4];
#pragma unroll
    for (int h = HS; h < 2; ++h) li[h] = p[32 * h + lane];
#pragma unroll
    for (int i = 0; i < 4; ++i) l[i] = p[4 * step + i];
    const Quad<float> inv = s.inv[step];
    const bool in = (lane >> 2) == blk, below = (lane >> 2) > blk;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float v = a[G][c][HS];
        Quad<float> u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float t = __shfl_sync(0xffffffffu, v, 4 * blk + i);
#pragma unroll
            for (int q = 0; q < i; ++q) t = fmaf(-l[i].v[q], u.v[q], t);
            u.v[i] = t * inv.v[i];
        }
        const float mine = (lane & 2) ? ((lane & 1) ? u.v[3] : u.v[2]) : ((lane & 1) ? u.v[1] : u.v[0]);
        const float upd = cp_dot_sub(v, li[HS], u);
        a[G][c][HS] = in ? mine : below ? upd : v;
        if (HS == 0) a[G][c][1] = cp_dot_sub(a[G][c][1], li[1], u);
    }
}

// the zeros among the pivots of columns z .. z + 3
static __device__ __noinline__ void getf_report_zero(Quad<float> piv, int z, int n, int *info, int info_base)
{
    if ((threadIdx.x & 31) == 0 && info)
        for (int j = 0; j < 4; ++j)
            if (piv.v[j] == 0.0f && z + j < n) atomicCAS(info, 0, info_base + z + j + 1);
}

// the owner's part of step 8 G + warp
template <int G>
__device__ __forceinline__ void getf_own(CpBlock<float> &a, GetfPanel &s, int n, float thr, int *d_first, int *info,
                                         int info_base)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, step = 8 * G + warp;
    Quad<float> *p = s.pan[step];
    const bool in = (lane >> 2) == warp;
    if (in) p[32 * G + lane] = {a[G][0][G], a[G][1][G], a[G][2][G], a[G][3][G]};
    __syncwarp();
    float l[4][4], inv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const Quad<float> v = p[4 * step + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) l[i][j] = v.v[j];
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        inv[j] = __frcp_rn(l[j][j]);
#pragma unroll
        for (int k = j + 1; k < 4; ++k) l[j][k] *= inv[j];
#pragma unroll
        for (int i = j + 1; i < 4; ++i)
#pragma unroll
            for (int k = j + 1; k < 4; ++k) l[i][k] = fmaf(-l[i][j], l[j][k], l[i][k]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        Quad<float> y;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v = a[G][j][h];
#pragma unroll
            for (int q = 0; q < j; ++q) v = fmaf(-y.v[q], l[q][j], v);
            y.v[j] = v;
        }
        if (h < G || (h == G && lane < 4 * warp)) {  // rows above: U already, no part in this step
            y = {0.0f, 0.0f, 0.0f, 0.0f};
        } else if (h == G && in) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if ((lane & 3) == i) {
                        a[G][j][h] = l[i][j];
                        y.v[j] = j <= i ? l[i][j] : 0.0f;
                    }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) a[G][j][h] = y.v[j];
        }
        p[32 * h + lane] = y;
    }
    if (lane == 0) s.inv[step] = {inv[0], inv[1], inv[2], inv[3]};
    // (before the step is published: the first zero pivot is the first to get
    // there; every lane knows the pivots, so the branch is the whole warp's)
    if (fminf(fminf(fabsf(l[0][0]), fabsf(l[1][1])), fminf(fabsf(l[2][2]), fabsf(l[3][3]))) == 0.0f)
        getf_report_zero({l[0][0], l[1][1], l[2][2], l[3][3]}, 4 * step, n, info, info_base);
    ptx::mbar_arrive(&s.bar[step]);
    if (lane == 0 && thr > 0.0f && d_first) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (4 * step + j < n && !(fabsf(l[j][j]) >= thr)) atomicMin(d_first, info_base + 4 * step + j);
    }
    __syncwarp();
}

__global__ void __launch_bounds__(256) getf2_leaf_kernel(int n, float *__restrict__ A, long lda, float thr, int *d_first,
                                                         int *info, int info_base, const CpWait wait)
{
    __shared__ GetfPanel s;
    const int w = threadIdx.x >> 5, steps = (n + 3) / 4;
    CpBlock<float> a;
    cp_panel_init(s.bar);
    cp_each<float>(a, [&](float &v, int r, int c) { v = (r < n && c < n) ? A[r + (long)c * lda] : (r == c ? 1.0f : 0.0f); });
    __syncthreads();
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < min(w, steps); ++i) {
        ok = cp_wait(&s.bar[i], 0, wait.us) && ok;
        getf_update<0, 0>(a, s, i);
        if (i < w - 1) getf_update<1, 0>(a, s, i);  // the next owner publishes first
    }
    if (w < steps) getf_own<0>(a, s, n, thr, d_first, info, info_base);
    if (steps > 8) {
        if (w > 0) getf_update<1, 0>(a, s, w - 1);
        getf_update<1, 0>(a, s, w);
#pragma unroll 1
        for (int i = w + 1; i < 8; ++i) {
            ok = cp_wait(&s.bar[i], 0, wait.us) && ok;
            getf_update<1, 0>(a, s, i);
        }
#pragma unroll 1
        for (int i = 8; i < min(8 + w, steps); ++i) {
            ok = cp_wait(&s.bar[i], 0, wait.us) && ok;
            getf_update<1, 1>(a, s, i);
        }
        if (8 + w < steps) getf_own<1>(a, s, n, thr, d_first, info, info_base);
    }
    if (!ok) wait.report();
    cp_each<float>(a, [&](float &v, int r, int c) {
        if (r < n && c < n) A[r + (long)c * lda] = v;
    });
}

// ---------------------------------------------------------------------------
// Exact unblocked threshold-pivoting LU of one n x n tile in global memory
// (the reference GETRF_PIVOT loop, xlu_kernels.c:516-545, with the pivot
// index of its CUDA branch), run by one CTA of 1024 threads.  It does
// nothing unless *d_first < n: the blocked factorisation that ran first met a
// pivot below the threshold, so the tile was restored from its copy and is
// factored again here with pivoting.  ipiv[z] = the column swapped with z at
// step z (z itself when the step pivoted in place), -1 when it did not pivot.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(1024) getrf_pivot_unblocked_kernel(int n, T *__restrict__ A, long lda, T thr,
                                                                     const int *d_first, int *ipiv, int *info)
{
    if (*d_first >= n) return;
    __shared__ double sval[32];
    __shared__ int sidx[32];
    __shared__ int s_p;
    __shared__ T s_piv;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int z = 0; z < n; ++z) {
        T *az = A + (long)z * lda;  // column z
        if (tid == 0) s_piv = az[z];
        __syncthreads();
        if (!(fabs((double)s_piv) >= (double)thr)) {
            // largest |a_zj|, j >= z (row z), first index on ties
            double best = -1.0;
            int bi = n;
            for (int j = z + tid; j < n; j += nt) {
                const double v = fabs((double)A[(long)z + (long)j * lda]);
                if (v > best) best = v, bi = j;
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_down_sync(0xffffffffu, best, o);
                const int oi = __shfl_down_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) best = ov, bi = oi;
            }
            if ((tid & 31) == 0) sval[tid >> 5] = best, sidx[tid >> 5] = bi;
            __syncthreads();
            if (tid == 0) {
                double b = sval[0];
                int p = sidx[0];
                for (int w = 1; w < nt / 32; ++w)
                    if (sval[w] > b || (sval[w] == b && sidx[w] < p)) b = sval[w], p = sidx[w];
                s_p = p < n ? p : z;
                ipiv[z] = s_p;
            }
            __syncthreads();
            const int p = s_p;
            if (p != z) {
                T *ap = A + (long)p * lda;
                for (int i = tid; i < n; i += nt) {
                    const T t = az[i];
                    az[i] = ap[i];
                    ap[i] = t;
                }
            }
            __syncthreads();
            if (tid == 0) s_piv = az[z];
        } else if (tid == 0) {
            ipiv[z] = -1;
        }
        __syncthreads();
        const T d = s_piv;
        if (tid == 0 && d == T(0) && info) atomicCAS(info, 0, z + 1);
        const T inv = lu_recip(d);
        for (int j = z + 1 + tid; j < n; j += nt) A[(long)z + (long)j * lda] *= inv;
        __syncthreads();
        // rank-1 update of the trailing block: a_ij -= a_iz * a_zj
        const int m = n - z - 1;
        for (long e = tid; e < (long)m * m; e += nt) {
            const int i = z + 1 + (int)(e % m), j = z + 1 + (int)(e / m);
            A[(long)i + (long)j * lda] = fma(-az[i], A[(long)z + (long)j * lda], A[(long)i + (long)j * lda]);
        }
        __syncthreads();
    }
}

// When a step of the blocked factorisation needed a pivot (*d_first < n):
// put the tile back from its copy (ld n) and clear the status word, so the
// pivoting factorisation starts from the input.
template <typename T>
__global__ void restore_if_flagged_kernel(int n, const T *__restrict__ copy, T *__restrict__ A, long lda,
                                          const int *d_first, int *info)
{
    if (*d_first >= n) return;
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e == 0 && info) *info = 0;
    if (e < (long)n * n) A[(e % n) + (e / n) * lda] = copy[e];
}

__global__ void lu_set_int_kernel(int *p, int v) { *p = v; }

// ---------------------------------------------------------------------------
// Column swaps of one tile in the order given (the reference PIVOT codelet,
// xlu_kernels.c:686-693): swap columns pairs[s].x and pairs[s].y for s = 0,
// 1, ...  One thread per row applies the whole sequence to its row.
// ---------------------------------------------------------------------------
constexpr int LU_SWAP_MAX = 1024;
struct LuSwapList {
    int count;
    int2 pairs[LU_SWAP_MAX];
};

template <typename T>
__global__ void __launch_bounds__(256) swap_columns_kernel(int m, T *__restrict__ A, long lda, const LuSwapList list)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    for (int s = 0; s < list.count; ++s) {
        const int2 p = list.pairs[s];
        T *x = A + i + (long)p.x * lda, *y = A + i + (long)p.y * lda;
        const T t = *x;
        *x = *y;
        *y = t;
    }
}

} // namespace gb300
