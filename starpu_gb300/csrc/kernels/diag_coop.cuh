// One cooperative launch that factors an FP32 matrix (lower Cholesky, in
// place) and, on request, builds its lower-triangular inverse (order <= 1024):
// the POTRF of the mixed solve's diagonal tile with the operand of its
// tensor-core panel TRSM (P <- P L_kk^-T as P * Linv^T), and the plain FP32
// factorisation of tiles and small matrices.
//
// The matrix is handled in 64 x 64 blocks, right-looking, as the tile loop of
// examples/cholesky/cholesky_implicit.c:244-318 with the POTRF/TRSM/SYRK/GEMM
// codelet arithmetic of cholesky_kernels.c.  Step k:
//   A  every CTA with a block row i >= k loads the diagonal block and its own
//      64 rows into registers and takes both through the leaf's 16 steps of
//      four columns together (chol_panel.cuh): the diagonal block is factored
//      by the same instructions in every CTA (bit-identical copies), the own
//      rows become L_ik = A_ik L_kk^-T on the way.  The CTA of row k solves
//      the identity instead, which gives the block's inverse, and stores the
//      factored block after the phase's barrier, when every CTA has read it;
//   B  the trailing blocks A_ij -= L_ik L_jk^T (k < j <= i) are spread over
//      the grid.
// The inverse X = L^-1 is built on the way, block row by block row from
// L X = I:  X_kj = -X_kk sum_{p=j}^{k-1} L_kp X_pj.  The products of row k
// run in phase B of step k, their sums and the X_kk multiply in phase A of
// step k+1, both in CTAs the factorisation leaves idle; only the last block
// row follows the factorisation.
//
// Bound by the chain of n / 64 steps: 16 dependent four-column steps, two
// grid barriers and two rounds of loads each.
//
// Phases are separated by grid barriers.  With a.bar: a launch counter that
// each CTA bumps, waited on with acquire loads, each wait bounded by
// %globaltimer; on a timeout the CTA sets *err and returns, and the CTAs
// still waiting time out in turn.  Without (callers that have no workspace):
// the cooperative launch's own barrier, which every CTA reaches.  Data other
// CTAs wrote is read through L2 (ld.global.cg), never from a stale L1 line.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "chol_panel.cuh"
#include "tile64.cuh"

namespace gb300 {

__device__ __forceinline__ uint64_t dc_timer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr int DC_MAXN = 1024;
constexpr int DC_ERR_TIMEOUT = 4;  // *err code of a barrier wait that ran out
constexpr uint64_t DC_WAIT_NS = 1000000000ull;

struct DiagCoopArgs {
    int n;
    float *A;
    long lda;
    float *Linv;  // n x n, strict upper part zeroed by the caller
    long ldi;
    float *T;  // scratch of the inverse's block products: n * n floats
    int *info;
    int info_base;
    unsigned *bar;  // barrier counter, zero at launch; null: the launch's own grid barrier
    int *err;       // word that err_code goes to when a wait ran out
    int err_code;   // DC_ERR_TIMEOUT (with bar), or CP_ERR_TIMEOUT where err is an info word
    unsigned wait_us;  // limit of a wait inside a panel
    int invert;  // 0: factor only (no inverse is written)
};

// a negative code takes the place of a pivot's info
__device__ __forceinline__ void dc_report(const DiagCoopArgs &a)
{
    if (a.err_code < 0) atomicMin(a.err, a.err_code);
    else atomicCAS(a.err, 0, a.err_code);
}

__device__ __forceinline__ unsigned dc_ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier number `phase` (1, 2, ...).  False: a wait timed out here or
// another CTA has flagged an error -- the caller returns.
__device__ __forceinline__ bool dc_sync(const DiagCoopArgs &a, unsigned phase, int *s_ok)
{
    if (!a.bar) {
        cooperative_groups::this_grid().sync();
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        const unsigned target = phase * gridDim.x;
        if (dc_ld_acquire(a.bar) < target) {
            const uint64_t t0 = dc_timer();
            while (dc_ld_acquire(a.bar) < target) {
                if (*(volatile int *)a.err || dc_timer() - t0 > DC_WAIT_NS) {
                    dc_report(a);
                    ok = 0;
                    break;
                }
            }
        }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// row index ii, column index jj <= ii of the t-th block of a lower triangle
// (row by row: (0,0), (1,0), (1,1), (2,0), ...)
__device__ __forceinline__ void dc_tri_index(int t, int &ii, int &jj)
{
    int i = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((i + 1) * (i + 2) / 2 <= t) ++i;
    while (i * (i + 1) / 2 > t) --i;
    ii = i;
    jj = t - i * (i + 1) / 2;
}

// The slot of the product L_kp X_pj (64 x 64, ld 64) in the scratch area.
__device__ __forceinline__ float *dc_slot(const DiagCoopArgs &a, int j, int p)
{
    return a.T + (long)(p * (p + 1) / 2 + j) * (DC_B * DC_B);
}

// slot(j, p) = L_kp X_pj (rows of block row k: rk), X_pj the inverse block
__device__ __forceinline__ void dc_inv_product(const DiagCoopArgs &a, int k, int j, int p, float *s0, float *s1, bool vec,
                                               bool vec_inv)
{
    const int rk = min(DC_B, a.n - k * DC_B);
    DcTile l, x;
    l.load(a.A + k * DC_B + (long)(p * DC_B) * a.lda, a.lda, rk, DC_B, vec);
    x.load(a.Linv + p * DC_B + (long)(j * DC_B) * a.ldi, a.ldi, DC_B, DC_B, vec_inv);
    __syncthreads();  // shared tiles free
    l.store(s0);
    x.store_t(s1);
    __syncthreads();
    float acc[4][4] = {};
    dc_mma(s0, s1, acc);
    const int tr = threadIdx.x & 15, tn = threadIdx.x >> 4;
    float *S = dc_slot(a, j, p);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
        *reinterpret_cast<float4 *>(S + 4 * tr + (4 * tn + jj) * DC_B) =
            make_float4(acc[0][jj], acc[1][jj], acc[2][jj], acc[3][jj]);
}

// X_kj = -X_kk (sum_{p = j}^{k-1} slot(j, p)), summed in p order
__device__ __forceinline__ void dc_inv_combine(const DiagCoopArgs &a, int k, int j, float *s0, float *s1, bool vec_inv)
{
    const int rk = min(DC_B, a.n - k * DC_B);
    DcTile x;
    x.load(a.Linv + k * DC_B + (long)(k * DC_B) * a.ldi, a.ldi, rk, rk, vec_inv);
    float v[DC_B * DC_B / DC_T] = {};
    for (int p = j; p < k; ++p) {
        const float *S = dc_slot(a, j, p) + threadIdx.x;
#pragma unroll
        for (int q = 0; q < DC_B * DC_B / DC_T; ++q) v[q] += __ldcg(S + q * DC_T);
    }
    __syncthreads();  // shared tiles free
#pragma unroll
    for (int q = 0; q < DC_B * DC_B / DC_T; ++q) {
        const int e = threadIdx.x + q * DC_T;
        s1[(e & (DC_B - 1)) * DC_LD + (e >> 6)] = v[q];
    }
    x.store(s0);
    __syncthreads();
    float acc[4][4] = {};
    dc_mma(s0, s1, acc);
    const int tr = threadIdx.x & 15, tn = threadIdx.x >> 4;
    float *X = a.Linv + k * DC_B + (long)(j * DC_B) * a.ldi;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (4 * tr + i < rk) X[4 * tr + i + (long)(4 * tn + jj) * a.ldi] = -acc[i][jj];
}

// ---------------------------------------------------------------------------
// The kernel.  Step k, phase A: the tasks t = blockIdx.x, + gridDim.x, ...
// of [factor block rows k .. nblk-1 | combine row k-1 of the inverse];
// phase B: [trailing tile updates | products of row k of the inverse].  The
// inverse is built row by row as X_kj = -X_kk sum_{p=j}^{k-1} L_kp X_pj
// (L X = I, block row k), in CTAs the factorisation leaves idle; only the
// last row runs after the factorisation.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(DC_T, 2) diag_coop_kernel(DiagCoopArgs a)
{
    // two operand tiles, or the panel's published columns (never both at a time)
    constexpr int TILE = DC_B * DC_LD * sizeof(float);
    __shared__ __align__(16) unsigned char shared[2 * TILE > sizeof(CpPanel<float, 2>) ? 2 * TILE : sizeof(CpPanel<float, 2>)];
    float *s0 = (float *)shared, *s1 = (float *)(shared + TILE);
    CpPanel<float, 2> &pan = *(CpPanel<float, 2> *)shared;
    __shared__ uint64_t bar[16];
    __shared__ int s_ok;
    __shared__ CpState st;
    const int n = a.n, nblk = (n + DC_B - 1) / DC_B, G = gridDim.x, b = blockIdx.x;
    const bool vec = ((reinterpret_cast<uintptr_t>(a.A) & 15) == 0) && ((a.lda & 3) == 0);
    const bool vec_inv = ((reinterpret_cast<uintptr_t>(a.Linv) & 15) == 0) && ((a.ldi & 3) == 0);
    unsigned phase = 0, panels = 0;
    cp_panel_init(bar);
    __syncthreads();

    for (int k = 0; k < nblk; ++k) {
        const int k0 = k * DC_B, bk = min(DC_B, n - k0);
        float *Akk = a.A + k0 + (long)k0 * a.lda;
        // ---- phase A
        const int nf = nblk - k, nc = (a.invert && k >= 2) ? k - 1 : 0;
        CpBlock<float> d, x;
        for (int t = b; t < nf + nc; t += G) {
            if (t < nf) {
                const int i0 = (k + t) * DC_B, ri = min(DC_B, n - i0);
                float *Aik = a.A + i0 + (long)k0 * a.lda;
                // the block (identity past bk, zeros above) and this CTA's rows
                cp_each<float>(d, [&](float &v, int r, int c) {
                    v = (r < bk && c <= r) ? __ldcg(Akk + r + (long)c * a.lda) : (r == c ? 1.0f : 0.0f);
                });
                cp_each<float>(x, [&](float &v, int r, int c) {
                    if (t == 0) v = r == c ? 1.0f : 0.0f;
                    else v = (r < ri && c < bk) ? __ldcg(Aik + r + (long)c * a.lda) : 0.0f;
                });
                __syncthreads();  // pan of the previous task is free
                if (!cp_panel<float, 2>(d, x, pan, bar, panels & 1, st, bk, a.info, a.info_base + k0, t == 0, a.wait_us))
                    dc_report(a);
                ++panels;
                if (t > 0)
                    cp_each<float>(x, [&](float &v, int r, int c) {
                        if (r < ri && c < bk) Aik[r + (long)c * a.lda] = v;
                    });
                else if (a.invert)  // I L^-T = X_kk^T
                    cp_each<float>(x, [&](float &v, int r, int c) {
                        if (c >= r && c < bk) a.Linv[(k0 + c) + (long)(k0 + r) * a.ldi] = v;
                    });
            } else {
                dc_inv_combine(a, k - 1, t - nf, s0, s1, vec_inv);
            }
        }
        if (!dc_sync(a, ++phase, &s_ok)) return;
        if (b == 0) {  // the factored block: every CTA has read the unfactored one
            cp_each<float>(d, [&](float &v, int r, int c) {
                if (r < bk && c < r) Akk[r + (long)c * a.lda] = v;
            });
            st.diagonal([&](int c, float v) {
                if (c < bk) Akk[c * (a.lda + 1)] = v;
            });
        }
        if (k == nblk - 1) break;
        // ---- phase B
        // (CTA 0, which stores the factored block, takes its tile last)
        const int m = nblk - k - 1, nu = m * (m + 1) / 2;
        const int np = (a.invert && k >= 1) ? k * (k + 1) / 2 : 0;
        for (int t = (b + G - 1) % G; t < nu + np; t += G) {
            if (t < nu) {
                int ii, jj;
                dc_tri_index(t, ii, jj);
                const int bi = k + 1 + ii, bj = k + 1 + jj;
                const int i0 = bi * DC_B, j0 = bj * DC_B, ri = min(DC_B, n - i0), rj = min(DC_B, n - j0);
                float *C = a.A + i0 + (long)j0 * a.lda;
                const bool whole = dc_whole(ri, rj, bi == bj, vec);
                DcTile li, lj;
                float c[4][4];
                li.load(a.A + i0 + (long)k0 * a.lda, a.lda, ri, bk, vec);
                lj.load(a.A + j0 + (long)k0 * a.lda, a.lda, rj, bk, vec);
                dc_sub_load(C, a.lda, ri, rj, bi == bj, whole, c);
                __syncthreads();  // the previous task's shared operands are free
                li.store(s0);
                lj.store(s1);
                __syncthreads();
                float acc[4][4] = {};
                dc_mma(s0, s1, acc);
                dc_sub_store(C, a.lda, ri, rj, bi == bj, whole, c, acc);
            } else {
                int p, j;
                dc_tri_index(t - nu, p, j);
                dc_inv_product(a, k, j, p, s0, s1, vec, vec_inv);
            }
        }
        if (!dc_sync(a, ++phase, &s_ok)) return;
    }

    // ---- the last row of the inverse
    if (a.invert && nblk >= 2) {
        const int k = nblk - 1;
        for (int t = b; t < k * (k + 1) / 2; t += G) {
            int p, j;
            dc_tri_index(t, p, j);
            dc_inv_product(a, k, j, p, s0, s1, vec, vec_inv);
        }
        if (!dc_sync(a, ++phase, &s_ok)) return;
        for (int t = b; t < k; t += G) dc_inv_combine(a, k, t, s0, s1, vec_inv);
    }
}

} // namespace gb300
