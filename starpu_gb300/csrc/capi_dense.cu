// C-ABI over the SIMT dense kernels: tile codelet bodies (POTRF/TRSM/SYRK/GEMM
// on one tile, FP32 and FP64) and the whole-matrix tiled factorisation and
// triangular solves composed from them.  Every entry point only enqueues work
// on the caller's stream and returns; nothing here synchronises or allocates.
#include "kernels/chol_panel.cuh"
#include "kernels/simt_blas.cuh"
#include "kernels/slice_update.cuh"
#include "kernels/trsv_sweep.cuh"
#include "gb300_internal.h"
#include "starpu_gb300_kernels.h"

#include <algorithm>
#include <type_traits>

namespace gb300 {

// fewest rows of an FP64 product or trailing update that runs on the tensor cores
constexpr int SLICE_MIN_M = 128;
// largest FP32 matrix (or diagonal tile) that one cooperative launch factors.
// Against tiles of 256, 512 or 1024 with a launch per tile, panel and update, the
// fastest of them: n = 600 131 and 187 us, 2048 543 and 588, 3000 958 and 1132,
// 4096 1562 and 1693; 5000 2394 and 2556, 6000 3496 and 3696, 8192 7383 and 6587.
// The line is below the crossing, since the launch rounds the trailing matrix
// every 64 columns instead of every tile.
constexpr int COOP_MAX_N = 4096;

static inline unsigned cdiv(long a, long b) { return (unsigned)((a + b - 1) / b); }

// C[m x n] -= A B^T in FP64 on the tensor cores (kernels/slice_update.cuh), A
// m x k and B n x k with the given element strides.  GEMM: any k, guarded;
// else k <= 64, for a panel of an SPD matrix.
template <bool GEMM>
static void slice_update(cudaStream_t s, bool lower, int m, int n, int k, const double *A, long a_rs, long a_ks,
                         const double *B, long b_rs, long b_ks, double *C, long ldc, int *err)
{
    if (m <= 0 || n <= 0 || k <= 0) return;
    if (gb300_func_dyn_smem((const void *)slice_update_kernel<GEMM>, SU_SMEM)) return;
    SliceUpdateArgs a;
    a.A = A, a.a_rs = a_rs, a.a_ks = a_ks, a.B = B, a.b_rs = b_rs, a.b_ks = b_ks;
    a.C = C, a.ldc = ldc, a.m = m, a.n = n, a.k = k, a.lower = lower ? 1 : 0;
    a.col_tiles = (n + SU_BN - 1) / SU_BN;
    a.err = err ? err : gb300_wait_status();
    if (!a.err) return;
    a.wait_budget_ns = gb300_wait_budget_ns();
    a.total = 0;
    for (int rb = 0; rb * SU_BM < m; ++rb)
        a.total += lower ? std::min(a.col_tiles, (SU_BM / SU_BN) * (rb + 1)) : a.col_tiles;
    gb300_count_launch(), slice_update_kernel<GEMM>
        <<<std::min(a.total, gb300_device_sms()), SU_THREADS, SU_SMEM, s>>>(a);
}

// Elements of C from which an FP64 product (alpha = -1, beta = 1) runs on the
// tensor cores.  The line is the solve's, which loses below it: POTRS of 64
// right-hand sides, us, with this line, on the FP64 units alone and with slices
// throughout: order 1000 488 488 626, 2000 1226 1206 1379, 3000 1893
// 2136 2061, 8000 5745 10172 5953.  Square products at the line (m = n = 320), slices
// and FP64 units: k = 16 23 and 17, 64 23 and 28, 256 45 and 77; at 256 23 and 16, 23 and
// 28, 46 and 79; at 640 24 and 25, 22 and 62, 46 and 207.
constexpr long SLICE_MIN_ELEMENTS = 96 * 1024;

template <typename T, bool TA, bool TB, int BM, int BN, int BK, int TM, int TN>
static void gemm_launch(cudaStream_t s, bool lower, int m, int n, int k, T alpha, const T *A, long lda, const T *B,
                        long ldb, T beta, T *C, long ldc)
{
    constexpr int NT = (BM / TM) * (BN / TN);
    // the lower-triangular form is only ever used as C -= A A^T (N,T)
    if constexpr (!TA && TB && BM == BN) {
        if (lower) {
            long tb = cdiv(m, BM);
            gb300_count_launch(), gemm_simt_kernel<T, TA, TB, BM, BN, BK, TM, TN, true>
                <<<dim3((unsigned)(tb * (tb + 1) / 2)), NT, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
            return;
        }
    }
    {
        gb300_count_launch(), gemm_simt_kernel<T, TA, TB, BM, BN, BK, TM, TN, false>
            <<<dim3(cdiv(m, BM), cdiv(n, BN)), NT, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    }
}

template <typename T> struct simt_cfg;
// CTAs of a product in bm x bm block tiles
static long gemm_ctas(bool lower, int m, int n, int bm)
{
    const long tm = cdiv(m, bm), tn = cdiv(n, bm);
    return lower ? tm * (tm + 1) / 2 : tm * tn;
}

static bool aligned16(const float *p, long ld) { return ((uintptr_t)p & 15) == 0 && (ld & 3) == 0; }

template <bool TB>
static void gemm_f32(cudaStream_t s, bool lower, int m, int n, int k, float alpha, const float *A, long lda,
                     const float *B, long ldb, float beta, float *C, long ldc)
{
    const unsigned tm = cdiv(m, 128), tn = cdiv(n, 128);
    if (TB && lower)
        gb300_count_launch(), gemm_f32_kernel<true, true>
            <<<tm * (tm + 1) / 2, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else
        gb300_count_launch(), gemm_f32_kernel<false, TB>
            <<<dim3(tm, tn), 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

// FP32: 128x128 block tiles, 8x8 per thread, from 64 of them on; smaller ones
// otherwise (the 64 and 32 tiles take a third and an eighth of the 128 tile's
// time each, so up to two waves of them are faster).  Alone, a 1024^3 product is
// faster in 64 tiles (86 us against 108) and a 512^3 one in 32 tiles (27 and 33),
// but a task graph runs eight of them side by side, where a third or a half
// more work per product counts: LU of order 16384 takes 195 ms in 32 x 32 tiles,
// 290 with smaller product tiles (from 152 instead of 64), and 105 and 127 ms in 16 x 16.
// Narrow variant for few columns.
template <> struct simt_cfg<float> {
    template <bool TA, bool TB>
    static void run(cudaStream_t s, bool lower, int m, int n, int k, float al, const float *A, long lda,
                    const float *B, long ldb, float be, float *C, long ldc)
    {
        if (!lower && n <= 32)
            gemm_launch<float, TA, TB, 128, 32, 8, 8, 2>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
        else if (!TA && gemm_ctas(lower, m, n, 128) >= 64 && aligned16(A, lda) && aligned16(B, ldb) && aligned16(C, ldc))
            gemm_f32<TB>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
        else if (gemm_ctas(lower, m, n, 128) >= 64)
            gemm_launch<float, TA, TB, 128, 128, 8, 8, 8>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
        else if (gemm_ctas(lower, m, n, 64) >= 64)
            gemm_launch<float, TA, TB, 64, 64, 16, 4, 4>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
        else
            gemm_launch<float, TA, TB, 32, 32, 32, 2, 2>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
    }
};
// FP64: 64x64 block tiles, 4x4 per thread, for several waves of them; 32x32
// tiles below that, so that every SM's FP64 units (2 FMA per clock) have work.
template <> struct simt_cfg<double> {
    template <bool TA, bool TB>
    static void run(cudaStream_t s, bool lower, int m, int n, int k, double al, const double *A, long lda,
                    const double *B, long ldb, double be, double *C, long ldc)
    {
        if (al == -1.0 && be == 1.0 && m >= SLICE_MIN_M && n >= 16 && k >= 16 &&
            (lower ? (long)m * (m + 1) / 2 : (long)m * n) >= SLICE_MIN_ELEMENTS)
            slice_update<true>(s, lower, m, n, k, A, TA ? lda : 1, TA ? 1 : lda, B, TB ? 1 : ldb, TB ? ldb : 1, C, ldc, nullptr);
        else if (!lower && n <= 16)
            gemm_launch<double, TA, TB, 64, 16, 8, 4, 2>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
        else if (gemm_ctas(lower, m, n, 64) >= 4L * gb300_device_sms())
            gemm_launch<double, TA, TB, 64, 64, 8, 4, 4>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
        else
            gemm_launch<double, TA, TB, 32, 32, 16, 2, 2>(s, lower, m, n, k, al, A, lda, B, ldb, be, C, ldc);
    }
};

template <typename T>
void gemm(cudaStream_t s, bool ta, bool tb, bool lower, int m, int n, int k, T alpha, const T *A, long lda,
          const T *B, long ldb, T beta, T *C, long ldc)
{
    if (m <= 0 || n <= 0) return;
    if (!ta && !tb) simt_cfg<T>::template run<false, false>(s, lower, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (!ta && tb) simt_cfg<T>::template run<false, true>(s, lower, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (ta && !tb) simt_cfg<T>::template run<true, false>(s, lower, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    else simt_cfg<T>::template run<true, true>(s, lower, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

// `batch` independent products C_z = alpha * A_z B_z + beta * C_z (no
// transposes), A_z = A + z * astride and likewise for B and C: one launch.
template <typename T>
void gemm_batched_nn(cudaStream_t s, int m, int n, int k, T alpha, const T *A, long lda, long astride, const T *B,
                     long ldb, long bstride, T beta, T *C, long ldc, long cstride, int batch)
{
    if (m <= 0 || n <= 0 || batch <= 0) return;
    if constexpr (std::is_same<T, float>::value)
        gb300_count_launch(), gemm_simt_kernel<T, false, false, 128, 128, 8, 8, 8, false>
            <<<dim3(cdiv(m, 128), cdiv(n, 128), batch), 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, -1,
                                                                    cstride, astride, bstride);
    else
        gb300_count_launch(), gemm_simt_kernel<T, false, false, 64, 64, 8, 4, 4, false>
            <<<dim3(cdiv(m, 64), cdiv(n, 64), batch), 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, -1,
                                                                  cstride, astride, bstride);
}

// Linv (n x n, ld ldi, strictly upper part zeroed) = inverse of the lower
// triangle of L: the 64 x 64 diagonal blocks by forward substitution, then
// doubling -- neighbouring inverted blocks of order h combine as
//   [L11 0; L21 L22]^-1 = [I11 0; -I22 (L21 I11)  I22],
// every pair of one level in one batched launch per product.  scratch holds
// >= n * n / 4 elements.
template <typename T>
void trtri_lower(cudaStream_t s, int n, const T *L, long ldl, T *Linv, long ldi, T *scratch)
{
    if (n <= 0) return;
    cudaMemset2DAsync(Linv, ldi * sizeof(T), 0, n * sizeof(T), n, s);
    gb300_count_launch(), invert_diag_blocks_kernel<T, 64>
        <<<cdiv(n, 64), 64, 0, s>>>(n, L, ldl, Linv, ldi, 64 * (ldi + 1), true);
    for (int h = 64; h < n; h *= 2) {
        const int full = n / (2 * h);  // pairs whose halves both have order h
        const long sl = 2L * h * (ldl + 1), si = 2L * h * (ldi + 1);
        if (full > 0) {
            gemm_batched_nn<T>(s, h, h, h, T(1), L + h, ldl, sl, Linv, ldi, si, T(0), scratch, h, (long)h * h, full);
            gemm_batched_nn<T>(s, h, h, h, T(-1), Linv + h + (long)h * ldi, ldi, si, scratch, h, (long)h * h, T(0),
                               Linv + h, ldi, si, full);
        }
        const int o = full * 2 * h, r = n - o - h;  // a last pair whose second half has order r < h
        if (r > 0) {
            gemm<T>(s, false, false, false, r, h, h, T(1), L + (o + h) + (long)o * ldl, ldl, Linv + o + (long)o * ldi,
                    ldi, T(0), scratch, r);
            gemm<T>(s, false, false, false, r, h, r, T(-1), Linv + (o + h) + (long)(o + h) * ldi, ldi, scratch, r, T(0),
                    Linv + (o + h) + (long)o * ldi, ldi);
        }
    }
}

// One launch of the slab solve X M^T = B (SlabArgs), n <= CP_TRSM_MAXN.
template <typename T, int SR> static void slab_launch(cudaStream_t s, const SlabArgs<T> &a)
{
    if (gb300_func_dyn_smem((const void *)trsm_slab_kernel<T, SR>, (int)cp_trsm_smem<T, SR>(CP_TRSM_MAXN))) return;
    gb300_count_launch(), trsm_slab_kernel<T, SR><<<cdiv(a.m, SR), 256, cp_trsm_smem<T, SR>(a.n), s>>>(a);
}

// X M^T = B in place: one launch per CP_TRSM_MAXN columns (rows are
// independent), then a GEMM update of the remaining columns.
template <typename T> void trsm_slab(cudaStream_t s, const SlabArgs<T> &a)
{
    if (a.m <= 0 || a.n <= 0) return;
    SlabArgs<T> c = a;
    for (int j0 = 0; j0 < a.n; j0 += CP_TRSM_MAXN) {
        c.n = std::min(CP_TRSM_MAXN, a.n - j0);
        c.M = a.M + j0 * (a.m_js + a.m_ps);
        c.B = a.B + j0 * a.b_js;
        // 16 rows per CTA once that fills the GPU; below, 4 spread the products
        // over more SMs (8 when one 64-column block has none)
        if (a.m >= 16 * 128) slab_launch<T, 16>(s, c);
        else if (a.n <= CP_W && a.m > 4 * gb300_device_sms()) slab_launch<T, 8>(s, c);
        else slab_launch<T, 4>(s, c);
        const int rest = a.n - j0 - c.n;
        if (rest <= 0) break;
        // B_rest -= X M_rest^T
        const T *M2 = c.M + c.n * a.m_js;
        T *B2 = c.B + c.n * a.b_js;
        if (a.b_js == 1 && a.m_js == 1)  // transposed: B2^T (rest x m) -= M_rest X^T
            gemm<T>(s, false, false, false, rest, a.m, c.n, T(-1), M2, a.m_ps, c.B, a.b_rs, T(1), B2, a.b_rs);
        else
            gemm<T>(s, false, a.m_js == 1, false, a.m, rest, c.n, T(-1), c.B, a.b_js, M2, a.m_js == 1 ? a.m_ps : a.m_js,
                    T(1), B2, a.b_js);
    }
}

// B[m x nc] <- B * L^{-T}
template <typename T>
void trsm_rltn(cudaStream_t s, int m, int nc, const T *L, long ldl, T *B, long ldb)
{
    trsm_slab<T>(s, {m, nc, L, 1, ldl, B, 1, ldb, false});
}

// B[m x n] <- L^{-1} B (LU block row)
template <typename T> void trsm_llnn(cudaStream_t s, int m, int n, const T *L, long ldl, T *B, long ldb)
{
    trsm_slab<T>(s, {n, m, L, 1, ldl, B, ldb, 1, false});
}

// B[m x n] <- B U^{-1}, U unit upper (LU block column)
template <typename T> void trsm_runu(cudaStream_t s, int m, int n, const T *U, long ldu, T *B, long ldb)
{
    trsm_slab<T>(s, {m, n, U, ldu, 1, B, 1, ldb, true});
}

// Trailing update of one step: C (m x m, lower) -= P P^T, P m x k.
static void trailing_update(cudaStream_t s, int m, int k, const float *P, long ldp, float *C, long ldc, int *)
{
    gemm<float>(s, false, true, true, m, m, k, -1.0f, P, ldp, P, ldp, 1.0f, C, ldc);
}
static void trailing_update(cudaStream_t s, int m, int k, const double *P, long ldp, double *C, long ldc, int *err)
{
    if (m < SLICE_MIN_M) gemm<double>(s, false, true, true, m, m, k, -1.0, P, ldp, P, ldp, 1.0, C, ldc);
    else slice_update<false>(s, true, m, m, k, P, 1, ldp, P, 1, ldp, C, ldc, err);
}

// Right-looking tiled Cholesky with tile nb: POTRF(k), TRSM of the whole
// column panel below it, then the lower-triangular trailing update.  This is
// the loop of examples/cholesky/cholesky_implicit.c:244-318 with the tasks of
// one step k fused into whole-panel launches.  FP32 diagonal blocks, and whole
// matrices up to COOP_MAX_N, are factored by one cooperative launch
// (kernels/diag_coop.cuh); FP64 goes in panels of CP_W columns.
template <typename T>
int potrf_tiled(cudaStream_t s, int n, T *A, long lda, int nb, int *info, int info_base)
{
    int rc = GB300_OK;
    if (nb <= 0) nb = n;
    const CpWait wait{gb300_wait_us(), info ? info : gb300_wait_status()};
    if (!wait.err) return GB300_ECUDA;
    if (std::is_same<T, float>::value && n <= COOP_MAX_N) nb = n;
    // FP64: the FP64 units would bound wider panels, the tensor-core update takes 64 columns
    if (std::is_same<T, double>::value) nb = std::min(nb, CP_W);
    for (int k0 = 0; k0 < n; k0 += nb) {
        const int kb = std::min(nb, n - k0);
        T *Akk = A + k0 + (long)k0 * lda;
        if (kb <= CP_W)
            gb300_count_launch(), potf2_leaf_kernel<<<1, 256, 0, s>>>(kb, Akk, lda, info, info_base + k0, wait);
        else if (std::is_same<T, float>::value && kb <= COOP_MAX_N)
            rc = potrf_coop(s, kb, (float *)Akk, lda, info, info_base + k0, wait.err);
        else
            rc = potrf_tiled<T>(s, kb, Akk, lda, CP_W, info, info_base + k0);
        if (rc) return rc;  // nothing is enqueued on a block that is not factored
        const int m = n - k0 - kb;
        if (m > 0) {
            T *P = A + (k0 + kb) + (long)k0 * lda;
            trsm_rltn<T>(s, m, kb, Akk, lda, P, lda);
            trailing_update(s, m, kb, P, lda, A + (k0 + kb) + (long)(k0 + kb) * lda, lda, wait.err);
        }
    }
    return GB300_OK;
}

// POTRS with a lower factor: L y = b (forward), then L^T x = y (backward),
// in blocks of CP_SB rows: solve the block, update the rows to come.
// min-dgels/base/SRC/dpotrs.c does the same two sweeps through dtrsm.
// C right-hand sides per CTA in the update.
template <typename T, int C, bool TRANS>
static void potrs_sweep_blocks(cudaStream_t s, int n, int nrhs, const T *L, long ldl, T *B, long ldb, const CpWait &wait)
{
    constexpr size_t sm_blk = cp_trsv_smem<T>(TRANS), sm_upd = cp_upd_smem<T, C>(TRANS);
    if (gb300_func_dyn_smem((const void *)trsv_blk_kernel<T, TRANS>, (int)sm_blk) ||
        gb300_func_dyn_smem((const void *)trsv_upd_kernel<T, C, TRANS>, (int)sm_upd))
        return;
    const int nblk = (n + CP_SB - 1) / CP_SB;
    for (int b = 0; b < nblk; ++b) {
        const int j0 = (TRANS ? nblk - 1 - b : b) * CP_SB, w = std::min(CP_SB, n - j0);
        gb300_count_launch(), trsv_blk_kernel<T, TRANS>
            <<<nrhs, 256, sm_blk, s>>>(w, L + j0 + (long)j0 * ldl, ldl, B + j0, ldb, wait);
        const int rest = TRANS ? j0 : n - j0 - w;
        if (rest <= 0) continue;
        if constexpr (std::is_same<T, double>::value) {
            // B_rest -= L X (or L^T X) on the tensor cores (SLICE_MIN_ELEMENTS)
            if (rest >= SLICE_MIN_M && nrhs >= 16 && (long)rest * nrhs >= SLICE_MIN_ELEMENTS) {
                slice_update<true>(s, false, rest, nrhs, w, TRANS ? L + j0 : L + (j0 + w) + (long)j0 * ldl,
                                   TRANS ? ldl : 1, TRANS ? 1 : ldl, B + j0, ldb, 1, TRANS ? B : B + j0 + w, ldb, wait.err);
                continue;
            }
        }
        gb300_count_launch(), trsv_upd_kernel<T, C, TRANS><<<dim3(cdiv(rest, 32), cdiv(nrhs, C)), 256, sm_upd, s>>>(
            rest, w, nrhs, TRANS ? L + j0 : L + (j0 + w) + (long)j0 * ldl, ldl, B + j0, TRANS ? B : B + j0 + w, ldb);
    }
}

template <typename T, int C>
static void potrs_sweeps(cudaStream_t s, int n, int nrhs, const T *L, long ldl, T *B, long ldb, const CpWait &wait)
{
    potrs_sweep_blocks<T, C, false>(s, n, nrhs, L, ldl, B, ldb, wait);
    potrs_sweep_blocks<T, C, true>(s, n, nrhs, L, ldl, B, ldb, wait);
}

template <typename T>
void potrs_blocked(cudaStream_t s, int n, int nrhs, const T *L, long ldl, T *B, long ldb, int *err)
{
    if (n <= 0 || nrhs <= 0) return;
    const CpWait wait{gb300_wait_us(), err ? err : gb300_wait_status()};
    if (!wait.err) return;
    if (nrhs == 1) potrs_sweeps<T, 1>(s, n, nrhs, L, ldl, B, ldb, wait);
    else if (nrhs <= 4) potrs_sweeps<T, 4>(s, n, nrhs, L, ldl, B, ldb, wait);
    else potrs_sweeps<T, 8>(s, n, nrhs, L, ldl, B, ldb, wait);
}

// ---- single-launch POTRS sweeps with inverted 64 x 64 diagonal blocks ------

template <typename T>
size_t potrs_sweep_workspace(int n)
{
    const size_t nblk = ((size_t)n + 63) / 64;
    return ((nblk * 64 * 64 * sizeof(T) + 255) & ~(size_t)255) + (((nblk + 2) * sizeof(int) + 255) & ~(size_t)255);
}

// Invert every diagonal 64 x 64 block of L (once per factorisation).
template <typename T>
void potrs_sweep_prepare(cudaStream_t s, int n, const T *L, long ldl, void *ws)
{
    if (n <= 0) return;
    const unsigned nblk = cdiv(n, 64);
    gb300_count_launch(), invert_diag_blocks_kernel<T, 64><<<nblk, 64, 0, s>>>(n, L, ldl, (T *)ws, 64, 64 * 64, false);
}

// L y = b then L^T x = y, one launch per sweep and group of 16 columns (FP32).
template <typename T>
void potrs_sweep(cudaStream_t s, int n, int nrhs, const T *L, long ldl, void *ws, T *B, long ldb, int *err)
{
    if (n <= 0 || nrhs <= 0) return;
    const int nblk = (int)cdiv(n, 64);
    const T *Linv = (const T *)ws;
    int *flags = (int *)((char *)ws + (((size_t)nblk * 64 * 64 * sizeof(T) + 255) & ~(size_t)255));
    unsigned *ticket = (unsigned *)(flags + nblk);
    const unsigned long long budget = gb300_wait_budget_ns();
    static_assert(std::is_same<T, float>::value, "the single-launch sweeps are FP32");
    if (gb300_func_dyn_smem((const void *)trsv_sweep_kernel<false>, SWEEP_SMEM) ||
        gb300_func_dyn_smem((const void *)trsv_sweep_kernel<true>, SWEEP_SMEM))
        return;
    for (int c0 = 0; c0 < nrhs; c0 += 16) {
        const int nr = std::min(16, nrhs - c0);
        cudaMemsetAsync(flags, 0, (nblk + 1) * sizeof(int), s);
        gb300_count_launch(), trsv_sweep_kernel<false>
            <<<nblk, 256, SWEEP_SMEM, s>>>(n, nr, L, ldl, Linv, B + (long)c0 * ldb, ldb, ticket, flags, err, budget);
        cudaMemsetAsync(flags, 0, (nblk + 1) * sizeof(int), s);
        gb300_count_launch(), trsv_sweep_kernel<true>
            <<<nblk, 256, SWEEP_SMEM, s>>>(n, nr, L, ldl, Linv, B + (long)c0 * ldb, ldb, ticket, flags, err, budget);
    }
}

template size_t potrs_sweep_workspace<float>(int);
template size_t potrs_sweep_workspace<double>(int);
template void potrs_sweep_prepare<float>(cudaStream_t, int, const float *, long, void *);
template void potrs_sweep_prepare<double>(cudaStream_t, int, const double *, long, void *);
template void potrs_sweep<float>(cudaStream_t, int, int, const float *, long, void *, float *, long, int *);

template void gemm<float>(cudaStream_t, bool, bool, bool, int, int, int, float, const float *, long, const float *,
                          long, float, float *, long);
template void gemm<double>(cudaStream_t, bool, bool, bool, int, int, int, double, const double *, long,
                           const double *, long, double, double *, long);
template void trsm_rltn<float>(cudaStream_t, int, int, const float *, long, float *, long);
template void trsm_rltn<double>(cudaStream_t, int, int, const double *, long, double *, long);
template void trsm_llnn<float>(cudaStream_t, int, int, const float *, long, float *, long);
template void trsm_llnn<double>(cudaStream_t, int, int, const double *, long, double *, long);
template void trsm_runu<float>(cudaStream_t, int, int, const float *, long, float *, long);
template void trsm_runu<double>(cudaStream_t, int, int, const double *, long, double *, long);
template int potrf_tiled<float>(cudaStream_t, int, float *, long, int, int *, int);
template void trtri_lower<float>(cudaStream_t, int, const float *, long, float *, long, float *);
template int potrf_tiled<double>(cudaStream_t, int, double *, long, int, int *, int);
template void potrs_blocked<float>(cudaStream_t, int, int, const float *, long, float *, long, int *);
template void potrs_blocked<double>(cudaStream_t, int, int, const double *, long, double *, long, int *);

} // namespace gb300

using namespace gb300;

#define GB300_STREAM(s) ((cudaStream_t)(s))

extern "C" {

// ---- tile codelet bodies -------------------------------------------------

int starpu_gb300_spotrf_tile(void *stream, int n, float *A, int lda, int *d_info)
{
    if (n < 0 || lda < (n > 1 ? n : 1)) return GB300_EINVAL;
    if (d_info) cudaMemsetAsync(d_info, 0, sizeof(int), GB300_STREAM(stream));
    const int rc = n ? potrf_tiled<float>(GB300_STREAM(stream), n, A, lda, CP_W, d_info, 0) : GB300_OK;
    const int last = gb300_last_launch_status();
    return rc ? rc : last;
}

int starpu_gb300_dpotrf_tile(void *stream, int n, double *A, int lda, int *d_info)
{
    if (n < 0 || lda < (n > 1 ? n : 1)) return GB300_EINVAL;
    if (d_info) cudaMemsetAsync(d_info, 0, sizeof(int), GB300_STREAM(stream));
    const int rc = n ? potrf_tiled<double>(GB300_STREAM(stream), n, A, lda, CP_W, d_info, 0) : GB300_OK;
    const int last = gb300_last_launch_status();
    return rc ? rc : last;
}

int starpu_gb300_spotrf_tile_status(void *stream, int n, float *A, int lda, int *d_status)
{
    if (n < 0 || lda < (n > 1 ? n : 1)) return GB300_EINVAL;
    const int rc = n ? potrf_tiled<float>(GB300_STREAM(stream), n, A, lda, CP_W, d_status, 0) : GB300_OK;
    const int last = gb300_last_launch_status();
    return rc ? rc : last;
}

int starpu_gb300_dpotrf_tile_status(void *stream, int n, double *A, int lda, int *d_status)
{
    if (n < 0 || lda < (n > 1 ? n : 1)) return GB300_EINVAL;
    const int rc = n ? potrf_tiled<double>(GB300_STREAM(stream), n, A, lda, CP_W, d_status, 0) : GB300_OK;
    const int last = gb300_last_launch_status();
    return rc ? rc : last;
}

int starpu_gb300_strsm_rltn_tile(void *stream, int m, int n, float alpha, const float *L, int ldl, float *B, int ldb)
{
    if (m < 0 || n < 0 || ldl < (n > 1 ? n : 1) || ldb < (m > 1 ? m : 1)) return GB300_EINVAL;
    if (alpha != 1.0f) return GB300_ENOTSUP;
    trsm_rltn<float>(GB300_STREAM(stream), m, n, L, ldl, B, ldb);
    return gb300_last_launch_status();
}

int starpu_gb300_dtrsm_rltn_tile(void *stream, int m, int n, double alpha, const double *L, int ldl, double *B, int ldb)
{
    if (m < 0 || n < 0 || ldl < (n > 1 ? n : 1) || ldb < (m > 1 ? m : 1)) return GB300_EINVAL;
    if (alpha != 1.0) return GB300_ENOTSUP;
    trsm_rltn<double>(GB300_STREAM(stream), m, n, L, ldl, B, ldb);
    return gb300_last_launch_status();
}

int starpu_gb300_ssyrk_ln_tile(void *stream, int n, int k, float alpha, const float *A, int lda, float beta, float *C,
                               int ldc)
{
    if (n < 0 || k < 0 || lda < (n > 1 ? n : 1) || ldc < (n > 1 ? n : 1)) return GB300_EINVAL;
    gemm<float>(GB300_STREAM(stream), false, true, true, n, n, k, alpha, A, lda, A, lda, beta, C, ldc);
    return gb300_last_launch_status();
}

int starpu_gb300_dsyrk_ln_tile(void *stream, int n, int k, double alpha, const double *A, int lda, double beta,
                               double *C, int ldc)
{
    if (n < 0 || k < 0 || lda < (n > 1 ? n : 1) || ldc < (n > 1 ? n : 1)) return GB300_EINVAL;
    gemm<double>(GB300_STREAM(stream), false, true, true, n, n, k, alpha, A, lda, A, lda, beta, C, ldc);
    return gb300_last_launch_status();
}

int starpu_gb300_sgemm_nt_tile(void *stream, int m, int n, int k, float alpha, const float *A, int lda, const float *B,
                               int ldb, float beta, float *C, int ldc)
{
    if (m < 0 || n < 0 || k < 0 || lda < (m > 1 ? m : 1) || ldb < (n > 1 ? n : 1) || ldc < (m > 1 ? m : 1))
        return GB300_EINVAL;
    gemm<float>(GB300_STREAM(stream), false, true, false, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    return gb300_last_launch_status();
}

int starpu_gb300_dgemm_nt_tile(void *stream, int m, int n, int k, double alpha, const double *A, int lda,
                               const double *B, int ldb, double beta, double *C, int ldc)
{
    if (m < 0 || n < 0 || k < 0 || lda < (m > 1 ? m : 1) || ldb < (n > 1 ? n : 1) || ldc < (m > 1 ? m : 1))
        return GB300_EINVAL;
    gemm<double>(GB300_STREAM(stream), false, true, false, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    return gb300_last_launch_status();
}

// ---- whole-matrix plain-precision factorisation and solve -----------------

int starpu_gb300_spotrf(void *stream, int n, float *A, int lda, int nb, int *d_info)
{
    if (n < 0 || lda < (n > 1 ? n : 1) || nb < 0) return GB300_EINVAL;
    if (d_info) cudaMemsetAsync(d_info, 0, sizeof(int), GB300_STREAM(stream));
    const int rc = n ? potrf_tiled<float>(GB300_STREAM(stream), n, A, lda, nb ? nb : 512, d_info, 0) : GB300_OK;
    const int last = gb300_last_launch_status();
    return rc ? rc : last;
}

int starpu_gb300_dpotrf(void *stream, int n, double *A, int lda, int nb, int *d_info)
{
    if (n < 0 || lda < (n > 1 ? n : 1) || nb < 0) return GB300_EINVAL;
    if (d_info) cudaMemsetAsync(d_info, 0, sizeof(int), GB300_STREAM(stream));
    const int rc = n ? potrf_tiled<double>(GB300_STREAM(stream), n, A, lda, nb ? nb : 512, d_info, 0) : GB300_OK;
    const int last = gb300_last_launch_status();
    return rc ? rc : last;
}

int starpu_gb300_spotrs(void *stream, int n, int nrhs, const float *L, int ldl, float *B, int ldb)
{
    if (n < 0 || nrhs < 0 || ldl < (n > 1 ? n : 1) || ldb < (n > 1 ? n : 1)) return GB300_EINVAL;
    potrs_blocked<float>(GB300_STREAM(stream), n, nrhs, L, ldl, B, ldb, nullptr);
    return gb300_last_launch_status();
}

int starpu_gb300_dpotrs(void *stream, int n, int nrhs, const double *L, int ldl, double *B, int ldb)
{
    if (n < 0 || nrhs < 0 || ldl < (n > 1 ? n : 1) || ldb < (n > 1 ? n : 1)) return GB300_EINVAL;
    potrs_blocked<double>(GB300_STREAM(stream), n, nrhs, L, ldl, B, ldb, nullptr);
    return gb300_last_launch_status();
}

size_t starpu_gb300_spotrs_sweep_workspace(int n)
{
    if (n <= 0) return 0;
    return potrs_sweep_workspace<float>(n) + 256;
}

int starpu_gb300_spotrs_sweep(void *stream, int n, int nrhs, const float *L, int ldl, float *B, int ldb, void *work,
                              size_t lwork, int *d_err)
{
    if (n < 0 || nrhs < 0 || ldl < (n > 1 ? n : 1) || ldb < (n > 1 ? n : 1)) return GB300_EINVAL;
    if (!n || !nrhs) return GB300_OK;
    if (!work || lwork < starpu_gb300_spotrs_sweep_workspace(n) || !d_err) return GB300_EINVAL;
    cudaStream_t s = GB300_STREAM(stream);
    potrs_sweep_prepare<float>(s, n, L, ldl, work);
    potrs_sweep<float>(s, n, nrhs, L, ldl, work, B, ldb, d_err);
    return gb300_last_launch_status();
}

} // extern "C"
