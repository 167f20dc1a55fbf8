// Products of 64 x 64 FP32 tiles by one CTA of 256 threads, for the persistent
// factorisations (diag_coop.cuh, batched_chol.cuh): tiles are read from
// column-major global matrices that other CTAs of the launch write (through
// L2), staged in shared memory and multiplied on the FP32 pipe.  The loads of
// both operands and of the updated tile are all in flight before the product
// (one memory latency per tile), 16 bytes each where a tile is whole.
#pragma once
#include <cuda_runtime.h>

namespace gb300 {

constexpr int DC_B = 64;         // block order
constexpr int DC_T = 256;        // threads per CTA
constexpr int DC_LD = DC_B + 4;  // pitch of a shared tile (column-major: s[c * DC_LD + r]); float4-aligned

// One thread's 16 elements of a 64 x 64 tile (rows x cols of a column-major
// global matrix, zero outside): all loads in flight together, 16 bytes each
// where the tile is whole and aligned (vec).
struct DcTile {
    float4 v[4];
    __device__ __forceinline__ void load(const float *g, long ld, int rows, int cols, bool vec)
    {
        if (vec && rows == DC_B && cols == DC_B) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = threadIdx.x + q * DC_T, r4 = e & 15, c = e >> 4;
                v[q] = __ldcg(reinterpret_cast<const float4 *>(g + 4 * r4 + (long)c * ld));
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = threadIdx.x + q * DC_T, r = 4 * (e & 15), c = e >> 4;
                const float *p = g + r + (long)c * ld;
                const bool in = c < cols;
                v[q].x = in && r < rows ? __ldcg(p) : 0.0f;
                v[q].y = in && r + 1 < rows ? __ldcg(p + 1) : 0.0f;
                v[q].z = in && r + 2 < rows ? __ldcg(p + 2) : 0.0f;
                v[q].w = in && r + 3 < rows ? __ldcg(p + 3) : 0.0f;
            }
        }
    }
    // to a shared tile: column-major (s[c * DC_LD + r]), or p-major (s[r * DC_LD + c])
    __device__ __forceinline__ void store(float *s) const
    {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = threadIdx.x + q * DC_T;
            *reinterpret_cast<float4 *>(s + (e >> 4) * DC_LD + 4 * (e & 15)) = v[q];
        }
    }
    __device__ __forceinline__ void store_t(float *s) const
    {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = threadIdx.x + q * DC_T, c = e >> 4, r = 4 * (e & 15);
            s[r * DC_LD + c] = v[q].x;
            s[(r + 1) * DC_LD + c] = v[q].y;
            s[(r + 2) * DC_LD + c] = v[q].z;
            s[(r + 3) * DC_LD + c] = v[q].w;
        }
    }
};

// acc += As * Bs for 64 x 64 shared tiles: As column-major (As[p * DC_LD + r]
// = A(r, p)), Bs stored p-major (Bs[p * DC_LD + c] = B(p, c)) -- which is how
// DcTile::store leaves a tile whose transpose is the operand (NT products).
// Thread (tr = tid % 16, tn = tid / 16) owns rows 4 tr .. 4 tr + 3 and
// columns 4 tn .. 4 tn + 3: two float4 shared loads per 16 FMAs.  kmax: terms.
__device__ __forceinline__ void dc_mma(const float *As, const float *Bs, float acc[4][4], int kmax = DC_B)
{
    const int tr = threadIdx.x & 15, tn = threadIdx.x >> 4;
#pragma unroll 8
    for (int p = 0; p < kmax; ++p) {
        const float4 av = *reinterpret_cast<const float4 *>(As + p * DC_LD + 4 * tr);
        const float4 bv = *reinterpret_cast<const float4 *>(Bs + p * DC_LD + 4 * tn);
        const float ar[4] = {av.x, av.y, av.z, av.w}, br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
    }
}

// The thread's 4 x 4 elements of C (rows x cols of a column-major global
// matrix; `lower` keeps only those on or below the diagonal), read before the
// product and written after it.  whole: every element, 16 bytes at a time.
__device__ __forceinline__ bool dc_whole(int rows, int cols, bool lower, bool vec)
{
    return vec && rows == DC_B && cols == DC_B && !lower;
}
__device__ __forceinline__ void dc_sub_load(const float *C, long ld, int rows, int cols, bool lower, bool whole,
                                            float (&c)[4][4])
{
    const int r0 = 4 * (threadIdx.x & 15), c0 = 4 * (threadIdx.x >> 4);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float *p = C + r0 + (long)(c0 + j) * ld;
        if (whole) {
            const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
            c[0][j] = v.x, c[1][j] = v.y, c[2][j] = v.z, c[3][j] = v.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                c[i][j] = c0 + j < cols && r0 + i < rows && (!lower || c0 + j <= r0 + i) ? __ldcg(p + i) : 0.0f;
        }
    }
}
__device__ __forceinline__ void dc_sub_store(float *C, long ld, int rows, int cols, bool lower, bool whole,
                                             const float (&c)[4][4], const float (&acc)[4][4])
{
    const int r0 = 4 * (threadIdx.x & 15), c0 = 4 * (threadIdx.x >> 4);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float *p = C + r0 + (long)(c0 + j) * ld;
        if (whole) {
            *reinterpret_cast<float4 *>(p) = make_float4(c[0][j] - acc[0][j], c[1][j] - acc[1][j], c[2][j] - acc[2][j],
                                                         c[3][j] - acc[3][j]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c0 + j < cols && r0 + i < rows && (!lower || c0 + j <= r0 + i)) p[i] = c[i][j] - acc[i][j];
        }
    }
}

} // namespace gb300
