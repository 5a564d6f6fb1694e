// Products on the FMA pipe: for the SpMM with fp32 blocks, whose split (simt_tile.cuh) every warp of a row would make of all of
// P, and for results of split products that are not finite.  128 threads = four warps, each of which owns a 32-row tile of the
// product and walks the contraction 32 elements ("a chunk") at a time out of shared memory.
//
// An SM multiplies 128 fp32 pairs per clock and issues four warp instructions per clock, so every issue slot that is not an FFMA
// costs arithmetic.  A thread's 4 x 8 outputs take 12 16-byte shared loads per 128 FFMAs (four steps of the contraction at
// once).  Lanes sit 8 (rows) x 4 (columns): rows are 8 apart, so that the 16-byte loads of a padded row-major tile (row stride = 4
// mod 32 words) touch each bank once.  Chunks travel by cp.async into the buffer the previous chunk has left (one
// __syncthreads per chunk); operands of 16-bit types are converted on the way in.
#pragma once
#include "simt_tile.cuh"

namespace sfb {
namespace fma_tile {

using tile::cp_async16;
using tile::kChunk;
using tile::kStride;
using tile::kThreads;

// A lane's place in the 8 x 4 grid of a warp tile.  Bits alternate between column and row, so that four neighbouring lanes
// make a 2 x 2 square: a 16-byte shared load then takes two wavefronts for either operand.  With the columns in the two
// low bits four neighbours read four different rows of the second operand, and that load takes four (measured).
__device__ __forceinline__ uint32_t lane_row(uint32_t lane) { return ((lane >> 1) & 1u) | ((lane >> 2) & 6u); }
__device__ __forceinline__ uint32_t lane_quad(uint32_t lane) { return (lane & 1u) | ((lane >> 1) & 2u); }    // lanes of one row: xor 1 and 4

// ROWS x COLS elements -> dst[r * stride + c] as fp32; element (r, c) is src[at + r * pitch + c]; columns from ncols on
// are zeros.  vec: 16-byte aligned rows (ncols then is a multiple of a 16-byte piece).  A thread keeps its piece of the
// row and steps down the rows, so a step is one pointer addition and one copy.
template <int DT, int ROWS, int COLS>
__device__ __forceinline__ void stage(float *dst, uint32_t stride, const void *src, size_t at, size_t pitch, uint32_t ncols, bool vec)
{
    if (vec) {
        constexpr int E = DT == SFB_F32 ? 4 : 8;              // elements per 16-byte piece
        constexpr int P = COLS / E, STEP = (int)kThreads / P;  // pieces per row, rows per step
        const uint32_t r0 = threadIdx.x / P, c = (threadIdx.x % P) * E;
        const bool in = c < ncols;
        float *d = dst + r0 * stride + c;
        if (DT == SFB_F32) {
            const float *q = (const float *)src + at + r0 * pitch + (in ? c : 0);
            const uint32_t bytes = in ? 16u : 0u;
#pragma unroll
            for (int i = 0; i < (ROWS + STEP - 1) / STEP; i++)
                if (ROWS % STEP == 0 || r0 + i * STEP < ROWS) cp_async16(d + i * STEP * stride, q + (size_t)i * STEP * pitch, bytes);
        } else {
            const uint16_t *q = (const uint16_t *)src + at + r0 * pitch + c;
#pragma unroll
            for (int i = 0; i < (ROWS + STEP - 1) / STEP; i++)
                if (ROWS % STEP == 0 || r0 + i * STEP < ROWS) {
                    uint4 u = make_uint4(0u, 0u, 0u, 0u);
                    if (in) u = __ldg((const uint4 *)(q + (size_t)i * STEP * pitch));
                    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
                    float v[8];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (DT == SFB_BF16) {
                            v[2 * k] = __uint_as_float(w[k] << 16);
                            v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
                        } else {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[k]));
                            v[2 * k] = f.x;
                            v[2 * k + 1] = f.y;
                        }
                    }
                    *(float4 *)(d + i * STEP * stride) = make_float4(v[0], v[1], v[2], v[3]);
                    *(float4 *)(d + i * STEP * stride + 4) = make_float4(v[4], v[5], v[6], v[7]);
                }
        }
    } else {
        for (uint32_t t = threadIdx.x; t < ROWS * COLS; t += kThreads) {
            const uint32_t r = t / COLS, c = t % COLS;
            dst[r * stride + c] = c < ncols ? Elem<DT>::load(src, at + r * pitch + c) : 0.f;
        }
    }
}

// ---- packed pairs: one fma.rn.f32x2 is two FFMAs in one issue slot
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t pair(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpair(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// TN columns of one row of the second operand, as TN / 2 pairs: contiguous groups of four (two when TN is 2), a lane's
// groups 16 apart
template <int TN>
__device__ __forceinline__ void load_cols(uint64_t (&v)[TN / 2], const float *row)
{
    if (TN == 2) {
        v[0] = *(const uint64_t *)row;
    } else {
#pragma unroll
        for (int j = 0; j < TN / 4; j++) {
            const ulonglong2 t = *(const ulonglong2 *)(row + 16 * j);
            v[2 * j] = t.x;
            v[2 * j + 1] = t.y;
        }
    }
}
// first column of this lane inside its warp's columns, and the column of acc[.][n]
template <int TN> __device__ __forceinline__ uint32_t lane_col(uint32_t lc) { return TN == 2 ? lc * 2 : lc * 4; }
template <int TN> __device__ __forceinline__ uint32_t acc_col(uint32_t lc, int n) { return TN == 2 ? lc * 2 + n : lc * 4 + (n >> 2) * 16 + (n & 3); }

// acc[m][n] += sum over one chunk of p[row m][k] * v[k][col n] on pairs of columns: p row-major along k (P . V).  p points
// at row lr.
template <int TN>
__device__ __forceinline__ void mma_nn(uint64_t (&acc)[4][TN / 2], const float *p, uint32_t p_stride, const float *v, uint32_t v_stride)
{
#pragma unroll 2
    for (uint32_t k = 0; k < kChunk; k += 4) {
        float4 x[4];
#pragma unroll
        for (int m = 0; m < 4; m++) x[m] = *(const float4 *)(p + m * 8 * p_stride + k);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint64_t y[TN / 2];
            load_cols<TN>(y, v + (k + j) * v_stride);
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const float s = j == 0 ? x[m].x : j == 1 ? x[m].y : j == 2 ? x[m].z : x[m].w;
                const uint64_t s2 = pair(s, s);
#pragma unroll
                for (int n = 0; n < TN / 2; n++) acc[m][n] = fma2(s2, y[n], acc[m][n]);
            }
        }
    }
}
// the same with p transposed in place, p[k][row] (P^T . V): this thread's four rows are neighbours; p points at its first
template <int TN>
__device__ __forceinline__ void mma_tn(uint64_t (&acc)[4][TN / 2], const float *p, uint32_t p_stride, const float *v, uint32_t v_stride)
{
#pragma unroll 8
    for (uint32_t k = 0; k < kChunk; k++) {
        const float4 x = *(const float4 *)(p + k * p_stride);
        uint64_t y[TN / 2];
        load_cols<TN>(y, v + k * v_stride);
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const float s = m == 0 ? x.x : m == 1 ? x.y : m == 2 ? x.z : x.w;
            const uint64_t s2 = pair(s, s);
#pragma unroll
            for (int n = 0; n < TN / 2; n++) acc[m][n] = fma2(s2, y[n], acc[m][n]);
        }
    }
}

// TN accumulators of one output row -> row (element offset of the warp's first column), columns from ncols on not written.
// AGAIN: only where what is there is not finite
template <int DT, int TN, bool AGAIN>
__device__ __forceinline__ void store_row(void *out, size_t row, uint32_t lc, const uint64_t (&acc)[TN / 2], uint32_t ncols, bool vec)
{
    float v[TN];
#pragma unroll
    for (int n = 0; n < TN / 2; n++) {
        const float2 f = unpair(acc[n]);
        v[2 * n] = f.x;
        v[2 * n + 1] = f.y;
    }
    if (vec && TN >= 4 && !AGAIN) {
#pragma unroll
        for (int j = 0; j < TN / 4; j++) {
            const uint32_t c = lc * 4 + 16 * j;
            if (c < ncols) {
                if (DT == SFB_F32) {
                    *(float4 *)((float *)out + row + c) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                } else {
                    uint2 w;
                    if (DT == SFB_BF16) {
                        w.x = to_bhalf_bits(v[4 * j]) | ((uint32_t)to_bhalf_bits(v[4 * j + 1]) << 16);
                        w.y = to_bhalf_bits(v[4 * j + 2]) | ((uint32_t)to_bhalf_bits(v[4 * j + 3]) << 16);
                    } else {
                        __half2 h0 = __floats2half2_rn(v[4 * j], v[4 * j + 1]), h1 = __floats2half2_rn(v[4 * j + 2], v[4 * j + 3]);
                        w.x = *reinterpret_cast<uint32_t *>(&h0);
                        w.y = *reinterpret_cast<uint32_t *>(&h1);
                    }
                    *(uint2 *)((uint16_t *)out + row + c) = w;
                }
            }
        }
    } else {
#pragma unroll
        for (int n = 0; n < TN; n++) {
            const uint32_t c = acc_col<TN>(lc, n);
            if (c < ncols && !(AGAIN && tile::finite(Elem<DT>::load(out, row + c)))) Elem<DT>::store(out, row + c, v[n]);
        }
    }
}

}  // namespace fma_tile
}  // namespace sfb
