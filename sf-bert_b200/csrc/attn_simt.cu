// FP32-arithmetic (CUDA-core) kernels of the block-sparse attention path: SDDMM, masked softmax,
// SpMM and the two block-row-owned fusions.  They serve fp32 operands (1e-5 parity with the CPU
// reference cannot be met on tensor cores) and every shape the tcgen05 kernels do not cover.
//
// SDDMM, SpMM, the fused attention and the fp32 element-sparse tiles are made of warp tiles of 4 x 8
// outputs per thread (simt_tile.cuh).  The fused SDDMM + softmax (fused_sddmm_softmax_kernel) has 256
// threads as a 16x16 grid; thread (ty,tx) owns rows ty+16m and columns tx+16n of a tile, so the 16
// lanes of a half-warp own one set of rows and row reductions are four shuffles.
#include "simt_tile.cuh"
#include "csr.cuh"
#include <float.h>
#include <math.h>

namespace sfb {

#define LOG2E_F 1.4426950408889634f


template <int BS>
struct MaskWord { typedef uint32_t type; };
template <>
struct MaskWord<64> { typedef uint64_t type; };

// loads rows [row0, row0+BS) x columns [k0, k0+KC) of a [*, HD] row-major operand into smem as
// dst[k][r] (k-major, row stride BS+1), zero beyond d
template <int DT, int BS, int KC>
__device__ __forceinline__ void load_tile_kmajor(float (*dst)[BS + 1], const void *src, size_t base, size_t HD,
                                                 uint32_t k0, uint32_t d)
{
    for (uint32_t e = threadIdx.x; e < BS * KC; e += 256) {
        uint32_t r = e / KC, k = e % KC;
        float v = 0.f;
        if (k0 + k < d) v = Elem<DT>::load(src, base + (size_t)r * HD + k0 + k);
        dst[k][r] = v;
    }
}

// ------------------------------------------------------------------------------------------------
// SDDMM.  A CTA (four warps) makes one 64x64 block, a 32x32 quarter per warp, or four consecutive 32x32 blocks of the LUT,
// one per warp.  Consecutive blocks mostly share their block-row (the LUT is in row-major scan order): its query rows
// are then staged once for the four.  Both operands come chunk by chunk (32 of d) through two buffers; the scores leave
// through shared memory, eight per lane, so that a row is written in whole pieces of 16 or 32 bytes.
template <int BS, int AB_DT, int C_DT>
__global__ void __launch_bounds__(tile::kThreads, 3) sddmm_nt_kernel(const uint2 *__restrict__ lut, const void *__restrict__ A,
                                                                   const void *__restrict__ Bm, void *__restrict__ C, AttnDims p, bool vec)
{
    using namespace tile;
    constexpr uint32_t PER = BS == 32 ? 4 : 1;               // blocks per CTA
    constexpr uint32_t ROWS = PER * BS;                      // staged rows of each operand: 128 or 64
    constexpr uint32_t BUF = 2 * ROWS * kStride;
    extern __shared__ __align__(16) float sm[];              // [2][A rows | B rows]
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane_row(lane), lc = lane_quad(lane);
    const uint32_t bid0 = blockIdx.x * PER, b = blockIdx.y, h = blockIdx.z;
    const uint32_t nblk = min(PER, p.blocks - bid0);
    const size_t HD = (size_t)p.H * p.d;
    const size_t head = (size_t)h * p.d;
    size_t offA[PER], offB[PER];
    bool shared_rows = true;
    {
        const uint2 *e = lut + (size_t)h * p.lut_stride + bid0;
        const uint32_t x0 = e[0].x;
#pragma unroll
        for (uint32_t k = 0; k < PER; k++) {
            const uint2 en = k < nblk ? e[k] : e[0];
            offA[k] = ((size_t)b * p.nb_a + en.x) * BS * HD + head;
            offB[k] = ((size_t)b * p.nb_b + en.y) * BS * HD + head;
            shared_rows = shared_rows && en.x == x0;
        }
    }
    auto issue = [&](uint32_t c) {
        float *buf = sm + (c & 1) * BUF;
        const uint32_t k0 = c * kChunk, left = p.d - k0;
#pragma unroll
        for (uint32_t g = 0; g < PER; g++)
            if (g < nblk) {
                if (g == 0 || !shared_rows) stage<AB_DT, BS, (int)kChunk>(buf + g * BS * kStride, kStride, A, offA[g] + k0, HD, left, vec);
                stage<AB_DT, BS, (int)kChunk>(buf + (ROWS + g * BS) * kStride, kStride, Bm, offB[g] + k0, HD, left, vec);
            }
        cp_commit();
    };
    const bool live = BS == 64 || warp < nblk;
    const uint32_t r0 = BS == 64 ? 32 * (warp >> 1) : (shared_rows ? 0 : 32 * warp), c0 = BS == 64 ? 32 * (warp & 1) : 32 * warp;
    uint64_t acc[4][8];
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int n = 0; n < 8; n++) acc[m][n] = 0;
    const uint32_t chunks = (p.d + kChunk - 1) / kChunk;
    issue(0);
    for (uint32_t c = 0; c < chunks; c++) {
        cp_wait_all();
        __syncthreads();
        if (c + 1 < chunks) issue(c + 1);
        const float *buf = sm + (c & 1) * BUF;
        if (live) mma_nt(acc, buf + (r0 + lr) * kStride, kStride, buf + (ROWS + c0 + lc) * kStride, kStride);
    }
    __syncthreads();
    if (!live) return;
    float *t = sm + warp * 32 * kStride;
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int n = 0; n < 8; n++) t[(lr + 8 * m) * kStride + lc + 4 * n] = half_sum(acc[m][n]);
    __syncwarp();
    const size_t baseC = (((size_t)b * p.H + h) * p.blocks + bid0 + (BS == 64 ? 0 : warp)) * BS * BS + (BS == 64 ? (size_t)r0 * BS + c0 : 0);
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const float *row = t + (lr + 8 * m) * kStride + lc * 8;
        const float4 u = *(const float4 *)row, w = *(const float4 *)(row + 4);
        const float v[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
        const size_t at = baseC + (size_t)(lr + 8 * m) * BS + lc * 8;
        if (vec) {
            if (C_DT == SFB_F32) {
                *(float4 *)((float *)C + at) = u;
                *(float4 *)((float *)C + at + 4) = w;
            } else {
                uint32_t q[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (C_DT == SFB_BF16) q[k] = to_bhalf_bits(v[2 * k]) | ((uint32_t)to_bhalf_bits(v[2 * k + 1]) << 16);
                    else {
                        __half2 hh = __floats2half2_rn(v[2 * k], v[2 * k + 1]);
                        q[k] = *reinterpret_cast<uint32_t *>(&hh);
                    }
                }
                *(uint4 *)((uint16_t *)C + at) = make_uint4(q[0], q[1], q[2], q[3]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) Elem<C_DT>::store(C, at + k, v[k]);
        }
    }
}

// ------------------------------------------------------------------------------------------------
template <int Y_DT>
__device__ __forceinline__ void store8(void *y, size_t idx, const float (&v)[8])
{
    if (Y_DT == SFB_F32) {
        float4 *p = (float4 *)((float *)y + idx);
        p[0] = make_float4(v[0], v[1], v[2], v[3]);
        p[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (Y_DT == SFB_BF16) {
                // probabilities: the hardware's round-to-nearest-even pack (one instruction per pair); it differs
                // from the reference's add-half-and-truncate rounding (ew_op_gpu.h:241-253) on exact ties only
                __nv_bfloat162 hb = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                w[i] = *reinterpret_cast<uint32_t *>(&hb);
            } else {
                __half2 hh = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                w[i] = *reinterpret_cast<uint32_t *>(&hh);
            }
        }
        *(uint4 *)((uint16_t *)y + idx) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// raw 16-byte (16-bit types) or 32-byte (fp32) load of 8 scores, kept unconverted so that many can be in flight
template <int X_DT> struct Raw8 { uint4 a; };
template <> struct Raw8<SFB_F32> { uint4 a, b; };

template <int X_DT>
__device__ __forceinline__ Raw8<X_DT> load_raw8(const void *x, size_t idx)
{
    Raw8<X_DT> r;
    if (X_DT == SFB_F32) {
        const uint4 *p = (const uint4 *)((const float *)x + idx);
        r.a = __ldg(p);
        ((Raw8<SFB_F32> &)r).b = __ldg(p + 1);
    } else {
        r.a = __ldg((const uint4 *)((const uint16_t *)x + idx));
    }
    return r;
}

template <int X_DT>
__device__ __forceinline__ void unpack8(float (&v)[8], const Raw8<X_DT> &r)
{
    if (X_DT == SFB_F32) {
        const Raw8<SFB_F32> &q = (const Raw8<SFB_F32> &)r;
        v[0] = __uint_as_float(q.a.x); v[1] = __uint_as_float(q.a.y); v[2] = __uint_as_float(q.a.z); v[3] = __uint_as_float(q.a.w);
        v[4] = __uint_as_float(q.b.x); v[5] = __uint_as_float(q.b.y); v[6] = __uint_as_float(q.b.z); v[7] = __uint_as_float(q.b.w);
    } else {
        const uint32_t w[4] = {r.a.x, r.a.y, r.a.z, r.a.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (X_DT == SFB_BF16) {
                v[2 * i] = __uint_as_float(w[i] << 16);
                v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
            } else {
                float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
                v[2 * i] = f.x;
                v[2 * i + 1] = f.y;
            }
        }
    }
}

__device__ __forceinline__ float ex2_fast(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Masked softmax: one CTA per block-row.  A lane owns 8 consecutive keys of one query row of one block
// (16 bytes of bf16), so a warp reads 512 contiguous bytes per block; the lanes of a row (BS/8 of them)
// combine with shuffles.
//
// NB > 0: the row has at most NB blocks.  All of them are loaded up front (NB independent 16-byte loads per
// lane in flight) and stay in registers: one pass over HBM, one exponential per element.
// NB == 0: rows of any length.  Pass 1 finds the row maximum, pass 2 the sum of exponentials, pass 3 writes;
// passes 2 and 3 re-read scores this CTA has just pulled through L2.
// SPLIT > 1: the block-row is shared by SPLIT CTAs of BS/SPLIT query rows each.  Registers decide how many of the
// register-resident CTAs an SM holds, and small CTAs fill what the register file leaves: with loads of some CTAs in
// flight while others compute and store, the 12- and 16-block rows run at the speed of a copy (0.98 of it; a CTA per
// whole block-row, one per SM, reached 0.6-0.7).
// The second launch bound asks for the number of CTAs per SM that the variant's registers allow anyway (it keeps the
// compiler from spending registers the occupancy needs).
template <int BS, int X_DT, int Y_DT, int NB, int SPLIT>
__global__ void __launch_bounds__(BS * BS / 8 / SPLIT, (NB > 0 && SPLIT > 1 && BS == 64 && X_DT != SFB_F32) ? (NB <= 12 ? 6 : NB <= 18 ? 5 : 4) : 1) softmax_kernel(const uint2 *__restrict__ lut,
                                                                const typename MaskWord<BS>::type *__restrict__ mask,
                                                                const void *__restrict__ X, void *__restrict__ Y, AttnDims p,
                                                                float scale_log2e, int rescale_in_place)
{
    typedef typename MaskWord<BS>::type W;
    constexpr int LPR = BS / 8;  // lanes per query row
    grid_dependency_wait();
    grid_launch_dependents();
    // last (batch, head) first: the scores were written in ascending order, and the last of them are still in L2
    const uint32_t i = blockIdx.x / SPLIT, b = gridDim.y - 1 - blockIdx.y, h = gridDim.z - 1 - blockIdx.z;
    const uint2 *nn = lut + (size_t)h * p.lut_stride;
    const uint2 head = nn[i];
    const uint32_t off = head.x, cnt = head.y;
    if (cnt == 0) return;
    const uint32_t r = (blockIdx.x % SPLIT) * (BS / SPLIT) + threadIdx.x / LPR;        // query row inside the block
    const uint32_t c0 = (threadIdx.x % LPR) * 8;  // first key of this lane
    const size_t base = ((size_t)b * p.H + h) * p.blocks * BS * BS + (size_t)r * BS + c0;
    const W *mrow = mask ? mask + (size_t)h * p.mask_stride + (size_t)r * p.blocks : nullptr;

    if (NB > 0) {
        constexpr int N = NB > 0 ? NB : 1;
        Raw8<X_DT> raw[N];
        uint32_t blks[N], bits[N];
#pragma unroll
        for (int j = 0; j < N; j++) {
            blks[j] = 0;
            bits[j] = 0;
            if (j < (int)cnt) {
                blks[j] = nn[off + j].x;
                raw[j] = load_raw8<X_DT>(X, base + (size_t)blks[j] * BS * BS);
                bits[j] = mrow ? (uint32_t)((__ldg(mrow + blks[j]) >> c0) & 0xffu) : 0xffu;
            }
        }
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < N; j++) {
            if (j < (int)cnt) {
                float v[8];
                unpack8<X_DT>(v, raw[j]);
#pragma unroll
                for (int t = 0; t < 8; t++)
                    if ((bits[j] >> t) & 1u) mx = fmaxf(mx, v[t]);
            }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float mxs = mx > -INFINITY ? mx * scale_log2e : 0.f;
        // second sweep: one exponential per score; the results replace the raw scores in their registers as
        // packed fp16 pairs (e is in (0, 1], 11 bits are more than the 16-bit output keeps)
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < N; j++) {
            if (j < (int)cnt) {
                float v[8];
                unpack8<X_DT>(v, raw[j]);
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    v[t] = ((bits[j] >> t) & 1u) ? ex2_fast(fmaf(v[t], scale_log2e, -mxs)) : 0.f;
                    sum += v[t];
                }
                if (Y_DT != SFB_F32) {   // fp32 outputs recompute the exponential below instead: fp16 would cost them bits
                    __half2 h0 = __floats2half2_rn(v[0], v[1]), h1 = __floats2half2_rn(v[2], v[3]);
                    __half2 h2 = __floats2half2_rn(v[4], v[5]), h3 = __floats2half2_rn(v[6], v[7]);
                    raw[j].a = make_uint4(*reinterpret_cast<uint32_t *>(&h0), *reinterpret_cast<uint32_t *>(&h1),
                                          *reinterpret_cast<uint32_t *>(&h2), *reinterpret_cast<uint32_t *>(&h3));
                }
            }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float inv = sum > 0.f ? 1.f / sum : 0.f;
#pragma unroll
        for (int j = 0; j < N; j++) {
            if (j < (int)cnt) {
                float v[8];
                if (Y_DT != SFB_F32) {
                    const uint32_t w[4] = {raw[j].a.x, raw[j].a.y, raw[j].a.z, raw[j].a.w};
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[t]));
                        v[2 * t] = f.x * inv;
                        v[2 * t + 1] = f.y * inv;
                    }
                } else {
                    unpack8<X_DT>(v, raw[j]);
#pragma unroll
                    for (int t = 0; t < 8; t++)
                        v[t] = ((bits[j] >> t) & 1u) ? ex2_fast(fmaf(v[t], scale_log2e, -mxs)) * inv : 0.f;
                }
                store8<Y_DT>(Y, base + (size_t)blks[j] * BS * BS, v);
            }
        }
        return;
    }

    // pass 1: the row maximum (packed bf16 max when there is no mask: 4 instructions per 8 scores)
    float mx = -INFINITY;
    if (X_DT == SFB_BF16 && !mrow) {
        uint32_t acc[4] = {0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u};   // pairs of -inf
        for (uint32_t e = 0; e < cnt; e++) {
            const uint32_t blk = nn[off + e].x;
            const Raw8<X_DT> r8 = load_raw8<X_DT>(X, base + (size_t)blk * BS * BS);
            const uint32_t w[4] = {r8.a.x, r8.a.y, r8.a.z, r8.a.w};
#pragma unroll
            for (int t = 0; t < 4; t++) {
                __nv_bfloat162 m2 = __hmax2(*reinterpret_cast<__nv_bfloat162 *>(&acc[t]), *reinterpret_cast<const __nv_bfloat162 *>(&w[t]));
                acc[t] = *reinterpret_cast<uint32_t *>(&m2);
            }
        }
#pragma unroll
        for (int t = 0; t < 4; t++)
            mx = fmaxf(mx, fmaxf(__uint_as_float(acc[t] << 16), __uint_as_float(acc[t] & 0xffff0000u)));
    } else {
        for (uint32_t e = 0; e < cnt; e++) {
            const uint32_t blk = nn[off + e].x;
            float v[8];
            unpack8<X_DT>(v, load_raw8<X_DT>(X, base + (size_t)blk * BS * BS));
            const uint32_t bits = mrow ? (uint32_t)((__ldg(mrow + blk) >> c0) & 0xffu) : 0xffu;
#pragma unroll
            for (int t = 0; t < 8; t++)
                if ((bits >> t) & 1u) mx = fmaxf(mx, v[t]);
        }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float mxs = mx > -INFINITY ? mx * scale_log2e : 0.f;
    // pass 2: one exponential per score; the unnormalised value goes to Y in the output type
    float sum = 0.f;
    for (uint32_t e = 0; e < cnt; e++) {
        const uint32_t blk = nn[off + e].x;
        float v[8];
        unpack8<X_DT>(v, load_raw8<X_DT>(X, base + (size_t)blk * BS * BS));
        if (mrow) {
            const uint32_t bits = (uint32_t)((__ldg(mrow + blk) >> c0) & 0xffu);
#pragma unroll
            for (int t = 0; t < 8; t++) v[t] = ((bits >> t) & 1u) ? ex2_fast(fmaf(v[t], scale_log2e, -mxs)) : 0.f;
        } else {
#pragma unroll
            for (int t = 0; t < 8; t++) v[t] = ex2_fast(fmaf(v[t], scale_log2e, -mxs));
        }
#pragma unroll
        for (int t = 0; t < 8; t++) sum += v[t];
        if (rescale_in_place) store8<Y_DT>(Y, base + (size_t)blk * BS * BS, v);
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    if (!rescale_in_place) {
        // pass 3 for long rows (their Y would not stay in L2 between two passes): exponentials again, from X
        for (uint32_t e = 0; e < cnt; e++) {
            const uint32_t blk = nn[off + e].x;
            float v[8];
            unpack8<X_DT>(v, load_raw8<X_DT>(X, base + (size_t)blk * BS * BS));
            const uint32_t bits = mrow ? (uint32_t)((__ldg(mrow + blk) >> c0) & 0xffu) : 0xffu;
#pragma unroll
            for (int t = 0; t < 8; t++) v[t] = ((bits >> t) & 1u) ? ex2_fast(fmaf(v[t], scale_log2e, -mxs)) * inv : 0.f;
            store8<Y_DT>(Y, base + (size_t)blk * BS * BS, v);
        }
        return;
    }
    // pass 3: every thread rescales the values it wrote itself (they are still in L2): packed multiplies
    for (uint32_t e = 0; e < cnt; e++) {
        const uint32_t blk = nn[off + e].x;
        const size_t idx = base + (size_t)blk * BS * BS;
        if (Y_DT == SFB_F32) {
            float4 *py = (float4 *)((float *)Y + idx);
            float4 y0 = py[0], y1 = py[1];
            py[0] = make_float4(y0.x * inv, y0.y * inv, y0.z * inv, y0.w * inv);
            py[1] = make_float4(y1.x * inv, y1.y * inv, y1.z * inv, y1.w * inv);
        } else {
            uint4 *py = (uint4 *)((uint16_t *)Y + idx);
            uint4 u = *py;
            uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (Y_DT == SFB_BF16) {
                    __nv_bfloat162 r2 = __hmul2(*reinterpret_cast<__nv_bfloat162 *>(&w[t]), __float2bfloat162_rn(inv));
                    w[t] = *reinterpret_cast<uint32_t *>(&r2);
                } else {
                    const float2 f = __half22float2(*reinterpret_cast<__half2 *>(&w[t]));
                    __half2 r2 = __floats2half2_rn(f.x * inv, f.y * inv);
                    w[t] = *reinterpret_cast<uint32_t *>(&r2);
                }
            }
            *py = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Softmax gradient: dx = (dy - sum over the query row of dy*y) * y * scale.  Same decomposition as the forward
// softmax: one CTA per block-row, a lane owns 8 consecutive keys of one query row of one block.
// NB > 0: the row has at most NB blocks; dy and y of all of them are loaded up front and stay in registers
// (one pass over HBM).  NB == 0: any length; the second sweep re-reads what the first pulled through L2.
// SPLIT > 1: the block-row is shared by SPLIT CTAs of BS/SPLIT query rows each -- fewer threads per CTA leave more
// registers per thread, which is what lets longer rows stay register-resident.
template <int BS, int DT, int NB, int SPLIT>
__global__ void __launch_bounds__(BS * BS / 8 / SPLIT) softmax_grad_kernel(const uint2 *__restrict__ lut, const void *__restrict__ DY,
                                                                     const void *__restrict__ Y, void *__restrict__ DX, AttnDims p,
                                                                     float scale)
{
    constexpr int LPR = BS / 8;  // lanes per query row
    grid_dependency_wait();
    grid_launch_dependents();
    // last (batch, head) first, as the softmax: dy was written in ascending order
    const uint32_t i = blockIdx.x / SPLIT, b = gridDim.y - 1 - blockIdx.y, h = gridDim.z - 1 - blockIdx.z;
    const uint2 *nn = lut + (size_t)h * p.lut_stride;
    const uint2 head = nn[i];
    const uint32_t off = head.x, cnt = head.y;
    if (cnt == 0) return;
    const uint32_t r = (blockIdx.x % SPLIT) * (BS / SPLIT) + threadIdx.x / LPR;
    const uint32_t c0 = (threadIdx.x % LPR) * 8;
    const size_t base = ((size_t)b * p.H + h) * p.blocks * BS * BS + (size_t)r * BS + c0;

    if (NB > 0) {
        constexpr int N = NB > 0 ? NB : 1;
        Raw8<DT> rdy[N], ry[N];
        uint32_t blks[N];
#pragma unroll
        for (int j = 0; j < N; j++) {
            blks[j] = 0;
            if (j < (int)cnt) {
                blks[j] = nn[off + j].x;
                rdy[j] = load_raw8<DT>(DY, base + (size_t)blks[j] * BS * BS);
                ry[j] = load_raw8<DT>(Y, base + (size_t)blks[j] * BS * BS);
            }
        }
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < N; j++)
            if (j < (int)cnt) {
                float a[8], c[8];
                unpack8<DT>(a, rdy[j]);
                unpack8<DT>(c, ry[j]);
#pragma unroll
                for (int t = 0; t < 8; t++) sum = fmaf(a[t], c[t], sum);
            }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int j = 0; j < N; j++)
            if (j < (int)cnt) {
                float a[8], c[8];
                unpack8<DT>(a, rdy[j]);
                unpack8<DT>(c, ry[j]);
#pragma unroll
                for (int t = 0; t < 8; t++) a[t] = (a[t] - sum) * c[t] * scale;
                store8<DT>(DX, base + (size_t)blks[j] * BS * BS, a);
            }
        return;
    }
    float sum = 0.f;
    for (uint32_t e = 0; e < cnt; e++) {
        const size_t at = base + (size_t)nn[off + e].x * BS * BS;
        float a[8], c[8];
        unpack8<DT>(a, load_raw8<DT>(DY, at));
        unpack8<DT>(c, load_raw8<DT>(Y, at));
#pragma unroll
        for (int t = 0; t < 8; t++) sum = fmaf(a[t], c[t], sum);
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    for (uint32_t e = 0; e < cnt; e++) {
        const size_t at = base + (size_t)nn[off + e].x * BS * BS;
        float a[8], c[8];
        unpack8<DT>(a, load_raw8<DT>(DY, at));
        unpack8<DT>(c, load_raw8<DT>(Y, at));
#pragma unroll
        for (int t = 0; t < 8; t++) a[t] = (a[t] - sum) * c[t] * scale;
        store8<DT>(DX, at, a);
    }
}

// ------------------------------------------------------------------------------------------------
// SpMM: one CTA per (block-row, slice of up to 128 of d).  TRANS = false: O = sum over the row's blocks of P . V (NN, the
// lut is the nn_lut).  TRANS = true: the backward products dV = P^T dO and dK = dS^T Q -- the lut is the tn_lut,
// "row" i is a block COLUMN, an entry names a block of that column and the block-row its B rows come from, and
// the block is used transposed (read as it lies, four neighbouring rows of P^T per 16-byte load).
// A chunk is 32 elements of the contraction: one 32x32 block, or half of a 64x64 one, with its 32 rows of V.
template <int BS, int DS> struct SpmmCfg {
    static constexpr int WC = BS == 32 ? 4 : 2;                          // warps side by side along d
    static constexpr int TN = DS / WC / 4;                               // columns per thread
    static constexpr uint32_t a_floats = BS == 32 ? 32 * tile::kStride : 64 * tile::kStride > 32 * (64 + 4) ? 64 * tile::kStride : 32 * (64 + 4);
    static constexpr uint32_t buf = a_floats + 32 * (DS + 4);
};
template <int BS, int DS, int A_DT, int BC_DT, bool TRANS>
__global__ void __launch_bounds__(tile::kThreads, 4) spmm_nn_kernel(const uint2 *__restrict__ lut, const void *__restrict__ Pm,
                                                                  const void *__restrict__ V, void *__restrict__ O, AttnDims p, bool avec,
                                                                  bool vec)
{
    using namespace tile;
    typedef SpmmCfg<BS, DS> Cfg;
    constexpr int TN = Cfg::TN;
    constexpr uint32_t PARTS = BS / 32;                                  // chunks per block
    constexpr uint32_t a_stride = TRANS ? BS + 4 : kStride;
    extern __shared__ __align__(16) float sm[];                          // [2][P chunk | V chunk]
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t nslice = (p.d + DS - 1) / DS;
    const uint32_t i = blockIdx.x / nslice, d0 = (blockIdx.x % nslice) * DS;
    const uint32_t b = blockIdx.y, h = blockIdx.z;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane_row(lane), lc = lane_quad(lane);
    const uint2 *nn = lut + (size_t)h * p.lut_stride;
    const uint2 head = nn[i];
    const size_t HD = (size_t)p.H * p.d;
    const size_t bh = (size_t)b * p.H + h;
    const uint32_t r0 = BS == 64 ? 32 * (warp >> 1) : 0, n0 = (BS == 64 ? warp & 1 : warp) * (DS / Cfg::WC);
    const uint32_t chunks = head.y * PARTS;

    auto issue = [&](uint32_t c) {
        const uint2 ent = nn[head.x + c / PARTS];
        const uint32_t part = c % PARTS;
        float *buf = sm + (c & 1) * Cfg::buf;
        const size_t baseP = (bh * p.blocks + ent.x) * BS * BS, baseV = ((size_t)b * p.nb_b + ent.y) * BS * HD + (size_t)h * p.d + d0;
        if (TRANS) stage<A_DT, 32, BS>(buf, a_stride, Pm, baseP + part * 32 * BS, BS, BS, avec);
        else stage<A_DT, BS, 32>(buf, a_stride, Pm, baseP + part * 32, BS, 32, avec);
        stage<BC_DT, 32, DS>(buf + Cfg::a_floats, DS + 4, V, baseV + (size_t)part * 32 * HD, HD, p.d - d0, vec);
        cp_commit();
    };
    uint64_t acc[4][TN / 2];
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int n = 0; n < TN / 2; n++) acc[m][n] = 0;
    if (chunks) issue(0);
    for (uint32_t c = 0; c < chunks; c++) {
        cp_wait_all();
        __syncthreads();
        if (c + 1 < chunks) issue(c + 1);
        const float *buf = sm + (c & 1) * Cfg::buf;
        const float *v = buf + Cfg::a_floats + n0 + lane_col<TN>(lc);
        if (TRANS) mma_tn<TN>(acc, buf + r0 + 4 * lr, a_stride, v, DS + 4);
        else mma_nn<TN>(acc, buf + (r0 + lr) * a_stride, a_stride, v, DS + 4);
    }
    // rows without blocks are written as zeros (blocksparse.h:949-962)
    const size_t baseO = ((size_t)b * p.nb_a + i) * BS * HD + (size_t)h * p.d + d0 + n0;
    const uint32_t left = p.d > d0 + n0 ? p.d - d0 - n0 : 0;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const uint32_t r = r0 + (TRANS ? 4 * lr + m : lr + 8 * m);
        store_cols<BC_DT, TN>(O, baseO + (size_t)r * HD, lc, acc[m], 1.f, left, vec);
    }
}

// ------------------------------------------------------------------------------------------------
// Block-row-owned fusions.  Dynamic smem: Qs[DMAX][BS+1] | Ks[DMAX][BS+1] | (attention only)
// Vs[BS][DMAX] | Ps[BS][BS+16].
template <int BS>
__device__ __forceinline__ void score_tile(float (&s)[BS / 16][BS / 16], const float (*Qs)[BS + 1],
                                           const float (*Ks)[BS + 1], uint32_t d, int tx, int ty)
{
    constexpr int T = BS / 16;
#pragma unroll
    for (int m = 0; m < T; m++)
#pragma unroll
        for (int n = 0; n < T; n++) s[m][n] = 0.f;
#pragma unroll 4
    for (uint32_t k = 0; k < d; k++) {
        float a[T], bb[T];
#pragma unroll
        for (int m = 0; m < T; m++) a[m] = Qs[k][ty + 16 * m];
#pragma unroll
        for (int n = 0; n < T; n++) bb[n] = Ks[k][tx + 16 * n];
#pragma unroll
        for (int m = 0; m < T; m++)
#pragma unroll
            for (int n = 0; n < T; n++) s[m][n] = fmaf(a[m], bb[n], s[m][n]);
    }
}

__device__ __forceinline__ float half_warp_max(float v)
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float half_warp_sum(float v)
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// SDDMM + softmax, probabilities out.  Pass 1 stores the raw scores (in the output type) into Y and
// tracks the row max / sum; pass 2 lets every thread turn the scores it wrote itself into
// probabilities, so no thread ever reads another thread's global writes.
template <int BS, int DMAX, int AB_DT, int Y_DT>
__global__ void __launch_bounds__(256) fused_sddmm_softmax_kernel(const uint2 *__restrict__ lut, const void *__restrict__ A,
                                                                 const void *__restrict__ Bm,
                                                                 const typename MaskWord<BS>::type *__restrict__ mask,
                                                                 void *__restrict__ Y, AttnDims p, float scale_log2e)
{
    typedef typename MaskWord<BS>::type W;
    constexpr int T = BS / 16;
    extern __shared__ float smem[];
    float (*Qs)[BS + 1] = (float (*)[BS + 1])smem;
    float (*Ks)[BS + 1] = (float (*)[BS + 1])(smem + DMAX * (BS + 1));
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t i = blockIdx.x, b = blockIdx.y, h = blockIdx.z;
    const uint2 *nn = lut + (size_t)h * p.lut_stride;
    const uint2 head = nn[i];
    if (head.y == 0) return;
    const size_t HD = (size_t)p.H * p.d;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const W *mh = mask ? mask + (size_t)h * p.mask_stride : nullptr;

    for (uint32_t k0 = 0; k0 < p.d; k0 += 32)
        load_tile_kmajor<AB_DT, BS, 32>(Qs + k0, A, ((size_t)b * p.nb_a * BS + (size_t)i * BS) * HD + (size_t)h * p.d, HD, k0, p.d);

    float mx[T], sum[T];
#pragma unroll
    for (int m = 0; m < T; m++) { mx[m] = -INFINITY; sum[m] = 0.f; }

    for (uint32_t e = 0; e < head.y; e++) {
        const uint2 ent = nn[head.x + e];
        __syncthreads();
        for (uint32_t k0 = 0; k0 < p.d; k0 += 32)
            load_tile_kmajor<AB_DT, BS, 32>(Ks + k0, Bm, ((size_t)b * p.nb_b * BS + (size_t)ent.y * BS) * HD + (size_t)h * p.d, HD, k0, p.d);
        __syncthreads();
        float s[T][T];
        score_tile<BS>(s, Qs, Ks, p.d, tx, ty);
        const size_t baseY = (((size_t)b * p.H + h) * p.blocks + ent.x) * BS * BS;
#pragma unroll
        for (int m = 0; m < T; m++) {
            const uint32_t r = ty + 16 * m;
            const W w = mh ? __ldg(mh + (size_t)ent.x * BS + r) : ~(W)0;
            float bm = -INFINITY, t[T];
#pragma unroll
            for (int n = 0; n < T; n++) {
                const uint32_t c = tx + 16 * n;
                // the stored (possibly 16-bit) score is what pass 2 will read: use it for the statistics too
                Elem<Y_DT>::store(Y, baseY + (size_t)r * BS + c, s[m][n]);
                float sv = Elem<Y_DT>::round(s[m][n]);
                t[n] = ((w >> c) & 1) ? sv * scale_log2e : -INFINITY;
                bm = fmaxf(bm, t[n]);
            }
            bm = half_warp_max(bm);
            if (bm > mx[m]) {
                sum[m] *= exp2f(mx[m] - bm);
                mx[m] = bm;
            }
            float ps = 0.f;
            if (mx[m] > -INFINITY) {
#pragma unroll
                for (int n = 0; n < T; n++) ps += exp2f(t[n] - mx[m]);
            }
            sum[m] += half_warp_sum(ps);
        }
    }
    for (uint32_t e = 0; e < head.y; e++) {
        const uint2 ent = nn[head.x + e];
        const size_t baseY = (((size_t)b * p.H + h) * p.blocks + ent.x) * BS * BS;
#pragma unroll
        for (int m = 0; m < T; m++) {
            const uint32_t r = ty + 16 * m;
            const W w = mh ? __ldg(mh + (size_t)ent.x * BS + r) : ~(W)0;
            const float inv = sum[m] > 0.f ? 1.f / sum[m] : 0.f;
#pragma unroll
            for (int n = 0; n < T; n++) {
                const uint32_t c = tx + 16 * n;
                float sv = Elem<Y_DT>::load(Y, baseY + (size_t)r * BS + c);
                float pv = (((w >> c) & 1) && inv > 0.f) ? exp2f(sv * scale_log2e - mx[m]) * inv : 0.f;
                Elem<Y_DT>::store(Y, baseY + (size_t)r * BS + c, pv);
            }
        }
    }
}

// SDDMM + softmax + SpMM with an online softmax; S and P never leave the SM.  One CTA (four warps) per block-row.
// A step takes four 32x32 key blocks (a 32x32 score tile per warp) or one 64x64 block (a quarter per warp): Q . K^T over
// chunks of 32 of d, the softmax in registers (row maxima meet in shared memory), P to shared memory, then O += P . V in
// chunks of 32 keys, each warp on its share of O's columns (and, for 64 rows, of its rows).  Keys and values flow through
// the same two buffers as one sequence of chunks.  Score and O rows of a thread are the same, so O is rescaled in place.
// ST chunk buffers: two let three CTAs share an SM; four keep three chunks on their way, for launches that do not fill the SMs
// anyway and wait for L2 chunk by chunk.
template <int BS, int D, int ST = 2> struct FaCfg {
    static constexpr uint32_t G = BS == 32 ? 4 : 1;                      // key blocks per step
    static constexpr uint32_t NK = G * BS;                               // keys per step
    static constexpr uint32_t WC = BS == 32 ? 4 : 2;                     // warps side by side (score columns, O columns)
    static constexpr int TN = D / (int)WC / 4;
    static constexpr uint32_t kbuf = NK * tile::kStride, vbuf = 32 * (D + 4), buf = kbuf > vbuf ? kbuf : vbuf;
    static constexpr uint32_t p_stride = NK + 4, q_stride = D + 4;
    static constexpr uint32_t floats = BS * q_stride + ST * buf + BS * p_stride + WC * BS;
    static constexpr int ctas = ST > 2 || (BS == 64 && D == 128) ? 2 : 3;            // what registers and shared memory allow per SM
};
template <int BS, int D, int DT, int ST>
__global__ void __launch_bounds__(tile::kThreads, (FaCfg<BS, D, ST>::ctas))
fused_attention_kernel(const uint2 *__restrict__ lut, const void *__restrict__ Q, const void *__restrict__ K, const void *__restrict__ V,
                       void *__restrict__ O, const typename MaskWord<BS>::type *__restrict__ mask, AttnDims p, float scale_log2e, bool vec)
{
    using namespace tile;
    typedef typename MaskWord<BS>::type W;
    typedef FaCfg<BS, D, ST> Cfg;
    constexpr int TN = Cfg::TN;
    constexpr uint32_t G = Cfg::G, WC = Cfg::WC, QS = Cfg::q_stride, PS = Cfg::p_stride;
    extern __shared__ __align__(16) float sm[];
    float *Qs = sm, *bufs = Qs + BS * QS, *Ps = bufs + ST * Cfg::buf, *red = Ps + BS * PS;
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane_row(lane), lc = lane_quad(lane);
    // rows are dealt from both ends: the long rows of the layouts at hand sit there and start first
    const uint32_t i = (blockIdx.x & 1u) ? p.nb_a - 1u - (blockIdx.x >> 1) : blockIdx.x >> 1, b = blockIdx.y, h = blockIdx.z;
    const uint2 *nn = lut + (size_t)h * p.lut_stride;
    const uint2 head = nn[i];
    const size_t HD = p.in_pitch ? (size_t)p.in_pitch : (size_t)p.H * p.d;      // row pitch of q, k, v
    const size_t HDo = p.out_pitch ? (size_t)p.out_pitch : (size_t)p.H * p.d;   // row pitch of o
    const W *mh = mask ? mask + (size_t)h * p.mask_stride : nullptr;
    const uint32_t r0 = BS == 64 ? 32 * (warp >> 1) : 0, wc = BS == 64 ? warp & 1 : warp;   // this warp's rows and column share
    const uint32_t n0 = wc * (D / WC);
    const uint32_t kchunks = (p.d + kChunk - 1) / kChunk;
    const uint32_t cnt = head.y;

    // the sequence of chunks: per step the key chunks, then the value chunks
    uint32_t is_e = 0, is_k = 0, is_n = 0;                               // next chunk to issue: step's first entry, index in the step, overall
    size_t koff[G];
    auto issue = [&]() {
        if (is_e >= cnt) {                                               // nothing left: an empty group keeps the count
            cp_commit();
            return;
        }
        const uint32_t nblk = min(G, cnt - is_e);
        if (is_k == 0) {
#pragma unroll
            for (uint32_t g = 0; g < G; g++)
                koff[g] = ((size_t)b * p.nb_b + nn[head.x + is_e + (g < nblk ? g : 0)].y) * BS * HD + (size_t)h * p.d;
        }
        float *buf = bufs + (is_n % ST) * Cfg::buf;
        if (is_k < kchunks) {
            const uint32_t k0 = is_k * kChunk;
#pragma unroll
            for (uint32_t g = 0; g < G; g++)
                if (g < nblk) stage<DT, BS, (int)kChunk>(buf + g * BS * kStride, kStride, K, koff[g] + k0, HD, p.d - k0, vec);
        } else {
            const uint32_t vc = is_k - kchunks;
            const size_t base = G > 1 ? (vc == 0 ? koff[0] : vc == 1 ? koff[1 % G] : vc == 2 ? koff[2 % G] : koff[3 % G]) : koff[0] + (size_t)vc * 32 * HD;
            stage<DT, 32, D>(buf, D + 4, V, base, HD, p.d, vec);
        }
        cp_commit();
        is_n++;
        if (++is_k == kchunks + nblk * (BS / 32)) {
            is_k = 0;
            is_e += G;
        }
    };

    if (cnt) {
        stage<DT, BS, D>(Qs, QS, Q, ((size_t)b * p.nb_a + i) * BS * HD + (size_t)h * p.d, HD, p.d, vec);
#pragma unroll
        for (int i = 0; i < ST - 1; i++) issue();
    }
    float mx[4], sum[4];
    uint64_t acc[4][TN / 2];
#pragma unroll
    for (int m = 0; m < 4; m++) {
        mx[m] = -INFINITY;
        sum[m] = 0.f;
#pragma unroll
        for (int n = 0; n < TN / 2; n++) acc[m][n] = 0;
    }
    uint32_t c = 0;
    for (uint32_t e = 0; e < cnt; e += G) {
        const uint32_t nblk = min(G, cnt - e);
        const bool live = G == 1 || warp < nblk;
        uint64_t s2[4][8];
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int n = 0; n < 8; n++) s2[m][n] = 0;
        for (uint32_t kc = 0; kc < kchunks; kc++, c++) {
            cp_wait<ST - 2>();
            __syncthreads();
            issue();
            const float *buf = bufs + (c % ST) * Cfg::buf;
            if (live) mma_nt(s2, Qs + (r0 + lr) * QS + kc * kChunk, QS, buf + (32 * wc + lc) * kStride, kStride);
        }
        const uint32_t blk = nn[head.x + e + (G > 1 && live ? warp : 0)].x;
        float s[4][8], bm[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const W w = live ? (mh ? __ldg(mh + (size_t)blk * BS + r0 + lr + 8 * m) : ~(W)0) : (W)0;
            bm[m] = -INFINITY;
#pragma unroll
            for (int n = 0; n < 8; n++) {
                const uint32_t col = (BS == 64 ? 32 * wc : 0) + lc + 4 * n;
                s[m][n] = ((w >> col) & 1) ? half_sum(s2[m][n]) * scale_log2e : -INFINITY;
                bm[m] = fmaxf(bm[m], s[m][n]);
            }
            bm[m] = fmaxf(bm[m], __shfl_xor_sync(0xffffffffu, bm[m], 1));
            bm[m] = fmaxf(bm[m], __shfl_xor_sync(0xffffffffu, bm[m], 4));
            if (lc == 0) red[wc * BS + r0 + lr + 8 * m] = bm[m];
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const uint32_t r = r0 + lr + 8 * m;
            float mn = mx[m];
#pragma unroll
            for (uint32_t k = 0; k < WC; k++) mn = fmaxf(mn, red[k * BS + r]);
            const float alpha = mn > mx[m] ? exp2f(mx[m] - mn) : 1.f;
            mx[m] = mn;
            float ps = 0.f;
#pragma unroll
            for (int n = 0; n < 8; n++) {
                const float pv = mn > -INFINITY ? exp2f(s[m][n] - mn) : 0.f;
                Ps[r * PS + 32 * wc + lc + 4 * n] = pv;
                ps += pv;
            }
            sum[m] = fmaf(sum[m], alpha, ps);                            // this thread's columns only; the shares meet at the end
            const uint64_t a2 = pair(alpha, alpha);
#pragma unroll
            for (int n = 0; n < TN / 2; n++) acc[m][n] = fma2(acc[m][n], a2, 0ull);
        }
        const uint32_t vchunks = nblk * (BS / 32);
        for (uint32_t vc = 0; vc < vchunks; vc++, c++) {
            cp_wait<ST - 2>();
            __syncthreads();
            issue();
            const float *buf = bufs + (c % ST) * Cfg::buf;
            mma_nn<TN>(acc, Ps + (r0 + lr) * PS + vc * 32, PS, buf + n0 + lane_col<TN>(lc), D + 4);
        }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 4; m++) {
        sum[m] += __shfl_xor_sync(0xffffffffu, sum[m], 1);
        sum[m] += __shfl_xor_sync(0xffffffffu, sum[m], 4);
        if (lc == 0) red[wc * BS + r0 + lr + 8 * m] = sum[m];
    }
    __syncthreads();
    const size_t baseO = (((size_t)b * p.nb_a + i) * BS) * HDo + (size_t)h * p.d + n0;
    const uint32_t left = p.d > n0 ? p.d - n0 : 0;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const uint32_t r = r0 + lr + 8 * m;
        float l = 0.f;
#pragma unroll
        for (uint32_t k = 0; k < WC; k++) l += red[k * BS + r];
        store_cols<DT, TN>(O, baseO + (size_t)r * HDo, lc, acc[m], l > 0.f ? 1.f / l : 0.f, left, vec);
    }
}

// ------------------------------------------------------------------------------------------------
// Element-sparse attention of one tile of 32 query rows on fp32 operands (csr.cu makes the tile's list of columns and
// row masks): the kernel above on keys gathered by column, 128 of them per step, a 32x32 score tile per warp.
template <int ROWS, int COLS>
__device__ __forceinline__ void stage_gather(float *dst, uint32_t stride, const float *src, const CsrTileArgs &a, uint32_t base, uint32_t top,
                                             uint32_t distinct, uint32_t first, uint32_t n, size_t pitch)
{
    using namespace tile;
    constexpr int P = COLS / 4, STEP = (int)kThreads / P;
    const uint32_t r0 = threadIdx.x / P, c = (threadIdx.x % P) * 4;
#pragma unroll
    for (int i = 0; i < ROWS / STEP; i++) {
        const uint32_t r = r0 + i * STEP;
        const bool in = first + r < n;                                   // rows behind the list arrive as zeros
        const uint32_t col = in ? csr_entry(a.entries, base, top, distinct, first + r).x : 0u;
        cp_async16(dst + r * stride + c, src + (size_t)col * pitch + c, in ? 16u : 0u);
    }
}
template <int D>
__global__ void __launch_bounds__(tile::kThreads, 3) csr_tile_f32_kernel(const CsrTileArgs a)
{
    using namespace tile;
    typedef FaCfg<32, D> Cfg;
    constexpr int TN = Cfg::TN;
    constexpr uint32_t NK = Cfg::NK, QS = Cfg::q_stride, PS = Cfg::p_stride, kchunks = D / kChunk;
    extern __shared__ __align__(16) float sm[];
    float *Qs = sm, *bufs = Qs + 32 * QS, *Ps = bufs + 2 * Cfg::buf, *red = Ps + 32 * PS;
    grid_dependency_wait();
    grid_launch_dependents();
    csr_write_bad(a);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane_row(lane), lc = lane_quad(lane);
    const uint32_t tl = a.tiles - 1u - blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const uint32_t *cnt = a.counts + kCsrCounts * tl;
    const uint32_t distinct = cnt[0], base = cnt[2], top = cnt[3], n = distinct + cnt[1];
    const size_t HD = (size_t)a.H * D, head = (size_t)b * a.L * HD + (size_t)h * D;
    const float *K = (const float *)a.K + head, *V = (const float *)a.V + head;
    const uint32_t n0 = warp * (D / 4);

    uint32_t is_e = 0, is_k = 0, is_n = 0;                               // next chunk to issue: step's first key, index in the step, overall
    auto issue = [&]() {
        float *buf = bufs + (is_n & 1) * Cfg::buf;
        if (is_k < kchunks) stage_gather<(int)NK, (int)kChunk>(buf, kStride, K + is_k * kChunk, a, base, top, distinct, is_e, n, HD);
        else stage_gather<32, D>(buf, D + 4, V, a, base, top, distinct, is_e + (is_k - kchunks) * 32, n, HD);
        cp_commit();
        is_n++;
        if (++is_k == kchunks + (min(NK, n - is_e) + 31) / 32) {
            is_k = 0;
            is_e += NK;
        }
    };
    if (n) {
        const uint32_t rows = min(32u, a.L - tl * 32);                   // rows behind the sequence: the last one again, not written
        constexpr int P = D / 4, STEP = (int)kThreads / P;
#pragma unroll
        for (int i = 0; i < 32 / STEP; i++) {
            const uint32_t r = threadIdx.x / P + i * STEP, c = (threadIdx.x % P) * 4;
            cp_async16(Qs + r * QS + c, (const float *)a.Q + head + (size_t)(tl * 32 + min(r, rows - 1)) * HD + c, 16u);
        }
        issue();
    }
    float mx[4], sum[4];
    uint64_t acc[4][TN / 2];
#pragma unroll
    for (int m = 0; m < 4; m++) {
        mx[m] = -INFINITY;
        sum[m] = 0.f;
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[m][j] = 0;
    }
    uint32_t c = 0;
    for (uint32_t e = 0; e < n; e += NK) {
        const uint32_t left = min(NK, n - e);
        const bool live = 32 * warp < left;
        uint64_t s2[4][8];
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int j = 0; j < 8; j++) s2[m][j] = 0;
        uint32_t mk[8];                                                  // the rows of this thread's eight columns
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t col = 32 * warp + lc + 4 * j;
            mk[j] = col < left ? csr_entry(a.entries, base, top, distinct, e + col).y : 0u;
        }
        for (uint32_t kc = 0; kc < kchunks; kc++, c++) {
            cp_wait_all();
            __syncthreads();
            issue();                                                     // a value chunk follows every key chunk of a step
            if (live) mma_nt(s2, Qs + lr * QS + kc * kChunk, QS, bufs + (c & 1) * Cfg::buf + (32 * warp + lc) * kStride, kStride);
        }
        float s[4][8], bm[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            bm[m] = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                s[m][j] = (mk[j] >> (lr + 8 * m)) & 1u ? half_sum(s2[m][j]) * a.scale_log2e : -INFINITY;
                bm[m] = fmaxf(bm[m], s[m][j]);
            }
            bm[m] = fmaxf(bm[m], __shfl_xor_sync(0xffffffffu, bm[m], 1));
            bm[m] = fmaxf(bm[m], __shfl_xor_sync(0xffffffffu, bm[m], 4));
            if (lc == 0) red[warp * 32 + lr + 8 * m] = bm[m];
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const uint32_t r = lr + 8 * m;
            float mn = mx[m];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) mn = fmaxf(mn, red[k * 32 + r]);
            const float alpha = mn > mx[m] ? exp2f(mx[m] - mn) : 1.f;
            mx[m] = mn;
            const float off = mn > -INFINITY ? mn : 0.f;                 // nothing kept so far: exp2(-inf) = 0, and NaN stays NaN
            float ps = 0.f;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float pv = exp2f(s[m][j] - off);
                Ps[r * PS + 32 * warp + lc + 4 * j] = pv;
                ps += pv;
            }
            sum[m] = fmaf(sum[m], alpha, ps);                            // this thread's columns only; the shares meet at the end
            const uint64_t a2 = pair(alpha, alpha);
#pragma unroll
            for (int j = 0; j < TN / 2; j++) acc[m][j] = fma2(acc[m][j], a2, 0ull);
        }
        const uint32_t vchunks = (left + 31) / 32;
        for (uint32_t vc = 0; vc < vchunks; vc++, c++) {
            cp_wait_all();
            __syncthreads();
            if (vc + 1 < vchunks || e + NK < n) issue();
            mma_nn<TN>(acc, Ps + lr * PS + vc * 32, PS, bufs + (c & 1) * Cfg::buf + n0 + lane_col<TN>(lc), D + 4);
        }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 4; m++) {
        sum[m] += __shfl_xor_sync(0xffffffffu, sum[m], 1);
        sum[m] += __shfl_xor_sync(0xffffffffu, sum[m], 4);
        if (lc == 0) red[warp * 32 + lr + 8 * m] = sum[m];
    }
    __syncthreads();
    uint32_t odd = 0;                                                    // this thread's rows with an output that is not finite
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const uint32_t r = lr + 8 * m;
        float l = 0.f;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) l += red[k * 32 + r];
        const float inv = l > 0.f ? 1.f / (l + 1e-6f) : 0.f;             // the reference's denominator (ewops.h:93, cuda_kernels.h:1022)
        if (tl * 32 + r < a.L) store_cols<SFB_F32, TN>(a.O, head + (size_t)(tl * 32 + r) * HD + n0, lc, acc[m], inv, D / 4, true);
        float zero = 0.f;                                                // stays 0 as long as every output is finite
#pragma unroll
        for (int j = 0; j < TN / 2; j++) {
            const float2 f = unpair(acc[m][j]);
            zero = fmaf(f.x, 0.f, fmaf(f.y, 0.f, zero));
        }
        if (!(zero == 0.f) && tl * 32 + r < a.L) odd |= 1u << r;
    }
    if (!__syncthreads_or(odd != 0)) return;
    // rows that are not finite are made again (csr_row_again), once every warp has written its columns of them
    uint32_t *again = (uint32_t *)red;
    if (threadIdx.x == 0) *again = 0;
    __syncthreads();
    if (odd) atomicOr(again, odd);
    __syncthreads();
    const uint32_t rows = *again;
    for (uint32_t r = warp; r < 32; r += 4)
        if ((rows >> r) & 1u) csr_row_again<SFB_F32, D>(a.rowptr, a.colidx, a.nnz, a.Q, a.K, a.V, a.O, a.L, a.H, b, h, tl * 32 + r, a.scale_log2e);
}

// ------------------------------------------------------------------------------------------------
// host-side dispatch
#define DISPATCH_BS(bs, ...)            \
    if (bs == 32) { constexpr int BS = 32; __VA_ARGS__ } else { constexpr int BS = 64; __VA_ARGS__ }
#define DISPATCH_DT(dt, NAME, ...)                                         \
    if (dt == SFB_F32) { constexpr int NAME = SFB_F32; __VA_ARGS__ }        \
    else if (dt == SFB_BF16) { constexpr int NAME = SFB_BF16; __VA_ARGS__ } \
    else { constexpr int NAME = SFB_F16; __VA_ARGS__ }

// the kernel's dynamic shared memory, asked for once per device and kernel
template <typename K>
static int set_smem(DeviceOnce &once, K kernel, size_t bytes)
{
    const int dev = current_device();
    if (bytes > 48 * 1024 && !once.done(dev)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return fail("cudaFuncSetAttribute(%zu bytes): %s", bytes, cudaGetErrorString(e));
        once.mark(dev);
    }
    return 0;
}

// 16-byte accesses to rows of a [.., pitch] tensor whose heads are d wide
static bool rows_vec(const void *ptr, int dtype, uint64_t pitch, uint32_t d)
{
    const uint32_t per = dtype == SFB_F32 ? 4 : 8;
    return ((uintptr_t)ptr & 15) == 0 && pitch % per == 0 && d % per == 0;
}

int simt_sddmm_nt(cudaStream_t s, const void *lut, const void *a, const void *b, void *c, int ab_dtype, int c_dtype,
                  uint32_t bs, const AttnDims &p)
{
    const uint64_t HD = (uint64_t)p.H * p.d;
    const bool vec = rows_vec(a, ab_dtype, HD, p.d) && rows_vec(b, ab_dtype, HD, p.d) && ((uintptr_t)c & 15) == 0;
#define SD_LAUNCH(CD)                                                                                             \
    {                                                                                                             \
        constexpr uint32_t per = BS == 32 ? 4 : 1;                                                                \
        const size_t bytes = sizeof(float) * 4 * per * BS * tile::kStride;                                        \
        auto kern = sddmm_nt_kernel<BS, AB, CD>;                                                                  \
        static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                                                      \
        launch_overlapped(kern, dim3((p.blocks + per - 1) / per, p.B, p.H), dim3(tile::kThreads), bytes, s, (const uint2 *)lut, a, b, c, p, vec); \
    }
    DISPATCH_BS(bs, DISPATCH_DT(ab_dtype, AB, {
        if (c_dtype == SFB_F32) SD_LAUNCH(SFB_F32) else if (c_dtype == SFB_BF16) SD_LAUNCH(SFB_BF16) else SD_LAUNCH(SFB_F16)
    }))
#undef SD_LAUNCH
    return check_launch("sfb_bst_sgemm_nt");
}

int simt_softmax(cudaStream_t s, const void *lut, const void *mask, const void *x, void *y, int x_dtype, int y_dtype,
                 uint32_t bs, const AttnDims &p, float scale, uint32_t max_lut)
{
    const float sl = scale * LOG2E_F;
    // The caller's max_lut (0 = unknown) picks the variant.  16-bit scores: rows of up to 20 blocks stay in registers,
    // one pass over HBM; from 9 blocks up a CTA takes a quarter of the block-row's query rows.  Longer or unknown rows
    // are streamed: three sweeps, the second and third over lines the CTA has just pulled through L2.  Measured and not
    // kept for rows of 17-32 blocks: two groups of lanes per query row, each holding every other block (0.68 of copy
    // bandwidth on 17-block rows against 0.77 with 20 slots per lane).
    const int inplace = max_lut != 0 && max_lut <= 12;   // streamed short rows: unnormalised values wait in L2 for the rescale
    int nb = 0;   // block slots of the register tile, 0 = stream
    if (x_dtype == SFB_BF16)
        nb = max_lut == 0 ? 0 : max_lut <= 4 ? 4 : max_lut <= 8 ? 8 : max_lut <= 12 ? 12 : max_lut <= 16 ? 16 : max_lut <= 18 ? 18 : max_lut <= 20 ? 20 : 0;
    else
        nb = (max_lut >= 3 && max_lut <= 4) ? 4 : (max_lut >= 7 && max_lut <= 8) ? 8 : (max_lut >= 14 && max_lut <= 16) ? 16 : 0;
#define SM_LAUNCH(XD, NBV, SPL)                                                                                        \
    DISPATCH_DT(y_dtype, YD, {                                                                                         \
        launch_overlapped_few(softmax_kernel<BS, XD, YD, NBV, SPL>, dim3(p.nb_a * SPL, p.B, p.H), dim3(BS * BS / 8 / SPL), 0, s, \
            (const uint2 *)lut, (const W *)mask, x, y, p, sl, inplace);                                                \
    })
    DISPATCH_BS(bs, {
        typedef typename MaskWord<BS>::type W;
        if (x_dtype == SFB_BF16) {
            if (nb == 4) { SM_LAUNCH(SFB_BF16, 4, 1) }
            else if (nb == 8) { SM_LAUNCH(SFB_BF16, 8, 1) }
            else if (nb == 12) { SM_LAUNCH(SFB_BF16, 12, 4) }
            else if (nb == 16) { SM_LAUNCH(SFB_BF16, 16, 4) }
            else if (nb == 18) { SM_LAUNCH(SFB_BF16, 18, 4) }
            else if (nb == 20) { SM_LAUNCH(SFB_BF16, 20, 4) }
            else { SM_LAUNCH(SFB_BF16, 0, 1) }
        } else {
            if (nb == 4) { SM_LAUNCH(SFB_F32, 4, 1) }
            else if (nb == 8) { SM_LAUNCH(SFB_F32, 8, 1) }
            else if (nb == 16) { SM_LAUNCH(SFB_F32, 16, 1) }
            else { SM_LAUNCH(SFB_F32, 0, 1) }
        }
    })
#undef SM_LAUNCH
    return check_launch("sfb_masked_softmax");
}

int simt_spmm_nn(cudaStream_t s, const void *lut, const void *a, const void *b, void *c, int a_dtype, int bc_dtype,
                 uint32_t bs, const AttnDims &p, bool trans)
{
    const uint64_t HD = (uint64_t)p.H * p.d;
    const bool avec = ((uintptr_t)a & 15) == 0, vec = rows_vec(b, bc_dtype, HD, p.d) && rows_vec(c, bc_dtype, HD, p.d);
#define SP_LAUNCH(DSV)                                                                                            \
    {                                                                                                             \
        const size_t bytes = sizeof(float) * 2 * SpmmCfg<BS, DSV>::buf;                                           \
        const dim3 grid(p.nb_a * ((p.d + DSV - 1) / DSV), p.B, p.H);                                              \
        if (trans) {                                                                                              \
            auto kern = spmm_nn_kernel<BS, DSV, AD, BD, true>;                                                    \
            static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                                                  \
            launch_overlapped(kern, grid, dim3(tile::kThreads), bytes, s, (const uint2 *)lut, a, b, c, p, avec, vec);                  \
        } else {                                                                                                  \
            auto kern = spmm_nn_kernel<BS, DSV, AD, BD, false>;                                                   \
            static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                                                  \
            launch_overlapped(kern, grid, dim3(tile::kThreads), bytes, s, (const uint2 *)lut, a, b, c, p, avec, vec);                  \
        }                                                                                                         \
    }
    DISPATCH_BS(bs, DISPATCH_DT(a_dtype, AD, DISPATCH_DT(bc_dtype, BD, {
        if (p.d <= 32) SP_LAUNCH(32) else if (p.d <= 64) SP_LAUNCH(64) else SP_LAUNCH(128)
    })))
#undef SP_LAUNCH
    return check_launch("sfb_bst_sgemm_xn");
}

int simt_softmax_grad(cudaStream_t s, const void *lut, const void *dy, const void *y, void *dx, int dtype, uint32_t bs,
                      const AttnDims &p, float scale, uint32_t max_lut)
{
    // rows of up to 8 blocks (24 for 16-bit types; the caller's max_lut says so) stay in registers: one pass over
    // HBM; 0 = unknown, stream.  The streamed variant re-reads dy and y, and at full size those re-reads miss L2.
    const bool wide = dtype != SFB_F32;
    const int nb = (max_lut >= 1 && max_lut <= 4) ? 4 : (max_lut >= 5 && max_lut <= 8) ? 8
                   : (max_lut >= 9 && max_lut <= 12 && wide) ? 12 : (max_lut >= 13 && max_lut <= 16 && wide) ? 16
                   : (max_lut >= 17 && max_lut <= 24 && wide) ? 24 : 0;
#define SG_LAUNCH(NBV, SPL)                                                                                            \
    DISPATCH_DT(dtype, DT, {                                                                                           \
        launch_overlapped_few(softmax_grad_kernel<BS, DT, NBV, SPL>, dim3(p.nb_a * SPL, p.B, p.H), dim3(BS * BS / 8 / SPL), 0, s, (const uint2 *)lut, dy, y, dx, p, scale); \
    })
    DISPATCH_BS(bs, {
        if (nb == 4) { SG_LAUNCH(4, 1) } else if (nb == 8) { SG_LAUNCH(8, 1) } else if (nb == 12) { SG_LAUNCH(12, 1) }
        else if (nb == 16) { SG_LAUNCH(16, 1) } else if (nb == 24) { SG_LAUNCH(24, 2) } else { SG_LAUNCH(0, 1) }
    })
#undef SG_LAUNCH
    return check_launch("sfb_masked_softmax_grad");
}

int simt_fused_sddmm_softmax(cudaStream_t s, const void *nn_lut, const void *a, const void *b, const void *mask, void *y,
                             int ab_dtype, int y_dtype, uint32_t bs, const AttnDims &p, float scale)
{
    SFB_REQUIRE(p.d <= 128, "sfb_fused_sddmm_softmax: state_dim %u > 128 not supported", p.d);
    dim3 grid(p.nb_a, p.B, p.H);
    const float sl = scale * LOG2E_F;
#define LAUNCH_FSS(DMAX)                                                                                         \
    {                                                                                                            \
        typedef typename MaskWord<BS>::type W;                                                                   \
        size_t bytes = sizeof(float) * 2 * DMAX * (BS + 1);                                                      \
        auto kern = fused_sddmm_softmax_kernel<BS, DMAX, AB, YD>;                                                \
        static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                                                     \
        launch_overlapped(kern, grid, dim3(256), bytes, s, (const uint2 *)nn_lut, a, b, (const W *)mask, y, p, sl);                   \
    }
    DISPATCH_BS(bs, DISPATCH_DT(ab_dtype, AB, DISPATCH_DT(y_dtype, YD, {
        if (p.d <= 64) LAUNCH_FSS(64) else LAUNCH_FSS(128)
    })))
#undef LAUNCH_FSS
    return check_launch("sfb_fused_sddmm_softmax");
}

int simt_fused_attention(cudaStream_t s, const void *nn_lut, const void *q, const void *k, const void *v, void *o,
                         const void *mask, int dtype, uint32_t bs, const AttnDims &p, float scale)
{
    SFB_REQUIRE(p.d <= 128, "sfb_fused_attention: state_dim %u > 128 not supported", p.d);
    dim3 grid(p.nb_a, p.B, p.H);
    const float sl = scale * LOG2E_F;
    const uint64_t HD = (uint64_t)p.H * p.d, in = p.in_pitch ? p.in_pitch : HD, on = p.out_pitch ? p.out_pitch : HD;
    const bool vec = rows_vec(q, dtype, in, p.d) && rows_vec(k, dtype, in, p.d) && rows_vec(v, dtype, in, p.d) && rows_vec(o, dtype, on, p.d);
    // a launch that two CTAs per SM hold at once waits for its chunks one after another: more of them on their way
    // (B 1, H 4, L 512, d 64: 64 CTAs)
    const int sms = device_sm_count(current_device());
    const bool few = (uint64_t)p.nb_a * p.B * p.H <= 2ull * (uint64_t)(sms > 0 ? sms : 0);
#define LAUNCH_FA_ST(DV, STV)                                                                                    \
    {                                                                                                            \
        typedef typename MaskWord<BS>::type W;                                                                   \
        const size_t bytes = sizeof(float) * FaCfg<BS, DV, STV>::floats;                                         \
        auto kern = fused_attention_kernel<BS, DV, DT, STV>;                                                     \
        static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                       \
        launch_overlapped(kern, grid, dim3(tile::kThreads), bytes, s, (const uint2 *)nn_lut, q, k, v, o, (const W *)mask, p, sl, vec); \
    }
#define LAUNCH_FA(DV) { if (few) LAUNCH_FA_ST(DV, 4) else LAUNCH_FA_ST(DV, 2) }
    DISPATCH_BS(bs, DISPATCH_DT(dtype, DT, {
        if (p.d <= 32) LAUNCH_FA(32) else if (p.d <= 64) LAUNCH_FA(64) else LAUNCH_FA(128)
    }))
#undef LAUNCH_FA_ST
#undef LAUNCH_FA
    return check_launch("sfb_fused_attention");
}

int csr_tile_f32(cudaStream_t s, const CsrTileArgs &a, uint32_t B, uint32_t d)
{
#define LAUNCH_CT(DV)                                                                                            \
    {                                                                                                            \
        const size_t bytes = sizeof(float) * FaCfg<32, DV>::floats;                                              \
        auto kern = csr_tile_f32_kernel<DV>;                                                                     \
        static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                       \
        launch_overlapped(kern, dim3(a.tiles, a.H, B), dim3(tile::kThreads), bytes, s, a);                       \
    }
    if (d == 32) LAUNCH_CT(32) else if (d == 64) LAUNCH_CT(64) else LAUNCH_CT(128)
#undef LAUNCH_CT
    return check_launch("sfb_csr_attention");
}

}  // namespace sfb
