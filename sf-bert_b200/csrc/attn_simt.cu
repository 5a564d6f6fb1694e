// Kernels of the block-sparse attention path that serve fp32 operands (1e-5 parity with the CPU reference, more than one
// 16-bit or tf32 product gives) and every shape the tcgen05 kernels do not cover: SDDMM, masked softmax, SpMM and the two
// block-row-owned fusions.
//
// SDDMM, SpMM, the fused attention and the fp32 element-sparse tiles take their products from warp-level tensor-core
// instructions on operands split into bf16 terms (simt_tile.cuh), the SpMM of fp32 blocks from FMAs (fma_tile.cuh).  The fused SDDMM + softmax (fused_sddmm_softmax_kernel) is on the
// FMA pipe: 256 threads as a 16x16 grid; thread (ty,tx) owns rows ty+16m and columns tx+16n of a tile, so the 16
// lanes of a half-warp own one set of rows and row reductions are four shuffles.
#include "fma_tile.cuh"
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
// The scores of a warp's 32x32 tile that are not finite, made again by plain FMAs (simt_tile.cuh says why), in place.  By a warp at a
// time and not inlined: the tile's registers are free by then.
template <int BS, int AB_DT, int C_DT>
__device__ __noinline__ void sddmm_again(float *buf, const void *A, const void *B, void *C, size_t rowA, size_t rowB, size_t at, size_t HD, uint32_t d)
{
    const uint32_t lane = threadIdx.x & 31;
    float s[32];
    tile::scores_again<AB_DT>(s, buf, A, B, rowA, rowB, HD, d, lane);
    // back to where a row's scores lie side by side: a lane per key
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 32; n++) buf[lane * 33 + n] = s[n];
    __syncwarp();
#pragma unroll 8
    for (uint32_t r = 0; r < 32; r++)
        if (!tile::finite(Elem<C_DT>::load(C, at + r * BS + lane))) Elem<C_DT>::store(C, at + r * BS + lane, buf[r * 33 + lane]);
}

// SDDMM.  A CTA (four warps) makes one 64x64 block, a 32x32 quarter per warp, or four consecutive 32x32 blocks of the LUT,
// one per warp.  The keys come chunk by chunk (32 of d) through a ring of the warps that use them; the query rows go straight to
// fragments, a chunk ahead in registers: consecutive blocks mostly share their block-row (the LUT is in row-major scan
// order), so three of the four warps find them in L1.  No warp waits for another one that does not share its keys.  A thread
// holds eight neighbouring scores of a row, so that they leave in whole pieces of 16 or 32 bytes.
template <int BS> struct SddmmCfg {
    static constexpr int TEAMS = BS == 32 ? 4 : 2, TT = 128 / TEAMS;      // teams that stage keys of their own
    static constexpr uint32_t buf = 32 * tile::kStride;
    static_assert(TEAMS * 2 * buf / 4 >= tile::kAgainFloats && tile::kAgainFloats >= 32 * 33, "a warp's share holds the tiles of sddmm_again");
};
template <int BS, int AB_DT, int C_DT>
__global__ void __launch_bounds__(tile::kThreads, 3) sddmm_nt_kernel(const uint2 *__restrict__ lut, const void *__restrict__ A,
                                                                   const void *__restrict__ Bm, void *__restrict__ C, AttnDims p, bool vec)
{
    using namespace tile;
    typedef SddmmCfg<BS> Cfg;
    constexpr uint32_t PER = BS == 32 ? 4 : 1;               // blocks per CTA
    constexpr int T = kTerms<AB_DT>, TT = Cfg::TT;
    extern __shared__ __align__(16) float sm[];              // [team][2][32 keys]
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t b = blockIdx.y, h = blockIdx.z;
    const uint32_t bid = blockIdx.x * PER + (BS == 32 ? warp : 0);
    if (bid >= p.blocks) return;
    const uint32_t r0 = BS == 64 ? 32 * (warp >> 1) : 0, team = BS == 64 ? warp & 1 : warp, c0 = BS == 64 ? 32 * team : 0;
    const uint32_t rank = BS == 64 ? 32 * (warp >> 1) + lane : lane;
    const size_t HD = (size_t)p.H * p.d;
    const uint2 en = lut[(size_t)h * p.lut_stride + bid];
    const size_t rowA = (((size_t)b * p.nb_a + en.x) * BS + r0) * HD + (size_t)h * p.d, rowB = (((size_t)b * p.nb_b + en.y) * BS + c0) * HD + (size_t)h * p.d;
    float *bufs = sm + team * 2 * Cfg::buf;
    Staged<AB_DT, TT, (int)kChunk> held_b;
    Raw4<AB_DT> held_a[8];                                   // [16-element half of the chunk][row 16 m + 8 half + g]
    const uint32_t chunks = (p.d + kChunk - 1) / kChunk;
    auto load_a = [&](uint32_t c) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t k = c * kChunk + 16 * (i >> 2) + 4 * t;
            load_raw4<AB_DT>(held_a[i], A, rowA + (size_t)(8 * (i & 3) + g) * HD + k, k < p.d ? p.d - k : 0u, vec);
        }
    };
    auto issue = [&](uint32_t c) {
        stage_begin(held_b, rank, bufs + (c & 1) * Cfg::buf, kStride, Bm, rowB + c * kChunk, HD, p.d - c * kChunk, vec);
        cp_commit();
    };
    float acc[2][4][4] = {};
    issue(0);
    load_a(0);
    stage_end(held_b, rank, bufs, kStride, vec);
    for (uint32_t c = 0; c < chunks; c++) {
        cp_wait<0>();
        meet<TT>(1 + team);
        if (c + 1 < chunks) issue(c + 1);
        Frag<T> fa[2][2];
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int m = 0; m < 2; m++) {
                float x0[4], x1[4];
                widen4<AB_DT>(x0, held_a[4 * k + 2 * m]);
                widen4<AB_DT>(x1, held_a[4 * k + 2 * m + 1]);
                split_rows<T>(fa[k][m], x0, x1);
            }
        if (c + 1 < chunks) load_a(c + 1);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            Four<T> fb[4];
            load_keys<T, true>(fb, bufs + (c & 1) * Cfg::buf, 16 * k, g, t);
#pragma unroll
            for (int m = 0; m < 2; m++) mma16<4, T, T>(acc[m], fa[k][m], fb);
        }
        if (c + 1 < chunks) stage_end(held_b, rank, bufs + ((c + 1) & 1) * Cfg::buf, kStride, vec);
    }
    const bool odd = T > 1 && !(zero_if_finite<4>(acc[1], zero_if_finite<4>(acc[0], 0.f)) == 0.f);
    const size_t baseC = (((size_t)b * p.H + h) * p.blocks + bid) * BS * BS + (size_t)r0 * BS + c0;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = acc[m][k >> 1][2 * half + (k & 1)];
            const size_t at = baseC + (size_t)(16 * m + 8 * half + g) * BS + 8 * t;
            if (vec) {
                if (C_DT == SFB_F32) {
                    *(float4 *)((float *)C + at) = make_float4(v[0], v[1], v[2], v[3]);
                    *(float4 *)((float *)C + at + 4) = make_float4(v[4], v[5], v[6], v[7]);
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
    // on the team's shared memory, when its other warp is past the products too
    if (T > 1 && (BS == 64 ? __syncthreads_or(odd) : __any_sync(0xffffffffu, odd)) && __any_sync(0xffffffffu, odd))
        sddmm_again<BS, AB_DT, C_DT>(sm + warp * (Cfg::TEAMS * 2 * Cfg::buf / 4), A, Bm, C, rowA, rowB, baseC, HD, p.d);
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
//
// By FMAs (fma_tile.cuh).  AGAIN: what the kernel below left that is not finite, made again by the same CTA (simt_tile.cuh says why).
template <int BS, int DS> struct SpmmFmaCfg {
    static constexpr int WC = BS == 32 ? 4 : 2;                          // warps side by side along d
    static constexpr int TN = DS / WC / 4;                               // columns per thread
    static constexpr uint32_t a_floats = BS == 32 ? 32 * tile::kStride : 64 * tile::kStride > 32 * (64 + 4) ? 64 * tile::kStride : 32 * (64 + 4);
    static constexpr uint32_t buf = a_floats + 32 * (DS + 4);
    static constexpr size_t bytes = sizeof(float) * 2 * buf;             // [2][P chunk | V chunk]
};
template <int BS, int DS, int A_DT, int BC_DT, bool TRANS, bool AGAIN>
__device__ __forceinline__ void spmm_fma(float *sm, const uint2 *__restrict__ lut, const void *__restrict__ Pm, const void *__restrict__ V, void *__restrict__ O,
                                         const AttnDims &p, bool avec, bool vec)
{
    using namespace fma_tile;
    typedef SpmmFmaCfg<BS, DS> Cfg;
    constexpr int TN = Cfg::TN;
    constexpr uint32_t PARTS = BS / 32;                                  // chunks per block
    constexpr uint32_t a_stride = TRANS ? BS + 4 : kStride;
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
        tile::cp_commit();
    };
    uint64_t acc[4][TN / 2];
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int n = 0; n < TN / 2; n++) acc[m][n] = 0;
    if (chunks) issue(0);
    for (uint32_t c = 0; c < chunks; c++) {
        tile::cp_wait<0>();
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
        store_row<BC_DT, TN, AGAIN>(O, baseO + (size_t)r * HD, lc, acc[m], left, vec);
    }
}
template <int BS, int DS, int A_DT, int BC_DT, bool TRANS>
__global__ void __launch_bounds__(tile::kThreads, 4) spmm_fma_kernel(const uint2 *__restrict__ lut, const void *__restrict__ Pm, const void *__restrict__ V,
                                                                   void *__restrict__ O, AttnDims p, bool avec, bool vec)
{
    extern __shared__ __align__(16) float sm[];
    grid_dependency_wait();
    grid_launch_dependents();
    spmm_fma<BS, DS, A_DT, BC_DT, TRANS, false>(sm, lut, Pm, V, O, p, avec, vec);
}
// Not inlined, and from the kernel's parameters alone: nothing is kept for it in registers while the split products are made
template <int BS, int DS, int A_DT, int BC_DT, bool TRANS>
__device__ __noinline__ void spmm_again(float *sm, const uint2 *lut, const void *Pm, const void *V, void *O, uint32_t H, uint32_t d, uint32_t nb_a, uint32_t nb_b,
                                        uint32_t blocks, uint32_t lut_stride, bool avec, bool vec)
{
    const AttnDims p = {0, H, d, nb_a, nb_b, blocks, lut_stride, 0, 0, 0};
    spmm_fma<BS, DS, A_DT, BC_DT, TRANS, true>(sm, lut, Pm, V, O, p, avec, vec);
}

// As split products (16-bit blocks).  A warp owns 32 output rows and a share of the columns; it stages its own columns of V (with
// the other warp that has them, where blocks are 64 rows) and reads P straight into fragments, a chunk ahead in registers: P is
// small beside V, and L1 has it for the other warps.
template <int BS, int DS> struct SpmmCfg {
    static constexpr int WC = BS == 32 ? 4 : 2;                          // warps side by side along d: each is a team with the ones below it
    static constexpr int TT = 128 / WC, NW = DS / WC, N = NW / 8;        // a team's threads and columns, n-tiles of 8 columns
    static constexpr uint32_t v_stride = NW + 8, buf = 32 * v_stride;
    static constexpr size_t own = sizeof(float) * 3 * WC * buf, bytes = own > SpmmFmaCfg<BS, DS>::bytes ? own : SpmmFmaCfg<BS, DS>::bytes;      // [team][3][32 rows of V], or spmm_again's
};
template <int BS, int DS, int A_DT, int BC_DT, bool TRANS>
__global__ void __launch_bounds__(tile::kThreads, BS == 64 && DS == 128 ? 3 : 4)
spmm_nn_kernel(const uint2 *__restrict__ lut, const void *__restrict__ Pm, const void *__restrict__ V, void *__restrict__ O, AttnDims p, bool avec, bool vec)
{
    using namespace tile;
    typedef SpmmCfg<BS, DS> Cfg;
    constexpr int N = Cfg::N, TT = Cfg::TT, VN = Cols<N>::VN;
    constexpr int TP = kTerms<A_DT>, TV = kTerms<BC_DT>;
    constexpr uint32_t PARTS = BS / 32;                                  // chunks per block
    extern __shared__ __align__(16) float sm[];                          // [team][3][32 rows of V]
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t nslice = (p.d + DS - 1) / DS;
    const uint32_t i = blockIdx.x / nslice, d0 = (blockIdx.x % nslice) * DS;
    const uint32_t b = blockIdx.y, h = blockIdx.z;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint2 *nn = lut + (size_t)h * p.lut_stride;
    const uint2 head = nn[i];
    const size_t HD = (size_t)p.H * p.d;
    const size_t bh = (size_t)b * p.H + h;
    const uint32_t r0 = BS == 64 ? 32 * (warp >> 1) : 0, team = BS == 64 ? warp & 1 : warp, n0 = d0 + team * Cfg::NW;
    const uint32_t rank = BS == 64 ? 32 * (warp >> 1) + lane : lane;
    const uint32_t chunks = head.y * PARTS, left = p.d > n0 ? p.d - n0 : 0;
    float *bufs = sm + team * 3 * Cfg::buf;

    // the row's entries, 32 at a time, one per lane, the next 32 ahead
    uint2 ent = lane < head.y ? nn[head.x + lane] : make_uint2(0u, 0u), ent2 = 32 + lane < head.y ? nn[head.x + 32 + lane] : make_uint2(0u, 0u);
    auto entry = [&](uint32_t c, uint32_t &part) {                       // called for c = 0, 1, 2, ... in turn
        const uint32_t e = c / PARTS;
        part = c % PARTS;
        if (e && e % 32 == 0 && part == 0) {
            ent = ent2;
            ent2 = e + 32 + lane < head.y ? nn[head.x + e + 32 + lane] : make_uint2(0u, 0u);
        }
        return make_uint2(__shfl_sync(0xffffffffu, ent.x, e % 32), __shfl_sync(0xffffffffu, ent.y, e % 32));
    };
    Staged<BC_DT, TT, Cfg::NW> held_v;
    Raw4<A_DT> held_p[8];                                                // [k16][row 16 m + 8 half + g], TRANS: [k16][element 4 t + i], rows 4 g to 4 g + 3
    size_t next_p = 0;                                                   // chunk c + 1's place in P
    auto issue = [&](uint32_t c) {                                       // V of chunk c; its P is asked for one chunk later
        if (c < chunks) {
            uint32_t part;
            const uint2 en = entry(c, part);
            next_p = (bh * p.blocks + en.x) * BS * BS + (TRANS ? (size_t)part * 32 * BS + r0 : (size_t)r0 * BS + part * 32);
            if (left) stage_begin(held_v, rank, bufs + (c % 3) * Cfg::buf, Cfg::v_stride, V, ((size_t)b * p.nb_b + en.y) * BS * HD + (size_t)part * 32 * HD + (size_t)h * p.d + n0, HD, left, vec);
        }
        cp_commit();
    };
    auto land = [&](uint32_t c) {                                        // the pieces of chunk c that are converted on the way
        if (c < chunks && left) stage_end(held_v, rank, bufs + (c % 3) * Cfg::buf, Cfg::v_stride, vec);
    };
    auto load_p = [&](size_t at) {
#pragma unroll
        for (int x = 0; x < 8; x++)
            load_raw4<A_DT>(held_p[x], Pm, at + (TRANS ? (size_t)(16 * (x >> 2) + 4 * t + (x & 3)) * BS + 4 * g : (size_t)(8 * (x & 3) + g) * BS + 16 * (x >> 2) + 4 * t), 4, avec);
    };
    float acc[2][N][4] = {};
    if (chunks) {
        issue(0);
        land(0);
        load_p(next_p);
        issue(1);
        land(1);
    }
    for (uint32_t c = 0; c < chunks; c++) {
        cp_wait<1>();
        meet<TT>(1 + team);
        Frag<TP> fp[2][2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            float x[4][4];
#pragma unroll
            for (int r = 0; r < 4; r++) widen4<A_DT>(x[r], held_p[4 * k + r]);
#pragma unroll
            for (int m = 0; m < 2; m++) {
                if (TRANS) {
                    const float y0[4] = {x[0][2 * m], x[1][2 * m], x[2][2 * m], x[3][2 * m]}, y1[4] = {x[0][2 * m + 1], x[1][2 * m + 1], x[2][2 * m + 1], x[3][2 * m + 1]};
                    split_rows<TP>(fp[k][m], y0, y1);
                } else {
                    split_rows<TP>(fp[k][m], x[2 * m], x[2 * m + 1]);
                }
            }
        }
        if (c + 1 < chunks) load_p(next_p);
        issue(c + 2);
        if (left) {
            const float *v = bufs + (c % 3) * Cfg::buf;
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int q = 0; q < Cols<N>::GROUPS; q++) {
                    Four<TV> fb[VN];
                    load_values<VN, TV>(fb, v + 16 * k * Cfg::v_stride + 32 * q, Cfg::v_stride, g, t);
#pragma unroll
                    for (int m = 0; m < 2; m++) mma16<VN, TP, TV>(&acc[m][VN * q], fp[k][m], fb);
                }
        }
        land(c + 2);
    }
    // rows without blocks are written as zeros (blocksparse.h:949-962)
    const size_t baseO = ((size_t)b * p.nb_a + i) * BS * HD + (size_t)h * p.d + n0;
    const bool odd = (TP > 1 || TV > 1) && !(zero_if_finite<N>(acc[1], zero_if_finite<N>(acc[0], 0.f)) == 0.f);
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const uint32_t r = r0 + (TRANS ? 4 * g + 2 * m + half : 16 * m + 8 * half + g);
            store_cols<BC_DT, N>(O, baseO + (size_t)r * HD, t, acc[m], half, 1.f, left, vec);
        }
    if ((TP > 1 || TV > 1) && __syncthreads_or(odd)) spmm_again<BS, DS, A_DT, BC_DT, TRANS>(sm, lut, Pm, V, O, p.H, p.d, p.nb_a, p.nb_b, p.blocks, p.lut_stride, avec, vec);
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

// The rows of a block-row whose outputs are not finite, made again by plain FMAs (simt_tile.cuh says why): the steps of the kernel
// below, by the same warps, on its shared memory, where the rows' flags come first.  q0, o0: first elements of the block-row; kv: of the keys and values;
// mask: this head's.
template <int BS, int NW> struct AgainCfg {
    static constexpr uint32_t red = BS, ps = red + 128, stage = ps + 128 * tile::kAgainRows;      // floats
    static constexpr uint32_t warp_floats = tile::kAgainFloats > tile::kAgain * tile::kAgainCols<NW> ? tile::kAgainFloats : tile::kAgain * tile::kAgainCols<NW>;
    static constexpr size_t bytes = 4 * (stage + 4 * warp_floats);
};
template <int BS, int DT, int NW>
__device__ __noinline__ void attention_again(float *sm, const uint2 *ent, uint32_t cnt, const void *Q, const void *K, const void *V, void *O,
                                             const typename MaskWord<BS>::type *mask, size_t q0, size_t kv, size_t o0, size_t HD, size_t HDo, uint32_t d, float scale_log2e)
{
    using namespace tile;
    typedef typename MaskWord<BS>::type W;
    typedef AgainCfg<BS, NW> Cfg;
    constexpr uint32_t G = BS == 32 ? 4 : 1, WC = BS == 32 ? 4 : 2;      // key blocks per step, warps per row
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wc = warp % WC, rg = warp / WC, r = 32 * rg + lane;
    const uint32_t n0 = wc * NW, left = d > n0 ? d - n0 : 0;
    float *red = sm + Cfg::red, *ps = sm + Cfg::ps + rg * 64 * kAgainRows, *buf = sm + Cfg::stage + warp * Cfg::warp_floats;
    float m = -INFINITY, l = 0.f, acc[NW] = {};
    for (uint32_t e = 0; e < cnt; e += G) {
        const uint32_t nblk = min(G, cnt - e);
        float s[32];
        if (G == 1 || wc < nblk) {
            const uint2 en = ent[e + (G == 1 ? 0 : wc)];
            scores_again<DT>(s, buf, Q, K, q0 + (size_t)(32 * rg) * HD, kv + ((size_t)en.y * BS + (G == 1 ? 32 * wc : 0)) * HD, HD, d, lane);
            const W w = mask ? mask[(size_t)en.x * BS + r] : ~(W)0;
#pragma unroll
            for (int n = 0; n < 32; n++) s[n] = (w >> (n + (G == 1 ? 32 * wc : 0))) & 1u ? s[n] * scale_log2e : -INFINITY;
        } else {
#pragma unroll
            for (int n = 0; n < 32; n++) s[n] = -INFINITY;
        }
        float mn = s[0];
#pragma unroll
        for (int n = 1; n < 32; n++) mn = fmaxf(mn, s[n]);
        red[warp * 32 + lane] = mn;
        __syncthreads();
        mn = m;
#pragma unroll
        for (uint32_t k = 0; k < WC; k++) mn = fmaxf(mn, red[(rg * WC + k) * 32 + lane]);
        const float alpha = mn > m ? exp2f(m - mn) : 1.f, off = mn > -INFINITY ? mn : 0.f;
        m = mn;
        l *= alpha;
#pragma unroll
        for (int n = 0; n < 32; n++) {
            const float pv = exp2f(s[n] - off);
            l += pv;
            ps[(32 * wc + n) * kAgainRows + lane] = pv;
        }
#pragma unroll
        for (int n = 0; n < NW; n++) acc[n] *= alpha;
        __syncthreads();
        if (left) {
            Again<kAgain, NW> v;
            v.template load<DT>(V, kv + (size_t)ent[e].y * BS * HD + n0, HD, left, lane);
            for (uint32_t k = 0; k < nblk * BS; k += kAgain) {
                __syncwarp();
                v.template put<kAgainCols<NW>, 1>(buf, lane);
                __syncwarp();
                const uint32_t next = k + kAgain;
                if (next < nblk * BS) v.template load<DT>(V, kv + ((size_t)ent[e + next / BS].y * BS + next % BS) * HD + n0, HD, left, lane);
                fma_again<NW>(acc, ps + k * kAgainRows, buf, lane);
            }
        }
    }
    __syncthreads();
    red[warp * 32 + lane] = l;
    __syncthreads();
    if (!((const uint32_t *)sm)[r]) return;
    l = 0.f;
#pragma unroll
    for (uint32_t k = 0; k < WC; k++) l += red[(rg * WC + k) * 32 + lane];
    const float inv = l > 0.f ? 1.f / l : l;                             // nothing kept: 0; NaN stays NaN
#pragma unroll
    for (int n = 0; n < NW; n++)
        if ((uint32_t)n < left) Elem<DT>::store(O, o0 + (size_t)r * HDo + n0 + n, acc[n] * inv);
}

// This warp's 32 x 32 probabilities as the A fragments of their product with the values: two of 16 keys per 16 rows (pitch: from
// one 16 rows to the next)
__device__ __forceinline__ void put_p(uint4 *at, uint32_t pitch, const float (&s)[2][4][4], uint32_t lane)
{
    using namespace tile;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float x0[4] = {s[m][2 * j][0], s[m][2 * j][1], s[m][2 * j + 1][0], s[m][2 * j + 1][1]};
            const float x1[4] = {s[m][2 * j][2], s[m][2 * j][3], s[m][2 * j + 1][2], s[m][2 * j + 1][3]};
            Frag<3> f;
            split_rows<3>(f, x0, x1);
            store_frag<3>(at + m * pitch + j * 3 * 32, lane, f);
        }
}

// SDDMM + softmax + SpMM with an online softmax; S and P never leave the SM.  One CTA (four warps) per block-row.
// A step takes four 32x32 key blocks (a 32x32 score tile per warp) or one 64x64 block (a quarter per warp): Q . K^T over
// chunks of 32 of d, the softmax in registers (row maxima meet in shared memory), P to shared memory as fragments, then
// O += P . V in chunks of 32 keys, each warp on its share of O's columns (and, for 64 rows, of its rows).  A warp stages
// the keys of its own scores and its own columns of the values (for 64 rows together with the warp that has the other half
// of the rows) as one sequence of chunks through a ring of ST buffers; all warps of a row meet twice per step, for the
// maxima and for P.  Score and O rows of a thread are the same, so O is rescaled in place.
// ST: two chunk buffers, three at blocks of 32 and d 128, where two CTAs share an SM and their memory has room; four for launches that the
// SMs hold at once: each CTA then waits alone.
// Measured (fp32, us, the FMA-pipe kernel before / this one with ex2.approx.ftz for the weights; exp2f, for their range, costs 1 to 3 % of it): B 1, H 4, L 512, d 64, fixed (64 CTAs) 14.8 / 12.1; B 8, H 4, L 2048, d 64, stride 179 / 136;
// d 128 317 / 245; blocks of 64, d 64 198 / 160; B 2, H 4, L 1024, d 64, full with a mask 77.5 / 57; B 32, H 4, L 1024, d 128, sawtooth 304 / 264.  At the
// last the tensor pipe is 41 % busy and a third of the issue slots are used, a quarter of them by the splits: the warps wait for fixed
// latencies, for their chunks and for the tensor pipe in turn.  Beside it were measured: eight warps of 16 keys and 16 columns 11.5 / 156 / 267 / 168 / 60 / 265;
// every warp a share of every key block of a step (no idle warps in a step of fewer than four) 13.2 / 138 / 254 / 159 / 71 / 267; keys and values
// straight to fragments without the ring, three CTAs per SM 291 at the last.
template <int BS, int D, int DT, int ST> struct FaCfg {
    static constexpr uint32_t G = BS == 32 ? 4 : 1;                      // key blocks per step
    static constexpr uint32_t NK = G * BS;                               // keys per step
    static constexpr uint32_t WC = BS == 32 ? 4 : 2;                     // teams: warps side by side (score columns, O columns)
    static constexpr int TT = 128 / WC, NW = D / WC, N = NW / 8;         // a team's threads and columns of O, n-tiles of 8 columns
    static constexpr uint32_t v_stride = NW + 8;
    static constexpr uint32_t kbuf = 32 * tile::kStride, vbuf = 32 * v_stride, buf = kbuf > vbuf ? kbuf : vbuf;
    static constexpr uint32_t T = tile::kTerms<DT>;
    static constexpr uint32_t qfrags = BS / 16 * (D / 16) * T * 32, pfrags = BS / 16 * (NK / 16) * 3 * 32;      // uint4
    static constexpr size_t bytes = 16 * (qfrags + pfrags) + 4 * (WC * ST * buf + WC * BS);
    static constexpr int ctas = bytes <= 75 * 1024 && N <= 4 ? 3 : bytes <= 113 * 1024 ? 2 : 1;       // what shared memory and registers allow per SM
};
template <int BS, int D, int DT, int ST>
__global__ void __launch_bounds__(tile::kThreads, (FaCfg<BS, D, DT, ST>::ctas))
fused_attention_kernel(const uint2 *__restrict__ lut, const void *__restrict__ Q, const void *__restrict__ K, const void *__restrict__ V,
                       void *__restrict__ O, const typename MaskWord<BS>::type *__restrict__ mask, AttnDims p, float scale_log2e, bool vec)
{
    using namespace tile;
    typedef typename MaskWord<BS>::type W;
    typedef FaCfg<BS, D, DT, ST> Cfg;
    constexpr int N = Cfg::N, T = Cfg::T, TT = Cfg::TT, ROWT = BS == 32 ? 128 : 64;      // ROWT: threads that share query rows
    constexpr uint32_t G = Cfg::G, WC = Cfg::WC, KQ = D / 16, KP = Cfg::NK / 16;
    extern __shared__ __align__(16) float sm[];
    uint4 *Qf = (uint4 *)sm, *Pf = Qf + Cfg::qfrags;
    float *bufs = (float *)(Pf + Cfg::pfrags), *red = bufs + WC * ST * Cfg::buf;
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // rows are dealt from both ends: the long rows of the layouts at hand sit there and start first
    const uint32_t i = (blockIdx.x & 1u) ? p.nb_a - 1u - (blockIdx.x >> 1) : blockIdx.x >> 1, b = blockIdx.y, h = blockIdx.z;
    const uint2 *nn = lut + (size_t)h * p.lut_stride;
    const uint2 head = nn[i];
    const size_t HD = p.in_pitch ? (size_t)p.in_pitch : (size_t)p.H * p.d;      // row pitch of q, k, v
    const size_t HDo = p.out_pitch ? (size_t)p.out_pitch : (size_t)p.H * p.d;   // row pitch of o
    const W *mh = mask ? mask + (size_t)h * p.mask_stride : nullptr;
    const uint32_t r0 = BS == 64 ? 32 * (warp >> 1) : 0, wc = BS == 64 ? warp & 1 : warp;   // this warp's rows and its team: score columns, columns of O
    const uint32_t rank = BS == 64 ? 32 * (warp >> 1) + lane : lane, n0 = wc * Cfg::NW;
    const uint32_t kchunks = (p.d + kChunk - 1) / kChunk;
    const uint32_t cnt = head.y, left = p.d > n0 ? p.d - n0 : 0;
    const size_t kv = (size_t)b * p.nb_b * BS * HD + (size_t)h * p.d;
    bufs += wc * ST * Cfg::buf;

    // the row's entries, 32 at a time, one per lane, the next 32 ahead
    uint32_t ent = lane < cnt ? nn[head.x + lane].y : 0u, ent2 = 32 + lane < cnt ? nn[head.x + 32 + lane].y : 0u;
    // the team's sequence of chunks: per step the key chunks of its block (if the step has one for it), then the value chunks
    uint32_t is_e = 0, is_k = 0, is_n = 0;                               // next chunk to issue: step's first entry, index in the step, overall
    Staged<DT, TT, (int)kChunk> held_k;
    Staged<DT, TT, Cfg::NW> held_v;
    uint32_t held = 0;                                                   // 16-bit pieces wait in registers: 1 keys, 2 values
    float *held_at = nullptr;
    auto issue = [&]() {
        held = 0;
        if (is_e < cnt) {
            const uint32_t nblk = min(G, cnt - is_e), mine = G == 1 || wc < nblk ? kchunks : 0;
            float *buf = bufs + (is_n % ST) * Cfg::buf;
            held_at = buf;
            if (is_k < mine) {
                const uint32_t key = __shfl_sync(0xffffffffu, ent, (is_e + (G == 1 ? 0 : wc)) % 32) * BS + (G == 1 ? 32 * wc : 0), k0 = is_k * kChunk;
                held = 1;
                stage_begin(held_k, rank, buf, kStride, K, kv + (size_t)key * HD + k0, HD, p.d - k0, vec);
            } else {
                const uint32_t vc = is_k - mine, key = __shfl_sync(0xffffffffu, ent, (is_e + (G == 1 ? 0 : vc)) % 32) * BS + (G == 1 ? 32 * vc : 0);
                held = 2;
                if (left) stage_begin(held_v, rank, buf, Cfg::v_stride, V, kv + (size_t)key * HD + n0, HD, left, vec);
            }
            is_n++;
            if (++is_k == mine + nblk * (BS / 32)) {
                is_k = 0;
                is_e += G;
                if (is_e % 32 == 0) {
                    ent = ent2;
                    ent2 = is_e + 32 + lane < cnt ? nn[head.x + is_e + 32 + lane].y : 0u;
                }
            }
        }
        cp_commit();                                                     // nothing left: an empty group keeps the count
    };
    auto land = [&]() {
        if (DT == SFB_F32) return;
        if (held == 1) stage_end(held_k, rank, held_at, kStride, vec);
        else if (held == 2 && left) stage_end(held_v, rank, held_at, Cfg::v_stride, vec);
    };

    if (cnt) {
#pragma unroll
        for (int k = 0; k < ST - 1; k++) {
            issue();
            land();
        }
        const size_t q0 = ((size_t)b * p.nb_a + i) * BS * HD + (size_t)h * p.d;
#pragma unroll 4
        for (uint32_t f = warp; f < BS / 16 * KQ; f += 4) {              // fragment f: rows 16 (f / KQ), elements 16 (f % KQ)
            const uint32_t k = 16 * (f % KQ) + 4 * t, n = k < p.d ? p.d - k : 0u;
            Raw4<DT> a0, a1;
            load_raw4<DT>(a0, Q, q0 + (size_t)(16 * (f / KQ) + g) * HD + k, n, vec);
            load_raw4<DT>(a1, Q, q0 + (size_t)(16 * (f / KQ) + 8 + g) * HD + k, n, vec);
            float x0[4], x1[4];
            widen4<DT>(x0, a0);
            widen4<DT>(x1, a1);
            Frag<T> fr;
            split_rows<T>(fr, x0, x1);
            store_frag<T>(Qf + f * T * 32, lane, fr);
        }
    }
    __syncthreads();
    float mx[4], sum[4];                                                 // of rows r0 + g + 8 q
    float acc[2][N][4] = {};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        mx[q] = -INFINITY;
        sum[q] = 0.f;
    }
    uint32_t c = 0;
    for (uint32_t e = 0; e < cnt; e += G) {
        const uint32_t nblk = min(G, cnt - e);
        const bool live = G == 1 || warp < nblk;
        float s[2][4][4] = {};
        if (live)
            for (uint32_t kc = 0; kc < kchunks; kc++, c++) {
                cp_wait<ST - 2>();
                meet<TT>(1 + wc);
                issue();
                const float *keys = bufs + (c % ST) * Cfg::buf;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    Four<T> fb[4];
                    load_keys<T, false>(fb, keys, 16 * k, g, t);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        Frag<T> fa;
                        load_frag<T>(fa, Qf + ((r0 / 16 + m) * KQ + 2 * kc + k) * T * 32, lane);
                        mma16<4, T, T>(s[m], fa, fb);
                    }
                }
                land();
            }
        const uint32_t blk = mh ? nn[head.x + e + (G > 1 && live ? warp : 0)].x : 0u;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t r = r0 + g + 8 * q;
            float bm = -INFINITY;
            if (mh) {
                const W w = live ? __ldg(mh + (size_t)blk * BS + r) : (W)0;
                const uint32_t bits = (uint32_t)(w >> (BS == 64 ? 32 * wc : 0));
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        float &v = s[q >> 1][j][2 * (q & 1) + k];
                        v = (bits >> score_key<false>(t, j, k)) & 1u ? v * scale_log2e : -INFINITY;
                        bm = fmaxf(bm, v);
                    }
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        float &v = s[q >> 1][j][2 * (q & 1) + k];
                        v = live ? v * scale_log2e : -INFINITY;
                        bm = fmaxf(bm, v);
                    }
            }
            bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
            bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
            if (t == 0) red[wc * BS + r] = bm;
        }
        meet<ROWT>(5 + (r0 >> 5));
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t r = r0 + g + 8 * q;
            float mn = mx[q];
#pragma unroll
            for (uint32_t k = 0; k < WC; k++) mn = fmaxf(mn, red[k * BS + r]);
            const float alpha = mn > mx[q] ? exp2f(mx[q] - mn) : 1.f;
            mx[q] = mn;
            const float off = mn > -INFINITY ? mn : 0.f;                 // nothing kept so far: exp2(-inf) = 0, and NaN stays NaN
            float ps = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    float &v = s[q >> 1][j][2 * (q & 1) + k];
                    v = exp2f(v - off);                              // not ex2_fast: that flushes weights below 2^-126 of the largest
                    ps += v;
                }
            sum[q] = fmaf(sum[q], alpha, ps);                            // this thread's columns only; the shares meet at the end
#pragma unroll
            for (int n = 0; n < N; n++) {
                acc[q >> 1][n][2 * (q & 1)] *= alpha;
                acc[q >> 1][n][2 * (q & 1) + 1] *= alpha;
            }
        }
        put_p(Pf + (r0 / 16 * KP + 2 * wc) * 3 * 32, KP * 3 * 32, s, lane);
        meet<ROWT>(5 + (r0 >> 5));
        const uint32_t vchunks = nblk * (BS / 32);
        for (uint32_t vc = 0; vc < vchunks; vc++, c++) {
            cp_wait<ST - 2>();
            meet<TT>(1 + wc);
            issue();
            if (left) mma_values<N, 3, T>(acc, Pf + (r0 / 16 * KP + 2 * vc) * 3 * 32, KP * 3 * 32, bufs + (c % ST) * Cfg::buf, Cfg::v_stride, lane);
            land();
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], 1);
        sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], 2);
        if (t == 0) red[wc * BS + r0 + g + 8 * q] = sum[q];
    }
    __syncthreads();
    const size_t baseO = (((size_t)b * p.nb_a + i) * BS) * HDo + (size_t)h * p.d;
    uint32_t odd = 0;                                                    // this thread's rows with an output that is not finite
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t r = r0 + g + 8 * q;
        float l = 0.f;
#pragma unroll
        for (uint32_t k = 0; k < WC; k++) l += red[k * BS + r];
        store_cols<DT, N>(O, baseO + (size_t)r * HDo + n0, t, acc[q >> 1], q & 1, l > 0.f ? 1.f / l : 0.f, left, vec);
        float zero = l * 0.f;
#pragma unroll
        for (int n = 0; n < N; n++) zero = fmaf(acc[q >> 1][n][2 * (q & 1)], 0.f, fmaf(acc[q >> 1][n][2 * (q & 1) + 1], 0.f, zero));
        if (!(zero == 0.f)) odd |= 1u << q;
    }
    if (!__syncthreads_or(odd != 0)) return;
    // such rows are made again by plain FMAs, once every warp has written its columns of them
    uint32_t *again = (uint32_t *)sm;
    if (threadIdx.x < BS) again[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++)
        if ((odd >> q) & 1u) again[r0 + g + 8 * q] = 1;
    __syncthreads();
    static_assert(Cfg::bytes >= AgainCfg<BS, Cfg::NW>::bytes, "attention_again works in the kernel's shared memory");
    attention_again<BS, DT, Cfg::NW>(sm, nn + head.x, cnt, Q, K, V, O, mh, ((size_t)b * p.nb_a + i) * BS * HD + (size_t)h * p.d, kv, baseO, HD, HDo, p.d, scale_log2e);
}

// ------------------------------------------------------------------------------------------------
// Element-sparse attention of one tile of 32 query rows on fp32 operands (csr.cu makes the tile's list of columns and
// row masks): the kernel above on keys gathered by column, 128 of them per step, a 32x32 score tile per warp.
template <int D> struct CsrF32Cfg : FaCfg<32, D, SFB_F32, D == 128 ? 3 : 2> {
    static constexpr int ST = D == 128 ? 3 : 2;
};
// 32 gathered rows x COLS elements by one warp: lane r has the column of row r, or -1 (zeros)
template <int COLS>
__device__ __forceinline__ void stage_gather(float *dst, uint32_t stride, const float *src, int32_t col, uint32_t lane, size_t pitch)
{
    using namespace tile;
    constexpr int P = COLS / 4, STEP = 32 / P;
    const uint32_t r0 = lane / P, c = (lane % P) * 4;
#pragma unroll
    for (int i = 0; i < 32 / STEP; i++) {
        const int32_t j = __shfl_sync(0xffffffffu, col, r0 + i * STEP);
        cp_async16(dst + (tile_row(r0) + tile_row(i * STEP)) * stride + c, src + (size_t)max(j, 0) * pitch + c, j < 0 ? 0u : 16u);
    }
}
template <int D>
__global__ void __launch_bounds__(tile::kThreads, CsrF32Cfg<D>::ctas) csr_tile_f32_kernel(const CsrTileArgs a)
{
    using namespace tile;
    typedef CsrF32Cfg<D> Cfg;
    constexpr int N = Cfg::N, ST = Cfg::ST;
    constexpr uint32_t NK = Cfg::NK, KQ = D / 16, KP = NK / 16, kchunks = D / kChunk;
    extern __shared__ __align__(16) float sm[];
    uint4 *Qf = (uint4 *)sm, *Pf = Qf + Cfg::qfrags;
    float *bufs = (float *)(Pf + Cfg::pfrags), *red = bufs + 4 * ST * Cfg::buf;
    grid_dependency_wait();
    grid_launch_dependents();
    csr_write_bad(a);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t tl = a.tiles - 1u - blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const uint32_t *cnt = a.counts + kCsrCounts * tl;
    const uint32_t distinct = cnt[0], base = cnt[2], top = cnt[3], n = distinct + cnt[1];
    const size_t HD = (size_t)a.H * D, head = (size_t)b * a.L * HD + (size_t)h * D;
    const float *K = (const float *)a.K + head, *V = (const float *)a.V + head;
    const uint32_t n0 = warp * (D / 4);
    bufs += warp * ST * Cfg::buf;

    // this warp's sequence of chunks: per step the key chunks of its 32 columns (if the step has any for it), then the value
    // chunks.  A chunk's columns are asked for when the one before is issued.
    uint32_t is_e = 0, is_k = 0, is_n = 0;                               // next chunk to issue: step's first key, index in the step, overall
    auto column = [&](uint32_t first) { return first + lane < n ? (int32_t)csr_entry(a.entries, base, top, distinct, first + lane).x : -1; };
    int32_t kcol = column(32 * warp), vcol = column(0);                  // of the key chunks at hand, of the next value chunk
    auto issue = [&]() {
        if (is_e < n) {
            const uint32_t left = min(NK, n - is_e), mine = 32 * warp < left ? kchunks : 0, vchunks = (left + 31) / 32;
            float *buf = bufs + (is_n % ST) * Cfg::buf;
            if (is_k < mine) {
                stage_gather<(int)kChunk>(buf, kStride, K + is_k * kChunk, kcol, lane, HD);
                if (is_k + 1 == mine) kcol = column(is_e + NK + 32 * warp);
            } else {
                const uint32_t vc = is_k - mine;
                stage_gather<(int)Cfg::NW>(buf, Cfg::v_stride, V + n0, vcol, lane, HD);
                vcol = column(vc + 1 < vchunks ? is_e + 32 * (vc + 1) : is_e + NK);
            }
            is_n++;
            if (++is_k == mine + vchunks) {
                is_k = 0;
                is_e += NK;
            }
        }
        cp_commit();                                                     // nothing left: an empty group keeps the count
    };
    if (n) {
#pragma unroll
        for (int k = 0; k < ST - 1; k++) issue();
        const uint32_t rows = min(32u, a.L - tl * 32);                   // rows behind the sequence: the last one again, not written
#pragma unroll 4
        for (uint32_t f = warp; f < 2 * KQ; f += 4) {
            float x[2][4];
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const uint32_t r = min(16 * (f / KQ) + 8 * half + g, rows - 1);
                const float4 v = __ldg((const float4 *)((const float *)a.Q + head + (size_t)(tl * 32 + r) * HD + 16 * (f % KQ) + 4 * t));
                x[half][0] = v.x; x[half][1] = v.y; x[half][2] = v.z; x[half][3] = v.w;
            }
            Frag<3> fr;
            split_rows<3>(fr, x[0], x[1]);
            store_frag<3>(Qf + f * 3 * 32, lane, fr);
        }
    }
    __syncthreads();
    float mx[4], sum[4];                                                 // of rows g + 8 q
    float acc[2][N][4] = {};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        mx[q] = -INFINITY;
        sum[q] = 0.f;
    }
    uint32_t c = 0;
    for (uint32_t e = 0; e < n; e += NK) {
        const uint32_t left = min(NK, n - e);
        const bool live = 32 * warp < left;
        float s[2][4][4] = {};
        uint32_t mk[8];                                                  // the rows of this thread's eight columns
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t col = 32 * warp + score_key<false>(t, j >> 1, j & 1);
            mk[j] = col < left ? csr_entry(a.entries, base, top, distinct, e + col).y : 0u;
        }
        if (live)
            for (uint32_t kc = 0; kc < kchunks; kc++, c++) {
                cp_wait<ST - 2>();
                __syncwarp();
                issue();
                const float *keys = bufs + (c % ST) * Cfg::buf;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    Four<3> fb[4];
                    load_keys<3, false>(fb, keys, 16 * k, g, t);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        Frag<3> fa;
                        load_frag<3>(fa, Qf + (m * KQ + 2 * kc + k) * 3 * 32, lane);
                        mma16<4, 3, 3>(s[m], fa, fb);
                    }
                }
            }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float bm = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float &v = s[q >> 1][j >> 1][2 * (q & 1) + (j & 1)];
                v = (mk[j] >> (g + 8 * q)) & 1u ? v * a.scale_log2e : -INFINITY;
                bm = fmaxf(bm, v);
            }
            bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
            bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
            if (t == 0) red[warp * 32 + g + 8 * q] = bm;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t r = g + 8 * q;
            float mn = mx[q];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) mn = fmaxf(mn, red[k * 32 + r]);
            const float alpha = mn > mx[q] ? exp2f(mx[q] - mn) : 1.f;
            mx[q] = mn;
            const float off = mn > -INFINITY ? mn : 0.f;                 // nothing kept so far: exp2(-inf) = 0, and NaN stays NaN
            float ps = 0.f;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float &v = s[q >> 1][j >> 1][2 * (q & 1) + (j & 1)];
                v = exp2f(v - off);                              // not ex2_fast: that flushes weights below 2^-126 of the largest
                ps += v;
            }
            sum[q] = fmaf(sum[q], alpha, ps);                            // this thread's columns only; the shares meet at the end
#pragma unroll
            for (int j = 0; j < N; j++) {
                acc[q >> 1][j][2 * (q & 1)] *= alpha;
                acc[q >> 1][j][2 * (q & 1) + 1] *= alpha;
            }
        }
        put_p(Pf + 2 * warp * 3 * 32, KP * 3 * 32, s, lane);
        __syncthreads();
        const uint32_t vchunks = (left + 31) / 32;
        for (uint32_t vc = 0; vc < vchunks; vc++, c++) {
            cp_wait<ST - 2>();
            __syncwarp();
            issue();
            mma_values<N, 3, 3>(acc, Pf + 2 * vc * 3 * 32, KP * 3 * 32, bufs + (c % ST) * Cfg::buf, Cfg::v_stride, lane);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], 1);
        sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], 2);
        if (t == 0) red[warp * 32 + g + 8 * q] = sum[q];
    }
    __syncthreads();
    uint32_t odd = 0;                                                    // this thread's rows with an output that is not finite
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t r = g + 8 * q;
        float l = 0.f;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) l += red[k * 32 + r];
        const float inv = l > 0.f ? 1.f / (l + 1e-6f) : 0.f;             // the reference's denominator (ewops.h:93, cuda_kernels.h:1022)
        if (tl * 32 + r < a.L) store_cols<SFB_F32, N>(a.O, head + (size_t)(tl * 32 + r) * HD + n0, t, acc[q >> 1], q & 1, inv, D / 4, true);
        float zero = 0.f;                                                // stays 0 as long as every output is finite
#pragma unroll
        for (int j = 0; j < N; j++) zero = fmaf(acc[q >> 1][j][2 * (q & 1)], 0.f, fmaf(acc[q >> 1][j][2 * (q & 1) + 1], 0.f, zero));
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
        const size_t bytes = sizeof(float) * 2 * SddmmCfg<BS>::TEAMS * SddmmCfg<BS>::buf;                         \
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

// FMAs: fp32 blocks, whose split every warp makes again for its own columns.  Split products / FMAs, us, transposed: sawtooth rows of
// eight, B 8, H 8, 24 block-rows of 32, d 32 33.1 / 19.2, d 64 38.1 / 27.8; full rows, B 1, H 4, 16 block-rows of 64, d 128 84.2 / 57.1;
// BigBird rows, B 4, H 8, 64 block-rows of 32, d 128, not transposed 184.6 / 211.6.  With 16-bit blocks of 32 at d 32, where a warp has eight columns to
// spend a fragment of P on, neither is ahead of the other: fp16, transposed, the sawtooth rows 28.3 / 23.4, full rows 11.8 / 15.3.
template <int BS, int DS, int AD, int BD, bool TRANS>
static int launch_spmm(cudaStream_t s, const void *lut, const void *a, const void *b, void *c, const AttnDims &p, bool avec, bool vec)
{
    static DeviceOnce once;
    const dim3 grid(p.nb_a * ((p.d + DS - 1) / DS), p.B, p.H);
    if constexpr (AD == SFB_F32) {
        if (set_smem(once, spmm_fma_kernel<BS, DS, AD, BD, TRANS>, SpmmFmaCfg<BS, DS>::bytes)) return 1;
        launch_overlapped(spmm_fma_kernel<BS, DS, AD, BD, TRANS>, grid, dim3(tile::kThreads), SpmmFmaCfg<BS, DS>::bytes, s, (const uint2 *)lut, a, b, c, p, avec, vec);
    } else {
        if (set_smem(once, spmm_nn_kernel<BS, DS, AD, BD, TRANS>, SpmmCfg<BS, DS>::bytes)) return 1;
        launch_overlapped(spmm_nn_kernel<BS, DS, AD, BD, TRANS>, grid, dim3(tile::kThreads), SpmmCfg<BS, DS>::bytes, s, (const uint2 *)lut, a, b, c, p, avec, vec);
    }
    return 0;
}
int simt_spmm_nn(cudaStream_t s, const void *lut, const void *a, const void *b, void *c, int a_dtype, int bc_dtype,
                 uint32_t bs, const AttnDims &p, bool trans)
{
    const uint64_t HD = (uint64_t)p.H * p.d;
    const bool avec = ((uintptr_t)a & 15) == 0, vec = rows_vec(b, bc_dtype, HD, p.d) && rows_vec(c, bc_dtype, HD, p.d);
#define SP_LAUNCH(DSV) { if (trans ? launch_spmm<BS, DSV, AD, BD, true>(s, lut, a, b, c, p, avec, vec) : launch_spmm<BS, DSV, AD, BD, false>(s, lut, a, b, c, p, avec, vec)) return 1; }
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
    // a launch that the SMs hold at once waits for its chunks one after another: more of them on their way
    // (B 1, H 4, L 512, d 64: 64 CTAs)
    const int sms = device_sm_count(current_device());
    const uint64_t ctas = (uint64_t)p.nb_a * p.B * p.H;
#define LAUNCH_FA_ST(DV, STV)                                                                                    \
    {                                                                                                            \
        typedef typename MaskWord<BS>::type W;                                                                   \
        const size_t bytes = FaCfg<BS, DV, DT, STV>::bytes;                                                      \
        auto kern = fused_attention_kernel<BS, DV, DT, STV>;                                                     \
        static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                       \
        launch_overlapped(kern, grid, dim3(tile::kThreads), bytes, s, (const uint2 *)nn_lut, q, k, v, o, (const W *)mask, p, sl, vec); \
    }
#define LAUNCH_FA(DV) { if (ctas <= (uint64_t)(sms > 0 ? sms : 0) * FaCfg<BS, DV, DT, 4>::ctas) LAUNCH_FA_ST(DV, 4) else LAUNCH_FA_ST(DV, (BS == 32 && DV == 128 ? 3 : 2)) }
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
        const size_t bytes = CsrF32Cfg<DV>::bytes;                                                               \
        auto kern = csr_tile_f32_kernel<DV>;                                                                     \
        static DeviceOnce once; if (set_smem(once, kern, bytes)) return 1;                                       \
        launch_overlapped(kern, dim3(a.tiles, a.H, B), dim3(tile::kThreads), bytes, s, a);                       \
    }
    if (d == 32) LAUNCH_CT(32) else if (d == 64) LAUNCH_CT(64) else LAUNCH_CT(128)
#undef LAUNCH_CT
    return check_launch("sfb_csr_attention");
}

}  // namespace sfb
