// Dense projection on the 5th-generation tensor cores: out[m, n] = act(x[m, k] . w[k, n] + bias[n]) for 16-bit
// x, w and out (fp32 accumulation, fp32 bias).  This is the product the encoder layer makes six times around the
// block-sparse attention (Q/K/V/output projections, the two FFN matrices), with the bias add and the GELU that
// the reference launches as separate kernels folded into the epilogue.
//
// Persistent, one CTA per SM.  A CTA tile is 128 rows x 256 columns: x arrives by TMA as a K-major A operand
// (128 x 64 per stage), w -- row-major [k, n], so n is the contiguous direction -- as an MN-major B operand
// (four 64 x 64 boxes per stage, one 128-byte swizzle span each; the descriptor's leading-dimension offset
// steps from one to the next), four stages of 48 KB.  One thread issues M128 N256 K16 tcgen05.mma into one of
// two 256-column accumulators in TMEM; eight epilogue warps drain the other one (tcgen05.ld, bias, activation,
// 32-byte stores), so the epilogue of a tile runs under the MMAs of the next.
// Every wait on an mbarrier is bounded; on a timeout the CTA records a status word and leaves through the
// common teardown.
#include "tc_common.cuh"

namespace sfb {
namespace tc {

constexpr uint32_t kGBM = 128, kGBN = 256, kGBK = 64;
constexpr uint32_t kGABytes = kGBM * kGBK * 2;           // 16 KB per 128 rows
constexpr uint32_t kGBBytes = kGBK * kGBN * 2;           // 32 KB: four 64 x 64 boxes
constexpr uint32_t kBiasBytes = 2 * 2 * 128 * 4;          // the epilogue's bias: [accumulator][column half][128]
constexpr int kGStages = 4, kGBufs = 2;
constexpr uint32_t kGStageBytes = kGABytes + kGBBytes;
constexpr size_t kGSmem = 1024 + kGStages * kGStageBytes + kBiasBytes + 256;

struct GShared {
    uint64_t full[kGStages], empty[kGStages], acc_full[2], acc_empty[2], drained;
    uint32_t tmem_base, abort_flag;
};
static_assert(sizeof(GShared) <= 256, "GShared outgrew its slot");

struct GParams {
    void *out;
    const float *bias;
    uint32_t M, N, K, tiles_m, tiles_n;
    int is_bf16, act;
    int w_transposed;   // w is [n, k] row-major (out = x . w^T, the tied-embedding logits): its tile is a K-major B operand
    uint32_t band;      // CTA-pair kernel: column tiles per band of the tile order (tile_coords)
    const void *resid;  // split kernel: [m, n] of x's type, added to the product (not out itself), or NULL
};

// Tile t of the CTA-pair kernel -> (row tile, column tile).  The tiles run band by band, a band being `band` column
// tiles wide, row tile by row tile inside it: the pairs that work at the same time then spread over `band` different
// w tiles and a stripe of x tiles, instead of all asking the same few L2 slices for one w tile at once (eight wide: the
// 74 pairs of a B200 then cover about nine row tiles by eight column tiles; measured against 1, 2 and 4).
__device__ __forceinline__ void tile_coords(const GParams &p, uint32_t t, uint32_t &tm, uint32_t &tn)
{
    const uint32_t per_band = p.tiles_m * p.band;
    const uint32_t b = t / per_band, rem = t - b * per_band;
    const uint32_t width = min(p.band, p.tiles_n - b * p.band);    // the last band may be narrower
    tm = rem / width;
    tn = b * p.band + (rem - tm * width);
}

// Four of the bias values of the 128 columns from n0 on, for this lane.  The epilogue reads them from shared memory: from
// global memory they cost it a trip to the cache per 16 columns, one after another.  Each epilogue warp keeps the values
// of its tile (fetched a tile ahead) in the slot of its column half and the tile's accumulator; the four warps that
// share a slot write the same values.  A warp writes the slot of tile i only once tile i's accumulator is full: that
// accumulator was emptied by every warp at tile i - 2, so none still reads the slot's earlier values.  (Written before that
// wait, a warp whose rows lie beyond the output, and which therefore stores nothing, could be two tiles ahead.)
__device__ __forceinline__ float4 fetch_bias(const GParams &p, uint32_t n0, uint32_t lane)
{
    return p.bias && n0 + lane * 4 < p.N ? __ldg((const float4 *)(p.bias + n0 + lane * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ float gelu_ref(float t)
{
    // x * sigmoid(1.702 x), the reference's GELU (gelu_gpu_v2, cuda_kernels.h:561-581), as
    // 0.5 x tanh(0.851 x) + 0.5 x: one MUFU operation per element instead of an exponential and a reciprocal
    // (tanh.approx: relative error about 2^-11, below half a unit of the 16-bit output)
    float th;
    asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(0.851f * t));
    const float h = 0.5f * t;
    return fmaf(h, th, h);
}

// One thread's share of a 128-row accumulator: row `row` of the output, 128 columns from n0 on, read from TMEM at
// tcol 32 columns at a time (the next 32 travel while these are written), bias and activation applied, 32-byte stores.
__device__ __forceinline__ void drain_rows(const GParams &p, uint32_t tcol, const float *bias, uint32_t row, uint32_t n0)
{
    const bool row_ok = row < p.M;
    const size_t off = (size_t)row * p.N + n0;
    uint32_t v[2][32];
    TMEM_LD_32((v[0]), tcol);
#pragma unroll
    for (uint32_t c = 0; c < 4; c++) {
        const uint32_t c0 = c * 32;
        tmem_wait_ld();
        if (c + 1 < 4) TMEM_LD_32((v[(c + 1) & 1]), tcol + c0 + 32);
        uint32_t(&cur)[32] = v[c & 1];
#pragma unroll
        for (uint32_t q = 0; q < 2; q++) {
            const uint32_t col = n0 + c0 + q * 16;
            if (row_ok && col < p.N) {      // N is a multiple of 16: a group of 16 is inside or outside as a whole
                float x[16];
#pragma unroll
                for (int j = 0; j < 16; j++) x[j] = __uint_as_float(cur[q * 16 + j]);
                if (p.bias) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float4 bb = *(const float4 *)(bias + c0 + q * 16 + 4 * j);   // the same address in every lane: one broadcast
                        x[4 * j] += bb.x; x[4 * j + 1] += bb.y; x[4 * j + 2] += bb.z; x[4 * j + 3] += bb.w;
                    }
                }
                if (p.act == 1) {
#pragma unroll
                    for (int j = 0; j < 16; j++) x[j] = gelu_ref(x[j]);
                }
                uint32_t w[8];
#pragma unroll
                for (int j = 0; j < 8; j++) w[j] = pack2(x[2 * j], x[2 * j + 1], p.is_bf16);
                asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"((uint16_t *)p.out + off + c0 + q * 16),
                             "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                             : "memory");
            }
        }
    }
}

// The same share of an accumulator, leaving through shared memory: the warp's 32 rows x 64 columns are packed into a
// staging tile in the tensor map's 128-byte swizzle (16-byte chunk c of row r at chunk c ^ (r % 8)) and one lane hands
// the tile to the TMA, twice per 128 columns.  The writes reach memory as whole 128-byte rows instead of 32 bytes per
// thread and instruction, and the storing threads are free as soon as the tile is in shared memory.
// row0 = first of the warp's 32 rows, n0 = first of its 128 columns.
__device__ __forceinline__ void drain_rows_staged(const GParams &p, const CUtensorMap *omap, uint32_t tcol, uint8_t *stage, const float *bias,
                                                  uint32_t row0, uint32_t n0, uint32_t lane)
{
    uint8_t *srow = stage + lane * 128;
    uint32_t v[2][32];
    TMEM_LD_32((v[0]), tcol);
#pragma unroll
    for (uint32_t c = 0; c < 4; c++) {
        const uint32_t c0 = c * 32;
        tmem_wait_ld();
        if (c + 1 < 4) TMEM_LD_32((v[(c + 1) & 1]), tcol + c0 + 32);
        if ((c & 1) == 0) {
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the store that used the tile has read it
            __syncwarp();
        }
        uint32_t(&cur)[32] = v[c & 1];
#pragma unroll
        for (uint32_t q = 0; q < 2; q++) {
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; j++) x[j] = __uint_as_float(cur[q * 16 + j]);
            if (p.bias) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 bb = *(const float4 *)(bias + c0 + q * 16 + 4 * j);
                    x[4 * j] += bb.x; x[4 * j + 1] += bb.y; x[4 * j + 2] += bb.z; x[4 * j + 3] += bb.w;
                }
            }
            if (p.act == 1) {
#pragma unroll
                for (int j = 0; j < 16; j++) x[j] = gelu_ref(x[j]);
            }
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 8; j++) w[j] = pack2(x[2 * j], x[2 * j + 1], p.is_bf16);
            const uint32_t ch = ((c & 1) * 32 + q * 16) >> 3;     // 16-byte chunk of the 128-byte row
            *(uint4 *)(srow + ((ch ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
            *(uint4 *)(srow + (((ch + 1) ^ (lane & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
        }
        if (c & 1) {
            fence_proxy_async();
            __syncwarp();
            const uint32_t col0 = n0 + (c0 - 32);
            if (lane == 0 && col0 < p.N && row0 < p.M) {      // rows and columns of the box beyond the tensor are not written
                asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                             ::"l"((uint64_t)omap), "r"(smem_u32(stage)), "r"((int32_t)col0), "r"((int32_t)row0) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        }
    }
}

__global__ void __launch_bounds__(320, 1)
linear_tc_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap, const GParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *tiles = smem;                                   // stage s: A (16 KB) then B (32 KB)
    float *bias_s = (float *)(tiles + kGStages * kGStageBytes);
    GShared *st = (GShared *)((uint8_t *)bias_s + kBiasBytes);

    const uint32_t warp = uniform_warp(), lane = threadIdx.x & 31;
    volatile uint32_t *abort_flag = &st->abort_flag;
    const uint32_t fmt = p.is_bf16 ? 1u : 0u;
    const uint32_t n_tiles = p.tiles_m * p.tiles_n;
    const uint32_t kblocks = (p.K + kGBK - 1) / kGBK;

    if (threadIdx.x == 0) {
        prefetch_map(amap);
        prefetch_map(bmap);
        for (int s = 0; s < kGStages; s++) { mbar_init(&st->full[s], 1); mbar_init(&st->empty[s], 1); }
        for (int s = 0; s < 2; s++) { mbar_init(&st->acc_full[s], 1); mbar_init(&st->acc_empty[s], 256); }
        mbar_init(&st->drained, 1);
        st->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&st->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = st->tmem_base;
    grid_dependency_wait();        // set-up done; x (and a w or bias written on the device) come from kernels before this one
    grid_launch_dependents();

    if (warp == 0) {
        // ===== TMA producer =====
        if (elect_one()) {
            uint32_t g = 0;   // k-blocks loaded so far (ring position)
            for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
                const int32_t m0 = (int32_t)((t % p.tiles_m) * kGBM), n0 = (int32_t)((t / p.tiles_m) * kGBN);
                bool alive = true;
                for (uint32_t kb = 0; kb < kblocks; kb++, g++) {
                    const uint32_t s = g % kGStages;
                    if (g >= kGStages && !mbar_wait(&st->empty[s], ((g / kGStages) - 1) & 1, abort_flag, 41)) { alive = false; break; }
                    const uint32_t base = smem_u32(tiles + s * kGStageBytes);
                    mbar_expect_tx(&st->full[s], kGStageBytes);   // boxes beyond the tensor arrive as zeros and still count
                    tma_load_2d(base, &amap, &st->full[s], (int32_t)(kb * kGBK), m0);
                    if (p.w_transposed) {
                        // 256 rows of w, 64 of k: one box
                        tma_load_2d(base + kGABytes, &bmap, &st->full[s], (int32_t)(kb * kGBK), n0);
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 4; j++)
                            tma_load_2d(base + kGABytes + j * kTileBytes, &bmap, &st->full[s], n0 + (int32_t)(j * 64), (int32_t)(kb * kGBK));
                    }
                }
                if (!alive) break;
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer =====
        if (elect_one()) {
            const uint32_t idesc = instr_desc(fmt, fmt, kGBM, kGBN, p.w_transposed ? 0 : 1);
            const uint32_t b_step = p.w_transposed ? 2u : 128u;   // descriptor units of 16 bytes per 16 of K
            uint32_t g = 0, i = 0;
            for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x, i++) {
                const uint32_t buf = i % kGBufs;
                bool alive = true;
                if (i >= (uint32_t)kGBufs && !mbar_wait(&st->acc_empty[buf], ((i / kGBufs) - 1) & 1, abort_flag, 42)) break;
                tcgen05_fence_after();
                for (uint32_t kb = 0; kb < kblocks; kb++, g++) {
                    const uint32_t s = g % kGStages;
                    if (!mbar_wait(&st->full[s], (g / kGStages) & 1, abort_flag, 43)) { alive = false; break; }
                    tcgen05_fence_after();
                    const uint32_t base = smem_u32(tiles + s * kGStageBytes);
                    // MN-major: the next 64 columns are one box further on; K-major: 256 rows of 128 bytes
                    const uint64_t b_desc = p.w_transposed ? smem_desc_sw128(base + kGABytes) : smem_desc_sw128(base + kGABytes, kTileBytes);
                    const uint64_t a_desc = smem_desc_sw128(base);
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++)   // 16 of K per MMA: +32 bytes in A's swizzled rows, +16 rows (2048 bytes) in B
                        umma_f16(tmem + buf * kGBN, a_desc + 2 * kk, b_desc + b_step * kk, idesc, (kb | kk) ? 1u : 0u);
                    umma_commit(&st->empty[s]);
                }
                if (!alive) break;
                umma_commit(&st->acc_full[buf]);
            }
        }
    } else {
        // ===== epilogue: eight warps; a thread takes one output row and half of the tile's 256 columns, 32 at a time =====
        const uint32_t quarter = warp & 3;                 // TMEM lanes this warp may touch
        const uint32_t chalf = (warp - 2) >> 2;            // which 128 columns
        const uint32_t r = quarter * 32 + lane;
        const uint32_t lane_field = (quarter * 32) << 16;
        uint32_t i = 0;
        float4 next = fetch_bias(p, (blockIdx.x / p.tiles_m) * kGBN + chalf * 128, lane);
        for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x, i++) {
            const uint32_t buf = i % kGBufs;
            const uint32_t n0 = (t / p.tiles_m) * kGBN + chalf * 128;
            float *bias = bias_s + ((i & 1) * 2 + chalf) * 128;
            if (!mbar_wait_warp(&st->acc_full[buf], (i / kGBufs) & 1, abort_flag, 44)) break;
            *(float4 *)(bias + lane * 4) = next;
            __syncwarp();
            if (t + gridDim.x < n_tiles) next = fetch_bias(p, ((t + gridDim.x) / p.tiles_m) * kGBN + chalf * 128, lane);
            tcgen05_fence_after();
            drain_rows(p, tmem + buf * kGBN + chalf * 128 + lane_field, bias, (t % p.tiles_m) * kGBM + r, n0);
            tcgen05_fence_before();
            mbar_arrive(&st->acc_empty[buf]);
        }
    }

    // ---- teardown (also the way out after a timeout) ----
    tcgen05_fence_before();
    __syncthreads();
    if (st->abort_flag) {
        if (warp == 1 && lane == 0) {
            umma_commit(&st->drained);
            for (uint32_t k = 0; k < kWaitLimit && !mbar_try_wait(&st->drained, 0); k++) {}
        }
        if (warp == 0 && lane == 0) {
            const uint64_t t0 = clock64();
            while (clock64() - t0 < 2000000ull) {}
        }
        __syncthreads();
    }
    if (warp == 0) {
        __syncwarp();
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- the same product on CTA pairs ------------------------------------------------------------------------
// With one CTA per tile the kernel above is bound by shared-memory bandwidth: an M128 N256 K16 MMA reads 4 KB of A and
// 8 KB of B from shared memory in its 128 cycles while the TMA writes the next stage at the same rate -- more than
// the 128 bytes per clock an SM's shared memory moves, which is where its 61 % tensor-pipe activity comes from.
// Here the two CTAs of a cluster (the two SMs of a TPC) share a 256 x 256 tile: each loads its own 128 rows of x and
// only HALF of the w tile (128 of the 256 columns), and one thread of the even CTA issues tcgen05.mma.cta_group::2
// (M 256), which reads A and its half of B from each CTA's own shared memory and writes each CTA's 128 rows of the
// accumulator into that CTA's TMEM.  Per CTA and MMA: 4 KB + 4 KB read, and stages of 32 KB instead of 48.
//   * Both producers signal the even CTA's `full` barrier (it expects the bytes of both); the commit after a stage's
//     MMAs arrives on the `empty` barrier of both CTAs, the commit after a tile on both `acc_full` barriers.
//   * Each CTA drains its own 128 rows (through per-warp staging tiles and TMA stores); its epilogue warps arrive on
//     the even CTA's `acc_empty` barrier.
//   * No load is a multicast: each CTA fetches what it multiplies.
#ifndef SFB_GEMM_PAIRS
#define SFB_GEMM_PAIRS 1
#endif
constexpr bool kUsePairs = SFB_GEMM_PAIRS != 0;
#ifndef SFB_GEMM_BAND
#define SFB_GEMM_BAND 8
#endif
constexpr uint32_t kPBand = SFB_GEMM_BAND;
constexpr uint32_t kPStages = 6;
constexpr uint32_t kPStagingBytes = 8 * 32 * 128;     // one 32-row x 64-column tile per epilogue warp
constexpr uint32_t kPABytes = kGBM * kGBK * 2;            // 16 KB: this CTA's 128 rows of x
constexpr uint32_t kPBBytes = kGBK * (kGBN / 2) * 2;      // 16 KB: this CTA's 128 columns of w
constexpr uint32_t kPStageBytes = kPABytes + kPBBytes;
// the shared window starts on a multiple of 1024 (aligned below): there is no room left for slack
constexpr size_t kPSmem = kPStages * kPStageBytes + kPStagingBytes + kBiasBytes + 256;
static_assert(kPSmem <= 227 * 1024, "shared memory budget");

struct PShared {
    uint64_t full[kPStages], empty[kPStages], acc_full[2], acc_empty[2], drained;
    uint32_t tmem_base, abort_flag;
};
static_assert(sizeof(PShared) <= 256, "PShared outgrew its slot");

__device__ __forceinline__ uint32_t cluster_ctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address, in the cluster's shared window, of this CTA's shared-memory address `addr` in CTA `rank`
__device__ __forceinline__ uint32_t mapa_rank(uint32_t addr, uint32_t rank)
{
    uint32_t d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
    return d;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// a tile into this CTA's shared memory, its bytes counted on a barrier that may live in the other CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster_addr, int32_t x, int32_t y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"((uint64_t)map), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar)
{
    const uint16_t both = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"(both)
                 : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1)
linear_tc_pair_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap,
                      const __grid_constant__ CUtensorMap omap, const GParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_aligned[];
    uint8_t *tiles = smem_aligned;                                   // stage s: A (16 KB) then this CTA's half of B (16 KB)
    uint8_t *staging = tiles + kPStages * kPStageBytes;      // the epilogue warps' output tiles (4 KB each)
    float *bias_s = (float *)(staging + kPStagingBytes);
    PShared *st = (PShared *)((uint8_t *)bias_s + kBiasBytes);

    const uint32_t warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();                 // 0: issues the MMAs of the pair
    const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    volatile uint32_t *abort_flag = &st->abort_flag;
    const uint32_t fmt = p.is_bf16 ? 1u : 0u;
    const uint32_t n_tiles = p.tiles_m * p.tiles_n;          // tiles of 256 x 256
    const uint32_t kblocks = (p.K + kGBK - 1) / kGBK;

    if (threadIdx.x == 0) {
        prefetch_map(amap);
        prefetch_map(bmap);
        prefetch_map(omap);
        for (uint32_t s = 0; s < kPStages; s++) { mbar_init(&st->full[s], 1); mbar_init(&st->empty[s], 1); }
        for (int s = 0; s < 2; s++) { mbar_init(&st->acc_full[s], 1); mbar_init(&st->acc_empty[s], 16); }   // 8 epilogue warps of each CTA
        mbar_init(&st->drained, 1);
        st->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&st->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();                                      // both CTAs' barriers exist before anything signals across
    tcgen05_fence_after();
    const uint32_t tmem = st->tmem_base;
    grid_dependency_wait();        // set-up done; nothing of global memory has been read yet
    grid_launch_dependents();

    if (warp == 0) {
        // ===== TMA producer (both CTAs): own rows of x, own half of the w tile; bytes counted on the even CTA's barrier =====
        if (elect_one()) {
            uint32_t g = 0;
            for (uint32_t t = pair; t < n_tiles; t += pairs) {
                uint32_t tm, tn;
                tile_coords(p, t, tm, tn);
                const int32_t m0 = (int32_t)(tm * 256 + rank * kGBM);
                const int32_t n0 = (int32_t)(tn * kGBN + rank * (kGBN / 2));
                bool alive = true;
                for (uint32_t kb = 0; kb < kblocks; kb++, g++) {
                    const uint32_t s = g % kPStages;
                    if (g >= kPStages && !mbar_wait(&st->empty[s], ((g / kPStages) - 1) & 1, abort_flag, 51)) { alive = false; break; }
                    const uint32_t base = smem_u32(tiles + s * kPStageBytes);
                    const uint32_t bar = mapa_rank(smem_u32(&st->full[s]), 0);
                    if (rank == 0) mbar_expect_tx(&st->full[s], 2 * kPStageBytes);   // both CTAs' bytes; boxes beyond the tensor arrive as zeros and still count
                    tma_load_2d_pair(base, &amap, bar, (int32_t)(kb * kGBK), m0);
                    if (p.w_transposed) {
                        tma_load_2d_pair(base + kPABytes, &bmap, bar, (int32_t)(kb * kGBK), n0);      // 128 rows of w, 64 of k
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 2; j++)
                            tma_load_2d_pair(base + kPABytes + j * kTileBytes, &bmap, bar, n0 + (int32_t)(j * 64), (int32_t)(kb * kGBK));
                    }
                }
                if (!alive) break;
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer: one thread of the even CTA for the pair =====
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = instr_desc(fmt, fmt, 256, kGBN, p.w_transposed ? 0 : 1);
            const uint32_t b_step = p.w_transposed ? 2u : 128u;
            uint32_t g = 0, i = 0;
            for (uint32_t t = pair; t < n_tiles; t += pairs, i++) {
                const uint32_t buf = i & 1;
                bool alive = true;
                if (i >= 2 && !mbar_wait(&st->acc_empty[buf], ((i >> 1) - 1) & 1, abort_flag, 52)) break;
                tcgen05_fence_after();
                for (uint32_t kb = 0; kb < kblocks; kb++, g++) {
                    const uint32_t s = g % kPStages;
                    if (!mbar_wait(&st->full[s], (g / kPStages) & 1, abort_flag, 53)) { alive = false; break; }
                    tcgen05_fence_after();
                    const uint32_t base = smem_u32(tiles + s * kPStageBytes);
                    const uint64_t a_desc = smem_desc_sw128(base);
                    const uint64_t b_desc = p.w_transposed ? smem_desc_sw128(base + kPABytes) : smem_desc_sw128(base + kPABytes, kTileBytes);
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++)
                        umma_f16_pair(tmem + buf * kGBN, a_desc + 2 * kk, b_desc + b_step * kk, idesc, (kb | kk) ? 1u : 0u);
                    umma_commit_pair(&st->empty[s]);
                }
                if (!alive) break;
                umma_commit_pair(&st->acc_full[buf]);
            }
        }
    } else {
        // ===== epilogue (both CTAs): this CTA's 128 rows of the tile; a warp takes 32 rows and 128 columns and stores them
        // through its own staging tile =====
        const uint32_t quarter = warp & 3;
        const uint32_t chalf = (warp - 2) >> 2;
        const uint32_t lane_field = (quarter * 32) << 16;
        const uint32_t acc_empty0[2] = {mapa_rank(smem_u32(&st->acc_empty[0]), 0), mapa_rank(smem_u32(&st->acc_empty[1]), 0)};
        uint32_t i = 0, tm, tn;
        tile_coords(p, pair, tm, tn);
        float4 next = fetch_bias(p, tn * kGBN + chalf * 128, lane);
        for (uint32_t t = pair; t < n_tiles; t += pairs, i++) {
            const uint32_t buf = i & 1;
            const uint32_t n0 = tn * kGBN + chalf * 128;
            const uint32_t m0 = tm * 256 + rank * kGBM;
            float *bias = bias_s + (buf * 2 + chalf) * 128;
            if (!mbar_wait_warp(&st->acc_full[buf], (i >> 1) & 1, abort_flag, 54)) break;
            *(float4 *)(bias + lane * 4) = next;
            __syncwarp();
            if (t + pairs < n_tiles) {
                tile_coords(p, t + pairs, tm, tn);
                next = fetch_bias(p, tn * kGBN + chalf * 128, lane);
            }
            tcgen05_fence_after();
            drain_rows_staged(p, &omap, tmem + buf * kGBN + chalf * 128 + lane_field, staging + (warp - 2) * 4096, bias, m0 + quarter * 32, n0, lane);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(buf ? acc_empty0[1] : acc_empty0[0]);
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the last tile has left shared memory
    }

    // ---- teardown (also the way out after a timeout) ----
    tcgen05_fence_before();
    __syncthreads();
    if (st->abort_flag) {
        if (warp == 1 && lane == 0 && rank == 0) {
            asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&st->drained)) : "memory");
            for (uint32_t k = 0; k < kWaitLimit && !mbar_try_wait(&st->drained, 0); k++) {}
        }
        if (warp == 0 && lane == 0) {
            const uint64_t t0 = clock64();
            while (clock64() - t0 < 2000000ull) {}
        }
        __syncthreads();
    }
    cluster_sync_all();      // neither CTA leaves, nor frees its TMEM, while the other may still read its shared memory or signal it
    if (warp == 0) {
        __syncwarp();
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- few tiles: the contraction split over a cluster -------------------------------------------------------------
// With fewer 128 x 256 tiles than SMs the kernels above leave most of the chip idle, and the tiles that do run walk the
// whole of k one after another (m = 320, n = 768, k = 3072: 9 CTAs, 20 us).  Here a tile is 128 x BN and a cluster of
// `split` CTAs shares it, each multiplying its share of the k-blocks; the fp32 accumulators meet in distributed shared
// memory: every CTA leaves its own in shared memory, and after the cluster's barrier each adds up its share of the
// rows from all of them, rank 0 first (the sum does not depend on timing), applies bias and activation and stores.
// One tile per CTA and deep stages: with few CTAs pulling through L2 the distance to it is what a k-block waits for.
// Measured, launches in sequence: m 320, n 768, k 3072 17.7 -> 8.6 us (two CTAs per 128 x 64 tile), m 320, n 768, k 768
// 8.4 -> 4.9 us (128 x 64), m 2048, n 768, k 3072 20.6 -> 14.0 us (128 x 128).
template <int BN, int ST> struct SCfg {
    static constexpr uint32_t stages = ST;
    static constexpr uint32_t stage_bytes = kGABytes + kGBK * BN * 2;
    static constexpr uint32_t acc_stride = BN + 4;                                  // floats
    static constexpr uint32_t acc_bytes = kGBM * acc_stride * 4;
    static constexpr uint32_t body = stages * stage_bytes > acc_bytes ? stages * stage_bytes : acc_bytes;
    static constexpr size_t smem = 1024 + body + BN * 4 + 256;
};
struct SShared {
    uint64_t full[8], empty[8], acc_full, drained;
    uint32_t tmem_base, abort_flag;
};
static_assert(sizeof(SShared) <= 256, "SShared outgrew its slot");

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
    return v;
}

// eight neighbouring outputs of one row: bias, activation, one 16-byte store
__device__ __forceinline__ void finish8(const GParams &p, float (&x)[8], const float *bias, const uint4 &resid, uint32_t row, uint32_t col)
{
    if (p.bias) {
        const float4 b0 = *(const float4 *)bias, b1 = *(const float4 *)(bias + 4);
        x[0] += b0.x; x[1] += b0.y; x[2] += b0.z; x[3] += b0.w;
        x[4] += b1.x; x[5] += b1.y; x[6] += b1.z; x[7] += b1.w;
    }
    if (p.act == 1) {
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = gelu_ref(x[j]);
    }
    uint32_t w[4];
    if (p.resid) {
        // the product is rounded to its type before the sum, as two separate operations do
        const uint32_t r[4] = {resid.x, resid.y, resid.z, resid.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t y = pack2(x[2 * j], x[2 * j + 1], p.is_bf16);
            const float2 a = unpack2(y, p.is_bf16), b = unpack2(r[j], p.is_bf16);
            x[2 * j] = a.x + b.x;
            x[2 * j + 1] = a.y + b.y;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = pack2(x[2 * j], x[2 * j + 1], p.is_bf16);
    *(uint4 *)((uint16_t *)p.out + (size_t)row * p.N + col) = make_uint4(w[0], w[1], w[2], w[3]);
}

template <int BN, int ST>
__global__ void __launch_bounds__(256, 1)
linear_tc_split_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap, const GParams p, const uint32_t split)
{
    typedef SCfg<BN, ST> Cfg;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float *bias_s = (float *)(smem + Cfg::body);           // the tile's bias: a read from L2 per column group would be on the critical path
    SShared *st = (SShared *)(smem + Cfg::body + BN * 4);
    float *acc_s = (float *)smem;                          // the accumulator's place once the stages are spent

    const uint32_t warp = uniform_warp(), lane = threadIdx.x & 31;
    volatile uint32_t *abort_flag = &st->abort_flag;
    const uint32_t fmt = p.is_bf16 ? 1u : 0u;
    const uint32_t tile = blockIdx.x / split, rank = blockIdx.x - tile * split;    // the cluster is `split` neighbouring CTAs
    const uint32_t tm = tile % p.tiles_m, tn = tile / p.tiles_m;
    const uint32_t kblocks = (p.K + kGBK - 1) / kGBK;
    const uint32_t kb0 = kblocks * rank / split, kb1 = kblocks * (rank + 1) / split;   // split <= kblocks: never empty

    if (threadIdx.x == 0) {
        prefetch_map(amap);
        prefetch_map(bmap);
        for (uint32_t s = 0; s < ST; s++) { mbar_init(&st->full[s], 1); mbar_init(&st->empty[s], 1); }
        mbar_init(&st->acc_full, 1);
        mbar_init(&st->drained, 1);
        st->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&st->tmem_base)), "r"((uint32_t)BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = st->tmem_base;
    grid_dependency_wait();
    grid_launch_dependents();

    if (warp == 0) {
        if (elect_one()) {
            for (uint32_t kb = kb0; kb < kb1; kb++) {
                const uint32_t g = kb - kb0, s = g % ST;
                if (g >= ST && !mbar_wait(&st->empty[s], ((g / ST) - 1) & 1, abort_flag, 61)) break;
                const uint32_t base = smem_u32(smem + s * Cfg::stage_bytes);
                mbar_expect_tx(&st->full[s], Cfg::stage_bytes);       // boxes beyond the tensor arrive as zeros and still count
                tma_load_2d(base, &amap, &st->full[s], (int32_t)(kb * kGBK), (int32_t)(tm * kGBM));
                if (p.w_transposed) {
                    tma_load_2d(base + kGABytes, &bmap, &st->full[s], (int32_t)(kb * kGBK), (int32_t)(tn * BN));
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < BN / 64; j++)
                        tma_load_2d(base + kGABytes + j * kTileBytes, &bmap, &st->full[s], (int32_t)(tn * BN + j * 64), (int32_t)(kb * kGBK));
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = instr_desc(fmt, fmt, kGBM, BN, p.w_transposed ? 0 : 1);
            const uint32_t b_step = p.w_transposed ? 2u : 128u;
            bool alive = true;
            for (uint32_t kb = kb0; kb < kb1; kb++) {
                const uint32_t g = kb - kb0, s = g % ST;
                if (!mbar_wait(&st->full[s], (g / ST) & 1, abort_flag, 62)) { alive = false; break; }
                tcgen05_fence_after();
                const uint32_t base = smem_u32(smem + s * Cfg::stage_bytes);
                const uint64_t a_desc = smem_desc_sw128(base);
                const uint64_t b_desc = p.w_transposed ? smem_desc_sw128(base + kGABytes) : smem_desc_sw128(base + kGABytes, kTileBytes);
#pragma unroll
                for (uint32_t kk = 0; kk < 4; kk++) umma_f16(tmem, a_desc + 2 * kk, b_desc + b_step * kk, idesc, (g | kk) ? 1u : 0u);
                umma_commit(&st->empty[s]);
            }
            if (alive) umma_commit(&st->acc_full);
        }
    }
    else if (warp == 2 && p.bias) {
        for (uint32_t c = lane; c < BN; c += 32) bias_s[c] = tn * BN + c < p.N ? __ldg(p.bias + tn * BN + c) : 0.f;
    }
    __syncwarp();
    // ===== all eight warps drain the accumulator: 32 rows and half of the columns each =====
    const uint32_t quarter = warp & 3, ch = warp >> 2, r = quarter * 32 + lane, lane_field = (quarter * 32) << 16;
    uint4 res[BN / 16];                                    // this thread's residuals, on their way while the products run
    if (p.resid && split == 1) {
        const uint32_t row = tm * kGBM + r;
#pragma unroll
        for (uint32_t q = 0; q < BN / 16; q++) {
            const uint32_t col = tn * BN + ch * (BN / 2) + q * 8;
            if (row < p.M && col < p.N) res[q] = *(const uint4 *)((const uint16_t *)p.resid + (size_t)row * p.N + col);
        }
    }
    const bool ok = mbar_wait_warp(&st->acc_full, 0, abort_flag, 63);
    __syncthreads();                                       // the bias is in place
    if (ok) {
        tcgen05_fence_after();
#pragma unroll
        for (uint32_t c0 = 0; c0 < BN / 2; c0 += 32) {
            const uint32_t c = ch * (BN / 2) + c0;
            uint32_t v[32];
            TMEM_LD_32((v), tmem + c + lane_field);
            tmem_wait_ld();
            if (split == 1) {
                const uint32_t row = tm * kGBM + r;
#pragma unroll
                for (uint32_t q = 0; q < 4; q++) {
                    const uint32_t col = tn * BN + c + q * 8;
                    if (row < p.M && col < p.N) {
                        float x[8];
#pragma unroll
                        for (int j = 0; j < 8; j++) x[j] = __uint_as_float(v[q * 8 + j]);
                        finish8(p, x, bias_s + c + q * 8, res[c0 / 8 + q], row, col);
                    }
                }
            } else {
                float4 *d = (float4 *)(acc_s + r * Cfg::acc_stride + c);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    d[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
            }
        }
        tcgen05_fence_before();
    }
    if (split > 1) {
        // every CTA of the cluster reaches both barriers, also after a timeout (the status word then says that the sums are not to be used)
        cluster_sync_all();
        const uint32_t rows = kGBM / split, first = rank * rows;      // split is 2 or 4
        const uint32_t mine = smem_u32(acc_s);
        constexpr uint32_t PIECES = BN / 8;
        for (uint32_t t = threadIdx.x; t < rows * PIECES; t += 256) {
            const uint32_t rr = first + t / PIECES, c = (t % PIECES) * 8;
            const uint32_t row = tm * kGBM + rr, col = tn * BN + c;
            if (row >= p.M || col >= p.N) continue;
            const uint32_t at = mine + (rr * Cfg::acc_stride + c) * 4;
            uint4 rs = make_uint4(0u, 0u, 0u, 0u);
            if (p.resid) rs = *(const uint4 *)((const uint16_t *)p.resid + (size_t)row * p.N + col);
            float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (uint32_t k = 0; k < split; k++) {
                const uint32_t a = mapa_rank(at, k);
                const float4 u = ld_cluster_f4(a), w = ld_cluster_f4(a + 16);
                x[0] += u.x; x[1] += u.y; x[2] += u.z; x[3] += u.w;
                x[4] += w.x; x[5] += w.y; x[6] += w.z; x[7] += w.w;
            }
            finish8(p, x, bias_s + c, rs, row, col);
        }
        __syncwarp();
        cluster_sync_all();                                           // the others have read this CTA's accumulator
    }

    // ---- teardown (also the way out after a timeout) ----
    __syncthreads();
    if (st->abort_flag) {
        if (warp == 1 && lane == 0) {
            umma_commit(&st->drained);
            for (uint32_t k = 0; k < kWaitLimit && !mbar_try_wait(&st->drained, 0); k++) {}
        }
        if (warp == 0 && lane == 0) {
            const uint64_t t0 = clock64();
            while (clock64() - t0 < 2000000ull) {}
        }
        __syncthreads();
    }
    if (warp == 0) {
        __syncwarp();
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN) : "memory");
    }
}

}  // namespace tc

// *refused: the device or partition cannot place the clusters, nothing was launched
template <int BN, int ST>
static int launch_split(cudaStream_t s, const CUtensorMap &am, const void *w, const tc::GParams &g, uint32_t split, int dev, bool *refused)
{
    using namespace tc;
    static DeviceOnce once;
    if (!once.done(dev)) {
        if (cudaFuncSetAttribute(linear_tc_split_kernel<BN, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCfg<BN, ST>::smem) != cudaSuccess)
            return fail("sfb_linear: cannot reserve %zu bytes of shared memory", SCfg<BN, ST>::smem);
        once.mark(dev);
    }
    CUtensorMap bm;
    if (g.w_transposed ? make_map_2d(&bm, w, g.N, g.K, g.is_bf16, BN) : make_map_2d(&bm, w, g.K, g.N, g.is_bf16, kGBK)) return 1;
    GParams prm = g;
    prm.tiles_m = (g.M + kGBM - 1) / kGBM;
    prm.tiles_n = (g.N + BN - 1) / BN;
    const cudaError_t e = launch_overlapped_cluster(linear_tc_split_kernel<BN, ST>, dim3(prm.tiles_m * prm.tiles_n * split), dim3(256),
                                                    SCfg<BN, ST>::smem, s, split, am, bm, prm, split);
    *refused = split > 1 && e != cudaSuccess;
    if (*refused) { (void)cudaGetLastError(); return 0; }
    return check_launch("sfb_linear");
}

// Which kernel and which tile: the one with the least estimated time, in microseconds.  Each estimate is a fixed part (the
// hand-over from the kernel before, the first load, the last tile's epilogue) plus the k-blocks of 64 that a CTA walks
// one after another, times what one costs -- which grows with the share of the SMs that pull operands through L2.
// Fitted to 36 shapes (m 64-32768, n 256-4096, k 256-4096, bf16, launches in sequence); within 8 % of all of them, and
// the shape's fastest variant or one within 4 % of it is the one taken:
//   128 x 64 and 128 x 128 tiles, one per CTA, only while all of them run at once: 2.7 + 0.165 and 3.7 + 0.175 per
//     k-block; sharing a tile between 2 (4) CTAs costs 1.9 (2.2) more, and clusters of four are only placed at once in a
//     third of the SMs (with twice as many CTAs they took two rounds);
//   128 x 256 tiles, persistent: 5.0 + 0.25 per k-block and round;  256 x 256 tiles on CTA pairs: 5.4 + 0.27.
struct LinearPlan {
    int kind;                  // 0: 128 x 256, 1: CTA pairs, 2: one tile per cluster
    uint32_t bn, split;
};
static LinearPlan plan_linear(uint32_t m, uint32_t n, uint32_t k, uint32_t sms)
{
    using namespace tc;
    const uint32_t kb = (k + kGBK - 1) / kGBK, tiles_m = (m + kGBM - 1) / kGBM, tiles_n = (n + kGBN - 1) / kGBN;
    auto waves = [&](uint64_t tiles, uint32_t slots, double fixed, double per, double load) {
        const uint64_t rounds = (tiles + slots - 1) / slots;
        const double share = tiles < slots ? (double)tiles / slots : 1.0;
        return fixed + (double)kb * (double)rounds * (per + load * share);
    };
    LinearPlan best = {0, kGBN, 1};
    double t_best = waves((uint64_t)tiles_m * tiles_n, sms, 5.0, 0.25, 0.13);
    if (kUsePairs && sms >= 2) {
        const double t = waves((uint64_t)((m + 255) / 256) * tiles_n, sms / 2, 5.4, 0.27, 0.09);
        if (t < t_best) { t_best = t; best = {1, kGBN, 1}; }
    }
    for (uint32_t bn = 64; bn <= 128; bn += 64) {
        const uint64_t tiles = (uint64_t)tiles_m * ((n + bn - 1) / bn);
        for (uint32_t split = 1; split <= 4 && split <= kb; split *= 2) {
            const uint64_t ctas = tiles * split;
            if (ctas > (split == 4 ? sms / 3 : sms)) break;
            const double t = (bn == 64 ? 2.7 : 3.7) + (split == 1 ? 0.0 : split == 2 ? 1.9 : 2.2) +
                             (double)((kb + split - 1) / split) * ((bn == 64 ? 0.165 : 0.175) + 0.04 * (double)ctas / sms);
            if (t < t_best) { t_best = t; best = {2, bn, split}; }
        }
    }
    return best;
}

// out += resid, 16 bytes per thread and step (what the kernels with large tiles leave to a pass of its own: read beside the
// accumulator, a row's residuals cost their epilogues more than the pass does)
template <bool BF16>
__global__ void __launch_bounds__(256) add_residual_kernel(void *out, const void *resid, size_t pieces)
{
    grid_dependency_wait();
    grid_launch_dependents();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < pieces; i += (size_t)gridDim.x * blockDim.x) {
        const uint4 a = ((const uint4 *)out)[i], b = ((const uint4 *)resid)[i];
        const uint32_t u[4] = {a.x, a.y, a.z, a.w}, v[4] = {b.x, b.y, b.z, b.w};
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = tc::unpack2(u[j], BF16), g = tc::unpack2(v[j], BF16);
            w[j] = tc::pack2(f.x + g.x, f.y + g.y, BF16);
        }
        ((uint4 *)out)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

static int linear_product(cudaStream_t s, void *out, const void *x, const void *w, const float *bias, uint32_t m, uint32_t n, uint32_t k,
                          int dtype, int act, bool w_transposed, const void *resid, bool *added)
{
    using namespace tc;
    const int is_bf16 = dtype == SFB_BF16;
    CUtensorMap am, bm;
    if (make_map_2d(&am, x, m, k, is_bf16, kGBM)) return 1;
    const int dev = current_device();
    const int sms = device_sm_count(dev);
    if (sms <= 0) return fail("sfb_linear: cannot read the SM count");
    const LinearPlan plan = plan_linear(m, n, k, (uint32_t)sms);
    const uint32_t tiles_n = (n + kGBN - 1) / kGBN;
    GParams prm = {out, bias, m, n, k, 0, tiles_n, is_bf16, act, w_transposed ? 1 : 0, 1, nullptr};
    // a device or a partition that cannot place clusters refuses their launch: the single-CTA kernel at the end takes over
    if (plan.kind == 2) {
        GParams few = prm;
        few.resid = resid;
        bool refused = false;
        const int rc = plan.bn == 64 ? launch_split<64, 8>(s, am, w, few, plan.split, dev, &refused) : launch_split<128, 6>(s, am, w, few, plan.split, dev, &refused);
        if (!refused) { *added = true; return rc; }
    }
    if (plan.kind == 1) {
        CUtensorMap bp;
        if (w_transposed ? make_map_2d(&bp, w, n, k, is_bf16, kGBN / 2) : make_map_2d(&bp, w, k, n, is_bf16, kGBK)) return 1;
        static DeviceOnce once_pair;
        if (!once_pair.done(dev)) {
            if (cudaFuncSetAttribute(linear_tc_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPSmem) != cudaSuccess)
                return fail("sfb_linear: cannot reserve %zu bytes of shared memory", kPSmem);
            once_pair.mark(dev);
        }
        CUtensorMap om;      // out as [m, n], boxes of 32 rows x 64 columns for the epilogue's stores
        if (make_map_2d(&om, out, m, n, is_bf16, 32)) return 1;
        prm.tiles_m = (m + 255) / 256;
        prm.band = tiles_n < kPBand ? tiles_n : kPBand;
        const uint64_t pair_tiles = (uint64_t)prm.tiles_m * tiles_n;
        const uint32_t pairs = pair_tiles < (uint64_t)(sms / 2) ? (uint32_t)pair_tiles : (uint32_t)(sms / 2);
        if (launch_overlapped(linear_tc_pair_kernel, dim3(2 * pairs), dim3(320), kPSmem, s, am, bp, om, prm) == cudaSuccess)
            return check_launch("sfb_linear");
        (void)cudaGetLastError();
    }
    if (w_transposed ? make_map_2d(&bm, w, n, k, is_bf16, kGBN) : make_map_2d(&bm, w, k, n, is_bf16, kGBK)) return 1;
    static DeviceOnce once;
    if (!once.done(dev)) {
        if (cudaFuncSetAttribute(linear_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGSmem) != cudaSuccess)
            return fail("sfb_linear: cannot reserve %zu bytes of shared memory", kGSmem);
        once.mark(dev);
    }
    prm.tiles_m = (m + kGBM - 1) / kGBM;
    prm.band = 1;
    const uint64_t tiles = (uint64_t)prm.tiles_m * prm.tiles_n;
    const uint32_t grid = tiles < (uint64_t)sms ? (uint32_t)tiles : (uint32_t)sms;
    launch_overlapped(linear_tc_kernel, dim3(grid), dim3(320), kGSmem, s, am, bm, prm);
    return check_launch("sfb_linear");
}

int tc_linear(cudaStream_t s, void *out, const void *x, const void *w, const float *bias, uint32_t m, uint32_t n, uint32_t k,
              int dtype, int act, bool w_transposed, const void *resid)
{
    bool added = false;
    if (linear_product(s, out, x, w, bias, m, n, k, dtype, act, w_transposed, resid, &added)) return 1;
    if (!resid || added) return 0;
    const size_t pieces = (size_t)m * n / 8;                            // n is a multiple of 16
    const int sms = device_sm_count(current_device());
    const size_t want = (pieces + 255) / 256, most = (size_t)(sms > 0 ? sms : 1) * 16;
    const dim3 grid((unsigned)(want < most ? want : most));
    if (dtype == SFB_BF16) launch_overlapped(add_residual_kernel<true>, grid, dim3(256), 0, s, out, resid, pieces);
    else launch_overlapped(add_residual_kernel<false>, grid, dim3(256), 0, s, out, resid, pieces);
    return check_launch("sfb_linear_residual");
}

int tc_status_clear_gemm()
{
    const uint32_t zero = 0;
    cudaError_t e = cudaMemcpyToSymbol(tc::g_status, &zero, sizeof(uint32_t));
    if (e != cudaSuccess) return fail("sfb_device_status_clear: %s", cudaGetErrorString(e));
    return 0;
}

int tc_status_gemm(uint32_t *out)
{
    cudaError_t e = cudaMemcpyFromSymbol(out, tc::g_status, sizeof(uint32_t));
    if (e != cudaSuccess) return fail("sfb_device_status: %s", cudaGetErrorString(e));
    return 0;
}

}  // namespace sfb
