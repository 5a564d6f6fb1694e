// Backward of the block-sparse attention on the tensor cores (tcgen05) for 16-bit operands, block_size 64, head size 64,
// from the saved probabilities P and the forward output O:
//   delta = rowsum(dO * O),  dS = P * (dO.V^T - delta) * scale,  dQ = dS.K,  dK = dS^T.Q,  dV = P^T.dO
// (the call order of transformer_attention_optimize.cu:924-964).  As separate operators this moves the block tensors five
// times (P in for dV and for dS, dS out, dS in for dK and for dQ); here dS never leaves the SM: one kernel walks pairs of
// block-rows and makes dQ, one walks pairs of block-columns and makes dK and dV, and each recomputes dS from its own read
// of P -- a product of tensor work per block, which is free next to 8 KB of P.  The row kernel also makes delta.
//
// Both are the same kernel, seen from the two sides (COL).  An item is 128 "own" positions (queries of two block-rows, or
// keys of two block-columns) of one (batch, head), and a walk over the union of their blocks; per step
//     dP  = X . Y^T           X: own rows of dO (V), an A operand that waits in TMEM; Y: the step's rows of V (dO), by TMA
//     dS  = P * (dP - delta)  256 threads, one own position and 32 of the 64 others each; dS goes back to TMEM, 16 bits
//     out += dS . Z           Z: the step's rows of K (Q)                              -> dQ (dK)
//     COL: dV += P^T . Y      the two blocks of P as one MN-major A operand
// A block that only one of the two rows (columns) keeps is fetched from beyond the tensor and arrives as zeros.
//
// Two CTAs per SM.  A CTA starts with the item of its own index and then takes over items that have not been started
// (cluster launch control: the grid is the items, and a running CTA cancels the launch of one and does its work), so that
// long rows and columns do not pile up on a few CTAs.  Everything an item needs before its first step is fetched under the
// item before it: the union by the planner warp, X and O as a stage of their own ahead of the item's first step.  With one
// item per CTA those dependent reads took 16 of every 38 thousand cycles, on a memory system busy with P; read by the
// threads themselves (16 bytes per row and lane) X and O still cost 9 thousand per item.
// The column kernel needs P transposed: it works on TMEM in fragment order (16x256b), so that one transposed ldmatrix
// brings eight probabilities per lane, where one key per lane meant 32 two-byte loads with their conflicts (1500 of 2600
// cycles per step).
// Warps: 0-7 dS and the epilogue, 8 TMA, 9 issues dP (and dV), 10 issues out, 11 plans.  Two issuing warps because each
// satisfied barrier wait costs its thread 250 cycles on a loaded SM: one thread's four waits per step were the step.
// TMEM (256 columns): dP 64, dS 32 (packed), X 32, the accumulators 64 + 64.  dP has one buffer: it is free again as soon as
// its values are in registers, so the next step's product runs under this step's arithmetic.
#include "tc_common.cuh"

namespace sfb {
namespace tc {

constexpr uint32_t kBwStages = 3;
constexpr uint32_t kBwStageBytes = 4 * kTileBytes;              // two blocks of P, Y, Z
constexpr uint32_t kBwThreads = 12 * 32;
constexpr uint32_t kBwMaxUnion = 256;

struct BwShared {
    uint64_t in_full[kBwStages], in_empty[kBwStages], x_ready, s_full, s_free, ds_full, ds_free, o_final, o_free;
    uint64_t list_ready[2], list_free[2], clc_bar, drained[2];
    alignas(16) uint32_t clc_response[4];
    uint32_t tmem_base, abort_flag, list_n[2], list_bh[2], list_own[2][2];      // list_own: the two rows (columns)
    alignas(16) float delta[kBwStages][64];                      // COL: the step's deltas
    float comb[2][2][128];                                       // rows: the halves of delta, of two items in turn
    UnionEntry lists[2][kBwMaxUnion];
};
constexpr size_t kBwSmem = 1024 + kBwStages * kBwStageBytes + sizeof(BwShared);
static_assert(2 * (kBwSmem + 1024) <= 228 * 1024, "two CTAs per SM");

struct BwParams {
    const uint2 *lut;          // nn_lut (rows) or tn_lut (columns)
    float *delta;              // [B, H, L] -scale * rowsum(dO * O): written by the row kernel, read by the column kernel
    void *out1, *out2;         // dQ, - or dK, dV
    uint32_t B, H, nb, blocks, lut_stride, p_rows;
    float scale;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(smem_u32(bar))
                 : "memory");
}

// 16 lanes x 32 fp32 columns of TMEM in fragment order: v[4 i + 0, 1] are lane t / 4, columns 8 i + 2 (t % 4) + {0, 1},
// v[4 i + 2, 3] the same columns of lane t / 4 + 8
#define TMEM_LD_FRAG(v, addr)                                                                                           \
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];" \
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),       \
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])   \
                 : "r"(addr)                                                                                             \
                 : "memory")
// 16 lanes x 16 words: w[2 i] is word 4 i + t % 4 of lane t / 4, w[2 i + 1] the same word of lane t / 4 + 8
#define TMEM_ST_FRAG(addr, w)                                                                                            \
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), \
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])                                                     \
                 : "memory")
// four 8 x 8 matrices of 16-bit elements, transposed: r[m] holds elements (2 (t % 4) + {0, 1}, t / 4) of matrix m, whose row
// i starts at the address that lane 8 m + i gives
__device__ __forceinline__ void ldmatrix_trans(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// P * (dP * scale + delta) for a pair, rounded to the 16-bit type
template <bool BF16>
__device__ __forceinline__ uint32_t ds_pair(uint32_t v0, uint32_t v1, uint32_t p_bits, uint64_t scale2, uint64_t delta2)
{
    const float2 pv = unpack2(p_bits, BF16);
    const uint64_t x = fma2p(pk64(__uint_as_float(v0), __uint_as_float(v1)), scale2, delta2);
    float e0, e1;
    up64(mul2p(x, pk64(pv.x, pv.y)), e0, e1);
    return pack2(e0, e1, BF16);
}

template <bool COL, bool BF16>
__global__ void __launch_bounds__(kBwThreads, 2)
backward_tc_kernel(const __grid_constant__ CUtensorMap pmap, const __grid_constant__ CUtensorMap ymap, const __grid_constant__ CUtensorMap zmap,
                   const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap omap, const BwParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    BwShared *st = (BwShared *)(smem + kBwStages * kBwStageBytes);

    const uint32_t warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t L = p.nb * 64;
    volatile uint32_t *abort_flag = &st->abort_flag;
    const uint32_t fmt = BF16 ? 1u : 0u;

    if (threadIdx.x == 0) {
        prefetch_map(pmap);
        prefetch_map(ymap);
        prefetch_map(zmap);
        prefetch_map(xmap);
        if (!COL) prefetch_map(omap);
        for (uint32_t s = 0; s < kBwStages; s++) { mbar_init(&st->in_full[s], 1); mbar_init(&st->in_empty[s], COL ? 2 : 1); }
        mbar_init(&st->x_ready, 8);
        mbar_init(&st->s_full, 1);
        mbar_init(&st->s_free, 8);
        mbar_init(&st->ds_full, 8);
        mbar_init(&st->ds_free, 1);
        mbar_init(&st->o_final, COL ? 2 : 1);
        mbar_init(&st->o_free, 8);
        for (int i = 0; i < 2; i++) {
            mbar_init(&st->list_ready[i], 1);
            mbar_init(&st->list_free[i], 11);      // TMA, two issuers, eight dS warps
            mbar_init(&st->drained[i], 1);
        }
        mbar_init(&st->clc_bar, 1);
        st->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&st->tmem_base)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = st->tmem_base;
    const uint32_t t_s = tmem, t_ds = tmem + 64, t_x = tmem + 96, t_o1 = tmem + 128, t_o2 = tmem + 192;
    grid_dependency_wait();
    grid_launch_dependents();

    if (warp == 11) {
        // ===== planner: the coming items and their unions, up to two ahead =====
        uint32_t id = blockIdx.x;
        const uint32_t first_pairs = p.lut_stride == 0 ? long_pairs(p.lut, p.nb, p.blocks, lane) : 0;
        for (uint32_t k = 0;; k++) {
            const uint32_t slot = k & 1;
            if (id != kNoItem && lane == 0) {
                fence_proxy_async();                          // the last answer has been read
                clc_request(st->clc_response, &st->clc_bar);
            }
            if (k >= 2 && !mbar_wait_warp(&st->list_free[slot], ((k >> 1) - 1) & 1, abort_flag, 70)) break;
            uint32_t n = 0, bh = kNoItem, own[2] = {kNoItem, kNoItem};
            if (id != kNoItem) {
                // head by head as the product before this call walks P; the row kernel backwards, the column kernel forwards again,
                // so that each starts with the blocks the kernel before it left in L2
                const ItemAt it = locate_item(p.lut, p.lut_stride, p.B, p.H, p.nb, p.blocks, first_pairs, id, lane, !COL);
                bh = it.b * p.H + it.h;
                own[0] = it.own[0];
                own[1] = it.own[1];
                n = warp_union(p.lut + (size_t)it.h * p.lut_stride, own, st->lists[slot], kBwMaxUnion, lane);
                if (n == kNoItem) {                           // more blocks than the caller's maximum: recorded, zeros written
                    if (lane == 0) atomicCAS(&g_status, 0u, (9u << 24) | (blockIdx.x & 0xffffffu));
                    n = 0;
                }
            }
            if (lane == 0) {
                st->list_n[slot] = n;
                st->list_bh[slot] = bh;
                st->list_own[slot][0] = own[0];
                st->list_own[slot][1] = own[1];
                mbar_arrive(&st->list_ready[slot]);
            }
            if (id == kNoItem) break;
            if (!mbar_wait_warp(&st->clc_bar, k & 1, abort_flag, 69)) break;
            id = clc_item(st->clc_response);
            __syncwarp();
        }
    } else if (warp == 8) {
        // ===== TMA producer =====
        if (elect_one()) {
            uint32_t g = 0;                                   // stages so far, over all items: X and O, then the steps
            bool alive = true;
            for (uint32_t k = 0; alive; k++) {
                const uint32_t slot = k & 1;
                if (!mbar_wait(&st->list_ready[slot], (k >> 1) & 1, abort_flag, 68)) break;
                const uint32_t bh = st->list_bh[slot], T = st->list_n[slot];
                if (bh == kNoItem) break;
                const uint32_t b = bh / p.H, h = bh - b * p.H;
                const int32_t x = (int32_t)(h * 64), row0 = (int32_t)(b * L), beyond = (int32_t)(p.B * L);
                const uint32_t bh_rows = bh * p.blocks * 64;  // first row of this (b,h) in the 2-D view of P
                for (uint32_t t = 0; T > 0 && t <= T; t++, g++) {
                    const uint32_t s = g % kBwStages;
                    if (g >= kBwStages && !mbar_wait(&st->in_empty[s], ((g / kBwStages) - 1) & 1, abort_flag, 71)) { alive = false; break; }
                    const uint32_t base = smem_u32(smem + s * kBwStageBytes);
                    if (t == 0) {
                        mbar_expect_tx(&st->in_full[s], (COL ? 2 : 4) * kTileBytes);
#pragma unroll
                        for (uint32_t o = 0; o < 2; o++) {
                            const int32_t y = st->list_own[slot][o] == kNoItem ? beyond : row0 + (int32_t)(st->list_own[slot][o] * 64);
                            tma_load_2d(base + o * kTileBytes, &xmap, &st->in_full[s], x, y);
                            if (!COL) tma_load_2d(base + (2 + o) * kTileBytes, &omap, &st->in_full[s], x, y);
                        }
                        continue;
                    }
                    const UnionEntry ent = st->lists[slot][t - 1];
                    mbar_expect_tx(&st->in_full[s], kBwStageBytes + (COL ? 256 : 0));
                    const int32_t y0 = (ent.flags & 1) ? (int32_t)(bh_rows + ent.blk[0] * 64) : (int32_t)p.p_rows;
                    const int32_t y1 = (ent.flags & 2) ? (int32_t)(bh_rows + ent.blk[1] * 64) : (int32_t)p.p_rows;
                    tma_load_2d(base, &pmap, &st->in_full[s], 0, y0);
                    tma_load_2d(base + kTileBytes, &pmap, &st->in_full[s], 0, y1);
                    tma_load_2d(base + 2 * kTileBytes, &ymap, &st->in_full[s], x, row0 + (int32_t)(ent.col * 64));
                    tma_load_2d(base + 3 * kTileBytes, &zmap, &st->in_full[s], x, row0 + (int32_t)(ent.col * 64));
                    if (COL) bulk_load(smem_u32(st->delta[s]), p.delta + (size_t)bh * L + (size_t)ent.col * 64, 256, &st->in_full[s]);
                }
                if (alive) mbar_arrive(&st->list_free[slot]);
            }
        }
    } else if (warp == 9) {
        // ===== dP = X . Y^T (and dV += P^T . Y) =====
        if (elect_one()) {
            const uint32_t idesc_dp = instr_desc(fmt, fmt, 128, 64, 0);                 // Y rows along N, K-major
            const uint32_t idesc_dv = instr_desc(fmt, fmt, 128, 64, 1) | (1u << 15);    // P transposed: A MN-major; Y rows along K
            uint32_t gs = 0, g = 0, kq = 0;                   // stages, steps, items with blocks
            bool alive = true;
            for (uint32_t k = 0; alive; k++) {
                const uint32_t slot = k & 1;
                if (!mbar_wait(&st->list_ready[slot], (k >> 1) & 1, abort_flag, 67)) break;
                const uint32_t T = st->list_n[slot];
                if (st->list_bh[slot] == kNoItem) break;
                if (T > 0) {
                    if (!mbar_wait(&st->x_ready, kq & 1, abort_flag, 72)) break;
                    mbar_arrive(&st->in_empty[gs % kBwStages]);       // X (and O) have been read out of their stage
                    if (COL) mbar_arrive(&st->in_empty[gs % kBwStages]);
                    gs++;
                }
                for (uint32_t t = 0; t < T; t++, g++, gs++) {
                    const uint32_t s = gs % kBwStages;
                    const bool ready = mbar_try_wait(&st->in_full[s], (gs / kBwStages) & 1);    // asked for together: one trip instead of two
                    if (g >= 1 && !mbar_wait(&st->s_free, (g - 1) & 1, abort_flag, 74)) { alive = false; break; }
                    if (!ready && !mbar_wait(&st->in_full[s], (gs / kBwStages) & 1, abort_flag, 73)) { alive = false; break; }
                    tcgen05_fence_after();
                    const uint32_t base = smem_u32(smem + s * kBwStageBytes);
                    const uint64_t y_desc = smem_desc_sw128(base + 2 * kTileBytes);
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) umma_f16_ts(t_s, t_x + 8 * kk, y_desc + 2 * kk, idesc_dp, kk);
                    umma_commit(&st->s_full);
                    if (COL) {
                        // the accumulator still holds the previous item's dV until its epilogue has read it
                        if (t == 0 && kq >= 1 && !mbar_wait(&st->o_free, (kq - 1) & 1, abort_flag, 66)) { alive = false; break; }
                        tcgen05_fence_after();
                        const uint64_t p_desc = smem_desc_sw128(base, kTileBytes);      // the second block is the next 64 along M
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; kk++) umma_f16(t_o2, p_desc + 128 * kk, y_desc + 128 * kk, idesc_dv, (t | kk) ? 1u : 0u);
                        umma_commit(&st->in_empty[s]);
                        if (t + 1 == T) umma_commit(&st->o_final);
                    }
                }
                if (T > 0) kq++;
                if (alive) mbar_arrive(&st->list_free[slot]);
            }
        }
    } else if (warp == 10) {
        // ===== out += dS . Z =====
        if (elect_one()) {
            const uint32_t idesc_out = instr_desc(fmt, fmt, 128, 64, 1);                // Z rows along K
            uint32_t gs = 0, g = 0, kq = 0;
            bool alive = true;
            for (uint32_t k = 0; alive; k++) {
                const uint32_t slot = k & 1;
                if (!mbar_wait(&st->list_ready[slot], (k >> 1) & 1, abort_flag, 65)) break;
                const uint32_t T = st->list_n[slot];
                if (st->list_bh[slot] == kNoItem) break;
                if (T > 0) gs++;                              // the stage of X and O
                if (T > 0 && kq >= 1 && !mbar_wait(&st->o_free, (kq - 1) & 1, abort_flag, 64)) break;
                for (uint32_t t = 0; t < T; t++, g++, gs++) {
                    const uint32_t s = gs % kBwStages;
                    if (!mbar_wait(&st->ds_full, g & 1, abort_flag, 75)) { alive = false; break; }
                    tcgen05_fence_after();
                    const uint64_t z_desc = smem_desc_sw128(smem_u32(smem + s * kBwStageBytes + 3 * kTileBytes));
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) umma_f16_ts(t_o1, t_ds + 8 * kk, z_desc + 128 * kk, idesc_out, (t | kk) ? 1u : 0u);
                    umma_commit(&st->ds_free);
                    umma_commit(&st->in_empty[s]);            // dP of this step is complete: its values made this dS
                    if (t + 1 == T) umma_commit(&st->o_final);
                }
                if (T > 0) kq++;
                if (alive) mbar_arrive(&st->list_free[slot]);
            }
        }
    } else {
        // ===== dS and the epilogue: own position r, half of the other side's 64 =====
        const uint32_t quarter = warp & 3, ch = warp >> 2;
        const uint32_t cb = ch * 32, r = quarter * 32 + lane, half = r >> 6;
        const uint32_t lane_field = (quarter * 32) << 16;
        const uint64_t scale2 = pk64(p.scale, p.scale);
        uint32_t gs = 0, g = 0, kq = 0, n_x = 0;             // stages, steps, items with blocks finished, X published
        float my_delta = 0.f, dot = 0.f;                     // rows: -scale * delta of this query; this thread's half of the sum
        // the coming item's X from its stage to TMEM (every dP of the item before is complete); rows: the sum over dO * O
        auto publish = [&]() -> bool {
            const uint32_t s = gs % kBwStages;
            if (!mbar_wait_warp(&st->in_full[s], (gs / kBwStages) & 1, abort_flag, 62)) return false;
            gs++;
            const uint8_t *xrow = smem + s * kBwStageBytes + half * kTileBytes + (r & 63) * 128;
            uint32_t w[16];
            dot = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t at = ((cb / 8 + j) ^ (r & 7)) << 4;
                const uint4 x = *(const uint4 *)(xrow + at);
                w[4 * j] = x.x; w[4 * j + 1] = x.y; w[4 * j + 2] = x.z; w[4 * j + 3] = x.w;
                if (!COL) {
                    const uint4 o = *(const uint4 *)(xrow + 2 * kTileBytes + at);
                    const uint32_t ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float2 xv = unpack2(w[4 * j + q], BF16), yv = unpack2(ov[q], BF16);
                        dot = fmaf(xv.x, yv.x, fmaf(xv.y, yv.y, dot));
                    }
                }
            }
            TMEM_ST_16(t_x + ch * 16 + lane_field, (w));
            tmem_wait_st();
            tcgen05_fence_before();
            if (!COL) st->comb[n_x & 1][ch][r] = dot;
            mbar_arrive_warp(&st->x_ready, lane);
            n_x++;
            return true;
        };

        bool alive = mbar_wait_warp(&st->list_ready[0], 0, abort_flag, 63);
        if (alive && st->list_n[0] > 0) alive = publish();
        for (uint32_t k = 0; alive; k++) {
            const uint32_t slot = k & 1;
            const uint32_t bh = st->list_bh[slot], T = st->list_n[slot];
            if (bh == kNoItem) break;
            if (!COL && T > 0) {
                // both halves of the row's sum are in place once every warp has published X
                if (!mbar_wait_warp(&st->x_ready, (n_x - 1) & 1, abort_flag, 60)) break;
                my_delta = -(dot + st->comb[(n_x - 1) & 1][ch ^ 1][r]) * p.scale;
                const uint32_t blk = st->list_own[slot][half];
                if (ch == 0 && blk != kNoItem) p.delta[(size_t)bh * L + (size_t)blk * 64 + (r & 63)] = my_delta;
            } else if (!COL) {
                // no blocks: dS is empty and dV, which alone would read it, gets nothing from this row
                const uint32_t blk = st->list_own[slot][half];
                if (ch == 0 && blk != kNoItem) p.delta[(size_t)bh * L + (size_t)blk * 64 + (r & 63)] = 0.f;
            }
            for (uint32_t t = 0; t < T; t++, g++, gs++) {
                const uint32_t s = gs % kBwStages;
                // Whether this row (column) has the step's block, the same for the whole warp (the vote says so to the compiler).
                // Where it has not, P is zeros but dP may be an infinity or NaN, and 0 times that is not 0: zeros are stored
                // instead.  A branch at the store alone: around the arithmetic it cost 2-4 % of the call, here 0.4-0.9.
                const bool mine = __any_sync(0xffffffffu, (st->lists[slot][t].flags >> half) & 1u);
                // P (and the deltas) came with the barrier the product waited for; observing it makes them visible to this thread
                const bool in_ok = mbar_try_wait(&st->in_full[s], (gs / kBwStages) & 1);
                if (!mbar_wait_warp(&st->s_full, g & 1, abort_flag, 76)) { alive = false; break; }
                tcgen05_fence_after();
                const uint8_t *tile = smem + s * kBwStageBytes + half * kTileBytes;
                bool ds_ok;
                if (COL) {
                    uint32_t v[2][16];
                    TMEM_LD_FRAG(v[0], t_s + lane_field + cb);
                    TMEM_LD_FRAG(v[1], t_s + lane_field + (16u << 16) + cb);
                    if (!__all_sync(0xffffffffu, in_ok) && !mbar_wait_warp(&st->in_full[s], (gs / kBwStages) & 1, abort_flag, 77)) { alive = false; break; }
                    ds_ok = g == 0 || mbar_try_wait(&st->ds_free, (g - 1) & 1);
                    tmem_wait_ld();
                    tcgen05_fence_before();
                    mbar_arrive_warp(&st->s_free, lane);
                    // a lane's addresses in the transposed loads: matrix lane / 8 is query group (lane / 16), key half (lane / 8) % 2
                    const uint32_t q_row = cb + ((lane >> 4) << 3) + (lane & 7), key_chunk = ((quarter & 1) << 2) + ((lane >> 3) & 1);
                    const uint32_t p_base = smem_u32(tile) + q_row * 128;
                    uint32_t w[2][8];
#pragma unroll
                    for (int kg = 0; kg < 2; kg++)
#pragma unroll
                        for (int i = 0; i < 4; i += 2) {
                            uint32_t pw[4];
                            ldmatrix_trans(pw, p_base + i * 1024 + (((key_chunk + 2 * kg) ^ (lane & 7)) << 4));
#pragma unroll
                            for (int j = 0; j < 2; j++) {
                                const uint64_t d2 = *(const uint64_t *)(st->delta[s] + cb + 8 * (i + j) + 2 * (lane & 3));
                                const uint32_t(&vv)[16] = v[kg];
                                const int e = 4 * (i + j);
                                w[kg][2 * (i + j)] = ds_pair<BF16>(vv[e], vv[e + 1], pw[2 * j], scale2, d2);
                                w[kg][2 * (i + j) + 1] = ds_pair<BF16>(vv[e + 2], vv[e + 3], pw[2 * j + 1], scale2, d2);
                            }
                        }
                    if (!__all_sync(0xffffffffu, ds_ok) && !mbar_wait_warp(&st->ds_free, (g - 1) & 1, abort_flag, 78)) { alive = false; break; }
                    tcgen05_fence_after();
                    if (mine) {
                        TMEM_ST_FRAG(t_ds + ch * 16 + lane_field, w[0]);
                        TMEM_ST_FRAG(t_ds + ch * 16 + lane_field + (16u << 16), w[1]);
                    } else {
                        const uint32_t none[8] = {};
                        TMEM_ST_FRAG(t_ds + ch * 16 + lane_field, none);
                        TMEM_ST_FRAG(t_ds + ch * 16 + lane_field + (16u << 16), none);
                    }
                } else {
                    uint32_t v[32], w[16];
                    TMEM_LD_32((v), t_s + lane_field + cb);
                    if (!__all_sync(0xffffffffu, in_ok) && !mbar_wait_warp(&st->in_full[s], (gs / kBwStages) & 1, abort_flag, 77)) { alive = false; break; }
                    ds_ok = g == 0 || mbar_try_wait(&st->ds_free, (g - 1) & 1);
                    tmem_wait_ld();
                    tcgen05_fence_before();
                    mbar_arrive_warp(&st->s_free, lane);
                    const uint8_t *prow = tile + (r & 63) * 128;
                    const uint64_t d2 = pk64(my_delta, my_delta);
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint4 u = *(const uint4 *)(prow + (((cb / 8 + c) ^ (r & 7)) << 4));
                        const uint32_t pw[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                        for (int j = 0; j < 4; j++) w[c * 4 + j] = ds_pair<BF16>(v[c * 8 + 2 * j], v[c * 8 + 2 * j + 1], pw[j], scale2, d2);
                    }
                    if (!__all_sync(0xffffffffu, ds_ok) && !mbar_wait_warp(&st->ds_free, (g - 1) & 1, abort_flag, 78)) { alive = false; break; }
                    tcgen05_fence_after();
                    if (mine) {
                        TMEM_ST_16(t_ds + ch * 16 + lane_field, (w));
                    } else {
                        const uint32_t none[16] = {};
                        TMEM_ST_16(t_ds + ch * 16 + lane_field, (none));
                    }
                }
                tmem_wait_st();
                tcgen05_fence_before();
                mbar_arrive_warp(&st->ds_full, lane);
            }
            if (!alive) break;
            // the next item's X before this item's epilogue: the issuer's next dP must not wait for it
            if (!mbar_wait_warp(&st->list_ready[slot ^ 1], ((k + 1) >> 1) & 1, abort_flag, 61)) break;
            if (st->list_n[slot ^ 1] > 0 && !publish()) break;
            if (T > 0 && !mbar_wait_warp(&st->o_final, kq & 1, abort_flag, 79)) break;
            tcgen05_fence_after();
            const uint32_t blk = st->list_own[slot][half], b = bh / p.H, h = bh - b * p.H;
            const size_t own = ((size_t)b * L + (size_t)blk * 64 + (r & 63)) * ((size_t)p.H * 64) + (size_t)h * 64 + cb;
#pragma unroll
            for (int o = 0; o < (COL ? 2 : 1); o++) {
                uint16_t *dst = (uint16_t *)(o ? p.out2 : p.out1) + own;
                uint32_t v[32];
                if (T > 0) {
                    TMEM_LD_32((v), (o ? t_o2 : t_o1) + lane_field + cb);
                    tmem_wait_ld();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = 0u;              // rows and columns without blocks have zero gradients
                }
                if (blk != kNoItem)
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        uint32_t y[8];
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            y[j] = pack2(__uint_as_float(v[16 * c + 2 * j]), __uint_as_float(v[16 * c + 2 * j + 1]), BF16);
                        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + 16 * c), "r"(y[0]), "r"(y[1]), "r"(y[2]),
                                     "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7])
                                     : "memory");
                    }
            }
            if (T > 0) {
                tcgen05_fence_before();
                mbar_arrive_warp(&st->o_free, lane);
                kq++;
            }
            mbar_arrive_warp(&st->list_free[slot], lane);
        }
    }

    // ---- teardown (also the way out after a timeout) ----
    tcgen05_fence_before();
    __syncthreads();
    if (st->abort_flag) {
        if ((warp == 9 || warp == 10) && lane == 0) {
            umma_commit(&st->drained[warp - 9]);
            for (uint32_t i = 0; i < kWaitLimit && !mbar_try_wait(&st->drained[warp - 9], 0); i++) {}
        }
        if (warp == 8 && lane == 0) {
            const uint64_t t0 = clock64();
            while (clock64() - t0 < 2000000ull) {}
        }
        __syncthreads();
    }
    if (warp == 8) {
        __syncwarp();
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
}

}  // namespace tc

bool tc_backward_supported(int dtype, uint32_t bs, const AttnDims &p, uint32_t nn_max, uint32_t tn_max, uint64_t pointers)
{
    return (dtype == SFB_BF16 || dtype == SFB_F16) && bs == 64 && p.d == 64 && p.blocks > 0 && (pointers & 31) == 0 && nn_max && tn_max &&
           (p.nb_a <= tc::kBwMaxUnion || (2 * (uint64_t)nn_max <= tc::kBwMaxUnion && 2 * (uint64_t)tn_max <= tc::kBwMaxUnion)) && (uint64_t)p.B * p.nb_a * 64 < (1ull << 31) &&
           (uint64_t)p.B * p.H * p.blocks * 64 < (1ull << 31) - 64;
}

template <bool BF16>
static int launch_backward(cudaStream_t s, const void *nn_lut, const void *tn_lut, const void *q, const void *k, const void *v, const void *pblk,
                           const void *o, const void *dout, float *delta, void *dq, void *dk, void *dv, const AttnDims &p, float scale)
{
    using namespace tc;
    const uint64_t rows = (uint64_t)p.B * p.nb_a * 64, prow = (uint64_t)p.B * p.H * p.blocks * 64;
    CUtensorMap pm, qm, km, vm, dm, om;
    if (make_map_2d(&pm, pblk, prow, 64, BF16, 64) || make_map(&qm, q, rows, p.H, BF16, 64) || make_map(&km, k, rows, p.H, BF16, 64) ||
        make_map(&vm, v, rows, p.H, BF16, 64) || make_map(&dm, dout, rows, p.H, BF16, 64) || make_map(&om, o, rows, p.H, BF16, 64))
        return 1;
    static DeviceOnce once;
    const int dev = current_device();
    if (!once.done(dev)) {
        if (cudaFuncSetAttribute(backward_tc_kernel<false, BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwSmem) != cudaSuccess ||
            cudaFuncSetAttribute(backward_tc_kernel<true, BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwSmem) != cudaSuccess)
            return fail("sfb_attention_backward: cannot reserve %zu bytes of shared memory", kBwSmem);
        once.mark(dev);
    }
    const uint32_t npairs = (p.nb_a + 1) / 2;
    const dim3 grid(npairs * p.B * p.H);
    const BwParams row = {(const uint2 *)nn_lut, delta, dq, nullptr, p.B, p.H, p.nb_a, p.blocks, p.lut_stride, (uint32_t)prow, scale};
    const BwParams col = {(const uint2 *)tn_lut, delta, dk, dv, p.B, p.H, p.nb_a, p.blocks, p.lut_stride, (uint32_t)prow, scale};
    launch_overlapped(backward_tc_kernel<false, BF16>, grid, dim3(kBwThreads), kBwSmem, s, pm, vm, km, dm, om, row);
    launch_overlapped(backward_tc_kernel<true, BF16>, grid, dim3(kBwThreads), kBwSmem, s, pm, dm, qm, vm, vm, col);
    return check_launch("sfb_attention_backward");
}

int tc_backward(cudaStream_t s, const void *nn_lut, const void *tn_lut, const void *q, const void *k, const void *v, const void *pblk, const void *o,
                const void *dout, float *delta, void *dq, void *dk, void *dv, int dtype, const AttnDims &p, float scale)
{
    return dtype == SFB_BF16 ? launch_backward<true>(s, nn_lut, tn_lut, q, k, v, pblk, o, dout, delta, dq, dk, dv, p, scale)
                             : launch_backward<false>(s, nn_lut, tn_lut, q, k, v, pblk, o, dout, delta, dq, dk, dv, p, scale);
}

int tc_status_clear_backward()
{
    const uint32_t zero = 0;
    cudaError_t e = cudaMemcpyToSymbol(tc::g_status, &zero, sizeof(uint32_t));
    if (e != cudaSuccess) return fail("sfb_device_status_clear: %s", cudaGetErrorString(e));
    return 0;
}

int tc_status_backward(uint32_t *out)
{
    cudaError_t e = cudaMemcpyFromSymbol(out, tc::g_status, sizeof(uint32_t));
    if (e != cudaSuccess) return fail("sfb_device_status: %s", cudaGetErrorString(e));
    return 0;
}

}  // namespace sfb
