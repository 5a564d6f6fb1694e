// Backward of the block-sparse attention on the tensor cores (tcgen05) for 16-bit operands, block_size 64, head size 64,
// from the saved probabilities P and the forward output O:
//   delta = rowsum(dO * O),  dS = P * (dO.V^T - delta) * scale,  dQ = dS.K,  dK = dS^T.Q,  dV = P^T.dO
// (the call order of transformer_attention_optimize.cu:924-964).  As separate operators this moves the block tensors five
// times (P in for dV and for dS, dS out, dS in for dK and for dQ); here dS never leaves the SM: one kernel walks pairs of
// block-rows and makes dQ, one walks pairs of block-columns and makes dK and dV, and each recomputes dS from its own read
// of P -- a product of tensor work per block, which is free next to 8 KB of P.  The row kernel also makes delta.
//
// Both are the same kernel, seen from the two sides (COL).  A CTA owns 128 "own" positions (queries of two block-rows, or
// keys of two block-columns) and walks the union of their blocks; per step
//     dP  = X . Y^T           X: own rows of dO (V), an A operand that waits in TMEM; Y: the step's rows of V (dO), by TMA
//     dS  = P * (dP - delta)  256 threads, one own position and 32 of the 64 others each; dS goes back to TMEM, 16 bits
//     out += dS . Z           Z: the step's rows of K (Q)                              -> dQ (dK)
//     COL: dV += P^T . Y      the two blocks of P as one MN-major A operand
// A block that only one of the two rows (columns) keeps is fetched from beyond the tensor and arrives as zeros.
// TMEM (256 columns, two CTAs per SM): dP 64, dS 32 (packed), X 32, the accumulators 64 + 64.  dP has one buffer: it is
// free again as soon as its values are in registers, so the next step's product runs under this step's arithmetic.
// Bound by HBM (P once per kernel: 16 KB per step against 128 bytes per clock of shared memory for 72 KB of operands);
// measured beside the code that launches it.
#include "tc_common.cuh"

namespace sfb {
namespace tc {

constexpr uint32_t kBwStages = 3;
constexpr uint32_t kBwStageBytes = 4 * kTileBytes + 256;        // two blocks of P, Y, Z, the step's 64 deltas (COL)
constexpr uint32_t kBwStagePitch = 4 * kTileBytes;              // the deltas live behind all stages (tiles want 1024-byte alignment)
constexpr int kBwThreads = 64 + 256;

struct BwShared {
    uint64_t in_full[kBwStages], in_empty[kBwStages], x_ready, s_full, s_free, ds_full, ds_free, o_final, drained;
    uint32_t tmem_base, n_union, abort_flag, pad;
    alignas(16) float delta[kBwStages][64];
    float comb[2][128];
    UnionEntry entries[kMaxUnion];
    uint2 cand[kMaxUnion];
};
constexpr size_t kBwSmem = 1024 + kBwStages * kBwStagePitch + sizeof(BwShared);
static_assert(2 * (kBwSmem + 1024) <= 228 * 1024, "two CTAs per SM");

struct BwParams {
    const uint2 *lut;          // nn_lut (rows) or tn_lut (columns)
    const void *X;             // dO (rows) or V (columns), read directly
    const void *O;             // rows: the forward output
    float *delta;              // [B, H, L] scale * rowsum(dO * O): written by the row kernel, read by the column kernel
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

template <bool COL, bool BF16>
__global__ void __launch_bounds__(kBwThreads, 2)
backward_tc_kernel(const __grid_constant__ CUtensorMap pmap, const __grid_constant__ CUtensorMap ymap, const __grid_constant__ CUtensorMap zmap,
                   const BwParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    BwShared *st = (BwShared *)(smem + kBwStages * kBwStagePitch);

    const uint32_t warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t pair = blockIdx.x, b = blockIdx.y, h = blockIdx.z;
    const uint32_t L = p.nb * 64;
    volatile uint32_t *abort_flag = &st->abort_flag;
    const uint32_t fmt = BF16 ? 1u : 0u;

    if (threadIdx.x == 0) {
        prefetch_map(pmap);
        prefetch_map(ymap);
        prefetch_map(zmap);
        for (uint32_t s = 0; s < kBwStages; s++) { mbar_init(&st->in_full[s], 1); mbar_init(&st->in_empty[s], 1); }
        mbar_init(&st->x_ready, 256);
        mbar_init(&st->s_full, 1);
        mbar_init(&st->s_free, 256);
        mbar_init(&st->ds_full, 256);
        mbar_init(&st->ds_free, 1);
        mbar_init(&st->o_final, 1);
        mbar_init(&st->drained, 1);
        st->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&st->tmem_base)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    grid_dependency_wait();
    grid_launch_dependents();
    build_union(p.lut + (size_t)h * p.lut_stride, pair, p.nb, st->entries, st->cand, &st->n_union, &st->abort_flag);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();

    const uint32_t T = st->n_union;
    const uint32_t tmem = st->tmem_base;
    const uint32_t t_s = tmem, t_ds = tmem + 64, t_x = tmem + 96, t_o1 = tmem + 128, t_o2 = tmem + 192;

    if (warp == 0) {
        // ===== TMA producer =====
        if (T > 0 && elect_one()) {
            const uint32_t bh_rows = ((b * p.H + h) * p.blocks) * 64;            // first row of this (b,h) in the 2-D view of P
            for (uint32_t t = 0; t < T; t++) {
                const uint32_t s = t % kBwStages;
                if (t >= kBwStages && !mbar_wait(&st->in_empty[s], ((t / kBwStages) - 1) & 1, abort_flag, 71)) break;
                const UnionEntry ent = st->entries[t];
                const uint32_t base = smem_u32(smem + s * kBwStagePitch);
                mbar_expect_tx(&st->in_full[s], COL ? kBwStageBytes : kBwStagePitch);
                const int32_t y0 = (ent.flags & 1) ? (int32_t)(bh_rows + ent.blk[0] * 64) : (int32_t)p.p_rows;
                const int32_t y1 = (ent.flags & 2) ? (int32_t)(bh_rows + ent.blk[1] * 64) : (int32_t)p.p_rows;
                tma_load_2d(base, &pmap, &st->in_full[s], 0, y0);
                tma_load_2d(base + kTileBytes, &pmap, &st->in_full[s], 0, y1);
                tma_load_2d(base + 2 * kTileBytes, &ymap, &st->in_full[s], (int32_t)(h * 64), (int32_t)(b * L + ent.col * 64));
                tma_load_2d(base + 3 * kTileBytes, &zmap, &st->in_full[s], (int32_t)(h * 64), (int32_t)(b * L + ent.col * 64));
                if (COL) bulk_load(smem_u32(st->delta[s]), p.delta + ((size_t)b * p.H + h) * L + (size_t)ent.col * 64, 256, &st->in_full[s]);
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer:  dP(0) | dP(1) out(0) | dP(2) out(1) | ...  =====
        if (T > 0 && elect_one()) {
            const uint32_t idesc_dp = instr_desc(fmt, fmt, 128, 64, 0);                 // Y rows along N, K-major
            const uint32_t idesc_out = instr_desc(fmt, fmt, 128, 64, 1);                // Z rows along K
            const uint32_t idesc_dv = idesc_out | (1u << 15);                           // P transposed: A MN-major
            bool alive = mbar_wait(&st->x_ready, 0, abort_flag, 72);
            for (uint32_t t = 0; alive && t <= T; t++) {
                if (t < T) {
                    const uint32_t s = t % kBwStages;
                    if (!mbar_wait(&st->in_full[s], (t / kBwStages) & 1, abort_flag, 73)) break;
                    if (t >= 1 && !mbar_wait(&st->s_free, (t - 1) & 1, abort_flag, 74)) break;
                    tcgen05_fence_after();
                    const uint32_t base = smem_u32(smem + s * kBwStagePitch);
                    const uint64_t y_desc = smem_desc_sw128(base + 2 * kTileBytes);
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) umma_f16_ts(t_s, t_x + 8 * kk, y_desc + 2 * kk, idesc_dp, kk);
                    umma_commit(&st->s_full);
                    if (COL) {
                        const uint64_t p_desc = smem_desc_sw128(base, kTileBytes);      // the second block is the next 64 along M
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; kk++) umma_f16(t_o2, p_desc + 128 * kk, y_desc + 128 * kk, idesc_dv, (t | kk) ? 1u : 0u);
                    }
                }
                if (t > 0) {
                    const uint32_t s = (t - 1) % kBwStages;
                    if (!mbar_wait(&st->ds_full, (t - 1) & 1, abort_flag, 75)) break;
                    tcgen05_fence_after();
                    const uint64_t z_desc = smem_desc_sw128(smem_u32(smem + s * kBwStagePitch + 3 * kTileBytes));
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) umma_f16_ts(t_o1, t_ds + 8 * kk, z_desc + 128 * kk, idesc_out, (t > 1 || kk) ? 1u : 0u);
                    umma_commit(&st->in_empty[s]);
                    umma_commit(&st->ds_free);
                    if (t == T) umma_commit(&st->o_final);
                }
            }
        }
    } else {
        // ===== dS and the epilogue: own position r, half of the other side's 64 =====
        const uint32_t quarter = warp & 3, ch = (warp - 2) >> 2;
        const uint32_t cb = ch * 32, r = quarter * 32 + lane, half = r >> 6;
        const uint32_t lane_field = (quarter * 32) << 16;
        const bool row_valid = half == 0 || pair * 2 + 1 < p.nb;
        const size_t own = ((size_t)b * L + (size_t)pair * 128 + r) * ((size_t)p.H * 64) + (size_t)h * 64 + cb;
        float my_delta = 0.f;                                // rows: scale * delta of this query
        {
            uint32_t w[16];
            float dot = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint4 u = make_uint4(0u, 0u, 0u, 0u), o = u;
                if (row_valid) {
                    u = *(const uint4 *)((const uint16_t *)p.X + own + 8 * j);
                    if (!COL) o = *(const uint4 *)((const uint16_t *)p.O + own + 8 * j);
                }
                w[4 * j] = u.x; w[4 * j + 1] = u.y; w[4 * j + 2] = u.z; w[4 * j + 3] = u.w;
                if (!COL) {
                    const uint32_t ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float2 x = unpack2(w[4 * j + q], BF16), y = unpack2(ov[q], BF16);
                        dot = fmaf(x.x, y.x, fmaf(x.y, y.y, dot));
                    }
                }
            }
            TMEM_ST_16(t_x + ch * 16 + lane_field, (w));
            tmem_wait_st();
            tcgen05_fence_before();
            mbar_arrive(&st->x_ready);
            if (!COL) {
                st->comb[ch][r] = dot;
                asm volatile("bar.sync 1, 256;" ::: "memory");           // nobody has given up yet: all 256 threads are here
                my_delta = (dot + st->comb[ch ^ 1][r]) * p.scale;
                if (ch == 0 && row_valid) p.delta[((size_t)b * p.H + h) * L + (size_t)pair * 128 + r] = my_delta;
            }
        }
        // COL: this key's 16 bits of row q of its block sit at q * 128 + (chunk ^ (q % 8)) * 16 + offset
        const uint32_t key = r & 63, key_chunk = key >> 3, key_off = (key & 7) * 2;
        bool alive = true;
        for (uint32_t t = 0; t < T; t++) {
            const uint32_t s = t % kBwStages;
            if (!mbar_wait_warp(&st->s_full, t & 1, abort_flag, 76)) { alive = false; break; }
            tcgen05_fence_after();
            uint32_t v[32];
            TMEM_LD_32((v), t_s + lane_field + cb);
            // P (and the deltas) came with the barrier the product waited for; observing it makes them visible to this thread
            if (!mbar_wait_warp(&st->in_full[s], (t / kBwStages) & 1, abort_flag, 77)) { alive = false; break; }
            tmem_wait_ld();
            tcgen05_fence_before();
            mbar_arrive(&st->s_free);
            const uint8_t *tile = smem + s * kBwStagePitch + half * kTileBytes;
            uint32_t w[16];
            if (COL) {
                const float *dl = st->delta[s] + cb;
#pragma unroll
                for (int q = 0; q < 32; q += 4) {
                    const float4 d4 = *(const float4 *)(dl + q);         // the same address in every lane
                    const float d[4] = {d4.x, d4.y, d4.z, d4.w};
                    float e[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const uint32_t qq = cb + q + j;
                        const uint16_t bits = *(const uint16_t *)(tile + qq * 128 + ((key_chunk ^ (qq & 7)) << 4) + key_off);
                        const float pv = BF16 ? __uint_as_float((uint32_t)bits << 16) : __half2float(__ushort_as_half(bits));
                        e[j] = pv * fmaf(__uint_as_float(v[q + j]), p.scale, -d[j]);
                    }
                    w[q / 2] = pack2(e[0], e[1], BF16);
                    w[q / 2 + 1] = pack2(e[2], e[3], BF16);
                }
            } else {
                const uint8_t *prow = tile + (r & 63) * 128;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint4 u = *(const uint4 *)(prow + (((cb / 8 + c) ^ (r & 7)) << 4));
                    const uint32_t pw[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float2 pv = unpack2(pw[j], BF16);
                        const int i = c * 8 + 2 * j;
                        w[c * 4 + j] = pack2(pv.x * fmaf(__uint_as_float(v[i]), p.scale, -my_delta),
                                             pv.y * fmaf(__uint_as_float(v[i + 1]), p.scale, -my_delta), BF16);
                    }
                }
            }
            if (t >= 1 && !mbar_wait_warp(&st->ds_free, (t - 1) & 1, abort_flag, 78)) { alive = false; break; }
            tcgen05_fence_after();
            TMEM_ST_16(t_ds + ch * 16 + lane_field, (w));
            tmem_wait_st();
            tcgen05_fence_before();
            mbar_arrive(&st->ds_full);
        }
        if (alive && T > 0) alive = mbar_wait_warp(&st->o_final, 0, abort_flag, 79);
        if (alive) {
            tcgen05_fence_after();
#pragma unroll
            for (int o = 0; o < (COL ? 2 : 1); o++) {
                uint32_t v[32];
                if (T > 0) {
                    TMEM_LD_32((v), (o ? t_o2 : t_o1) + lane_field + cb);
                    tmem_wait_ld();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = 0u;              // rows and columns without blocks have zero gradients
                }
                if (row_valid) {
                    uint4 *dst = (uint4 *)((uint16_t *)(o ? p.out2 : p.out1) + own);
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        uint32_t y[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) y[j] = pack2(__uint_as_float(v[8 * c + 2 * j]), __uint_as_float(v[8 * c + 2 * j + 1]), BF16);
                        dst[c] = make_uint4(y[0], y[1], y[2], y[3]);
                    }
                }
            }
        }
    }

    // ---- teardown (also the way out after a timeout) ----
    tcgen05_fence_before();
    __syncthreads();
    if (st->abort_flag) {
        if (warp == 1 && lane == 0) {
            umma_commit(&st->drained);
            for (uint32_t i = 0; i < kWaitLimit && !mbar_try_wait(&st->drained, 0); i++) {}
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
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
}

}  // namespace tc

bool tc_backward_supported(int dtype, uint32_t bs, const AttnDims &p, uint32_t nn_max, uint32_t tn_max, uint64_t pointers)
{
    return (dtype == SFB_BF16 || dtype == SFB_F16) && bs == 64 && p.d == 64 && p.blocks > 0 && (pointers & 15) == 0 && nn_max && tn_max &&
           2 * (uint64_t)nn_max <= tc::kMaxUnion && 2 * (uint64_t)tn_max <= tc::kMaxUnion && (uint64_t)p.B * p.nb_a * 64 < (1ull << 31) &&
           (uint64_t)p.B * p.H * p.blocks * 64 < (1ull << 31) - 64;
}

template <bool BF16>
static int launch_backward(cudaStream_t s, const void *nn_lut, const void *tn_lut, const void *q, const void *k, const void *v, const void *pblk,
                           const void *o, const void *dout, float *delta, void *dq, void *dk, void *dv, const AttnDims &p, float scale)
{
    using namespace tc;
    const uint64_t rows = (uint64_t)p.B * p.nb_a * 64, prow = (uint64_t)p.B * p.H * p.blocks * 64;
    CUtensorMap pm, qm, km, vm, dm;
    if (make_map_2d(&pm, pblk, prow, 64, BF16, 64) || make_map(&qm, q, rows, p.H, BF16, 64) || make_map(&km, k, rows, p.H, BF16, 64) ||
        make_map(&vm, v, rows, p.H, BF16, 64) || make_map(&dm, dout, rows, p.H, BF16, 64))
        return 1;
    static DeviceOnce once;
    const int dev = current_device();
    if (!once.done(dev)) {
        if (cudaFuncSetAttribute(backward_tc_kernel<false, BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwSmem) != cudaSuccess ||
            cudaFuncSetAttribute(backward_tc_kernel<true, BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwSmem) != cudaSuccess)
            return fail("sfb_attention_backward: cannot reserve %zu bytes of shared memory", kBwSmem);
        once.mark(dev);
    }
    const dim3 grid((p.nb_a + 1) / 2, p.B, p.H);
    const BwParams row = {(const uint2 *)nn_lut, dout, o, delta, dq, nullptr, p.B, p.H, p.nb_a, p.blocks, p.lut_stride, (uint32_t)prow, scale};
    const BwParams col = {(const uint2 *)tn_lut, v, nullptr, delta, dk, dv, p.B, p.H, p.nb_a, p.blocks, p.lut_stride, (uint32_t)prow, scale};
    launch_overlapped(backward_tc_kernel<false, BF16>, grid, dim3(kBwThreads), kBwSmem, s, pm, vm, km, row);
    launch_overlapped(backward_tc_kernel<true, BF16>, grid, dim3(kBwThreads), kBwSmem, s, pm, dm, qm, col);
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
