// Element-sparse (CSR) attention: the alternative sparse format the reference prototypes with one thread per query row
// (csr_sddmm / csr_softmax / csr_spmm and fused_attention, cuda_kernels.h:976-1075; mask generators ewops.h:430-459).
// One CSR pattern (rowptr [L+1], colidx [nnz], int32) is shared by every (batch, head).
//
//   csr_from_layout_kernel   block layout -> the CSR pattern of all elements of its kept blocks
//   csr_plan_kernel          the pattern by tiles of 32 query rows: the columns any of them has, in ascending order, each with
//                            a 32-bit mask of the rows that have it
//   csr_tile_kernel          O for one tile and (batch, head) over those columns, 16-bit operands, on warp MMAs
//   csr_tile_f32_kernel      (attn_simt.cu) the same for fp32 operands, split into bf16 terms
//   csr_attention_split_kernel   one warp per query row, four lanes per key: callers without a workspace for the plan, and
//                            sequences whose columns do not fit the plan's shared memory
// Row by row every query gathers its own keys through L2 (294 keys, 75 KB, per row of a 256-token window with strided and
// random columns): 626 us at B 2, H 12, L 4096, d 64, with the FMA pipes half idle.  32 neighbouring rows mostly want the
// same keys, so a tile fetches each column once and masks the rows that do not have it: a ninth of the bytes, and the
// products are contractions again.  The plan is made once per call and shared by the batch's heads.
#include "attn.cuh"
#include "csr.cuh"

namespace sfb {

// one CTA per block-row; dynamic smem: uint32 cols[nb] (kept column blocks of this row)
__global__ void csr_from_layout_kernel(const uint8_t *__restrict__ layout, uint32_t nb, uint32_t bs, int32_t *__restrict__ rowptr,
                                       int32_t *__restrict__ colidx)
{
    extern __shared__ uint32_t cols[];
    __shared__ uint32_t before, mine;
    const uint32_t bi = blockIdx.x;
    if (threadIdx.x == 0) {
        uint32_t b = 0, m = 0;
        for (uint32_t r = 0; r < bi; r++)
            for (uint32_t j = 0; j < nb; j++) b += layout[(size_t)r * nb + j] != 0;
        for (uint32_t j = 0; j < nb; j++)
            if (layout[(size_t)bi * nb + j]) cols[m++] = j;
        before = b;
        mine = m;
    }
    __syncthreads();
    const size_t base = (size_t)before * bs * bs;           // nonzeros of all earlier block-rows
    const uint32_t per_row = mine * bs;
    for (uint32_t r = threadIdx.x; r < bs; r += blockDim.x) rowptr[(size_t)bi * bs + r + 1] = (int32_t)(base + (size_t)(r + 1) * per_row);
    if (bi == 0 && threadIdx.x == 0) rowptr[0] = 0;
    for (size_t e = threadIdx.x; e < (size_t)bs * per_row; e += blockDim.x) {
        const uint32_t within = (uint32_t)(e % per_row);
        colidx[base + e] = (int32_t)(cols[within / bs] * bs + within % bs);
    }
}

// One warp per query row.
template <int DT, int D, int LPK>
__global__ void __launch_bounds__(128) csr_attention_split_kernel(const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
                                                                 const void *__restrict__ Q, const void *__restrict__ K,
                                                                 const void *__restrict__ V, void *__restrict__ O, uint32_t L,
                                                                 uint32_t H, float scale_log2e, uint32_t *bad)
{
    const uint32_t i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i < L) csr_row<DT, D, LPK>(colidx, rowptr[i], rowptr[i + 1], Q, K, V, O, L, H, blockIdx.y, blockIdx.z, i, scale_log2e, bad);
}

// ---- the plan -------------------------------------------------------------------------------------------------
// One CTA per tile of 32 query rows.  Every element sets its row's bit in its column's mask in shared memory; what is set
// is written out column by column.  A column that a row names twice counts twice, as it does row by row: the second one
// becomes an entry of its own at the end.  The tile's entries start at its first row's offset in colidx: there are never
// more of them than elements.  Columns outside the sequence are counted and dropped.
// HALVES: the distinct columns come in three groups: those that only the tile's first 16 rows have, those of both halves,
// those of the last 16 rows alone.  Scattered columns mostly belong to one row; the kernels whose warps work for 16 rows
// (D 128) leave out the group of the other half.
// A warp per row, whose elements are on their way at once (plan and tiles of the window pattern, B 2, H 12, L 4096, d 64:
// 105.8 us against 108.7 with two rows per warp).  The tiles' launch is not let in early: their CTAs would crowd the SMs that the plan left free and stay
// there (128 tiles, B 1, H 1: 24.4 us, 17.4 like this).
constexpr uint32_t kPlanThreads = 1024;
constexpr uint32_t kPlanMaxL = 48 * 1024;                    // columns whose masks fit shared memory
template <bool HALVES>
__global__ void __launch_bounds__(kPlanThreads) csr_plan_kernel(const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx, uint32_t L,
                                                                uint32_t nnz, uint2 *__restrict__ entries, uint32_t *__restrict__ counts,
                                                                uint32_t *__restrict__ bad)
{
    extern __shared__ uint32_t mask[];                       // [L]
    constexpr uint32_t NG = HALVES ? 3 : 1;                  // groups of columns
    __shared__ uint32_t warp_count[NG][kPlanThreads / 32], n_twice, n_bad;
    grid_dependency_wait();
    const uint32_t tile = blockIdx.x, row0 = tile * 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rows = min(32u, L - row0);
    const uint32_t base = min((uint32_t)max(rowptr[row0], 0), nnz), top = min((uint32_t)max(rowptr[row0 + rows], 0), nnz);
    if (threadIdx.x == 0) n_twice = n_bad = 0;
    for (uint32_t j = threadIdx.x; j < L; j += kPlanThreads) mask[j] = 0;
    __syncthreads();
    for (uint32_t r = warp; r < rows; r += kPlanThreads / 32) {
        const int32_t lo = max(rowptr[row0 + r], 0), hi = (int32_t)min((uint32_t)max(rowptr[row0 + r + 1], 0), nnz);
        for (int32_t e0 = lo + (int32_t)lane; e0 < hi; e0 += 32 * 8) {
            int32_t col[8];                                  // eight reads on their way at once
#pragma unroll
            for (int u = 0; u < 8; u++) col[u] = e0 + 32 * u < hi ? __ldg(colidx + e0 + 32 * u) : 0;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (e0 + 32 * u >= hi) break;
                const int32_t j = col[u];
                if (j < 0 || (uint32_t)j >= L) { atomicAdd(&n_bad, 1u); continue; }
                if (atomicOr(&mask[j], 1u << r) & (1u << r)) {
                    const uint32_t at = top - 1u - atomicAdd(&n_twice, 1u);      // from the end of the tile's share backwards
                    if (at >= base && at < nnz) entries[at] = make_uint2((uint32_t)j, 1u << r);
                }
            }
        }
    }
    __syncthreads();
    // every warp takes a run of columns: count by group, prefix over the groups and warps, write
    auto group = [](uint32_t m) { return !m ? NG : !HALVES || !(m >> 16) ? 0u : m & 0xffffu ? 1u : 2u; };
    const uint32_t per = ((L + kPlanThreads / 32 - 1) / (kPlanThreads / 32) + 31) & ~31u;
    const uint32_t from = min(warp * per, L), to = min(from + per, L);
    uint32_t at[NG] = {}, all[NG] = {};
    for (uint32_t j0 = from; j0 < to; j0 += 32) {
        const uint32_t g = group(j0 + lane < to ? mask[j0 + lane] : 0);
#pragma unroll
        for (uint32_t k = 0; k < NG; k++) at[k] += __popc(__ballot_sync(0xffffffffu, g == k));
    }
#pragma unroll
    for (uint32_t k = 0; k < NG; k++)
        if (lane == k) warp_count[k][warp] = at[k];
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (uint32_t k = 0; k < NG; k++) {
        const uint32_t c = lane < kPlanThreads / 32 ? warp_count[k][lane] : 0;
        at[k] = base + total + __reduce_add_sync(0xffffffffu, lane < warp ? c : 0);
        all[k] = __reduce_add_sync(0xffffffffu, c);
        total += all[k];
    }
    for (uint32_t j0 = from; j0 < to; j0 += 32) {
        const uint32_t m = j0 + lane < to ? mask[j0 + lane] : 0, g = group(m);
#pragma unroll
        for (uint32_t k = 0; k < NG; k++) {
            const uint32_t votes = __ballot_sync(0xffffffffu, g == k), dst = at[k] + __popc(votes & ((1u << lane) - 1u));
            if (g == k && dst < nnz) entries[dst] = make_uint2(j0 + lane, m);
            at[k] += __popc(votes);
        }
    }
    if (threadIdx.x == 0) {
        uint32_t *c = counts + kCsrCounts * tile;
        c[0] = min(total, nnz - base);
        c[1] = min(n_twice, top - min(base, top));
        c[2] = base;
        c[3] = top;
        if (HALVES) {
            c[4] = all[0];
            c[5] = all[NG - 1];
        }
        bad[tile] = n_bad;
    }
}

// ---- one tile of 32 query rows x one (batch, head), 16-bit operands ------------------------------------------------
// Four warps share the tile's columns, a chunk of KC of them at a time each (two warps share a chunk when D is 128: 16 rows
// each), with no barrier between them: a warp fetches its chunk's K and V rows into its own two buffers (cp.async, one
// chunk ahead), multiplies on warp MMAs (m16n8k16), and keeps its own running maximum, sum and output; the four meet at
// the end.  Warp MMAs rather than tcgen05: the columns of a tile are rows scattered over K and V, and 32 rows is where
// neighbouring queries still share them.
// The queries are read from shared memory as they are needed and the chunks are small: what bounds the kernel is latency
// (40 % of the issue slots, tensor pipe 43 %, L2 18 %: a chunk is 360 instructions of 7.5 cycles each on one of three warps; 32 columns per
// chunk 96.8 us instead of 95.1), so the registers go to more CTAs (D 128: two per SM became three, 226 -> 170 us for
// the window pattern at B 2, H 12, L 4096) or keep the accumulators out of local memory (D 64: 114.4 -> 105.8, at four CTAs
// per SM 119).
// P enters P.V as two 16-bit terms (the rounded value and what the rounding left), so the product keeps the fp32
// probabilities to 16 bits (bf16) and 22 bits (fp16).
constexpr float kCsrGrow = 8.f;
template <int D> struct CsrCfg {
    static constexpr int MT = D == 128 ? 1 : 2;              // 16-row tiles per warp
    static constexpr int SPLITS = D == 128 ? 2 : 4;          // warps that take different chunks
    static constexpr int KC = D >= 64 ? 16 : 32;             // columns per chunk
    static constexpr uint32_t tile_bytes = KC * D * 2;
    static constexpr int CTAS = D >= 64 ? 3 : 4;             // per SM: what their registers admit
    static constexpr uint32_t o_stride = D + 4;              // floats; the outputs take the buffers' place at the end
    static constexpr uint32_t o_bytes = MT * 16 * o_stride * 4, kv_bytes = 4 * tile_bytes;       // K and V, two buffers
    static constexpr uint32_t warp_bytes = o_bytes > kv_bytes ? o_bytes : kv_bytes;
    static constexpr size_t smem = 4 * warp_bytes + 32 * D * 2;      // the tile's queries behind the warps' buffers
};
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_trans(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    if (BF16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float a, float b)
{
    uint32_t y;
    if (BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(y) : "f"(b), "f"(a));
    else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(y) : "f"(b), "f"(a));
    return y;
}
template <bool BF16>
__device__ __forceinline__ float2 unpack16(uint32_t v)
{
    if (BF16) return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    return __half22float2(*reinterpret_cast<const __half2 *>(&v));
}
__device__ __forceinline__ float ex2f(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// pairs of floats: one issue slot for two operations
__device__ __forceinline__ uint64_t pair2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpair2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

template <bool BF16, int D>
__global__ void __launch_bounds__(128, CsrCfg<D>::CTAS) csr_tile_kernel(const CsrTileArgs a)
{
    typedef CsrCfg<D> Cfg;
    constexpr int MT = Cfg::MT, KC = Cfg::KC, NT = KC / 8, CH = D / 8, DN = D / 8;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ __align__(8) uint32_t masks[4][2][KC];
    __shared__ float2 ml[4][MT * 16];
    grid_dependency_wait();
    grid_launch_dependents();
    csr_write_bad(a);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane >> 2, tq = lane & 3;
    const uint32_t tile = a.tiles - 1u - blockIdx.x, h = blockIdx.y, b = blockIdx.z;     // causal patterns: the long rows first
    const uint32_t *cnt = a.counts + kCsrCounts * tile;
    const uint32_t distinct = cnt[0], twice = cnt[1], base = cnt[2], top = cnt[3];
    const uint32_t split = MT == 2 ? warp : warp >> 1, rg = MT == 2 ? 0 : warp & 1;        // this warp's chunks and 16-row tile
    // with 16 rows per warp: not the other half's columns (entries of columns named twice are behind all of them)
    const uint32_t first = MT == 1 && rg == 1 ? min(cnt[4], distinct) : 0;
    const uint32_t n = MT == 1 && rg == 0 && twice == 0 ? distinct - min(cnt[5], distinct) : distinct + twice;
    const uint32_t chunks = (n - first + KC - 1) / KC;
    const size_t HD = (size_t)a.H * D;
    const uint16_t *K = (const uint16_t *)a.K + (size_t)b * a.L * HD + (size_t)h * D, *V = (const uint16_t *)a.V + (size_t)b * a.L * HD + (size_t)h * D;
    uint8_t *buf = sm + warp * Cfg::warp_bytes;

    uint4 q_piece[CH / 4];                                   // this thread's share of the queries, on its way to shared memory
#pragma unroll
    for (int i = 0; i < CH / 4; i++) {
        const uint32_t t = i * 128 + threadIdx.x, row = tile * 32 + t / CH;
        const uint16_t *src = (const uint16_t *)a.Q + ((size_t)b * a.L + row) * HD + (size_t)h * D + t % CH * 8;
        q_piece[i] = row < a.L ? __ldg((const uint4 *)src) : make_uint4(0u, 0u, 0u, 0u);
    }
    float o[MT][DN][4], m[MT][2];
    uint64_t l[MT][2];                                       // two partial sums of a row, one per column of a pair
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        m[mt][0] = m[mt][1] = -INFINITY;
        l[mt][0] = l[mt][1] = 0ull;
#pragma unroll
        for (int d = 0; d < DN; d++)
#pragma unroll
            for (int j = 0; j < 4; j++) o[mt][d][j] = 0.f;
    }
    auto entry = [&](uint32_t c) {
        const uint32_t i = first + c * KC + lane;
        return (KC == 32 || lane < KC) && i < n ? csr_entry(a.entries, base, top, distinct, i) : make_uint2(0u, 0u);
    };
    // 16-byte chunk c of row r of a tile sits at chunk c ^ (r % 8) (64-byte rows: c ^ (r / 2 % 4)): no bank twice in a ldmatrix
    auto place = [](uint32_t r, uint32_t c) { return r * (D * 2) + ((c ^ (D == 32 ? (r >> 1) & 3u : r & 7u)) << 4); };
    static_assert(32 % CH == 0, "a lane keeps its piece of the row");
    const uint32_t pitch = (uint32_t)(HD * 2);               // bytes; 32 bits, so that an address is one wide multiply-add
    const uint64_t klane = (uint64_t)(K + lane % CH * 8), vlane = (uint64_t)(V + lane % CH * 8);
    auto issue = [&](const uint2 &e, uint32_t s) {
        const uint32_t kt = (uint32_t)__cvta_generic_to_shared(buf + s * 2 * Cfg::tile_bytes), vt = kt + Cfg::tile_bytes;
#pragma unroll
        for (int i = 0; i < KC * CH / 32; i++) {
            const uint32_t r = i * (32 / CH) + lane / CH;
            const uint64_t at = (uint64_t)__shfl_sync(0xffffffffu, e.x, r) * pitch;
            const uint32_t off = place(r, lane % CH);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(kt + off), "l"(klane + at) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vt + off), "l"(vlane + at) : "memory");
        }
        if (KC == 32 || lane < KC) masks[warp][s][lane % KC] = e.y;
    };
    const uint32_t qt = (uint32_t)__cvta_generic_to_shared(sm + 4 * Cfg::warp_bytes);
    const uint64_t scale2 = pair2(a.scale_log2e, a.scale_log2e), one2 = pair2(1.f, 1.f), minus2 = pair2(-1.f, -1.f);
    uint2 e_next = make_uint2(0u, 0u);
    if (split < chunks) {
        issue(entry(split), 0);
        if (split + Cfg::SPLITS < chunks) e_next = entry(split + Cfg::SPLITS);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int i = 0; i < CH / 4; i++) {
        const uint32_t t = i * 128 + threadIdx.x;
        *(uint4 *)(sm + 4 * Cfg::warp_bytes + place(t / CH, t % CH)) = q_piece[i];
    }
    __syncthreads();
    uint32_t s = 0;
    for (uint32_t c = split; c < chunks; c += Cfg::SPLITS, s ^= 1) {
        if (c + Cfg::SPLITS < chunks) {
            issue(e_next, s ^ 1);
            if (c + 2 * Cfg::SPLITS < chunks) e_next = entry(c + 2 * Cfg::SPLITS);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const uint32_t kt = (uint32_t)__cvta_generic_to_shared(buf + s * 2 * Cfg::tile_bytes), vt = kt + Cfg::tile_bytes;
        // S = Q . K^T
        float sc[MT][NT][4];
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int j = 0; j < 4; j++) sc[mt][t][j] = 0.f;
#pragma unroll
        for (int kk = 0; kk < D / 16; kk++) {
            uint32_t q[MT][4], f[NT / 2][4];
#pragma unroll
            for (int mt = 0; mt < MT; mt++) ldsm(q[mt], qt + place((rg + mt) * 16 + (lane & 15), 2 * kk + (lane >> 4)));
#pragma unroll
            for (int t = 0; t < NT; t += 2) ldsm(f[t / 2], kt + place(t * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)));
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int mt = 0; mt < MT; mt++) mma16816<BF16>(sc[mt][t], q[mt], f[t / 2][2 * (t & 1)], f[t / 2][2 * (t & 1) + 1]);
        }
        // mask: bit `row` of a column's word
        uint2 mk[NT];
        uint32_t all = 0xffffffffu;
#pragma unroll
        for (int t = 0; t < NT; t++) {
            mk[t] = *(const uint2 *)&masks[warp][s][t * 8 + 2 * tq];
            all &= mk[t].x & mk[t].y;
        }
        if (__any_sync(0xffffffffu, all != 0xffffffffu)) {
#pragma unroll
            for (int t = 0; t < NT; t++) {
                const uint32_t x = mk[t].x >> (rg * 16 + quad), y = mk[t].y >> (rg * 16 + quad);
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    sc[mt][t][0] = (x >> (16 * mt)) & 1u ? sc[mt][t][0] : -INFINITY;
                    sc[mt][t][1] = (y >> (16 * mt)) & 1u ? sc[mt][t][1] : -INFINITY;
                    sc[mt][t][2] = (x >> (16 * mt + 8)) & 1u ? sc[mt][t][2] : -INFINITY;
                    sc[mt][t][3] = (y >> (16 * mt + 8)) & 1u ? sc[mt][t][3] : -INFINITY;
                }
            }
        }
        // The reference maximum of a row (shared by its quad of lanes, in units of log2 after the scale) moves only when a score
        // outgrows it by 2^8: P stays below that, its two terms are as precise there, and a chunk of 16 columns, in which nearly
        // always one of 32 rows has a new maximum, needs neither the row's shuffles nor a rescaled output.
        float x[MT][2];
        bool grow = false;
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                x[mt][e] = fmaxf(sc[mt][0][2 * e], sc[mt][0][2 * e + 1]);
#pragma unroll
                for (int t = 1; t < NT; t++) x[mt][e] = fmaxf(x[mt][e], fmaxf(sc[mt][t][2 * e], sc[mt][t][2 * e + 1]));
                x[mt][e] *= a.scale_log2e;
                grow |= x[mt][e] > m[mt][e] + kCsrGrow;
            }
        if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    float top = x[mt][e];
                    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                    const float old = m[mt][e], nm = top > old + kCsrGrow ? top : old;
                    const float f = old > -INFINITY ? ex2f(old - nm) : 0.f;
                    m[mt][e] = nm;
                    l[mt][e] = fma2(l[mt][e], pair2(f, f), 0ull);
#pragma unroll
                    for (int d = 0; d < DN; d++) {
                        o[mt][d][2 * e] *= f;
                        o[mt][d][2 * e + 1] *= f;
                    }
                }
        }
        float neg[MT][2];
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int e = 0; e < 2; e++) neg[mt][e] = m[mt][e] > -INFINITY ? -m[mt][e] : 0.f;
        // P.V, 16 columns at a time
#pragma unroll
        for (int j = 0; j < NT / 2; j++) {
            uint32_t hi[MT][4], lo[MT][4];
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int t = 0; t < 2; t++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const float2 z = unpair2(fma2(pair2(sc[mt][2 * j + t][2 * e], sc[mt][2 * j + t][2 * e + 1]), scale2, pair2(neg[mt][e], neg[mt][e])));
                        const float p0 = ex2f(z.x), p1 = ex2f(z.y);
                        const uint64_t p2 = pair2(p0, p1);
                        l[mt][e] = fma2(p2, one2, l[mt][e]);
                        const uint32_t w = pack16<BF16>(p0, p1);
                        const float2 r = unpack16<BF16>(w), d = unpair2(fma2(pair2(r.x, r.y), minus2, p2));
                        hi[mt][2 * t + e] = w;
                        lo[mt][2 * t + e] = pack16<BF16>(d.x, d.y);
                    }
            uint32_t f[DN / 2][4];
#pragma unroll
            for (int d = 0; d < DN; d += 2) ldsm_trans(f[d / 2], vt + place(j * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), d + (lane >> 4)));
#pragma unroll
            for (int term = 0; term < 2; term++)
#pragma unroll
                for (int d = 0; d < DN; d++)
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) mma16816<BF16>(o[mt][d], term ? lo[mt] : hi[mt], f[d / 2][2 * (d & 1)], f[d / 2][2 * (d & 1) + 1]);
        }
        __syncwarp();                                        // the buffer may be filled again
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    // the warps' outputs, maxima and sums meet in shared memory
    float *ow = (float *)buf;
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float2 l2 = unpair2(l[mt][e]);
            float sum = l2.x + l2.y;
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            const uint32_t r = mt * 16 + quad + 8 * e;
            if (tq == 0) ml[warp][r] = make_float2(m[mt][e], sum);
#pragma unroll
            for (int d = 0; d < DN; d++) *(float2 *)(ow + r * Cfg::o_stride + d * 8 + 2 * tq) = make_float2(o[mt][d][2 * e], o[mt][d][2 * e + 1]);
        }
    __syncthreads();
    const uint32_t r = threadIdx.x >> 2, row = tile * 32 + r, d0 = (threadIdx.x & 3) * (D / 4);
    const uint32_t w0 = MT == 2 ? 0 : r >> 4, wr = MT == 2 ? r : r & 15;                  // the warps that hold this row
    constexpr uint32_t WS = MT == 2 ? 1 : 2;
    float M = -INFINITY, sum = 0.f, f[Cfg::SPLITS];
#pragma unroll
    for (int k = 0; k < Cfg::SPLITS; k++) M = fmaxf(M, ml[w0 + k * WS][wr].x);
#pragma unroll
    for (int k = 0; k < Cfg::SPLITS; k++) {
        const float2 x = ml[w0 + k * WS][wr];
        f[k] = x.x > -INFINITY ? ex2f(x.x - M) : 0.f;
        sum = fmaf(x.y, f[k], sum);
    }
    // the reference's denominator (ewops.h:93, cuda_kernels.h:1022); the sum may stand 2^8 above the reference's, where 1e-6 counts less
    const float inv = sum > 0.f ? 1.f / (sum + 1e-6f) : 0.f;
    uint16_t *dst = (uint16_t *)a.O + ((size_t)b * a.L + row) * HD + (size_t)h * D + d0;
    float zero = 0.f;                                          // stays 0 as long as every output is finite
#pragma unroll
    for (int c = 0; c < D / 4; c += 8) {
        float y[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < Cfg::SPLITS; k++) {
            const float *src = (const float *)(sm + (w0 + k * WS) * Cfg::warp_bytes) + wr * Cfg::o_stride + d0 + c;
#pragma unroll
            for (int j = 0; j < 8; j++) y[j] = fmaf(src[j], f[k], y[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) zero = fmaf(y[j], 0.f, zero);
        if (row < a.L)
            *(uint4 *)(dst + c) = make_uint4(pack16<BF16>(y[0] * inv, y[1] * inv), pack16<BF16>(y[2] * inv, y[3] * inv),
                                             pack16<BF16>(y[4] * inv, y[5] * inv), pack16<BF16>(y[6] * inv, y[7] * inv));
    }
    // a warp has written rows of its own, four lanes each: it makes those that are not finite again (csr_row_again)
    uint32_t odd = __ballot_sync(0xffffffffu, row < a.L && !(zero == 0.f));
    while (odd) {
        const uint32_t first_lane = __ffs(odd) - 1u, rr = (warp * 32 + first_lane) >> 2;
        odd &= ~(0xfu << (first_lane & ~3u));
        csr_row_again<BF16 ? SFB_BF16 : SFB_F16, D>(a.rowptr, a.colidx, a.nnz, a.Q, a.K, a.V, a.O, a.L, a.H, b, h, tile * 32 + rr, a.scale_log2e);
    }
}

template <bool BF16, int D>
static int launch_csr_tile(cudaStream_t s, const CsrTileArgs &a, uint32_t B)
{
    static DeviceOnce once;
    const int dev = current_device();
    if (!once.done(dev)) {
        if (cudaFuncSetAttribute(csr_tile_kernel<BF16, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CsrCfg<D>::smem) != cudaSuccess)
            return fail("sfb_csr_attention: cannot reserve %zu bytes of shared memory", CsrCfg<D>::smem);
        once.mark(dev);
    }
    launch_overlapped(csr_tile_kernel<BF16, D>, dim3(a.tiles, a.H, B), dim3(128), CsrCfg<D>::smem, s, a);
    return check_launch("sfb_csr_attention");
}

// entries of 8 bytes, one per element, then the counts and a bad-column count per tile of 32 rows
static size_t csr_workspace(uint64_t nnz, uint32_t L) { return nnz * 8 + (size_t)((L + 31) / 32) * (kCsrCounts + 1) * sizeof(uint32_t); }

static int csr_attention_planned(cudaStream_t s, const int32_t *rowptr, const int32_t *colidx, uint32_t nnz, const void *q, const void *k,
                                 const void *v, void *o, int dtype, uint32_t B, uint32_t L, uint32_t H, uint32_t d, float scale, uint32_t *bad,
                                 void *workspace)
{
    const uint32_t tiles = (L + 31) / 32;
    uint2 *entries = (uint2 *)workspace;
    uint32_t *counts = (uint32_t *)(entries + nnz);
    static DeviceOnce once;
    const int dev = current_device();
    if (!once.done(dev)) {
        if (cudaFuncSetAttribute(csr_plan_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kPlanMaxL * sizeof(uint32_t))) != cudaSuccess ||
            cudaFuncSetAttribute(csr_plan_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kPlanMaxL * sizeof(uint32_t))) != cudaSuccess)
            return fail("sfb_csr_attention: cannot reserve %u bytes of shared memory", kPlanMaxL * 4u);
        once.mark(dev);
    }
    launch_overlapped(dtype != SFB_F32 && d == 128 ? csr_plan_kernel<true> : csr_plan_kernel<false>, dim3(tiles), dim3(kPlanThreads), L * sizeof(uint32_t), s, rowptr, colidx, L, nnz, entries, counts, counts + kCsrCounts * tiles);
    const CsrTileArgs a = {entries, counts, counts + kCsrCounts * tiles, rowptr, colidx, nnz, q, k, v, o, L, H, tiles, B * H, scale * 1.4426950408889634f, bad};
    if (dtype == SFB_F32) return csr_tile_f32(s, a, B, d);
#define CSR_TILE(BF) return d == 32 ? launch_csr_tile<BF, 32>(s, a, B) : d == 64 ? launch_csr_tile<BF, 64>(s, a, B) : launch_csr_tile<BF, 128>(s, a, B)
    if (dtype == SFB_BF16) CSR_TILE(true);
    CSR_TILE(false);
#undef CSR_TILE
}

int csr_from_layout(cudaStream_t s, const uint8_t *layout, uint32_t nb, uint32_t bs, int32_t *rowptr, int32_t *colidx)
{
    csr_from_layout_kernel<<<nb, 256, nb * sizeof(uint32_t), s>>>(layout, nb, bs, rowptr, colidx);
    return check_launch("sfb_csr_from_layout");
}

int csr_attention(cudaStream_t s, const int32_t *rowptr, const int32_t *colidx, const void *q, const void *k, const void *v, void *o,
                  int dtype, uint32_t B, uint32_t L, uint32_t H, uint32_t d, float scale, uint32_t *bad)
{
    if (bad) cudaMemsetAsync(bad, 0, sizeof(uint32_t), s);
    const dim3 grid((L + 3) / 4, B, H);
    const float sl = scale * 1.4426950408889634f;
#define CSR_BY_D(DTV)                                                                                                               \
    do {                                                                                                                            \
        if (d == 32) csr_attention_split_kernel<DTV, 32, 4><<<grid, 128, 0, s>>>(rowptr, colidx, q, k, v, o, L, H, sl, bad);         \
        else if (d == 64) csr_attention_split_kernel<DTV, 64, 4><<<grid, 128, 0, s>>>(rowptr, colidx, q, k, v, o, L, H, sl, bad);    \
        else csr_attention_split_kernel<DTV, 128, 4><<<grid, 128, 0, s>>>(rowptr, colidx, q, k, v, o, L, H, sl, bad);                \
    } while (0)
    if (dtype == SFB_F32) CSR_BY_D(SFB_F32);
    else if (dtype == SFB_BF16) CSR_BY_D(SFB_BF16);
    else CSR_BY_D(SFB_F16);
#undef CSR_BY_D
    return check_launch("sfb_csr_attention");
}

}  // namespace sfb

extern "C" int sfb_csr_from_layout(sfb_stream_t stream, const uint8_t *layout, uint32_t nb, uint32_t block_size, int32_t *rowptr,
                                   int32_t *colidx)
{
    SFB_REQUIRE(layout && rowptr && colidx, "sfb_csr_from_layout: NULL pointer");
    SFB_REQUIRE(nb >= 1 && nb <= 4096 && block_size >= 1 && block_size <= 128, "sfb_csr_from_layout: bad nb=%u block_size=%u", nb, block_size);
    SFB_REQUIRE((uint64_t)nb * nb * block_size * block_size < (1ull << 31), "sfb_csr_from_layout: the pattern may exceed 2^31 entries");
    return sfb::csr_from_layout((cudaStream_t)stream, layout, nb, block_size, rowptr, colidx);
}

static int csr_check(const char *who, const int32_t *rowptr, const int32_t *colidx, const void *q, const void *k, const void *v, void *o,
                     int dtype, uint32_t batch_dim, uint32_t head_dim, uint32_t state_dim)
{
    SFB_REQUIRE(rowptr && colidx && q && k && v && o, "%s: NULL pointer", who);
    SFB_REQUIRE(dtype == SFB_F32 || dtype == SFB_BF16 || dtype == SFB_F16, "%s: unknown dtype", who);
    SFB_REQUIRE(state_dim == 32 || state_dim == 64 || state_dim == 128, "%s: state_dim %u not supported (32, 64 or 128)", who, state_dim);
    SFB_REQUIRE(batch_dim >= 1 && batch_dim <= 65535 && head_dim >= 1 && head_dim <= 65535, "%s: bad batch_dim=%u head_dim=%u", who, batch_dim, head_dim);
    SFB_REQUIRE((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o) & 15) == 0, "%s: q, k, v, o must be 16-byte aligned", who);
    return 0;
}

extern "C" int sfb_csr_attention(sfb_stream_t stream, const int32_t *rowptr, const int32_t *colidx, const void *q, const void *k,
                                 const void *v, void *o, int dtype, uint32_t batch_dim, uint32_t seq_len, uint32_t head_dim,
                                 uint32_t state_dim, float scale, uint32_t *bad_columns)
{
    if (csr_check("sfb_csr_attention", rowptr, colidx, q, k, v, o, dtype, batch_dim, head_dim, state_dim)) return 1;
    if (seq_len == 0) { sfb::clear_error(); return 0; }
    return sfb::csr_attention((cudaStream_t)stream, rowptr, colidx, q, k, v, o, dtype, batch_dim, seq_len, head_dim, state_dim, scale,
                              bad_columns);
}

extern "C" uint64_t sfb_csr_workspace(uint32_t nnz, uint32_t seq_len)
{
    return seq_len <= sfb::kPlanMaxL ? (uint64_t)sfb::csr_workspace(nnz, seq_len) : 0;
}

extern "C" int sfb_csr_attention_planned(sfb_stream_t stream, const int32_t *rowptr, const int32_t *colidx, uint32_t nnz, const void *q,
                                         const void *k, const void *v, void *o, int dtype, uint32_t batch_dim, uint32_t seq_len,
                                         uint32_t head_dim, uint32_t state_dim, float scale, uint32_t *bad_columns, void *workspace)
{
    const char *who = "sfb_csr_attention_planned";
    if (csr_check(who, rowptr, colidx, q, k, v, o, dtype, batch_dim, head_dim, state_dim)) return 1;
    SFB_REQUIRE(workspace && ((uintptr_t)workspace & 15) == 0, "%s: workspace is NULL or not 16-byte aligned", who);
    SFB_REQUIRE(seq_len <= sfb::kPlanMaxL, "%s: seq_len %u > %u", who, seq_len, sfb::kPlanMaxL);
    SFB_REQUIRE(nnz < (1u << 31), "%s: too many elements", who);
    if (seq_len == 0) { sfb::clear_error(); return 0; }
    return sfb::csr_attention_planned((cudaStream_t)stream, rowptr, colidx, nnz, q, k, v, o, dtype, batch_dim, seq_len, head_dim, state_dim, scale,
                                      bad_columns, workspace);
}
