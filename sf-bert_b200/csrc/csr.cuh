// What the plan of an element-sparse pattern hands to the tile kernels (csr.cu, attn_simt.cu).
#pragma once
#include "common.cuh"

namespace sfb {

constexpr uint32_t kCsrCounts = 6;
struct CsrTileArgs {
    const uint2 *entries;            // (column, mask of the tile's rows that have it)
    // per tile: [distinct columns, entries of columns named twice, first entry, behind the last; for 16-bit operands with
    // d 128: distinct columns of the first 16 rows alone, of the last 16 alone], bad columns
    const uint32_t *counts, *bad;
    const void *Q, *K, *V;
    void *O;
    uint32_t L, H, tiles, BH;
    float scale_log2e;
    uint32_t *bad_out;
};
// entry i of a tile's list: the distinct columns, then (from the end of the tile's share backwards) the ones named twice
__device__ __forceinline__ uint2 csr_entry(const uint2 *entries, uint32_t base, uint32_t top, uint32_t distinct, uint32_t i)
{
    return __ldg(entries + (i < distinct ? base + i : top - 1u - (i - distinct)));
}
// the first CTA writes the number of columns outside the sequence, once per (batch, head) as every one of them meets it
__device__ __forceinline__ void csr_write_bad(const CsrTileArgs &a)
{
    if (blockIdx.x || blockIdx.y || blockIdx.z || !a.bad_out || threadIdx.x >= 32) return;
    uint32_t n = 0;
    for (uint32_t t = threadIdx.x; t < a.tiles; t += 32) n += a.bad[t];
    n = __reduce_add_sync(0xffffffffu, n);
    if (threadIdx.x == 0) *a.bad_out = n * a.BH;
}

int csr_tile_f32(cudaStream_t s, const CsrTileArgs &a, uint32_t B, uint32_t d);     // attn_simt.cu

}  // namespace sfb
