// What the plan of an element-sparse pattern hands to the tile kernels (csr.cu, attn_simt.cu), and one row of it by one warp.
#pragma once
#include "common.cuh"

namespace sfb {

constexpr uint32_t kCsrCounts = 6;
struct CsrTileArgs {
    const uint2 *entries;            // (column, mask of the tile's rows that have it)
    // per tile: [distinct columns, entries of columns named twice, first entry, behind the last; for 16-bit operands with
    // d 128: distinct columns of the first 16 rows alone, of the last 16 alone], bad columns
    const uint32_t *counts, *bad;
    const int32_t *rowptr, *colidx;  // the pattern itself: nnz elements
    uint32_t nnz;
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

// 16-byte pieces -> floats, by element type
template <int DT> struct Piece;
template <> struct Piece<SFB_F32> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(float *v, const uint4 &t)
    {
        v[0] = __uint_as_float(t.x); v[1] = __uint_as_float(t.y); v[2] = __uint_as_float(t.z); v[3] = __uint_as_float(t.w);
    }
};
template <> struct Piece<SFB_BF16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(float *v, const uint4 &t)
    {
        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 4; j++) { v[2 * j] = __uint_as_float(w[j] << 16); v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u); }
    }
};
template <> struct Piece<SFB_F16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(float *v, const uint4 &t)
    {
        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 4; j++) { const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[j])); v[2 * j] = f.x; v[2 * j + 1] = f.y; }
    }
};

// Query row i of (batch b, head h) over the elements lo to hi - 1 of colidx: one warp, LPK lanes per key, each owning a share of the head dimension; the key's K and V pieces are all
// requested before the first is used.  The lanes of a key join their partial scores by shuffles and carry the same running
// max and sum; the groups' softmaxes are merged at the end.  A score of -inf is a weight of 0, also while nothing else has
// been met; one of +inf makes the row NaN.
template <int DT, int D, int LPK>
__device__ __forceinline__ void csr_row(const int32_t *__restrict__ colidx, int32_t lo, int32_t hi, const void *__restrict__ Q, const void *__restrict__ K,
                                        const void *__restrict__ V, void *__restrict__ O, uint32_t L, uint32_t H, uint32_t b, uint32_t h, uint32_t i,
                                        float scale_log2e, uint32_t *bad)
{
    constexpr int HD2 = D / LPK;                     // elements per lane
    constexpr int KPI = 32 / LPK;                    // keys per warp and step
    constexpr int NP = HD2 / Piece<DT>::N;           // 16-byte pieces per lane and operand
    constexpr int ESZ = 16 / Piece<DT>::N;
    const uint32_t lane = threadIdx.x & 31, hp = lane % LPK, pi = lane / LPK;
    const size_t HD = (size_t)H * D;
    const size_t row_off = ((size_t)b * L + i) * HD + (size_t)h * D + hp * HD2;
    float q[HD2], acc[HD2];
    {
        const uint4 *src = (const uint4 *)((const uint8_t *)Q + row_off * ESZ);
#pragma unroll
        for (int n = 0; n < NP; n++) Piece<DT>::unpack(q + n * Piece<DT>::N, __ldg(src + n));
    }
    if (scale_log2e < 0.f) {                         // the largest score is the one that counts, so the sign goes to the query
        scale_log2e = -scale_log2e;
#pragma unroll
        for (int x = 0; x < HD2; x++) q[x] = -q[x];
    }
#pragma unroll
    for (int x = 0; x < HD2; x++) acc[x] = 0.f;
    float m = -INFINITY, l = 0.f;
    for (int32_t base = lo; base < hi; base += KPI) {          // the same trip count for every lane: the shuffle below is full-warp
        const int32_t e = base + (int32_t)pi;
        bool valid = e < hi;
        int32_t j = 0;
        if (valid) {
            j = __ldg(colidx + e);
            if (j < 0 || (uint32_t)j >= L) {                   // a column outside the sequence: counted once, not read
                if (bad && hp == 0) atomicAdd(bad, 1u);
                valid = false;
            }
        }
        uint4 kr[NP], vr[NP];
        if (valid) {
            const size_t key_off = (((size_t)b * L + (uint32_t)j) * HD + (size_t)h * D + hp * HD2) * ESZ;
            const uint4 *ks = (const uint4 *)((const uint8_t *)K + key_off), *vs = (const uint4 *)((const uint8_t *)V + key_off);
#pragma unroll
            for (int n = 0; n < NP; n++) kr[n] = __ldg(ks + n);
#pragma unroll
            for (int n = 0; n < NP; n++) vr[n] = __ldg(vs + n);
        }
        float part = 0.f;
        if (valid) {
#pragma unroll
            for (int n = 0; n < NP; n++) {
                float t[Piece<DT>::N];
                Piece<DT>::unpack(t, kr[n]);
#pragma unroll
                for (int x = 0; x < Piece<DT>::N; x++) part = fmaf(q[n * Piece<DT>::N + x], t[x], part);
            }
        }
        float sc = part;
#pragma unroll
        for (int o = 1; o < LPK; o <<= 1) sc += __shfl_xor_sync(0xffffffffu, sc, o);
        if (valid) {
            if (sc > m) {
                const float f = exp2f((m - sc) * scale_log2e);   // 0 on the first key
                l *= f;
#pragma unroll
                for (int x = 0; x < HD2; x++) acc[x] *= f;
                m = sc;
            }
            const float p = exp2f((sc - (m > -INFINITY ? m : 0.f)) * scale_log2e);
            l += p;
#pragma unroll
            for (int n = 0; n < NP; n++) {
                float t[Piece<DT>::N];
                Piece<DT>::unpack(t, vr[n]);
#pragma unroll
                for (int x = 0; x < Piece<DT>::N; x++) acc[n * Piece<DT>::N + x] = fmaf(p, t[x], acc[n * Piece<DT>::N + x]);
            }
        }
    }
    // merge the groups' softmaxes (the LPK lanes of a group hold the same max and sum: offsets from LPK on)
    float M = m;
#pragma unroll
    for (int o = 16; o >= LPK; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    const float f = m > -INFINITY ? exp2f((m - M) * scale_log2e) : 0.f;
    l *= f;
#pragma unroll
    for (int o = 16; o >= LPK; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const float inv = l > 0.f ? 1.f / (l + 1e-6f) : 0.f;   // the reference's denominator (ewops.h:93, cuda_kernels.h:1022)
#pragma unroll
    for (int x = 0; x < HD2; x++) {
        float a = acc[x] * f;
#pragma unroll
        for (int o = 16; o >= LPK; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        // every lane with this share of the head holds the element now; group x % KPI writes it
        if ((x % KPI) == (int)pi) Elem<DT>::store(O, row_off + x, a * inv);
    }
}

// The same for a row of a tile whose output is not finite.  The tile kernels multiply the values of all of a tile's columns with
// every row's probabilities, which are 0 where the row does not have the column: an infinity or a NaN among the values of a
// column then reaches rows that do not have it (0 * inf), and must not.  Such rows are made again on their own columns.  Not
// inlined: the tile kernels' registers are for the tiles; arguments one by one: with the kernel's parameters passed by their
// address every read of them in the kernel got slower (D 128 139.5 -> 145 us on a block pattern).
template <int DT, int D>
__device__ __noinline__ void csr_row_again(const int32_t *rowptr, const int32_t *colidx, uint32_t nnz, const void *Q, const void *K, const void *V,
                                           void *O, uint32_t L, uint32_t H, uint32_t b, uint32_t h, uint32_t i, float scale_log2e)
{
    const int32_t lo = max(rowptr[i], 0), hi = (int32_t)min((uint32_t)max(rowptr[i + 1], 0), nnz);
    csr_row<DT, D, 4>(colidx, lo, hi, Q, K, V, O, L, H, b, h, i, scale_log2e, nullptr);
}

int csr_tile_f32(cudaStream_t s, const CsrTileArgs &a, uint32_t B, uint32_t d);     // attn_simt.cu

}  // namespace sfb
