// The matmul core of the kernels on fp32 operands (and of every shape that the tcgen05 kernels do not take): 128 threads =
// four warps, each of which owns a 32-row tile of the product and walks the contraction 32 elements ("a chunk") at a time,
// on warp-level tensor-core instructions.
//
// fp32 products on bf16 operands.  An fp32 number is the sum of three bf16 numbers, x = h + m + l (8 + 8 + 8 bits, each
// rounded from what the one before left), exact down to 2^-109; of a smaller number a multiple of 2^-133 is left (the last place
// of the smallest bf16 numbers), so its products are off by up to 2^-134 of the other factor.  x * y is then six products of them,
// hh + hm + mh + hl + mm + lh, up to 2^-24 of it.  The tensor core's products are exact and its sums truncate (measured: an aligned addend keeps one bit
// below the last place), which over a long contraction is a bias; so the small products go first, and every 16 elements of
// the contraction are summed from zero and added to the fp32 accumulator by rounded additions.  Measured relative error of
// scores against 64 bits at d = 32 / 64 / 128: 5.5e-8 / 6.3e-8 / 7.4e-8; two FMA chains, as the thread tiles before this had
// them, 7.9e-8 / 1.07e-7 / 1.47e-7; two tf32 terms and three products 9.9e-8 / 1.04e-7 / 1.10e-7 at the same tensor time.
// bf16 operands are one term, fp16 operands two (8 + 3 bits), both exact.
//
// Why.  An SM makes 1024 bf16 products per clock by mma.sync (measured), a sixth of that is 170 fp32 products against the 128
// of the FMA pipe, of which thread tiles of 4 x 8 outputs reached half, being bound by issue slots and shared memory: an MMA
// is one issue slot for 2048 products.  What is left to issue is the split (22 slots for four elements), so an operand that
// several warps use is split once: the queries when they arrive, the probabilities where they are made, both kept
// in shared memory as fragments.
//
// What is not finite.  inf splits into inf and inf - inf, so products with it come out as NaN, as do those with a finite number
// that rounds to a bf16 infinity; callers make every result that is not finite again with plain FMAs, a tile at a time (fma_again below,
// fma_tile.cuh).  A call whose every result is NaN takes two to five times as long as one on finite operands (SDDMM 2.4 to 3.8, SpMM
// 2.2 to 3.8, attention 3.1 to 4.6, blocks of 32 and 64, d 64 and 128); element by element, and a row per warp, it took 7 to 70 times as long.
//
// Keys and values travel by cp.async through rings of chunks, and only as far as the warps that use them: a team (one warp, or
// the two that share columns) stages its own keys and its own columns of the values, and waits for nobody else.
#pragma once
#include "attn.cuh"

namespace sfb {
namespace tile {

constexpr uint32_t kThreads = 128;
constexpr uint32_t kChunk = 32;               // elements of the contraction per chunk
constexpr uint32_t kStride = kChunk + 4;      // row stride, in floats, of a tile whose rows are one chunk long

// Row r of a staged tile lies at tile_row(r): inside each group of 16 the two bit pairs are swapped.  Fragments are read as 16
// bytes along a row, eight lanes at a time from rows r and r + 1 (keys of the scores), or from rows 0, 4, 8, 12 of a group
// (values).  With the swap the first are four rows apart, which at a stride of 4 mod 32 words are different banks,
// and the second are neighbours, different banks at 8 mod 32.
__device__ __host__ __forceinline__ constexpr uint32_t tile_row(uint32_t r) { return (r & ~15u) | ((r >> 2) & 3u) | ((r & 3u) << 2); }

__device__ __forceinline__ void cp_async16(float *dst, const void *src, uint32_t bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst, const void *src, uint32_t bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// THREADS threads (whole warps) meet; id: 1 to 15, the same for all of them and nobody else at the time
template <int THREADS> __device__ __forceinline__ void meet(uint32_t id)
{
    if (THREADS == 32) __syncwarp();
    else if (THREADS == (int)kThreads) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}

// 16-byte piece of a 16-bit type -> eight floats
template <int DT> __device__ __forceinline__ void widen2(float &a, float &b, uint32_t w)
{
    if (DT == SFB_BF16) {
        a = __uint_as_float(w << 16);
        b = __uint_as_float(w & 0xffff0000u);
    } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w));
        a = f.x;
        b = f.y;
    }
}

// 32 rows x COLS elements -> dst[tile_row(r) * stride + c] as fp32, by a team of TT threads (rank: this thread's place in it);
// element (r, c) is src[at + r * pitch + c]; columns from ncols on are zeros.  vec: 16-byte aligned rows (ncols then is a
// multiple of a 16-byte piece).  A thread keeps its piece of the row and steps down the rows.  STEP is a power of two, so
// tile_row(r0 + i * STEP) is tile_row(r0) + tile_row(i * STEP).
// In two halves: stage_begin asks for everything (fp32 pieces by cp.async straight to where they belong), stage_end
// converts the 16-bit pieces that have waited in registers meanwhile.
template <int DT, int TT, int COLS> struct Staged {
    static constexpr int E = DT == SFB_F32 ? 4 : 8;                       // elements per 16-byte piece
    static constexpr int P = COLS / E, STEP = TT / P;                      // pieces per row, rows per step
    static constexpr int N = (32 + STEP - 1) / STEP;
    static_assert(TT % P == 0, "a row's pieces divide the team");
    uint4 held[DT == SFB_F32 ? 1 : N];
};
template <int DT, int TT, int COLS>
__device__ __forceinline__ void stage_begin(Staged<DT, TT, COLS> &st, uint32_t rank, float *dst, uint32_t stride, const void *src, size_t at, size_t pitch,
                                            uint32_t ncols, bool vec)
{
    typedef Staged<DT, TT, COLS> S;
    if (vec) {
        const uint32_t r0 = rank / S::P, c = (rank % S::P) * S::E;
        const bool in = c < ncols;
        if (DT == SFB_F32) {
            float *d = dst + tile_row(r0) * stride + c;
            const float *q = (const float *)src + at + r0 * pitch + (in ? c : 0);
            const uint32_t bytes = in ? 16u : 0u;
#pragma unroll
            for (int i = 0; i < S::N; i++)
                if (32 % S::STEP == 0 || r0 + i * S::STEP < 32) cp_async16(d + tile_row(i * S::STEP) * stride, q + (size_t)i * S::STEP * pitch, bytes);
        } else {
            const uint16_t *q = (const uint16_t *)src + at + r0 * pitch + c;
#pragma unroll
            for (int i = 0; i < S::N; i++) {
                uint4 u = make_uint4(0u, 0u, 0u, 0u);
                if (in && (32 % S::STEP == 0 || r0 + i * S::STEP < 32)) u = __ldg((const uint4 *)(q + (size_t)i * S::STEP * pitch));
                st.held[DT == SFB_F32 ? 0 : i] = u;
            }
        }
    } else {
        uint32_t first = rank;
        // Nothing of this is worked out ahead and kept in registers that the aligned rows need (SpMM, bf16 blocks of 32, fp32, d 128, BigBird
        // rows 163 us otherwise, 135 so).  For 16-bit operands the unrolled loads count: attention at block 64, d 30 416 us against 792,
        // but fp16 SpMM at d 128 up to 10 % longer.
        asm volatile("" : "+r"(first));
#pragma unroll 8
        for (uint32_t t = first; t < 32 * COLS; t += TT) {
            const uint32_t r = t / COLS, c = t % COLS;
            float *d = dst + tile_row(r) * stride + c;
            if (DT == SFB_F32) cp_async4(d, (const float *)src + at + (c < ncols ? r * pitch + c : 0), c < ncols ? 4u : 0u);
            else *d = c < ncols ? Elem<DT>::load(src, at + r * pitch + c) : 0.f;
        }
    }
}
template <int DT, int TT, int COLS>
__device__ __forceinline__ void stage_end(const Staged<DT, TT, COLS> &st, uint32_t rank, float *dst, uint32_t stride, bool vec)
{
    typedef Staged<DT, TT, COLS> S;
    if (DT == SFB_F32 || !vec) return;
    const uint32_t r0 = rank / S::P, c = (rank % S::P) * S::E;
    float *d = dst + tile_row(r0) * stride + c;
#pragma unroll
    for (int i = 0; i < S::N; i++)
        if (32 % S::STEP == 0 || r0 + i * S::STEP < 32) {
            const uint4 u = st.held[DT == SFB_F32 ? 0 : i];
            float v[8];
            widen2<DT>(v[0], v[1], u.x);
            widen2<DT>(v[2], v[3], u.y);
            widen2<DT>(v[4], v[5], u.z);
            widen2<DT>(v[6], v[7], u.w);
            *(float4 *)(d + tile_row(i * S::STEP) * stride) = make_float4(v[0], v[1], v[2], v[3]);
            *(float4 *)(d + tile_row(i * S::STEP) * stride + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
}

// four neighbouring elements on their way to a fragment, unconverted
template <int DT> struct Raw4 { uint2 w; };
template <> struct Raw4<SFB_F32> { float4 w; };
template <int DT>
__device__ __forceinline__ void load_raw4(Raw4<DT> &r, const void *p, size_t at, uint32_t n, bool vec)      // n: how many of them exist
{
    if (vec) {
        if (n) r.w = __ldg((const decltype(r.w) *)((const typename Elem<DT>::type *)p + at));
        else r.w = decltype(r.w){};
    } else {
        typename Elem<DT>::type e[4] = {};
#pragma unroll
        for (uint32_t i = 0; i < 4; i++)
            if (i < n) e[i] = ((const typename Elem<DT>::type *)p)[at + i];
        memcpy(&r.w, e, sizeof r.w);
    }
}
template <int DT>
__device__ __forceinline__ void widen4(float (&x)[4], const Raw4<DT> &r)
{
    if constexpr (DT == SFB_F32) {
        x[0] = r.w.x; x[1] = r.w.y; x[2] = r.w.z; x[3] = r.w.w;
    } else {
        widen2<DT>(x[0], x[1], r.w.x);
        widen2<DT>(x[2], x[3], r.w.y);
    }
}

// ---- products
template <int DT> constexpr int kTerms = DT == SFB_F32 ? 3 : DT == SFB_F16 ? 2 : 1;      // bf16 numbers that an element is the sum of

// c (+)= a . b, 16 x 8 x 16.  Lane = 4 g + t.  a: (row g, slots 2t, 2t + 1), (g + 8, the same), (g, 2t + 8, 2t + 9), (g + 8, the same);
// b: (slots 2t, 2t + 1, column g), (2t + 8, 2t + 9, column g); c: (row g, columns 2t, 2t + 1), (g + 8, the same).  Which element of the contraction
// a slot is does not matter as long as a and b agree.
__device__ __forceinline__ void mma_zero(float (&c)[4], const uint4 &a, const uint32_t (&b)[2])
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void mma_add(float (&c)[4], const uint4 &a, const uint32_t (&b)[2])
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b[0]), "r"(b[1]));
}
// two rounded additions in one issue slot
__device__ __forceinline__ void add2(float &a0, float &a1, float b0, float b1)
{
    asm("{.reg .b64 a, b; mov.b64 a, {%0, %1}; mov.b64 b, {%2, %3}; add.rn.f32x2 a, a, b; mov.b64 {%0, %1}, a;}" : "+f"(a0), "+f"(a1) : "f"(b0), "f"(b1));
}
// a pair as T packed bf16 pairs
__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
template <int T>
__device__ __forceinline__ void split2(uint32_t (&w)[T], float a, float b)
{
    if constexpr (T == 1) {
        w[0] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);       // bf16 numbers: their upper halves
    } else {
#pragma unroll
        for (int i = 0; i < T; i++) {
            w[i] = pack2(a, b);
            if (i + 1 < T) {
                a -= __uint_as_float(w[i] << 16);
                b -= __uint_as_float(w[i] & 0xffff0000u);
            }
        }
    }
}
// four elements of the contraction: slots 2t, 2t + 1 and 2t + 8, 2t + 9
template <int T> struct Four { uint32_t w[T][2]; };
template <int T>
__device__ __forceinline__ void split4(Four<T> &f, const float (&x)[4])
{
    uint32_t lo[T], hi[T];
    split2<T>(lo, x[0], x[1]);
    split2<T>(hi, x[2], x[3]);
#pragma unroll
    for (int i = 0; i < T; i++) {
        f.w[i][0] = lo[i];
        f.w[i][1] = hi[i];
    }
}
// an A fragment (16 rows x 16 elements) per term
template <int T> struct Frag { uint4 w[T]; };
template <int T>
__device__ __forceinline__ void split_rows(Frag<T> &f, const float (&x0)[4], const float (&x1)[4])      // rows g and g + 8
{
    Four<T> a, b;
    split4<T>(a, x0);
    split4<T>(b, x1);
#pragma unroll
    for (int i = 0; i < T; i++) f.w[i] = make_uint4(a.w[i][0], b.w[i][0], a.w[i][1], b.w[i][1]);
}
// fragments in shared memory: a fragment's terms follow each other, 16 bytes per lane
template <int T> __device__ __forceinline__ void store_frag(uint4 *at, uint32_t lane, const Frag<T> &f)
{
#pragma unroll
    for (int i = 0; i < T; i++) at[i * 32 + lane] = f.w[i];
}
template <int T> __device__ __forceinline__ void load_frag(Frag<T> &f, const uint4 *at, uint32_t lane)
{
#pragma unroll
    for (int i = 0; i < T; i++) f.w[i] = at[i * 32 + lane];
}
// acc[n] += a . b[n], 16 elements of the contraction: small products first, from zero
template <int N, int TA, int TB>
__device__ __forceinline__ void mma16(float (*acc)[4], const Frag<TA> &a, const Four<TB> *b)
{
    constexpr int TOP = TA + TB - 2 < 2 ? TA + TB - 2 : 2;
    float t[N][4];
#pragma unroll
    for (int s = TOP; s >= 0; s--)
#pragma unroll
        for (int i = TA - 1; i >= 0; i--) {
            const int j = s - i;
            if (j < 0 || j >= TB) continue;
            const bool first = s == TOP && (i == TA - 1 || s - (i + 1) < 0);
#pragma unroll
            for (int n = 0; n < N; n++)
                if (first) mma_zero(t[n], a.w[i], b[n].w[j]);
                else mma_add(t[n], a.w[i], b[n].w[j]);
        }
#pragma unroll
    for (int n = 0; n < N; n++) {
        add2(acc[n][0], acc[n][1], t[n][0], t[n][1]);
        add2(acc[n][2], acc[n][3], t[n][2], t[n][3]);
    }
}

// Scores.  acc[m][j][2 * half + e] is row 16 m + 8 half + g and key score_key<WIDE>(t, j, e): a thread's keys of a row are two
// groups of four neighbours, which makes them (m, 2 j2), (m, 2 j2 + 1) the A fragment of keys 16 j2 to 16 j2 + 15 of the
// product with the values.  WIDE: eight neighbours, to be stored.
template <bool WIDE> __device__ __forceinline__ constexpr uint32_t score_key(uint32_t t, uint32_t j, uint32_t e)
{
    return WIDE ? 8 * t + 2 * j + e : 16 * (j >> 1) + 4 * t + 2 * (j & 1) + e;
}
// the keys b[j] over 16 elements (offset k) of the staged chunk at `keys`
template <int T, bool WIDE>
__device__ __forceinline__ void load_keys(Four<T> (&b)[4], const float *keys, uint32_t k, uint32_t g, uint32_t t)
{
    const float *p = keys + tile_row(score_key<WIDE>(g >> 1, 0, g & 1)) * kStride + 4 * t + k;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float4 v = *(const float4 *)(p + tile_row(score_key<WIDE>(0, j, 0)) * kStride);
        const float x[4] = {v.x, v.y, v.z, v.w};
        split4<T>(b[j], x);
    }
}

// Outputs: N n-tiles of 8 columns, in groups of up to four: a group is 8 x VN columns of which lane row g loads the VN neighbours
// from VN * g on, and of which a thread's accumulators hold the 2 VN neighbours from 2 VN t on.
template <int N> struct Cols { static constexpr int VN = N < 4 ? N : 4, GROUPS = N / VN; };
template <int VN>
__device__ __forceinline__ void load_cols(float (&v)[VN], const float *p)
{
    if constexpr (VN == 4) {
        const float4 q = *(const float4 *)p;
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else if constexpr (VN == 2) {
        const float2 q = *(const float2 *)p;
        v[0] = q.x; v[1] = q.y;
    } else {
        v[0] = *p;
    }
}
// the columns b[n] of one group over 16 elements of the contraction: element 4 t + i of them is row t + 4 i of the staged tile
template <int VN, int T>
__device__ __forceinline__ void load_values(Four<T> (&b)[VN], const float *v, uint32_t stride, uint32_t g, uint32_t t)
{
    float x[4][VN];
#pragma unroll
    for (int i = 0; i < 4; i++) load_cols<VN>(x[i], v + (t + 4 * i) * stride + VN * g);
#pragma unroll
    for (int n = 0; n < VN; n++) {
        const float y[4] = {x[0][n], x[1][n], x[2][n], x[3][n]};
        split4<T>(b[n], y);
    }
}
// acc += 32 rows of p, fragments [m][k16 of this chunk][term] (pitch: uint4 from one m to the next), times one staged chunk of values
template <int N, int TP, int TV>
__device__ __forceinline__ void mma_values(float (&acc)[2][N][4], const uint4 *p, uint32_t pitch, const float *v, uint32_t stride, uint32_t lane)
{
    constexpr int VN = Cols<N>::VN;
    const uint32_t g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
        for (int q = 0; q < Cols<N>::GROUPS; q++) {
            Four<TV> b[VN];
            load_values<VN, TV>(b, v + 16 * k * stride + 32 * q, stride, g, t);
#pragma unroll
            for (int m = 0; m < 2; m++) {
                Frag<TP> a;
                load_frag<TP>(a, p + m * pitch + k * TP * 32, lane);
                mma16<VN, TP, TV>(&acc[m][VN * q], a, b);
            }
        }
}
// stays 0 while every v is finite
template <int N>
__device__ __forceinline__ float zero_if_finite(const float (*v)[4], float z)
{
#pragma unroll
    for (int n = 0; n < N; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) z = fmaf(v[n][i], 0.f, z);
    return z;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// ---- results that are not finite, made again by plain FMAs: a warp's 32 rows, one per lane, times N columns, kAgain elements of the
// contraction at a time from shared memory (the rows' elements at a, the columns' at b, both with the contraction outermost: a lane's own
// element is one conflict-free load, four columns are one broadcast)
constexpr uint32_t kAgain = 16, kAgainRows = 33;
template <int N> constexpr uint32_t kAgainCols = N + 4;
constexpr uint32_t kAgainFloats = kAgain * (kAgainRows + kAgainCols<32>);
// ROWS x COLS elements on their way there, by one warp: element (r, c) = src[at + r * pitch + c] -> dst[r * ROW + c * COL]; columns from ncols on are zeros
template <int ROWS, int COLS> struct Again {
    float x[ROWS * COLS / 32];
    template <int DT> __device__ __forceinline__ void load(const void *src, size_t at, size_t pitch, uint32_t ncols, uint32_t lane)
    {
#pragma unroll
        for (int i = 0; i < ROWS * COLS / 32; i++) {
            const uint32_t r = (32 * i + lane) / COLS, c = (32 * i + lane) % COLS;
            x[i] = c < ncols ? Elem<DT>::load(src, at + r * pitch + c) : 0.f;
        }
    }
    template <int ROW, int COL> __device__ __forceinline__ void put(float *dst, uint32_t lane) const
    {
#pragma unroll
        for (int i = 0; i < ROWS * COLS / 32; i++) dst[(32 * i + lane) / COLS * ROW + (32 * i + lane) % COLS * COL] = x[i];
    }
};
template <int N>
__device__ __forceinline__ void fma_again(float (&acc)[N], const float *a, const float *b, uint32_t lane)
{
#pragma unroll 4
    for (uint32_t k = 0; k < kAgain; k++) {
        const float x = a[k * kAgainRows + lane];
#pragma unroll
        for (int n = 0; n < N; n += 4) {
            const float4 v = *(const float4 *)(b + k * kAgainCols<N> + n);
            acc[n] = fmaf(x, v.x, acc[n]);
            acc[n + 1] = fmaf(x, v.y, acc[n + 1]);
            acc[n + 2] = fmaf(x, v.z, acc[n + 2]);
            acc[n + 3] = fmaf(x, v.w, acc[n + 3]);
        }
    }
}
// scores of the rows at rowA, rowA + HD, ... and the keys at rowB, rowB + HD, ... (element offsets), d elements
template <int DT>
__device__ __forceinline__ void scores_again(float (&s)[32], float *buf, const void *A, const void *B, size_t rowA, size_t rowB, size_t HD, uint32_t d, uint32_t lane)
{
#pragma unroll
    for (int n = 0; n < 32; n++) s[n] = 0.f;
    Again<32, kAgain> x, y;
    x.template load<DT>(A, rowA, HD, d, lane);
    y.template load<DT>(B, rowB, HD, d, lane);
    for (uint32_t k = 0; k < d; k += kAgain) {
        __syncwarp();
        x.template put<1, kAgainRows>(buf, lane);
        y.template put<1, kAgainCols<32>>(buf + kAgain * kAgainRows, lane);
        __syncwarp();
        if (k + kAgain < d) {
            x.template load<DT>(A, rowA + k + kAgain, HD, d - k - kAgain, lane);
            y.template load<DT>(B, rowB + k + kAgain, HD, d - k - kAgain, lane);
        }
        fma_again<32>(s, buf, buf + kAgain * kAgainRows, lane);
    }
}

// the column of accumulator n of a row, e = 0 or 1
template <int N> __device__ __forceinline__ uint32_t out_col(uint32_t t, int n, int e)
{
    constexpr int VN = Cols<N>::VN;
    return 32 * (n / VN) + VN * (2 * t + e) + n % VN;
}
// One output row (half 0 or 1 of acc[n]), times mul -> row (element offset of the warp's first column), columns from ncols on not written
template <int DT, int N>
__device__ __forceinline__ void store_cols(void *out, size_t row, uint32_t t, const float (*acc)[4], int half, float mul, uint32_t ncols, bool vec)
{
    constexpr int VN = Cols<N>::VN;
#pragma unroll
    for (int q = 0; q < Cols<N>::GROUPS; q++) {
        float v[2 * VN];
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
            for (int n = 0; n < VN; n++) v[e * VN + n] = acc[VN * q + n][2 * half + e] * mul;
        const uint32_t c = 32 * q + 2 * VN * t;
        if (vec && VN >= 2) {
#pragma unroll
            for (int j = 0; j < 2 * VN; j += 4) {
                if (c + j < ncols) {
                    const float w0 = v[j], w1 = v[(j + 1) % (2 * VN)], w2 = v[(j + 2) % (2 * VN)], w3 = v[(j + 3) % (2 * VN)];
                    if (DT == SFB_F32) {
                        *(float4 *)((float *)out + row + c + j) = make_float4(w0, w1, w2, w3);
                    } else {
                        uint2 w;
                        if (DT == SFB_BF16) {
                            w.x = to_bhalf_bits(w0) | ((uint32_t)to_bhalf_bits(w1) << 16);
                            w.y = to_bhalf_bits(w2) | ((uint32_t)to_bhalf_bits(w3) << 16);
                        } else {
                            __half2 h0 = __floats2half2_rn(w0, w1), h1 = __floats2half2_rn(w2, w3);
                            w.x = *reinterpret_cast<uint32_t *>(&h0);
                            w.y = *reinterpret_cast<uint32_t *>(&h1);
                        }
                        *(uint2 *)((uint16_t *)out + row + c + j) = w;
                    }
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 2 * VN; j++)
                if (c + j < ncols) Elem<DT>::store(out, row + c + j, v[j]);
        }
    }
}

}  // namespace tile
}  // namespace sfb
