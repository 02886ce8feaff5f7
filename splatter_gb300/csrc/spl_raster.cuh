// What the rasteriser and its backward share (sm_103a): batches of a tile's records and the masks of the pixels
// that each record may draw.
#pragma once
#include "spl_device.cuh"

namespace spl {

constexpr int RASTER_BATCH = 256;
constexpr int RASTER_WORDS = RASTER_BATCH / 32;
constexpr uint32_t RASTER_CTAS = 6;  // of k_raster per SM
constexpr float RASTER_NEAR_MARGIN = 9.0f;  // up to this margin a covered pixel's exponent stays above -87

// Two float operations per instruction on packed pairs (the results of the scalar operations, each rounded
// to nearest).  The assembler contracts a packed product and a packed sum that takes it into a packed fma
// even where plain contraction is off, so a product that is to be rounded before a sum is a product with a
// zero addend (fma2, the same value for a non-negative product) or its sum is scalar.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mul.rn.f32x2 d, a, b; mov.b64 {%0, %1}, d;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; add.rn.f32x2 d, a, b; mov.b64 {%0, %1}, d;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{.reg .b64 a, b, c, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %7}; "
        "fma.rn.f32x2 d, a, b, c; mov.b64 {%0, %1}, d;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// The CTA's tile and its pair range: the next entry of the tile order, or row-major without one.
__device__ __forceinline__ void ordered_tile(const uint2* ranges, const uint4* tile_order, uint2& range, int& tile) {
    if (tile_order) {
        const uint4 e = __ldg(tile_order + blockIdx.x);
        range = make_uint2(e.x, e.y);
        tile = (int)e.z;
    } else {
        range = __ldg(ranges + blockIdx.x);
        tile = (int)blockIdx.x;
    }
}

// Highest set bit of x (x != 0).
__device__ __forceinline__ uint32_t top_bit(uint32_t x) {
    uint32_t r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}

// Columns a .. b - 1 of a row of 16 as a bit mask (a, b <= 16, in their low five bits; empty when a >= b).
__device__ __forceinline__ uint32_t row_columns(uint32_t a, uint32_t b) {
    return __funnelshift_l(0u, 0xFFFFu, a) & ~__funnelshift_l(0u, 0xFFFFFFFFu, b) & 0xFFFFu;
}

// Slots of a batch of n records whose masks are listed: a whole number of list words, 1, 2, 4 or 8 of them, so that
// short lists, which most tiles of a frame have (5018 of 8160 tiles up to 32 records, 45 on average, for 1M splats at
// 1080p), take no more transposes than their records need.  With the barrier after the last batch left out: frames of 1M
// splats 181.2 -> 177.7 us, 24 served frames 2,237 -> 2,203 us, a training step 2,712 -> 2,691 us, 6M splats the same.
// Slower: short batches staged by two to eight threads a record, each for some of the strips (object 92.2 for 91.5 us).
__device__ __forceinline__ uint32_t listed_slots(uint32_t n) {
    return n <= 32u ? 32u : (n <= 64u ? 64u : (n <= 128u ? 128u : (uint32_t)RASTER_BATCH));
}

// The pixels that a record with first three words r0, r1, r2 may draw in the tile at (wx0, ty0), as
// s_pm[strip][slot]: strip w is the rows 2w, 2w + 1, the low half of its word the columns of the first.  Rows
// that the record misses are left as they are (zero).
template <bool RECT>
__device__ __forceinline__ void mask_rows(uint32_t (&s_pm)[8][RASTER_BATCH], uint32_t slot, float4 r0, float4 r1, float4 r2,
                                          int wx0, int ty0, float margin) {
    // The record's lane mask for each of the tile's eight strips (rows 2w, 2w + 1), one 16-bit half
    // per row: the pixels inside its pixel box and, for rectangles, only those whose centre may lie in
    // the rectangle: along a row tc is c + x A, so |c + x A| <= T is the interval (-c +- T) / A of
    // columns x.  T is the margin widened by a rounding bound far above the errors of the
    // per-pixel FMA chains and of this arithmetic (1e-6 of each term of c and of T itself), the
    // interval by another 1e-3 columns.  Pixels left out are not drawn by the record: the image
    // is unchanged.
    const uint32_t lo = __float_as_uint(r1.w), hi = __float_as_uint(r2.w);
    const int x0 = (int)(lo & 0xFFFFu), y0 = (int)(lo >> 16);
    const int x1 = (int)(hi & 0xFFFFu), y1 = (int)(hi >> 16);
    if (x0 <= x1 && y0 <= y1) {
        const int ra = max(y0 - ty0, 0), rb = min(y1 - ty0, 15);  // the box's rows and columns here
        const uint32_t box = row_columns((uint32_t)max(x0 - wx0, 0), (uint32_t)min(x1 - wx0, 15) + 1u);
        float2 c = make_float2(0.0f, 0.0f), step = c, half = make_float2(1e9f, 1e9f);
        if (RECT) {
            // column 0 of row ra; row after row the interval's centre moves by step
            const float Xc = (float)wx0 + 0.5f, Yc = (float)(ty0 + ra) + 0.5f;
            const float Xm = (float)(wx0 + 16), Ym = (float)(ty0 + 16);
            if (fabsf(r0.x) > 1e-30f) {
                const float s = -1.0f / r0.x;
                const float T = margin + 1e-6f * (fabsf(r0.x) * Xm + fabsf(r0.y) * Ym + fabsf(r0.z) + margin);
                c.x = fmaf(r0.y, Yc, fmaf(r0.x, Xc, r0.z)) * s;
                step.x = r0.y * s;
                half.x = T * fabsf(s) + 1e-3f;
            }
            if (fabsf(r0.w) > 1e-30f) {
                const float s = -1.0f / r0.w;
                const float T = margin + 1e-6f * (fabsf(r0.w) * Xm + fabsf(r1.x) * Ym + fabsf(r1.y) + margin);
                c.y = fmaf(r1.x, Yc, fmaf(r0.w, Xc, r1.y)) * s;
                step.y = r1.x * s;
                half.y = T * fabsf(s) + 1e-3f;
            }
        }
        for (int row = ra; row <= rb; ++row) {
            uint32_t m = box;
            if (RECT) {
                const float k = (float)(row - ra);
                const float2 q = fma2(make_float2(k, k), step, c);
                const float2 qa = add2(q, make_float2(-half.x, -half.y)), qb = add2(q, half);
                // first column: the bound rounded up; one past the last: rounded down, plus one
                const float fa = fminf(fmaxf(fmaxf(qa.x, qa.y), 0.0f), 16.0f);
                const float fb = fmaxf(fminf(fminf(qb.x, qb.y), 15.0f), -1.0f);
                m &= row_columns(__float_as_uint(__fadd_ru(fa, 8388608.0f)),
                                 __float_as_uint(__fadd_rd(fb, 8388609.0f)));
            }
            // Strip row / 2, half row & 1.  Copied as bytes: an assignment through a pointer to 16-bit words might be
            // moved before the caller's clearing of the 32-bit words or after their use (g++ does).  Both rows of a
            // strip in one 32-bit store, which takes a branch per row, is slower: frames of 100k splats 86.5 -> 88.4
            // us, 1M 174.6 -> 181.4 us, 6M at 2160p 1,521 -> 1,578 us.
            const uint16_t half_word = (uint16_t)m;
            memcpy(__builtin_assume_aligned(reinterpret_cast<unsigned char*>(&s_pm[row >> 1][slot]) + 2 * (row & 1), 2), &half_word,
                   2);
        }
    }
}

}  // namespace spl
