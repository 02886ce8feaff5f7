// Device-side building blocks shared by the splat-pipeline kernels (sm_103a).
//
// Floating point: every translation unit is compiled with -fmad=false and IEEE division/sqrt, so
// the FP32 results follow the written operation order exactly (the WGSL order of
// Lichtso/splatter src/shaders.wgsl).  Where a fused multiply-add is wanted it is written as
// fmaf() explicitly.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "spl_types.h"

namespace spl {

constexpr uint32_t FULL_MASK = 0xFFFFFFFFu;

// ------------------------------------------------------------------------------------------------
// A frame's kernels, and those of its backward, are launched with programmatic dependence (launch_after): a kernel's blocks may start when
// every block of the kernel before it has ended or called start_next, instead of after a full launch latency.
// Every kernel but one calls frame_step before it touches memory: it waits until the kernel before has ended and its
// writes are visible (at once, where a kernel is launched plainly), so a kernel sees all kernels before it
// complete.  The exception is the vertex stage beside the depth sort (below), which reads only what was complete before
// that sort began: a kernel between the two, or one more input of the vertex stage that the sort or a kernel between
// writes, would break it.  The pointers that it reads through the read-only path are given to frame_step: the compiler
// takes what such loads read for unchanging and might read it before the wait otherwise.
// Frames of 2k splats 44.6 -> 38.3 us, of 100k 101.4 -> 99.4 us, of 1M 188.3 -> 187.1 us, of 6M the same; the backward of
// eight views of 1M splats 1829 -> 1762 us.
// start_next is called by the kernels of one block (frame start, tile order: thumbnails and 1M splats gain
// 0.4 and 1.3 us); called by all, the next kernel's waiting blocks take room from the last wave (100k splats
// 105.5 us, 6M +10 us), and the cooperative sorts stay plain dependents for the same reason.
// The cooperative depth sort calls it too, when all that the vertex stage reads is complete (the sort itself is launched
// plainly and starts after the cull kernel has ended): the vertex stage then runs beside the sort without a wait at its
// start, and its first block waits at its end, so that the kernels after it, which wait for it alone, find both complete.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P>
__device__ __forceinline__ void frame_step(P&... read_only) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (([&] { asm volatile("" : "+l"(read_only)::"memory"); }()), ...);
}

template <class... Params, class... Args>
inline cudaError_t launch_after(void (*kernel)(Params...), uint32_t grid, uint32_t threads, cudaStream_t st, Args... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// ------------------------------------------------------------------------------------------------
// Decoupled look-back status words: [epoch:32 | INC:1 | AGG:1 | value:30].  A word is only valid
// when its epoch equals the frame's epoch, so status arrays never need clearing between frames.
// ------------------------------------------------------------------------------------------------
constexpr uint32_t LB_AGG = 0x40000000u;
constexpr uint32_t LB_INC = 0x80000000u;
constexpr uint32_t LB_VAL = 0x3FFFFFFFu;

__device__ __forceinline__ uint64_t lb_pack(uint32_t epoch, uint32_t flags, uint32_t value) {
    return ((uint64_t)epoch << 32) | (uint64_t)(flags | (value & LB_VAL));
}
__device__ __forceinline__ void lb_store(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t lb_load(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Look-back for a single running total (stream compaction, bin offsets), called by all 32 lanes of one warp;
// returns the exclusive prefix of `tile` (sum of all earlier tiles): 32 x WORDS words at a time, down to the nearest
// inclusive prefix.  The steps are a chain of L2 round trips, so a step is wide where the registers allow it; and
// every tile's word has a line of its own (lb_word): the tiles of a wave publish and wait at the same time, and
// stores to a line that many others read cost some 20 ns each.  With 16 words to a line a wait of 245 tiles
// whose predecessors had all published took 6-7 us instead of 1.
// Every wait is bounded: after spin_limit polls, or once another wait has run out, the error flag is raised and the
// missing predecessors count as zero, so the kernel always terminates.
__device__ __forceinline__ size_t lb_word(size_t tile) { return tile * LB_LINE; }
template <int WORDS>
__device__ __forceinline__ uint32_t lookback_single(const uint64_t* status, uint32_t tile, uint32_t epoch,
                                                    uint32_t spin_limit, uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t excl = 0;
    for (uint32_t end = tile; end > 0u; end -= 32u * WORDS) {
        uint64_t v[WORDS];
#pragma unroll
        for (uint32_t j = 0; j < (uint32_t)WORDS; ++j) {
            const uint32_t off = lane + 32u * j;
            v[j] = off < end ? lb_load(status + lb_word(end - 1u - off)) : lb_pack(epoch, LB_INC, 0);
        }
        uint32_t nearest, spins = 0;
        for (;;) {
            nearest = 0xFFFFFFFFu;
            uint32_t first_missing = 0xFFFFFFFFu;
#pragma unroll
            for (uint32_t j = 0; j < (uint32_t)WORDS; ++j) {
                const uint32_t off = lane + 32u * j, f = (uint32_t)v[j];
                const bool ready = (uint32_t)(v[j] >> 32) == epoch && (f & (LB_AGG | LB_INC)) != 0u;
                if (ready && (f & LB_INC) != 0u) nearest = min(nearest, off);
                if (!ready) first_missing = min(first_missing, off);
            }
            nearest = __reduce_min_sync(FULL_MASK, nearest);
            if (__reduce_min_sync(FULL_MASK, first_missing) > nearest ||
                (nearest == 0xFFFFFFFFu && __all_sync(FULL_MASK, first_missing == 0xFFFFFFFFu)))
                break;
            if (++spins > spin_limit || ((spins & 1023u) == 0u && (ld_relaxed_u32(err) & SPL_DEV_ERR_LOOKBACK))) {
                if (lane == 0u) atomicOr(err, SPL_DEV_ERR_LOOKBACK);
                return excl;
            }
            if (spins > 4u) __nanosleep(40);
#pragma unroll
            for (uint32_t j = 0; j < (uint32_t)WORDS; ++j) {
                const uint32_t off = lane + 32u * j;
                const bool ready = (uint32_t)(v[j] >> 32) == epoch && ((uint32_t)v[j] & (LB_AGG | LB_INC)) != 0u;
                if (!ready && off <= nearest) v[j] = lb_load(status + lb_word(end - 1u - off));
            }
        }
        uint32_t sum = 0u;
#pragma unroll
        for (uint32_t j = 0; j < (uint32_t)WORDS; ++j) sum += lane + 32u * j <= nearest ? (uint32_t)v[j] & LB_VAL : 0u;
        excl += __reduce_add_sync(FULL_MASK, sum);
        if (nearest != 0xFFFFFFFFu) break;  // always in the window that holds the first tile
    }
    return excl;
}

// Per-thread look-back for one digit of a onesweep pass (status has 256 words per tile): eight predecessors' words
// in flight at a time, nearest first, so that a tile whose predecessors have published but not yet looked back, as
// all of a first wave have, sums them in a few L2 round trips and not in one after another.
__device__ __forceinline__ uint32_t lookback_digit(const uint64_t* status, uint32_t tile, uint32_t digit,
                                                   uint32_t epoch, uint32_t spin_limit, uint32_t* err) {
    constexpr uint32_t WORDS = 8;
    uint32_t excl = 0, end = tile;  // tiles before `end` are still to be added
    while (end > 0u) {
        const uint32_t m = min(end, WORDS);
        uint64_t v[WORDS];
#pragma unroll
        for (uint32_t j = 0; j < WORDS; ++j)
            v[j] = j < m ? lb_load(status + (size_t)(end - 1u - j) * 256u + digit) : 0u;
#pragma unroll
        for (uint32_t j = 0; j < WORDS; ++j) {
            if (j >= m) break;
            uint32_t spins = 0;
            while ((uint32_t)(v[j] >> 32) != epoch || ((uint32_t)v[j] & (LB_AGG | LB_INC)) == 0u) {
                if (++spins > spin_limit) {
                    atomicOr(err, SPL_DEV_ERR_LOOKBACK);
                    return excl;
                }
                if (spins > 16u) __nanosleep(64);
                v[j] = lb_load(status + (size_t)(end - 1u - j) * 256u + digit);
            }
            excl += (uint32_t)v[j] & LB_VAL;
            if ((uint32_t)v[j] & LB_INC) return excl;
        }
        end -= m;
    }
    return excl;
}

// ------------------------------------------------------------------------------------------------
// exp: Cody–Waite range reduction (x = n*ln2 + r with ln2 split into a 16-bit head and a tail),
// degree-7 Taylor polynomial of e^r on |r| <= ln2/2 in Horner form with fused multiply-adds, and a
// two-factor scaling by 2^n that keeps both factors normal.  Bit-identical to the oracle's exp.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float spl_expf(float x) {
    if (x != x) return x;
    if (x > 88.72283935546875f) return __int_as_float(0x7f800000);
    if (x < -103.97208404541015625f) return 0.0f;
    const float n = rintf(__fmul_rn(x, 1.44269502162933349609375f));
    float r = fmaf(n, -0.693145751953125f, x);
    r = fmaf(n, -1.428606765330187045e-06f, r);
    float p = 1.98412698412698412e-04f;
    p = fmaf(p, r, 1.38888888888888889e-03f);
    p = fmaf(p, r, 8.33333333333333333e-03f);
    p = fmaf(p, r, 4.16666666666666667e-02f);
    p = fmaf(p, r, 1.66666666666666667e-01f);
    p = fmaf(p, r, 0.5f);
    p = fmaf(p, r, 1.0f);
    p = fmaf(p, r, 1.0f);
    const int ni = (int)n;
    const int h = ni / 2;
    const float s1 = __int_as_float((h + 127) << 23);
    const float s2 = __int_as_float((ni - h + 127) << 23);
    return __fmul_rn(__fmul_rn(p, s1), s2);
}

// spl_expf restricted to finite x <= 0 (the fragment falloff): the same result bit for bit.  Adding
// 1.5 x 2^23 rounds x log2(e) to the nearest integer n, ties to even as rintf does, and leaves n in the
// sum's low bits, so that the scaling by 2^n (p 2^n is normal for n >= -125) is one integer shift-add and no
// float-to-integer conversion is needed.  FAR: x may lie below -87 (or be NaN), the general path's case.
template <bool FAR>
__device__ __forceinline__ float spl_expf_falloff(float x) {
    if (FAR && !(x >= -87.0f)) return spl_expf(x);
    const float m = __fadd_rn(__fmul_rn(x, 1.44269502162933349609375f), 12582912.0f);
    const float n = m - 12582912.0f;
    float r = fmaf(n, -0.693145751953125f, x);
    r = fmaf(n, -1.428606765330187045e-06f, r);
    float p = 1.98412698412698412e-04f;
    p = fmaf(p, r, 1.38888888888888889e-03f);
    p = fmaf(p, r, 8.33333333333333333e-03f);
    p = fmaf(p, r, 4.16666666666666667e-02f);
    p = fmaf(p, r, 1.66666666666666667e-01f);
    p = fmaf(p, r, 0.5f);
    p = fmaf(p, r, 1.0f);
    p = fmaf(p, r, 1.0f);
    return __uint_as_float(__float_as_uint(p) + (__float_as_uint(m) << 23));
}

// 1/255 as a sum of two floats: k UNORM_HI + (k UNORM_LO rounded), in one fma, is k / 255 correctly rounded
// for k = 0 .. 255.
constexpr float UNORM_HI = 0x1.010102p-8f, UNORM_LO = -0x1.fdfdfep-33f;

// The loader's transform of one splat (Scene::load_chunk, scene.rs:225-250): quaternion normalised,
// log-scales clamped to their mean +- 5 and exponentiated, opacity logit through the sigmoid.
__device__ __forceinline__ void activate_splat(float q0, float q1, float q2, float q3, float l0, float l1, float l2,
                                               float logit, float4& rot, float4& scale_alpha) {
    const float inv = 1.0f / sqrtf(((q0 * q0 + q1 * q1) + q2 * q2) + q3 * q3);
    rot = make_float4(q0 * inv, q1 * inv, q2 * inv, q3 * inv);
    const float avg = ((l0 + l1) + l2) / 3.0f;
    const float lo = avg - 5.0f, hi = avg + 5.0f;
    const float s0 = spl_expf(fminf(fmaxf(l0, lo), hi));
    const float s1 = spl_expf(fminf(fmaxf(l1, lo), hi));
    const float s2 = spl_expf(fminf(fmaxf(l2, lo), hi));
    const float a = 1.0f / (1.0f + spl_expf(-logit));
    scale_alpha = make_float4(s0, s1, s2, a);
}

__device__ __forceinline__ float clamp01(float x) { return fminf(fmaxf(x, 0.0f), 1.0f); }

// WGSL u32(f32): truncate, saturate, NaN -> 0.
__device__ __forceinline__ uint32_t sat_u32(float x) { return __float2uint_rz(x); }

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Lanes whose 8-bit digit equals this lane's (valid lanes only), from eight ballots: the warp-level
// multisplit match without MATCH.ANY, whose latency dominated the ranking.
__device__ __forceinline__ uint32_t match_digit(uint32_t d, bool valid) {
    uint32_t peers = __ballot_sync(FULL_MASK, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(FULL_MASK, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// Block-wide exclusive scan of one u32 per thread (blockDim.x == 256).  `scratch` holds 8 words.
__device__ __forceinline__ uint32_t block_exclusive_scan_256(uint32_t v, uint32_t* scratch, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) scratch[w] = x;
    __syncthreads();
    uint32_t wpre = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t s = scratch[i];
        wpre += (uint32_t)i < w ? s : 0u;
        tot += s;
    }
    __syncthreads();
    *total = tot;
    return wpre + x - v;
}

}  // namespace spl
