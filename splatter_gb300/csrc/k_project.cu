// Projection side of the splat pipeline (sm_103a):
//   k_frame_begin   - per-frame counter reset + epoch bump (replaces buffer clears, renderer.rs:412,422-427)
//   k_cull_key      - worldToClipSpace + isInFrustum + depth key + digit histograms (radixSortA,
//                     shaders.wgsl:298-336) fused with ORDERED stream compaction of the visible splats
//                     (warp ballots + decoupled look-back), so only visible keys are sorted
//   k_preprocess    - the vertex stage (shaders.wgsl:507-573): SH colour, exact perspective conic of the
//                     ellipsoid, its decomposition and the rotated rectangle, emitted once per visible
//                     splat as a 64-byte screen-space record for the compute rasteriser
//   k_load_records  - Scene::load_chunk transform (scene.rs:225-250) on the device
//
// Compiled with -fmad=false: all FP32 expressions follow the WGSL operation order and are
// bit-identical to the oracle's FP32 restatement.
#include <cstdio>

#include "spl_vertex.cuh"

namespace spl {

// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void counters_begin(FrameCounters* fc, uint32_t* epoch_word) {
    uint4* w = reinterpret_cast<uint4*>(fc);
    for (uint32_t i = threadIdx.x; i < sizeof(FrameCounters) / 16; i += blockDim.x) w[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t e = *epoch_word + 1u;
        if (e == 0u) e = 1u;  // epoch 0 marks never-written status words
        *epoch_word = e;
        fc->epoch = e;
    }
}

__global__ void k_counters_begin(FrameCounters* fc, uint32_t* epoch_word, uint32_t count) {
    counters_begin(fc, epoch_word);
    if (threadIdx.x == 0) fc->visible = count;
}

// A frame's first kernel: the counters as above, and the frame's uniform block and scene view
// (kernel parameters here, so that a captured frame graph takes a new camera and scene by updating
// this one node) published to device memory for the kernels that follow.
__global__ void k_frame_begin(FrameCounters* fc, uint32_t* epoch_word, Uniforms u, Uniforms* d_u, SceneView sv,
                              SceneView* d_sv) {
    start_next();
    frame_step();
    if (threadIdx.x < sizeof(Uniforms) / 4)
        reinterpret_cast<uint32_t*>(d_u)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&u)[threadIdx.x];
    if (threadIdx.x < sizeof(SceneView) / 4)
        reinterpret_cast<uint32_t*>(d_sv)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&sv)[threadIdx.x];
    counters_begin(fc, epoch_word);
}

void launch_frame_begin(FrameCounters* fc, uint32_t* epoch_word, uint32_t count, cudaStream_t st) {
    k_counters_begin<<<1, 256, 0, st>>>(fc, epoch_word, count);
}

void launch_frame_begin(FrameCounters* fc, uint32_t* epoch_word, const Uniforms& u, Uniforms* d_u, const SceneView& sv,
                        SceneView* d_sv, cudaStream_t st) {
    k_frame_begin<<<1, 256, 0, st>>>(fc, epoch_word, u, d_u, sv, d_sv);
}

const void* frame_begin_kernel() { return reinterpret_cast<const void*>(&k_frame_begin); }

// The frame's uniform block and scene view staged in shared memory (one word per thread of the
// first warps; the caller synchronises).
__device__ __forceinline__ void stage_frame(const Uniforms* __restrict__ d_u, Uniforms& s_u,
                                            const SceneView* __restrict__ d_sv, SceneView& s_sv) {
    if (threadIdx.x < sizeof(Uniforms) / 4)
        reinterpret_cast<uint32_t*>(&s_u)[threadIdx.x] = __ldg(reinterpret_cast<const uint32_t*>(d_u) + threadIdx.x);
    if (threadIdx.x < sizeof(SceneView) / 4)
        reinterpret_cast<uint32_t*>(&s_sv)[threadIdx.x] = __ldg(reinterpret_cast<const uint32_t*>(d_sv) + threadIdx.x);
}

// ------------------------------------------------------------------------------------------------
// Cull + key + histogram + ordered compaction.  One CTA handles a tile of 256 x PER_LANE consecutive splats; warp w
// owns an eighth of the tile and lane l handles its elements 32*j + l, so loads are coalesced and the ballot
// order is the index order.
// Bound by latency: the ticket and the uniform block, the loads, some 120 instructions per splat, the look-back.
// 6M splats 66 -> 50 us (look-back words in lines of their own and 256 of them per step: 52 us; tiles of 2048 splats
// instead of 4096, four CTAs per SM: 50 us, tiles of 1024: 61 us), 1M 26 -> 21 us; frames of up to 2^19 splats,
// which fit one wave in tiles of 1024, take those: 100k 18 -> 15 us, 350k 19 -> 16 us (whole frames of 131k 67.8 -> 66.4 us,
// 400k 84.8 -> 84.5, 2^19 the same, 700k 103.0 -> 105.0, 1M 121.5 -> 123.6).
template <int MODE, bool HIST, int PER_LANE>
__global__ void __launch_bounds__(256, 4) k_cull_key(const SceneView* __restrict__ d_sv, const Uniforms* __restrict__ d_u,
                                                  FrameCounters* fc,
                                                  const uint32_t* __restrict__ epoch_word, uint64_t* status,
                                                  uint32_t* __restrict__ keys_out, uint32_t* __restrict__ idx_out,
                                                  uint32_t spin_limit) {
    __shared__ uint32_t s_hist[HIST ? 1024 : 1];
    __shared__ uint32_t s_wcnt[8];
    __shared__ uint32_t s_tile, s_epoch, s_base;
    __shared__ Uniforms s_u;
    __shared__ SceneView s_sv;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    if (HIST)
        for (uint32_t i = tid; i < 1024u; i += 256u) s_hist[i] = 0u;
    frame_step(d_sv, d_u, epoch_word);
    stage_frame(d_u, s_u, d_sv, s_sv);
    if (tid == 0) {
        s_tile = atomicAdd(&fc->tile_counter[0].v, 1u);
        s_epoch = *epoch_word;
    }
    __syncthreads();
    const Uniforms& u = s_u;
    const SceneView& s = s_sv;
    const uint32_t tile = s_tile, epoch = s_epoch, n = s.n;
    constexpr uint32_t TILE = 256u * PER_LANE;
    const uint32_t ntiles = (n + TILE - 1) / TILE;
    if (tile >= ntiles) return;  // a grid sized for a larger scene (captured frames)
    const uint32_t base = tile * TILE + w * (TILE / 8u) + lane;

    float px[PER_LANE], py[PER_LANE], pz[PER_LANE];
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const uint32_t e = base + 32u * j;
        if (e < n) {
            px[j] = __ldg(s.x + e);
            py[j] = __ldg(s.y + e);
            pz[j] = __ldg(s.z + e);
        } else {
            px[j] = py[j] = pz[j] = 0.0f;
        }
    }
    uint32_t key[PER_LANE], pos[PER_LANE];
    uint32_t vis_bits = 0u, wtotal = 0u, all_ones = 0u, top_ff = 0u;
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const uint32_t e = base + 32u * j;
        float h[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
            h[r] = ((u.vp[0 * 4 + r] * px[j] + u.vp[1 * 4 + r] * py[j]) + u.vp[2 * 4 + r] * pz[j]) + u.vp[3 * 4 + r] * 1.0f;
        bool vis;
        uint32_t k;
        if (MODE == DS_CPU) {
            // renderer.rs:381-387: reciprocal multiply, no epsilon, key = bits(z)
            const float rw = 1.0f / h[3];
            const float cx = h[0] * rw, cy = h[1] * rw, cz = h[2] * rw;
            vis = fabsf(cx) < u.tol && fabsf(cy) < u.tol && fabsf(cz - 0.5f) < 0.5f;
            k = __float_as_uint(cz);
        } else {
            // shaders.wgsl:54-61, 318-324
            const float den = h[3] + 1e-7f;
            const float cx = h[0] / den, cy = h[1] / den, cz = h[2] / den;
            vis = fabsf(cx) < u.tol && fabsf(cy) < u.tol && fabsf(cz - 0.5f) < 0.5f;
            k = sat_u32(cz * 65535.0f) << 16;
            k |= sat_u32((cx * 0.5f + 0.5f) * 255.0f) << 8;
            k |= sat_u32((cy * 0.5f + 0.5f) * 255.0f);
        }
        vis = vis && e < n;
        const uint32_t b = __ballot_sync(FULL_MASK, vis);
        pos[j] = wtotal + __popc(b & lt);
        wtotal += __popc(b);
        key[j] = k;
        if (vis) {
            vis_bits |= 1u << j;
            if (HIST) {
                atomicAdd(&s_hist[k & 255u], 1u);
                atomicAdd(&s_hist[256u + ((k >> 8) & 255u)], 1u);
                atomicAdd(&s_hist[512u + ((k >> 16) & 255u)], 1u);
                atomicAdd(&s_hist[768u + (k >> 24)], 1u);
            }
            all_ones += k == 0xFFFFFFFFu;
            top_ff += (k >> 24) == 0xFFu;
        }
    }
    if (lane == 0) s_wcnt[w] = wtotal;
    __syncthreads();
    uint32_t wpre = 0, ttot = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t c = s_wcnt[i];
        wpre += i < w ? c : 0u;
        ttot += c;
    }
    if (w == 0) {
        if (lane == 0) lb_store(status + lb_word(tile), lb_pack(epoch, tile == 0 ? LB_INC : LB_AGG, ttot));
        const uint32_t excl = lookback_single<8>(status, tile, epoch, spin_limit, &fc->err);
        if (lane == 0) {
            if (tile != 0) lb_store(status + lb_word(tile), lb_pack(epoch, LB_INC, excl + ttot));
            s_base = excl;
            if (tile == ntiles - 1) fc->visible = excl + ttot;
        }
    }
    __syncthreads();
    const uint32_t out0 = s_base + wpre;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        if (vis_bits & (1u << j)) {
            keys_out[out0 + pos[j]] = key[j];
            idx_out[out0 + pos[j]] = base + 32u * j;
        }
    }
    if (HIST) {
        for (uint32_t i = tid; i < 1024u; i += 256u) {
            const uint32_t v = s_hist[i];
            if (v) atomicAdd(&fc->hist_depth[0][0] + i, v);
        }
    }
    if (MODE != DS_CPU) {
        const uint32_t a = __reduce_add_sync(FULL_MASK, all_ones), t = __reduce_add_sync(FULL_MASK, top_ff);
        if (lane == 0 && a) atomicAdd(&fc->keys_all_ones, a);
        if (lane == 0 && t) atomicAdd(&fc->keys_top_ff, t);
    }
}

void launch_cull_key(int mode, bool hist, uint32_t grid_n, const SceneView* d_sv, const Uniforms* u,
                     FrameCounters* fc, const uint32_t* epoch_word, uint64_t* status, uint32_t* keys_out,
                     uint32_t* idx_out, uint32_t spin_limit, cudaStream_t st) {
    if (grid_n == 0) return;
    const bool small = grid_n <= CULL_SMALL_MAX;
    const uint32_t tile = small ? CULL_TILE_SMALL : CULL_TILE, grid = (grid_n + tile - 1) / tile;
    constexpr int L = CULL_TILE / 256, S = CULL_TILE_SMALL / 256;
    auto k = mode == DS_CPU ? (hist ? (small ? k_cull_key<DS_CPU, true, S> : k_cull_key<DS_CPU, true, L>)
                                    : (small ? k_cull_key<DS_CPU, false, S> : k_cull_key<DS_CPU, false, L>))
                            : (hist ? (small ? k_cull_key<DS_GPU, true, S> : k_cull_key<DS_GPU, true, L>)
                                    : (small ? k_cull_key<DS_GPU, false, S> : k_cull_key<DS_GPU, false, L>));
    launch_after(k, grid, 256, st, d_sv, u, fc, epoch_word, status, keys_out, idx_out, spin_limit);
}

// ------------------------------------------------------------------------------------------------
// Vertex stage, a warp for 32 visible splats at a time.  STAGED: their SH rows (NV 16-byte pieces of the
// 192-byte rows) come through shared memory: lane l of load k copies piece (32 k + l) of the warp's 32 NV
// pieces, so that a load's lanes cover whole rows.  One row per lane instead touches 32 different 128-byte
// lines with every load, and the L1's line accesses bound the kernel.  The copies are asynchronous: the shape
// is computed while they are in flight.  6M splats, SH 3, 4.33M visible: 246 -> 219 us, 91% of the copy
// bandwidth on 312 bytes per visible splat (seven CTAs of four warps per SM at 72 registers; six 223 us; eight
// 219 us, but slower than seven below 1M splats; a grid of the resident CTAs alone 228 us).  Where one wave of
// warps holds all splats the detour only adds latency (before the stage ran beside the sort, frames of 2k, 100k
// and 350k splats 0.8-1.2 us longer; since, with nearly all splats visible, 262k 151.3 -> 152.6 us, 400k 202.3
// -> 202.1, 2^19 234.4 -> 230.5, 1M 332.8 -> 324.0): below PRE_STAGED_MIN splats, and for degree 0, whose rows
// are one piece, each lane reads its own row.
constexpr uint32_t PRE_STAGED_MIN = 1u << 19;

template <int SHO, bool STAGED>
struct PreShape {
    static constexpr int NV = (3 * (SHO + 1) * (SHO + 1) + 3) / 4;  // 1, 3, 7 or 12 pieces of a row
    static constexpr int STRIDE = NV | 1;  // in shared memory, odd: a lane per row reads without bank conflicts
    static constexpr int WARPS = STAGED ? 4 : 8, CTAS = STAGED ? 7 : 3;
};

__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int SHO, bool COV, bool RECT, bool STAGED>
__global__ void __launch_bounds__(PreShape<SHO, STAGED>::WARPS * 32, PreShape<SHO, STAGED>::CTAS) k_preprocess(const SceneView* __restrict__ d_sv,
                                                    const Uniforms* __restrict__ d_u,
                                                    const uint32_t* __restrict__ idx,
                                                    const FrameCounters* __restrict__ fc, float4* __restrict__ rec,
                                                    uint2* __restrict__ boxes, bool beside) {
    constexpr int NV = PreShape<SHO, STAGED>::NV, STRIDE = PreShape<SHO, STAGED>::STRIDE;
    __shared__ float4 s_sh[PreShape<SHO, STAGED>::WARPS][STAGED ? 32 * STRIDE : 1];
    __shared__ Uniforms s_u;
    __shared__ SceneView s_sv;
    if (!beside) frame_step(d_sv, d_u, idx, fc);
    stage_frame(d_u, s_u, d_sv, s_sv);
    __syncthreads();
    const Uniforms& u = s_u;
    const SceneView& s = s_sv;
    const uint32_t V = fc->visible, lane = threadIdx.x & 31u;
    float4* rows = s_sh[threadIdx.x >> 5];
    const uint32_t step = gridDim.x * blockDim.x;
    uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t i = STAGED && slot < V ? __ldg(idx + slot) : 0u;
    for (; slot - lane < V; slot += step) {  // the warp's 32 slots; lanes past V only help to copy
        const uint32_t live = min(32u, V - (slot - lane));
        if constexpr (STAGED) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const uint32_t piece = 32u * k + lane, row = piece / NV, col = piece - row * NV;
                const uint32_t ir = __shfl_sync(FULL_MASK, i, (int)row);
                if (row < live) copy16_async(rows + row * STRIDE + col, s.sh + (size_t)ir * 48 + col * 4);
            }
        } else {
            if (slot >= V) break;
            i = __ldg(idx + slot);
        }
        const bool mine = !STAGED || lane < live;
        float cx = 0.0f, cy = 0.0f, cz = 0.0f;
        float4 rot = make_float4(0.0f, 0.0f, 0.0f, 0.0f), sca = rot;
        float c[3];
        if (mine) {
            cx = __ldg(s.x + i);
            cy = __ldg(s.y + i);
            cz = __ldg(s.z + i);
            rot = __ldg(s.rot + i);
            sca = __ldg(s.scale_alpha + i);
        }
        if constexpr (!STAGED) {
            float4 row[NV];
            const float4* r = reinterpret_cast<const float4*>(s.sh + (size_t)i * 48);
#pragma unroll
            for (int k = 0; k < NV; ++k) row[k] = __ldg(r + k);
            vertex_colour<SHO, STAGED>(u, cx, cy, cz, row, c);
        }
        if (STAGED) i = slot + step < V ? __ldg(idx + slot + step) : 0u;  // the next iteration's splat
        VertexShape<float> o;
        vertex_shape<COV, float>(u, cx, cy, cz, rot.x, rot.y, rot.z, rot.w, sca.x, sca.y, sca.z, o);
        // pixel box of the rectangle (or AA square) and validity
        const float vw = u.view_size[0], vh = u.view_size[1];
        const float Wf = (float)u.image_size[0], Hf = (float)u.image_size[1];
        const float psx = (2.0f * vw) / Wf, psy = -((2.0f * vh) / Hf);
        const float m = u.margin;
        float ex, ey, R = 0.0f;
        if (RECT) {
            ex = m * (fabsf(o.Xx) + fabsf(o.Yx));
            ey = m * (fabsf(o.Xy) + fabsf(o.Yy));
        } else {
            R = sqrtf(fmaxf(o.Xx * o.Xx + o.Xy * o.Xy, o.Yx * o.Yx + o.Yy * o.Yy)) * m;
            ex = R;
            ey = R;
        }
        const float cxp = (o.t0 + vw) / psx, exq = ex / psx;
        const float cyp = (o.t1 - vh) / psy, eyq = ey / (-psy);
        // pixels whose centre (p + 0.5) lies in the exact box, widened by 1/64 px against rounding
        const float eps = 0.015625f;
        const float fx0 = ceilf(((cxp - exq) - eps) - 0.5f), fx1 = floorf(((cxp + exq) + eps) - 0.5f);
        const float fy0 = ceilf(((cyp - eyq) - eps) - 0.5f), fy1 = floorf(((cyp + eyq) + eps) - 0.5f);
        const float al = sca.w;
        if constexpr (STAGED) {
            wait_copies();
            __syncwarp();
            vertex_colour<SHO, STAGED>(u, cx, cy, cz, rows + lane * STRIDE, c);
            __syncwarp();  // the rows are read before the next iteration's copies
        }
        bool ok = isfinite(o.A00) && isfinite(o.A01) && isfinite(o.B0) && isfinite(o.A10) && isfinite(o.A11) &&
                  isfinite(o.B1) && isfinite(c[0]) && isfinite(c[1]) && isfinite(c[2]) && isfinite(fx0) &&
                  isfinite(fx1) && isfinite(fy0) && isfinite(fy1) && isfinite(R) && isfinite(o.bx) && isfinite(o.by) &&
                  (al >= 1.0f / 255.0f);
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
        if (ok) {
            const float cx0 = fmaxf(fx0, 0.0f), cx1 = fminf(fx1, Wf - 1.0f);
            const float cy0 = fmaxf(fy0, 0.0f), cy1 = fminf(fy1, Hf - 1.0f);
            if (cx0 <= cx1 && cy0 <= cy1) {
                lo = (uint32_t)(int)cx0 | ((uint32_t)(int)cy0 << 16);
                hi = (uint32_t)(int)cx1 | ((uint32_t)(int)cy1 << 16);
            }
        }
        if (mine) {
            float4* q = rec + (size_t)slot * 4;
            q[0] = make_float4(o.A00, o.A01, o.B0, o.A10);
            q[1] = make_float4(o.A11, o.B1, al, __uint_as_float(lo));
            q[2] = make_float4(c[0], c[1], c[2], __uint_as_float(hi));
            q[3] = RECT ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : make_float4(o.bx, o.by, R, 0.0f);
            boxes[slot] = make_uint2(lo, hi);  // compact copy for the binning kernel
        }
    }
    // This kernel's end is the next one's sign that both are done: one block waits for the kernel before.
    if (beside && blockIdx.x == 0) frame_step();
}

template <int SHO, bool COV, bool RECT, bool STAGED>
static void launch_pre3(const SceneView* s, const Uniforms* u, const uint32_t* idx, const FrameCounters* fc, float4* rec,
                        uint2* boxes, uint32_t max_n, bool beside, cudaStream_t st) {
    constexpr uint32_t threads = PreShape<SHO, STAGED>::WARPS * 32;
    // grid stride beyond 4096 threads per SM
    const uint32_t blocks = (max_n + threads - 1) / threads, cap = device_sm_count() * (4096u / threads);
    launch_after(k_preprocess<SHO, COV, RECT, STAGED>, blocks < cap ? blocks : cap, threads, st, s, u, idx, fc, rec, boxes,
                 beside);
}
template <int SHO>
static void launch_pre(bool cov, bool rect, const SceneView* s, const Uniforms* u, const uint32_t* idx,
                       const FrameCounters* fc, float4* rec, uint2* boxes, uint32_t max_n, bool beside, cudaStream_t st) {
    constexpr bool CAN_STAGE = SHO > 0;
    const bool staged = CAN_STAGE && max_n >= PRE_STAGED_MIN;
    auto run = cov ? (rect ? (staged ? launch_pre3<SHO, true, true, CAN_STAGE> : launch_pre3<SHO, true, true, false>)
                           : (staged ? launch_pre3<SHO, true, false, CAN_STAGE> : launch_pre3<SHO, true, false, false>))
                   : (rect ? (staged ? launch_pre3<SHO, false, true, CAN_STAGE> : launch_pre3<SHO, false, true, false>)
                           : (staged ? launch_pre3<SHO, false, false, CAN_STAGE> : launch_pre3<SHO, false, false, false>));
    run(s, u, idx, fc, rec, boxes, max_n, beside, st);
}

void launch_preprocess(int sh_order, bool covariance, bool rect, const SceneView* s, const Uniforms* u,
                       const uint32_t* idx, const FrameCounters* fc, float4* rec, uint2* boxes, uint32_t max_n,
                       bool beside, cudaStream_t st) {
    if (max_n == 0) return;
    auto run = sh_order == 0 ? launch_pre<0> : (sh_order == 1 ? launch_pre<1> : (sh_order == 2 ? launch_pre<2> : launch_pre<3>));
    run(covariance, rect, s, u, idx, fc, rec, boxes, max_n, beside, st);
}

// ------------------------------------------------------------------------------------------------
// Loader: 62-float PLY records -> SoA (scene.rs:225-250).  A block stages 256 records in shared
// memory with coalesced 16-byte loads, transforms one record per thread, and writes the 48 SH
// floats of its 256 splats back as one contiguous, coalesced range.
constexpr int LOAD_BLOCK = 256;

__global__ void __launch_bounds__(LOAD_BLOCK) k_load_records(const float* __restrict__ recs, uint32_t count,
                                                             float* x, float* y, float* z, float4* rot,
                                                             float4* scale_alpha, float* sh) {
    extern __shared__ float4 s_buf4[];
    float* s_buf = reinterpret_cast<float*>(s_buf4);
    const uint32_t first = blockIdx.x * LOAD_BLOCK;
    const uint32_t nrec = min((uint32_t)LOAD_BLOCK, count - first);
    const uint32_t nflt = nrec * 62u;
    const float* src = recs + (size_t)first * 62u;  // 256*62*4 bytes per block: 16-byte aligned
    const uint32_t nvec = nflt / 4u;
    for (uint32_t k = threadIdx.x; k < nvec; k += LOAD_BLOCK) s_buf4[k] = __ldg(reinterpret_cast<const float4*>(src) + k);
    for (uint32_t k = nvec * 4u + threadIdx.x; k < nflt; k += LOAD_BLOCK) s_buf[k] = __ldg(src + k);
    __syncthreads();
    const uint32_t t = threadIdx.x;
    if (t < nrec) {
        const float* r = s_buf + t * 62u;
        const uint32_t i = first + t;
        float4 q, sa;
        activate_splat(r[58], r[59], r[60], r[61], r[55], r[56], r[57], r[54], q, sa);
        rot[i] = q;
        scale_alpha[i] = sa;
        x[i] = r[0];
        y[i] = r[1];
        z[i] = r[2];
    }
    float* dst = sh + (size_t)first * 48u;
    for (uint32_t k = threadIdx.x; k < nrec * 48u; k += LOAD_BLOCK) {
        const uint32_t rr = k / 48u, c = k - rr * 48u;
        dst[k] = s_buf[rr * 62u + 6u + c];
    }
}

void launch_load_records(const float* records62, uint32_t count, float* x, float* y, float* z, float4* rot,
                         float4* scale_alpha, float* sh, cudaStream_t st) {
    if (count == 0) return;
    static bool attr = false;
    const int smem = LOAD_BLOCK * 62 * 4;
    if (!attr) {
        cudaFuncSetAttribute(k_load_records, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        attr = true;
    }
    const uint32_t grid = (count + LOAD_BLOCK - 1) / LOAD_BLOCK;
    k_load_records<<<grid, LOAD_BLOCK, smem, st>>>(records62, count, x, y, z, rot, scale_alpha, sh);
}

// 60-float device splats of the reference (scene.rs:32, shaders.wgsl:28-35) <-> SoA.
__global__ void k_splats60_to_soa(const float* __restrict__ s60, uint32_t count, float* x, float* y, float* z,
                                  float4* rot, float4* scale_alpha, float* sh) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float4* r = reinterpret_cast<const float4*>(s60 + (size_t)i * 60);
        const float4 a = r[0], b = r[1], c = r[2];
        rot[i] = a;
        x[i] = b.x;
        y[i] = b.y;
        z[i] = b.z;
        scale_alpha[i] = c;
        float4* d = reinterpret_cast<float4*>(sh + (size_t)i * 48);
#pragma unroll
        for (int k = 0; k < 12; ++k) d[k] = r[3 + k];
    }
}

__global__ void k_soa_to_splats60(SceneView s, uint32_t start, uint32_t count, float* s60) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        const uint32_t i = start + t;
        float4* r = reinterpret_cast<float4*>(s60 + (size_t)t * 60);
        r[0] = s.rot[i];
        r[1] = make_float4(s.x[i], s.y[i], s.z[i], 0.0f);
        r[2] = s.scale_alpha[i];
        const float4* q = reinterpret_cast<const float4*>(s.sh + (size_t)i * 48);
#pragma unroll
        for (int k = 0; k < 12; ++k) r[3 + k] = q[k];
    }
}

void launch_splats60_to_soa(const float* s60, uint32_t count, float* x, float* y, float* z, float4* rot,
                            float4* scale_alpha, float* sh, cudaStream_t st) {
    if (count == 0) return;
    uint32_t grid = (count + 255) / 256;
    if (grid > 4096) grid = 4096;
    k_splats60_to_soa<<<grid, 256, 0, st>>>(s60, count, x, y, z, rot, scale_alpha, sh);
}

void launch_soa_to_splats60(const SceneView& s, uint32_t start, uint32_t count, float* s60, cudaStream_t st) {
    if (count == 0) return;
    uint32_t grid = (count + 255) / 256;
    if (grid > 4096) grid = 4096;
    k_soa_to_splats60<<<grid, 256, 0, st>>>(s, start, count, s60);
}

// Sorted entries (key, splat index) for readback (the reference's commented debug readback,
// renderer.rs:456-464).  slots == nullptr for the unsorted (None) mode.
__global__ void k_gather_entries(const uint32_t* keys, const uint32_t* slots, const uint32_t* idx,
                                 const FrameCounters* fc, uint32_t* keys_out, uint32_t* idx_out, uint32_t cap) {
    const uint32_t V = min(fc->visible, cap);
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < V; r += gridDim.x * blockDim.x) {
        if (slots) {
            keys_out[r] = keys[r];
            idx_out[r] = idx[slots[r]];
        } else {
            keys_out[r] = keys[r];
            idx_out[r] = idx[r];
        }
    }
}

void launch_gather_entries(const uint32_t* keys, const uint32_t* slots, const uint32_t* idx, const FrameCounters* fc,
                           int mode, uint32_t* keys_out, uint32_t* idx_out, uint32_t cap, cudaStream_t st) {
    (void)mode;
    if (cap == 0) return;
    uint32_t grid = (cap + 255) / 256;
    if (grid > 4096) grid = 4096;
    k_gather_entries<<<grid, 256, 0, st>>>(keys, slots, idx, fc, keys_out, idx_out, cap);
}

// Fault-free check of the bounded look-back: one warp acts as tile 1 of a scan whose tile 0 never
// publishes (status[0] is never written).  The wait runs out after spin_limit polls, raises the
// error bit and returns; out[0] = prefix it gave up with, out[1] = error word.
__global__ void k_lookback_probe(uint64_t* status, uint32_t* err, uint32_t spin_limit, uint32_t* out) {
    const uint32_t excl = lookback_single<8>(status, 1u, 7u, spin_limit, err);
    __syncwarp();
    if (threadIdx.x == 0) {
        out[0] = excl;
        out[1] = ld_relaxed_u32(err);
    }
}

void launch_lookback_probe(uint64_t* status, uint32_t* err, uint32_t spin_limit, uint32_t* out, cudaStream_t st) {
    k_lookback_probe<<<1, 32, 0, st>>>(status, err, spin_limit, out);
}

}  // namespace spl
