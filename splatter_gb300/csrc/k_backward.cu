// Backward pass of the splat pipeline (sm_103a), fp32 blend mode.  No reference counterpart: the
// reference only renders.  The forward it differentiates is the one k_raster/k_preprocess compute:
//
//   per pixel, front to back over the tile's depth-ordered list:
//     alpha = a * exp(-|tc|^2 / 2)            (skipped when alpha < 1/255)
//     s_c = sat(rgb_c * alpha), sa = sat(alpha)
//     C_c += s_c * T,  T *= (1 - sa)          (stops once T < 1e-4)
//
// k_raster_backward re-walks each tile front to back, RECOMPUTING the transmittance instead of
// storing it.  With C_final and T_final from the forward image, the colour still to come after
// splat i is S = C_final - C_(<=i), so
//     dL/ds_c  = dL/dC_c * T_i
//     dL/dsa   = -(dL/dC . S + dL/dT * T_final) / (1 - sa)
// and the chain through sat(), the falloff and tc = A (X, Y) + B gives per-splat gradients of the
// record (A00, A01, B0, A10, A11, B1, a, r, g, b), reduced over each 4x2-pixel group before one
// set of global float atomics per (splat, group).  A is accumulated against pixel offsets from the
// centre of the splat's pixel box and B at that centre (well conditioned; see vertex_vjp_t).
//
// k_preprocess_backward maps those record gradients to the splat parameters (centre, rotation,
// scale, opacity, SH) in reverse mode (vertex_vjp_t): one sweep of the vertex stage's values, one
// sweep of adjoints back through the same formulas, in float; needles and discs (needs_double_sweep)
// are left to k_preprocess_backward_double, which sweeps them in double.  SH coefficient gradients
// are the basis values times the colour gradients.
#include "spl_raster.cuh"
#include "spl_vertex.cuh"

namespace spl {

constexpr int GR = 10;  // gradient words per record

__global__ void k_zero_grad_rec(float* grad_rec, const FrameCounters* fc, uint32_t* deferred) {
    frame_step();
    if (blockIdx.x == 0 && threadIdx.x == 0) deferred[0] = 0u;
    const uint32_t n = fc->visible * GR;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) grad_rec[i] = 0.0f;
}

// Sums 10 values over the 8 lanes of a lane group (lane index li = lane & 7) in three exchange steps that halve the
// values each lane carries: afterwards lane li holds the sum of value k0 in v0 and, for li = 0 and 4, of k0 + 1 in v1.
__device__ __forceinline__ uint32_t reduce10_over8(const float* g, uint32_t li, float& v0, float& v1) {
    const bool h4 = (li & 4u) != 0u, h2 = (li & 2u) != 0u, h1 = (li & 1u) != 0u;
    float a[5], b[3];
#pragma unroll
    for (int i = 0; i < 5; ++i) {  // keep values 5..9 (h4) or 0..4
        const float send = h4 ? g[i] : g[i + 5], keep = h4 ? g[i + 5] : g[i];
        a[i] = keep + __shfl_xor_sync(FULL_MASK, send, 4);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {  // keep a[3..4] (h2) or a[0..2]
        const float hi = i < 2 ? a[i + 3] : 0.0f;
        const float send = h2 ? a[i] : hi, keep = h2 ? hi : a[i];
        b[i] = keep + __shfl_xor_sync(FULL_MASK, send, 2);
    }
    // h2 lanes carry two values (b0, b1): keep b1 (h1) or b0; the others three: keep b2 (h1) or b0, b1
    const float send0 = h1 ? b[0] : (h2 ? b[1] : b[2]);
    const float keep0 = h1 ? (h2 ? b[1] : b[2]) : b[0];
    const float send1 = (h1 && !h2) ? b[1] : 0.0f;
    const float keep1 = (!h1 && !h2) ? b[1] : 0.0f;
    v0 = keep0 + __shfl_xor_sync(FULL_MASK, send0, 1);
    v1 = keep1 + __shfl_xor_sync(FULL_MASK, send1, 1);
    return (h4 ? 5u : 0u) + (h2 ? (h1 ? 4u : 3u) : (h1 ? 2u : 0u));
}

// One CTA per tile, its warps as in k_raster (strips of two rows), a warp's lanes in four groups of 4x2 pixels.
// A group walks its own list of the batch's records, those whose row masks (mask_rows) touch one of its pixels,
// all eight lanes on the same record, so that the record's ten gradients are summed over the group before they
// are added to grad_rec.  The lists are record indices in shared memory: four ballots per 32 records give every
// (record, group) its place, and the walk has no list bookkeeping but a counter.
// Bound by instruction issue (74% of the slots, DRAM 5%): what counts is the number of walk iterations, i.e. how well the lists fit, and
// what one costs.  A training step of eight views of 1M splats at 1024x1024, per view: groups listed by their boxes and
// walked in lockstep over 32 records 167 us; lists from the row masks, walked over the whole batch as bit words, 134 us;
// as record indices 125 us (106 us as a launch alone).
// Groups of 2x2 pixels take 111 us (99 us), with fewer idle lanes, but twice as many additions to grad_rec: one after
// another to one float, their error grows with the square root of their number, 2.31e-7 of a sum for 1.72e-7
// (root mean square of colour gradients over some 130 groups of 4x2), and the vertex stage's sweep passes a thousandfold
// of it on to the rotations of nearly round splats (the worst splat of a million against the 4x2 groups in another order,
// nine in ten of 70 scenes: below 6.0e-4 of its gradient with 2x2, 2.4e-4 with 4x2).
// Sums in double of either group have neither, but cost more than the smaller groups save (a step 2,931 us with 4x2 and
// float, 3,030 with 2x2 and double, 3,087 with 4x2 and double) and twice the scratch.
template <bool RECT, bool FAR>
__global__ void __launch_bounds__(256, 4) k_raster_backward(const uint2* __restrict__ ranges,
                                                         const uint4* __restrict__ tile_order,
                                                         const uint32_t* __restrict__ pair_vals,
                                                         const float4* __restrict__ rec, int W, int H, int tiles_x,
                                                         float margin, float psx, float psy,
                                                         const float4* __restrict__ image,
                                                         const float4* __restrict__ grad_image,
                                                         float* __restrict__ grad_rec) {
    // (A00, A10, A01, A11) (B0, B1, alpha, r) (g, b, centre of the pixel box)
    __shared__ float4 s_a[RASTER_BATCH], s_b[RASTER_BATCH], s_c[RASTER_BATCH];
    __shared__ float4 s_q3[RECT ? 1 : RASTER_BATCH];
    __shared__ uint32_t s_row[RASTER_BATCH], s_pm[8][RASTER_BATCH];  // the record's row of grad_rec; its row masks
    __shared__ uint8_t s_list[8][4][RASTER_BATCH];                   // [warp][group]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5, lt = lanemask_lt();
    const uint32_t grp = lane >> 3, li = lane & 7u;
    frame_step(ranges, tile_order, pair_vals, rec, image, grad_image);
    // the forward's most-pairs-first order of this frame's tiles, when it made one
    uint2 rg;
    int tile;
    ordered_tile(ranges, tile_order, rg, tile);
    const int tx = tile % tiles_x, ty = tile / tiles_x;
    const int wx0 = tx * TILE_PIXELS, ty0 = ty * TILE_PIXELS;
    const uint32_t col = 4u * grp + (li & 3u), row = li >> 2;
    const int px = wx0 + (int)col, py = ty0 + 2 * (int)w + (int)row;
    const float X = (float)px + 0.5f, Y = (float)py + 0.5f;
    const uint32_t my_pixel = 1u << (16u * row + col);  // in a strip's row mask
    const bool inside = px < W && py < H;
    float Cf[3] = {0.0f, 0.0f, 0.0f}, gC[3] = {0.0f, 0.0f, 0.0f}, Tf = 1.0f, gT = 0.0f;
    if (inside) {
        const size_t pix = (size_t)py * (size_t)W + (size_t)px;
        const float4 im = image[pix], gi = grad_image[pix];
        Cf[0] = im.x; Cf[1] = im.y; Cf[2] = im.z; Tf = im.w;
        gC[0] = gi.x; gC[1] = gi.y; gC[2] = gi.z; gT = gi.w;
    }
    const float kT = gT * Tf;
    bool done = !inside;
    float T = 1.0f, Ca[3] = {0.0f, 0.0f, 0.0f};
    const float alpha_min = 1.0f / 255.0f;
    for (uint32_t b = rg.x; b < rg.y; b += RASTER_BATCH) {
        const uint32_t i = b + tid, n_left = rg.y - b, slots = listed_slots(n_left);
        if (tid < slots) {
#pragma unroll
            for (int sw = 0; sw < 8; ++sw) s_pm[sw][tid] = 0u;
        }
        if (i < rg.y) {
            const uint32_t rs = __ldg(pair_vals + i);
            const float4* r = rec + (size_t)rs * 4;
            const float4 r0 = __ldg(r + 0), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
            const uint32_t lo = __float_as_uint(r1.w), hi = __float_as_uint(r2.w);
            s_row[tid] = rs;
            s_a[tid] = make_float4(r0.x, r0.w, r0.y, r1.x);
            s_b[tid] = make_float4(r0.z, r1.y, r1.z, r2.x);
            s_c[tid] = make_float4(r2.y, r2.z, 0.5f * (float)((lo & 0xFFFFu) + (hi & 0xFFFFu) + 1u),
                                   0.5f * (float)((lo >> 16) + (hi >> 16) + 1u));
            if (!RECT) s_q3[tid] = __ldg(r + 3);
            mask_rows<RECT>(s_pm, tid, r0, r1, r2, wx0, ty0, margin);
        }
        __syncthreads();
        if (__any_sync(FULL_MASK, !done)) {
            uint32_t count = 0u, longest = 0u;  // entries of this lane's group's list, and of the warp's longest
            {
                uint32_t n[4] = {};
#pragma unroll 1
                for (uint32_t c = 0; c < slots; c += 32u) {
                    const uint32_t m = s_pm[w][c + lane];
                    if (!__any_sync(FULL_MASK, m != 0u)) continue;
#pragma unroll
                    for (uint32_t q = 0; q < 4u; ++q) {
                        const bool hit = (m & (0x000F000Fu << (4u * q))) != 0u;
                        const uint32_t hits = __ballot_sync(FULL_MASK, hit);
                        if (hit) s_list[w][q][n[q] + __popc(hits & lt)] = (uint8_t)(c + lane);
                        n[q] += __popc(hits);
                    }
                }
#pragma unroll
                for (uint32_t q = 0; q < 4u; ++q) {
                    count = grp == q ? n[q] : count;
                    longest = max(longest, n[q]);
                }
                __syncwarp();
            }
            // every lane runs every iteration (no early exits) so the group reductions are legal
            for (uint32_t k = 0; k < longest; ++k) {
                uint32_t j = 0u;
                bool contrib = false;
                float g[GR];
#pragma unroll
                for (int m = 0; m < GR; ++m) g[m] = 0.0f;
                if (k < count) {
                    j = s_list[w][grp][k];
                    if (!done && (s_pm[w][j] & my_pixel) != 0u) {
                        const float4 qa = s_a[j], qb = s_b[j];
                        const float2 tc = fma2(make_float2(qa.z, qa.w), make_float2(Y, Y),
                                               fma2(make_float2(qa.x, qa.y), make_float2(X, X), make_float2(qb.x, qb.y)));
                        bool cov;
                        if (RECT) {
                            cov = fabsf(tc.x) <= margin && fabsf(tc.y) <= margin;
                        } else {
                            const float4 q3 = s_q3[j];
                            const float dx = fmaf(psx, X, q3.x), dy = fmaf(psy, Y, q3.y);
                            cov = fabsf(dx) <= q3.z && fabsf(dy) <= q3.z;
                        }
                        const float power = fmaf(tc.x, tc.x, tc.y * tc.y);
                        const float a = qb.z;
                        float E = 0.0f, alpha = 0.0f;
                        if (cov) {
                            E = spl_expf_falloff<FAR>(-0.5f * power);
                            alpha = a * E;
                        }
                        if (cov && !(alpha < alpha_min)) {
                            contrib = true;
                            const float4 qc = s_c[j];
                            const float rgb[3] = {qb.w, qc.x, qc.y};
                            float s[3], dS[3];
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                s[c] = __saturatef(rgb[c] * alpha);
                                dS[c] = gC[c] * T;
                                Ca[c] = s[c] * T + Ca[c];  // the forward's operation order
                            }
                            const float om = 1.0f - __saturatef(alpha);
                            float dsa = 0.0f;
                            if (om > 0.0f) {  // om in (0, 1]: the fast divide is within 2 ulp
                                const float Sdot =
                                    (gC[0] * (Cf[0] - Ca[0]) + gC[1] * (Cf[1] - Ca[1])) + gC[2] * (Cf[2] - Ca[2]);
                                dsa = __fdividef(-(Sdot + kT), om);
                            }
                            T = T * om;
                            done = T < FP32_T_MIN;
                            float dalpha = alpha < 1.0f ? dsa : 0.0f;
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                if (s[c] > 0.0f && s[c] < 1.0f) {  // the clamp passes it on
                                    dalpha += dS[c] * rgb[c];
                                    g[7 + c] = dS[c] * alpha;
                                }
                            }
                            g[6] = dalpha * E;
                            const float dpow = -0.5f * (dalpha * a * E);
                            const float dtx = 2.0f * dpow * tc.x, dty = 2.0f * dpow * tc.y;
                            // A against offsets from the box centre (Xr, Yr), B at that centre
                            const float ox = X - qc.z, oy = Y - qc.w;
                            g[0] = dtx * ox;
                            g[1] = dtx * oy;
                            g[2] = dtx;
                            g[3] = dty * ox;
                            g[4] = dty * oy;
                            g[5] = dty;
                        }
                    }
                }
                // reduce over the lanes of the group (all hold the same record this iteration)
                const uint32_t gm = __ballot_sync(FULL_MASK, contrib);
                if (gm != 0u) {
                    float v0, v1;
                    const uint32_t k0 = reduce10_over8(g, li, v0, v1);
                    if ((gm >> (grp * 8u)) & 0xFFu) {
                        float* dst = grad_rec + (size_t)s_row[j] * GR + k0;
                        atomicAdd(dst, v0);
                        if ((li & 3u) == 0u) atomicAdd(dst + 1, v1);
                    }
                }
            }
        }
        // no wait for the other warps after the last batch
        if (n_left <= (uint32_t)RASTER_BATCH || __syncthreads_and(done)) break;
    }
}

// One splat's inputs to the vertex-stage backward: its parameters and SH coefficients, and the view-plane
// position of its record's reference pixel (the centre of the record's pixel box).
template <int SHO>
struct VjpInputs {
    float cx, cy, cz, rx, ry;
    float4 rot, sca;
    float sh[48];
    __device__ __forceinline__ void load(const SceneView& s, const Uniforms& u, uint32_t i, uint2 bb) {
        cx = __ldg(s.x + i);
        cy = __ldg(s.y + i);
        cz = __ldg(s.z + i);
        rot = __ldg(s.rot + i);
        sca = __ldg(s.scale_alpha + i);
        // 16-byte loads of the row's first NF coefficients (rows are 192 bytes, 16-byte aligned; the
        // last load of SH degree 2 also reads coefficient 27, inside the row)
        constexpr int NF4 = (3 * (SHO + 1) * (SHO + 1) + 3) / 4;
        const float4* p = reinterpret_cast<const float4*>(s.sh + (size_t)i * 48);
#pragma unroll
        for (int k = 0; k < NF4; ++k) {
            const float4 v = __ldg(p + k);
            sh[4 * k + 0] = v.x;
            sh[4 * k + 1] = v.y;
            sh[4 * k + 2] = v.z;
            sh[4 * k + 3] = v.w;
        }
        const float Xr = 0.5f * (float)((bb.x & 0xFFFFu) + (bb.y & 0xFFFFu) + 1u);
        const float Yr = 0.5f * (float)((bb.x >> 16) + (bb.y >> 16) + 1u);
        const float vw = u.view_size[0], vh = u.view_size[1];
        rx = Xr * ((2.0f * vw) / (float)u.image_size[0]) - vw;
        ry = vh - Yr * ((2.0f * vh) / (float)u.image_size[1]);
    }
    template <class T, bool COV, int PARTS>
    __device__ __forceinline__ void vjp(const Uniforms& u, const float* g, T* gin) const {
        vertex_vjp_t<T, SHO, COV, PARTS>(u, cx, cy, cz, rot.x, rot.y, rot.z, rot.w, sca.x, sca.y, sca.z, sh, rx, ry, g,
                                             gin);
    }
};

__device__ __forceinline__ bool load_record_gradient(const float* grad_rec, uint32_t slot, float* g) {
    const float2* gr = reinterpret_cast<const float2*>(grad_rec + (size_t)slot * GR);  // 40-byte rows
    bool any = false;
#pragma unroll
    for (int k = 0; k < GR / 2; ++k) {
        const float2 v = gr[k];
        g[2 * k] = v.x;
        g[2 * k + 1] = v.y;
        any = any || v.x != 0.0f || v.y != 0.0f;
    }
    return any;  // false: not drawn, or no gradient reached it
}

// The centre, rotation, scale and opacity gradients of splat i (set, or added to what is there).
__device__ __forceinline__ void store_splat_gradient(uint32_t i, const float* gin, float galpha, float* gx, float* gy,
                                                     float* gz, float4* grot, float4* gscale_alpha, bool accumulate) {
    if (accumulate) {  // several frames' gradients summed in place, one frame after another
        // loaded and stored: reductions in the L2 take subnormal sums to zero (and are no faster: a step of eight views of
        // 1M splats 3,002 us with them, 2,989 us so)
        const float4 r0 = grot[i], s0 = gscale_alpha[i];
        gx[i] += gin[0];
        gy[i] += gin[1];
        gz[i] += gin[2];
        grot[i] = make_float4(r0.x + gin[3], r0.y + gin[4], r0.z + gin[5], r0.w + gin[6]);
        gscale_alpha[i] = make_float4(s0.x + gin[7], s0.y + gin[8], s0.z + gin[9], s0.w + galpha);
    } else {
        gx[i] = gin[0];
        gy[i] = gin[1];
        gz[i] = gin[2];
        grot[i] = make_float4(gin[3], gin[4], gin[5], gin[6]);
        gscale_alpha[i] = make_float4(gin[7], gin[8], gin[9], galpha);
    }
}

// Float sweep of every drawn splat but the needles and discs (needs_double_sweep), whose slots go to
// `deferred` ([0] the count, then the slots) for k_preprocess_backward_double; SH gradients of all.
template <int SHO, bool COV>
__global__ void __launch_bounds__(128, 4) k_preprocess_backward(SceneView s, Uniforms u, const uint32_t* __restrict__ idx,
                                                             const FrameCounters* __restrict__ fc,
                                                             const uint2* __restrict__ boxes,
                                                             const float* __restrict__ grad_rec, float* gx, float* gy,
                                                             float* gz, float4* grot, float4* gscale_alpha,
                                                             float* gsh, uint32_t* deferred, uint32_t deferred_cap,
                                                             bool accumulate) {
    frame_step(idx, fc, boxes, grad_rec);
    const uint32_t V = fc->visible;
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < V; slot += gridDim.x * blockDim.x) {
        float g[GR];
        if (!load_record_gradient(grad_rec, slot, g)) continue;
        const uint32_t i = __ldg(idx + slot);
        VjpInputs<SHO> in;
        in.load(s, u, i, __ldg(boxes + slot));
        if (needs_double_sweep(in.sca.x, in.sca.y, in.sca.z)) {
            const uint32_t pos = atomicAdd(deferred, 1u);
            if (pos < deferred_cap) deferred[1 + pos] = slot;
        } else {
            float gin[10];
            in.template vjp<float, COV, VJP_ALL>(u, g, gin);
#pragma unroll
            for (int m = 0; m < 10; ++m) gin[m] = finite_gradient(gin[m]);
            store_splat_gradient(i, gin, g[6], gx, gy, gz, grot, gscale_alpha, accumulate);
        }
        // SH: rgb_c = 0.5 + sum_k B_k(d) sh[3k + c]
        const float vx = in.cx - u.camera[12], vy = in.cy - u.camera[13], vz = in.cz - u.camera[14];
        const float len = sqrtf((vx * vx + vy * vy) + vz * vz);
        float B[16];
        sh_basis<SHO>(vx / len, vy / len, vz / len, B);
        // coefficient m = 3 k + c gets B[k] g[7 + c]: whole 16-byte groups, then the tail
        constexpr int NF = 3 * (SHO + 1) * (SHO + 1), NV = NF / 4;
        float v[NF];
#pragma unroll
        for (int m = 0; m < NF; ++m) v[m] = B[m / 3] * g[7 + m % 3];
        float* o = gsh + (size_t)i * 48;
        float4* o4 = reinterpret_cast<float4*>(o);
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            float4 x = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            if (accumulate) {
                const float4 y = o4[k];
                x = make_float4(y.x + x.x, y.y + x.y, y.z + x.z, y.w + x.w);
            }
            o4[k] = x;
        }
#pragma unroll
        for (int m = 4 * NV; m < NF; ++m) o[m] = accumulate ? o[m] + v[m] : v[m];
    }
}

// The deferred needles and discs, swept in double (same formulas, same float forward values).  
// A double operation holds its scheduler's pipe for some 30 cycles whatever the number of lanes, so that even one
// splat's sweep, some 2000 of them one after another, took 65 us, as long as the float sweep of 500k splats; fused
// products and shared reciprocals take it to 41 us.  A block takes 32 splats, a warp each for the gradients' three
// parts: 26 us.  (Computing what the parts share again costs more than it gives above some 40k needles: 150k of 1M
// splats, eight views' backward 3338 us, 2980 us with a thread per splat, 3420 us before; a branch to that in the same
// kernel makes the few needles' sweep 36 us.)
template <int SHO, bool COV>
__global__ void __launch_bounds__(96) k_preprocess_backward_double(SceneView s, Uniforms u,
                                                                    const uint32_t* __restrict__ idx,
                                                                    const uint2* __restrict__ boxes,
                                                                    const float* __restrict__ grad_rec, float* gx,
                                                                    float* gy, float* gz, float4* grot,
                                                                    float4* gscale_alpha,
                                                                    const uint32_t* __restrict__ deferred,
                                                                    uint32_t deferred_cap, bool accumulate) {
    frame_step(idx, boxes, grad_rec, deferred);
    const uint32_t n = min(deferred[0], deferred_cap);
    __shared__ double s_part[2][10][32];
    const uint32_t lane = threadIdx.x & 31u, part = threadIdx.x >> 5;
    for (uint32_t k0 = blockIdx.x * 32u; k0 < n; k0 += gridDim.x * 32u) {
        const uint32_t k = k0 + lane;
        float g[GR];
        double gin[10];
        uint32_t i = 0;
        if (k < n) {
            const uint32_t slot = deferred[1 + k];
            load_record_gradient(grad_rec, slot, g);
            i = __ldg(idx + slot);
            VjpInputs<SHO> in;
            in.load(s, u, i, __ldg(boxes + slot));
            if (part == 0)
                in.template vjp<double, COV, VJP_OUTLINE>(u, g, gin);
            else if (part == 1)
                in.template vjp<double, COV, VJP_AXES>(u, g, gin);
            else
                in.template vjp<double, COV, VJP_COLOUR>(u, g, gin);
            if (part != 0) {
#pragma unroll
                for (int m = 0; m < 10; ++m) s_part[part - 1][m][lane] = gin[m];
            }
        }
        __syncthreads();
        if (part == 0 && k < n) {
            float sum[10];
#pragma unroll
            for (int m = 0; m < 10; ++m) sum[m] = finite_gradient(gin[m] + s_part[0][m][lane] + s_part[1][m][lane]);
            store_splat_gradient(i, sum, g[6], gx, gy, gz, grot, gscale_alpha, accumulate);
        }
        __syncthreads();
    }
}

void launch_backward(int sh_order, bool covariance, bool rect, const SceneView& s, const Uniforms& u,
                     const uint32_t* idx, const FrameCounters* fc, const uint2* boxes, const uint2* ranges,
                     const uint4* tile_order, const uint32_t* pair_vals, const float4* rec, const float4* image,
                     const float4* grad_image, float* grad_rec, uint32_t* deferred,
                     uint32_t max_n, float* gx, float* gy, float* gz, float4* grot, float4* gscale_alpha, float* gsh,
                     bool accumulate, cudaStream_t st) {
    const int W = (int)u.image_size[0], H = (int)u.image_size[1];
    const int tiles_x = (W + TILE_PIXELS - 1) / TILE_PIXELS, tiles_y = (H + TILE_PIXELS - 1) / TILE_PIXELS;
    const float psx = (2.0f * u.view_size[0]) / (float)W;
    const float psy = -((2.0f * u.view_size[1]) / (float)H);
    uint32_t zg = (max_n * GR + 255) / 256;
    if (zg > device_sm_count() * 8u) zg = device_sm_count() * 8u;
    if (zg == 0) zg = 1;
    launch_after(k_zero_grad_rec, zg, 256, st, grad_rec, fc, deferred);
    const int grid = tiles_x * tiles_y;
    if (!raster_orders_tiles((uint64_t)grid)) tile_order = nullptr;
    if (grid > 0) {
        auto k = !rect ? k_raster_backward<false, true>
                       : (fabsf(u.margin) <= RASTER_NEAR_MARGIN ? k_raster_backward<true, false> : k_raster_backward<true, true>);
        launch_after(k, (uint32_t)grid, 256, st, ranges, tile_order, pair_vals, rec, W, H, tiles_x, u.margin, psx, psy, image,
                     grad_image, grad_rec);
    }
    if (max_n == 0) return;
    uint32_t blocks = (max_n + 127) / 128;
    if (blocks > device_sm_count() * 16u) blocks = device_sm_count() * 16u;
    // the double sweep's grid: a few blocks per SM (needles and discs are few; the count is on the device)
    const uint32_t dblocks = device_sm_count() * 2u;
#define PB(SHO, COV)                                                                                          \
    do {                                                                                                      \
        launch_after(k_preprocess_backward<SHO, COV>, blocks, 128, st, s, u, idx, fc, boxes, grad_rec, gx, gy, gz, \
                     grot, gscale_alpha, gsh, deferred, max_n, accumulate);                                        \
        launch_after(k_preprocess_backward_double<SHO, COV>, dblocks, 96, st, s, u, idx, boxes, grad_rec, gx, gy, \
                     gz, grot, gscale_alpha, deferred, max_n, accumulate);                                         \
    } while (0)
    switch (sh_order * 2 + (covariance ? 1 : 0)) {
        case 0: PB(0, false); break;
        case 1: PB(0, true); break;
        case 2: PB(1, false); break;
        case 3: PB(1, true); break;
        case 4: PB(2, false); break;
        case 5: PB(2, true); break;
        case 6: PB(3, false); break;
        default: PB(3, true); break;
    }
#undef PB
}

}  // namespace spl
