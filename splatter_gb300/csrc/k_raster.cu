// Compute rasteriser for the splat records (sm_103a).  The reference draws each splat as a rotated
// rectangle (triangle strip, renderer.rs:275-283) through the fixed-function rasteriser, runs the
// Gaussian fragment (shaders.wgsl:580-592) and blends front-to-back into a Bgra8Unorm target with
// destination alpha as transmittance (renderer.rs:260-271).  There is no fixed-function unit here,
// so the frame is tiled into 16x16-pixel tiles:
//   k_bin          - for each drawn entry in depth order, the tiles its pixel box touches; emitted as
//                    (tile id, record slot) pairs at offsets from a decoupled look-back scan, emitted in
//                    chunks of 128 pairs dealt to the CTA's warps and, for the onesweep sort, the
//                    tile-id digit histograms
//   (a stable radix sort of the pairs by tile id, so each tile's list stays in depth order)
//   k_tile_ranges  - start/end of each tile's run in the sorted pair list
//   k_tile_order   - the raster's tile order: most pairs first
//   k_raster       - one CTA per tile, one thread per pixel; records staged through shared memory in
//                    batches of 256, per-pixel record lists from the boxes (bit-transposed ballots),
//                    exact coverage test, falloff, blend, and early exit once every pixel of the tile
//                    is opaque
#include "spl_raster.cuh"

namespace spl {

// ------------------------------------------------------------------------------------------------
// Bound by latency (the ticket, the entries' boxes in a random gather, the look-back).  Emission in chunks dealt to
// the warps instead of 1024 pairs at a time by the CTA with four barriers: 66 -> 59 us at 6M splats, 1080p, 102 -> 86
// us at 3840x2160; tiles of 512 entries instead of 1024: 59 and 70 us, 1M splats 22 -> 16 us (tiles of 256: 14 us at
// 1M, but 83 us at 6M, where 17k tickets at some 5 ns each set the pace; tiles of 2048: 94 us).
constexpr int BIN_LB = 2, BIN_CTAS = 8;
constexpr uint32_t BIN_CHUNK = 128;  // pairs that a warp emits at a time
constexpr int BIN_PER = BIN_TILE / 256;  // consecutive draw entries per thread (depth order)
template <bool ORDERED, bool HIST>
__global__ void __launch_bounds__(256, BIN_CTAS) k_bin(const uint32_t* __restrict__ order, const uint2* __restrict__ boxes,
                                             FrameCounters* fc, int mode, const uint32_t* __restrict__ epoch_word,
                                             uint64_t* status, uint32_t* __restrict__ pair_keys,
                                             uint32_t* __restrict__ pair_vals, uint32_t pair_cap, int tiles_x,
                                             uint2* __restrict__ ranges, uint32_t tiles, uint32_t spin_limit) {
    __shared__ uint32_t s_off[BIN_TILE + 1];  // exclusive pair offsets of the tile's entries, and their sum
    __shared__ uint32_t s_slot[BIN_TILE];
    __shared__ uint32_t s_box[BIN_TILE];  // tx0 | ty0 << 16
    __shared__ uint16_t s_bw[BIN_TILE];
    __shared__ uint4 s_map[8][BIN_CHUNK / 4];  // [warp]: entry + 1 at each entry's first place in the chunk
    __shared__ uint32_t s_hist[HIST ? 768 : 1];
    __shared__ uint32_t s_scan[8];
    __shared__ uint32_t s_tile, s_epoch, s_base, s_draw;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    frame_step(order, boxes, epoch_word);
    // every tile's range starts empty
    for (uint32_t i = blockIdx.x * 256u + tid; i < tiles; i += gridDim.x * 256u) ranges[i] = make_uint2(0u, 0u);
    if (tid == 0) {
        s_tile = atomicAdd(&fc->tile_counter[8].v, 1u);
        s_epoch = *epoch_word;
        const uint32_t V = fc->visible;
        uint32_t draw = V;
        if (mode == DS_GPU) draw = V - fc->keys_all_ones;
        else if (mode == DS_GPU_INDIRECT) draw = V - fc->keys_top_ff;
        s_draw = draw;
    }
    if (HIST) {
        s_hist[tid] = 0u;
        s_hist[tid + 256] = 0u;
        s_hist[tid + 512] = 0u;
    }
    __syncthreads();
    const uint32_t tile = s_tile, epoch = s_epoch, draw = s_draw;
    const uint32_t ntiles = (draw + BIN_TILE - 1) / BIN_TILE;
    if (tile >= ntiles) {
        if (tile == 0 && tid == 0) {  // nothing to draw at all
            fc->draw = 0;
            fc->pairs = 0;
        }
        return;
    }
    if (tile == 0 && tid == 0) fc->draw = draw;
    // per-entry tile counts (consecutive entries per thread keep the thread order = depth order)
    uint32_t cnt[BIN_PER], tsum = 0;
#pragma unroll
    for (int e = 0; e < BIN_PER; ++e) {
        const uint32_t r = tile * BIN_TILE + tid * (uint32_t)BIN_PER + e;
        uint32_t c = 0, slot = 0, box = 0, bw = 0;
        if (r < draw) {
            slot = ORDERED ? __ldg(order + r) : r;
            const uint2 bb = __ldg(boxes + slot);
            const uint32_t lo = bb.x, hi = bb.y;
            const uint32_t x0 = lo & 0xFFFFu, y0 = lo >> 16, x1 = hi & 0xFFFFu, y1 = hi >> 16;
            if (x0 <= x1 && y0 <= y1) {
                const uint32_t tx0 = x0 / TILE_PIXELS, tx1 = x1 / TILE_PIXELS;
                const uint32_t ty0 = y0 / TILE_PIXELS, ty1 = y1 / TILE_PIXELS;
                bw = tx1 - tx0 + 1u;
                c = bw * (ty1 - ty0 + 1u);
                box = tx0 | (ty0 << 16);
            }
        }
        cnt[e] = c;
        s_slot[tid * BIN_PER + e] = slot;
        s_box[tid * BIN_PER + e] = box;
        s_bw[tid * BIN_PER + e] = (uint16_t)bw;
        tsum += c;
    }
    uint32_t btot;
    uint32_t off = block_exclusive_scan_256(tsum, s_scan, &btot);
#pragma unroll
    for (int e = 0; e < BIN_PER; ++e) {
        s_off[tid * BIN_PER + e] = off;
        off += cnt[e];
    }
    if (tid == 255u) s_off[BIN_TILE] = off;
    if (tid < 32) {
        if (tid == 0) lb_store(status + lb_word(tile), lb_pack(epoch, tile == 0 ? LB_INC : LB_AGG, btot));
        const uint32_t excl = lookback_single<BIN_LB>(status, tile, epoch, spin_limit, &fc->err);
        if (tid == 0) {
            if (tile != 0) lb_store(status + lb_word(tile), lb_pack(epoch, LB_INC, excl + btot));
            s_base = excl;
            if (tile == ntiles - 1) {
                fc->pairs = excl + btot;
                if (excl + btot > pair_cap) atomicOr(&fc->err, SPL_DEV_ERR_PAIR_OVERFLOW);
            }
        }
    }
    __syncthreads();
    const uint32_t gbase = s_base;
    // Emission in chunks of 128 pairs, dealt to the warps in turn (the nearest splats, first in the order, may
    // cover thousands of tiles each), no CTA barriers: the warp finds the entry of the chunk's first pair by two
    // ballots over the offsets, entries that start in the chunk mark their first place (entry + 1), and the last mark
    // at or before a place is its entry.  Lanes emit consecutive pairs.
    uint32_t* map = reinterpret_cast<uint32_t*>(s_map[w]);
    const uint32_t le = 0xFFFFFFFFu >> (31u - lane);
    for (uint32_t q0 = w * BIN_CHUNK; q0 < btot; q0 += 8u * BIN_CHUNK) {
        s_map[w][lane] = make_uint4(0u, 0u, 0u, 0u);
        // the last entry that starts at or before q0 (offsets rise; the first one is 0): a 32nd of the tile, then entry
        constexpr uint32_t B = BIN_TILE / 32;
        const uint32_t blk = (uint32_t)__popc(__ballot_sync(FULL_MASK, s_off[B * lane] <= q0)) - 1u;
        uint32_t first = B * blk + (uint32_t)__popc(__ballot_sync(FULL_MASK, lane < B && s_off[B * blk + lane] <= q0)) - 1u;
        const uint32_t before = first + 1u;  // as a mark
        __syncwarp();
        for (bool more = true; more; first += 32u) {
            const uint32_t e = first + 1u + lane;
            const uint32_t o = e < (uint32_t)BIN_TILE ? s_off[e] : btot;
            if (o < q0 + BIN_CHUNK && o < btot && s_off[e + 1u] != o) map[o - q0] = e + 1u;
            more = __all_sync(FULL_MASK, o < q0 + BIN_CHUNK && o < btot);
        }
        __syncwarp();
        uint32_t carry = before;
#pragma unroll
        for (uint32_t k = 0; k < BIN_CHUNK; k += 32u) {
            const uint32_t q = q0 + k + lane;
            const uint32_t mark = map[k + lane];
            const uint32_t upto = __ballot_sync(FULL_MASK, mark != 0u) & le;
            const uint32_t found = __shfl_sync(FULL_MASK, mark, upto ? 31 - __clz(upto) : 0);
            const uint32_t e = (upto ? found : carry) - 1u;
            carry = __shfl_sync(FULL_MASK, e, 31) + 1u;
            if (q < btot) {
                const uint32_t li = q - s_off[e];
                const uint32_t bw = s_bw[e], box = s_box[e];
                // li / bw and li % bw (li < 2^24): float estimate, corrected by one step
                uint32_t dy = __float2uint_rz(__fdividef((float)li, (float)bw));
                int32_t dx = (int32_t)(li - dy * bw);
                if (dx < 0) {
                    --dy;
                    dx += (int32_t)bw;
                } else if (dx >= (int32_t)bw) {
                    ++dy;
                    dx -= (int32_t)bw;
                }
                const uint32_t tid_tile = ((box >> 16) + dy) * (uint32_t)tiles_x + (box & 0xFFFFu) + (uint32_t)dx;
                const uint32_t g = gbase + q;
                if (g < pair_cap) {
                    pair_keys[g] = tid_tile;
                    pair_vals[g] = s_slot[e];
                    if (HIST) {
                        atomicAdd(&s_hist[tid_tile & 255u], 1u);
                        atomicAdd(&s_hist[256u + ((tid_tile >> 8) & 255u)], 1u);
                        atomicAdd(&s_hist[512u + ((tid_tile >> 16) & 255u)], 1u);
                    }
                }
            }
        }
        __syncwarp();
    }
    if (HIST) {
        __syncthreads();
        for (uint32_t i = tid; i < 768u; i += 256u) {
            const uint32_t v = s_hist[i];
            if (v) atomicAdd(&fc->hist_pairs[0][0] + i, v);
        }
    }
}

void launch_bin(int mode, bool hist, const uint32_t* order, const uint2* boxes, FrameCounters* fc,
                const uint32_t* epoch_word, uint64_t* status, uint32_t* pair_keys, uint32_t* pair_vals,
                uint32_t pair_cap, int tiles_x, uint2* ranges, uint32_t tiles, uint32_t max_n, uint32_t spin_limit,
                cudaStream_t st) {
    const uint32_t grid = max_n == 0 ? 1u : (max_n + BIN_TILE - 1) / BIN_TILE;
    auto k = order ? (hist ? k_bin<true, true> : k_bin<true, false>) : (hist ? k_bin<false, true> : k_bin<false, false>);
    launch_after(k, grid, 256, st, order, boxes, fc, mode, epoch_word, status, pair_keys, pair_vals, pair_cap, tiles_x,
                 ranges, tiles, spin_limit);
}

// ------------------------------------------------------------------------------------------------
__global__ void k_tile_ranges(const uint32_t* __restrict__ keys, const FrameCounters* __restrict__ fc,
                              uint32_t pair_cap, uint2* ranges) {
    frame_step(keys, fc);
    const uint32_t P = min(fc->pairs, pair_cap);
    // four keys per thread (one 16-byte load; the neighbours across the group edges loaded singly)
    const uint32_t groups = (P + 3u) / 4u;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < groups; g += gridDim.x * blockDim.x) {
        const uint32_t i0 = g * 4u;
        uint32_t k[4];
        if (i0 + 4u <= P) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(keys + i0));
            k[0] = v.x;
            k[1] = v.y;
            k[2] = v.z;
            k[3] = v.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) k[j] = i0 + j < P ? __ldg(keys + i0 + j) : 0u;
        }
        const bool has_prev = i0 > 0u, has_next = i0 + 4u < P;
        const uint32_t prev = has_prev ? __ldg(keys + i0 - 1u) : 0u;
        const uint32_t next = has_next ? __ldg(keys + i0 + 4u) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t i = i0 + j;
            if (i >= P) break;
            const bool starts = j > 0 ? k[j - 1] != k[j] : (!has_prev || prev != k[j]);
            const bool ends = i + 1u == P || (j < 3 ? k[j + 1] != k[j] : next != k[j]);
            if (starts) ranges[k[j]].x = i;
            if (ends) ranges[k[j]].y = i + 1u;
        }
    }
}

void launch_tile_ranges(const uint32_t* pair_keys, const FrameCounters* fc, uint32_t pair_cap, uint2* ranges,
                        cudaStream_t st) {
    if (pair_cap == 0) return;
    uint32_t grid = (pair_cap + 255) / 256;
    if (grid > device_sm_count() * 8u) grid = device_sm_count() * 8u;
    launch_after(k_tile_ranges, grid, 256, st, pair_keys, fc, pair_cap, ranges);
}

// ------------------------------------------------------------------------------------------------
// The raster's tile order: tiles with more (tile, splat) pairs first, in buckets of half an octave of
// the pair count (2 buckets per power of two), empty tiles last.  Tiles take very different times
// (dense clusters against open sky); started in row-major order, a few heavy tiles could begin in
// the last wave and set the kernel's end, while heavy-first is close to the longest-processing-time
// schedule.  Tiles are independent, so the order changes no pixel.  One CTA: bucket counts per warp, their scan in
// (bucket, warp) order, and a scatter of (pair range, tile) entries, which spare the raster a dependent load.
// Viewports whose tiles are all resident at once (up to 912) are not ordered.
// Lanes of the same bucket are found by five ballots instead of MATCH.ANY, which loops over the distinct values:
// 12.8 -> 9.3 us (one launch alone, cold) for 8,160 tiles, and the raster stage of 1M splats 80.6 -> 78.5 us with the
// ranges in the entries; frames of 2k splats 37.0 -> 35.5 us without the launch.
constexpr int ORDER_BUCKETS = 32;

__device__ __forceinline__ uint32_t order_bucket(uint2 r) {
    const uint32_t c = r.y - r.x;
    if (c == 0u) return ORDER_BUCKETS - 1;
    const uint32_t l = 31u - __clz(c);                         // floor(log2 c)
    const uint32_t half = l > 0u ? (c >> (l - 1u)) & 1u : 0u;  // the bit after the leading one
    return 30u - min(2u * l + half, 30u);                      // more pairs -> smaller bucket; 2^15 pairs on: 0
}

__device__ __forceinline__ uint32_t match_bucket(uint32_t b, bool valid) {
    uint32_t peers = __ballot_sync(FULL_MASK, valid);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const bool bit = (b >> k) & 1u;
        const uint32_t m = __ballot_sync(FULL_MASK, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

__global__ void __launch_bounds__(1024) k_tile_order(const uint2* __restrict__ ranges, uint32_t ntiles,
                                                     uint4* __restrict__ order) {
    __shared__ uint32_t cnt[ORDER_BUCKETS][33];  // [bucket][warp]: counts, then places
    __shared__ uint32_t tot[ORDER_BUCKETS];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5, lt = lanemask_lt();
    cnt[lane][w] = 0u;
    start_next();
    frame_step(ranges);
    __syncthreads();
    for (uint32_t t0 = 0; t0 < ntiles; t0 += 4096u) {
        uint2 r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t t = t0 + 1024u * k + tid;
            r[k] = t < ntiles ? __ldg(ranges + t) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (t0 + 1024u * k >= ntiles) break;
            const uint32_t b = order_bucket(r[k]), peers = match_bucket(b, t0 + 1024u * k + tid < ntiles);
            if (((peers >> lane) & 1u) != 0u && (peers & lt) == 0u) cnt[b][w] += __popc(peers);
            __syncwarp();
        }
    }
    __syncthreads();
    {  // warp w scans bucket w's counts over the warps, then all warps the totals
        const uint32_t v = cnt[w][lane];
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL_MASK, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31u) tot[w] = x;
        __syncthreads();
        const uint32_t below = __reduce_add_sync(FULL_MASK, lane < w ? tot[lane] : 0u);
        cnt[w][lane] = below + x - v;
    }
    __syncthreads();
    for (uint32_t t0 = 0; t0 < ntiles; t0 += 4096u) {
        uint2 r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t t = t0 + 1024u * k + tid;
            r[k] = t < ntiles ? __ldg(ranges + t) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t t = t0 + 1024u * k + tid;
            if (t0 + 1024u * k >= ntiles) break;
            const uint32_t b = order_bucket(r[k]), peers = match_bucket(b, t < ntiles);
            const uint32_t at = cnt[b][w];
            __syncwarp();
            if (t < ntiles) {
                if ((peers & lt) == 0u) cnt[b][w] = at + __popc(peers);
                order[at + __popc(peers & lt)] = make_uint4(r[k].x, r[k].y, t, 0u);
            }
            __syncwarp();
        }
    }
}

// ------------------------------------------------------------------------------------------------

// One CTA per 16x16 tile, one thread per pixel.  Warp w owns the strip of rows 2w, 2w+1; lane l holds
// column l & 15 and row 2w + l / 16.  The tile's records (depth order) are staged through shared memory in batches of 256,
// last record in slot 0, so that the highest set bit of a list word is its first record; the thread staging a
// record also forms its mask of the lanes (pixels) it may draw in each of the eight strips.  Warp-wide bit
// transposes, four 32-record words at a time, turn its strip's masks into each pixel's list of the batch's
// records, in place.  The warp then walks the 32 lists of the whole batch at once: in every iteration each
// pixel takes its next record, so one pass of the per-pixel code serves as many splats as there are lanes
// with work (most splats here cover a few pixels).  Per pixel: coverage test, falloff, 1/255 discard, blend —
// the operations of the oracle's raster_tile in the same order, so the image is bit-identical.  Lists are
// walked in depth order per pixel, a warp whose pixels are all finished skips the rest, and the CTA stops
// once every pixel is finished (T == 0 in unorm8 mode, T < 1e-4 in fp32 mode).
//
// Bound by instruction issue (3M splats, 1080p: 81% of issue slots, 194 M warp instructions, DRAM 16%), so the
// work per list entry and per record is what counts:
// * lists exact to a pixel row (column interval per row) instead of to a 2x2 block: a walk iteration's lanes
//   rarely miss the rectangle.  6M splats, 1080p: 400 -> 360 us; 3840x2160: 1,002 -> 924 us;
// * packed float pairs, the unorm8 target held as k / 255 in floats, no float-to-integer conversions or table
//   look-ups in the walk, byte permutes and rotations in the transposes, 40 bytes of shared memory read per
//   list entry instead of 48, two CTA barriers per batch instead of three: 483 -> 400 us; 1,207 -> 1,002 us
//   (without the packed pairs 417 and 1,062 us).
// Batches of 512 records (fewer, longer walks) lose more to the fewer resident CTAs: 483 us; five CTAs per
// SM at 48 registers, without spills: 416 us.

// The unorm8 value nearest to v in [0, 1] (k / 255, k = v * 255 rounded to nearest even), as the float
// nearest to k / 255: adding 2^23 leaves the integer k in the mantissa's last bits, and k / 255 is the
// product with the reciprocal's two-float expansion (equal to the correctly rounded quotient for all 256
// values).  No integer conversions (a quarter of the float rate or less) and no table look-ups.
__device__ __forceinline__ float2 quantise2(float2 v) {
    const float2 t = fma2(v, make_float2(255.0f, 255.0f), make_float2(0.0f, 0.0f));
    const float2 m = add2(t, make_float2(8388608.0f, 8388608.0f));
    const float2 k = add2(m, make_float2(-8388608.0f, -8388608.0f));
    const float2 lo = mul2(k, make_float2(UNORM_LO, UNORM_LO));
    return fma2(k, make_float2(UNORM_HI, UNORM_HI), lo);
}

// N 32x32 bit-matrix transposes across the warp: afterwards bit i of x[c] in lane l is bit l of the
// old x[c] in lane i.  Each step d exchanges lane-index bit d with bit-index bit d: whole bytes move by one
// byte permute for d = 16 and 8, smaller groups by a rotation and one bitwise select.  The N words go
// through each step together, so their independent shuffle chains overlap their latency (one word
// at a time, the list building took a quarter of the raster's warp time at 6M splats, 1080p).
template <int N>
__device__ __forceinline__ void transpose_lane_bits_n(uint32_t* x, uint32_t lane) {
    const uint32_t sel16 = (lane & 16u) ? 0x3276u : 0x5410u, sel8 = (lane & 8u) ? 0x3715u : 0x6240u;
#pragma unroll
    for (int c = 0; c < N; ++c) x[c] = __byte_perm(x[c], __shfl_xor_sync(FULL_MASK, x[c], 16), sel16);
#pragma unroll
    for (int c = 0; c < N; ++c) x[c] = __byte_perm(x[c], __shfl_xor_sync(FULL_MASK, x[c], 8), sel8);
    const uint32_t masks[3] = {0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t d = 4u >> k;
        const bool up = (lane & d) != 0u;
        const uint32_t keep = up ? ~masks[k] : masks[k], rot = up ? 32u - d : d;
#pragma unroll
        for (int c = 0; c < N; ++c) {
            const uint32_t p = __shfl_xor_sync(FULL_MASK, x[c], (int)d);
            x[c] = (x[c] & keep) | (__funnelshift_l(p, p, rot) & ~keep);
        }
    }
}

// Words c0 ... c0 + N - 1 of the warp's lists (see k_raster), in place.  A group whose records all miss the strip
// stays zero.
template <int N>
__device__ __forceinline__ void list_words(uint32_t (&masks)[RASTER_BATCH], uint32_t c0, uint32_t lane, uint32_t& nz) {
    uint32_t t[N], any = 0u;
#pragma unroll
    for (int c = 0; c < N; ++c) any |= t[c] = masks[(c0 + c) * 32u + lane];
    if (!__any_sync(FULL_MASK, any != 0u)) return;
    transpose_lane_bits_n<N>(t, lane);
#pragma unroll
    for (int c = 0; c < N; ++c) {
        masks[(c0 + c) * 32u + lane] = t[c];
        nz |= (t[c] != 0u ? 1u : 0u) << (c0 + c);
    }
}

// FAR: a covered pixel's exponent may fall below -87 (axis-aligned squares, or a margin above
// RASTER_NEAR_MARGIN), where the falloff takes spl_expf's general path.
template <bool RECT, int BLEND, bool FAR>
__global__ void __launch_bounds__(256, RASTER_CTAS) k_raster(const uint2* __restrict__ ranges, const uint4* __restrict__ tile_order,
                                                const uint32_t* __restrict__ pair_vals,
                                                const float4* __restrict__ rec, int W, int H, int tiles_x, float margin,
                                                float psx, float psy, void* __restrict__ out) {
    // the batch's records, rearranged for packed arithmetic: (A00, A10, A01, A11) (B0, B1, alpha, r) (g, b)
    __shared__ float4 s_a[RASTER_BATCH], s_b[RASTER_BATCH];
    __shared__ float2 s_c[RASTER_BATCH];
    __shared__ float4 s_q3[RECT ? 1 : RASTER_BATCH];
    // [strip][record]: lane masks of the batch's records; then [strip][word * 32 + lane]: the pixels' lists
    __shared__ uint32_t s_pm[8][RASTER_BATCH];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    frame_step(ranges, tile_order, pair_vals, rec);
    uint2 rg;
    int tile;
    ordered_tile(ranges, tile_order, rg, tile);
    const int tx = tile % tiles_x, ty = tile / tiles_x;
    const int wx0 = tx * TILE_PIXELS;
    const int px = wx0 + (int)(lane & 15u), py = ty * TILE_PIXELS + 2 * (int)w + (int)(lane >> 4);
    const float X = (float)px + 0.5f, Y = (float)py + 0.5f;
    const bool inside = px < W && py < H;
    bool done = !inside;
    bool warp_done = __all_sync(FULL_MASK, done);
    // (r, g) and (b, T): unorm8 values as floats k / 255, or the fp32 target
    float2 rgv = make_float2(0.0f, 0.0f), bt = make_float2(0.0f, 1.0f);
    const float alpha_min = 1.0f / 255.0f;
    for (uint32_t b = rg.x; b < rg.y; b += RASTER_BATCH) {
        const uint32_t i = b + tid, slot = RASTER_BATCH - 1u - tid;
        const uint32_t n = rg.y - b;  // records from here on; the batch has 256 of them at most
        if (tid < listed_slots(n)) {
#pragma unroll
            for (int sw = 0; sw < 8; ++sw) s_pm[sw][slot] = 0u;
        }
        if (i < rg.y) {
            const uint32_t rs = __ldg(pair_vals + i);
            const float4* r = rec + (size_t)rs * 4;
            const float4 r0 = __ldg(r + 0), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
            s_a[slot] = make_float4(r0.x, r0.w, r0.y, r1.x);
            s_b[slot] = make_float4(r0.z, r1.y, r1.z, r2.x);
            s_c[slot] = make_float2(r2.y, r2.z);
            if (!RECT) s_q3[slot] = __ldg(r + 3);
            mask_rows<RECT>(s_pm, slot, r0, r1, r2, wx0, ty * TILE_PIXELS, margin);
        }
        __syncthreads();
        if (!warp_done) {
            // Per-pixel lists of the batch: the strip's lane masks of slots 32c + l, transposed so that lane p
            // holds word c of pixel p's list (bit i: slot 32c + i); bit c of `nz` marks a non-empty word.
            uint32_t nz = 0u;
            if (n <= 32u) {
                list_words<1>(s_pm[w], 7u, lane, nz);
            } else if (n <= 64u) {
                list_words<2>(s_pm[w], 6u, lane, nz);
            } else {
                if (n > 128u) list_words<4>(s_pm[w], 0u, lane, nz);
                list_words<4>(s_pm[w], 4u, lane, nz);
            }
            // Walk the 32 lists at once across the whole batch: in every iteration each pixel takes its
            // next record.  The warp leaves once every pixel is finished or has walked its list.
            if (done) nz = 0u;
            uint32_t cur = 0u, cbase = 0u;
            while (true) {
                if (cur == 0u && nz != 0u) {
                    const uint32_t c = top_bit(nz);
                    nz ^= 1u << c;
                    cbase = c * 32u;
                    cur = s_pm[w][cbase + lane];
                }
                if (!__any_sync(FULL_MASK, cur != 0u)) break;
                if (cur == 0u) continue;
                const uint32_t bit = top_bit(cur);
                const uint32_t j = cbase + bit;
                cur ^= 1u << bit;
                const float4 qa = s_a[j], qb = s_b[j];
                const float2 tc = fma2(make_float2(qa.z, qa.w), make_float2(Y, Y),
                                       fma2(make_float2(qa.x, qa.y), make_float2(X, X), make_float2(qb.x, qb.y)));
                if (RECT) {
                    if (!(fabsf(tc.x) <= margin && fabsf(tc.y) <= margin)) continue;
                } else {
                    const float4 q3 = s_q3[j];
                    const float dx = fmaf(psx, X, q3.x), dy = fmaf(psy, Y, q3.y);
                    if (!(fabsf(dx) <= q3.z && fabsf(dy) <= q3.z)) continue;
                }
                const float power = fmaf(tc.x, tc.x, tc.y * tc.y);
                const float alpha = qb.z * spl_expf_falloff<FAR>(-0.5f * power);
                if (alpha < alpha_min) continue;
                const float2 qc = s_c[j];
                // __saturatef == clamp to [0, 1] (NaN -> 0)
                const float sr = __saturatef(qb.w * alpha), sg = __saturatef(qc.x * alpha);
                const float sb = __saturatef(qc.y * alpha), om = 1.0f - __saturatef(alpha);
                const float2 TT = make_float2(bt.y, bt.y);
                const float2 u = mul2(make_float2(sr, sg), TT), v = mul2(make_float2(sb, om), TT);
                if (BLEND == 0) {
                    rgv = quantise2(make_float2(__saturatef(u.x + rgv.x), __saturatef(u.y + rgv.y)));
                    bt = quantise2(make_float2(__saturatef(v.x + bt.x), v.y));
                    done = bt.y == 0.0f;
                } else {
                    rgv = make_float2(u.x + rgv.x, u.y + rgv.y);
                    bt = make_float2(v.x + bt.x, v.y);
                    done = bt.y < FP32_T_MIN;
                }
                if (done) cur = nz = 0u;
            }
            warp_done = __all_sync(FULL_MASK, done);
        }
        // no wait for the other warps after the last batch
        if (n <= (uint32_t)RASTER_BATCH || __syncthreads_and(done)) break;
    }
    if (inside) {
        const size_t pix = (size_t)py * (size_t)W + (size_t)px;
        if (BLEND == 0) {
            const auto byte = [](float v) { return (unsigned char)__float2int_rn(v * 255.0f); };
            reinterpret_cast<uchar4*>(out)[pix] = make_uchar4(byte(rgv.x), byte(rgv.y), byte(bt.x), byte(bt.y));
        } else {
            reinterpret_cast<float4*>(out)[pix] = make_float4(rgv.x, rgv.y, bt.x, bt.y);
        }
    }
}

bool raster_orders_tiles(uint64_t tiles) { return tiles > (uint64_t)device_sm_count() * RASTER_CTAS; }

typedef void (*RasterKernel)(const uint2*, const uint4*, const uint32_t*, const float4*, int, int, int, float,
                             float, float, void*);
static RasterKernel pick_raster(bool rect, int blend, float margin) {
    if (!rect) return blend == 0 ? k_raster<false, 0, true> : k_raster<false, 1, true>;
    if (fabsf(margin) <= RASTER_NEAR_MARGIN) return blend == 0 ? k_raster<true, 0, false> : k_raster<true, 1, false>;
    return blend == 0 ? k_raster<true, 0, true> : k_raster<true, 1, true>;
}

const void* raster_kernel(bool rect, int blend, float margin) {
    return reinterpret_cast<const void*>(pick_raster(rect, blend, margin));
}

void launch_raster(bool rect, int blend, const uint2* ranges, uint4* tile_order, const uint32_t* pair_vals,
                   const float4* rec, const Uniforms& u, void* out, cudaStream_t st) {
    const int W = (int)u.image_size[0], H = (int)u.image_size[1];
    const int tiles_x = (W + TILE_PIXELS - 1) / TILE_PIXELS, tiles_y = (H + TILE_PIXELS - 1) / TILE_PIXELS;
    const int grid = tiles_x * tiles_y;
    if (grid == 0) return;
    const float psx = (2.0f * u.view_size[0]) / (float)W;
    const float psy = -((2.0f * u.view_size[1]) / (float)H);
    if (!raster_orders_tiles((uint64_t)grid)) tile_order = nullptr;
    if (tile_order) launch_after(k_tile_order, 1, 1024, st, ranges, (uint32_t)grid, tile_order);
    launch_after(pick_raster(rect, blend, u.margin), (uint32_t)grid, 256, st, ranges, tile_order, pair_vals, rec, W, H,
                 tiles_x, u.margin, psx, psy, out);
}

}  // namespace spl
