// All passes of a stable LSD radix sort in ONE cooperative launch (sm_103a).
//
// The reference's GPU depth sort (radixSortA/B/C, Lichtso/splatter src/shaders.wgsl:298-498) is a
// onesweep sort whose tiles learn their global digit offsets through a decoupled look-back chain.
// At splat-pipeline sizes (a few million keys, L2-resident) that chain — one L2 round trip per
// tile — dominates.  Here every CTA is resident (cooperative launch, two 512-thread CTAs per SM) and
// owns one contiguous segment of the input; each 8-bit pass is:
//   1. digit counts of the segment.  A segment of at most one sub-tile (4096 keys) is loaded and ranked
//      at once (warp-level multisplit), which gives its counts; a longer one is counted first
//   2. the counts exchanged: every CTA publishes its 256 counts as tagged 64-bit words (epoch, pass, count:
//      valid words are recognised by themselves, so nothing is cleared and no barrier is waited for) and
//      reads those of its group of 16 CTAs; the group's last CTA publishes the group's sums, and every CTA
//      reads the sums of all groups.  Up to 32 CTAs read one another's counts directly.  The sums over all
//      CTAs give the digits' global bases, those over the CTAs before it this CTA's offsets
//   3. the keys and values, staged together through shared memory in digit order, written as runs,
//      sub-tile by sub-tile
//   4. a bounded grid barrier (the next pass reads this pass's output); none after the last pass
// The ranking keeps equal digits in input order, so every pass is stable, like the onesweep passes.
//
// What bounds it: a long pass (4.3M keys, 14k per CTA) is bound by the ranking's shared-memory and integer
// pipes (6 us per sub-tile and pair of CTAs), a short one (100k keys) by the chain of L2 round trips of the exchange
// and the barrier.  Measured (frame stages, four depth passes / two tile passes): counts exchanged by tagged
// words instead of two grid barriers around a scan, ranks before counts in short segments, no barrier after the
// last pass: 96k keys 47 -> 30 us, 340k 59 -> 36 us, 540k pairs 33 -> 22 us; lanes matched by shared atomics and
// ballots in turn (atomics alone 132 us, ballots alone 144), the next sub-tile's loads and the exchange behind
// other work, four CTA barriers per sub-tile instead of five: 4.3M keys 147 -> 122 us, 6M pairs 100 -> 81 us.
// Slower: 1024-thread CTAs (178 us: twice the count rows to scan), three CTAs per SM at 40 registers (180 us:
// spills), MATCH.ANY (183 us), sub-tiles of 8192 keys (165 us: spills).
// Every wait is bounded: on timeout the error bit is raised and the kernel runs to its end
// (writes stay in bounds), so a missing CTA can never hang the GPU.  The barrier word counts the
// launch's arrivals and must be zero when the launch starts (each sort of a frame has its own word in
// the frame counters, which the frame start zeroes).
#include <atomic>

#include "spl_device.cuh"

namespace spl {

constexpr int CS_THREADS = 512;               // two CTAs per SM
constexpr int CS_WARPS = CS_THREADS / 32;
constexpr int CS_KPT = 8;
constexpr int CS_TILE = CS_THREADS * CS_KPT;  // 4096 keys per sub-tile
constexpr int CS_MIN_SEG = CS_THREADS * 4;    // shortest segment of a sort of several CTAs
constexpr int CS_GROUP = 16;                  // CTAs of a group in the exchange of counts
constexpr int CS_DIRECT = 32;                 // up to this many CTAs exchange counts without groups
constexpr int CS_MAX_GRID = 512;
// Keys up to which the sort leaves room on the SMs for a kernel beside it: its CTAs have 32 K registers each, and
// one of two on an SM leaves (622 k keys) or ends early (a little above).  With 966 k keys a frame of 1M splats takes
// 331 us with the vertex stage beside the sort and 324 us without, with 799 k 253.7 and 256.0 us.
constexpr uint32_t CS_START_MAX = 3u << 18;
static_assert(CS_THREADS == 512 && CS_WARPS == 16, "the sub-tile scan maps digit t / 2 and 8 warps to thread t, "
                                                   "the exchange digit t & 255 and half of the words");

struct CoopSmem {
    uint2 buf[CS_TILE];                // (key, value) of the sub-tile in digit order
    uint32_t wcnt[CS_WARPS][256];      // per-warp digit counts -> exclusive prefixes
    uint32_t mask[CS_WARPS][256];      // per-warp lanes of each digit in the row being ranked; zero between rows
    uint32_t part[2][2][256];          // halves of a digit's prefix and total
    uint32_t next[256];                // global place of this CTA's next key of each digit
    uint32_t place[256];               // global place of sub-tile place 0 for keys of each digit
    uint32_t count[256];               // the sub-tile's digit counts
    uint32_t scan[CS_WARPS];
};

// A count as a word that is valid for one pass of one launch: [epoch:32 | pass:2 | count:30].
__device__ __forceinline__ uint64_t count_word(uint32_t epoch, uint32_t pass, uint32_t count) {
    return ((uint64_t)epoch << 32) | (pass << 30) | count;
}

struct CountTable {
    uint64_t* rows;    // [CTA][256], then [group][256]
    uint32_t epoch, pass, spin_limit;
    uint32_t* err;
    __device__ __forceinline__ uint64_t* group(uint32_t g) const { return rows + ((size_t)gridDim.x + g) * 256; }
    __device__ __forceinline__ void publish(uint64_t* p, uint32_t count) const { lb_store(p, count_word(epoch, pass, count)); }
    // Adds the counts of rows first, first + 2, ... < end (word d of each) to tot, those before `mine` to pre;
    // eight loads in flight.  A word that does not become valid in time counts as zero (the error bit is set).
    __device__ __forceinline__ void sum(const uint64_t* table, uint32_t d, uint32_t first, uint32_t end, uint32_t mine,
                                        uint32_t& pre, uint32_t& tot) const {
        const uint32_t tag = pass << 30;
        for (uint32_t k0 = first; k0 < end; k0 += 16u) {
            uint64_t v[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i)
                v[i] = k0 + 2u * i < end ? lb_load(table + (size_t)(k0 + 2u * i) * 256 + d) : 0u;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t k = k0 + 2u * i;
                if (k >= end) break;
                uint32_t spins = 0;
                while ((uint32_t)(v[i] >> 32) != epoch || ((uint32_t)v[i] & 0xC0000000u) != tag) {
                    if (++spins > spin_limit ||
                        ((spins & 1023u) == 0u && (ld_relaxed_u32(err) & SPL_DEV_ERR_LOOKBACK))) {
                        atomicOr(err, SPL_DEV_ERR_LOOKBACK);
                        v[i] = 0u;
                        break;
                    }
                    if (spins > 32u) __nanosleep(32);
                    v[i] = lb_load(table + (size_t)k * 256 + d);
                }
                const uint32_t c = (uint32_t)v[i] & 0x3FFFFFFFu;
                tot += c;
                if (k < mine) pre += c;
            }
        }
    }
};

// Grid barrier on a word that only counts arrivals (zero when the launch starts): the b-th barrier of
// the launch (b = 0, 1, ...) waits until *bar reaches (b + 1) * nblocks.  Releasing takes only the
// last arrival's atomic: no reset and no generation word on the critical path (those cost two more
// L2 round trips per barrier).
__device__ __forceinline__ void grid_barrier(uint32_t* bar, uint32_t target, uint32_t spin_limit, uint32_t* err) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        const volatile uint32_t* v = bar;
        uint32_t spins = 0;
        while (*v < target) {
            if (++spins > spin_limit) {
                atomicOr(err, SPL_DEV_ERR_LOOKBACK);
                break;
            }
            // a wait of this launch already timed out: the later ones would too, each after its own
            // spin limit; stop waiting (the frame reports the error)
            if ((spins & 1023u) == 0u && (*(volatile uint32_t*)err & SPL_DEV_ERR_LOOKBACK)) break;
            if (spins > 32) __nanosleep(32);
        }
        __threadfence();
    }
    __syncthreads();
}

// Block-wide exclusive scan over 256 values held by threads 0..255 (other threads pass 0 and ignore
// the result).  Uses sm->scan; every thread of the CTA must call it.
__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t* scan, uint32_t* total) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31 && w < 8) scan[w] = x;
    __syncthreads();
    uint32_t pre = 0, tot = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t s = scan[i];
        pre += i < w ? s : 0u;
        tot += s;
    }
    __syncthreads();
    *total = tot;
    return pre + x - v;
}

// A sub-tile's keys and values: key[j] is element wb + 32 j (warp w owns 32 R consecutive elements), valid
// below `end`.  FULL: all are.
template <int R, bool FULL>
__device__ __forceinline__ void load_subtile(uint32_t (&key)[R], uint32_t (&val)[R], const uint32_t* kin,
                                             const uint32_t* vin, bool iota, uint32_t wb, uint32_t end) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const uint32_t e = wb + 32u * j;
        key[j] = FULL || e < end ? __ldcg(kin + e) : 0u;
    }
    if (iota) {
#pragma unroll
        for (int j = 0; j < R; ++j) val[j] = wb + 32u * j;
    } else {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t e = wb + 32u * j;
            val[j] = FULL || e < end ? __ldcg(vin + e) : 0u;
        }
    }
}

// Ranks a sub-tile's keys by the digit at `shift` (warp-level multisplit: equal digits keep their input
// order): pos[j] is the key's rank among its warp's keys of the digit, sm.wcnt each (warp, digit)'s first
// place in the sub-tile's digit order.  The thread that owns digit tid / 2 (odd tid) gets the digit's first
// place and count.  Every thread of the CTA calls it; sm.wcnt is complete after the next CTA barrier.
template <int R, bool FULL>
__device__ __forceinline__ void rank_subtile(CoopSmem& sm, const uint32_t (&key)[R], uint32_t (&pos)[R], uint32_t wb,
                                             uint32_t end, int shift, uint32_t lt, uint32_t& first, uint32_t& count) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
#pragma unroll
    for (int k = 0; k < 8; ++k) sm.wcnt[w][lane + 32 * k] = 0u;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const bool valid = FULL || wb + 32u * j < end;
        const uint32_t d = (key[j] >> shift) & 255u;
        // the lanes of each digit: by shared atomics and by ballots in turn, so that neither the shared-memory
        // pipe nor the integer pipe sets the pace alone
        const bool ballots = (j & 1) != 0;
        uint32_t peers;
        if (ballots) {
            peers = match_digit(d, valid);
        } else {
            if (valid) atomicOr(&sm.mask[w][d], 1u << lane);
            __syncwarp();
            peers = sm.mask[w][d];
        }
        const uint32_t cur = sm.wcnt[w][d], before = peers & lt;
        pos[j] = cur + __popc(before);
        __syncwarp();
        if (valid && before == 0u) {  // the digit's first lane
            sm.wcnt[w][d] = cur + __popc(peers);
            if (!ballots) sm.mask[w][d] = 0u;
        }
        __syncwarp();
    }
    __syncthreads();
    // One exclusive scan of the count table in (digit, warp) order gives every (warp, digit) its
    // first position in the sub-tile: thread t owns digit t / 2 and half of the warps; the thread
    // sums go through a warp scan and the warp totals.
    constexpr int HW = CS_WARPS / 2;
    const uint32_t d = tid >> 1, w0 = (tid & 1u) * HW;
    uint32_t c8[HW], sum = 0;
#pragma unroll
    for (int k = 0; k < HW; ++k) {
        c8[k] = sm.wcnt[w0 + k][d];
        sum += c8[k];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31u) sm.scan[w] = x;
    __syncthreads();
    const uint32_t wpre = __reduce_add_sync(FULL_MASK, lane < w ? sm.scan[lane] : 0u);
    const uint32_t excl = wpre + x - sum;
    uint32_t run = excl;
#pragma unroll
    for (int k = 0; k < HW; ++k) {
        sm.wcnt[w0 + k][d] = run;
        run += c8[k];
    }
    first = __shfl_xor_sync(FULL_MASK, excl, 1);  // the digit's other half
    count = run - first;
}

// Puts the ranked keys and values into digit order in sm.buf.
template <int R, bool FULL>
__device__ __forceinline__ void place_subtile(CoopSmem& sm, const uint32_t (&key)[R], const uint32_t (&val)[R],
                                              const uint32_t (&pos)[R], uint32_t wb, uint32_t end, int shift) {
    const uint32_t w = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < R; ++j)
        if (FULL || wb + 32u * j < end)
            sm.buf[pos[j] + sm.wcnt[w][(key[j] >> shift) & 255u]] = make_uint2(key[j], val[j]);
}

// Writes a placed sub-tile of tn keys: each digit's run is consecutive in the output.
template <int R, bool FULL>
__device__ __forceinline__ void write_subtile(const CoopSmem& sm, uint32_t* kout, uint32_t* vout, uint32_t tn, uint32_t n,
                                              int shift) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const uint32_t i = threadIdx.x + CS_THREADS * j;
        if (FULL || i < tn) {
            const uint2 kv = sm.buf[i];
            const uint32_t g = sm.place[(kv.x >> shift) & 255u] + i;
            if (g < n) {  // always, unless a wait timed out
                kout[g] = kv.x;
                vout[g] = kv.y;
            }
        }
    }
}

// The exchange of the pass's counts, in two parts so that work fits between them.  First, after every thread
// of the CTA has seen its counts published in row c: the sums over this thread's share of the group's earlier
// CTAs; the group's last CTA publishes the group's sums.  `own`: this CTA's count of digit tid & 255.
__device__ __forceinline__ uint32_t sum_group(CoopSmem& sm, const CountTable& t, uint32_t c, uint32_t G, uint32_t own) {
    const uint32_t tid = threadIdx.x, d = tid & 255u, h = tid >> 8;
    uint32_t pre = 0, unused = 0;
    if (G > (uint32_t)CS_DIRECT) {
        const uint32_t g = c / CS_GROUP, g0 = g * CS_GROUP;
        t.sum(t.rows, d, g0 + h, c, c, pre, unused);
        if (c == min(g0 + CS_GROUP, G) - 1u) {
            sm.part[0][h][d] = pre;
            __syncthreads();
            if (tid < 256) t.publish(t.group(g) + d, sm.part[0][0][d] + sm.part[0][1][d] + own);
            __syncthreads();
        }
    }
    return pre;
}

// Then the sums over all groups (or all CTAs): thread d < 256 gets the global output base of the CTA's first
// key of digit d.  `pre`: sum_group's result.  Every thread of the CTA calls it.
__device__ __forceinline__ uint32_t finish_exchange(CoopSmem& sm, const CountTable& t, uint32_t c, uint32_t G, uint32_t pre) {
    const uint32_t tid = threadIdx.x, d = tid & 255u, h = tid >> 8;
    uint32_t tot = 0;
    if (G <= (uint32_t)CS_DIRECT)
        t.sum(t.rows, d, h, G, c, pre, tot);
    else
        t.sum(t.group(0), d, h, (G + CS_GROUP - 1) / CS_GROUP, c / CS_GROUP, pre, tot);
    sm.part[0][h][d] = pre;
    sm.part[1][h][d] = tot;
    __syncthreads();
    uint32_t all;
    const uint32_t bases = scan256(tid < 256 ? sm.part[1][0][d] + sm.part[1][1][d] : 0u, sm.scan, &all);
    return bases + sm.part[0][0][d] + sm.part[0][1][d];
}

// One pass of a segment of at most CS_THREADS * R keys: ranked first, so that its counts need no pass of
// their own, and staged in shared memory while the other CTAs' counts arrive.
template <int R>
__device__ __forceinline__ void short_pass(CoopSmem& sm, const CountTable& t, const uint32_t* kin, const uint32_t* vin,
                                           uint32_t* kout, uint32_t* vout, bool iota, uint32_t s_begin, uint32_t s_end,
                                           uint32_t n, int shift, uint32_t c, uint32_t G, uint32_t lt) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    uint32_t key[R], val[R], pos[R], first, count;
    const uint32_t wb = s_begin + w * (32u * R) + lane;
    load_subtile<R, false>(key, val, kin, vin, iota, wb, s_end);
    rank_subtile<R, false>(sm, key, pos, wb, s_end, shift, lt, first, count);
    if (tid & 1u) {
        t.publish(t.rows + (size_t)c * 256 + (tid >> 1), count);
        sm.count[tid >> 1] = count;
        sm.next[tid >> 1] = first;
    }
    __syncthreads();
    place_subtile<R, false>(sm, key, val, pos, wb, s_end, shift);
    const uint32_t pre = sum_group(sm, t, c, G, sm.count[tid & 255u]);
    const uint32_t base = finish_exchange(sm, t, c, G, pre);
    if (tid < 256) sm.place[tid] = base - sm.next[tid];
    __syncthreads();
    write_subtile<R, false>(sm, kout, vout, s_end - s_begin, n, shift);
}

// One pass of a segment of more than a sub-tile: counted, then ranked and written sub-tile by sub-tile.
__device__ __forceinline__ void long_pass(CoopSmem& sm, const CountTable& t, const uint32_t* kin, const uint32_t* vin,
                                          uint32_t* kout, uint32_t* vout, bool iota, uint32_t s_begin, uint32_t s_end,
                                          uint32_t n, int shift, uint32_t c, uint32_t G, uint32_t lt) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    // count: per-warp histograms (shared atomics)
#pragma unroll
    for (int k = 0; k < 8; ++k) sm.wcnt[w][lane + 32 * k] = 0u;
    __syncwarp();
    {
        // 16-byte loads (segments start 256-aligned), four in flight per thread; the loads bypass
        // L1 because the previous pass's output was written by other CTAs of this launch
        const uint32_t v_begin = s_begin >> 2, v_end = s_end >> 2;
        const uint4* kin4 = reinterpret_cast<const uint4*>(kin);
        for (uint32_t v0 = v_begin; v0 < v_end; v0 += 4u * CS_THREADS) {
            uint4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t vi = v0 + (uint32_t)u * CS_THREADS + tid;
                q[u] = vi < v_end ? __ldcg(kin4 + vi) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (v0 + (uint32_t)u * CS_THREADS + tid < v_end) {
                    atomicAdd(&sm.wcnt[w][(q[u].x >> shift) & 255u], 1u);
                    atomicAdd(&sm.wcnt[w][(q[u].y >> shift) & 255u], 1u);
                    atomicAdd(&sm.wcnt[w][(q[u].z >> shift) & 255u], 1u);
                    atomicAdd(&sm.wcnt[w][(q[u].w >> shift) & 255u], 1u);
                }
            }
        }
        // tail (fewer than 4 keys past the last 16-byte group)
        for (uint32_t e = (v_end << 2) + tid; e < s_end; e += CS_THREADS)
            atomicAdd(&sm.wcnt[w][(__ldcg(kin + e) >> shift) & 255u], 1u);
    }
    __syncthreads();
    {
        const uint32_t d = tid & 255u, h = tid >> 8;
        uint32_t acc = 0;
#pragma unroll
        for (int k = 0; k < CS_WARPS / 2; ++k) acc += sm.wcnt[CS_WARPS / 2 * h + k][d];
        sm.part[0][h][d] = acc;
    }
    __syncthreads();
    const uint32_t own = sm.part[0][0][tid & 255u] + sm.part[0][1][tid & 255u];
    if (tid < 256) t.publish(t.rows + (size_t)c * 256 + tid, own);
    uint32_t key[CS_KPT], val[CS_KPT], pos[CS_KPT], first, count;
    const uint32_t wo = w * (32u * CS_KPT) + lane;
    uint32_t tb = s_begin;
    if (s_begin + CS_TILE <= s_end) {
        // The first sub-tile is ranked and placed while the other CTAs' counts arrive.
        load_subtile<CS_KPT, true>(key, val, kin, vin, iota, tb + wo, s_end);
        rank_subtile<CS_KPT, true>(sm, key, pos, tb + wo, s_end, shift, lt, first, count);
        if (tid & 1u) {
            sm.place[tid >> 1] = first;
            sm.count[tid >> 1] = count;
        }
        __syncthreads();
        const uint32_t pre = sum_group(sm, t, c, G, own);
        place_subtile<CS_KPT, true>(sm, key, val, pos, tb + wo, s_end, shift);
        tb += CS_TILE;
        if (tb + CS_TILE <= s_end) load_subtile<CS_KPT, true>(key, val, kin, vin, iota, tb + wo, s_end);
        const uint32_t base = finish_exchange(sm, t, c, G, pre);
        if (tid < 256) {
            sm.place[tid] = base - sm.place[tid];
            sm.next[tid] = base + sm.count[tid];
        }
        __syncthreads();
        write_subtile<CS_KPT, true>(sm, kout, vout, CS_TILE, n, shift);
        // The other full sub-tiles, each one's keys loaded while the one before is written.  Four CTA barriers:
        // ranked, scanned, counts placed, keys placed; the writes of one sub-tile need none against the next
        // one's ranking, whose first barrier comes before anything they read is changed.
        while (tb + CS_TILE <= s_end) {
            rank_subtile<CS_KPT, true>(sm, key, pos, tb + wo, s_end, shift, lt, first, count);
            if (tid & 1u) {
                const uint32_t at = sm.next[tid >> 1];
                sm.place[tid >> 1] = at - first;
                sm.next[tid >> 1] = at + count;
            }
            __syncthreads();
            place_subtile<CS_KPT, true>(sm, key, val, pos, tb + wo, s_end, shift);
            tb += CS_TILE;
            if (tb + CS_TILE <= s_end) load_subtile<CS_KPT, true>(key, val, kin, vin, iota, tb + wo, s_end);
            __syncthreads();
            write_subtile<CS_KPT, true>(sm, kout, vout, CS_TILE, n, shift);
        }
    } else {  // the input's end, less than a sub-tile
        __syncthreads();  // every thread has its count from part
        const uint32_t pre = sum_group(sm, t, c, G, own);
        const uint32_t base = finish_exchange(sm, t, c, G, pre);
        if (tid < 256) sm.next[tid] = base;
    }
    if (tb < s_end) {  // the rest
        load_subtile<CS_KPT, false>(key, val, kin, vin, iota, tb + wo, s_end);
        rank_subtile<CS_KPT, false>(sm, key, pos, tb + wo, s_end, shift, lt, first, count);
        if (tid & 1u) sm.place[tid >> 1] = sm.next[tid >> 1] - first;
        __syncthreads();
        place_subtile<CS_KPT, false>(sm, key, val, pos, tb + wo, s_end, shift);
        __syncthreads();
        write_subtile<CS_KPT, false>(sm, kout, vout, s_end - tb, n, shift);
    }
}

// `passes` passes starting at bit `shift0` (the buffers: SortBuffers).  For at most one sub-tile of keys only the
// last pass's buffers are written.
__global__ void __launch_bounds__(CS_THREADS, 2)
    k_sort_coop(SortBuffers io, const uint32_t* n_ptr, uint32_t n_cap, int passes, int shift0, uint64_t* table,
                const uint32_t* epoch_word, uint32_t* bar, uint32_t spin_limit, uint32_t* err, bool start_dependent) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CoopSmem& sm = *reinterpret_cast<CoopSmem*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    const uint32_t c = blockIdx.x;
    frame_step(n_ptr, epoch_word);
    const uint32_t n = min(*n_ptr, n_cap);
    if (start_dependent && n <= CS_START_MAX) start_next();
    // Contiguous segments, 256-aligned: up to one sub-tile of keys is one CTA's work, more are spread over
    // the grid in segments of at least CS_MIN_SEG.  The live count is read on the device (a captured graph
    // replays with any count up to n_cap), so the grid is sized for n_cap; CTAs past the last segment
    // leave at once, and only the G CTAs that work wait for one another.
    uint32_t seg = (n + gridDim.x - 1) / gridDim.x;
    seg = n <= (uint32_t)CS_TILE ? (uint32_t)CS_TILE : max((seg + 255u) & ~255u, (uint32_t)CS_MIN_SEG);
    const uint32_t G = (n + seg - 1) / seg;
    if (c >= G) return;
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int k = 0; k < 8; ++k) sm.mask[w][lane + 32 * k] = 0u;
    __syncwarp();
    if (G == 1u) {
        // n <= CS_TILE: one sub-tile.  Every pass ranks and stages it in shared memory (no count
        // table, no grid barriers); the keys are read once and written once.
        uint32_t key[CS_KPT], val[CS_KPT], pos[CS_KPT], first, count;
        const uint32_t wb = w * (32u * CS_KPT) + lane;
        load_subtile<CS_KPT, false>(key, val, io.keys_in, io.vals_in, io.vals_in == nullptr, wb, n);
        for (int p = 0; p < passes; ++p) {
            rank_subtile<CS_KPT, false>(sm, key, pos, wb, n, shift0 + 8 * p, lt, first, count);
            __syncthreads();
            place_subtile<CS_KPT, false>(sm, key, val, pos, wb, n, shift0 + 8 * p);
            __syncthreads();
            if (p + 1 < passes) {
#pragma unroll
                for (int j = 0; j < CS_KPT; ++j) {
                    const uint32_t e = wb + 32u * j;
                    if (e < n) {
                        const uint2 kv = sm.buf[e];
                        key[j] = kv.x;
                        val[j] = kv.y;
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < CS_KPT; ++j) {
            const uint32_t i = tid + CS_THREADS * j;
            if (i < n) {
                const uint2 kv = sm.buf[i];
                io.keys_out[i] = kv.x;
                io.vals_out[i] = kv.y;
            }
        }
        return;
    }
    CountTable t{table, *epoch_word, 0u, spin_limit, err};
    const uint32_t s_begin = c * seg, s_end = min(s_begin + seg, n);
    for (int p = 0; p < passes; ++p) {
        const bool last = p + 1 == passes;
        const uint32_t* kin = p == 0 ? io.keys_in : (p & 1) ? io.keys[1] : io.keys[0];
        const uint32_t* vin = p == 0 ? io.vals_in : (p & 1) ? io.vals[1] : io.vals[0];
        uint32_t* kout = last ? io.keys_out : (p & 1) ? io.keys[0] : io.keys[1];
        uint32_t* vout = last ? io.vals_out : (p & 1) ? io.vals[0] : io.vals[1];
        const bool iota = vin == nullptr;
        t.pass = (uint32_t)p;
        if (seg <= 4u * CS_THREADS)
            short_pass<4>(sm, t, kin, vin, kout, vout, iota, s_begin, s_end, n, shift0 + 8 * p, c, G, lt);
        else if (seg <= (uint32_t)CS_TILE)
            short_pass<CS_KPT>(sm, t, kin, vin, kout, vout, iota, s_begin, s_end, n, shift0 + 8 * p, c, G, lt);
        else
            long_pass(sm, t, kin, vin, kout, vout, iota, s_begin, s_end, n, shift0 + 8 * p, c, G, lt);
        if (!last) grid_barrier(bar, (uint32_t)(p + 1) * G, spin_limit, err);
    }
}

// CTAs of the grid on the current device, asked of each device once: they are what the device holds at a time, and the
// kernel's shared memory (above the 48 KB that every kernel may have) is allowed device by device.
int sort_coop_grid() {
    static std::atomic<int> cache[64];
    int dev = 0;
    const bool known = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64;
    int grid = known ? cache[dev].load(std::memory_order_relaxed) : 0;
    if (grid == 0) {
        int sms = 0, per = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(k_sort_coop, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CoopSmem));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sort_coop, CS_THREADS, sizeof(CoopSmem));
        grid = sms * (per > 0 ? per : 1);
        if (grid > CS_MAX_GRID) grid = CS_MAX_GRID;
        if (known) cache[dev].store(grid, std::memory_order_relaxed);
    }
    return grid;
}

// CTAs launched for at most n_cap keys.
static uint32_t coop_grid_for(uint64_t n_cap) {
    const uint64_t grid = (uint64_t)sort_coop_grid(), want = (n_cap + CS_MIN_SEG - 1) / CS_MIN_SEG;
    return (uint32_t)(want < 1 ? 1 : (want < grid ? want : grid));
}

size_t sort_coop_table_words(uint64_t n_cap) {
    const size_t grid = coop_grid_for(n_cap);
    return (grid + (grid + CS_GROUP - 1) / CS_GROUP) * 256;
}

cudaError_t launch_sort_coop(const SortBuffers& io, const uint32_t* n_ptr, uint32_t n_cap, int passes, int shift0,
                             uint64_t* table, const uint32_t* epoch_word, uint32_t* bar, uint32_t spin_limit,
                             uint32_t* err, bool start_dependent, cudaStream_t st) {
    if (n_cap == 0 || passes == 0) return cudaSuccess;
    void* args[] = {(void*)&io, (void*)&n_ptr, &n_cap, &passes, &shift0, &table, (void*)&epoch_word, &bar, &spin_limit, &err,
                    &start_dependent};
    return cudaLaunchCooperativeKernel((const void*)k_sort_coop, dim3(coop_grid_for(n_cap)), dim3(CS_THREADS), args,
                                       sizeof(CoopSmem), st);
}

}  // namespace spl
