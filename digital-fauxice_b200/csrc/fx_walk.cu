// fx_walk.cu -- the serial RNG walk, parallelised by speculation.
//
// The chain of RNG-dependent channels (see fx_writer.cu) is a function of
// one integer: E_i, the number of extra draws before channel i.  The state
// at channel i's first draw is T_i = G^(pos_i + 1 + E_i)(T0) (G = one LCG step
// in T space), the channel draws an extra time iff T_i misses its copy
// intervals, and E_{i+1} = E_i + extra_i.  The walk carries S = G^E(T0):
// T_i is an affine map of S that depends on the channel alone (AmbEntry), and
// S takes one LCG step where the channel draws an extra time.  So a segment
// of channels maps an entry count E_in to an exit count E_out, and:
//   * two candidates E < E' keep their order and merge for good once equal
//     (E'_k - E_k moves by -1, 0 or +1 per channel), so merges only ever
//     happen between neighbours in E order;
//   * candidates merge quickly (the gap is a lazy random walk absorbed at 0).
//
// A wave of segments is one launch of k_wave.  Its blocks each walk one
// segment for a window of candidate E_in values around the predicted value
// (expected extras from the exact state-space measure of every copy set,
// summed per chunk by k_coef), merging candidates as they meet and
// compacting the survivors, and write a compact survivor list.  The block
// that finishes last of a group of kGroup segments composes the group's
// lists (every survivor of the first list followed through the others), and
// the block that completes the last group chains the exact E through the
// groups and looks up every segment's exact entry count.  When E falls
// outside a window the wave ends there and the next one starts at that
// segment, its windows centred on the exact count again (the launches hold a
// few waves in reserve; without one left the segment is walked exactly), so
// correctness never depends on the prediction.  No block waits for another.
//
// Every 512 channels a block also keeps its survivors (entry count and
// state): from them k_rewalk starts one lane per 512 channels, in parallel,
// at the exact state and writes the extra draws of every channel.  With one
// segment covering the whole chain, k_rewalk alone is the plain serial walk.
#include <algorithm>
#include <cmath>

#include "fx_internal.cuh"

namespace fx {

constexpr int kWinThreads = 256;
constexpr int kWinWarps = kWinThreads / 32;
constexpr int kWinBlocksPerSM = 4;                  // segments resident per SM
constexpr int kWinSlots = 8;                        // candidates per thread
constexpr int kWinBatch = 32 * kWinSlots;           // candidates a warp walks at once
// Widest window.  A wave's reach is at most per_wave x kWalkAvgMax chunks,
// 2.7 M channels, and a channel's variance at most 1/4, so 4.5 standard
// deviations either side (at most 7425 + 33 candidates) always fit.
constexpr int kWinMax = 8192;
// The first kWinFirst channels (the first chunk, where too many are left then)
// are walked by every warp on its own share of the window, in batches of
// kWinBatch; about a quarter of a batch is left then and waits in the warp's
// region of the list.
constexpr uint32_t kWinFirst = 64;
constexpr int kWinRegion = 2 * kWinBatch;
constexpr int kWinChunk = kWalkChunk;               // channels staged per chunk
constexpr int kWinRing = 3;                         // staged chunks in flight
constexpr uint32_t kPiece = 512;                    // channels per kept survivor list
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kSerialBelow = 1024;             // short chains: one serial walk
// The window half-width is kDefaultWindowSigmas (4.5) standard deviations of
// the predicted entry count, plus 16.  A count outside its window never
// changes a result: it ends the wave, or costs one exact serial walk of that
// segment (200 us for the longest).  Heavily damaged frames drift out of 4.5
// sigma now and then and stay out for the rest of the wave: 239 segments and
// 51.6 ms on one frame with exact walks alone, 4.6 ms with restarts.
// fx_set_walk_window narrows the windows, so tests can force misses.
constexpr uint32_t kSpareWaves = 2;  // launches beyond the waves a chain needs

struct SegWindow {
    uint32_t lo, hi;  // candidate E_in range, inclusive
};

// Powers of the LCG step: g_pow[j][d] = G^(d * 64^j); states repeat after 2^24
// steps, so the four low base-64 digits of n give G^n on states.
__device__ Affine g_pow[4][64];

__device__ __forceinline__ uint32_t jump_t(uint32_t t0, uint32_t n) {
    uint32_t t = t0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const Affine f = g_pow[j][(n >> (6 * j)) & 63u];
        t = f.a * t + f.c;
    }
    return t;
}

// Steps n with G^n(from) = to (T space, 24-bit state in the high bits), by
// matching one bit per round: G^(2^j) leaves the bits below j unchanged and
// flips bit j (full-period LCG: multiplier 1 mod 4, odd increment).
__device__ __forceinline__ uint32_t lcg_distance_t(uint32_t from_t, uint32_t to_t) {
    uint32_t cur = from_t >> 8, target = to_t >> 8, a = 125u, c = 1u, d = 0u;
#pragma unroll
    for (int j = 0; j < 24; ++j) {
        const uint32_t bit = 1u << j;
        if ((cur ^ target) & bit) {
            cur = (a * cur + c) & 0xFFFFFFu;
            d |= bit;
        }
        c = (a + 1u) * c;
        a = a * a;
    }
    return d;
}

// One channel: S takes one LCG step unless the channel copies.  e = (a, b, w,
// two).  Inline PTX keeps the step at three instructions (multiply-add,
// compare, predicated multiply-add).
__device__ __forceinline__ void step_one(const uint4 &e, uint32_t &S) {
    asm("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\t"
        "mad.lo.u32 t, %1, %0, %2;\n\t"
        "setp.gt.u32 p, t, %3;\n\t"
        "@p mad.lo.u32 %0, %0, 125, 256;\n\t}"
        : "+r"(S)
        : "r"(e.x), "r"(e.y), "r"(e.z));
}

// Whether the channel copies at state S; `second` is read only where the
// entry has a second interval.
__device__ __forceinline__ bool copies(const uint4 &e, const SecondInterval *second, uint32_t S) {
    const uint32_t t = e.x * S + e.y;
    bool c = t <= e.z;
    if (e.w) {
        const SecondInterval q = *second;
        c |= (t + q.d) <= q.w;
    }
    return c;
}

__device__ __forceinline__ void step_two(const uint4 &e, const SecondInterval *second,
                                         uint32_t &S) {
    if (!copies(e, second, S)) S = 125u * S + 256u;
}

// ---------------------------------------------------------------------------
// Window walk
// ---------------------------------------------------------------------------

constexpr int kListMax = 384;  // survivors kept in a segment's list (wave ends have 210 to
                               // 260 whatever the segment length: window and survivor
                               // density both go with its root)
constexpr int kGroup = 20;     // segments composed by one block
constexpr uint32_t kTooMany = 0xFFFFu;  // list count: more than kListMax survivors

// Compact result of one window [lo, hi]: survivors in E_in order as 16-bit
// offsets (E_in - lo, E_out - lo).
struct __align__(16) SegList {
    uint32_t count;
    SegWindow win;
    uint32_t pad;
    uint16_t ein[kListMax];
    uint16_t eout[kListMax];
};
static_assert(sizeof(SegList) % 16 == 0, "lists are copied in 16-byte vectors");

// The survivors of a segment at a piece boundary: E_in - lo and state, in
// pools shared by all segments.  Indexed by the boundary's chunk.
struct KeptHead {
    uint32_t offset, count;  // count 0: not kept (the pool was full)
};
__host__ __device__ inline int64_t kept_pool(int64_t capacity) {
    return capacity - capacity / 4 + 65536;  // measured use: 0.4 per channel
}

struct WindowSmem {
    AmbEntry ring[kWinRing][kWinChunk];
    uint32_t t[kWinWarps * kWinRegion];    // survivors in E_in order: state,
    uint16_t ein[kWinWarps * kWinRegion];  // and E_in less the window's lowest
    uint32_t wfirst[kWinWarps], wlast[kWinWarps], wcount[kWinWarps];
    double pred[kWinWarps][2];
    uint32_t kept_at;
};
static_assert(kWinMax <= 65536, "candidates are 16-bit offsets in their window");

// One warp steps its candidates over LEN staged channels, starting at staged
// channel r (`second` is the chunk's).  The entries do not depend on the
// candidates, so all LEN are loaded first.  Dead candidates (merged into a
// neighbour) keep stepping: skipping them would put a divergent branch on
// every step, and their state stays that of the neighbour they merged into.
template <int SLOTS, int LEN, bool TWO>
__device__ __forceinline__ void walk_group(const uint4 *r4, const SecondInterval *second,
                                           uint32_t r, uint32_t (&rS)[kWinSlots],
                                           uint32_t live_mask, uint32_t &steps) {
    uint4 e[LEN];
#pragma unroll
    for (int k = 0; k < LEN; ++k) e[k] = r4[r + k];
    steps += (uint32_t)__popc(live_mask & ((1u << SLOTS) - 1u)) * LEN;
#pragma unroll
    for (int k = 0; k < LEN; ++k) {
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            if (TWO) step_two(e[k], second + r + k, rS[s]);
            else step_one(e[k], rS[s]);
        }
    }
}

// Walk channels [r, stop) of the staged ring for one warp.  TWO: some entry
// of the staged chunk has two copy intervals.
template <int SLOTS, bool TWO>
__device__ __forceinline__ void walk_span(const uint4 *r4, const SecondInterval *second,
                                          uint32_t r, uint32_t stop, uint32_t (&rS)[kWinSlots],
                                          uint32_t live_mask, uint32_t &steps) {
    // many slots give their own parallelism: stage fewer channels at once
    constexpr int kLen = TWO ? 1 : (SLOTS <= 2 ? 8 : (SLOTS <= 4 ? 4 : 2));
    for (; r + kLen <= stop; r += kLen)
        walk_group<SLOTS, kLen, TWO>(r4, second, r, rS, live_mask, steps);
    for (; r < stop; ++r) walk_group<SLOTS, 1, TWO>(r4, second, r, rS, live_mask, steps);
}

// Slots per lane for `live` candidates (at most kWinThreads * kWinSlots).  Warp w holds
// list positions [w * slots * 32, (w + 1) * slots * 32).  More than 32
// candidates go at least two per lane, into the fewest warps: two slots in
// four warps measured 1.48x the candidate-step rate of one slot in eight, and
// warps with no candidate left do not step.
__device__ __forceinline__ int window_slots(uint32_t live) {
    if (live <= 32u) return 1;
    const uint32_t s = (live + kWinThreads - 1u) / kWinThreads;
    return s < 2u ? 2 : (int)s;
}

// Pointers of one pass's walk scratch.
struct WalkBuffers {
    const AmbEntry *entries;
    const SecondInterval *second;
    const uint8_t *chunk_two;
    const ChunkStat *chunk_stat;
    WalkState *st;
    uint2 *wave;           // per wave: first chunk, exact E there (one more: its end)
    SegWindow *windows;    // per segment of every wave
    uint32_t *e_in;        // per segment: exact entry count
    SegList *lists;        // per segment of a wave
    uint32_t *path;        // per segment of a wave: kListMax exit counts, one per survivor
                           // of its group's first list (kNone: left a window)
    uint32_t *group_done;  // per group of a wave: segments finished
    KeptHead *kept;        // per chunk
    uint32_t *kept_state;
    uint16_t *kept_ein;
    uint32_t kept_size;
};

// Segments that hold channels of a wave that starts at chunk c0 (the last
// wave may be short).
__device__ __forceinline__ uint32_t wave_segments(const WalkPlan &plan, uint32_t c0) {
    if (c0 >= plan.chunks) return 0u;
    const uint32_t left = plan.chunks - c0;
    if (left >= plan.wave_chunks) return plan.segs;
    uint32_t l = 0, h = plan.segs;  // start(l) < left <= start(h)
    while (h - l > 1u) {
        const uint32_t mid = (l + h) / 2u;
        if (plan.start(mid) < left) l = mid;
        else h = mid;
    }
    return h;
}

// One segment's window walk: segment x of wave w, channels [i0, i1).
__device__ __forceinline__ void window_block(const WalkBuffers &B, WindowSmem &S, uint32_t c_wave,
                                             uint32_t e0, uint32_t i0, uint32_t i1, uint32_t j, uint32_t x,
                                             uint32_t t0, double sigmas) {
    const uint32_t tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const uint32_t len = i1 - i0;

    auto stage = [&](uint32_t first, int b) {
        if (first < i1) {
            const uint32_t avail = min((uint32_t)kWinChunk, i1 - first);
            const uint4 *src = reinterpret_cast<const uint4 *>(B.entries + first);
            uint4 *dst = reinterpret_cast<uint4 *>(S.ring[b]);
            for (uint32_t v = tid; v < avail; v += kWinThreads) {
                const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst + v);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(src + v));
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    // Three staged chunks: chunk c+2 is fetched into the buffer of chunk c-1
    // right after the barrier that ends every warp's work on chunk c-1.
    stage(i0, 0);
    stage(i0 + kWinChunk, 1);

    // window of candidate entry counts around the prediction: the chunks of
    // the wave before this segment, each channel drawing an extra with
    // probability p = 1 - copying states / 2^24.  The prediction only
    // centres the window: any summation order.
    {
        double mu = 0.0, var = 0.0;
        const uint32_t c1 = i0 / kWalkChunk;
#pragma unroll 4
        for (uint32_t c = c_wave + tid; c < c1; c += kWinThreads) {
            const uint2 q = __ldg(reinterpret_cast<const uint2 *>(B.chunk_stat) + c);
            mu += (double)kWalkChunk - (double)q.x * 0x1p-23;
            var += (double)q.y * 0x1p-25;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mu += __shfl_down_sync(0xFFFFFFFFu, mu, o);
            var += __shfl_down_sync(0xFFFFFFFFu, var, o);
        }
        if (lane == 0) {
            S.pred[warp][0] = mu;
            S.pred[warp][1] = var;
        }
    }
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();  // the prediction and the first chunk
    double center = 0.0, var = 0.0;
#pragma unroll
    for (int w = 0; w < kWinWarps; ++w) {
        center += S.pred[w][0];
        var += S.pred[w][1];
    }
    double half = sigmas * sqrt(var) + 16.0;
    const uint32_t before = i0 - c_wave * kWalkChunk;  // channels since the wave start

    // A warp's candidates, in order k = slot * 32 + lane of its share.  Slots
    // hold the state S; the entry count of position k is ein[k] of the share.
    uint32_t rS[kWinSlots];
    uint32_t live_mask = 0;
    uint32_t steps = 0;
    uint32_t *const wt = S.t + warp * kWinRegion;

    // Merges the warp's candidates: equal states mean equal counts (distinct
    // counts of one window are far closer than the LCG's 2^24 period), a
    // merged candidate keeps the state of its left neighbour, and neighbours
    // in list order are the lane to the left or the last lane of the slot
    // before.
    auto warp_dedupe = [&](int slots) {
        uint32_t last = 0;
#pragma unroll
        for (int s = 0; s < kWinSlots; ++s) {
            if (s < slots) {
                uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, rS[s], 1);
                if (lane == 0) prev = last;
                if ((s || lane) && prev == rS[s]) live_mask &= ~(1u << s);
                last = __shfl_sync(0xFFFFFFFFu, rS[s], 31);
            }
        }
    };
    // The warp's live candidates (entry counts from list position e_at on)
    // into list positions at.., in order; returns how many.
    auto warp_store = [&](int slots, uint32_t e_at, uint32_t at) -> uint32_t {
        uint32_t ein[kWinSlots];
#pragma unroll
        for (int s = 0; s < kWinSlots; ++s)
            if (s < slots && (live_mask & (1u << s))) ein[s] = S.ein[e_at + s * 32 + lane];
        __syncwarp();
        uint32_t run = 0;
#pragma unroll
        for (int s = 0; s < kWinSlots; ++s) {
            if (s < slots) {
                const bool alive = live_mask & (1u << s);
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, alive);
                if (alive) {
                    const uint32_t k = at + run + __popc(bal & ((1u << lane) - 1u));
                    S.ein[k] = (uint16_t)ein[s];
                    S.t[k] = rS[s];
                }
                run += __popc(bal);
            }
        }
        __syncwarp();
        return run;
    };
    // `n` list entries from position `at` into the warp's registers
    auto warp_load = [&](uint32_t at, uint32_t n, int slots) {
        live_mask = 0;
#pragma unroll
        for (int s = 0; s < kWinSlots; ++s) {
            if (s < slots) {
                const uint32_t k = (uint32_t)(s * 32 + lane);
                if (k < n) {
                    live_mask |= 1u << s;
                    rS[s] = S.t[at + k];
                }
            }
        }
    };
    // Channels [r, stop) of a staged chunk.
    auto walk = [&](const uint4 *r4, const SecondInterval *sec, bool two, int slots, uint32_t r,
                    uint32_t stop) {
        if (slots == 0) return;
        if (two) {
            // rare: one code path for every slot count (idle slots step too)
            walk_span<kWinSlots, true>(r4, sec, r, stop, rS, live_mask, steps);
            return;
        }
        switch (slots) {
#define FX_WALK_CASE(K)                                                    \
    case K:                                                                \
        walk_span<K, false>(r4, sec, r, stop, rS, live_mask, steps);       \
        break;
            FX_WALK_CASE(1) FX_WALK_CASE(2) FX_WALK_CASE(3) FX_WALK_CASE(4)
            FX_WALK_CASE(5) FX_WALK_CASE(6) FX_WALK_CASE(7)
        default:
            walk_span<kWinSlots, false>(r4, sec, r, stop, rS, live_mask, steps);
            break;
#undef FX_WALK_CASE
        }
    };
    // Slots a warp needs for n candidates.
    auto slots_for = [](uint32_t n) { return (int)((n + 31u) / 32u); };

    // ---- the first channels, every warp on its share of the window -----------
    uint32_t first = min(kWinFirst, len);
    const uint4 *ring0 = reinterpret_cast<const uint4 *>(S.ring[0]);
    const bool two0 = B.chunk_two[i0 / kWalkChunk] != 0;
    uint32_t wlo, count;
    uint32_t mine;  // survivors in the warp's region
    for (;;) {
        int64_t lo = (int64_t)floor(center - half), hi = (int64_t)ceil(center + half);
        lo = lo < 0 ? 0 : lo;
        hi = hi > (int64_t)before ? (int64_t)before : hi;
        if (lo > (int64_t)before) lo = before;
        if (hi < lo) hi = lo;
        if (hi - lo + 1 > kWinMax) {
            lo = (int64_t)center - kWinMax / 2;
            lo = lo < 0 ? 0 : lo;
            hi = lo + kWinMax - 1;
            if (hi > (int64_t)before) {
                hi = before;
                lo = hi - kWinMax + 1;
            }
        }
        wlo = e0 + (uint32_t)lo;
        count = (uint32_t)(hi - lo + 1);
        const uint32_t share = (count + kWinWarps - 1) / kWinWarps;
        const uint32_t k_end = min(count, (warp + 1) * share);
        mine = 0;
        bool full = false;
        for (uint32_t b0 = warp * share; b0 < k_end; b0 += kWinBatch) {
            uint32_t n = min((uint32_t)kWinBatch, k_end - b0);
            if (mine > (uint32_t)(kWinRegion - kWinBatch)) {  // no room for another batch
                full = true;
                break;
            }
            const uint32_t at = warp * kWinRegion + mine;
            uint32_t t = jump_t(t0, wlo + b0 + lane);
            const Affine stride = g_pow[0][32];
            live_mask = 0;
            int slots = slots_for(n);
#pragma unroll
            for (int s = 0; s < kWinSlots; ++s) {
                rS[s] = t;
                const uint32_t k = (uint32_t)(s * 32 + lane);
                if (k < n) {
                    live_mask |= 1u << s;
                    S.ein[at + k] = (uint16_t)(b0 + k);
                }
                t = stride.a * t + stride.c;
            }
            __syncwarp();
            uint32_t r = 0;
            for (uint32_t stop = 8; r < first; stop *= 2) {
                stop = min(stop, first);
                walk(ring0, B.second + i0, two0, slots, r, stop);
                r = stop;
                warp_dedupe(slots);
                // against the batch before (whose survivors are at `first` too)
                if (r == first && mine && lane == 0 && wt[mine - 1] == rS[0]) live_mask &= ~1u;
                n = warp_store(slots, at, at);
                if (r < first) {
                    slots = slots_for(n);
                    warp_load(at, n, slots);
                }
            }
            mine += n;
        }
        full |= mine > (uint32_t)kWinBatch;
        if (!__syncthreads_or(full)) break;
        // Too many are left (a stretch of channels that hardly merges): more
        // channels first, then half the window, at the risk of a miss.
        if (first < min((uint32_t)kWinChunk, len)) first = min((uint32_t)kWinChunk, len);
        else half *= 0.5;
    }

    // ---- the rest of the segment ---------------------------------------------
    int slots = slots_for(mine);  // of this warp
    uint32_t at = warp * kWinRegion;  // list position of the warp's candidates
    warp_load(at, mine, slots);
    uint32_t live = count;  // of the block, at the last block-wide compaction
    bool packed = false;    // the settled phase ran two candidates per lane
    bool settled = false;

    // Block-wide merge and compaction: the warps' survivors (already in
    // registers) into one list from position 0, then dealt out again.  A
    // warp's first survivor may repeat the last one of the warps before.
    auto block_compact = [&]() {
        warp_dedupe(slots);
        uint32_t cnt = 0, firstv = kNone, lastv = kNone;
#pragma unroll
        for (int s = 0; s < kWinSlots; ++s) {
            if (s < slots) {
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, live_mask & (1u << s));
                if (bal) {
                    const uint32_t f = __shfl_sync(0xFFFFFFFFu, rS[s], __ffs(bal) - 1);
                    if (cnt == 0) firstv = f;
                    lastv = __shfl_sync(0xFFFFFFFFu, rS[s], 31 - __clz(bal));
                }
                cnt += __popc(bal);
            }
        }
        if (lane == 0) {
            S.wfirst[warp] = firstv;
            S.wlast[warp] = lastv;
            S.wcount[warp] = cnt;
        }
        uint32_t ein[kWinSlots];
#pragma unroll
        for (int s = 0; s < kWinSlots; ++s)
            if (s < slots && (live_mask & (1u << s))) ein[s] = S.ein[at + s * 32 + lane];
        __syncthreads();
        uint32_t base = 0, total = 0, prev = kNone;
        bool drop = false;
#pragma unroll
        for (int w = 0; w < kWinWarps; ++w) {
            const uint32_t n = S.wcount[w];
            const bool d = n && S.wfirst[w] == prev;
            if (w == warp) {
                base = total;
                drop = d;
            }
            total += n - (d ? 1u : 0u);
            if (n) prev = S.wlast[w];
        }
        uint32_t run = 0;
#pragma unroll
        for (int s = 0; s < kWinSlots; ++s) {
            if (s < slots) {
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, live_mask & (1u << s));
                if (live_mask & (1u << s)) {
                    const uint32_t rank = run + __popc(bal & ((1u << lane) - 1u));
                    if (!(drop && rank == 0)) {
                        const uint32_t k = base + rank - (drop ? 1u : 0u);
                        S.ein[k] = (uint16_t)ein[s];
                        S.t[k] = rS[s];
                    }
                }
                run += __popc(bal);
            }
        }
        __syncthreads();
        live = total;
        settled = live <= (uint32_t)kWinThreads;
        const int per = window_slots(live);
        at = (uint32_t)(warp * per * 32);
        mine = live > at ? min(live - at, (uint32_t)per * 32u) : 0u;
        slots = slots_for(mine);
        warp_load(at, mine, slots);
        packed |= settled && per == 2;
    };
    block_compact();
    if (tid == 0 && len > kPiece) S.kept_at = atomicAdd(&B.st->kept_next, live);

    uint32_t next_compact = first > kWinFirst ? kPiece : 2 * kWinFirst;  // then 256, 512,
                                                                         // every kPiece channels
    int b = 0;
    for (uint32_t c0 = i0; c0 < i1; c0 += kWinChunk) {
        const uint32_t c1 = min(i1, c0 + (uint32_t)kWinChunk);
        if (c0 > i0) {
            asm volatile("cp.async.wait_group 1;\n" ::);
            __syncthreads();
        }
        stage(c0 + 2 * kWinChunk, (b + 2) % kWinRing);
        const uint4 *r4 = reinterpret_cast<const uint4 *>(S.ring[b]);
        uint32_t r = c0 == i0 ? first : 0u;
        const uint32_t clen = c1 - c0;
        const bool two = B.chunk_two[c0 / kWinChunk] != 0;  // block-uniform
        while (r < clen) {
            const uint32_t stop = min(clen, r + (next_compact - ((c0 - i0) + r)));
            walk(r4, B.second + c0, two, slots, r, stop);
            r = stop;
            const uint32_t done = (c0 - i0) + r;
            if (done == len || done % kPiece == 0) {
                block_compact();
                if (done < len) {  // keep the survivors here
                    const uint32_t off = S.kept_at;
                    const bool room = off + live <= B.kept_size && off + live >= off;
                    if (room) {
                        for (uint32_t k = tid; k < live; k += kWinThreads) {
                            B.kept_state[off + k] = S.t[k];
                            B.kept_ein[off + k] = S.ein[k];
                        }
                    }
                    if (tid == 0) B.kept[(i0 + done) / kWalkChunk] = KeptHead{off, room ? live : 0u};
                    __syncthreads();
                    // the next list's place: survivors never grow in number
                    if (tid == 0 && len - done > kPiece)
                        S.kept_at = atomicAdd(&B.st->kept_next, live);
                }
            } else if (done == next_compact && !settled) {  // inside the warps only
                warp_dedupe(slots);
                mine = warp_store(slots, at, at);
                slots = slots_for(mine);
                warp_load(at, mine, slots);
            }
            if (done == next_compact) next_compact = min(2 * next_compact, done + kPiece);
        }
        b = (b + 1) % kWinRing;
    }
    asm volatile("cp.async.wait_group 0;\n" ::);

    // Exit counts: a survivor's state is G^E(t0), so E - wlo is its LCG
    // distance from the state of count wlo (exact: the difference is at most
    // count + len, far under the 2^24 period).
    SegList *list = B.lists + x;
    if (live <= (uint32_t)kListMax) {
        const uint32_t t_ref = jump_t(t0, wlo);
        for (uint32_t k = tid; k < live; k += kWinThreads) {
            list->ein[k] = S.ein[k];
            list->eout[k] = (uint16_t)lcg_distance_t(t_ref, S.t[k]);
        }
    }
    if (tid == 0) {
        const SegWindow win{wlo, wlo + count - 1};
        B.windows[j] = win;
        list->win = win;
        list->count = (live <= (uint32_t)kListMax) ? live : kTooMany;
        atomicAdd(&B.st->window_sum, (unsigned long long)count);
        atomicAdd(&B.st->survivor_sum, (unsigned long long)live);
        if (packed) atomicAdd(&B.st->packed, 1u);
    }
    for (int o = 16; o > 0; o >>= 1) steps += __shfl_down_sync(0xFFFFFFFFu, steps, o);
    if (lane == 0 && steps) atomicAdd(&B.st->candidate_steps, (unsigned long long)steps);
}

// Exact serial walk of one segment from a known entry count (a miss), by one
// warp: the lanes load 32 entries at a time, the next 32 while the current
// ones are stepped, and every lane steps the same state.
__device__ __noinline__ uint32_t walk_segment_exact(const AmbEntry *entries,
                                                    const SecondInterval *second, uint32_t i0,
                                                    uint32_t i1, uint32_t e_in, uint32_t t0) {
    const int lane = threadIdx.x & 31;
    const uint4 *e4 = reinterpret_cast<const uint4 *>(entries);
    uint32_t S = jump_t(t0, e_in);
    uint32_t E = e_in;
    uint4 cur = i0 + lane < i1 ? __ldg(e4 + i0 + lane) : make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t i = i0; i < i1; i += 32) {
        const uint32_t nat = i + 32 + lane;
        const uint4 nxt = nat < i1 ? __ldg(e4 + nat) : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t cnt = min(32u, i1 - i);
        for (uint32_t q = 0; q < cnt; ++q) {
            uint4 e;
            e.x = __shfl_sync(0xFFFFFFFFu, cur.x, q);
            e.y = __shfl_sync(0xFFFFFFFFu, cur.y, q);
            e.z = __shfl_sync(0xFFFFFFFFu, cur.z, q);
            e.w = __shfl_sync(0xFFFFFFFFu, cur.w, q);
            if (!copies(e, second + i + q, S)) {
                S = 125u * S + 256u;
                E += 1u;
            }
        }
        cur = nxt;
    }
    return E;
}

// Position of the last of `n` ascending entries at or below q (the first is
// at or below every q asked).
__device__ __forceinline__ uint32_t last_at_or_below(const uint16_t *e, uint32_t n, uint32_t q) {
    uint32_t l = 0, h = n;
    while (h - l > 1u) {
        const uint32_t mid = (l + h) / 2u;
        if (e[mid] <= q) l = mid;
        else h = mid;
    }
    return l;
}

// Composition of a group's lists: every survivor of the first list followed
// through the others, one thread each, by binary search in shared memory.
// The exit counts after every segment go to B.path; a count that leaves a
// window, or meets a list that overflowed, is kNone from there on.  The
// lists are read through L2 only (the same scratch is rewritten every wave,
// and a line this SM cached in an earlier wave must not be read).
struct GroupSmem {
    uint32_t count[kGroup];
    SegWindow win[kGroup];
    uint16_t ein[kGroup][kListMax], eout[kGroup][kListMax];
};

__device__ void compose_group(const WalkBuffers &B, GroupSmem &S, uint32_t x0, uint32_t n) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t s = warp; s < n; s += kWinWarps) {
        const SegList *L = B.lists + x0 + s;
        const uint4 head = __ldcg(reinterpret_cast<const uint4 *>(L));
        const uint32_t cnt = head.x <= (uint32_t)kListMax ? head.x : 0u;
        if (lane == 0) {
            S.count[s] = cnt;
            S.win[s] = SegWindow{head.y, head.z};
        }
        for (uint32_t v = lane; v < (cnt + 7u) / 8u; v += 32) {
            reinterpret_cast<uint4 *>(S.ein[s])[v] = __ldcg(reinterpret_cast<const uint4 *>(L->ein) + v);
            reinterpret_cast<uint4 *>(S.eout[s])[v] =
                __ldcg(reinterpret_cast<const uint4 *>(L->eout) + v);
        }
    }
    __syncthreads();
    for (uint32_t k = tid; k < S.count[0]; k += kWinThreads) {
        uint32_t E = S.win[0].lo + S.eout[0][k];
        B.path[(size_t)x0 * kListMax + k] = E;
        for (uint32_t s = 1; s < n; ++s) {
            const SegWindow w = S.win[s];
            if (E != kNone && S.count[s] && E >= w.lo && E <= w.hi)
                E = w.lo + S.eout[s][last_at_or_below(S.ein[s], S.count[s], E - w.lo)];
            else
                E = kNone;
            B.path[(size_t)(x0 + s) * kListMax + k] = E;
        }
    }
}

// End of a wave: chain the exact E through the groups (warp 0, one lookup
// per group: the survivor of E in the group's first list gives its exit
// count, as an offset in the next group's first window), then every
// segment's exact entry count from the survivor chosen in its group.
constexpr int kMaxGroups = 32;
struct FinalSmem {
    uint32_t count[kMaxGroups];              // survivors of the first list
    SegWindow win[kMaxGroups + 1];           // its window (then an empty one)
    uint32_t pick[kMaxGroups];               // survivor chosen; kNone: written already
    uint32_t stop;                           // segments resolved
    uint16_t ein[kMaxGroups][kListMax];
    uint16_t next[kMaxGroups][kListMax];     // 0xFFFF: not in the next group's window
};
constexpr size_t kWaveSmem =
    sizeof(FinalSmem) > sizeof(WindowSmem)
        ? (sizeof(FinalSmem) > sizeof(GroupSmem) ? sizeof(FinalSmem) : sizeof(GroupSmem))
        : (sizeof(WindowSmem) > sizeof(GroupSmem) ? sizeof(WindowSmem) : sizeof(GroupSmem));
static_assert(kWinBlocksPerSM * (kWaveSmem + 1024) <= 228 * 1024, "window blocks per SM");

__device__ void resolve_wave(const WalkBuffers &B, FinalSmem &S, const WalkPlan &plan, uint32_t n,
                             uint32_t wave, uint32_t launches, uint32_t per_wave, uint32_t c_wave,
                             uint32_t e0, uint32_t here, uint32_t t0) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a miss at segment x ends the wave there, if the launches left can still
    // cover the chain from it
    const auto restarts = [&](uint32_t x) {
        const uint32_t left = plan.chunks - (c_wave + plan.start(x));
        return (left + plan.wave_chunks - 1u) / plan.wave_chunks <= launches - (wave + 1u);
    };
    const uint32_t groups = (here + kGroup - 1) / kGroup;
    if (tid <= (int)groups && tid < kMaxGroups + 1) {
        uint4 head = make_uint4(0u, 1u, 0u, 0u);  // past the last: an empty window
        if (tid < (int)groups)
            head = __ldcg(reinterpret_cast<const uint4 *>(B.lists + (size_t)tid * kGroup));
        S.win[tid] = SegWindow{head.y, head.z};
        if (tid < (int)groups) S.count[tid] = head.x <= (uint32_t)kListMax ? head.x : 0u;
    }
    __syncthreads();
    for (uint32_t g = warp; g < groups; g += kWinWarps) {
        const uint32_t x0 = g * kGroup, last = min(here, x0 + kGroup) - 1u;
        const SegList *L = B.lists + x0;
        const uint32_t cnt = S.count[g];
        const SegWindow nw = S.win[g + 1];
        for (uint32_t k = lane; k < cnt; k += 32) {
            S.ein[g][k] = __ldcg(L->ein + k);
            const uint32_t E = __ldcg(B.path + (size_t)last * kListMax + k);
            const bool in = E != kNone && E >= nw.lo && E <= nw.hi;
            S.next[g][k] = in ? (uint16_t)(E - nw.lo) : (uint16_t)0xFFFFu;
        }
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t E = e0;
        uint32_t fallbacks = 0;
        uint32_t stop = here;  // segments resolved
        for (uint32_t g = 0; g < groups && stop == here; ++g) {
            const uint32_t x0 = g * kGroup, end = min(here, x0 + kGroup);
            const uint32_t cnt = S.count[g];
            const SegWindow win = S.win[g];
            if (lane == 0) B.e_in[wave * per_wave + x0] = E;
            if (cnt && E >= win.lo && E <= win.hi) {
                const uint32_t q = E - win.lo;
                uint32_t below = 0;
#pragma unroll
                for (int m = 0; m < kListMax / 32; ++m) {
                    const uint32_t k = m * 32 + lane;
                    below += (k < cnt && S.ein[g][k] <= q) ? 1u : 0u;
                }
                below = __reduce_add_sync(0xFFFFFFFFu, below);
                const uint32_t k = below - 1u;
                const uint32_t nx = S.next[g][k];
                uint32_t Ex = S.win[g + 1].lo + nx;
                if (nx == 0xFFFFu) Ex = __ldcg(B.path + (size_t)(end - 1u) * kListMax + k);
                if (Ex != kNone) {
                    if (lane == 0) S.pick[g] = k;
                    E = Ex;
                    continue;
                }
            }
            // a miss inside the group: segment by segment
            for (uint32_t x = x0; x < end; ++x) {
                const SegList *L = B.lists + x;
                const uint4 head = __ldcg(reinterpret_cast<const uint4 *>(L));
                const bool listed =
                    head.x <= (uint32_t)kListMax && head.x > 0 && E >= head.y && E <= head.z;
                if (!listed) {
                    ++fallbacks;
                    if (x > 0 && restarts(x)) {
                        stop = x;
                        break;
                    }
                }
                if (lane == 0) B.e_in[wave * per_wave + x] = E;
                if (listed) {
                    const uint32_t q = E - head.y;
                    uint32_t below = 0;
                    for (uint32_t k = lane; k < head.x; k += 32) below += __ldcg(L->ein + k) <= q;
                    below = __reduce_add_sync(0xFFFFFFFFu, below);
                    E = head.y + __ldcg(L->eout + below - 1u);
                } else {
                    const uint32_t c = c_wave + plan.start(x), ce = c_wave + plan.start(x + 1);
                    E = walk_segment_exact(B.entries, B.second, c * kWalkChunk,
                                           min(n, ce * kWalkChunk), E, t0);
                }
            }
            if (lane == 0) S.pick[g] = kNone;
        }
        if (lane == 0) {
            const uint32_t end = min(plan.chunks, c_wave + plan.start(stop));
            B.wave[wave + 1] = make_uint2(end, E);
            B.st->waves = wave + 1;
            B.st->fallbacks += fallbacks;
            B.st->groups_done = 0;  // for the next wave
            S.stop = stop;
        }
    }
    __syncthreads();
    // the other segments of a group: the exit count of the one before
    for (uint32_t x = tid; x < S.stop; x += kWinThreads) {
        const uint32_t k = S.pick[x / kGroup];
        if (x % kGroup && k != kNone)
            B.e_in[wave * per_wave + x] = __ldcg(B.path + (size_t)(x - 1) * kListMax + k);
    }
}

// One wave of the speculative walk: one block per segment.
__global__ void __launch_bounds__(kWinThreads, kWinBlocksPerSM)
    k_wave(WalkBuffers B, const uint32_t *__restrict__ n_ptr, int64_t capacity, uint32_t wave,
           uint32_t launches, uint32_t per_wave, uint32_t t0, uint32_t serial_below, double sigmas, uint32_t *err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_last;
    grid_dependency();
    if (pass_stopped(err)) return;
    const uint32_t n = (uint32_t)min((int64_t)*n_ptr, capacity);
    if (n < serial_below) return;  // the chain is walked serially instead
    const WalkPlan plan = walk_plan(n, per_wave);
    // where this wave starts: written by the wave before, never during this one
    const uint2 from = __ldcg(B.wave + wave);
    const uint32_t c_wave = from.x;
    const uint32_t here = wave_segments(plan, c_wave);
    const uint32_t x = blockIdx.x;
    if (here == 0 && x == 0 && threadIdx.x == 0) B.wave[wave + 1] = from;  // nothing left
    if (x >= here) return;  // past the chain
    const uint32_t i0 = (c_wave + plan.start(x)) * kWalkChunk;
    const uint32_t i1 = min(n, (c_wave + plan.start(x + 1)) * kWalkChunk);
    window_block(B, *reinterpret_cast<WindowSmem *>(smem_raw), c_wave, from.y, i0, i1,
                 wave * per_wave + x, x, t0, sigmas);
    // the last of a group composes it; the last group resolves the wave
    const uint32_t g = x / kGroup, size = min((uint32_t)kGroup, here - g * kGroup);
    const uint32_t groups = (here + kGroup - 1) / kGroup;
    __threadfence();
    __syncthreads();  // every output of the segment is written
    if (threadIdx.x == 0) s_last = atomicAdd(B.group_done + g, 1u) == size - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) B.group_done[g] = 0u;  // for the next wave
    compose_group(B, *reinterpret_cast<GroupSmem *>(smem_raw), g * kGroup, size);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&B.st->groups_done, 1u) == groups - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    resolve_wave(B, *reinterpret_cast<FinalSmem *>(smem_raw), plan, n, wave, launches, per_wave,
                 c_wave, from.y, here, t0);
}

// ---------------------------------------------------------------------------
// Per-channel extra draws: one lane per piece of kPiece channels, from the
// exact state at the piece's start.
// ---------------------------------------------------------------------------

// A lane finds its piece's start from the segment's exact entry count: the
// survivor of that count in the list the window block kept there.  The warp
// stages the 32 pieces' entries 32 channels at a time (one cp.async
// instruction per piece: 512 consecutive bytes), rows padded by 16 bytes so
// the lanes' 16-byte reads of one channel spread over all banks.  A step is
// one dependent chain of 23 cycles, so a piece takes 512 of them, and the
// pieces of a native frame are about one warp per scheduler.  Walking each
// 4096-channel segment on one lane took 124 us whatever the frame's size;
// this takes 60 us on a native frame (8.9 M channels) and 15 us on 256x256.
// A serial walk (a short chain, or all of one) is one lane: only its row is
// staged, and the idle lanes don't hold it off the unrolled steps (113.9 ->
// 45.2 ms for the 2.2 M channels of a 2892x1973 frame; a warp of pieces that
// end apart gains as well, 78 -> 60 us).
constexpr int kRewalkChunk = 32;  // channels per staged chunk
constexpr int kRewalkRing = 3;

struct RewalkSmem {
    uint4 e[kRewalkRing][32][kRewalkChunk + 1];
};

__global__ void __launch_bounds__(32)
    k_rewalk(WalkBuffers B, const uint32_t *__restrict__ n_ptr, int64_t capacity,
             uint32_t per_wave, uint32_t t0, ExtraWord *__restrict__ extra, uint32_t serial_below,
             const uint32_t *__restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RewalkSmem &S = *reinterpret_cast<RewalkSmem *>(smem_raw);
    grid_dependency();
    if (pass_stopped(err)) return;
    const int lane = threadIdx.x;
    const uint32_t n = (uint32_t)min((int64_t)*n_ptr, capacity);
    const uint32_t p = blockIdx.x * 32 + lane;
    uint32_t from = 0, a = 0, b = 0;  // walk [from, b), write from a (from < a: replay)
    uint32_t T = t0, E = 0;
    if (n < serial_below) {  // a short chain (or the serial mode): one lane from E = 0
        if (blockIdx.x) return;
        if (n == 0 && lane == 0) extra[0] = ExtraWord{0u, 0u};  // read by every site's lookup
        b = p == 0 ? n : 0u;
    } else {
        // pieces of segment x of a wave take the places from start(x) / 2 + x
        // on (a segment of c chunks has at most c / 2 + 1 pieces)
        const WalkPlan plan = walk_plan(n, per_wave);
        const uint32_t places = plan.wave_chunks / 2u + plan.segs;
        const uint32_t w = p / places, q = p % places;
        if (w < B.st->waves) {
            const uint32_t c_wave = B.wave[w].x, c_end = B.wave[w + 1].x;
            uint32_t l = 0, h = plan.segs;
            while (h - l > 1u) {
                const uint32_t mid = (l + h) / 2u;
                if (plan.start(mid) / 2u + mid <= q) l = mid;
                else h = mid;
            }
            const uint32_t s0 = plan.start(l), m = q - (s0 / 2u + l);
            const uint32_t c0 = c_wave + s0;
            const uint32_t c1 = min(c_end, c_wave + plan.start(l + 1));
            const uint32_t c = c0 + m * (kPiece / kWalkChunk);
            if (c < c1) {
                const uint32_t j = w * per_wave + l;
                a = c * kWalkChunk;
                b = min(n, min(c1 * kWalkChunk, a + kPiece));
                from = c0 * kWalkChunk;
                E = B.e_in[j];
                T = jump_t(t0, E);
                const SegWindow win = B.windows[j];
                if (m > 0 && E >= win.lo && E <= win.hi) {
                    const KeptHead k = B.kept[c];
                    if (k.count) {  // else replayed from the segment's start
                        // the last survivor at or below the entry count
                        const uint32_t at =
                            k.offset + last_at_or_below(B.kept_ein + k.offset, k.count, E - win.lo);
                        T = B.kept_state[at];
                        E = win.lo + lcg_distance_t(jump_t(t0, win.lo), T);
                        from = a;
                    }
                }
            }
        }
    }
    const uint32_t mine = (b - from + kRewalkChunk - 1) / kRewalkChunk;
    const uint32_t chunks = __reduce_max_sync(0xFFFFFFFFu, mine);
    if (chunks == 0) return;
    // lanes up to the last with channels (one alone on a serial walk)
    const int rows = 32 - __clz(__ballot_sync(0xFFFFFFFFu, mine > 0u));
    auto issue = [&](uint32_t k) {
        if (k < chunks) {
#pragma unroll 8
            for (int q = 0; q < rows; ++q) {
                const uint32_t f = __shfl_sync(0xFFFFFFFFu, from, q) + k * kRewalkChunk + lane;
                if (f < __shfl_sync(0xFFFFFFFFu, b, q)) {
                    const uint32_t sa =
                        (uint32_t)__cvta_generic_to_shared(&S.e[k % kRewalkRing][q][lane]);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa),
                                 "l"(reinterpret_cast<const uint4 *>(B.entries) + f));
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
#pragma unroll
    for (int k = 0; k < kRewalkRing - 1; ++k) issue(k);
    for (uint32_t k = 0; k < chunks; ++k) {
        issue(k + kRewalkRing - 1);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kRewalkRing - 1));
        __syncwarp();
        const uint32_t i = from + k * kRewalkChunk;
        const uint32_t cnt = i < b ? min((uint32_t)kRewalkChunk, b - i) : 0u;
        const uint4 *row = S.e[k % kRewalkRing][lane];
        const bool two = cnt && B.chunk_two[i / kWalkChunk] != 0;
        uint32_t bits = 0;
        // a lane past its end steps through whatever its row holds; its state
        // and count are not used again
        if (__all_sync(0xFFFFFFFFu, cnt == 0u || (cnt == (uint32_t)kRewalkChunk && !two))) {
#pragma unroll
            for (int r = 0; r < kRewalkChunk; ++r) {
                const uint4 e = row[r];
                const bool x = e.x * T + e.y > e.z;
                bits |= x ? 1u << r : 0u;
                T = x ? 125u * T + 256u : T;
            }
        } else {
            for (uint32_t r = 0; r < cnt; ++r) {
                const bool x = !copies(row[r], B.second + i + r, T);
                bits |= x ? 1u << r : 0u;
                T = x ? 125u * T + 256u : T;
            }
        }
        if (cnt) {
            if (i >= a) extra[i / 32] = ExtraWord{E, bits};
            E += (uint32_t)__popc(bits);
        }
        __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    if (b == n && b > from && (n & 31u) == 0u) extra[n / 32] = ExtraWord{E, 0u};
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// Waves launched for a chain of the list's capacity: spare ones where a miss
// is expensive (long segments).
static uint32_t wave_launches(const WalkPlan &plan) {
    return plan.waves + (plan.even ? 0u : kSpareWaves);
}

constexpr size_t kWalkZeroGroups = 128, kWalkZeroWaves = 256;
static_assert(sizeof(WalkState) <= kWalkZeroGroups &&
                  kWalkZeroGroups + kMaxGroups * sizeof(uint32_t) <= kWalkZeroWaves,
              "the cleared part's layout");
size_t walk_zero_bytes(int64_t capacity) {
    // a wave has at least one segment, so at least kWalkAvgMax chunks
    return kWalkZeroWaves +
           (walk_chunks(capacity) / kWalkAvgMax + 2 + kSpareWaves) * sizeof(uint2);
}

static uint32_t walk_channels(int64_t capacity) {
    return (uint32_t)std::min<int64_t>(capacity, 0xFFFFFF00ll);
}

// Segment records (window, entry count) of a walk in waves of `per_wave`.
int64_t walk_segments(int64_t capacity, int per_wave) {
    const WalkPlan plan = walk_plan(walk_channels(capacity), (uint32_t)per_wave);
    return (int64_t)wave_launches(plan) * per_wave;
}

// Segment records that hold a walk in waves of any number of segments up to
// `widest`: c chunks in waves of s segments are ceil(c / (kWalkAvgMax s))
// waves (at least one) and kSpareWaves more, so at most c / kWalkAvgMax +
// (1 + kSpareWaves) s records.  A narrower wave can need more records than the
// widest: one of 591 segments ramps from 2364 chunks on, with spare waves, one
// of 592 from 2368 on.
int64_t walk_segments_reserved(int64_t capacity, int widest) {
    const WalkPlan plan = walk_plan(walk_channels(capacity), (uint32_t)widest);
    return plan.chunks / kWalkAvgMax + (int64_t)(1u + kSpareWaves) * widest;
}

// Device layout of the walk scratch for lists of up to `capacity` channels and
// waves of up to `widest` segments; returns its size.
static size_t walk_layout(void *scratch, void *zero, int64_t capacity, int widest,
                          WalkBuffers *B) {
    const size_t segments = (size_t)walk_segments_reserved(capacity, widest);
    char *base = reinterpret_cast<char *>(scratch);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *r = base + off;
        off += (bytes + 255) & ~(size_t)255;
        return r;
    };
    WalkBuffers b{};
    b.windows = (SegWindow *)take(segments * sizeof(SegWindow));
    b.e_in = (uint32_t *)take(segments * sizeof(uint32_t));
    b.lists = (SegList *)take((size_t)widest * sizeof(SegList));
    b.path = (uint32_t *)take((size_t)widest * kListMax * sizeof(uint32_t));
    b.kept = (KeptHead *)take(walk_chunks(capacity) * sizeof(KeptHead));
    const int64_t pool = kept_pool(capacity);
    b.kept_state = (uint32_t *)take((size_t)pool * sizeof(uint32_t));
    b.kept_ein = (uint16_t *)take((size_t)pool * sizeof(uint16_t));
    b.kept_size = (uint32_t)std::min<int64_t>(pool, 0xFFFFFFFFll);
    // the cleared part: state, group counters, the waves' starts
    b.st = (WalkState *)zero;
    b.group_done = (uint32_t *)((char *)zero + kWalkZeroGroups);
    b.wave = (uint2 *)((char *)zero + kWalkZeroWaves);
    if (B) *B = b;
    return off;
}

size_t walk_scratch_bytes(int64_t capacity, int widest) {
    return walk_layout(nullptr, nullptr, capacity, widest, nullptr);
}

// Segments per wave: the blocks that fit the SMs, so every block of a wave is
// resident at once (a block left waiting for a slot would start late, and it
// would be the wave's last, widest window).
int walk_per_wave(int sms) { return std::min(kWinBlocksPerSM * sms, kMaxGroups * kGroup); }

cudaError_t walk_init() {
    Affine tab[4][64];
    Affine step{125u, 256u};  // G^(64^j)
    for (int j = 0; j < 4; ++j) {
        Affine acc{1u, 0u};
        for (int d = 0; d < 64; ++d) {
            tab[j][d] = acc;
            acc = affine_compose(step, acc);
        }
        step = acc;
    }
    cudaError_t e = cudaMemcpyToSymbol(g_pow, tab, sizeof(tab));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_wave, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWaveSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_rewalk, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(RewalkSmem));
}

// Enqueue the walk.  The channel count stays on the device (n_ptr): the
// launch shape is sized from the list capacity and every kernel exits early
// beyond the count, so nothing waits for the host.  Chains shorter than
// kSerialBelow (or every chain, when `parallel` is off) are walked by one
// lane instead of the speculative windows.
cudaError_t launch_walk(const AmbEntry *entries, const SecondInterval *second,
                        const uint32_t *n_ptr, int64_t capacity, uint32_t s0, void *scratch,
                        void *zero, int widest, int per_wave, bool parallel, double window_sigmas,
                        const uint8_t *chunk_two, const ChunkStat *chunk_stat, ExtraWord *extra,
                        const uint32_t *err, cudaStream_t stream, int priority) {
    WalkBuffers B;
    walk_layout(scratch, zero, capacity, widest, &B);
    B.entries = entries;
    B.second = second;
    B.chunk_two = chunk_two;
    B.chunk_stat = chunk_stat;
    const uint32_t t0 = (s0 & kLcgMask) << 8;
    const uint32_t serial_below = parallel ? kSerialBelow : 0xFFFFFFFFu;
    int64_t places = 1;
    if (parallel) {
        const WalkPlan plan = walk_plan(walk_channels(capacity), (uint32_t)per_wave);
        const uint32_t blocks = std::min((uint32_t)per_wave, plan.chunks);
        const uint32_t launches = wave_launches(plan);
        // half a wave's chunks (a shorter chain may have longer waves than the
        // capacity's) and per_wave places a wave
        const uint32_t reach = std::min(plan.chunks, (uint32_t)per_wave * kWalkAvgMax);
        places = (int64_t)launches * (reach / 2 + per_wave + 2);
        for (uint32_t w = 0; w < launches; ++w) {
            const cudaError_t e =
                launch_chained(k_wave, dim3(blocks), dim3(kWinThreads), kWaveSmem, stream, priority,
                            B, n_ptr, capacity, w, launches, (uint32_t)per_wave, t0, serial_below,
                            window_sigmas, const_cast<uint32_t *>(err));
            if (e != cudaSuccess) return e;
        }
    }
    cudaError_t e = launch_chained(k_rewalk, dim3((unsigned)((places + 31) / 32)), dim3(32),
                                sizeof(RewalkSmem), stream, priority, B, n_ptr, capacity,
                                (uint32_t)per_wave, t0, extra, serial_below, err);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace fx
