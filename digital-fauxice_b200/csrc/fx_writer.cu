// fx_writer.cu -- the sequential dither writer, restructured for the GPU.
//
// The reference writes attempted sites in strict row-major order, threading
// one 24-bit LCG through every conditional draw (reconstruction.py:916-982,
// dither.py:59-104, rng.py:159-172).  The number of draws a channel takes is
// a function of the state only when its first draw happens, the floor gate
// is on and the floor comparison is not settled by the largest possible
// |delta|.  So:
//   1. k_stencil / k_startup classify every channel: 0, 1 or 2 fixed draws,
//      or "RNG-dependent" (one or two).
//   2. k_seg_sums: exclusive prefix of fixed draws and of RNG-dependent
//      channels along the chain (startup sites, then public sites in
//      row-major order).
//   3. k_coef: lists the RNG-dependent channels and finds, for each, the set
//      of first-draw states that copy the original, as at most two state
//      intervals (by binary search on the exact binary64 expressions, which
//      are monotone in the state), as a test on the extra draws before it
//      (the channel's fixed draws folded into an affine LCG jump).
//   4. the walk (fx_walk.cu) visits only the RNG-dependent channels: a
//      multiply-add, a test and a conditional LCG step per channel,
//      parallelised over segments by speculation.  Output: the running count of extra draws.
//   5. k_apply: every public site makes its draws and computes its values from
//      its own start state g^(fixed + extra before it)(s0), in parallel, and
//      emits public RGB16 with the counters.  Draws that differ from what steps
//      1 and 4 say fail the pass.
#include <algorithm>

#include "fx_internal.cuh"

namespace fx {

struct alignas(16) DevCounters {
    unsigned long long attempted, written, public_advances, changed;
    unsigned long long su_attempted[6], su_advances[6];
    unsigned long long public_base, public_amb;
    uint32_t final_state, su_final_state;
    uint32_t startup_base, startup_amb, startup_extra;
    uint32_t n_amb;
    uint32_t walk_fallbacks;
    uint32_t walk_packed;
    unsigned long long walk_stats[3];  // candidate steps, window sum, survivor sum
    uint32_t su_base[6], su_amb[6];    // per startup row, for the last block's chain
    uint32_t seg_done;                 // k_seg_sums's finished blocks
    uint32_t coef_next;                // k_coef's next ticket
    uint32_t apply_next;               // k_apply's next ticket
    uint32_t apply_done;               // k_apply's finished blocks
};

// Extra draws of the first `count` RNG-dependent channels (clamped to the
// list capacity; an overflowing frame is rerun by the host).
__device__ __forceinline__ uint32_t extra_before(const ExtraWord *extra, uint32_t count,
                                                 int64_t capacity) {
    if (count == 0) return 0u;
    const uint32_t i = (uint32_t)((int64_t)count < capacity ? (int64_t)count : capacity);
    const uint2 w = __ldg(reinterpret_cast<const uint2 *>(extra) + (i >> 5));
    return w.x + (uint32_t)__popc(w.y & ((1u << (i & 31u)) - 1u));
}

// (fixed draws << 16) | RNG-dependent channels of the four sites of one
// meta word.  Per channel code k (bits 2c, 2c+1): fixed draws k, except 1
// for k = 3, and one RNG-dependent channel when k = 3; so over the lows
// (k & 1), highs (k >> 1) and both: fixed = lows + 2 highs - 2 both.
__device__ __forceinline__ uint32_t packed_word(uint32_t w) {
    const uint32_t lo = w & 0x15151515u, hi = (w >> 1) & 0x15151515u;
    const uint32_t amb = (uint32_t)__popc(lo & hi);
    const uint32_t base = (uint32_t)__popc(lo) + 2u * (uint32_t)__popc(hi) - 2u * amb;
    return (base << 16) | amb;
}

constexpr int kSegWarps = 8;  // segments per block of the chain kernels (one per warp)

static_assert(kSegWarps == kSegGroup, "a k_seg_sums block sums one group of segments");

// The chain prefix's partial sums (seg_raw_words): per-segment sums, then
// the groups' exclusive prefixes of fixed draws and RNG-dependent channels.
struct SegRaw {
    uint32_t *seg, *grp_base, *grp_amb;
};
__device__ __forceinline__ SegRaw seg_raw_view(uint32_t *raw, int64_t segs) {
    const int64_t groups = (segs + kSegGroup - 1) / kSegGroup;
    SegRaw v;
    v.seg = raw;
    v.grp_base = raw + ((segs + 63) / 64) * 64;
    v.grp_amb = v.grp_base + ((groups + 63) / 64) * 64;
    return v;
}

// Fixed draws and RNG-dependent channels of every segment (packed as
// fixed << 16 | RNG-dependent), and of every group of eight segments: one
// warp per segment, 32 sites per lane in two 16-byte loads (the meta array
// starts on a 256-byte boundary and segments on multiples of 1024 sites),
// one block per group.  The last block to finish scans the groups' sums into
// their exclusive prefixes, over tiles of 4096 groups (a native frame has 2.8
// k): a tile is loaded coalesced into shared memory, each thread scans 16
// neighbouring groups, and one block scan of (fixed << 32 | RNG-dependent)
// pairs gives the threads' offsets (the RNG-dependent total stays below 2^32:
// at most three per site).  seg_base[segs] and seg_amb[segs] get the totals;
// k_coef adds a segment's offset inside its group.
__global__ void __launch_bounds__(kSegWarps * 32)
    k_seg_sums(const uint8_t *__restrict__ meta, int64_t sites, int64_t segs,
               uint32_t *__restrict__ raw, uint32_t *__restrict__ seg_base,
               uint32_t *__restrict__ seg_amb, DevCounters *ctr,
               const uint32_t *__restrict__ err) {
    constexpr int kPerThread = 16, kTile = kSegWarps * 32 * kPerThread;
    __shared__ uint32_t s_warp[kSegWarps];
    __shared__ uint32_t tile[kTile];
    __shared__ unsigned long long ws[kSegWarps];
    __shared__ bool s_last;
    grid_dependency();
    if (pass_stopped(err)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t seg = (int64_t)blockIdx.x * kSegWarps + warp;
    const SegRaw v = seg_raw_view(raw, segs);
    uint32_t packed = 0;
    const int64_t first = seg * kSegment + lane * 32;
    if (seg < segs) {
        if (first + 32 <= sites) {
            const uint4 *q = reinterpret_cast<const uint4 *>(meta + first);
            const uint4 u = q[0], w = q[1];
            packed = packed_word(u.x) + packed_word(u.y) + packed_word(u.z) + packed_word(u.w) +
                     packed_word(w.x) + packed_word(w.y) + packed_word(w.z) + packed_word(w.w);
        } else {
            for (int i = 0; i < 32; ++i)
                if (first + i < sites) packed += packed_word(meta[first + i]);
        }
    }
    packed = __reduce_add_sync(0xFFFFFFFFu, packed);
    if (lane == 0) {
        if (seg < segs) v.seg[seg] = packed;
        s_warp[warp] = packed;
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t g = 0;  // at most 8 x 6144 fixed draws and 8 x 3072 channels
#pragma unroll
        for (int k = 0; k < kSegWarps; ++k) g += s_warp[k];
        v.grp_amb[blockIdx.x] = g;  // the sum, until the scan below
        __threadfence();
        s_last = atomicAdd(&ctr->seg_done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int64_t groups = gridDim.x;
    unsigned long long carry = 0;
    for (int64_t t0 = 0; t0 < groups; t0 += kTile) {
        for (int j = tid; j < kTile; j += kSegWarps * 32)
            tile[j] = t0 + j < groups ? __ldcg(v.grp_amb + t0 + j) : 0u;
        __syncthreads();
        unsigned long long mine = 0;
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
            const uint32_t g = tile[kPerThread * tid + k];
            mine += ((unsigned long long)(g >> 16) << 32) | (g & 0xFFFFu);
        }
        unsigned long long x = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        unsigned long long run = carry + x - mine;
        for (int k = 0; k < kSegWarps; ++k) {
            if (k < warp) run += ws[k];
            carry += ws[k];
        }
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
            const int64_t i = t0 + kPerThread * tid + k;
            const uint32_t g = tile[kPerThread * tid + k];
            if (i < groups) {
                v.grp_base[i] = (uint32_t)(run >> 32);
                v.grp_amb[i] = (uint32_t)run;
            }
            run += ((unsigned long long)(g >> 16) << 32) | (g & 0xFFFFu);
        }
        __syncthreads();  // the tile and the warp sums are consumed
    }
    if (tid == 0) {
        seg_base[segs] = (uint32_t)(carry >> 32);
        seg_amb[segs] = (uint32_t)carry;
    }
}

// Affine jump tables: g_jump[j][d] = g^(d * 64^j) in T space.  States repeat
// after 2^24 draws, so the low four base-64 digits of a draw count give its
// map on states.
constexpr int kJumpDigits = 4;
__device__ Affine g_jump[kJumpDigits][64];

// Powers of the LCG step for short jumps: g_short[j][d] = g^(d * 128^j) in T
// space, so a jump below 2^14 draws is two lookups.
__device__ Affine g_short[2][128];

// ---------------------------------------------------------------------------
// Copy intervals of one RNG-dependent channel
// ---------------------------------------------------------------------------

struct ChannelView {
    double cand, cd, env, od;
    float span;
    DitherConst dc;
    __device__ double raw(uint32_t s1) const { return dither_raw_delta(cd, env, span, s1); }
    __device__ bool low_ok(double d) const { return dc.low < cd + d; }
    __device__ bool high_ok(double d) const { return cd + d < dc.high; }
    __device__ bool floor_test(double d) const { return cand + d <= od; }
};

// Estimate of the state s1 at which base + raw(s1) reaches target (the delta
// is affine in s1 before rounding), inside [1, 2^24 - 2].  `inverse` is 1 /
// (env * span) to about 2^-45; the search checks the exact predicate, so the
// estimate changes only its cost.
__device__ __forceinline__ uint32_t crossing(double base, double target, double inverse) {
    constexpr double kScale = 1.0 / kNormalization, kOffset = 0.5 / kNormalization - 1.0;
    const double guess = (target - base) * (inverse * kScale) + kOffset;
    // the conversion saturates, and gives 0 for NaN
    return min(max(__double2uint_rz(guess), 1u), kLcgMask - 1u);
}

// First state where a monotone predicate differs from its value p0 at state 0
// (it does differ at 2^24 - 1).  Two probes around the estimate x settle
// nearly every search; otherwise the search gallops from x to a bracket and
// bisects inside.
template <class F>
__device__ __forceinline__ uint32_t switch_point(F pred, bool p0, uint32_t x) {
    const bool px = pred(x), py = pred(x + 1u);
    if (px == p0 && py != p0) return x + 1u;
    // invariant: pred(lo) == p0, pred(hi) != p0, lo < hi
    uint32_t lo = 0u, hi = kLcgMask;
    uint32_t step = 1u;
    if (px == p0) {
        lo = x + 1u;
        while (hi - lo > step) {
            const uint32_t y = lo + step;
            if (pred(y) != p0) {
                hi = y;
                break;
            }
            lo = y;
            step <<= 1;
        }
    } else {
        hi = x;
        while (hi - lo > step) {
            const uint32_t y = hi - step;
            if (pred(y) == p0) {
                lo = y;
                break;
            }
            hi = y;
            step <<= 1;
        }
    }
    while (hi - lo > 1u) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (pred(mid) == p0) lo = mid;
        else hi = mid;
    }
    return hi;
}

// Copy set of one channel in T space: copy iff (T - l1) <= w1 or
// (T - l2) <= w2 (modulo 2^32); l = 0x80 marks an empty interval.
struct CopySet {
    uint32_t l1, w1, l2, w2;
};

// A state copies when its delta, or none if the delta leaves (low, high),
// passes the floor test.  Each of the three tests is monotone in the state,
// so its values at both ends and its switch point give it everywhere.
__device__ __forceinline__ void copy_intervals(const ChannelView &cv, CopySet &e, uint32_t *err) {
    constexpr uint32_t kNever = kLcgMask + 1u;
    const double d0 = cv.raw(0u), d1 = cv.raw(kLcgMask);
    const bool low0 = cv.low_ok(d0), low1 = cv.low_ok(d1);
    const bool high0 = cv.high_ok(d0), high1 = cv.high_ok(d1);
    const bool floor0 = cv.floor_test(d0), floor1 = cv.floor_test(d1);
    // one Newton step on the binary32 reciprocal; out of its range (and for
    // 0) the estimates are infinite or NaN and the searches gallop
    const double scale = cv.env * (double)cv.span;
    const double r = (double)__frcp_rn((float)scale);
    const double inverse = r * (2.0 - scale * r);
    uint32_t bf = kNever;
    if (floor0 != floor1)
        bf = switch_point([&](uint32_t s) { return cv.floor_test(cv.raw(s)); }, floor0,
                          crossing(cv.cand, cv.od, inverse));
    // empty interval: l = 0x80 can never match a T value (low byte zero)
    e.l1 = 0x80u; e.w1 = 0u; e.l2 = 0x80u; e.w2 = 0u;
    if (low0 && low1 && high0 && high1) {
        // every delta stays in range (all but a few channels): the floor test
        // alone decides, on the states up to or from its switch point
        const uint32_t lo = floor0 ? 0u : bf, hi = floor0 ? bf - 1u : kLcgMask;
        if (lo <= hi) { e.l1 = lo << 8; e.w1 = (hi - lo) << 8; }
        return;
    }
    const uint32_t bl = low0 == low1 ? kNever
                                     : switch_point(
                                           [&](uint32_t s) { return cv.low_ok(cv.raw(s)); }, low0,
                                           crossing(cv.cd, cv.dc.low, inverse));
    const uint32_t bh = high0 == high1 ? kNever
                                       : switch_point(
                                             [&](uint32_t s) { return cv.high_ok(cv.raw(s)); },
                                             high0, crossing(cv.cd, cv.dc.high, inverse));
    const bool still = cv.floor_test(0.0);  // no delta
    // the pieces between the sorted switch points, in order
    const uint32_t b0 = min(min(bl, bh), bf), b2 = max(max(bl, bh), bf);
    const uint32_t b1 = max(min(bl, bh), min(max(bl, bh), bf));
    uint32_t lo0 = 0u, hi0 = 0u, lo1 = 0u, hi1 = 0u, first = 0u;
    int intervals = 0;
    bool open = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t end = i == 0 ? b0 : (i == 1 ? b1 : (i == 2 ? b2 : kNever));
        if (end == first) continue;  // empty piece
        const bool low = low0 != (first >= bl), high = high0 != (first >= bh);
        const bool copy = low && high ? floor0 != (first >= bf) : still;
        if (copy) {
            if (!open) {
                if (intervals == 0) lo0 = first;
                else if (intervals == 1) lo1 = first;
                else { raise_error(err, FX_ERR_INTERNAL); return; }
                ++intervals;
            }
            if (intervals == 1) hi0 = end - 1u;
            else hi1 = end - 1u;
        }
        open = copy;
        first = end;
    }
    if (intervals == 2 && lo0 == 0u && hi1 == kLcgMask) {
        // [0, hi0] and [lo1, 2^24 - 1] meet across the wrap: one cyclic
        // interval from lo1 (the test (T - l) <= w wraps modulo 2^32)
        e.l1 = lo1 << 8;
        e.w1 = (hi0 - lo1) << 8;
        return;
    }
    if (intervals >= 1) { e.l1 = lo0 << 8; e.w1 = (hi0 - lo0) << 8; }
    if (intervals == 2) { e.l2 = lo1 << 8; e.w2 = (hi1 - lo1) << 8; }
}

// Copy test and state map of every RNG-dependent channel.  Every warp takes
// units of 256 sites, a quarter of a chain segment (or 64, see unit_sites): the segment's meta bytes
// give the chain offsets of the unit's sites, the channels are listed in the
// warp's shared memory (at most three per site), and the list is processed
// densely, one channel per lane, written to consecutive entries.  One
// round's candidates and samples are in flight while the round before
// searches.
//
// Bound: instruction issue (binary64 probes, list building), with the first
// candidates of a unit waiting on memory.  A native frame's 9.3 M channels
// take 173 us, at 5% coverage 17.4 M take 250.  Listing the channels in a
// kernel of its own, through memory, and evaluating every piece between the
// switch points anew took 300 and 500.  Five blocks per SM at 48 registers:
// four at 60 registers measured 6% more, six (with spills) 5% more.
constexpr int kCoefWarps = 8, kCoefBlocksPerSM = 5;
constexpr int kUnitSites = 256;  // most sites of a unit
static_assert(kSegment == 1024 && kUnitSites == 32 * 8, "32 and 8 meta bytes per lane");

// Sites of a unit of k_coef and k_apply (template instances).  256 keep a
// warp's lists dense; where 64 still give every resident warp of k_coef at most
// one unit, the frame is bound by one unit's latency and 64 are faster: a
// 256x256 frame's chain 29 -> 19 us and apply 24 -> 20, of 580x600 34 -> 23 and
// 25 -> 25.
static int unit_sites(int64_t segments, int resident_warps) {
    return segments * (kSegment / 64) <= resident_warps ? 64 : kUnitSites;
}

// Meta bytes of a unit of US sites: this lane's 8 sites (US / 8 lanes have
// any), and the packed sums (fixed << 16 | RNG-dependent) of the segment's
// sites before the unit on this lane.
struct UnitMeta {
    uint32_t word[2];
    uint32_t ahead;
};
template <int US>
__device__ __forceinline__ UnitMeta unit_meta(const uint8_t *__restrict__ meta, int64_t sites,
                                              int64_t seg, int part) {
    const int lane = threadIdx.x & 31;
    const int64_t first = seg * kSegment + part * US;
    const int64_t mine = first + lane * 8, far = seg * kSegment + lane * 32;
    UnitMeta u{{0u, 0u}, 0u};
    if (first + US <= sites) {
        if (lane < part * (US / 32)) {
            const uint4 *q = reinterpret_cast<const uint4 *>(meta + far);
            const uint4 a = q[0], b = q[1];
            u.ahead = packed_word(a.x) + packed_word(a.y) + packed_word(a.z) + packed_word(a.w) +
                      packed_word(b.x) + packed_word(b.y) + packed_word(b.z) + packed_word(b.w);
        }
        if (lane < US / 8) {
            const uint2 v = *reinterpret_cast<const uint2 *>(meta + mine);
            u.word[0] = v.x;
            u.word[1] = v.y;
        }
    } else {  // the chain's last unit
        if (lane < part * (US / 32))
            for (int i = 0; i < 32; ++i) u.ahead += packed_word(meta[far + i]);
        for (int i = 0; i < 8; ++i)
            if (lane < US / 8 && mine + i < sites) u.word[i >> 2] |= (uint32_t)meta[mine + i] << (8 * (i & 3));
    }
    return u;
}

template <int US>
__global__ void __launch_bounds__(kCoefWarps * 32, kCoefBlocksPerSM)
    k_coef(AmbEntry *__restrict__ entries, SecondInterval *__restrict__ second, int64_t capacity,
           const uint8_t *__restrict__ meta, int64_t sites, int64_t segs,
           uint32_t *__restrict__ raw, uint32_t *__restrict__ seg_base,
           uint32_t *__restrict__ seg_amb, const double *__restrict__ cand, int w,
           const uint16_t *__restrict__ rgbi, const float *__restrict__ lut, fx_params p,
           uint8_t *__restrict__ chunk_two, ChunkStat *__restrict__ chunk_stat, DevCounters *ctr,
           uint32_t *err) {
    __shared__ Affine s_jump[2][128];
    // listed channels: site in the unit | channel << 8 | fixed draws before it
    // in the segment << 10
    __shared__ uint32_t s_list[kCoefWarps][3 * US];
    grid_dependency();
    if (pass_stopped(err)) return;
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < 256; i += kCoefWarps * 32)
        s_jump[i >> 7][i & 127] = g_short[i >> 7][i & 127];
    __syncthreads();
    uint32_t *list = s_list[threadIdx.x >> 5];
    const DitherConst dc = dither_const(p);
    const int64_t su = 6 * (int64_t)w;
    const SegRaw v = seg_raw_view(raw, segs);
    constexpr int kPerSegment = kSegment / US;
    const int64_t units = segs * kPerSegment;
    // two units per ticket on large frames (the counter is one address)
    const int grab = units > 8 * (int64_t)gridDim.x * kCoefWarps ? 2 : 1;
    int64_t unit = 0;
    for (int left = 0;; --left, ++unit) {
        if (left == 0) {
            uint32_t ticket = 0;
            if (lane == 0) ticket = atomicAdd(&ctr->coef_next, 1u);
            unit = (int64_t)__shfl_sync(0xFFFFFFFFu, ticket, 0) * grab;
            left = grab;
        }
        if (unit >= units) break;
        const int64_t seg = unit / kPerSegment;
        const int part = (int)(unit % kPerSegment);
        const int64_t first = seg * kSegment + part * US;
        if (first >= sites) continue;
        const UnitMeta u = unit_meta<US>(meta, sites, seg, part);
        // the segment's prefix: its group's, plus the segments before it in
        // the group (fewer than eight, so the packed halves cannot carry);
        // its first unit writes it for the kernels after the walk
        const int64_t grp = seg / kSegGroup, k0 = grp * kSegGroup;
        const uint32_t before =
            __reduce_add_sync(0xFFFFFFFFu, (k0 + lane < seg) ? v.seg[k0 + lane] : 0u);
        const uint32_t seg_p = v.grp_base[grp] + (before >> 16);
        const uint32_t seg_a = v.grp_amb[grp] + (before & 0xFFFFu);
        if (part == 0 && lane == 0) {
            seg_base[seg] = seg_p;
            seg_amb[seg] = seg_a;
        }
        const uint32_t sum = packed_word(u.word[0]) + packed_word(u.word[1]);
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += y;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, inc, 31) & 0xFFFFu;
        const uint32_t ahead = __reduce_add_sync(0xFFFFFFFFu, u.ahead);
        if (total == 0) continue;
        __syncwarp();  // the previous list is consumed
        {
            uint32_t slot = (inc - sum) & 0xFFFFu;
            uint32_t pos = (ahead + inc - sum) >> 16;  // fixed draws, relative to the segment
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint8_t mi = (uint8_t)(u.word[i >> 2] >> (8 * (i & 3)));
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int code = meta_code(mi, c);
                    if (code == 3) list[slot++] = (uint32_t)(lane * 8 + i) | (c << 8) | (pos << 10);
                    pos += code == 3 ? 1u : (uint32_t)code;
                }
            }
        }
        __syncwarp();
        // G^(draws before the segment + 1): a channel's map starts there
        Affine base{1u, 0u};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            base = affine_compose(g_jump[j][((seg_p + 1u) >> (6 * j)) & 63u], base);
        const uint32_t a0 = seg_a + (ahead & 0xFFFFu);  // list index of the unit's first
        struct Channel {
            uint32_t item, sample;
            double cand;
        };
        auto fetch = [&](uint32_t k) {
            Channel q{0u, 0u, 1.0};
            if (k < total) {
                q.item = list[k];
                const int64_t site = first + (q.item & 0xFFu);
                const int c = (q.item >> 8) & 3;
                const int64_t pixel = site < su ? site % w : site - su;  // startup rows: row 0
                q.sample = rgbi[4 * pixel + c];
                q.cand = cand[3 * site + c];
            }
            return q;
        };
        Channel cur = fetch(lane);
        for (uint32_t k = 0; k < total; k += 32) {
            const Channel q = cur;
            cur = fetch(k + 32 + lane);
            const uint32_t i = a0 + k + lane;
            const bool live = k + lane < total && (int64_t)i < capacity;
            uint32_t m = 0;  // copying states
            if (live) {
                const int c = (q.item >> 8) & 3;
                ChannelView cv;
                cv.cand = q.cand;
                cv.cd = (double)(float)cv.cand;
                cv.dc = dc;
                cv.env = ((dc.high - cv.cd) * (cv.cd - dc.low)) * dc.coefficient;
                cv.span = (float)((double)p.dither_scales[c] * cv.cd);
                cv.od = (double)__ldg(lut + q.sample);
                CopySet e;
                copy_intervals(cv, e, err);
                // a chunk of walk channels with a two-interval entry steps with
                // both interval tests (every other chunk with one)
                if (e.l2 != 0x80u) chunk_two[i / kWalkChunk] = 1;
                if (e.l1 != 0x80u) m += (e.w1 >> 8) + 1u;
                if (e.l2 != 0x80u) m += (e.w2 >> 8) + 1u;
                // G^(pos + 1) less the first interval's start
                const uint32_t pos = q.item >> 10;
                const Affine f = affine_compose(
                    s_jump[1][pos >> 7], affine_compose(s_jump[0][pos & 127u], base));
                entries[i] = AmbEntry{f.a, f.c - e.l1, e.w1, e.l2 != 0x80u ? 1u : 0u};
                if (e.l2 != 0x80u) second[i] = SecondInterval{e.l1 - e.l2, e.w2};
            }
            // the walk's prediction: m copying states of 2^24 (an extra draw
            // with probability p = 1 - m / 2^24), summed per chunk with the
            // spread p (1 - p); a round's entries lie in one or two chunks
            const uint32_t spread =
                live ? (uint32_t)(((unsigned long long)m * ((1u << 24) - m)) >> 23) : 0u;
            const uint32_t chunk = (a0 + k) / kWalkChunk;
            const bool next = live && i / kWalkChunk != chunk;
            uint32_t ms = __reduce_add_sync(0xFFFFFFFFu, next ? 0u : m >> 1);
            uint32_t qs = __reduce_add_sync(0xFFFFFFFFu, next ? 0u : spread);
            if (lane == 0 && ms + qs) {
                atomicAdd(&chunk_stat[chunk].copy, ms);
                atomicAdd(&chunk_stat[chunk].spread, qs);
            }
            if (__any_sync(0xFFFFFFFFu, next)) {
                ms = __reduce_add_sync(0xFFFFFFFFu, next ? m >> 1 : 0u);
                qs = __reduce_add_sync(0xFFFFFFFFu, next ? spread : 0u);
                if (lane == 0) {
                    atomicAdd(&chunk_stat[chunk + 1].copy, ms);
                    atomicAdd(&chunk_stat[chunk + 1].spread, qs);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Apply + emit, counters, final state
// ---------------------------------------------------------------------------

// Emitted value of a table index (output.py:61-73).
__device__ __forceinline__ uint16_t emit_index(uint32_t idx, const uint32_t *hi,
                                               const uint32_t *lo) {
    const unsigned long long prod = (unsigned long long)hi[idx >> 8] * lo[idx & 0xFFu];
    return (uint16_t)((prod >> 20) - 1ull);
}

// Table index of a finite value: trunc(v + 0.5) clipped to 0..65535.  The
// reference adds in binary64, where the sum is exact; v's integer and
// fractional parts are exact in binary32, so this is the same index.
__device__ __forceinline__ uint32_t emit_index_of(float v) {
    const float c = fminf(fmaxf(v, 0.0f), 65535.0f);
    const uint32_t u = (uint32_t)c;
    return u + (c - (float)u >= 0.5f ? 1u : 0u);
}

// Identity emits: ident[v] = emit(lut[v]), the output of a channel whose value
// is its original (every unattempted pixel, and the comparison emit of an
// attempted one).  *bad is set when a LUT value is not finite.
__global__ void k_identity(const float *__restrict__ lut, const uint32_t *__restrict__ hi,
                           const uint32_t *__restrict__ lo, uint16_t *__restrict__ ident,
                           uint32_t *bad) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= 65536) return;
    const float x = lut[v];
    if (!isfinite(x)) atomicOr(bad, 1u);
    ident[v] = isfinite(x) ? emit_index(emit_index_of(x), hi, lo) : (uint16_t)0;
}

cudaError_t writer_identity_table(const float *lut, const uint32_t *hi, const uint32_t *lo,
                                  uint16_t *ident, uint32_t *bad, cudaStream_t stream) {
    cudaMemsetAsync(bad, 0, sizeof(uint32_t), stream);
    k_identity<<<256, 256, 0, stream>>>(lut, hi, lo, ident, bad);
    return cudaGetLastError();
}

constexpr int kApplyBlocksPerSM = 4;  // k_apply's resident blocks per SM
static int g_apply_blocks = kApplyBlocksPerSM * 148;
static int g_coef_blocks = kCoefBlocksPerSM * 148;

int host_write_site(const fx_params &p, bool floor_enabled, const double cand[3],
                    const float orig[3], uint32_t meta, uint32_t redraw, uint32_t *state,
                    float values[3], int32_t *draws) {
    uint32_t s = *state & kLcgMask;
    const WrittenSite out = write_site(cand, orig, floor_enabled, p.dither_scales, dither_const(p),
                                       (uint8_t)meta, redraw, s);
    for (int c = 0; c < 3; ++c) values[c] = out.value[c];
    *draws = (int32_t)out.draws;
    *state = s;
    return out.agrees ? FX_OK : FX_ERR_INTERNAL;
}

cudaError_t writer_init() {
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
        sms > 0) {
        g_apply_blocks = kApplyBlocksPerSM * sms;
        g_coef_blocks = kCoefBlocksPerSM * sms;
    }
    Affine tab[kJumpDigits][64];
    Affine step{125u, 256u};  // g^(64^j)
    for (int j = 0; j < kJumpDigits; ++j) {
        Affine acc{1u, 0u};
        for (int d = 0; d < 64; ++d) {
            tab[j][d] = acc;
            acc = affine_compose(step, acc);
        }
        step = acc;
    }
    cudaError_t e = cudaMemcpyToSymbol(g_jump, tab, sizeof(tab));
    if (e != cudaSuccess) return e;
    Affine brief[2][128];
    Affine one{125u, 256u};  // g^(128^j)
    for (int j = 0; j < 2; ++j) {
        Affine acc{1u, 0u};
        for (int d = 0; d < 128; ++d) {
            brief[j][d] = acc;
            acc = affine_compose(one, acc);
        }
        one = acc;
    }
    return cudaMemcpyToSymbol(g_short, brief, sizeof(brief));
}

// Every warp takes units of 256 sites, a quarter of a chain segment (64 on
// small frames: unit_sites), with no block barrier:
//   * the segment's meta bytes give the chain offsets before the unit and of
//     its sites, and the attempted sites are listed in the warp's shared
//     memory;
//   * the sites that were not attempted are emitted, one pixel per lane
//     (their output is the identity emit);
//   * the list is processed densely, one attempted site per lane, from its
//     own start state: the segment's, advanced by the draws inside it.
// Every draw is evaluated again and compared with the classification and the
// walk's bits (write_site).  The first six units are the startup rows' counts;
// the last block to finish chains the rows and writes the final state.
// Bound: instruction issue and the gathers' L1.  Measured on a native frame
// with half its pixels attempted, every draw evaluated: 505 us as blocks of 256
// threads with a block scan, four pixels per thread and a six-digit jump per
// site; 396 us so.  Four blocks per SM: five at 48 registers 403; with the next
// 32 sites' loads in flight, four blocks took 424, five 457 and three 453.
// Without the comparison, at most one draw a channel, it took 330.  The gathers' L1 decides
// the rest: with the samples staged in shared memory five blocks took 505 us
// and six 866, with a 128 KB emit table instead of the two factor tables 420.
constexpr int kApplyWarps = 8;

__device__ void apply_final(const uint32_t *seg_base, const uint32_t *seg_amb, int64_t segments,
                            const ExtraWord *extra, uint32_t s0, DevCounters *ctr,
                            const WalkState *walk, uint32_t *err, int64_t capacity) {
    uint32_t a_run = 0, p_run = 0;
    for (int r = 0; r < 6; ++r) {
        const uint32_t rb = __ldcg(&ctr->su_base[r]), ra = __ldcg(&ctr->su_amb[r]);
        const uint32_t e_start = extra_before(extra, a_run, capacity);
        const uint32_t e_end = extra_before(extra, a_run + ra, capacity);
        ctr->su_advances[r] = (unsigned long long)rb + (e_end - e_start);
        a_run += ra;
        p_run += rb;
    }
    const uint32_t e_su = extra_before(extra, a_run, capacity);
    ctr->startup_base = p_run;
    ctr->startup_amb = a_run;
    ctr->startup_extra = e_su;
    ctr->su_final_state = lcg_jump(s0, (uint64_t)p_run + e_su);
    const uint32_t p_total = seg_base[segments];
    const uint32_t a_total = seg_amb[segments];
    const uint32_t e_total = extra_before(extra, a_total, capacity);
    ctr->n_amb = a_total;
    ctr->walk_fallbacks = walk->fallbacks;
    ctr->walk_packed = walk->packed;
    ctr->walk_stats[0] = walk->candidate_steps;
    ctr->walk_stats[1] = walk->window_sum;
    ctr->walk_stats[2] = walk->survivor_sum;
    ctr->final_state = lcg_jump(s0, (uint64_t)p_total + e_total);
    const unsigned long long expect =
        (unsigned long long)(p_total - p_run) + (e_total - e_su);
    if ((int64_t)a_total <= capacity && expect != __ldcg(&ctr->public_advances))
        raise_error(err, FX_ERR_INTERNAL);
}

template <int US>
__global__ void __launch_bounds__(kApplyWarps * 32, kApplyBlocksPerSM)
    k_apply(const uint8_t *__restrict__ meta, const double *__restrict__ cand, int64_t sites,
            int w, const uint16_t *__restrict__ rgbi, const float *__restrict__ lut,
            const uint32_t *__restrict__ g_high, const uint32_t *__restrict__ g_low,
            const uint16_t *__restrict__ ident, const fx_stage *__restrict__ stages, fx_params p,
            const uint32_t *__restrict__ seg_base, const uint32_t *__restrict__ seg_amb,
            const ExtraWord *__restrict__ extra, uint32_t s0, uint16_t *__restrict__ rgb_out,
            uint8_t *__restrict__ changed_out, DevCounters *ctr,
            const WalkState *__restrict__ walk, uint32_t *err, int64_t capacity) {
    __shared__ Affine s_jump[2][128];
    __shared__ uint32_t hi[256], lo[256];  // emit factors
    // attempted sites: x = site in the segment | meta << 16, y = fixed draws
    // before it in the segment | RNG-dependent channels before it << 16
    __shared__ uint2 s_list[kApplyWarps][US];
    __shared__ unsigned long long s_sums[kApplyWarps][4];
    __shared__ bool s_last;
    grid_dependency();
    if (pass_stopped(err)) return;  // cancelled: the output stays untouched
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < 256; i += kApplyWarps * 32) {
        s_jump[i >> 7][i & 127] = g_short[i >> 7][i & 127];
        hi[i] = g_high[i];
        lo[i] = g_low[i];
    }
    __syncthreads();
    const int64_t su = 6 * (int64_t)w;
    const int64_t segs = (sites + kSegment - 1) / kSegment;
    const DitherConst dc = dither_const(p);
    uint2 *list = s_list[warp];
    unsigned long long att = 0, written = 0, changed = 0, draws_total = 0;
    bool ok = true;
    constexpr int kPerSegment = kSegment / US;
    const int64_t units = 6 + segs * kPerSegment;
    // two units per ticket on large frames (the ticket counter is one address),
    // one on small ones
    const int grab = units > 8 * (int64_t)gridDim.x * kApplyWarps ? 2 : 1;
    int64_t unit = 0;
    for (int left = 0;; --left, ++unit) {
        if (left == 0) {
            uint32_t ticket = 0;
            if (lane == 0) ticket = atomicAdd(&ctr->apply_next, 1u);
            unit = (int64_t)__shfl_sync(0xFFFFFFFFu, ticket, 0) * grab;
            left = grab;
        }
        if (unit >= units) break;
        if (unit < 6) {  // counts of a startup row
            uint32_t a = 0, fixed = 0, amb = 0;
            const uint8_t *row = meta + unit * w;
#pragma unroll 4
            for (int x = lane; x < w; x += 32) {
                const uint32_t m = row[x];
                const uint32_t k = packed_word(m);
                a += m >> 7;
                fixed += k >> 16;
                amb += k & 0xFFFFu;
            }
            a = __reduce_add_sync(0xFFFFFFFFu, a);
            fixed = __reduce_add_sync(0xFFFFFFFFu, fixed);
            amb = __reduce_add_sync(0xFFFFFFFFu, amb);
            if (lane == 0) {
                ctr->su_attempted[unit] = a;
                ctr->su_base[unit] = fixed;
                ctr->su_amb[unit] = amb;
            }
            continue;
        }
        const int64_t seg = (unit - 6) / kPerSegment;
        const int part = (int)((unit - 6) % kPerSegment);
        const int64_t first = seg * kSegment + part * US;
        if (first >= sites) continue;
        // the state at the segment's first draw
        const uint32_t seg_a = seg_amb[seg], seg_p = seg_base[seg];
        // ---- meta: the segment's sites before the unit, this lane's 8 sites ---
        const UnitMeta um = unit_meta<US>(meta, sites, seg, part);
        const uint32_t *m2 = um.word;
        const int64_t mine = first + lane * 8;
        uint32_t sum = 0;
        // attempted public sites of the lane (bit i: site i)
        const int pub = (int)(su - mine < 0 ? 0 : (su - mine > 8 ? 8 : su - mine));
        uint32_t bits = 0;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            sum += packed_word(m2[q]);
            const uint32_t hi = (m2[q] >> 7) & 0x01010101u;
            bits |= ((hi * 0x01020408u) >> 24 & 0xFu) << (4 * q);
        }
        bits &= 0xFFu << pub & 0xFFu;
        const uint32_t listed = __popc(bits);
        // fixed << 16 | RNG-dependent fits (at most 6144 and 3072 a segment)
        uint32_t inc = sum, slot = listed;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            const uint32_t z = __shfl_up_sync(0xFFFFFFFFu, slot, o);
            if (lane >= o) {
                inc += y;
                slot += z;
            }
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, slot, 31);
        uint32_t run = __reduce_add_sync(0xFFFFFFFFu, um.ahead) + inc - sum;
        slot -= listed;
        __syncwarp();  // the previous list is consumed
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t m = (m2[i >> 2] >> (8 * (i & 3))) & 0xFFu;
            if ((bits >> i) & 1u) {
                list[slot] = make_uint2((uint32_t)(part * US + lane * 8 + i) | (m << 16),
                                        (run >> 16) | (run << 16));
                ++slot;
            }
            run += packed_word(m);
        }
        // ---- sites that were not attempted: identity emits -------------------
#pragma unroll
        for (int r = 0; r < US / 32; ++r) {
            const int64_t site = first + 32 * r + lane;
            // the bits of site's lane say whether it was attempted
            const uint32_t b = __shfl_sync(0xFFFFFFFFu, bits, 4 * r + (lane >> 3));
            if (site >= su && site < sites && !((b >> (lane & 7)) & 1u)) {
                const int64_t pixel = site - su;
                const uint2 raw = reinterpret_cast<const uint2 *>(rgbi)[pixel];
                uint16_t *o = rgb_out + 3 * pixel;
                o[0] = __ldg(ident + (raw.x & 0xFFFFu));
                o[1] = __ldg(ident + (raw.x >> 16));
                o[2] = __ldg(ident + (raw.y & 0xFFFFu));
                if (changed_out) changed_out[pixel] = 0;
            }
        }
        if (total == 0) continue;
        const uint32_t seg_e = extra_before(extra, seg_a, capacity);
        uint32_t seg_t = s0 << 8;
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // states repeat after 2^24 draws
            const Affine f = g_jump[j][((seg_p + seg_e) >> (6 * j)) & 63u];
            seg_t = f.a * seg_t + f.c;
        }
        __syncwarp();  // the list is complete
        // ---- attempted sites, densely ------------------------------------------
        for (uint32_t k = lane; k < total; k += 32) {
            const uint2 entry = list[k];
            const int64_t site = seg * kSegment + (entry.x & 0xFFFFu);
            const uint32_t pixel = (uint32_t)(site - su);  // H*W < 2^31
            const uint2 raw = reinterpret_cast<const uint2 *>(rgbi)[pixel];
            const uint32_t lanes[3] = {raw.x & 0xFFFFu, raw.x >> 16, raw.y & 0xFFFFu};
            uint16_t e0[3];
            float orig[3];
            double c3[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                c3[c] = cand[3 * site + c];
                e0[c] = __ldg(ident + lanes[c]);
                orig[c] = __ldg(lut + lanes[c]);
            }
            // the walk's bits of this site's RNG-dependent channels, and the
            // extra draws before them
            const uint8_t mi = (uint8_t)(entry.x >> 16);
            const uint32_t a = (uint32_t)min((int64_t)(seg_a + (entry.y >> 16)), capacity);
            const uint32_t sh = a & 31u;
            const uint2 words = __ldg(reinterpret_cast<const uint2 *>(extra) + (a >> 5));
            uint32_t redraw = words.y >> sh;
            if (sh + (uint32_t)meta_amb(mi) > 32u)
                redraw |= __ldg(&extra[(a >> 5) + 1].bits) << (32u - sh);
            const uint32_t n = (entry.y & 0xFFFFu) + words.x +
                               (uint32_t)__popc(words.y & ((1u << sh) - 1u)) - seg_e;
            const Affine f0 = s_jump[0][n & 127u], f1 = s_jump[1][(n >> 7) & 127u];
            uint32_t state = (f1.a * (f0.a * seg_t + f0.c) + f1.c) >> 8;
            const bool floor_enabled =
                p.driver_gate_primary || stages[pixel / (uint32_t)w + 6].gate_secondary;
            const WrittenSite out =
                write_site(c3, orig, floor_enabled, p.dither_scales, dc, mi, redraw, state);
            // (a list past its capacity is run again with a longer one)
            if (!out.agrees && (int64_t)(seg_a + (entry.y >> 16)) + meta_amb(mi) <= capacity)
                raise_error(err, FX_ERR_INTERNAL);
            draws_total += out.draws;
            bool wrote = false, differs = false;
            uint16_t *o = rgb_out + 3 * (int64_t)pixel;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                uint16_t e = e0[c];
                if (!out.kept[c]) {
                    if (!isfinite(out.value[c])) ok = false;
                    else e = emit_index(emit_index_of(out.value[c]), hi, lo);
                    wrote |= !(out.value[c] == orig[c]);
                }
                differs |= e != e0[c];
                o[c] = e;
            }
            att += 1;
            written += wrote;
            changed += differs;
            if (changed_out) changed_out[pixel] = differs ? 1 : 0;
        }
    }
    if (!ok) raise_error(err, FX_ERR_NONFINITE_WORK);
    // the four counters in one reduction: warps, then thread 0
    unsigned long long v4[4] = {att, written, changed, draws_total};
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v4[q] += __shfl_down_sync(0xFFFFFFFFu, v4[q], o);
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q) s_sums[warp][q] = v4[q];
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t4[4] = {0, 0, 0, 0};
        for (int wq = 0; wq < kApplyWarps; ++wq)
#pragma unroll
            for (int q = 0; q < 4; ++q) t4[q] += s_sums[wq][q];
        if (t4[0]) atomicAdd(&ctr->attempted, t4[0]);
        if (t4[1]) atomicAdd(&ctr->written, t4[1]);
        if (t4[2]) atomicAdd(&ctr->changed, t4[2]);
        if (t4[3]) atomicAdd(&ctr->public_advances, t4[3]);
        __threadfence();
        s_last = atomicAdd(&ctr->apply_done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    apply_final(seg_base, seg_amb, segs, extra, s0, ctr, walk, err, capacity);
}

// ---------------------------------------------------------------------------
// Launcher
// ---------------------------------------------------------------------------

cudaError_t launch_writer(const Geometry &g, const uint8_t *meta, const double *cand,
                          const uint16_t *rgbi, const float *lut, const uint32_t *high,
                          const uint32_t *low, const uint16_t *ident, const fx_stage *stages,
                          const fx_params &p,
                          uint32_t s0, const WriterBuffers &b, uint16_t *rgb_out,
                          uint8_t *changed_out, uint32_t *err, cudaStream_t stream,
                          const Marks &marks) {
    const int64_t segs = g.segments;
    DevCounters *ctr = reinterpret_cast<DevCounters *>(b.counters);  // cleared, as b.walk_zero
    cudaError_t e = launch_gate(b.cancel, err, stream);
    if (e != cudaSuccess) return e;
    // the chain and the walk are latency-bound: launched with b.priority, so
    // that with several frames in flight their blocks are dispatched ahead
    // of other frames' stencil and apply blocks, which fill the SMs they
    // leave idle
    const int pr = b.priority;
    const unsigned seg_blocks = (unsigned)((segs + kSegWarps - 1) / kSegWarps);
    e = launch_chained(k_seg_sums, dim3(seg_blocks), dim3(kSegWarps * 32), 0, stream, pr, meta,
                    g.sites, segs, b.seg_raw, b.seg_base, b.seg_amb, ctr, err);
    if (e != cudaSuccess) return e;
    const uint32_t *n_amb = b.seg_amb + segs;
    const int us = unit_sites(segs, g_coef_blocks * kCoefWarps);
    const int64_t unit_blocks = (segs * (kSegment / us) + kCoefWarps - 1) / kCoefWarps;
    e = launch_chained(us == 64 ? k_coef<64> : k_coef<kUnitSites>,
                    dim3((unsigned)std::min<int64_t>(unit_blocks, g_coef_blocks)),
                    dim3(kCoefWarps * 32), 0, stream, pr, b.entries, b.second, b.capacity, meta,
                    g.sites, segs, b.seg_raw, b.seg_base, b.seg_amb, cand, g.w, rgbi, lut, p,
                    b.chunk_two, b.chunk_stat, ctr, err);
    if (e != cudaSuccess) return e;
    marks.mark(5, stream);
    e = launch_gate(b.cancel, err, stream);
    if (e != cudaSuccess) return e;
    e = launch_walk(b.entries, b.second, n_amb, b.capacity, s0, b.walk_scratch, b.walk_zero,
                    b.widest_wave, b.per_wave, b.parallel_walk, b.window_sigmas, b.chunk_two, b.chunk_stat,
                    b.extra, err, stream, pr);
    if (e != cudaSuccess) return e;
    marks.mark(6, stream);
    e = launch_gate(b.cancel, err, stream);
    if (e != cudaSuccess) return e;
    const int64_t apply_blocks =
        (segs * (kSegment / us) + 6 + kApplyWarps - 1) / kApplyWarps;
    e = launch_chained(us == 64 ? k_apply<64> : k_apply<kUnitSites>,
                       dim3((unsigned)std::min<int64_t>(apply_blocks, g_apply_blocks)),
                       dim3(kApplyWarps * 32), 0, stream, 0, meta, cand, g.sites, g.w, rgbi, lut,
                       high, low, ident, stages, p, b.seg_base, b.seg_amb, b.extra, s0 & kLcgMask,
                       rgb_out, changed_out, ctr,
                       reinterpret_cast<const WalkState *>(b.walk_zero), err, b.capacity);
    if (e != cudaSuccess) return e;
    marks.mark(7, stream);
    return cudaGetLastError();
}

// One thread: a cancel request seen here stops every later kernel of the pass.
__global__ void k_gate(const volatile uint32_t *cancel, uint32_t *err) {
    if (*cancel && err[1] == 0u) {
        err[1] = 1u;
        atomicCAS(err, 0u, (uint32_t)FX_ERR_CANCELLED);
    }
}

cudaError_t launch_gate(const uint32_t *cancel, uint32_t *err, cudaStream_t stream) {
    if (!cancel) return cudaSuccess;
    k_gate<<<1, 1, 0, stream>>>(cancel, err);
    return cudaGetLastError();
}

size_t dev_counters_bytes() { return sizeof(DevCounters); }

void counters_to_host(const void *dev_copy, fx_counters *out) {
    const DevCounters &c = *reinterpret_cast<const DevCounters *>(dev_copy);
    out->attempted = (int64_t)c.attempted;
    out->written = (int64_t)c.written;
    out->public_advances = (int64_t)c.public_advances;
    out->changed = (int64_t)c.changed;
    out->final_state = c.final_state;
    out->startup_final_state = c.su_final_state;
    for (int k = 0; k < 6; ++k) {
        out->startup_attempted[k] = (int64_t)c.su_attempted[k];
        out->startup_advances[k] = (int64_t)c.su_advances[k];
    }
    out->rng_dependent = (int64_t)c.n_amb;
    out->walk_fallbacks = (int64_t)c.walk_fallbacks;
    out->walk_candidate_steps = (int64_t)c.walk_stats[0];
    out->walk_candidates = (int64_t)c.walk_stats[1];
    out->walk_survivors = (int64_t)c.walk_stats[2];
    out->walk_packed_segments = (int64_t)c.walk_packed;
    out->capacity_reruns = 0;  // set by the host when the pass runs again
}

uint32_t counters_n_amb(const void *dev_copy) {
    return reinterpret_cast<const DevCounters *>(dev_copy)->n_amb;
}

}  // namespace fx
