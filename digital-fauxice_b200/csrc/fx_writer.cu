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
//   2. k_seg_sums + k_seg_scan: exclusive prefix of fixed draws and of
//      RNG-dependent channels along the chain (startup sites, then public
//      sites in row-major order).
//   3. k_amb: for each RNG-dependent channel, the set of first-draw states
//      that copy the original, as at most two state intervals (found by
//      binary search on the exact binary64 expressions, which are monotone
//      in the state).
//   4. k_coef: the interval test of each such channel as a function of the
//      extra draws before it (the channel's fixed draws folded into an affine
//      LCG jump).
//   5. the walk (fx_walk.cu) visits only the RNG-dependent channels: a
//      multiply-add, a test and a conditional LCG step per channel,
//      parallelised over segments by speculation.  Output: the running count of extra draws.
//   6. k_apply: every public site computes its values from its own start
//      state g^(fixed + extra before it)(s0), in parallel, and emits public
//      RGB16 with the counters.
#include <algorithm>

#include "fx_internal.cuh"

namespace fx {

struct DevCounters {
    unsigned long long attempted, written, public_advances, changed;
    unsigned long long su_attempted[6], su_advances[6];
    unsigned long long public_base, public_amb;
    uint32_t final_state, su_final_state;
    uint32_t startup_base, startup_amb, startup_extra;
    uint32_t n_amb;
    uint32_t walk_fallbacks;
    uint32_t walk_packed;              // written together with walk_fallbacks
    unsigned long long walk_stats[3];  // candidate steps, window sum, survivor sum
    uint32_t su_base[6], su_amb[6];    // per startup row, for the last block's chain
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

__device__ __forceinline__ uint32_t packed_site(uint8_t m) {
    return ((uint32_t)meta_base(m) << 16) | (uint32_t)meta_amb(m);
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
// one block per group.  The group sums go where k_seg_scan writes the
// groups' prefixes.
__global__ void __launch_bounds__(kSegWarps * 32)
    k_seg_sums(const uint8_t *__restrict__ meta, int64_t sites, int64_t segs,
               uint32_t *__restrict__ raw, const uint32_t *__restrict__ err) {
    __shared__ uint32_t s_warp[kSegWarps];
    if (pass_stopped(err)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
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
                if (first + i < sites) packed += packed_site(meta[first + i]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) packed += __shfl_xor_sync(0xFFFFFFFFu, packed, o);
    if (lane == 0) {
        if (seg < segs) v.seg[seg] = packed;
        s_warp[warp] = packed;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t g = 0;  // at most 8 x 6144 fixed draws and 8 x 3072 channels
#pragma unroll
        for (int k = 0; k < kSegWarps; ++k) g += s_warp[k];
        v.grp_base[blockIdx.x] = g;
    }
}

// Exclusive scan of the groups' sums into the groups' prefixes; seg_base[n]
// and seg_amb[n] get the totals (n segments).  One block of 1024 threads,
// over tiles of 4096 groups (a native frame has 2.8 k): a tile is loaded
// coalesced into shared memory, each thread scans four neighbouring groups,
// and one block scan of (fixed << 32 | RNG-dependent) pairs gives the
// threads' offsets (the RNG-dependent total stays below 2^32: at most three
// per site).  k_amb adds a segment's offset inside its group.
__global__ void __launch_bounds__(1024)
    k_seg_scan(uint32_t *__restrict__ raw, int64_t n, uint32_t *__restrict__ seg_base,
               uint32_t *__restrict__ seg_amb, const uint32_t *__restrict__ err) {
    constexpr int kPerThread = 4, kTile = 1024 * kPerThread;
    __shared__ uint32_t tb[kTile], ta[kTile];
    __shared__ unsigned long long ws[32];
    if (pass_stopped(err)) return;
    const SegRaw v = seg_raw_view(raw, n);
    const int64_t groups = (n + kSegGroup - 1) / kSegGroup;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long carry = 0;
    for (int64_t t0 = 0; t0 < groups; t0 += kTile) {
        for (int j = tid; j < kTile; j += 1024) {
            const int64_t i = t0 + j;
            const uint32_t g = i < groups ? v.grp_base[i] : 0u;
            tb[j] = g >> 16;
            ta[j] = g & 0xFFFFu;
        }
        __syncthreads();
        unsigned long long mine = 0;
#pragma unroll
        for (int k = 0; k < kPerThread; ++k)
            mine += ((unsigned long long)tb[kPerThread * tid + k] << 32) | ta[kPerThread * tid + k];
        unsigned long long x = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        if (warp == 0) {
            unsigned long long w = ws[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, w, o);
                if (lane >= o) w += y;
            }
            ws[lane] = w;
        }
        __syncthreads();
        unsigned long long run = carry + (warp ? ws[warp - 1] : 0ull) + x - mine;
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
            const int j = kPerThread * tid + k;
            const unsigned long long val = ((unsigned long long)tb[j] << 32) | ta[j];
            tb[j] = (uint32_t)(run >> 32);
            ta[j] = (uint32_t)run;
            run += val;
        }
        carry += ws[31];
        __syncthreads();
        for (int j = tid; j < kTile; j += 1024) {
            const int64_t i = t0 + j;
            if (i < groups) {
                v.grp_base[i] = tb[j];
                v.grp_amb[i] = ta[j];
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        seg_base[n] = (uint32_t)(carry >> 32);
        seg_amb[n] = (uint32_t)carry;
    }
}

struct SiteInfo {
    float orig[3];
    bool floor_enabled;
};

__device__ __forceinline__ SiteInfo site_info(int64_t site, int w, const uint16_t *rgbi,
                                              const float *lut, const fx_stage *stages,
                                              const fx_params &p) {
    SiteInfo si;
    const int64_t su = 6 * (int64_t)w;
    int64_t pixel;
    int stage_index;
    if (site < su) {
        pixel = site % w;  // startup originals are row 0 (startup.py:327-336)
        stage_index = (int)(site / w);
    } else {
        pixel = site - su;
        stage_index = (int)(pixel / w) + 6;
    }
    const uint2 raw = reinterpret_cast<const uint2 *>(rgbi)[pixel];
    si.orig[0] = __ldg(lut + (raw.x & 0xFFFFu));
    si.orig[1] = __ldg(lut + (raw.x >> 16));
    si.orig[2] = __ldg(lut + (raw.y & 0xFFFFu));
    si.floor_enabled = p.driver_gate_primary || stages[stage_index].gate_secondary;
    return si;
}

// Affine jump tables: g_jump[j][d] = g^(d * 64^j) in T space.  States repeat
// after 2^24 draws, so the low four base-64 digits of a draw count give its
// map on states.
constexpr int kJumpDigits = 4;
__device__ Affine g_jump[kJumpDigits][64];

// ---------------------------------------------------------------------------
// Copy intervals of one RNG-dependent channel
// ---------------------------------------------------------------------------

struct ChannelView {
    double cand, cd, env, od;
    float span;
    DitherConst dc;
    __device__ double raw(uint32_t s1) const { return dither_raw_delta(cd, env, span, s1); }
    __device__ bool low_ok(uint32_t s1) const { return dc.low < cd + raw(s1); }
    __device__ bool high_ok(uint32_t s1) const { return cd + raw(s1) < dc.high; }
    __device__ bool floor_test(uint32_t s1) const { return cand + raw(s1) <= od; }
    __device__ bool copies(uint32_t s1) const {
        const double d = raw(s1);
        const double changed = cd + d;
        const double eff = (dc.low < changed && changed < dc.high) ? d : 0.0;
        return cand + eff <= od;
    }
};

// First state where a monotone predicate differs from its value at 0
// (2^24 when it never does).  `guess` estimates that state; the search
// gallops from it to a bracket checked on the exact predicate and bisects
// inside, so the estimate changes only the cost, never the result.
template <class F>
__device__ __forceinline__ uint32_t switch_point(F pred, double guess) {
    const bool p0 = pred(0u);
    if (pred(kLcgMask) == p0) return kLcgMask + 1u;
    // invariant: pred(lo) == p0, pred(hi) != p0, lo < hi
    uint32_t lo = 0u, hi = kLcgMask;
    uint32_t x = kLcgMask / 2u;
    if (guess == guess) {  // not NaN
        const double top = (double)(kLcgMask - 1u);
        x = (uint32_t)(guess < 1.0 ? 1.0 : (guess > top ? top : guess));
    }
    uint32_t step = 1u;
    if (pred(x) == p0) {
        lo = x;
        while (hi - lo > 1u) {
            if (hi - lo <= step) break;
            const uint32_t y = lo + step;
            if (pred(y) == p0) {
                lo = y;
                step <<= 1;
            } else {
                hi = y;
                break;
            }
        }
    } else {
        hi = x;
        while (hi - lo > 1u) {
            if (hi - lo <= step) break;
            const uint32_t y = hi - step;
            if (pred(y) != p0) {
                hi = y;
                step <<= 1;
            } else {
                lo = y;
                break;
            }
        }
    }
    while (hi - lo > 1u) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (pred(mid) == p0) lo = mid;
        else hi = mid;
    }
    return hi;
}

// The state s1 at which base + raw(s1) would reach `target` if the delta
// were computed exactly (it is affine in s1): a starting point for
// switch_point.
__device__ __forceinline__ double crossing(const ChannelView &cv, double base, double target) {
    const double scale = cv.env * (double)cv.span;
    return ((target - base) / scale + 0.5) / kNormalization - 1.0;
}

// Copy set of one channel in T space: copy iff (T - l1) <= w1 or
// (T - l2) <= w2 (modulo 2^32); l = 0x80 marks an empty interval.
struct CopySet {
    uint32_t l1, w1, l2, w2;
};

__device__ void copy_intervals(const ChannelView &cv, CopySet &e, uint32_t *err) {
    uint32_t b[3] = {
        switch_point([&](uint32_t s) { return cv.low_ok(s); }, crossing(cv, cv.cd, cv.dc.low)),
        switch_point([&](uint32_t s) { return cv.high_ok(s); }, crossing(cv, cv.cd, cv.dc.high)),
        switch_point([&](uint32_t s) { return cv.floor_test(s); }, crossing(cv, cv.cand, cv.od))};
    // sort the three breakpoints
    if (b[0] > b[1]) { const uint32_t t = b[0]; b[0] = b[1]; b[1] = t; }
    if (b[1] > b[2]) { const uint32_t t = b[1]; b[1] = b[2]; b[2] = t; }
    if (b[0] > b[1]) { const uint32_t t = b[0]; b[0] = b[1]; b[1] = t; }
    uint32_t starts[4];
    int n = 0;
    starts[n++] = 0u;
    for (int i = 0; i < 3; ++i)
        if (b[i] <= kLcgMask && b[i] != starts[n - 1]) starts[n++] = b[i];
    uint32_t lo[2], hi[2];
    int intervals = 0;
    bool open = false;
    for (int i = 0; i < n; ++i) {
        const uint32_t first = starts[i];
        const uint32_t last = (i + 1 < n) ? starts[i + 1] - 1u : kLcgMask;
        const bool c = cv.copies(first);
        if (c) {
            if (open) {
                hi[intervals - 1] = last;
            } else {
                if (intervals == 2) { raise_error(err, FX_ERR_INTERNAL); return; }
                lo[intervals] = first;
                hi[intervals] = last;
                ++intervals;
                open = true;
            }
        } else {
            open = false;
        }
    }
    // empty interval: l = 0x80 can never match a T value (low byte zero)
    e.l1 = 0x80u; e.w1 = 0u; e.l2 = 0x80u; e.w2 = 0u;
    if (intervals == 2 && lo[0] == 0u && hi[1] == kLcgMask) {
        // [0, hi0] and [lo1, 2^24 - 1] meet across the wrap: one cyclic
        // interval from lo1 (the test (T - l) <= w wraps modulo 2^32)
        e.l1 = lo[1] << 8;
        e.w1 = (hi[0] - lo[1]) << 8;
        return;
    }
    if (intervals >= 1) { e.l1 = lo[0] << 8; e.w1 = (hi[0] - lo[0]) << 8; }
    if (intervals == 2) { e.l2 = lo[1] << 8; e.w2 = (hi[1] - lo[1]) << 8; }
}

// Lists every RNG-dependent channel in chain order: entry a gets its site
// (site_of[a], a compact array so the writes coalesce) and its draw
// position; k_coef fills in the intervals and jumps.  One warp per segment,
// in 16 rounds of 64 consecutive sites, two neighbouring sites per lane (all
// the segment's meta loads issued first); a round's offsets come from one
// warp scan, so a round's entries are written by consecutive lanes to
// consecutive list positions.
__global__ void __launch_bounds__(kSegWarps * 32)
    k_amb(const uint8_t *__restrict__ meta, int64_t sites, int64_t segs,
          uint32_t *__restrict__ raw, uint32_t *__restrict__ seg_base,
          uint32_t *__restrict__ seg_amb, uint32_t *__restrict__ site_of,
          uint32_t *__restrict__ pos_out, int64_t capacity, const uint32_t *__restrict__ err) {
    if (pass_stopped(err)) return;
    const int lane = threadIdx.x & 31;
    const int64_t seg = (int64_t)blockIdx.x * kSegWarps + (threadIdx.x >> 5);
    if (seg >= segs) return;
    const int64_t first = seg * kSegment + 2 * lane;  // sites first + 64 r, + 1
    uint32_t m2[16];  // the two meta bytes of round r
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int64_t s0 = first + 64 * r;
        if (s0 + 1 < sites)
            m2[r] = *reinterpret_cast<const uint16_t *>(meta + s0);  // even offset
        else
            m2[r] = s0 < sites ? meta[s0] : 0u;
    }
    // the segment's prefix: its group's, plus the segments before it in the
    // group (fewer than eight, so the packed halves cannot carry); written
    // for the kernels after the walk
    const SegRaw v = seg_raw_view(raw, segs);
    const int64_t grp = seg / kSegGroup, k0 = grp * kSegGroup;
    uint32_t before = (k0 + lane < seg) ? v.seg[k0 + lane] : 0u;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
    before = __shfl_sync(0xFFFFFFFFu, before, 0);
    uint32_t P = v.grp_base[grp] + (before >> 16), A = v.grp_amb[grp] + (before & 0xFFFFu);
    if (lane == 0) {
        seg_base[seg] = P;
        seg_amb[seg] = A;
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const uint8_t mb[2] = {(uint8_t)(m2[r] & 0xFFu), (uint8_t)(m2[r] >> 8)};
        const uint32_t x0 = packed_site(mb[0]), x = x0 + packed_site(mb[1]);
        uint32_t inc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += y;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, inc, 31);
        if (x & 0xFFFFu) {
            const uint32_t ex = inc - x;
            uint32_t pos = P + (ex >> 16), a = A + (ex & 0xFFFFu);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint8_t mi = mb[h];
                pos = P + ((ex + (h ? x0 : 0u)) >> 16);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int code = meta_code(mi, c);
                    if (code == 3) {
                        if ((int64_t)a < capacity) {
                            site_of[a] = (uint32_t)(first + 64 * r + h);
                            pos_out[a] = pos;
                        }
                        ++a;
                        pos += 1u;
                    } else {
                        pos += (uint32_t)code;
                    }
                }
            }
        }
        P += total >> 16;
        A += total & 0xFFFFu;
    }
}

// k_coef's inputs of one entry, gathered in two dependent steps: the list
// (coalesced) gives the site, the site gives its meta, pixel and candidates.
struct CoefList {
    uint32_t site, pos;  // pos: fixed draws before the channel
    int k;               // this entry is the k-th of its site
};
struct CoefSite {
    uint8_t meta;
    uint2 raw;
    double cand[3];
};

__device__ __forceinline__ CoefList coef_list(const uint32_t *__restrict__ site_of,
                                              const uint32_t *__restrict__ pos, uint32_t i,
                                              uint32_t n) {
    CoefList l{0u, 0u, 0};
    if (i >= n) return l;
    l.site = site_of[i];
    // a site's RNG-dependent channels are listed in channel order
    l.k = (i >= 1 && site_of[i - 1] == l.site) ? ((i >= 2 && site_of[i - 2] == l.site) ? 2 : 1)
                                                : 0;
    l.pos = pos[i];
    return l;
}

__device__ __forceinline__ CoefSite coef_site(const CoefList &l, bool live, int64_t su, int w,
                                              const uint8_t *__restrict__ meta,
                                              const double *__restrict__ cand,
                                              const uint16_t *__restrict__ rgbi) {
    CoefSite c{};
    if (!live) return c;
    const int64_t site = l.site;
    const int64_t pixel = site < su ? site % w : site - su;
    c.meta = meta[site];
    c.raw = reinterpret_cast<const uint2 *>(rgbi)[pixel];
    c.cand[0] = cand[3 * site];
    c.cand[1] = cand[3 * site + 1];
    c.cand[2] = cand[3 * site + 2];
    return c;
}

// Copy intervals and state map of every RNG-dependent channel.  A thread's
// entries i, i + stride, ... run through a three-stage software pipeline:
// while entry i's interval search computes, the site of entry i + 2 stride
// and the meta, pixel and candidates of entry i + stride are in flight, so
// the dependent gathers overlap the arithmetic instead of stalling it.
__global__ void __launch_bounds__(256, 4) k_coef(AmbEntry *__restrict__ entries, SecondInterval *__restrict__ second,
                       const uint32_t *__restrict__ pos,
                       const uint32_t *__restrict__ n_amb_ptr, int64_t capacity,
                       const uint32_t *__restrict__ site_of, const uint8_t *__restrict__ meta,
                       const double *__restrict__ cand, int w, const uint16_t *__restrict__ rgbi,
                       const float *__restrict__ lut, fx_params p, uint32_t *err,
                       uint8_t *__restrict__ chunk_two, ChunkStat *__restrict__ chunk_stat) {
    // powers of the LCG step: states repeat after 2^24 draws, so the four
    // low base-64 digits of a draw count give its map on states
    __shared__ Affine s_jump[4][64];
    if (pass_stopped(err)) return;
    for (int j = threadIdx.x; j < 4 * 64; j += blockDim.x) s_jump[j / 64][j % 64] = g_jump[j / 64][j % 64];
    __syncthreads();
    const uint32_t n = (uint32_t)min((int64_t)*n_amb_ptr, capacity);
    const DitherConst dc = dither_const(p);
    const int64_t su = 6 * (int64_t)w;
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    CoefList l0 = coef_list(site_of, pos, i, n);
    CoefSite s0 = coef_site(l0, i < n, su, w, meta, cand, rgbi);
    CoefList l1 = coef_list(site_of, pos, i + stride, n);
    for (; i < n; i += stride) {
        const uint32_t i1 = i + stride, i2 = i1 + stride;
        const CoefSite s1 = coef_site(l1, i1 < n && i1 > i, su, w, meta, cand, rgbi);
        const CoefList l2 = coef_list(site_of, pos, i2 > i1 ? i2 : n, n);
        const uint8_t mi = s0.meta;
        int c = 0;
        for (int seen = 0; c < 3; ++c)
            if (meta_code(mi, c) == 3 && seen++ == l0.k) break;
        const uint2 raw = s0.raw;
        const uint32_t lane = c == 0 ? (raw.x & 0xFFFFu) : (c == 1 ? (raw.x >> 16) : (raw.y & 0xFFFFu));
        ChannelView cv;
        cv.cand = c == 0 ? s0.cand[0] : (c == 1 ? s0.cand[1] : s0.cand[2]);
        cv.cd = (double)(float)cv.cand;
        cv.dc = dc;
        cv.env = ((dc.high - cv.cd) * (cv.cd - dc.low)) * dc.coefficient;
        cv.span = (float)((double)p.dither_scales[c] * cv.cd);
        cv.od = (double)__ldg(lut + lane);
        CopySet e;
        copy_intervals(cv, e, err);
        // a chunk of walk channels with a two-interval entry steps with both
        // interval tests (every other chunk with one)
        if (e.l2 != 0x80u) chunk_two[i / kWalkChunk] = 1;
        // the walk's prediction: m copying states of 2^24 (an extra draw with
        // probability p = 1 - m / 2^24), summed per chunk with the spread
        // p (1 - p).  A warp holds 32 consecutive entries of one chunk; the
        // lanes past the chain's end have left the loop.
        {
            uint32_t m = 0;
            if (e.l1 != 0x80u) m += (e.w1 >> 8) + 1u;
            if (e.l2 != 0x80u) m += (e.w2 >> 8) + 1u;
            const uint32_t q = (uint32_t)(((unsigned long long)m * ((1u << 24) - m)) >> 23);
            const uint32_t lane = threadIdx.x & 31, live = n - (i - lane);
            const uint32_t mask = live >= 32u ? 0xFFFFFFFFu : ((1u << live) - 1u);
            const uint32_t ms = __reduce_add_sync(mask, m >> 1), qs = __reduce_add_sync(mask, q);
            if (lane == 0) {
                atomicAdd(&chunk_stat[i / kWalkChunk].copy, ms);
                atomicAdd(&chunk_stat[i / kWalkChunk].spread, qs);
            }
        }
        // G^(pos + 1) less the first interval's start
        const uint32_t draws = l0.pos + 1u;
        Affine f = s_jump[0][draws & 63u];
#pragma unroll
        for (int j = 1; j < 4; ++j)
            f = affine_compose(s_jump[j][(draws >> (6 * j)) & 63u], f);
        entries[i] = AmbEntry{f.a, f.c - e.l1, e.w1, e.l2 != 0x80u ? 1u : 0u};
        if (e.l2 != 0x80u) second[i] = SecondInterval{e.l1 - e.l2, e.w2};
        l0 = l1;
        s0 = s1;
        l1 = l2;
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

constexpr int kApplyBlocksPerSM = 5;  // k_apply's resident blocks per SM
static int g_apply_blocks = kApplyBlocksPerSM * 148;

// Powers of the LCG step for short jumps: g_short[j][d] = g^(d * 128^j) in T
// space, so a jump below 2^14 draws is two lookups.
__device__ Affine g_short[2][128];

cudaError_t writer_init() {
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
        sms > 0)
        g_apply_blocks = kApplyBlocksPerSM * sms;
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

// Every warp takes units of 256 sites, a quarter of a chain segment, with no
// block barrier:
//   * the segment's meta bytes give the chain offsets before the unit and of
//     its sites, and the attempted sites are listed in the warp's shared
//     memory;
//   * the sites that were not attempted are emitted, one pixel per lane
//     (their output is the identity emit);
//   * the list is processed densely, one attempted site per lane, from its
//     own start state: the segment's, advanced by the draws inside it.
// A channel's classification and the walk's bit say which of its draws
// decides its value, so at most one is evaluated, and none where the original
// is copied.  The first six units are the startup rows' counts; the last block
// to finish chains the rows and writes the final state.
// Measured on a native frame with half its pixels attempted: 505 us as blocks
// of 256 threads with a block scan, four pixels per thread, both draws of
// every channel and a six-digit jump per site (564 warp instructions per 32
// pixels, 357 now); 332 us so.  The gathers' L1 decides the rest: with the
// samples staged in shared memory five blocks took 505 us and six 866, with a
// 128 KB emit table instead of the two factor tables 420.
constexpr int kApplyWarps = 8;
constexpr int kApplySites = 256;  // sites of a unit
static_assert(kSegment == 1024 && kApplySites == 32 * 8, "32 and 8 meta bytes per lane");

__device__ void apply_final(const uint32_t *seg_base, const uint32_t *seg_amb, int64_t segments,
                            const ExtraWord *extra, uint32_t s0, DevCounters *ctr, uint32_t *err,
                            int64_t capacity) {
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
    ctr->final_state = lcg_jump(s0, (uint64_t)p_total + e_total);
    const unsigned long long expect =
        (unsigned long long)(p_total - p_run) + (e_total - e_su);
    if ((int64_t)a_total <= capacity && expect != __ldcg(&ctr->public_advances))
        raise_error(err, FX_ERR_INTERNAL);
}

__global__ void __launch_bounds__(kApplyWarps * 32, kApplyBlocksPerSM)
    k_apply(const uint8_t *__restrict__ meta, const double *__restrict__ cand, int64_t sites,
            int w, const uint16_t *__restrict__ rgbi, const float *__restrict__ lut,
            const uint32_t *__restrict__ g_high, const uint32_t *__restrict__ g_low,
            const uint16_t *__restrict__ ident, const fx_stage *__restrict__ stages, fx_params p,
            const uint32_t *__restrict__ seg_base, const uint32_t *__restrict__ seg_amb,
            const ExtraWord *__restrict__ extra, uint32_t s0, uint16_t *__restrict__ rgb_out,
            uint8_t *__restrict__ changed_out, DevCounters *ctr, uint32_t *err,
            int64_t capacity) {
    __shared__ Affine s_jump[2][128];
    __shared__ uint32_t hi[256], lo[256];  // emit factors
    // attempted sites: x = site in the segment | meta << 16, y = fixed draws
    // before it in the segment | RNG-dependent channels before it << 16
    __shared__ uint2 s_list[kApplyWarps][kApplySites];
    __shared__ unsigned long long s_sums[kApplyWarps][4];
    __shared__ bool s_last;
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
    const int64_t units = 6 + segs * (kSegment / kApplySites);
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
        const int64_t seg = (unit - 6) / (kSegment / kApplySites);
        const int part = (int)((unit - 6) % (kSegment / kApplySites));
        const int64_t first = seg * kSegment + part * kApplySites;
        if (first >= sites) continue;
        // the state at the segment's first draw
        const uint32_t seg_a = seg_amb[seg], seg_p = seg_base[seg];
        // ---- meta: the segment's sites before the unit, this lane's 8 sites ---
        uint32_t sum = 0, ahead = 0;
        uint32_t m2[2] = {0u, 0u};
        const int64_t mine = first + lane * 8, far = seg * kSegment + lane * 32;
        if (first + kApplySites <= sites) {
            if (lane < part * (kApplySites / 32)) {
                const uint4 *q = reinterpret_cast<const uint4 *>(meta + far);
                const uint4 u = q[0], v = q[1];
                ahead = packed_word(u.x) + packed_word(u.y) + packed_word(u.z) +
                        packed_word(u.w) + packed_word(v.x) + packed_word(v.y) +
                        packed_word(v.z) + packed_word(v.w);
            }
            const uint2 v = *reinterpret_cast<const uint2 *>(meta + mine);
            m2[0] = v.x;
            m2[1] = v.y;
        } else {  // the chain's last unit
            if (lane < part * (kApplySites / 32))
                for (int i = 0; i < 32; ++i) ahead += packed_word(meta[far + i]);
            for (int i = 0; i < 8; ++i)
                if (mine + i < sites) m2[i >> 2] |= (uint32_t)meta[mine + i] << (8 * (i & 3));
        }
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
        uint32_t run = __reduce_add_sync(0xFFFFFFFFu, ahead) + inc - sum;
        slot -= listed;
        __syncwarp();  // the previous list is consumed
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t m = (m2[i >> 2] >> (8 * (i & 3))) & 0xFFu;
            if ((bits >> i) & 1u) {
                list[slot] = make_uint2((uint32_t)(part * kApplySites + lane * 8 + i) | (m << 16),
                                        (run >> 16) | (run << 16));
                ++slot;
            }
            run += packed_word(m);
        }
        // ---- sites that were not attempted: identity emits -------------------
#pragma unroll
        for (int r = 0; r < 8; ++r) {
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
        // ---- attempted sites, densely: one round's loads are in flight while
        // the round before is computed ------------------------------------------
        struct Site {
            uint2 entry, raw, words;  // list entry, samples, extra draws
            double cand[3];
        };
        auto fetch = [&](uint32_t k) {
            Site q;
            if (k < total) {
                q.entry = list[k];
                const int64_t site = seg * kSegment + (q.entry.x & 0xFFFFu);
                q.raw = reinterpret_cast<const uint2 *>(rgbi)[site - su];
                const uint32_t a =
                    (uint32_t)min((int64_t)(seg_a + (q.entry.y >> 16)), capacity);
                q.words = __ldg(reinterpret_cast<const uint2 *>(extra) + (a >> 5));
#pragma unroll
                for (int c = 0; c < 3; ++c) q.cand[c] = cand[3 * site + c];
            }
            return q;
        };
        Site cur = fetch(lane);
        for (uint32_t k = lane; k < total; k += 32) {
            const Site q = cur;
            cur = fetch(k + 32);
            const uint8_t mi = (uint8_t)(q.entry.x >> 16);
            // H*W < 2^31
            const uint32_t pixel = (uint32_t)(seg * kSegment + (q.entry.x & 0xFFFFu) - su);
            const uint32_t lanes[3] = {q.raw.x & 0xFFFFu, q.raw.x >> 16, q.raw.y & 0xFFFFu};
            uint16_t e0[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) e0[c] = __ldg(ident + lanes[c]);
            // the walk's bits of this site's RNG-dependent channels, and the
            // extra draws before them
            const uint32_t a = (uint32_t)min((int64_t)(seg_a + (q.entry.y >> 16)), capacity);
            const uint32_t sh = a & 31u;
            uint32_t redraw = q.words.y >> sh;
            if (sh + (uint32_t)meta_amb(mi) > 32u)
                redraw |= __ldg(&extra[(a >> 5) + 1].bits) << (32u - sh);
            const uint32_t n = (q.entry.y & 0xFFFFu) + q.words.x +
                               (uint32_t)__popc(q.words.y & ((1u << sh) - 1u)) - seg_e;
            const Affine f0 = s_jump[0][n & 127u], f1 = s_jump[1][(n >> 7) & 127u];
            uint32_t state = (f1.a * (f0.a * seg_t + f0.c) + f1.c) >> 8;
            const bool floor_enabled =
                p.driver_gate_primary || stages[pixel / (uint32_t)w + 6].gate_secondary;
            bool valid = true;
            if ((mi & 0x3Fu) == 0u)  // no draws: all channels outside the bounds, or invalid
#pragma unroll
                for (int c = 0; c < 3; ++c) valid &= isfinite(q.cand[c]) && q.cand[c] > 0.0;
            bool wrote = false, differs = false;
            uint16_t *o = rgb_out + 3 * (int64_t)pixel;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                int code = meta_code(mi, c);
                if (code == 3) {  // one draw and a copy, or two
                    code = (redraw & 1u) ? 2 : 1;
                    redraw >>= 1;
                }
                // the draw that decides the value (the first draw copies the
                // original where the floor gate is on)
                if (code >= 1) state = (125u * state + 1u) & kLcgMask;
                if (code == 2) state = (125u * state + 1u) & kLcgMask;
                draws_total += (uint32_t)code;
                uint16_t e = e0[c];
                if (valid && !(code == 1 && floor_enabled)) {
                    const double c3 = q.cand[c];
                    float v;
                    bool copied = false;
                    if (code == 0) {
                        const float orig = __ldg(lut + lanes[c]);
                        copied = floor_enabled && c3 <= (double)orig;
                        v = (float)c3;
                    } else {
                        const DitherChannel ch = dither_channel(c3, p.dither_scales[c], dc);
                        const double d = dither_raw_delta(ch.cand, ch.envelope, ch.span, state);
                        const double moved = ch.cand + d;
                        v = (float)(c3 + ((dc.low < moved && moved < dc.high) ? d : 0.0));
                    }
                    if (!copied) {
                        if (!isfinite(v)) ok = false;
                        else e = emit_index(emit_index_of(v), hi, lo);
                        // an output that differs was written; one that does not
                        // may still come from another value
                        wrote |= e != e0[c] || !(v == __ldg(lut + lanes[c]));
                    }
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
    apply_final(seg_base, seg_amb, segs, extra, s0, ctr, err, capacity);
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
    DevCounters *ctr = reinterpret_cast<DevCounters *>(b.counters);
    cudaMemsetAsync(ctr, 0, sizeof(DevCounters), stream);
    cudaError_t e = launch_gate(b.cancel, err, stream);
    if (e != cudaSuccess) return e;
    // the chain and the walk are latency-bound: launched with b.priority, so
    // that with several frames in flight their blocks are dispatched ahead
    // of other frames' stencil and apply blocks, which fill the SMs they
    // leave idle
    const int pr = b.priority;
    const unsigned seg_blocks = (unsigned)((segs + kSegWarps - 1) / kSegWarps);
    e = launch_prio(k_seg_sums, dim3(seg_blocks), dim3(kSegWarps * 32), 0, stream, pr, meta,
                    g.sites, segs, b.seg_raw, err);
    if (e != cudaSuccess) return e;
    e = launch_prio(k_seg_scan, dim3(1), dim3(1024), 0, stream, pr, b.seg_raw, segs, b.seg_base,
                    b.seg_amb, err);
    if (e != cudaSuccess) return e;
    e = launch_prio(k_amb, dim3(seg_blocks), dim3(kSegWarps * 32), 0, stream, pr, meta, g.sites,
                    segs, b.seg_raw, b.seg_base, b.seg_amb, b.site_of, b.pos, b.capacity,
                    err);
    if (e != cudaSuccess) return e;
    const uint32_t *n_amb = b.seg_amb + segs;
    cudaMemsetAsync(b.chunk_two, 0, walk_chunks(b.capacity), stream);
    cudaMemsetAsync(b.chunk_stat, 0, walk_chunks(b.capacity) * sizeof(ChunkStat), stream);
    e = launch_prio(k_coef, dim3(1184), dim3(256), 0, stream, pr, b.entries, b.second, b.pos, n_amb,
                    b.capacity, b.site_of, meta, cand, g.w, rgbi, lut, p, err, b.chunk_two,
                    b.chunk_stat);
    if (e != cudaSuccess) return e;
    marks.mark(5, stream);
    e = launch_gate(b.cancel, err, stream);
    if (e != cudaSuccess) return e;
    e = launch_walk(b.entries, b.second, n_amb, b.capacity, s0, b.walk_scratch, b.per_wave,
                    b.parallel_walk, b.window_sigmas, b.chunk_two, b.chunk_stat, b.extra,
                    &ctr->walk_fallbacks, ctr->walk_stats, err, stream, pr);
    if (e != cudaSuccess) return e;
    marks.mark(6, stream);
    e = launch_gate(b.cancel, err, stream);
    if (e != cudaSuccess) return e;
    const int64_t apply_blocks =
        (segs * (kSegment / kApplySites) + 6 + kApplyWarps - 1) / kApplyWarps;
    k_apply<<<(unsigned)std::min<int64_t>(apply_blocks, g_apply_blocks), kApplyWarps * 32, 0,
              stream>>>(meta, cand, g.sites, g.w, rgbi, lut, high, low, ident, stages, p,
                        b.seg_base, b.seg_amb, b.extra, s0 & kLcgMask, rgb_out, changed_out, ctr,
                        err, b.capacity);
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
