// fx_route.cu -- device primitives of the at-floor routing census.
//
// The routing step downstream of the diagnostics (hybrid routing.py:447-682,
// route_at_floor_mask) measures the 8-connected components of the at-floor
// mask, routes the large ones, dilates them by a square margin and labels
// the result again.  Every per-pixel step runs here; the per-component
// bookkeeping (reasons, budget, overlap tables, the JSON census) is host
// logic in fauxice_b200/routing.py.
//
//   k_ccl_*        8-connected components by lock-free union-find over
//                  segments: a segment is a run of set pixels inside one
//                  32-pixel word of a row, and its first pixel's slot is its
//                  node.  A root is only ever linked under a smaller root, so
//                  each root is its component's smallest raster index and the
//                  final ids (1..K by root order) follow
//                  scipy.ndimage.label's raster order of first pixels.
//   k_dist_*       chessboard distance to the nearest in-frame background
//                  pixel (distance_transform_cdt, metric "chessboard"): exact
//                  up to 63 from a bit plane, deeper pixels by Jacobi
//                  relaxation in shared-memory tiles until no change.
//   k_stats        per-label area, bounding box and maximum of a plane.
//   k_dilate_*     square (Chebyshev) dilation, separable: on bits in
//                  shared-memory tiles up to radius 31, beyond it the nearest
//                  set pixel along each column, then along each row, within
//                  a radius clipped to the frame.
//   k_pairs        (label, label) pairs of two label planes, emitted only
//                  where a pixel starts a new pair locally (the host removes
//                  the remaining duplicates).
#include <utility>

#include "fx_internal.cuh"

namespace fx {

constexpr int kRouteThreads = 256;
constexpr uint32_t kFindLimit = 1u << 26;  // bounds every pointer walk

// Root of x.  Path halving (each visited slot is pointed at its
// grandparent) only ever stores an ancestor, so concurrent finds and links
// stay consistent.
__device__ __forceinline__ int32_t find_root(int32_t *parent, int32_t x, uint32_t *err) {
    uint32_t steps = 0;
    int32_t p = parent[x];
    while (p != x) {
        const int32_t gp = parent[p];
        if (gp != p) parent[x] = gp;
        x = p;
        p = parent[x];
        if (++steps > kFindLimit) {
            raise_error(err, FX_ERR_INTERNAL);
            break;
        }
    }
    return x;
}

// A bit plane holds 32-pixel words, words_per_row(w) per row, bit x % 32 of
// word x / 32; bits past the row's end are 0.
__host__ __device__ __forceinline__ int words_per_row(int w) { return (w + 31) / 32; }

// Walks the words of a plane in steps of a grid: row and word of the first,
// kept by additions (one 64-bit division per thread instead of one per word).
struct WordWalk {
    int64_t y, sy;
    int x, sx, wpr;
    __device__ WordWalk(int64_t first, int64_t step, int words_a_row)
        : y(first / words_a_row), sy(step / words_a_row), x((int)(first % words_a_row)),
          sx((int)(step % words_a_row)), wpr(words_a_row) {}
    __device__ void next() {
        y += sy;
        x += sx;
        if (x >= wpr) {
            x -= wpr;
            ++y;
        }
    }
    // j words further on (small j)
    __device__ void at(int j, int64_t &yy, int &xx) const {
        yy = y;
        xx = x + j;
        while (xx >= wpr) {
            xx -= wpr;
            ++yy;
        }
    }
};

// First pixel (bit) of the segment of word `bits` that holds bit x.
__device__ __forceinline__ int segment_start(uint32_t bits, int x) {
    return 32 - __clz(~bits & ((1u << x) - 1u));
}

// The mask as a bit plane, and (when `parent` is given) every segment's node
// as its own root.  One warp packs a word by ballot, four words in flight:
// everything after works on 1/8 byte per pixel instead of the mask's byte
// and a 4-byte slot of every pixel.
__global__ void __launch_bounds__(kRouteThreads)
    k_pack(const uint8_t *__restrict__ mask, int h, int w, uint32_t *__restrict__ bits,
           int32_t *parent) {
    const int lane = threadIdx.x & 31;
    const int wpr = words_per_row(w);
    const int64_t words = (int64_t)h * wpr;
    const int64_t warps = (int64_t)gridDim.x * (kRouteThreads / 32);
    int64_t k0 = (blockIdx.x * (int64_t)(kRouteThreads / 32) + (threadIdx.x >> 5)) * 4;
    WordWalk at(k0, warps * 4, wpr);
    for (; k0 < words; k0 += warps * 4, at.next()) {
        bool set[4];
        int64_t px[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t k = k0 + j;
            int64_t y;
            int wx;
            at.at(j, y, wx);
            const int x = wx * 32 + lane;
            px[j] = y * w + x;
            set[j] = k < words && x < w && mask[px[j]];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, set[j]);
            if (k0 + j < words && lane == 0) bits[k0 + j] = b;
            if (parent && set[j] && (lane == 0 || !((b >> (lane - 1)) & 1u)))
                parent[px[j]] = (int32_t)px[j];
        }
    }
}

// Link the components of pixel a and pixel b: the larger root goes under the
// smaller one.  A failed link (the root moved meanwhile) retries from the
// new roots; each retry strictly lowers the larger root, so the loop ends.
__device__ void ccl_union(int32_t *parent, int32_t a, int32_t b, uint32_t *err) {
    for (uint32_t tries = 0; tries < kFindLimit; ++tries) {
        a = find_root(parent, a, err);
        b = find_root(parent, b, err);
        if (a == b) return;
        if (a < b) {
            const int32_t t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(&parent[a], a, b) == a) return;
    }
    raise_error(err, FX_ERR_INTERNAL);
}

// Links between the segments of a word and their neighbours: the segment to
// the left across the word boundary, and the row above.  A contact with the row
// above is linked where its first pixel shows it (a pixel whose left neighbour
// already touches the same segment above is skipped), so links are per pair of
// segments rather than per pixel.  One thread per two pixels of a word: a
// thread's links are serial, and a word of noise or of one-pixel stripes has up
// to 16.  Labels of 300x300 half-set noise take 109 us so, 148 with a thread
// per word, of stripes 701x933 198 and 580; of a native frame's floor mask 209
// and 216.  A thread per pixel costs masks of long runs 20%.
constexpr int kUnionParts = 16, kUnionBits = 32 / kUnionParts;
__global__ void __launch_bounds__(kRouteThreads)
    k_ccl_union(const uint32_t *__restrict__ bits, int h, int w, int32_t *parent, uint32_t *err) {
    const int wpr = words_per_row(w);
    const int64_t parts = (int64_t)h * wpr * kUnionParts;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < parts;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = i / kUnionParts;
        const uint32_t c = bits[k];
        const int part = (int)(i % kUnionParts);
        const uint32_t own = ((1u << kUnionBits) - 1u) << (part * kUnionBits);
        if (!(c & own)) continue;
        const int64_t y = k / wpr;
        const int wx = (int)(k - y * wpr);
        const int32_t row = (int32_t)(y * w + wx * 32);  // pixel of bit 0
        if (part == 0 && wx > 0 && (c & 1u)) {
            const uint32_t p = bits[k - 1];
            if (p >> 31) ccl_union(parent, row, row - 32 + segment_start(p, 31), err);
        }
        if (y == 0) continue;
        const int64_t u = k - wpr;
        const uint32_t a = bits[u];
        const uint32_t al = wx > 0 ? bits[u - 1] : 0u;
        const uint32_t ar = wx + 1 < wpr ? bits[u + 1] : 0u;
        if (!(a | (al >> 31) | (ar & 1u))) continue;
        const int32_t up = row - w;
        const uint32_t ul = (a << 1) | (al >> 31), ur = (a >> 1) | (ar << 31);
        // straight up, unless the pixel to the left has the same contact
        for (uint32_t m = c & a & ~((c << 1) & ul) & own; m; m &= m - 1u) {
            const int x = __ffs(m) - 1;
            ccl_union(parent, row + segment_start(c, x), up + segment_start(a, x), err);
        }
        // up-left of a segment's first pixel, up-right of its last
        for (uint32_t m = c & ~a & ul & ~(c << 1) & own; m; m &= m - 1u) {
            const int x = __ffs(m) - 1;
            const int32_t other = x > 0 ? up + segment_start(a, x - 1)
                                        : up - 32 + segment_start(al, 31);
            ccl_union(parent, row + segment_start(c, x), other, err);
        }
        for (uint32_t m = c & ~a & ur & ~(c >> 1) & own; m; m &= m - 1u) {
            const int x = __ffs(m) - 1;
            const int32_t other = x < 31 ? up + segment_start(a, x + 1) : up + 32;
            ccl_union(parent, row + segment_start(c, x), other, err);
        }
    }
}

// After every link: point each node straight at its root and count the roots
// per block of 256 words.  The walk only reads (every slot it meets holds an
// ancestor, the old one or the root), and each slot is written only by its
// own thread, so every slot ends up holding its root.
__global__ void __launch_bounds__(kRouteThreads)
    k_ccl_flatten(const uint32_t *__restrict__ bits, int h, int w, int32_t *parent,
                  uint32_t *block_roots, uint32_t *err) {
    const int wpr = words_per_row(w);
    const int64_t words = (int64_t)h * wpr;
    const int64_t k = blockIdx.x * (int64_t)kRouteThreads + threadIdx.x;
    uint32_t roots = 0;
    if (k < words) {
        const uint32_t c = bits[k];
        const int64_t y = c ? k / wpr : 0;
        const int32_t row = (int32_t)(y * w + (k - y * wpr) * 32);
        for (uint32_t m = c & ~(c << 1); m; m &= m - 1u) {
            const int32_t node = row + __ffs(m) - 1;
            int32_t x = parent[node];
            uint32_t steps = 0;
            int32_t p = parent[x];
            while (p != x) {
                x = p;
                p = parent[x];
                if (++steps > kFindLimit) {
                    raise_error(err, FX_ERR_INTERNAL);
                    break;
                }
            }
            parent[node] = x;
            roots += x == node;
        }
    }
    const int total = __syncthreads_count(roots > 0);  // most blocks hold none
    __shared__ uint32_t sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    if (total && roots) atomicAdd(&sum, roots);
    __syncthreads();
    if (threadIdx.x == 0) block_roots[blockIdx.x] = sum;
}

// Exclusive scan of the per-block root counts (one block); total at [n].
__global__ void k_ccl_scan(uint32_t *block_roots, int64_t nblocks) {
    __shared__ uint32_t warp_sums[32];
    uint32_t carry = 0;
    for (int64_t base = 0; base < nblocks; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const uint32_t v = i < nblocks ? block_roots[i] : 0u;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
                if (lane >= o) s += y;
            }
            warp_sums[lane] = s;
        }
        __syncthreads();
        const uint32_t prefix = (warp ? warp_sums[warp - 1] : 0u) + x - v;
        if (i < nblocks) block_roots[i] = carry + prefix;
        carry += warp_sums[(blockDim.x >> 5) - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) block_roots[nblocks] = carry;
}

// Ids 1..K to the roots in raster order (word order inside a block by a
// block scan), stored in the root's own slot as -(id) - 1.  Each thread
// reads and writes only its own words' slots.
__global__ void __launch_bounds__(kRouteThreads)
    k_ccl_number(const uint32_t *__restrict__ bits, int h, int w, int32_t *parent,
                 const uint32_t *block_base) {
    __shared__ uint32_t warp_sums[kRouteThreads / 32];
    const int wpr = words_per_row(w);
    const int64_t words = (int64_t)h * wpr;
    const int64_t k = blockIdx.x * (int64_t)kRouteThreads + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t nodes = 0, mine = 0;
    int32_t row = 0;
    if (k < words) {
        const uint32_t c = bits[k];
        const int64_t y = c ? k / wpr : 0;
        row = (int32_t)(y * w + (k - y * wpr) * 32);
        for (uint32_t m = c & ~(c << 1); m; m &= m - 1u) {
            const int x = __ffs(m) - 1;
            if (parent[row + x] == row + x) nodes |= 1u << x;
        }
        mine = __popc(nodes);
    }
    uint32_t x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += v;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    uint32_t id = block_base[blockIdx.x] + x - mine;
    for (int q = 0; q < warp; ++q) id += warp_sums[q];
    for (; nodes; nodes &= nodes - 1u) {
        ++id;
        parent[row + __ffs(nodes) - 1] = -(int32_t)id - 1;
    }
}

// Labels: a numbered root's slot holds -(id) - 1, every other node its
// root's index (flattened).  One warp per word, four words in flight; the
// words are packed again from the mask, since the bit plane lives in the
// label plane until here.
__global__ void __launch_bounds__(kRouteThreads)
    k_ccl_labels(const uint8_t *__restrict__ mask, const int32_t *__restrict__ parent, int h,
                 int w, int32_t *__restrict__ labels) {
    const int lane = threadIdx.x & 31;
    const int wpr = words_per_row(w);
    const int64_t words = (int64_t)h * wpr;
    const int64_t warps = (int64_t)gridDim.x * (kRouteThreads / 32);
    int64_t k0 = (blockIdx.x * (int64_t)(kRouteThreads / 32) + (threadIdx.x >> 5)) * 4;
    WordWalk at(k0, warps * 4, wpr);
    for (; k0 < words; k0 += warps * 4, at.next()) {
        bool set[4], in[4];
        int64_t px[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t k = k0 + j;
            int64_t y;
            int wx;
            at.at(j, y, wx);
            const int x = wx * 32 + lane;
            px[j] = y * w + x;
            in[j] = k < words && x < w;
            set[j] = in[j] && mask[px[j]];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, set[j]);
            int32_t label = 0;
            if (set[j]) {
                int32_t p = parent[px[j] - lane + segment_start(b, lane)];
                if (p >= 0) p = parent[p];
                label = -p - 1;
            }
            if (in[j]) labels[px[j]] = label;
        }
    }
}

// ---------------------------------------------------------------------------
// Chessboard distance: dist = 0 on background; foreground relaxes to
// min(dist, min over the 8 neighbours + 1).  A block relaxes a 32x32 tile
// with an 8-pixel halo in shared memory for 8 steps (the tile's centre is
// exact for those steps), and reports whether anything changed.
// ---------------------------------------------------------------------------

constexpr int kDistTile = 32, kDistHalo = 8, kDistSide = kDistTile + 2 * kDistHalo;
constexpr int32_t kDistInf = 0x3FFFFFFF;

// Distances up to kDistNear from the bit plane.  A pixel's distance is the
// least over the rows y +- k of max(k, distance along that row), and only rows
// with k below the best so far can lower it; the row distances come from the
// 64 bits to either side of the pixel.  A block covers 16 rows x 256 columns
// with 64 pixels of halo in shared memory (7 KB); a tile without a set
// pixel only writes zeros.  Tiles are numbered along x: a tall mask has more
// rows of them than the 65,535 blocks of the other axes.  Pixels outside the frame are no background.  A
// deeper pixel gets kDistInf, from which the relaxation finishes it.
// (Relaxing every tile from scratch took four launches of 500 us on a native
// frame; this takes one of 140 us after 35 us of packing, 39 instead of 80 us on
// 701x933; tiles of 64 rows left a small frame 44 blocks: 77 us.)
constexpr int kDistNear = 63;
constexpr int kNearRows = 16, kNearWords = 8;

__global__ void __launch_bounds__(kRouteThreads)
    k_dist_near(const uint32_t *__restrict__ bits, int h, int w, int32_t *__restrict__ dist,
                uint32_t *deep) {
    constexpr int kRows = kNearRows + 2 * 64, kCols = kNearWords + 4;
    __shared__ uint32_t t[kRows][kCols + 1];
    const int wpr = words_per_row(w);
    const unsigned across = (wpr + kNearWords - 1) / kNearWords;
    const int y0 = blockIdx.x / across * kNearRows, w0 = blockIdx.x % across * kNearWords;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool any = false;
    for (int k = threadIdx.x; k < kRows * kCols; k += kRouteThreads) {
        const int r = k / kCols, c = k % kCols;
        const int y = y0 - 64 + r, wx = w0 - 2 + c;
        uint32_t v = 0xFFFFFFFFu;  // outside the frame: no background
        if (y >= 0 && y < h && wx >= 0 && wx < wpr) {
            v = bits[(int64_t)y * wpr + wx];
            any |= v && r >= 64 && r < 64 + kNearRows && c >= 2 && c < 2 + kNearWords;
            if (wx == wpr - 1 && (w & 31)) v |= 0xFFFFFFFFu << (w & 31);
        }
        t[r][c] = v;
    }
    any = __syncthreads_or(any);
    bool left = false;
    for (int k = warp; k < kNearRows * kNearWords; k += kRouteThreads / 32) {
        const int r = k / kNearWords, c = k % kNearWords;
        const int y = y0 + r, x = (w0 + c) * 32 + lane;
        if (y >= h || x >= w) continue;
        int32_t best = 0;
        if (any && ((t[r + 64][c + 2] >> lane) & 1u)) {
            best = kDistNear + 1;
            for (int d = 0; d < best; ++d) {
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const uint32_t *q = t[r + 64 + (side ? d : -d)] + c;
                    // 64 pixels ending at x (bit 63 = x), and 64 starting there
                    const uint32_t lo = __funnelshift_r(q[0], q[1], (lane + 1) & 31);
                    const uint32_t mid = __funnelshift_r(q[1], q[2], (lane + 1) & 31);
                    const unsigned long long before =
                        lane == 31 ? ((unsigned long long)q[2] << 32) | q[1]
                                   : ((unsigned long long)mid << 32) | lo;
                    const unsigned long long after =
                        ((unsigned long long)__funnelshift_r(q[3], q[4], lane) << 32) |
                        __funnelshift_r(q[2], q[3], lane);
                    const int gl = __clzll(~before);                        // 64: none
                    const int gr = ~after ? __ffsll((long long)~after) - 1 : 64;
                    const int g = min(gl, gr);
                    best = min(best, max(d, g));
                }
            }
            if (best > kDistNear) {
                best = kDistInf;
                left = true;
            }
        }
        dist[(int64_t)y * w + x] = best;
    }
    if (__syncthreads_or(left) && threadIdx.x == 0) atomicOr(deep, 1u);
}

__global__ void __launch_bounds__(kRouteThreads)
    k_dist_relax(const int32_t *__restrict__ in, int32_t *__restrict__ out, int h, int w,
                 uint32_t *changed) {
    __shared__ int32_t t[2][kDistSide][kDistSide];
    const unsigned across = (unsigned)(((int64_t)w + kDistTile - 1) / kDistTile);
    const int y0 = blockIdx.x / across * kDistTile - kDistHalo;
    const int x0 = blockIdx.x % across * kDistTile - kDistHalo;
    for (int k = threadIdx.x; k < kDistSide * kDistSide; k += blockDim.x) {
        const int r = k / kDistSide, c = k % kDistSide;
        const int y = y0 + r, x = x0 + c;
        // outside the frame: no background and no path (never lowers a value)
        t[0][r][c] = (y >= 0 && y < h && x >= 0 && x < w) ? in[(int64_t)y * w + x] : kDistInf;
    }
    __syncthreads();
    int b = 0;
    for (int step = 0; step < kDistHalo; ++step) {
        for (int k = threadIdx.x; k < kDistSide * kDistSide; k += blockDim.x) {
            const int r = k / kDistSide, c = k % kDistSide;
            int32_t v = t[b][r][c];
            if (v > 0 && r > 0 && r < kDistSide - 1 && c > 0 && c < kDistSide - 1) {
                int32_t m = kDistInf;
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                    for (int dx = -1; dx <= 1; ++dx) m = min(m, t[b][r + dy][c + dx]);
                if (m < kDistInf && m + 1 < v) v = m + 1;
            }
            t[b ^ 1][r][c] = v;
        }
        __syncthreads();
        b ^= 1;
    }
    bool any = false;
    for (int k = threadIdx.x; k < kDistTile * kDistTile; k += blockDim.x) {
        const int r = k / kDistTile + kDistHalo, c = k % kDistTile + kDistHalo;
        const int y = y0 + r, x = x0 + c;
        if (y < h && x < w) {
            const int32_t v = t[b][r][c];
            const int64_t o = (int64_t)y * w + x;
            any |= v != in[o];
            out[o] = v;
        }
    }
    if (__syncthreads_or(any) && threadIdx.x == 0) atomicOr(changed, 1u);
}

// ---------------------------------------------------------------------------
// Per-label statistics: area, bounding box [y0, x0, y1, x1) and maximum of
// an optional plane.
// ---------------------------------------------------------------------------

__global__ void k_stats_init(int64_t k, unsigned long long *area, int32_t *box, int32_t *vmax) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < k;
         i += (int64_t)gridDim.x * blockDim.x) {
        area[i] = 0;
        box[4 * i] = box[4 * i + 1] = 0x7FFFFFFF;
        box[4 * i + 2] = box[4 * i + 3] = -1;
        if (vmax) vmax[i] = -1;
    }
}

// One warp per 32-pixel word of a row, four words in flight.  Neighbouring
// pixels of one label are one run: its first lane adds the run's length, box
// and maximum, so a run costs five or six atomics instead of every pixel.
__global__ void __launch_bounds__(kRouteThreads)
    k_stats(const int32_t *__restrict__ labels, const int32_t *__restrict__ plane, int h, int w,
            int64_t k_max, unsigned long long *area, int32_t *box, int32_t *vmax) {
    const int lane = threadIdx.x & 31;
    const int wpr = words_per_row(w);
    const int64_t words = (int64_t)h * wpr;
    const int64_t warps = (int64_t)gridDim.x * (kRouteThreads / 32);
    int64_t k0 = (blockIdx.x * (int64_t)(kRouteThreads / 32) + (threadIdx.x >> 5)) * 4;
    WordWalk at(k0, warps * 4, wpr);
    for (; k0 < words; k0 += warps * 4, at.next()) {
        int32_t lab[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t k = k0 + j;
            int64_t y;
            int wx;
            at.at(j, y, wx);
            const int x = wx * 32 + lane;
            lab[j] = k < words && x < w ? labels[y * w + x] : 0;
            if (lab[j] > k_max) lab[j] = 0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t l = lab[j] > 0 ? lab[j] : 0;
            if (!__any_sync(0xFFFFFFFFu, l)) continue;
            int64_t yy;
            int wx;
            at.at(j, yy, wx);
            const int y = (int)yy, x = wx * 32 + lane;
            const int32_t prev = __shfl_up_sync(0xFFFFFFFFu, l, 1);
            const uint32_t starts = __ballot_sync(0xFFFFFFFFu, lane == 0 || prev != l);
            const uint32_t after = lane < 31 ? starts >> (lane + 1) : 0u;
            const int len = after ? __ffs(after) : 32 - lane;  // to the next run's start
            int32_t v = -1;
            if (vmax) {
                v = l ? plane[(int64_t)y * w + x] : -1;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t u = __shfl_down_sync(0xFFFFFFFFu, v, o);
                    if (o < len) v = max(v, u);
                }
            }
            if (l && ((starts >> lane) & 1u)) {
                const int64_t q = (int64_t)l - 1;
                atomicAdd(&area[q], (unsigned long long)len);
                atomicMin(&box[4 * q], y);
                atomicMin(&box[4 * q + 1], x);
                atomicMax(&box[4 * q + 2], y + 1);
                atomicMax(&box[4 * q + 3], x + len);
                if (vmax) atomicMax(&vmax[q], v);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Square dilation, separable: a pixel is set when a set pixel lies within
// `r` along the row, then within `r` along the column.
//
// Radii up to kDilateBits: a block packs its 32 x 256 tile and the halo into
// bits, dilates the rows with shifts (doubling: the union over shifts 0..n
// becomes 0..2n + 1 in one step) and ORs 2 r + 1 rows.
constexpr int kDilateBits = 31;
constexpr int kDilateRows = 32, kDilateWords = 8;

__global__ void __launch_bounds__(kRouteThreads)
    k_dilate_tile(const uint8_t *__restrict__ in, int h, int w, int rv, int rh,
                  uint8_t *__restrict__ out) {
    __shared__ uint32_t t[kDilateRows + 2 * kDilateBits][kDilateWords + 2];
    __shared__ uint32_t u[kDilateRows + 2 * kDilateBits][kDilateWords];
    const int y0 = blockIdx.y * kDilateRows, w0 = blockIdx.x * kDilateWords;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rows = kDilateRows + 2 * rv;
    for (int k0 = warp * 4; k0 < rows * (kDilateWords + 2); k0 += kRouteThreads / 32 * 4) {
        bool set[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + j;
            const int y = y0 - rv + k / (kDilateWords + 2);
            const int x = (w0 - 1 + k % (kDilateWords + 2)) * 32 + lane;
            set[j] = k < rows * (kDilateWords + 2) && y >= 0 && y < h && x >= 0 && x < w &&
                     in[(int64_t)y * w + x];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, set[j]);
            const int k = k0 + j;
            if (lane == 0 && k < rows * (kDilateWords + 2))
                t[k / (kDilateWords + 2)][k % (kDilateWords + 2)] = b;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < rows * kDilateWords; k += kRouteThreads) {
        const int r = k / kDilateWords, c = k % kDilateWords;
        unsigned long long a = ((unsigned long long)t[r][c + 1] << 32) | t[r][c];
        unsigned long long b = ((unsigned long long)t[r][c + 2] << 32) | t[r][c + 1];
        for (int n = 0; n < rh;) {
            const int s = min(n + 1, rh - n);
            a |= a << s;
            b |= b >> s;
            n += s;
        }
        u[r][c] = (uint32_t)(a >> 32) | (uint32_t)b;
    }
    __syncthreads();
    for (int k = warp; k < kDilateRows * kDilateWords; k += kRouteThreads / 32) {
        const int r = k / kDilateWords, c = k % kDilateWords;
        const int y = y0 + r, x = (w0 + c) * 32 + lane;
        if (y >= h) break;
        uint32_t v = 0;
        for (int d = lane; d <= 2 * rv; d += 32) v |= u[r + d][c];
        v = __reduce_or_sync(0xFFFFFFFFu, v);
        if (x < w) out[(int64_t)y * w + x] = (v >> lane) & 1u;
    }
}

// Larger radii, and a dilation in place: each thread sweeps one column or one
// row twice (nearest set pixel before and after), so any radius costs the same.
__global__ void k_dilate_cols(const uint8_t *__restrict__ in, int h, int w, int r,
                              uint8_t *__restrict__ out) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= w) return;
    int last = -0x3FFFFFFF;  // last set row at or above y
    for (int y = 0; y < h; ++y) {
        if (in[(int64_t)y * w + x]) last = y;
        out[(int64_t)y * w + x] = (y - last) <= r;
    }
    int next = 0x3FFFFFFF;  // next set row at or below y
    for (int y = h - 1; y >= 0; --y) {
        if (in[(int64_t)y * w + x]) next = y;
        if (next - y <= r) out[(int64_t)y * w + x] = 1;
    }
}

__global__ void k_dilate_rows(const uint8_t *__restrict__ in, int h, int w, int r,
                              uint8_t *__restrict__ out) {
    const int y = blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= h) return;
    const uint8_t *row = in + (int64_t)y * w;
    uint8_t *dst = out + (int64_t)y * w;
    int last = -0x3FFFFFFF;
    for (int x = 0; x < w; ++x) {
        if (row[x]) last = x;
        dst[x] = (x - last) <= r;
    }
    int next = 0x3FFFFFFF;
    for (int x = w - 1; x >= 0; --x) {
        if (row[x]) next = x;
        if (next - x <= r) dst[x] = 1;
    }
}

// ---------------------------------------------------------------------------
// (a, b) label pairs where both are positive and the pixel has no earlier
// 8-neighbour (W, NW, N, NE) carrying the same pair; every distinct pair has
// at least one such pixel.
// ---------------------------------------------------------------------------

__global__ void k_pairs(const int32_t *__restrict__ la, const int32_t *__restrict__ lb, int h,
                        int w, int64_t capacity, int2 *pairs, unsigned long long *count) {
    const int64_t n = (int64_t)h * w;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t a = la[i];
        if (a <= 0) continue;
        const int32_t b = lb[i];
        if (b <= 0) continue;
        const int y = (int)(i / w), x = (int)(i % w);
        auto same = [&](int64_t j) { return la[j] == a && lb[j] == b; };
        bool seen = x > 0 && same(i - 1);
        if (!seen && y > 0) {
            const int64_t u = i - w;
            seen = (x > 0 && same(u - 1)) || same(u) || (x + 1 < w && same(u + 1));
        }
        if (seen) continue;
        const unsigned long long at = atomicAdd(count, 1ull);
        if ((int64_t)at < capacity) pairs[at] = make_int2(a, b);
    }
}

static unsigned grid_for(int64_t n) {
    const int64_t b = (n + kRouteThreads - 1) / kRouteThreads;
    return (unsigned)(b < 4096 ? (b > 0 ? b : 1) : 4096);
}

}  // namespace fx

using namespace fx;

// Launch kRouteThreads (or `threads`) a block; false when the launch is refused.
template <typename... KArgs, typename... Args>
static bool launch(void (*kernel)(KArgs...), dim3 grid, cudaStream_t stream, int threads,
                   Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    if (cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...) == cudaSuccess) return true;
    cudaGetLastError();  // reported by the caller's status
    return false;
}

// Tiles of rows x cols pixels that cover h x w, as a one-dimensional grid.
static unsigned tiles_of(int64_t h, int64_t w, int rows, int cols) {
    return (unsigned)((h + rows - 1) / rows * ((w + cols - 1) / cols));
}

// Copies a word back and waits for the stream.
static bool fetch(void *dst, const void *src, size_t bytes, cudaStream_t stream) {
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream) == cudaSuccess &&
           cudaStreamSynchronize(stream) == cudaSuccess;
}

// Blocks of a grid-stride kernel with one warp per four 32-pixel words.
static unsigned grid_for_words(int64_t words) {
    const int64_t b = (words + kRouteThreads / 8 - 1) / (kRouteThreads / 8);
    return (unsigned)(b < 2368 ? (b > 0 ? b : 1) : 2368);  // 16 per SM
}

// Work buffers are the caller's (device): forest int32[n] (distinct from
// labels), block_scratch ceil(n / 256) + 1 uint32, err one uint32.  The bit
// plane (at most one word per pixel) lives in the label plane until the
// labels are written.
FX_API int fx_label8(const uint8_t *d_mask, int32_t h, int32_t w, int32_t *d_labels,
                     int32_t *d_forest, uint32_t *d_block_scratch, uint32_t *d_err,
                     int64_t *count, void *stream) {
    if (!d_mask || !d_labels || !d_forest || !d_block_scratch || !d_err || !count || h < 1 ||
        w < 1 || (int64_t)h * w >= ((int64_t)1 << 31))
        return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int64_t words = (int64_t)h * words_per_row(w);
    const int64_t nblocks = (words + kRouteThreads - 1) / kRouteThreads;
    uint32_t *bits = reinterpret_cast<uint32_t *>(d_labels);
    if (cudaMemsetAsync(d_err, 0, sizeof(uint32_t), st) != cudaSuccess) return FX_ERR_CUDA;
    const unsigned nb = (unsigned)nblocks;
    uint32_t total = 0, err = 0;
    if (!launch(k_pack, grid_for_words(words), st, kRouteThreads, d_mask, h, w, bits, d_forest) ||
        !launch(k_ccl_union, grid_for(words * kUnionParts), st, kRouteThreads, bits, h, w, d_forest, d_err) ||
        !launch(k_ccl_flatten, nb, st, kRouteThreads, bits, h, w, d_forest, d_block_scratch,
                d_err) ||
        !launch(k_ccl_scan, 1, st, 1024, d_block_scratch, nblocks) ||
        !launch(k_ccl_number, nb, st, kRouteThreads, bits, h, w, d_forest, d_block_scratch) ||
        !launch(k_ccl_labels, grid_for_words(words), st, kRouteThreads, d_mask, d_forest, h, w,
                d_labels) ||
        cudaMemcpyAsync(&total, d_block_scratch + nblocks, sizeof(uint32_t),
                        cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        !fetch(&err, d_err, sizeof(uint32_t), st))
        return FX_ERR_CUDA;
    if (err) return FX_ERR_INTERNAL;
    *count = total;
    return FX_OK;
}

FX_API int fx_chessboard_distance(const uint8_t *d_mask, int32_t h, int32_t w, int32_t *d_dist,
                                  int32_t *d_work, uint32_t *d_flag, void *stream) {
    if (!d_mask || !d_dist || !d_work || !d_flag || h < 1 || w < 1) return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int64_t n = (int64_t)h * w;
    // the near distances; the bit plane lives in d_work until the relaxation
    uint32_t *bits = reinterpret_cast<uint32_t *>(d_work);
    const int wpr = words_per_row(w);
    uint32_t changed = 0;
    if (cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), st) != cudaSuccess) return FX_ERR_CUDA;
    if (!launch(k_pack, grid_for_words((int64_t)h * wpr), st, kRouteThreads, d_mask, h, w, bits,
                static_cast<int32_t *>(nullptr)) ||
        !launch(k_dist_near, tiles_of(h, wpr, kNearRows, kNearWords), st, kRouteThreads, bits, h,
                w, d_dist, d_flag) ||
        !fetch(&changed, d_flag, sizeof(uint32_t), st))
        return FX_ERR_CUDA;
    if (!changed) return FX_OK;
    const unsigned grid = tiles_of(h, w, kDistTile, kDistTile);
    int32_t *a = d_dist, *b = d_work;
    // every launch moves each front by up to kDistHalo pixels; the distance
    // of any pixel is below max(h, w), which bounds the launches
    const int64_t limit = (h > w ? h : w) / kDistHalo + 2;
    for (int64_t it = 0; it < limit && changed; ++it) {
        changed = 0;
        if (cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), st) != cudaSuccess) return FX_ERR_CUDA;
        if (!launch(k_dist_relax, grid, st, kRouteThreads, a, b, h, w, d_flag) ||
            !fetch(&changed, d_flag, sizeof(uint32_t), st))
            return FX_ERR_CUDA;
        int32_t *t = a;
        a = b;
        b = t;
    }
    if (changed) return FX_ERR_INTERNAL;
    if (a != d_dist &&
        cudaMemcpyAsync(d_dist, a, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToDevice, st) !=
            cudaSuccess)
        return FX_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
}

FX_API int fx_label_stats(const int32_t *d_labels, const int32_t *d_plane, int32_t h, int32_t w,
                          int64_t k, unsigned long long *d_area, int32_t *d_box, int32_t *d_vmax,
                          void *stream) {
    if (!d_labels || !d_area || !d_box || h < 1 || w < 1 || k < 0) return FX_ERR_INVALID_ARGUMENT;
    if (k == 0) return FX_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int32_t *vmax = d_plane ? d_vmax : nullptr;
    if (!launch(k_stats_init, grid_for(k), st, kRouteThreads, k, d_area, d_box, vmax) ||
        !launch(k_stats, grid_for_words((int64_t)h * words_per_row(w)), st, kRouteThreads,
                d_labels, d_plane, h, w, k, d_area, d_box, vmax))
        return FX_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
}

FX_API int fx_dilate_square(const uint8_t *d_in, int32_t h, int32_t w, int32_t radius,
                            uint8_t *d_work, uint8_t *d_out, void *stream) {
    if (!d_in || !d_work || !d_out || h < 1 || w < 1 || radius < 0) return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int rv = radius < h - 1 ? radius : h - 1, rh = radius < w - 1 ? radius : w - 1;
    // a block of the tile kernel reads its halo from d_in while others write
    // d_out; planes that overlap take the two sweeps through d_work
    const uintptr_t in = reinterpret_cast<uintptr_t>(d_in), out = reinterpret_cast<uintptr_t>(d_out);
    const uintptr_t n = (uintptr_t)h * (uintptr_t)w;
    const bool apart = in + n <= out || out + n <= in;
    if (apart && rv <= kDilateBits && rh <= kDilateBits) {
        const dim3 grid((words_per_row(w) + kDilateWords - 1) / kDilateWords,
                        (h + kDilateRows - 1) / kDilateRows);
        if (grid.y <= 65535u) {
            if (!launch(k_dilate_tile, grid, st, kRouteThreads, d_in, h, w, rv, rh, d_out))
                return FX_ERR_CUDA;
            return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
        }
    }
    if (!launch(k_dilate_cols, tiles_of(1, w, 1, 128), st, 128, d_in, h, w, rv, d_work) ||
        !launch(k_dilate_rows, tiles_of(1, h, 1, 128), st, 128, d_work, h, w, rh, d_out))
        return FX_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
}

FX_API int fx_label_pairs(const int32_t *d_a, const int32_t *d_b, int32_t h, int32_t w,
                          int64_t capacity, int32_t *d_pairs, unsigned long long *d_count,
                          int64_t *count, void *stream) {
    if (!d_a || !d_b || !d_pairs || !d_count || !count || h < 1 || w < 1)
        return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), st) != cudaSuccess)
        return FX_ERR_CUDA;
    unsigned long long c = 0;
    if (!launch(k_pairs, grid_for((int64_t)h * w), st, kRouteThreads, d_a, d_b, h, w, capacity,
                reinterpret_cast<int2 *>(d_pairs), d_count) ||
        !fetch(&c, d_count, sizeof(c), st))
        return FX_ERR_CUDA;
    *count = (int64_t)c;
    return (int64_t)c > capacity ? FX_ERR_OUT_OF_MEMORY : FX_OK;
}

// ---------------------------------------------------------------------------
// Label-plane helpers of the routing census
// ---------------------------------------------------------------------------

namespace fx {

__global__ void k_map_labels(const int32_t *__restrict__ labels, int64_t n,
                             const int32_t *__restrict__ map, int64_t k, int32_t *out_i32,
                             uint8_t *out_u8) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t l = labels[i];
        const int32_t v = (l >= 0 && l <= k) ? map[l] : 0;
        if (out_i32) out_i32[i] = v;
        if (out_u8) out_u8[i] = v != 0;
    }
}

__global__ void k_clear_label(uint8_t *mask, const int32_t *__restrict__ labels, int64_t n,
                              int32_t id, unsigned long long *cleared) {
    unsigned long long mine = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (labels[i] == id) {
            mine += mask[i] != 0;
            mask[i] = 0;
        }
    }
    if (mine) atomicAdd(cleared, mine);
}

// One warp per 32 pixels, four groups in flight; neighbouring pixels of one
// key are counted together (one atomic per run, not per pixel).
__global__ void __launch_bounds__(kRouteThreads)
    k_count_where(const int32_t *__restrict__ key, const int32_t *__restrict__ cond, int64_t n,
                  int64_t k, unsigned long long *counts) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (kRouteThreads / 32);
    for (int64_t i0 = (blockIdx.x * (int64_t)(kRouteThreads / 32) + (threadIdx.x >> 5)) * 128;
         i0 < n; i0 += warps * 128) {
        int32_t l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t i = i0 + 32 * j + lane;
            l[j] = i < n ? key[i] : 0;
            if (l[j] < 0 || l[j] > k) l[j] = 0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!__any_sync(0xFFFFFFFFu, l[j])) continue;
            const bool hit = l[j] && cond[i0 + 32 * j + lane] > 0;
            const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
            const int32_t prev = __shfl_up_sync(0xFFFFFFFFu, l[j], 1);
            const uint32_t starts = __ballot_sync(0xFFFFFFFFu, lane == 0 || prev != l[j]);
            if (l[j] && ((starts >> lane) & 1u)) {
                const uint32_t after = lane < 31 ? starts >> (lane + 1) : 0u;
                const int len = after ? __ffs(after) : 32 - lane;
                const uint32_t run = (len < 32 ? (1u << len) - 1u : 0xFFFFFFFFu) << lane;
                const int c = __popc(hits & run);
                if (c) atomicAdd(&counts[l[j]], (unsigned long long)c);
            }
        }
    }
}

__global__ void k_tile_extract(const int32_t *__restrict__ labels, int w, int y0, int x0, int th,
                               int tw, int32_t id, uint8_t *tile) {
    const int64_t n = (int64_t)th * tw;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int ty = (int)(i / tw), tx = (int)(i % tw);
        tile[i] = labels[(int64_t)(y0 + ty) * w + (x0 + tx)] == id;
    }
}

__global__ void k_tile_scatter(const int32_t *__restrict__ tile_labels, int w, int y0, int x0,
                               int th, int tw, int32_t base, int32_t *plane) {
    const int64_t n = (int64_t)th * tw;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t l = tile_labels[i];
        if (l > 0) plane[(int64_t)(y0 + i / tw) * w + (x0 + i % tw)] = base + l;
    }
}

}  // namespace fx

// out[i] = map[labels[i]] (int32 and/or nonzero as uint8); map holds k + 1
// entries, labels outside 0..k map to 0.
FX_API int fx_map_labels(const int32_t *d_labels, int64_t n, const int32_t *d_map, int64_t k,
                         int32_t *d_out_i32, uint8_t *d_out_u8, void *stream) {
    if (!d_labels || !d_map || (!d_out_i32 && !d_out_u8) || n < 1 || k < 0)
        return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (!launch(k_map_labels, grid_for(n), st, kRouteThreads, d_labels, n, d_map, k, d_out_i32,
                d_out_u8))
        return FX_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
}

// Clear mask where labels == id; *cleared = how many of those were set.
FX_API int fx_clear_label(uint8_t *d_mask, const int32_t *d_labels, int64_t n, int32_t id,
                          unsigned long long *d_scratch, int64_t *cleared, void *stream) {
    if (!d_mask || !d_labels || !d_scratch || !cleared || n < 1) return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(d_scratch, 0, sizeof(unsigned long long), st) != cudaSuccess)
        return FX_ERR_CUDA;
    unsigned long long c = 0;
    if (!launch(k_clear_label, grid_for(n), st, kRouteThreads, d_mask, d_labels, n, id,
                d_scratch) ||
        !fetch(&c, d_scratch, sizeof(c), st))
        return FX_ERR_CUDA;
    *cleared = (int64_t)c;
    return FX_OK;
}

// counts[key] += 1 over pixels where 0 < key <= k and cond > 0; counts holds
// k + 1 entries and is cleared first.
FX_API int fx_count_where(const int32_t *d_key, const int32_t *d_cond, int64_t n, int64_t k,
                          unsigned long long *d_counts, void *stream) {
    if (!d_key || !d_cond || !d_counts || n < 1 || k < 0) return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(d_counts, 0, (size_t)(k + 1) * sizeof(unsigned long long), st) !=
        cudaSuccess)
        return FX_ERR_CUDA;
    if (!launch(k_count_where, grid_for_words((n + 31) / 32), st, kRouteThreads, d_key, d_cond, n,
                k, d_counts))
        return FX_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
}

// Tile of a label plane: tile = (labels[y0 + ty][x0 + tx] == id), th x tw.
FX_API int fx_tile_extract(const int32_t *d_labels, int32_t h, int32_t w, int32_t y0, int32_t x0,
                           int32_t th, int32_t tw, int32_t id, uint8_t *d_tile, void *stream) {
    if (!d_labels || !d_tile || th < 1 || tw < 1 || y0 < 0 || x0 < 0 || y0 + th > h ||
        x0 + tw > w)
        return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (!launch(k_tile_extract, grid_for((int64_t)th * tw), st, kRouteThreads, d_labels, w, y0, x0,
                th, tw, id, d_tile))
        return FX_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
}

// plane[y0 + ty][x0 + tx] = base + tile_labels[ty][tx] where tile_labels > 0.
FX_API int fx_tile_scatter(const int32_t *d_tile_labels, int32_t h, int32_t w, int32_t y0,
                           int32_t x0, int32_t th, int32_t tw, int32_t base, int32_t *d_plane,
                           void *stream) {
    if (!d_tile_labels || !d_plane || th < 1 || tw < 1 || y0 < 0 || x0 < 0 || y0 + th > h ||
        x0 + tw > w)
        return FX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (!launch(k_tile_scatter, grid_for((int64_t)th * tw), st, kRouteThreads, d_tile_labels, w, y0,
                x0, th, tw, base, d_plane))
        return FX_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? FX_OK : FX_ERR_CUDA;
}
