// si_sisi_ip.cu -- intersect-path (ip) for one pair of sorted sets.
//
// Replaces findDiagonals (include/helpers.cuh:75-166) + intersectPath
// (src/ip.cu:207-245) for the single-instance case.  Same two-level idea --
// split the merge path of (A, B) into CTA tiles, then each thread takes a
// sub-diagonal of its tile and merges serially (include/helpers.cuh:24-61) --
// re-designed for B200:
//
//  * Grid level (ip_split_kernel, ip_fine_kernel): tile t covers merged
//    positions [t kTile, (t + 1) kTile).  One warp finds where a tile's diagonal
//    crosses the path with a 32-ary search (four round trips for 2^20 elements);
//    of very many tiles the warps take every 64th, and one thread each the rest,
//    between its two neighbours.
//  * Staging: a tile's A and B ranges go into shared memory by two bulk copies
//    (TMA) of their 16-byte aligned supersets, each range with its successor
//    element.  The successors stand for the next tile's first elements, so that
//    an equal pair whose two halves fall into neighbouring tiles is found by the
//    tile that holds the A element (no "augmentation" atomic, quirk of
//    include/helpers.cuh:121-124).
//  * Thread level: merge-path split per thread in shared memory with one tie
//    rule (A first on ties), then kVT merge steps of eight instructions; a match
//    is an A element taken while the head of B equals it.
//  * Output (ip_tile_kernel, up to kPlaceTiles tiles): merged once for the
//    tiles' counts and once more to write each tile's matches behind those of
//    the tiles before it.  No CTA waits for another.  More tiles
//    (ip_group_kernel): once, with a decoupled look-back per group of tiles.
//
// A pair of one tile is a single launch of one CTA, which clears the header
// itself.  Eight CTAs per SM (the group kernel six) hide each other's staging and
// searches, so a tile has no warps of its own for them.  What bounds it: counting
// large pairs, shared memory's banks (the threads' reads are kVT / 2 words apart,
// 2.9 wavefronts a load; 82 % of the LSU's data pipe) and issue slots (80 %); the
// group kernel, at 57 % and 58 % of those, the latency of global memory; small
// pairs, latency.
//
// Measured, device time with elements out / counts only (in brackets: a
// persistent kernel with producer, consumer and output warps on tiles cut at
// value pivots): 1000 x 1000 3.8 / 3.4 us (18 / 16), 2^20 x 2^20 17 / 8 us (42 /
// 24), 2^24 x 2^24 77 / 49 us (96 / 68), 2^27 x 2^27 453 / 261 us (584 / 409).
// 256 threads with 17 steps took 578 / 335 us at 2^27 x 2^27, with 23 steps 477 /
// 284; a look-back per tile 1066 us (every tile's CTA polls the same words).
//
// Techniques bitmap (and auto for large pairs of similar size) and hi run the
// stream engine of si_sisi_bitmap.cu.
#include <algorithm>

#include "si_device.cuh"
#include "si_internal.h"
#include "si_stream.cuh"

namespace si {
namespace {

constexpr int kIpThreads = 192;
constexpr int kIpWarps = kIpThreads / 32;
constexpr int kVT = 27;  // merge steps per thread: odd, so that consecutive threads' shared loads spread over the banks
constexpr uint32_t kTile = kIpThreads * kVT;
static_assert(kTile == kIpOneTile, "the engine's choice counts tiles");
constexpr int kIpCtasPerSm = 8;
// both ranges, their successors, the alignment of both, and the steps by which
// a thread's reads can run over when the sets are not sorted
constexpr uint32_t kStaged = kTile + 2 * 8 + 8 + 32;
// Element output of up to this many tiles merges them twice; of more, once with
// a look-back.
constexpr uint64_t kPlaceTiles = 2048;  // 10.6 M merged elements
constexpr uint64_t kFineTiles = 4096;        // more tiles than this are split in two steps
constexpr uint32_t kCoarse = 64;             // tiles per coarse split
static_assert(kVT <= 31, "a thread's matches are a 32-bit mask");

constexpr uint64_t kFlagAgg = 1ull << 62;
constexpr uint64_t kFlagInc = 2ull << 62;
constexpr uint64_t kValMask = (1ull << 62) - 1;

// Workspace: header ([0..16) error words), the groups' look-back status or the
// tiles' counts, the tiles' splits (A elements before each tile).
constexpr size_t kIpHeader = 256;
struct Layout {
    uint64_t nTiles = 0;
    size_t off_status = 0, off_split = 0, total = 0;
};

Layout make_layout(uint64_t nA, uint64_t nB) {
    Layout L;
    L.nTiles = std::max<uint64_t>(1, (nA + nB + kTile - 1) / kTile);
    size_t o = kIpHeader;
    L.off_status = o;
    o = align_up(o + L.nTiles * 8, 256);
    L.off_split = o;
    o = align_up(o + (L.nTiles + 1) * 8, 256);
    L.total = o;
    return L;
}

// A elements among the first d merged ones (A first on ties): the first i with
// A[i] > B[d - 1 - i], by a warp.
__device__ __forceinline__ uint64_t warp_diagonal(const uint32_t* __restrict__ A, const uint32_t* __restrict__ B,
                                                  uint64_t d, uint64_t lo, uint64_t hi) {
    return warp_first_true(lo, hi, [&](uint64_t i) { return __ldg(A + i) > __ldg(B + d - 1 - i); });
}

// Splits of tiles 0, step, 2 step, ... and nTiles; clears the header, the
// look-back status and the count.
__global__ void __launch_bounds__(256) ip_split_kernel(const uint32_t* __restrict__ A, uint64_t nA,
                                                       const uint32_t* __restrict__ B, uint64_t nB, uint64_t nTiles,
                                                       uint32_t step, uint64_t* __restrict__ split,
                                                       uint64_t* __restrict__ zero, uint64_t nzero,
                                                       uint64_t* __restrict__ d_count) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint64_t tid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x, threads = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = tid; i < nzero; i += threads) zero[i] = 0;
    if (tid == 0) {
        *d_count = 0;
        split[0] = 0;
        split[nTiles] = nA;
    }
    for (uint64_t t = (tid / 32 + 1) * step; t < nTiles; t += threads / 32 * step) {
        const uint64_t d = t * kTile;
        const uint64_t s = warp_diagonal(A, B, d, d > nB ? d - nB : 0, d < nA ? d : nA);
        if ((threadIdx.x & 31) == 0) split[t] = s;
    }
}

// The splits between those of every kCoarse-th tile, one thread each.
__global__ void __launch_bounds__(256) ip_fine_kernel(const uint32_t* __restrict__ A, const uint32_t* __restrict__ B,
                                                      uint64_t nTiles, uint64_t n, uint64_t* split) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the coarse splits
    for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < nTiles; t += uint64_t(gridDim.x) * blockDim.x) {
        if (t % kCoarse == 0) continue;
        const uint64_t t0 = t / kCoarse * kCoarse, t1 = min(t0 + kCoarse, nTiles);
        const uint64_t a0 = split[t0], a1 = split[t1], d = t * kTile;
        const uint64_t b0 = t0 * kTile - a0, b1 = min(t1 * kTile, n) - a1;
        uint64_t lo = d > b1 ? max(a0, d - b1) : a0;
        const uint64_t hi = min(a1, d - b0);
        uint64_t len = hi > lo ? hi - lo : 0;
        while (len > 0) {
            const uint64_t half = len >> 1, i = lo + half;
            const bool before = __ldg(A + i) <= __ldg(B + d - 1 - i);
            lo = before ? i + 1 : lo;
            len = before ? len - half - 1 : half;
        }
        split[t] = lo;
    }
}

constexpr int kLookBackPerLane = 4;  // status words per lane per round trip
__device__ __forceinline__ uint64_t look_back(uint64_t* status, uint64_t t, uint32_t* err) {
    // Warp-wide; returns the exclusive prefix of group t (t > 0).  Flag and
    // value share one 64-bit word, so relaxed accesses suffice.  Each round
    // trip reads the 128 nearest unvisited predecessors, lane l holding
    // tiles base - 4l - 1 ... base - 4l - 4.
    const int lane = threadIdx.x & 31;
    uint64_t prefix = 0;
    int64_t base = static_cast<int64_t>(t);
    while (true) {
        uint64_t s[kLookBackPerLane];
        WaitBudget budget;
        bool gave_up = false;
        while (true) {
            // ready when every status nearer than the nearest inclusive one
            // in the window is published (those beyond it do not matter)
            int first_inc = kLookBackPerLane, first_pending = kLookBackPerLane;
#pragma unroll
            for (int q = kLookBackPerLane - 1; q >= 0; --q) {
                const int64_t p = base - 1 - lane * kLookBackPerLane - q;
                s[q] = p >= 0 ? ld_relaxed_u64(status + p) : kFlagInc;
                if ((s[q] >> 62) == 2) first_inc = q;
                if ((s[q] >> 62) == 0) first_pending = q;
            }
            const uint32_t inc_lanes = __ballot_sync(kFullMask, first_inc < kLookBackPerLane);
            const int inc_lane = inc_lanes ? __ffs(inc_lanes) - 1 : 32;
            const int inc_q = __shfl_sync(kFullMask, first_inc, inc_lane & 31);
            // a pending status nearer than (inc_lane, inc_q) blocks
            const bool blocks = first_pending < kLookBackPerLane &&
                                (lane < inc_lane || (lane == inc_lane && first_pending < inc_q));
            if (!__any_sync(kFullMask, blocks)) break;
            if (__any_sync(kFullMask, budget.expired())) {  // warp-uniform exit
                gave_up = true;
                break;
            }
            __nanosleep(32);
        }
        if (gave_up) {
            if (lane == 0) record_error(err, SI_ERR_TIMEOUT, 1, static_cast<uint32_t>(t));
            return prefix;
        }
        // nearest inclusive status in this window: lane-major, then q
        int first_q = kLookBackPerLane;
#pragma unroll
        for (int q = kLookBackPerLane - 1; q >= 0; --q)
            if ((s[q] >> 62) == 2) first_q = q;
        const uint32_t inc_mask = __ballot_sync(kFullMask, first_q < kLookBackPerLane);
        uint64_t v = 0;
        if (inc_mask) {
            const int first_lane = __ffs(inc_mask) - 1;
#pragma unroll
            for (int q = 0; q < kLookBackPerLane; ++q) {
                const bool take = lane < first_lane || (lane == first_lane && q <= first_q);
                v += take ? (s[q] & kValMask) : 0ull;
            }
            return prefix + warp_sum_u64(v);
        }
#pragma unroll
        for (int q = 0; q < kLookBackPerLane; ++q) v += s[q] & kValMask;
        prefix += warp_sum_u64(v);
        base -= 32 * kLookBackPerLane;
    }
}

// A tile's ranges and where they are staged.
struct TileRange {
    uint64_t a0, a1, b0, b1;
    __device__ __forceinline__ uint32_t na() const { return static_cast<uint32_t>(a1 - a0); }
    __device__ __forceinline__ uint32_t nb() const { return static_cast<uint32_t>(b1 - b0); }
};

__device__ __forceinline__ TileRange tile_range(uint64_t t, uint64_t nA, uint64_t nB, const uint64_t* split,
                                                uint64_t nTiles, uint32_t* err) {
    TileRange r;
    r.a0 = nTiles > 1 ? split[t] : 0;
    r.a1 = nTiles > 1 ? split[t + 1] : nA;
    r.b0 = t * kTile - r.a0;
    r.b1 = min((t + 1) * kTile, nA + nB) - r.a1;
    const bool sane = r.a0 <= r.a1 && r.a1 <= nA && r.a1 - r.a0 <= kTile && r.b0 <= r.b1 && r.b1 <= nB &&
                      r.b1 - r.b0 <= kTile;
    if (!sane) {  // only sets that are not sorted split like this
        if (threadIdx.x == 0) record_error(err, SI_ERR_INVALID_INPUT, 12, static_cast<uint32_t>(t));
        r.a0 = r.a1 = r.b0 = r.b1 = 0;
    }
    return r;
}

// Where a tile's ranges lie in its stage: each range and its successor, at
// their 16-byte phase; every 16-byte block copied holds an element of its set.
struct Staging {
    const void *a_src, *b_src;
    uint32_t bytes_a, bytes_b;
    uint32_t a_at, b_at;  // words of the stage where the first elements are
    __device__ __forceinline__ Staging(const uint32_t* A, uint64_t nA, const uint32_t* B, uint64_t nB,
                                       const TileRange& r) {
        const uint64_t a_end = r.a1 < nA ? r.a1 + 1 : r.a1, b_end = r.b1 < nB ? r.b1 + 1 : r.b1;
        const uintptr_t a_lo = reinterpret_cast<uintptr_t>(A + r.a0) & ~uintptr_t(15);
        const uintptr_t b_lo = reinterpret_cast<uintptr_t>(B + r.b0) & ~uintptr_t(15);
        a_src = reinterpret_cast<const void*>(a_lo);
        b_src = reinterpret_cast<const void*>(b_lo);
        bytes_a = a_end > r.a0
                      ? static_cast<uint32_t>(((reinterpret_cast<uintptr_t>(A + a_end) + 15) & ~uintptr_t(15)) - a_lo)
                      : 0u;
        bytes_b = b_end > r.b0
                      ? static_cast<uint32_t>(((reinterpret_cast<uintptr_t>(B + b_end) + 15) & ~uintptr_t(15)) - b_lo)
                      : 0u;
        a_at = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(A + r.a0) & 15u) >> 2);
        // (+ 4: room for A's end mark)
        b_at = bytes_a / 4 + 4 + static_cast<uint32_t>((reinterpret_cast<uintptr_t>(B + r.b0) & 15u) >> 2);
    }
    // By one thread.
    __device__ __forceinline__ void issue(uint32_t* stage, uint64_t* landed) const {
        mbar_arrive_expect_tx(landed, bytes_a + bytes_b);
        if (bytes_a) bulk_g2s(stage, a_src, bytes_a, landed);
        if (bytes_b) bulk_g2s(stage + (b_at & ~3u), b_src, bytes_b, landed);
    }
};

// Waits for the staged tile and merges it along its path: the thread's A
// elements r.a0 + i0 + x with bit x of the mask set are in B.  False when the
// wait gave up (in every thread).
__device__ __forceinline__ bool merge_tile(uint64_t nA, uint64_t nB, const TileRange& r, const Staging& st, uint64_t t,
                                           uint32_t* staged, uint64_t* landed, uint32_t phase, uint32_t* err,
                                           uint32_t& mask, uint32_t& i0) {
    const uint32_t tid = threadIdx.x;
    const uint32_t na = r.na(), nb = r.nb(), total = na + nb;
    uint32_t *sA = staged + st.a_at, *sB = staged + st.b_at;
    const bool ok = mbar_wait_bounded(landed, phase, err, 5, static_cast<uint32_t>(t));
    const bool ends = r.a1 == nA && r.b1 == nB;
    if (r.a1 == nA && tid == 0) sA[na] = 0xffffffffu;
    if (r.b1 == nB && tid == 1) sB[nb] = 0xffffffffu;
    if (!__syncthreads_and(ok)) return false;
    mask = 0;
    i0 = 0;
    if (na == 0) return true;
    const uint32_t d0 = min(tid * kVT, total), d1 = min(d0 + kVT, total);
    uint32_t lo = d0 > nb ? d0 - nb : 0u, len = min(d0, na) - lo;
    while (len > 0) {
        const uint32_t half = len >> 1, mid = lo + half;
        const bool c = sA[mid] <= sB[d0 - 1 - mid];
        lo = c ? mid + 1 : lo;
        len = c ? len - half - 1 : half;
    }
    i0 = lo;
    // The heads after the ranges' ends are the successors, or 2^32 - 1 past the
    // end of a set: right as long as the other set does not hold that value
    // here, which only its last element can be.
    const bool top = ends && (sA[na - 1] == 0xffffffffu || (nb && sB[nb - 1] == 0xffffffffu));
    if (!top) {
        uint32_t pa = smem_addr(sA + i0), pb = smem_addr(sB + (d0 - i0)), bit = 1;
        uint32_t a = lds_u32(pa), b = lds_u32(pb);
        auto merge_step = [&]() {
            if (a == b) mask |= bit;
            if (a <= b) {
                bit <<= 1;
                pa += 4;
                a = lds_u32(pa);
            } else {
                pb += 4;
                b = lds_u32(pb);
            }
        };
        if (total == kTile) {
#pragma unroll
            for (int s = 0; s < kVT; ++s) merge_step();
        } else {
            for (uint32_t s = d0; s < d1; ++s) merge_step();
        }
    } else {
        uint32_t i = i0, j = d0 - i0;
        for (uint32_t s = d0; s < d1; ++s) {
            const bool a_ok = i < na, b_ok = j < nb;
            const uint32_t a = a_ok ? sA[i] : 0u, b = b_ok ? sB[j] : 0u;
            const bool take_a = a_ok && (!b_ok || a <= b);
            if (take_a && b_ok && a == b) mask |= 1u << (i - i0);
            if (take_a) ++i; else ++j;
        }
    }
    // a thread of sets that are not sorted can step past the tile's A elements:
    // no match is read from there
    if (na - i0 < 32) mask &= (1u << (na - i0)) - 1;
    return true;
}

// Matches before this thread's in the tile, and the tile's (two barriers' worth
// of s_warp: the caller synchronises before the next call).
__device__ __forceinline__ uint32_t tile_scan(uint32_t cnt, uint32_t* s_warp, uint32_t& tile_count) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_inclusive_scan(cnt);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = incl - cnt;
    tile_count = 0;
#pragma unroll
    for (uint32_t w = 0; w < kIpWarps; ++w) {
        before += w < warp ? s_warp[w] : 0u;
        tile_count += s_warp[w];
    }
    return before;
}

// One tile per CTA.  kCount: its matches are added to the count.  kTileCounts:
// they are stored, for a kPlace launch after it, which merges the tile again
// and writes its matches behind those of the tiles before it.  A pair of one
// tile needs kPlace alone.
enum TileMode { kCount = 0, kTileCounts = 1, kPlace = 2 };
template <int kMode>
__global__ void __launch_bounds__(kIpThreads, kIpCtasPerSm) ip_tile_kernel(
    const uint32_t* __restrict__ A, uint64_t nA, const uint32_t* __restrict__ B, uint64_t nB, const uint64_t* split,
    uint64_t nTiles, uint32_t* header, uint32_t* tile_counts, uint32_t* __restrict__ out, uint64_t out_cap,
    uint64_t* __restrict__ d_count) {
    __shared__ __align__(16) uint32_t staged[kStaged];
    __shared__ __align__(8) uint64_t landed;
    __shared__ uint32_t s_warp[kIpWarps];
    __shared__ uint64_t s_sum[kIpWarps];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t t = blockIdx.x;
    if (tid == 0) {
        mbar_init(&landed, 1);
        fence_mbar_init();
    }
    if (nTiles == 1) {
        if (tid < kIpHeader / 4) header[tid] = 0;
    } else {
        if (kMode == kTileCounts) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the splits and the cleared header; the tiles' counts
    }
    __syncthreads();
    const TileRange r = tile_range(t, nA, nB, split, nTiles, header);
    uint64_t sum = 0;
    if (kMode == kPlace && nTiles > 1) {  // the matches of the tiles before this one
        for (uint64_t x = tid; x < t; x += kIpThreads) sum += __ldcg(tile_counts + x);
        sum = warp_sum_u64(sum);
        if (lane == 0) s_sum[warp] = sum;
    }
    const Staging st(A, nA, B, nB, r);
    if (tid == 0) st.issue(staged, &landed);
    uint32_t mask, i0;
    if (!merge_tile(nA, nB, r, st, t, staged, &landed, 0, header, mask, i0)) return;
    const uint32_t cnt = __popc(mask);
    uint32_t tile_count;
    const uint32_t before = tile_scan(cnt, s_warp, tile_count);
    if constexpr (kMode == kCount) {
        if (tid == 0) {
            if (nTiles == 1) *d_count = tile_count;
            else if (tile_count) atomicAdd(reinterpret_cast<unsigned long long*>(d_count), tile_count);
        }
    } else if constexpr (kMode == kTileCounts) {
        if (tid == 0) tile_counts[t] = tile_count;
    } else {
        uint64_t prefix = 0;
        if (nTiles > 1)
#pragma unroll
            for (uint32_t w = 0; w < kIpWarps; ++w) prefix += s_sum[w];
        const uint32_t* mine = staged + st.a_at + i0;
        uint64_t pos = prefix + before;
        bool overflow = false;
        for (uint32_t m = mask; m; m &= m - 1, ++pos) {
            if (pos < out_cap) out[pos] = mine[__ffs(m) - 1];
            else overflow = true;
        }
        if (overflow) record_error(header, SI_ERR_OUTPUT_OVERFLOW, 9, static_cast<uint32_t>(t));
        if (tid == 0 && t + 1 == nTiles) *d_count = prefix + tile_count;
    }
}

// Element output of many tiles in one pass: persistent CTAs take groups of
// kGroup consecutive tiles round robin, merge them, find the group's offset by
// a decoupled look-back over the groups before it and write the matches from
// the sets (a group's tiles are still in L2).  A group's look-back and writes
// come after the next group's merge, when the groups before it have long
// published their counts.  The launch is cooperative: all CTAs are resident and
// a CTA's groups come in order, so a look-back only waits for groups that are
// being merged.
constexpr uint32_t kGroup = 4;
struct GroupMatches {
    uint32_t mask[kGroup][kIpThreads];  // each thread's own
    uint16_t i0[kGroup][kIpThreads], before[kGroup][kIpThreads];
    uint32_t count[kGroup];
};
constexpr int kIpGroupCtasPerSm = 6;  // 33 KiB of shared memory each
__global__ void __launch_bounds__(kIpThreads, kIpGroupCtasPerSm) ip_group_kernel(
    const uint32_t* __restrict__ A, uint64_t nA, const uint32_t* __restrict__ B, uint64_t nB, const uint64_t* split,
    uint64_t nTiles, uint32_t* header, uint64_t* status, uint32_t* __restrict__ out, uint64_t out_cap,
    uint64_t* __restrict__ d_count) {
    __shared__ __align__(16) uint32_t staged[kStaged];
    __shared__ __align__(8) uint64_t landed;
    __shared__ uint32_t s_warp[kIpWarps];
    __shared__ GroupMatches s_group[2];
    __shared__ uint64_t s_prefix;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&landed, 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t phase = 0, total = 0, last_total = 0;
    const uint64_t nGroups = (nTiles + kGroup - 1) / kGroup;
    uint32_t buf = 0;
    for (uint64_t g = blockIdx.x; g < nGroups + gridDim.x; g += gridDim.x, buf ^= 1) {
        const uint64_t t0 = g * kGroup;
        if (g < nGroups) {
            GroupMatches& gm = s_group[buf];
            const uint32_t n = static_cast<uint32_t>(min(uint64_t(kGroup), nTiles - t0));
            total = 0;
            for (uint32_t q = 0; q < n; ++q) {
                const TileRange r = tile_range(t0 + q, nA, nB, split, nTiles, header);
                const Staging st(A, nA, B, nB, r);
                if (tid == 0) st.issue(staged, &landed);
                uint32_t mask, i0, count;
                if (!merge_tile(nA, nB, r, st, t0 + q, staged, &landed, phase, header, mask, i0)) return;
                phase ^= 1;
                const uint32_t before = tile_scan(__popc(mask), s_warp, count);
                gm.mask[q][tid] = mask;
                gm.i0[q][tid] = static_cast<uint16_t>(i0);
                gm.before[q][tid] = static_cast<uint16_t>(before);
                if (tid == 0) gm.count[q] = count;
                total += count;
                // the tile is read before the next one is copied over it
                fence_proxy_async_smem();
                __syncthreads();
            }
            if (tid == 0) st_relaxed_u64(status + g, (g == 0 ? kFlagInc : kFlagAgg) | total);
        }
        if (g >= gridDim.x) {  // the group before, gd
            const uint64_t gd = g - gridDim.x, td = gd * kGroup;
            if (warp == 0) {
                const uint64_t p = gd > 0 ? look_back(status, gd, header) : 0;
                if (lane == 0) {
                    if (gd > 0) st_relaxed_u64(status + gd, kFlagInc | ((p + last_total) & kValMask));
                    s_prefix = p;
                }
            }
            __syncthreads();
            uint64_t prefix = s_prefix;
            const GroupMatches& gm = s_group[buf ^ 1];
            const uint32_t n = static_cast<uint32_t>(min(uint64_t(kGroup), nTiles - td));
            bool overflow = false;
            for (uint32_t q = 0; q < n; ++q) {
                const uint32_t* mine = A + split[td + q] + gm.i0[q][tid];
                uint64_t pos = prefix + gm.before[q][tid];
                for (uint32_t m = gm.mask[q][tid]; m; m &= m - 1, ++pos) {
                    if (pos < out_cap) out[pos] = __ldg(mine + __ffs(m) - 1);
                    else overflow = true;
                }
                prefix += gm.count[q];
            }
            if (overflow) record_error(header, SI_ERR_OUTPUT_OVERFLOW, 9, static_cast<uint32_t>(gd));
            if (tid == 0 && td + n == nTiles) *d_count = prefix;
            __syncthreads();  // the group's words are read before a later group writes them
        }
        last_total = total;
    }
}

}  // namespace

size_t ip_workspace_size(uint64_t nA, uint64_t nB) { return make_layout(nA, nB).total; }

si_status ip_sisi(const uint32_t* dA, uint64_t nA, const uint32_t* dB, uint64_t nB, uint64_t* d_count,
                  uint32_t* d_out, uint64_t out_cap, void* ws, size_t ws_bytes, cudaStream_t stream) {
    const Layout L = make_layout(nA, nB);
    if (ws_bytes < L.total) return SI_ERR_WORKSPACE_TOO_SMALL;
    if (L.nTiles > 0x7fffffffull) return SI_ERR_INVALID_ARGUMENT;
    unsigned char* w = static_cast<unsigned char*>(ws);
    uint64_t* status = reinterpret_cast<uint64_t*>(w + L.off_status);
    uint64_t* split = reinterpret_cast<uint64_t*>(w + L.off_split);
    uint32_t* header = reinterpret_cast<uint32_t*>(w);
    const bool fine = L.nTiles > kFineTiles, grouped = d_out && L.nTiles > kPlaceTiles;
    if (L.nTiles > 1) {
        PhaseTimer timer("sisi_split", stream);
        const uint32_t step = fine ? kCoarse : 1;
        const uint64_t warps = (L.nTiles + step - 1) / step;
        ip_split_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, stream>>>(
            dA, nA, dB, nB, L.nTiles, step, split, reinterpret_cast<uint64_t*>(w),
            grouped ? L.off_split / 8 : kIpHeader / 8, d_count);
        SI_LAUNCH_CHECK("ip_split_kernel");
        if (fine) {
            const si_status st = launch_dependent(
                ip_fine_kernel, dim3(static_cast<unsigned>(std::min<uint64_t>((L.nTiles + 255) / 256, 65535))),
                dim3(256), 0, stream, dA, dB, L.nTiles, nA + nB, split);
            if (st != SI_OK) return st;
        }
    }
    PhaseTimer timer("sisi_tile", stream);
    const dim3 grid(static_cast<unsigned>(L.nTiles)), block(kIpThreads);
    const uint64_t* csplit = split;
    uint32_t* tile_counts = reinterpret_cast<uint32_t*>(status);
    if (grouped) {
        int per_sm = 0;
        SI_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ip_group_kernel, kIpThreads, 0));
        if (per_sm < 1) return SI_ERR_UNSUPPORTED;
        const uint64_t nGroups = (L.nTiles + kGroup - 1) / kGroup;
        const unsigned ctas =
            static_cast<unsigned>(std::min<uint64_t>(nGroups, static_cast<uint64_t>(sm_count()) * per_sm));
        uint64_t nTiles = L.nTiles;
        void* args[] = {&dA, &nA, &dB, &nB, &csplit, &nTiles, &header, &status, &d_out, &out_cap, &d_count};
        SI_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(ip_group_kernel), dim3(ctas), block, args,
                                                0, stream));
        return SI_OK;
    }
    if (L.nTiles == 1) {
        const auto kernel = d_out ? ip_tile_kernel<kPlace> : ip_tile_kernel<kCount>;
        kernel<<<grid, block, 0, stream>>>(dA, nA, dB, nB, csplit, L.nTiles, header, tile_counts, d_out, out_cap,
                                           d_count);
        SI_LAUNCH_CHECK("ip_tile_kernel");
        return SI_OK;
    }
    const si_status st =
        launch_dependent(d_out ? ip_tile_kernel<kTileCounts> : ip_tile_kernel<kCount>, grid, block, 0, stream, dA, nA,
                         dB, nB, csplit, L.nTiles, header, tile_counts, d_out, out_cap, d_count);
    if (st != SI_OK || !d_out) return st;
    return launch_dependent(ip_tile_kernel<kPlace>, grid, block, 0, stream, dA, nA, dB, nB, csplit, L.nTiles, header,
                            tile_counts, d_out, out_cap, d_count);
}

}  // namespace si
