// si_batch.cu -- counts of a batch of uneven pairs of one collection in one
// persistent launch.
//
// The reference has no batched mode: every pair is a host-loop iteration with
// its own launches (src/ip.cu:141-177 for one tile pair; a single pair costs
// the 3-kernel SISI path).  Here a list of (a, b) pairs of a CSR collection is
// counted by two persistent kernels over one work queue:
//
//  * Work queue: the pairs are ordered by class of estimated cost, largest
//    first (a counting sort of 12-bit keys: kernel, cost class, a hash of the
//    larger set, whose pairs then find it in L2), merge
//    and search pairs first, hash and bitmap pairs after them; every warp takes
//    the next pair of its kernel's part from an atomic ticket, so the long
//    pairs start first and the short ones fill the tail.  Pairs that are a
//    good part of a warp's share of all the work are first taken by whole CTAs,
//    each warp an eighth of the larger set's range.  The merge / search
//    kernel runs 32 warps per SM (search is latency-bound), the hash / bitmap
//    kernel 24 with 8 KiB of shared memory each; the second starts as the first
//    one's CTAs end.
//  * Six technique codes per pair, picked per bucket of (density class of the
//    larger set, log2 of the smaller size, log2 of the size ratio) from a
//    1024-entry table:
//      MERGE (ip): the warp takes a window of 256 elements of each set into
//        shared memory; every round finalises the elements up to the smaller of
//        the two window maxima and merges them along the merge path (each lane
//        an equal share of the merged positions after a split search, as the
//        reference's intersectPath splits a partition, src/ip.cu:207-245), while
//        the next windows are loaded into registers.
//      SEARCH (obs): sets of similar size stream the larger one through shared
//        memory, the smaller one's elements searching its windows.  Otherwise
//        the warp takes the smaller set 256 elements at a time, bounds the
//        window of the larger set that can hold them, caches 256 samples of a
//        long window in shared memory, and every lane runs 8 interleaved binary
//        searches in the gaps between samples.
//      HASH (hi, windows of 1024 or 512 elements): the smaller set S is cut
//        into windows of consecutive elements; each window goes into the
//        warp's 2048-slot open-addressing table (load <= 1/2 or 1/4) and the
//        elements of the larger set up to the window's last value probe it
//        (src/hi.cu:361-418 hashes one partition the same way).
//      BITMAP (windows of 16384 or 32768 values): both sets set bits in the
//        warp's two bitmaps of the window's values and the AND's popcount is
//        the window's count; the next window starts at the larger of the two
//        sets' next elements (src/bitmap_dynamic.cu:279-319 probes a set's
//        bitmap; this is the window form of si_sisi_bitmap.cu's engine).
//    HASH and BITMAP read both sets as 256-element streams (si_stream.cuh).
//  * The table comes from si_batch_tune, which times every technique on a
//    sample of every populated bucket, or the default rule.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "si_device.cuh"
#include "si_internal.h"
#include "si_stream.cuh"

namespace si {
namespace {

constexpr int kBThreads = 256;           // 8 warps
constexpr int kBWarps = kBThreads / 32;
// Two kernels share the queue: the merge / search one (64 registers a thread,
// 32 KiB of windows: 4 CTAs, 32 warps per SM; search is latency-bound and wants
// the warps) and the stream one for hash and bitmap (80 registers, 8 KiB a
// warp: 3 CTAs, 24 warps per SM).
constexpr int kSearchCtasPerSm = 4;
constexpr int kStreamCtasPerSm = 3;
constexpr uint32_t kWarpSmem = 8192;     // stream kernel: shared bytes per warp, hash table or bitmaps
constexpr uint32_t kBSmem = kBWarps * kWarpSmem + 4096;  // + the skew to a 4 KiB boundary
constexpr uint32_t kW = 256;             // window (block) per set per round
constexpr int kVT = kW / 32;             // elements per lane per block
// header: [0..16) error words, then per kernel (merge / search, stream) u32
// tickets of the warps [16, 24) and of the CTAs [24, 32), u32 pairs in the
// queue's first part (merge / search) [32], u64 cost of each part [40, 56)
constexpr size_t kBatchHeader = 256;
constexpr size_t kWarpTicket = 16, kCtaTicket = 24, kNFirst = 32, kPartCost = 40;
// technique codes: the table's bytes (si.h SI_BATCH_*)
constexpr uint8_t kMerge = 0, kSearch = 1, kHash1024 = 2, kHash512 = 3, kBitmap16K = 4, kBitmap32K = 5;
constexpr uint8_t kTechCodes = 6;
constexpr uint32_t kTableSize = 1024;    // 4 density classes x 16 size classes x 16 ratio classes

// The queue's bins: part (1 bit), falling cost class (7 bits), a hash of the
// larger set (4 bits), so that the pairs of a set run close together in time and
// find it in L2.  A pair's 16-bit key has its technique above the bin.  shift = 1
// leaves out the hash's last bit.
constexpr uint32_t kBins = 4096;
__host__ __device__ constexpr uint32_t key_bin(uint32_t key, uint32_t shift) { return (key & (kBins - 1)) >> shift; }
__host__ __device__ constexpr uint32_t key_class(uint32_t key) { return 127u - ((key >> 4) & 127u); }
__host__ __device__ constexpr uint8_t key_tech(uint32_t key) { return static_cast<uint8_t>((key >> 12) & 7u); }
constexpr int kKeyThreads = 256;
constexpr uint32_t kKeyPairs = 4;  // pairs per thread of the key and queue kernels
// Up to kPlanMost pairs are ordered by one CTA, whose histogram needs no room
// outside it, and up to kHalfBins the others' has half of the bins: two 64-bit
// words a pair of workspace are enough for a batch of any size.  A whole call,
// one CTA against two kernels: 1 short pair 16.5 us against 17.2, 1000 pairs 20.7
// and 24.6, 3000 26.4 and 26.2, 4500 29.5 and 27.3.  200000 pairs with half of the
// bins: 8.48 ms against 8.39.
constexpr int kPlanThreads = 1024;
constexpr uint32_t kPlanPairs = 3;  // per thread
constexpr uint64_t kPlanMost = uint64_t(kPlanThreads) * kPlanPairs;
constexpr uint64_t kHalfBins = 8192;

struct BatchLayout {
    uint32_t shift = 0;
    size_t off_hist = 0, off_cursor = 0, off_bins = 0, off_queue = 0, total = 0;
};

BatchLayout batch_layout(uint64_t npairs) {
    BatchLayout L;
    L.shift = npairs <= kHalfBins ? 1 : 0;
    const size_t bins = npairs > kPlanMost ? kBins >> L.shift : 0;
    size_t o = kBatchHeader;
    L.off_hist = o;    o += bins * 4;  // the header, the histogram and the cursors start at zero
    L.off_cursor = o;  o += bins * 4;
    L.off_bins = o;    o = align_up(o + npairs * 2, 256);
    L.off_queue = o;   o = align_up(o + npairs * 8, 256);
    L.total = o;
    return L;
}

// Class of a cost: its exponent and two more bits (a class spans a quarter of
// its cost).
__device__ __forceinline__ uint32_t cost_class(uint64_t cost) {
    const uint32_t c = static_cast<uint32_t>(min(cost, uint64_t(0xffffffffu)));
    if (c < 4) return c;
    const uint32_t e = 31 - __clz(c);
    return (e - 1) * 4 + ((c >> (e - 2)) & 3u);
}

__host__ __device__ inline uint32_t log2_floor(uint64_t x) {  // x >= 1
#ifdef __CUDA_ARCH__
    return 63u - static_cast<uint32_t>(__clzll(static_cast<long long>(x)));
#else
    uint32_t r = 0;
    while (x >>= 1) ++r;
    return r;
#endif
}

// Density class of a set from its first and last values and size: the mean
// gap between consecutive values is < 4, < 32, < 256 or larger (class 0..3).
__host__ __device__ inline uint32_t density_class(uint32_t first, uint32_t last, uint64_t n) {
    if (n < 2) return 3;
    const uint64_t gap = static_cast<uint64_t>(last - first) / (n - 1);
    return gap < 4 ? 0u : gap < 32 ? 1u : gap < 256 ? 2u : 3u;
}

// Bucket of a pair: (density class of the larger set, log2 of the smaller
// size, log2 of larger / smaller): 2 + 4 + 4 bits.
__host__ __device__ inline uint32_t pair_bucket(uint64_t na, uint64_t nb, uint32_t dclass) {
    const uint64_t s = na < nb ? na : nb, l = na < nb ? nb : na;
    const uint32_t ls = s ? min(15u, log2_floor(s)) : 0u;
    const uint32_t lr = s ? min(15u, log2_floor(l / s)) : 15u;
    return (dclass << 8) | (ls << 4) | lr;
}

struct TechTable {
    uint8_t t[kTableSize];
};

// Costs are in warp instructions, about: a merge takes one per element; the
// streamed search two per element of the smaller set and a quarter per element
// of the larger; the sampled search eight per element.
constexpr uint64_t kStreamRatio = 32;  // below this ratio a search streams the larger set
__device__ __forceinline__ uint64_t search_cost(uint64_t s, uint64_t l) {
    return l < kStreamRatio * s ? 2 * s + l / 4 : 8 * s;
}

struct PairSets {
    uint64_t a0, na, b0, nb;
};

__device__ __forceinline__ PairSets pair_sets(const uint64_t* off, uint32_t a, uint32_t b) {
    PairSets p;
    p.a0 = off[a];
    p.na = off[a + 1] - p.a0;
    p.b0 = off[b];
    p.nb = off[b + 1] - p.b0;
    return p;
}

// The pair's bucket: its larger set's density class comes from that set's end values.
__device__ __forceinline__ uint32_t device_bucket(const uint32_t* el, const PairSets& p) {
    const bool a_large = p.na >= p.nb;
    const uint64_t l0 = a_large ? p.a0 : p.b0, nl = a_large ? p.na : p.nb;
    const uint32_t dc = nl >= 2 ? density_class(__ldg(el + l0), __ldg(el + l0 + nl - 1), nl) : 3u;
    return pair_bucket(p.na, p.nb, dc);
}

__host__ __device__ constexpr bool is_stream_tech(uint8_t t) { return t >= kHash1024 && t < kTechCodes; }

// A pair's key and cost.  A stream technique falls back to merge for a pair whose
// larger set has 2^32 - 1024 elements or more (stream positions are 32-bit).
__device__ __forceinline__ uint32_t pair_key(const uint32_t* __restrict__ el, const uint64_t* __restrict__ off,
                                             const uint32_t* __restrict__ pairs, uint64_t p, uint32_t k,
                                             const TechTable& table, int forced, unsigned char* header,
                                             uint64_t& cost) {
    const uint32_t a = pairs[2 * p], b = pairs[2 * p + 1];
    cost = 0;
    uint32_t larger = 0;
    uint8_t t = kMerge;
    if (a >= k || b >= k) {
        record_error(reinterpret_cast<uint32_t*>(header), SI_ERR_INVALID_INPUT, 50, static_cast<uint32_t>(p));
    } else {
        const PairSets ps = pair_sets(off, a, b);
        t = forced >= 0 ? static_cast<uint8_t>(forced) : table.t[device_bucket(el, ps)];
        if (t >= kTechCodes || (is_stream_tech(t) && max(ps.na, ps.nb) >= kMaxStream)) t = kMerge;
        cost = t == kSearch ? search_cost(min(ps.na, ps.nb), max(ps.na, ps.nb)) : ps.na + ps.nb;
        larger = ps.na > ps.nb ? a : b;
    }
    return uint32_t(t) << 12 | uint32_t(is_stream_tech(t)) << 11 | (127u - cost_class(cost)) << 4 |
           (larger * 0x9e3779b1u) >> 28;
}
__host__ __device__ constexpr uint32_t key_part(uint32_t key) { return (key >> 11) & 1u; }

// Each pair's key, the bins' histogram and the parts' total cost.
__global__ void __launch_bounds__(kKeyThreads) batch_keys_kernel(
    const uint32_t* __restrict__ el, const uint64_t* __restrict__ off, const uint32_t* __restrict__ pairs,
    uint64_t npairs, uint32_t k, const __grid_constant__ TechTable table, int forced, uint32_t shift,
    uint16_t* __restrict__ bins, uint32_t* __restrict__ hist, unsigned char* header) {
    __shared__ uint32_t s_hist[kBins];
    __shared__ unsigned long long s_cost[2];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (uint32_t i = threadIdx.x; i < kBins >> shift; i += kKeyThreads) s_hist[i] = 0;
    if (threadIdx.x < 2) s_cost[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t p0 = uint64_t(blockIdx.x) * kKeyThreads * kKeyPairs + threadIdx.x;
    uint64_t part_cost[2] = {0, 0};
#pragma unroll
    for (uint32_t u = 0; u < kKeyPairs; ++u) {
        const uint64_t p = p0 + u * kKeyThreads;
        if (p >= npairs) continue;
        uint64_t cost;
        const uint32_t key = pair_key(el, off, pairs, p, k, table, forced, header, cost);
        bins[p] = static_cast<uint16_t>(key);
        atomicAdd(&s_hist[key_bin(key, shift)], 1u);
        part_cost[key_part(key)] += cost;
    }
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        const uint64_t c = warp_sum_u64(part_cost[part]);
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_cost[part], static_cast<unsigned long long>(c));
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kBins >> shift; i += kKeyThreads)
        if (s_hist[i]) atomicAdd(hist + i, s_hist[i]);
    if (threadIdx.x < 2 && s_cost[threadIdx.x])
        atomicAdd(reinterpret_cast<unsigned long long*>(header + kPartCost) + threadIdx.x, s_cost[threadIdx.x]);
}

// The queue of up to kPlanMost pairs, by one CTA.
__global__ void __launch_bounds__(kPlanThreads) batch_plan_kernel(
    const uint32_t* __restrict__ el, const uint64_t* __restrict__ off, const uint32_t* __restrict__ pairs,
    uint32_t npairs, uint32_t k, const __grid_constant__ TechTable table, int forced, uint64_t* __restrict__ queue,
    unsigned char* header) {
    __shared__ __align__(8) uint32_t s_hist[kBins / 2];  // the bins' pairs, then where the next pair of each goes
    __shared__ uint32_t s_warp[kPlanThreads / 32];
    __shared__ unsigned long long s_cost[2];
    constexpr uint32_t kPer = kBins / 2 / kPlanThreads;
    static_assert(kPer == 2, "a thread scans 8 bytes of the histogram");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint2* h2 = reinterpret_cast<uint2*>(s_hist);
    h2[tid] = make_uint2(0u, 0u);
    if (tid < 2) s_cost[tid] = 0;
    __syncthreads();
    uint32_t key[kPlanPairs];
    uint64_t part_cost[2] = {0, 0};
#pragma unroll
    for (uint32_t u = 0; u < kPlanPairs; ++u) {
        const uint32_t p = u * kPlanThreads + tid;
        key[u] = ~0u;
        if (p >= npairs) continue;
        uint64_t cost;
        key[u] = pair_key(el, off, pairs, p, k, table, forced, header, cost);
        atomicAdd(&s_hist[key_bin(key[u], 1)], 1u);
        part_cost[key_part(key[u])] += cost;
    }
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        const uint64_t c = warp_sum_u64(part_cost[part]);
        if (lane == 0 && c) atomicAdd(&s_cost[part], static_cast<unsigned long long>(c));
    }
    __syncthreads();
    const uint2 v = h2[tid];
    const uint32_t sum = v.x + v.y, incl = warp_inclusive_scan(sum);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t o = incl - sum;
    for (uint32_t w = 0; w < warp; ++w) o += s_warp[w];
    h2[tid] = make_uint2(o, o + v.x);
    if (tid < 2) reinterpret_cast<unsigned long long*>(header + kPartCost)[tid] = s_cost[tid];
    if (tid == kPlanThreads / 2) *reinterpret_cast<uint32_t*>(header + kNFirst) = o;
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kPlanPairs; ++u)
        if (key[u] != ~0u)
            queue[atomicAdd(&s_hist[key_bin(key[u], 1)], 1u)] = uint64_t(key[u]) << 32 | (u * kPlanThreads + tid);
}

// The queue: every pair (its key in bits 32.., its index below) at its bin's
// offset.  A CTA scans the histogram itself and reserves room in each bin once;
// the order within a bin does not matter.
__global__ void __launch_bounds__(kKeyThreads) batch_queue_kernel(const uint16_t* bins, uint64_t npairs, uint32_t shift,
                                                                  const uint32_t* hist, uint32_t* __restrict__ cursor,
                                                                  uint64_t* __restrict__ queue,
                                                                  unsigned char* header) {
    __shared__ uint32_t s_off[kBins];    // the bin's offset, then where this CTA's next pair of it goes
    __shared__ uint32_t s_count[kBins];  // this CTA's pairs of the bin
    __shared__ uint32_t s_warp[kKeyThreads / 32];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (uint32_t i = threadIdx.x; i < kBins >> shift; i += kKeyThreads) s_count[i] = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the bins and their histogram
    constexpr uint32_t kPer = kBins / kKeyThreads;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t v[kPer], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q) {
        v[q] = threadIdx.x * kPer + q < kBins >> shift ? hist[threadIdx.x * kPer + q] : 0u;
        sum += v[q];
    }
    const uint32_t incl = warp_inclusive_scan(sum);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t o = incl - sum;
    for (uint32_t w = 0; w < warp; ++w) o += s_warp[w];
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q) {
        s_off[threadIdx.x * kPer + q] = o;
        o += v[q];
    }
    uint32_t key[kKeyPairs];
    const uint64_t p0 = uint64_t(blockIdx.x) * kKeyThreads * kKeyPairs + threadIdx.x;
#pragma unroll
    for (uint32_t u = 0; u < kKeyPairs; ++u) {
        const uint64_t p = p0 + u * kKeyThreads;
        key[u] = p < npairs ? bins[p] : ~0u;
        if (key[u] != ~0u) atomicAdd(&s_count[key_bin(key[u], shift)], 1u);
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<uint32_t*>(header + kNFirst) = s_off[(kBins >> shift) / 2];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kBins >> shift; i += kKeyThreads)
        if (s_count[i]) s_off[i] += atomicAdd(cursor + i, s_count[i]);
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kKeyPairs; ++u)
        if (key[u] != ~0u)
            queue[atomicAdd(&s_off[key_bin(key[u], shift)], 1u)] = uint64_t(key[u]) << 32 | (p0 + u * kKeyThreads);
}

// ------------------------------------------------------ per-warp techniques --
// Elements [i, i + kW) of x (below n) into registers, the next window.
__device__ __forceinline__ void fetch_window(const uint32_t* x, uint64_t i, uint64_t n, uint32_t lane,
                                             uint32_t (&r)[kVT]) {
#pragma unroll
    for (int t = 0; t < kVT; ++t) {
        const uint64_t k = i + lane + 32u * t;
        r[t] = k < n ? __ldg(x + k) : 0xffffffffu;
    }
}

__device__ __forceinline__ void store_window(uint32_t* w, uint32_t lane, const uint32_t (&r)[kVT]) {
#pragma unroll
    for (int t = 0; t < kVT; ++t) w[lane + 32u * t] = r[t];
}

// Number of a window's kW elements that are <= v (v below its end marks),
// warp-cooperative: lane l tests element 8 l, then the first eight lanes the
// elements of the one group of eight the answer ends in (two shared loads and
// two ballots per lane).  Every lane gets the result.
__device__ __forceinline__ uint32_t window_count_le(const uint32_t* w, uint32_t v, uint32_t lane) {
    const uint32_t k = __popc(__ballot_sync(kFullMask, w[8 * lane] <= v));
    if (k == 0) return 0;
    const bool c = lane < 8 && w[8 * (k - 1) + (lane & 7)] <= v;
    return 8 * (k - 1) + __popc(__ballot_sync(kFullMask, c));
}

// MERGE: |A ∩ B|, a window of kW elements of each set at a time in the warp's
// shared memory (kMergeWords words).  A round finalises the elements of both
// windows up to the smaller window maximum and merges them along the merge path
// (each lane an equal share of the merged positions after a split search; ties
// to A), while the windows that start after them are already being loaded into
// registers.  Neither set holds 2^32 - 1 here (matched apart), which marks the
// positions past a set's or a window's end.
//
// A merge step is eight instructions, a round of some 500 elements of sets of
// similar size about 330.  200000 pairs of 20000 sets of 32 .. 2^18 elements, all
// merged (most of very different sizes): 1.35 warp instructions per element,
// 15.1 ms, bound by issue and the shared-memory pipe (100000 pairs of 10000 such
// sets: 90 % of issue slots, 88 % of the LSU's data pipe); rings of
// blocks with masked indexes and clamped ends took 2.7 and 21.6 ms.
constexpr uint32_t kMergeWords = 2 * (kW + 32);  // per set: the window, then end marks that a lane's steps may run into
__device__ uint32_t merge_pair(const uint32_t* A, uint64_t na, const uint32_t* B, uint64_t nb, uint32_t* win,
                               uint32_t lane) {
    if (na == 0 || nb == 0) return 0;
    const uint32_t last_a = __ldg(A + na - 1), last_b = __ldg(B + nb - 1);
    uint32_t hits = lane == 0 && last_a == 0xffffffffu && last_b == 0xffffffffu ? 1u : 0u;
    na -= last_a == 0xffffffffu;
    nb -= last_b == 0xffffffffu;
    if (na == 0 || nb == 0 || last_a < __ldg(B) || last_b < __ldg(A))  // nothing else, or value ranges apart
        return __reduce_add_sync(kFullMask, hits);
    uint32_t* wa = win;
    uint32_t* wb = win + kW + 32;
    wa[kW + lane] = 0xffffffffu;
    wb[kW + lane] = 0xffffffffu;
    uint32_t ra[kVT], rb[kVT];
    uint64_t ia = 0, ib = 0;
    fetch_window(A, 0, na, lane, ra);
    fetch_window(B, 0, nb, lane, rb);
    for (;;) {
        __syncwarp();  // the last round's windows have been read
        store_window(wa, lane, ra);
        store_window(wb, lane, rb);
        __syncwarp();
        // a window that ends with its set holds end marks: its last element is
        // then the largest value, and the other window bounds the round
        const uint32_t max_a = wa[kW - 1], max_b = wb[kW - 1], m = min(max_a, max_b);
        const bool last_round = m == 0xffffffffu;  // both sets end in these windows
        const uint32_t cA = max_a <= m && !last_round ? kW : window_count_le(wa, m - (last_round ? 1u : 0u), lane);
        const uint32_t cB = max_b <= m && !last_round ? kW : window_count_le(wb, m - (last_round ? 1u : 0u), lane);
        ia += cA;
        ib += cB;
        // both sets end in a last round's windows; in sets padded with 2^32 - 1
        // it may take nothing, so it also ends the loop
        const bool more = !last_round && ia < na && ib < nb;
        if (more) {  // the next windows, in flight during the merge
            fetch_window(A, ia, na, lane, ra);
            fetch_window(B, ib, nb, lane, rb);
        }
        // lane l takes merged positions [st l, st l + st) of the cA + cB (<= 512);
        // st is odd, so that the lanes' reads spread over the banks
        const uint32_t tot = cA + cB, st = (tot + 31) / 32 | 1;
        const uint32_t d = min(st * lane, tot), steps = min(st, tot - d);
        uint32_t lo = d > cB ? d - cB : 0u, hi = min(d, cA);
        while (lo < hi) {  // the first a with A[a] > B[d - 1 - a]
            const uint32_t mid = (lo + hi) >> 1;
            const bool right = wa[mid] <= wb[d - 1 - mid];
            lo = right ? mid + 1 : lo;
            hi = right ? hi : mid;
        }
        uint32_t pa = smem_addr(wa + lo), pb = smem_addr(wb + (d - lo));
        uint32_t a = lds_u32(pa), b = lds_u32(pb);
#pragma unroll 4
        for (uint32_t x = 0; x < st; ++x) {  // warp-uniform
            if (a == b && x < steps) ++hits;
            if (a <= b) {
                pa += 4;
                a = lds_u32(pa);
            } else {
                pb += 4;
                b = lds_u32(pb);
            }
        }
        if (!more) break;
    }
    return __reduce_add_sync(kFullMask, hits);
}

// SEARCH of sets of similar size (the larger below kStreamRatio times the
// smaller): L streams through shared memory in windows of kSWin elements, the
// next one landing (cp.async, 16 bytes a lane, coalesced) while the elements of
// S up to the window's last value are binary-searched in this one, 32 at a time.
// Reads every element of L once, 4 nl / ns bytes per element of S, where the
// sampled search below takes some six random sectors; per element of S 2.4 warp
// instructions at a ratio of 4 and 6 at 32, against 6.4.  The same pairs, all
// searched: 9.6 ms with both, 15.2 ms with the sampled search alone.
constexpr uint32_t kSWin = 512;
constexpr uint32_t kSearchWords = 2 * kSWin;  // per warp
static_assert(kSearchWords >= kMergeWords, "one region serves both");
__device__ uint32_t stream_search_pair(const uint32_t* S, uint64_t ns, const uint32_t* L, uint64_t nl, uint32_t* win,
                                       uint32_t lane) {
    const uint32_t lo_v = max(__ldg(S), __ldg(L));
    if (__ldg(S + ns - 1) < lo_v || __ldg(L + nl - 1) < lo_v) return 0;  // value ranges apart
    const uint64_t s0 = warp_first_true(0, ns, [&](uint64_t i) { return __ldg(S + i) >= lo_v; });
    const uint64_t l0 = warp_first_true(0, nl, [&](uint64_t i) { return __ldg(L + i) >= lo_v; });
    // positions count from the 16-byte boundary below L[l0]; elements are [v0, v1)
    const uint32_t v0 = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(L + l0) & 15u) >> 2);
    const uint32_t* base = L + l0 - v0;
    const uint32_t v1 = v0 + static_cast<uint32_t>(nl - l0), last_group = (v1 - 1) & ~3u;
    const uint32_t at = smem_addr(win) + 16 * lane;
    auto issue = [&](uint32_t w) {  // window w into its half; groups past the last read it again
#pragma unroll
        for (uint32_t q = 0; q < kSWin / 128; ++q)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + (w & 1) * kSWin * 4 + q * 512),
                         "l"(base + min(w * kSWin + q * 128 + 4 * lane, last_group))
                         : "memory");
    };
    uint64_t is = s0;
    uint32_t hits = 0;
    uint32_t v = is + lane < ns ? __ldg(S + is + lane) : 0xffffffffu;
    const uint32_t windows = (v1 + kSWin - 1) / kSWin;
    issue(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (uint32_t w = 0; w < windows && is < ns; ++w) {
        if (w + 1 < windows) issue(w + 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        uint32_t* sm = win + (w & 1) * kSWin;
        // positions that are no elements get copies of the nearest one
        if (w == 0 && lane < v0) sm[lane] = sm[v0];
        if (w + 1 == windows) {
            const uint32_t n = v1 - w * kSWin, last = sm[n - 1];
            __syncwarp();
            for (uint32_t x = n + lane; x < kSWin; x += 32) sm[x] = last;
        }
        __syncwarp();
        const uint32_t top = sm[kSWin - 1];
        for (;;) {
            const bool valid = is + lane < ns && v <= top;
            const uint32_t n = __popc(__ballot_sync(kFullMask, valid));  // valid lanes are a prefix
            if (n) {
                uint32_t pos = 0;
#pragma unroll
                for (uint32_t step = kSWin / 2; step > 0; step >>= 1) pos = sm[pos + step] <= v ? pos + step : pos;
                hits += valid && sm[pos] == v ? 1u : 0u;
                is += n;
                v = is + lane < ns ? __ldg(S + is + lane) : 0xffffffffu;
            }
            if (n < 32) break;
        }
        __syncwarp();  // the half is read before the window after next lands in it
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    return __reduce_add_sync(kFullMask, hits);
}

// SEARCH: every element of the smaller set S, binary-searched in the larger
// L, 256 elements of S at a time.  The window of L that can hold the block
// comes from two 32-ary warp searches; a window longer than 512 elements is
// sampled at 256 evenly spaced positions into shared memory (one load round
// for the warp, the cached top of the search tree, as the reference's obs
// caches it, src/obs.cu:275-438), every element finds its gap between two
// samples there, and only the gap is searched in global memory, 8 searches
// interleaved per lane.  samp: the warp's 256 words of shared memory.
constexpr uint32_t kSample = 256;
__device__ uint32_t search_pair(const uint32_t* S, uint64_t ns, const uint32_t* L, uint64_t nl, uint32_t* samp,
                               int lane) {
    if (ns == 0 || nl == 0) return 0;
    if (ns >= 32 && nl < kStreamRatio * ns && nl < kMaxStream) return stream_search_pair(S, ns, L, nl, samp, lane);
    uint32_t hits = 0;
    uint64_t from = 0;  // the windows advance monotonically
    for (uint64_t base = 0; base < ns; base += kW) {
        const uint64_t last_i = min(base + kW, ns) - 1;
        // a smaller set of one block searches all of L (its samples bound the
        // gaps as well as a narrowed window would, without the two searches)
        // later blocks start where the previous one's window ended (the L
        // elements between are below this block's first value: harmless)
        uint64_t lo = 0, hi = nl;
        if (ns > kW) {
            const uint32_t v1 = __ldg(S + last_i);
            if (base == 0) {
                const uint32_t v0 = __ldg(S);
                lo = warp_first_true(0, nl, [&](uint64_t i) { return __ldg(L + i) >= v0; });
            } else {
                lo = from;
            }
            hi = warp_first_true(lo, nl, [&](uint64_t i) { return __ldg(L + i) > v1; });
        }
        from = hi;
        if (lo >= hi) continue;
        const uint64_t W = hi - lo;
        const bool sampled = W > 2 * kSample;
        if (sampled) {
#pragma unroll
            for (uint32_t t = 0; t < kSample / 32; ++t) {
                const uint32_t j = lane + 32 * t;
                samp[j] = __ldg(L + lo + W * j / kSample);
            }
            __syncwarp();
        }
        if (W >= (uint64_t(1) << 32)) {  // a window past 32-bit offsets: one plain search after another
            for (uint32_t t = 0; t < kVT; ++t) {
                const uint64_t i = base + lane + 32u * t;
                if (i > last_i) break;
                const uint32_t v = __ldg(S + i);
                uint64_t p = lo, len = W;
                while (len > 1) {
                    const uint64_t half = len >> 1;
                    const bool c = __ldg(L + p + half) <= v;
                    p = c ? p + half : p;
                    len = c ? len - half : half;
                }
                hits += __ldg(L + p) == v ? 1u : 0u;
            }
            __syncwarp();  // the samples are not read, and written again by the next block
            continue;
        }
        const uint32_t* Lw = L + lo;
        const uint32_t W32 = static_cast<uint32_t>(W);
        uint32_t v[kVT], o32[kVT], n32[kVT];
#pragma unroll
        for (int t = 0; t < kVT; ++t) {
            const uint64_t i = base + lane + 32u * t;
            v[t] = i <= last_i ? __ldg(S + i) : 0u;
            o32[t] = 0;
            n32[t] = i <= last_i ? W32 : 0u;
        }
        if (sampled) {
#pragma unroll
            for (int t = 0; t < kVT; ++t) {
                // c = samples <= v; the answer lies between samples c - 1 and c
                uint32_t c = 0;
#pragma unroll
                for (uint32_t step = kSample / 2; step > 0; step >>= 1)
                    c = samp[c + step - 1] <= v[t] ? c + step : c;
                c = (c == kSample - 1 && samp[kSample - 1] <= v[t]) ? kSample : c;
                const uint32_t p0 = static_cast<uint32_t>(uint64_t(W32) * (c ? c - 1 : 0) / kSample);
                const uint32_t p1 = static_cast<uint32_t>(uint64_t(W32) * c / kSample);  // W32 for c == kSample
                o32[t] = p0;
                n32[t] = c == 0 || n32[t] == 0 ? 0u : p1 - p0;  // c == 0: v is below L[lo]
            }
            __syncwarp();  // the samples are read before the next block writes them
        }
        // interleaved searches for the last element <= v: kVT independent load
        // chains per lane; 4-ary steps (three independent loads, a quarter of the
        // gap left) while the gap allows, then binary: half the dependent load
        // rounds of a binary search
        bool more = true;
        while (more) {
            more = false;
#pragma unroll
            for (int t = 0; t < kVT; ++t) {
                const uint32_t n = n32[t];
                if (n >= 4) {
                    const uint32_t q1 = n >> 2, q2 = n >> 1, q3 = q1 + q2;
                    const uint32_t o = o32[t];
                    const bool c1 = __ldg(Lw + o + q1) <= v[t];
                    const bool c2 = __ldg(Lw + o + q2) <= v[t];
                    const bool c3 = __ldg(Lw + o + q3) <= v[t];
                    const uint32_t lo_q = c3 ? q3 : c2 ? q2 : c1 ? q1 : 0u;
                    const uint32_t hi_q = c3 ? n : c2 ? q3 : c1 ? q2 : q1;
                    o32[t] = o + lo_q;
                    n32[t] = hi_q - lo_q;
                    more |= n32[t] > 1;
                } else if (n > 1) {
                    const uint32_t half = n >> 1;
                    const bool c = __ldg(Lw + o32[t] + half) <= v[t];
                    o32[t] = c ? o32[t] + half : o32[t];
                    n32[t] = c ? n - half : half;
                    more |= n32[t] > 1;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < kVT; ++t) hits += (n32[t] == 1 && __ldg(Lw + o32[t]) == v[t]) ? 1u : 0u;
    }
    return __reduce_add_sync(kFullMask, hits);
}

// ---------------------------------------------------------------- HASH --
// HASH: |S ∩ L| (S the smaller set), windows of kWinChunks chunks of S.
template <uint32_t kWinChunks>
__device__ uint32_t hash_pair(const uint32_t* S, uint64_t ns, const uint32_t* L, uint64_t nl, uint32_t* tab,
                              uint32_t lane) {
    static_assert(kWinChunks * kChunk <= kWinHashSlots / 2, "a window fills at most half of the table");
    if (ns == 0 || nl == 0) return 0;
    // the value 2^32 - 1 marks empty slots: a match of it is counted here and
    // it leaves both sets (it can only be their last element)
    const bool s_top = __ldg(S + ns - 1) == kWinHashEmpty, l_top = __ldg(L + nl - 1) == kWinHashEmpty;
    const uint32_t extra = s_top && l_top ? 1u : 0u;
    ns -= s_top;
    nl -= l_top;
    if (ns == 0 || nl == 0) return extra;
    const uint32_t lo = max(__ldg(S), __ldg(L));
    if (__ldg(S + ns - 1) < lo || __ldg(L + nl - 1) < lo) return extra;  // value ranges apart
    const uint64_t s0 = warp_first_true(0, ns, [&](uint64_t i) { return __ldg(S + i) >= lo; });
    const uint64_t l0 = warp_first_true(0, nl, [&](uint64_t i) { return __ldg(L + i) >= lo; });
    SetStream ss, sl;
    stream_init(ss, S, s0, ns, lane);
    stream_init(sl, L, l0, nl, lane);
    const uint32_t lv0 = sl.v1 - static_cast<uint32_t>(nl - l0);  // L's first stream position
    uint4* tab4 = reinterpret_cast<uint4*>(tab);
    uint32_t hits = 0;
    for (;;) {
        for (uint32_t i = lane; i < kWinHashSlots / 4; i += 32)
            tab4[i] = make_uint4(kWinHashEmpty, kWinHashEmpty, kWinHashEmpty, kWinHashEmpty);
        __syncwarp();
        // the window: the next kWinChunks chunks of S, up to its last value hi
        uint32_t hi = 0;
        bool more_s = true;
        for (uint32_t c = 0; c < kWinChunks && more_s; ++c) {
            if (ss.ph == 0)
                chunk_hash_insert(tab, ss.a0, ss.a1);
            else
                chunk_hash_insert(tab, ss.b0, ss.b1);
            hi = ss.last;
            more_s = stream_next(ss, lane);
        }
        __syncwarp();
        // L's elements up to hi probe it; a chunk reaching past hi stays
        bool more_l = true;
        for (;;) {
            if (sl.ph == 0)
                hits += __popc(chunk_hash_probe(tab, sl.a0, sl.a1, probe_mask(sl, sl.a0, sl.a1, lv0, hi, lane)));
            else
                hits += __popc(chunk_hash_probe(tab, sl.b0, sl.b1, probe_mask(sl, sl.b0, sl.b1, lv0, hi, lane)));
            if (sl.last > hi) break;
            more_l = stream_next(sl, lane);
            if (!more_l) break;
        }
        if (!more_l || !more_s) break;
        __syncwarp();  // the probes are done before the table is cleared
    }
    return __reduce_add_sync(kFullMask, hits) + extra;
}

// -------------------------------------------------------------- BITMAP --
// BITMAP: |X ∩ Y| by windows of 32 kWords values; bmx: the warp's two
// kWords-word bitmaps (bmx, bmx + kWords), each aligned to its size.
template <uint32_t kWords>
__device__ uint32_t bitmap_pair(const uint32_t* X, uint64_t nx, const uint32_t* Y, uint64_t ny, uint32_t* bmx,
                                uint32_t lane) {
    constexpr uint32_t kWinV = 32 * kWords;
    if (nx == 0 || ny == 0) return 0;
    const uint32_t lo = max(__ldg(X), __ldg(Y));
    if (__ldg(X + nx - 1) < lo || __ldg(Y + ny - 1) < lo) return 0;  // value ranges apart
    uint4* bx4 = reinterpret_cast<uint4*>(bmx);
    uint4* by4 = reinterpret_cast<uint4*>(bmx + kWords);
    for (uint32_t i = lane; i < kWords / 2; i += 32) bx4[i] = make_uint4(0u, 0u, 0u, 0u);  // both bitmaps
    const uint64_t x0 = warp_first_true(0, nx, [&](uint64_t i) { return __ldg(X + i) >= lo; });
    const uint64_t y0 = warp_first_true(0, ny, [&](uint64_t i) { return __ldg(Y + i) >= lo; });
    SetStream sx, sy;
    stream_init(sx, X, x0, nx, lane);
    stream_init(sy, Y, y0, ny, lane);
    const uint32_t sbx = smem_addr(bmx), sby = smem_addr(bmx + kWords);
    uint32_t a = max(__ldg(X + x0), __ldg(Y + y0));
    uint32_t hits = 0;
    __syncwarp();
    for (;;) {
        const uint64_t e = static_cast<uint64_t>(a) + kWinV;
        const uint32_t lim = e > 0xffffffffull ? static_cast<uint32_t>(0x100000000ull - a) : kWinV;
        const bool more_x = stream_fill<kWords>(sx, sbx, a, lim, e, lane);
        const bool more_y = stream_fill<kWords>(sy, sby, a, lim, e, lane);
        __syncwarp();
#pragma unroll
        for (uint32_t h = 0; h < kWords / 128; ++h) {
            const uint32_t i = 32 * h + lane;
            const uint4 p = bx4[i], q = by4[i];
            bx4[i] = make_uint4(0u, 0u, 0u, 0u);
            by4[i] = make_uint4(0u, 0u, 0u, 0u);
            hits += __popc(p.x & q.x) + __popc(p.y & q.y) + __popc(p.z & q.z) + __popc(p.w & q.w);
        }
        __syncwarp();
        if (!more_x || !more_y) break;
        a = max(stream_first_from(sx, e), stream_first_from(sy, e));
    }
    return __reduce_add_sync(kFullMask, hits);
}

// --------------------------------------------------------------- kernel --
struct BatchParams {
    const uint32_t* el;
    const uint64_t* off;
    const uint32_t* pairs;
    uint32_t k;
    const uint64_t* queue;   // key in bits 32.., pair index below
    const uint32_t* subset;  // when non-null: the queue is these pair indices, in order, all by `forced`
    uint64_t nqueue;         // queue length (all pairs, or the subset)
    uint32_t* counts;
    unsigned char* header;
    int forced;
    bool first;              // the first kernel after the queue's
};

// |S ∩ L| by one warp.
template <bool kStream>
__device__ __forceinline__ uint32_t count_pair(uint8_t tech, const uint32_t* S, uint64_t ns, const uint32_t* L,
                                               uint64_t nl, uint32_t* region, uint32_t lane) {
    if constexpr (kStream) {
        if (nl >= kMaxStream) tech = kMerge;  // only reachable with a tuner subset
        switch (tech) {
            case kMerge: return merge_pair(S, ns, L, nl, region, lane);
            case kHash512: return hash_pair<2>(S, ns, L, nl, region, lane);
            case kBitmap16K: return bitmap_pair<512>(L, nl, S, ns, region, lane);
            case kBitmap32K: return bitmap_pair<1024>(L, nl, S, ns, region, lane);
            default: return hash_pair<4>(S, ns, L, nl, region, lane);
        }
    } else {
        return tech == kSearch ? search_pair(S, ns, L, nl, region, lane) : merge_pair(S, ns, L, nl, region, lane);
    }
}

// Pairs of more than a kCoopShare-th of a warp's share of the part's cost are
// taken by whole CTAs when they are worth the searches that divide them.  Their
// warps would otherwise hold up the end.  Merge and search, shares of 1/2, 2 and
// 8 warps' work: 20000 pairs of 5000 sets of up to 2^18 elements 1.88, 1.25 and
// 1.04 ms by the default rule (12.1 without), 2000 pairs 0.29, 0.30 and 0.28 ms
// (10.1); 200000 pairs by search 16.3, 15.4 and 15.2 ms (15.3).  Hash and bitmap:
// 11.5, 6.2 and 5.1 ms, and 8.3, 8.2 and 9.2 ms for the 20000.
constexpr uint64_t kCoopCost = 8192;
template <bool kStream>
constexpr uint64_t kCoopShareOf = kStream ? 2 : 8;

// One kernel per part of the queue.  kStream = false: merge and search pairs
// (the first part), windows in static shared memory; kStream = true: hash and
// bitmap pairs (the rest), 8 KiB of dynamic shared memory per warp.  With a
// subset (the tuner) the kernel of the forced technique takes it all.
template <bool kStream>
__global__ void __launch_bounds__(kBThreads, kStream ? kStreamCtasPerSm : kSearchCtasPerSm)
    batch_kernel(BatchParams p) {
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ uint32_t s_q, s_hits[kBWarps];
    // the part of the queue left, in shared memory: the counting below wants the registers
    __shared__ uint64_t s_q0, s_q1;
    __shared__ uint32_t s_class;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // stream kernel: the warp's 8 KiB, 4 KiB aligned (the bitmaps' word
    // addresses are one LOP3); merge / search kernel: the warp's two windows
    uint32_t* region;
    if constexpr (kStream) {
        const uint32_t skew = ((smem_addr(smem) + 4095u) & ~4095u) - smem_addr(smem);
        region = smem + skew / 4 + warp * (kWarpSmem / 4);
    } else {
        __shared__ __align__(16) uint32_t windows[kBWarps][kSearchWords];
        region = windows[warp];
    }
    // the queue is ready when its kernel's first successor runs; the second one
    // may then start while the first one's last CTAs run.  It has not waited for
    // the queue's kernel itself, so it (the stream kernel) reads the queue from
    // L2, where it lies whole
    if (p.first) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        uint64_t q0 = 0, q1 = p.nqueue;
        uint32_t cls = 0;
        if (!p.subset) {
            const uint32_t nf = *reinterpret_cast<const volatile uint32_t*>(p.header + kNFirst);
            q0 = kStream ? nf : 0;
            q1 = kStream ? p.nqueue : nf;
            const uint64_t cost = reinterpret_cast<const volatile uint64_t*>(p.header + kPartCost)[kStream];
            cls = cost_class(max(kCoopCost, cost / kCoopShareOf<kStream> / (uint64_t(gridDim.x) * kBWarps)));
        }
        s_q0 = q0;
        s_q1 = q1;
        s_class = cls;
    }
    __syncthreads();
    auto key_of = [&](uint64_t q) { return kStream ? ld_relaxed_u64(p.queue + q) : p.queue[q]; };
    auto is_small = [&](uint64_t q) { return key_class(static_cast<uint32_t>(key_of(q) >> 32)) < s_class; };
    bool coop = !p.subset && s_q0 < s_q1 && !is_small(s_q0);  // CTA-uniform; the queue falls in cost
    for (;;) {
        uint64_t q;
        if (coop) {
            __syncthreads();
            if (threadIdx.x == 0) s_q = atomicAdd(reinterpret_cast<uint32_t*>(p.header + kCtaTicket) + kStream, 1u);
            __syncthreads();
            q = s_q0 + s_q;
            if (q >= s_q1 || is_small(q)) {  // the rest goes to the warps
                coop = false;
                const uint64_t q0 = warp_first_true(s_q0, s_q1, is_small);
                __syncthreads();
                if (threadIdx.x == 0) s_q0 = q0;
                __syncthreads();
                continue;
            }
        } else {
            uint32_t t = 0;
            if (lane == 0) t = atomicAdd(reinterpret_cast<uint32_t*>(p.header + kWarpTicket) + kStream, 1u);
            q = s_q0 + __shfl_sync(kFullMask, t, 0);
            if (q >= s_q1) break;
        }
        uint32_t pi;
        uint8_t tech;
        if (p.subset) {
            pi = p.subset[q];
            tech = static_cast<uint8_t>(p.forced);
        } else {
            const uint64_t key = key_of(q);
            pi = static_cast<uint32_t>(key);
            tech = key_tech(static_cast<uint32_t>(key >> 32));
        }
        const uint32_t a = p.pairs[2 * uint64_t(pi)], b = p.pairs[2 * uint64_t(pi) + 1];
        if (a >= p.k || b >= p.k) continue;  // recorded by the key kernel (cost 0: never taken by a CTA)
        const PairSets ps = pair_sets(p.off, a, b);
        const bool as = ps.na <= ps.nb;  // A is the smaller set
        const uint32_t* S = p.el + (as ? ps.a0 : ps.b0);
        const uint32_t* L = p.el + (as ? ps.b0 : ps.a0);
        uint64_t ns = as ? ps.na : ps.nb, nl = as ? ps.nb : ps.na;
        if (coop) {  // an eighth of L, and the elements of S from its first to the next one's
            const uint64_t l0 = nl * warp / kBWarps, l1 = nl * (warp + 1) / kBWarps;
            uint64_t s0 = 0, s1 = ns;
            if (warp > 0) {
                const uint32_t v = __ldg(L + l0);
                s0 = warp_first_true(0, ns, [&](uint64_t i) { return __ldg(S + i) >= v; });
            }
            if (warp + 1 < kBWarps) {
                const uint32_t v = __ldg(L + l1);
                s1 = warp_first_true(s0, ns, [&](uint64_t i) { return __ldg(S + i) >= v; });
            }
            S += s0;
            L += l0;
            ns = s1 - s0;
            nl = l1 - l0;
            if (ns > nl) {
                const uint32_t* x = S;
                S = L;
                L = x;
                const uint64_t n = ns;
                ns = nl;
                nl = n;
            }
        }
        const uint32_t c = count_pair<kStream>(tech, S, ns, L, nl, region, lane);
        if (coop) {
            if (lane == 0) s_hits[warp] = c;
            __syncthreads();
            if (threadIdx.x == 0) {
                uint32_t sum = 0;
#pragma unroll
                for (int w = 0; w < kBWarps; ++w) sum += s_hits[w];
                p.counts[pi] = sum;
            }
        } else {
            if (lane == 0) p.counts[pi] = c;
            __syncwarp();
        }
    }
    // this kernel does not end before the one it started beside
    if (!p.first) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Default rule, from every technique's time on pairs of each bucket over pools
// of 2^14 .. 2^26 values.  Dense larger sets (mean gap below 32): window bitmaps
// of 32768 values, but search when the smaller set is short or 16 times smaller
// (gap 8..32, 1024 against 8192 elements: bitmap 18 ns a pair, search 20, merge
// 25, hash 81; 512 against 32768: 37, 23, 73, 186).  Sparse ones: search from a
// ratio of 4 on, else merge (gap 64..256, 8192 against 12000: merge 71 ns, search
// 152, bitmap 116, hash 285).  Hash is never the fastest.
TechTable default_table() {
    TechTable T;
    for (uint32_t b = 0; b < kTableSize; ++b) {
        const uint32_t d = b >> 8, ls = (b >> 4) & 15u, lr = b & 15u;
        if (d <= 1)
            T.t[b] = lr >= 4 || (ls < 9 && lr >= 2) ? kSearch : ls < 8 ? kMerge : kBitmap32K;
        else
            T.t[b] = lr >= 2 ? kSearch : kMerge;
    }
    return T;
}

// Resident CTAs per SM of the two batch kernels on the current device (the
// stream kernel's shared-memory attribute is set per device, once).
struct BatchOccupancy {
    int search = 0, stream = 0;
};
BatchOccupancy batch_occupancy() {
    constexpr int kMaxDevices = 64;
    static BatchOccupancy cached[kMaxDevices];
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return {};
    std::lock_guard<std::mutex> lk(mu);
    BatchOccupancy& o = cached[dev];
    if (o.search == 0 || o.stream == 0) {
        int a = 0, b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, batch_kernel<false>, kBThreads, 0) != cudaSuccess ||
            cudaFuncSetAttribute(batch_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBSmem) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, batch_kernel<true>, kBThreads, kBSmem) != cudaSuccess)
            return {};
        o.search = a;
        o.stream = b;
    }
    return o;
}

si_status batch_launch(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, const uint32_t* d_pairs,
                       uint64_t npairs, const TechTable& table, int forced, const uint32_t* d_subset,
                       uint64_t nsubset, uint32_t* d_counts, void* ws, size_t ws_bytes, cudaStream_t stream) {
    const BatchLayout L = batch_layout(npairs);
    if (ws_bytes < L.total) return SI_ERR_WORKSPACE_TOO_SMALL;
    unsigned char* w = static_cast<unsigned char*>(ws);
    SI_CUDA_TRY(cudaMemsetAsync(w, 0, d_subset ? kBatchHeader : L.off_bins, stream));
    if (npairs == 0) return SI_OK;
    uint64_t* queue = reinterpret_cast<uint64_t*>(w + L.off_queue);
    BatchParams prm;
    prm.el = d_elements;
    prm.off = d_offsets;
    prm.pairs = d_pairs;
    prm.k = k;
    prm.queue = queue;
    prm.subset = d_subset;
    prm.nqueue = d_subset ? nsubset : npairs;
    prm.counts = d_counts;
    prm.header = w;
    prm.forced = forced;
    if (!d_subset) {
        PhaseTimer timer("batch_plan", stream);
        uint32_t* hist = reinterpret_cast<uint32_t*>(w + L.off_hist);
        uint32_t* cursor = reinterpret_cast<uint32_t*>(w + L.off_cursor);
        uint16_t* bins = reinterpret_cast<uint16_t*>(w + L.off_bins);
        if (npairs <= kPlanMost) {
            batch_plan_kernel<<<1, kPlanThreads, 0, stream>>>(d_elements, d_offsets, d_pairs,
                                                              static_cast<uint32_t>(npairs), k, table, forced, queue, w);
            SI_LAUNCH_CHECK("batch_plan_kernel");
        } else {
            const unsigned g = static_cast<unsigned>((npairs + kKeyThreads * kKeyPairs - 1) / (kKeyThreads * kKeyPairs));
            batch_keys_kernel<<<g, kKeyThreads, 0, stream>>>(d_elements, d_offsets, d_pairs, npairs, k, table, forced,
                                                             L.shift, bins, hist, w);
            SI_LAUNCH_CHECK("batch_keys_kernel");
            const si_status st = launch_dependent(batch_queue_kernel, dim3(g), dim3(kKeyThreads), 0, stream,
                                                  static_cast<const uint16_t*>(bins), npairs, L.shift,
                                                  static_cast<const uint32_t*>(hist), cursor, queue, w);
            if (st != SI_OK) return st;
        }
    }
    const BatchOccupancy occ = batch_occupancy();
    const int search_per_sm = occ.search, stream_per_sm = occ.stream;
    if (search_per_sm == 0 || stream_per_sm == 0) return cuda_fail(cudaGetLastError(), "batch_kernel attributes");
    // the subset of the tuner runs in its technique's kernel; the whole queue
    // in both, one part each (no stream part when every pair merges or searches,
    // nor the other when every pair is forced to the stream kernel: those too
    // large for it, which merge there, are in the first part)
    const bool forced_stream = forced >= 0 && is_stream_tech(static_cast<uint8_t>(forced));
    const bool run_search = d_subset ? !forced_stream : true;
    const bool run_stream = d_subset ? forced_stream : forced < 0 || forced_stream;
    PhaseTimer timer("batch_count", stream);
    prm.first = true;
    if (run_search) {
        const si_status st = launch_dependent(batch_kernel<false>, dim3(static_cast<unsigned>(sm_count() * search_per_sm)),
                                              dim3(kBThreads), 0, stream, prm);
        if (st != SI_OK) return st;
        prm.first = false;
    }
    if (run_stream)
        return launch_dependent(batch_kernel<true>, dim3(static_cast<unsigned>(sm_count() * stream_per_sm)),
                                dim3(kBThreads), kBSmem, stream, prm);
    return SI_OK;
}

__global__ void bucket_kernel(const uint32_t* __restrict__ el, const uint64_t* __restrict__ off,
                              const uint32_t* __restrict__ pairs, uint64_t npairs, uint32_t k,
                              uint16_t* __restrict__ bucket) {
    for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < npairs; p += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t a = pairs[2 * p], b = pairs[2 * p + 1];
        bucket[p] = (a < k && b < k) ? static_cast<uint16_t>(device_bucket(el, pair_sets(off, a, b))) : 0;
    }
}

}  // namespace

size_t batch_workspace_size(uint64_t npairs) { return batch_layout(npairs).total; }

si_status batch_count(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, const uint32_t* d_pairs,
                      uint64_t npairs, si_technique t, const uint8_t* table, uint32_t* d_counts, void* ws,
                      size_t ws_bytes, cudaStream_t stream) {
    TechTable T = default_table();
    if (table) std::memcpy(T.t, table, kTableSize);
    const int forced = t == SI_TECH_IP       ? kMerge
                       : t == SI_TECH_OBS    ? kSearch
                       : t == SI_TECH_HI     ? kHash1024
                       : t == SI_TECH_BITMAP ? kBitmap16K
                                             : -1;
    return batch_launch(d_elements, d_offsets, k, d_pairs, npairs, T, forced, nullptr, 0, d_counts, ws, ws_bytes,
                        stream);
}

si_status batch_tune(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, const uint32_t* d_pairs,
                     uint64_t npairs, uint32_t sample, uint32_t* d_counts, void* ws, size_t ws_bytes,
                     cudaStream_t stream, uint8_t* table_out) {
    TechTable T = default_table();
    std::memcpy(table_out, T.t, kTableSize);
    const BatchLayout L = batch_layout(npairs);
    if (ws_bytes < L.total) return SI_ERR_WORKSPACE_TOO_SMALL;
    // the error words: a batch without a bucket of 32 pairs launches nothing else that clears them
    SI_CUDA_TRY(cudaMemsetAsync(ws, 0, kBatchHeader, stream));
    if (npairs == 0) return SI_OK;
    // bucket of every pair, on the device, read back
    unsigned char* w = static_cast<unsigned char*>(ws);
    uint16_t* d_bucket = reinterpret_cast<uint16_t*>(w + L.off_bins);
    const unsigned g = static_cast<unsigned>(std::min<uint64_t>((npairs + 255) / 256, uint64_t(sm_count()) * 8));
    bucket_kernel<<<g, 256, 0, stream>>>(d_elements, d_offsets, d_pairs, npairs, k, d_bucket);
    SI_LAUNCH_CHECK("bucket_kernel");
    std::vector<uint16_t> bucket(npairs);
    SI_CUDA_TRY(cudaMemcpyAsync(bucket.data(), d_bucket, npairs * 2, cudaMemcpyDeviceToHost, stream));
    SI_CUDA_TRY(cudaStreamSynchronize(stream));
    std::vector<std::vector<uint32_t>> members(kTableSize);
    for (uint64_t p = 0; p < npairs; ++p)
        if (members[bucket[p]].size() < sample) members[bucket[p]].push_back(static_cast<uint32_t>(p));
    // sample lists on the device, in the queue's room
    uint32_t* d_subset = reinterpret_cast<uint32_t*>(w + L.off_queue);  // npairs * 8 bytes of room
    cudaEvent_t e0, e1;
    SI_CUDA_TRY(cudaEventCreate(&e0));
    SI_CUDA_TRY(cudaEventCreate(&e1));
    si_status st = SI_OK;
    for (uint32_t b = 0; b < kTableSize && st == SI_OK; ++b) {
        const auto& m = members[b];
        if (m.size() < 32) continue;  // too few pairs to matter: keep the default
        if (cudaMemcpyAsync(d_subset, m.data(), m.size() * 4, cudaMemcpyHostToDevice, stream) != cudaSuccess) {
            st = cuda_fail(cudaGetLastError(), "batch_tune copy");
            break;
        }
        float ms[kTechCodes] = {};
        for (uint8_t tech = 0; tech < kTechCodes && st == SI_OK; ++tech) {
            // three runs: the first warms the caches, the faster of the other two counts
            ms[tech] = 0.f;
            for (int rep = 0; rep < 3 && st == SI_OK; ++rep) {
                cudaEventRecord(e0, stream);
                st = batch_launch(d_elements, d_offsets, k, d_pairs, npairs, T, tech, d_subset, m.size(), d_counts,
                                  ws, ws_bytes, stream);
                cudaEventRecord(e1, stream);
                if (st != SI_OK || rep == 0) continue;
                if (cudaEventSynchronize(e1) != cudaSuccess) {
                    st = cuda_fail(cudaGetLastError(), "batch_tune");
                    break;
                }
                float t = 0.f;
                cudaEventElapsedTime(&t, e0, e1);
                ms[tech] = rep == 1 ? t : std::min(ms[tech], t);
            }
            if (st != SI_OK) break;
        }
        if (st != SI_OK) break;
        // another technique replaces the default only when it is 3 % faster
        uint8_t best = T.t[b];
        for (uint8_t tech = 0; tech < kTechCodes; ++tech)
            if (ms[tech] < 0.97f * ms[best]) best = tech;
        table_out[b] = best;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return st;
}

}  // namespace si
