// si_sisi_obs.cu -- optimized binary search (obs) for one pair of sorted sets.
//
// The reference's obs (src/obs.cu:275-358, warpBasedOBS; :439-522 for the
// single pair) caches the first levels of the larger set's binary-search tree
// in shared memory and lets every element of the smaller set search the cache
// first (phase 1), then the larger set in global memory (phase 2).  Same two
// phases here, re-designed for B200, where all of it is dependent loads of
// lines that are not in cache: latency while there are few searches, sectors
// fetched when there are many.
//
//  * Phase 1: every CTA gathers 256 or 1024 evenly spaced elements of the larger
//    set L into shared memory itself (one round of loads in flight).  8192
//    samples, gathered once by a kernel before, narrowed a search further, but
//    cost that kernel and 32 KiB of copies per CTA.
//  * Phase 2: the values on both sides of a window say where in it an element
//    should lie (interpolation search: Peterson, 1957; Perl, Itai, Avni, 1978).
//    For evenly spread values the place is off by half the square root of the
//    window's length or less, so a step probes that far to both sides, two
//    loads at once: windows of 2^18 elements are down to 512 after one step and
//    to some twenty after two, where halving takes eight and fourteen, each a
//    miss and a sector.  After three steps, or below 64 elements, the window
//    is cut in four by three loads at once, then halved, so that values that
//    are spread in no such way cost the three steps at most.
//  * Each warp owns 32 J consecutive elements of S, the smaller set, J (1..32)
//    chosen so that the grid holds about one search per resident thread (its
//    occupancy on the device).
//  * The hits of 32 consecutive elements are one word of a hit mask in global
//    memory, and each CTA counts its chunk's hits.
//  * A second kernel, a programmatic dependent of the first, compacts S by the
//    hit mask: every CTA adds up the chunk counts before its own, a warp takes
//    up to 32 mask words at a time, lanes on bits.  The result is ascending
//    because S is.  Without element output one CTA adds up the counts, unless
//    a single CTA has searched (S of up to kObsThreads elements), which knows
//    the count: 3.0 us a call against 4.0, 16 to 128 elements in 16384.
//
// Elements out, L not in cache (in cache), against 13 or more halving steps
// after 8192 samples, in three launches: 2^16 elements in 2^26 23.6 (9.4)
// against 42 (19.4) us, 2^18 in 2^26 42 (19.5) against 93 (71), 2^20 in 2^26 77
// (57) against 192 (175), 2^20 in 2^20 25 against 34.  Values that cluster at
// twelve scales, 2^16 in 2^25: 27.6 against 33.7.
// Work is |S| searches, so the technique pays off when |S| << |L| (skewed
// pairs); it is exact for any sizes.
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "si_device.cuh"
#include "si_internal.h"

namespace si {
namespace {

constexpr uint32_t kTop = 1024;             // most samples a CTA caches
constexpr uint32_t kTopMany = 256;          // what it caches where many CTAs gather them
constexpr uint64_t kTopChunks = 148;        // chunks up to which kTop are gathered
constexpr int kGuess = 3;                   // interpolation steps of a search
constexpr uint32_t kGuessLen = 64;          // shorter windows are not guessed in
constexpr int kObsThreads = 256;
static_assert(kObsThreads == kObsOneChunk, "the engine's choice counts searches");
constexpr int kObsWarps = kObsThreads / 32;
constexpr size_t kObsHeader = 256;          // error words

struct ObsLayout {
    uint64_t nChunks = 0, nWords = 0;
    uint32_t J = 1;                          // mask words per warp
    uint64_t chunk = 0;                      // elements of S per CTA: kObsThreads J
    size_t off_mask = 0, off_ccount = 0, total = 0;
};

// threads: resident threads of the search kernel on the GPU.
ObsLayout obs_layout(uint64_t nS, uint64_t threads) {
    ObsLayout L;
    // J elements per thread: about one search per resident thread
    L.J = static_cast<uint32_t>(std::min<uint64_t>(32, std::max<uint64_t>(1, (nS + threads - 1) / threads)));
    L.chunk = uint64_t(kObsThreads) * L.J;
    L.nChunks = (nS + L.chunk - 1) / L.chunk;
    L.nWords = L.nChunks * L.chunk / 32;
    // sized for any J, so the workspace size depends on the sizes only
    const uint64_t max_words = nS / 32 + 256;
    const uint64_t max_chunks = (nS + 255) / 256;
    size_t o = kObsHeader;
    L.off_mask = o;
    o = align_up(o + max_words * 4, 256);
    L.off_ccount = o;
    o = align_up(o + max_chunks * 4, 256);
    L.total = o;
    return L;
}

// Phase 1: the last of n cached samples <= x (branch-free; top2: the largest
// power of two below n); x >= top[0].
__device__ __forceinline__ uint32_t top_find(uint32_t x, const uint32_t* __restrict__ top, uint32_t n, uint32_t top2) {
    uint32_t pos = 0;  // invariant: top[pos] <= x
    for (uint32_t step = top2; step > 0; step >>= 1) {
        const uint32_t p = pos + step;
        pos = (p < n && top[p] <= x) ? p : pos;
    }
    return pos;
}

// Phase 2: is x among the len elements from L, where L[0] = a <= x < b and b is
// the element after them (or above it)?  a and b only say where to look.
__device__ __forceinline__ bool gap_find(uint32_t x, uint32_t a, uint32_t b, const uint32_t* __restrict__ L,
                                         uint32_t len) {
#pragma unroll 1
    for (int round = 0; round < kGuess && len > kGuessLen; ++round) {
        // d: half of sqrt(len), two standard deviations at the window's ends and
        // one in its middle; 2^18 in 2^26: 40.0 us, with sqrt(len) 44.1
        const float est = __fdividef(static_cast<float>(x - a), static_cast<float>(b - a)) * static_cast<float>(len);
        const uint32_t d = static_cast<uint32_t>(0.5f * sqrtf(static_cast<float>(len)));
        const uint32_t e = min(static_cast<uint32_t>(est), len - 1);
        const uint32_t p0 = e > d ? e - d : 0u, p1 = min(e + d, len - 1);
        const uint32_t v0 = __ldg(L + p0), v1 = __ldg(L + p1);
        if (x < v0) {
            b = v0;
            len = p0;
        } else if (x >= v1) {
            a = v1;
            L += p1;
            len -= p1;
        } else {
            a = v0;
            b = v1;
            L += p0;
            len = p1 - p0;
        }
    }
    while (len > 8) {
        const uint32_t q = len >> 2;
        const uint32_t u = __ldg(L + q), v = __ldg(L + 2 * q), w = __ldg(L + 3 * q);
        const uint32_t m = (u <= x) + (v <= x) + (w <= x);
        L += m * q;
        len = m == 3 ? len - 3 * q : q;
    }
    while (len > 1) {
        const uint32_t half = len >> 1;
        const bool c = __ldg(L + half) <= x;
        L += c ? half : 0u;
        len = c ? len - half : half;
    }
    return __ldg(L) == x;
}

// Phase 1 + 2 for one chunk of S per CTA: hit mask words and chunk counts.
// T: elements between the nTop samples.  Also clears the workspace's error words.
constexpr int kObsSearchCtasPerSm = 8;  // 32 registers
template <bool kOut>
__global__ void __launch_bounds__(kObsThreads, kObsSearchCtasPerSm)
    obs_search_kernel(const uint32_t* __restrict__ S, uint64_t nS, const uint32_t* __restrict__ L, uint64_t nL,
                      uint32_t* __restrict__ mask, uint32_t* __restrict__ ccount, uint64_t nChunks, uint32_t J,
                      uint32_t T, uint32_t nTop, uint32_t* __restrict__ header, uint64_t* __restrict__ d_count) {
    __shared__ uint32_t top[kTop];
    __shared__ uint32_t s_warp[kObsWarps];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (blockIdx.x == 0 && threadIdx.x < kObsHeader / 4) header[threadIdx.x] = 0;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t top2 = nTop > 1 ? 1u << (31 - __clz(nTop - 1)) : 0u;
#pragma unroll 4
    for (uint32_t w = threadIdx.x; w < nTop; w += kObsThreads) top[w] = __ldg(L + uint64_t(w) * T);
    __syncthreads();
    for (uint64_t c = blockIdx.x; c < nChunks; c += gridDim.x) {
        const uint64_t first = c * kObsThreads * J;
        const uint64_t base = first + uint64_t(warp) * 32 * J;
        uint32_t hits = 0;
#pragma unroll 1
        for (uint32_t j = 0; j < J; ++j) {
            const uint64_t i = base + uint64_t(j) * 32 + lane;
            bool hit = false;
            if (i < nS) {
                const uint32_t x = __ldg(S + i);
                if (x >= top[0]) {
                    const uint32_t pos = top_find(x, top, nTop, top2);
                    const uint64_t at = uint64_t(pos) * T;
                    hit = gap_find(x, top[pos], pos + 1 < nTop ? top[pos + 1] : 0xffffffffu, L + at,
                                   nL - at < T ? static_cast<uint32_t>(nL - at) : T);
                }
            }
            const uint32_t word = __ballot_sync(kFullMask, hit);
            if (kOut && lane == 0) mask[(base >> 5) + j] = word;
            hits += __popc(word);
        }
        if (lane == 0) s_warp[warp] = hits;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t total = 0;
            for (int w = 0; w < kObsWarps; ++w) total += s_warp[w];
            ccount[c] = total;
            if (!kOut && nChunks == 1) *d_count = total;
        }
        __syncthreads();
    }
}

// Compaction.  CTA b takes `per` chunks of W mask words.  It adds up the
// counts of all chunks before them, then takes its words 8 seg at a time, a
// warp seg (1..32) of them: lane i holds word i, scans of the words' hits over
// the lanes and the warps give each word's place, and the warp writes word by
// word: lane b copies element 32 w + b when bit b of word w is set, so loads
// of S and stores of out are coalesced.  The last CTA knows the total; without
// element output it is the only one and has no words.
template <bool kOut>
__global__ void __launch_bounds__(kObsThreads) obs_compact_kernel(const uint32_t* __restrict__ S,
                                                                  const uint32_t* mask, const uint32_t* ccount,
                                                                  uint32_t* __restrict__ out,
                                                                  uint64_t* __restrict__ d_count, uint64_t nChunks,
                                                                  uint64_t per, uint32_t W, uint32_t seg) {
    __shared__ uint64_t s_sum[kObsWarps];
    __shared__ uint32_t s_warp[kObsWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the mask and the counts
    const uint64_t c0 = kOut ? blockIdx.x * per : nChunks;
    uint64_t sum = 0;
#pragma unroll 8
    for (uint64_t i = threadIdx.x; i < c0; i += kObsThreads) sum += ccount[i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(kFullMask, sum, d);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    uint64_t base = 0;
#pragma unroll
    for (int w = 0; w < kObsWarps; ++w) base += s_sum[w];
    if constexpr (kOut) {
        const uint64_t end = (c0 + per < nChunks ? c0 + per : nChunks) * W;
        for (uint64_t b = c0 * W; b < end; b += uint64_t(kObsWarps) * seg) {
            const uint64_t w0 = b + uint64_t(warp) * seg;
            const uint32_t word = lane < seg && w0 + lane < end ? mask[w0 + lane] : 0u;
            const uint32_t n = __popc(word);
            const uint32_t incl = warp_inclusive_scan(n);
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            uint64_t mine = base + incl - n;  // the place of word `lane`
#pragma unroll
            for (int w = 0; w < kObsWarps; ++w) {
                mine += w < static_cast<int>(warp) ? s_warp[w] : 0u;
                base += s_warp[w];
            }
            const uint32_t below = (1u << lane) - 1u;
            for (uint32_t i = 0; i < seg; ++i) {
                const uint32_t wd = __shfl_sync(kFullMask, word, i);
                if (wd == 0) continue;  // warp-uniform
                const uint64_t o = __shfl_sync(kFullMask, mine, i);
                if ((wd >> lane) & 1u) out[o + __popc(wd & below)] = __ldg(S + (w0 + i) * 32 + lane);
            }
            __syncthreads();
        }
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *d_count = base;
}

// Resident threads of the search kernel (with or without element output) on
// the current device, cached per device.
uint64_t obs_resident_threads(bool out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
    static std::mutex mu;
    static std::unordered_map<int, uint64_t> cache[2];
    std::lock_guard<std::mutex> lk(mu);
    const auto it = cache[out].find(dev);
    if (it != cache[out].end()) return it->second;
    int per_sm = 0;
    const cudaError_t e = out ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, obs_search_kernel<true>,
                                                                              kObsThreads, 0)
                              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, obs_search_kernel<false>,
                                                                              kObsThreads, 0);
    if (e != cudaSuccess || per_sm <= 0) {
        (void)cudaGetLastError();
        per_sm = 1;
    }
    const uint64_t r = uint64_t(per_sm) * kObsThreads * uint64_t(sm_count());
    cache[out][dev] = r;
    return r;
}

}  // namespace

size_t obs_workspace_size(uint64_t nA, uint64_t nB) {
    return obs_layout(std::min(nA, nB), 1).total;  // the sizes do not depend on the threads
}

si_status obs_sisi(const uint32_t* dA, uint64_t nA, const uint32_t* dB, uint64_t nB, uint64_t* d_count,
                   uint32_t* d_out, void* ws, size_t ws_bytes, cudaStream_t stream) {
    // S: the smaller set (A on ties), searched for in the larger set L
    const bool a_small = nA <= nB;
    const uint32_t* S = a_small ? dA : dB;
    const uint32_t* Lp = a_small ? dB : dA;
    const uint64_t nS = a_small ? nA : nB, nL = a_small ? nB : nA;
    const ObsLayout Lo = obs_layout(nS, obs_resident_threads(d_out != nullptr));
    if (ws_bytes < Lo.total) return SI_ERR_WORKSPACE_TOO_SMALL;
    unsigned char* w = static_cast<unsigned char*>(ws);
    if (nS == 0 || nL == 0) {
        SI_CUDA_TRY(cudaMemsetAsync(w, 0, kObsHeader, stream));
        SI_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), stream));
        return SI_OK;
    }
    uint32_t* header = reinterpret_cast<uint32_t*>(w);
    uint32_t* mask = reinterpret_cast<uint32_t*>(w + Lo.off_mask);
    uint32_t* ccount = reinterpret_cast<uint32_t*>(w + Lo.off_ccount);
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(Lo.nChunks, uint64_t(sm_count()) * 8));
    // every CTA gathers the samples for itself, so many CTAs take fewer: 2^20
    // elements in 2^20, 1024 CTAs: 25.3 us with 256 against 28.7 with 1024;
    // 16 in 10000, one CTA: 4.6 against 4.2
    const uint64_t samples = Lo.nChunks <= kTopChunks ? kTop : kTopMany;
    const uint32_t T = static_cast<uint32_t>((nL + samples - 1) / samples);
    const uint32_t nTop = static_cast<uint32_t>((nL + T - 1) / T);
    {
        PhaseTimer timer("obs_search", stream);
        auto kernel = d_out ? obs_search_kernel<true> : obs_search_kernel<false>;
        kernel<<<grid, kObsThreads, 0, stream>>>(S, nS, Lp, nL, mask, ccount, Lo.nChunks, Lo.J, T, nTop, header,
                                                 d_count);
    }
    SI_LAUNCH_CHECK("obs_search_kernel");
    if (!d_out && Lo.nChunks == 1) return SI_OK;  // it has written the count
    PhaseTimer timer("obs_compact", stream);
    const uint32_t* cmask = mask;
    const uint32_t* ccounts = ccount;
    if (!d_out)
        return launch_dependent(obs_compact_kernel<false>, dim3(1), dim3(kObsThreads), 0, stream, S, cmask, ccounts,
                                d_out, d_count, Lo.nChunks, uint64_t(0), 0u, 1u);
    // chunks per CTA: up to 8 CTAs an SM; mask words per warp and round: all 32
    // lanes hold one where the CTA has that many
    const uint64_t ctas = std::min<uint64_t>(Lo.nChunks, uint64_t(sm_count()) * 8);
    const uint64_t per = (Lo.nChunks + ctas - 1) / ctas;
    const uint32_t W = static_cast<uint32_t>(Lo.chunk / 32);  // mask words per chunk: at least one a warp
    const uint32_t seg = static_cast<uint32_t>(std::min<uint64_t>(32, per * W / kObsWarps));
    return launch_dependent(obs_compact_kernel<true>, dim3(static_cast<unsigned>((Lo.nChunks + per - 1) / per)),
                            dim3(kObsThreads), 0, stream, S, cmask, ccounts, d_out, d_count, Lo.nChunks, per, W, seg);
}

}  // namespace si
