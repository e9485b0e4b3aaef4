// si_misi_slab.cuh -- the value-major bit matrix of the all-pairs bitmap
// technique: what si_misi.cu (plan, fallback) and si_misi_slab.cu (the kernel)
// share.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "si.h"

namespace si {

// The matrix: one entry of 32 E row bits per value, E = 16, 8 or 4 words.
// 64 MiB hold 2^20 values of 512 rows, 2^21 of 256 or 2^22 of 128, and half
// of the L2 cache holds 64 MiB.
constexpr uint32_t kSlabMaxWords = 16;
constexpr uint32_t kSlabMinWords = 4;
constexpr uint64_t kSlabValues = 1ull << 20;  // values of an entry of kSlabMaxWords words
constexpr size_t kSlabBytes = (kSlabValues + 16) * kSlabMaxWords * 4;
// Collections of fewer rows keep the probe kernel: a group of rows fills less
// than a quarter of the narrowest entry.
constexpr uint32_t kSlabMinRows = 32;
// So do small collections of small sets, where the matrix' clears and grid
// barriers cost more than the probes: with sets of up to 32 elements, hash,
// 32 sets 32 us a call by the probe kernel and 53 by the matrix, 200 sets 48 and
// 62, 1000 sets 119 and 118-125; bitmap, 32 sets 32 and 42, 200 sets 48 and 48.
constexpr uint32_t kSlabSmallSet = 64;
constexpr uint32_t kSlabSmallRows = 128;
constexpr uint32_t kSlabSmallRowsHash = 1024;

// Words of the all-pairs header that the plan and both kernels use.
constexpr size_t kMisiTicket = 16;      // u32 ticket of the probe kernel
constexpr size_t kMisiValueMin = 20;    // u32 ~(smallest first value of a set), 0 when every set is empty
constexpr size_t kMisiValueMax = 24;    // u32 largest last value of a set
constexpr size_t kMisiSlabTicket = 28;  // u32 slices handed out in the current group
constexpr size_t kMisiSlabBarrier = 32;  // u32 arrivals at the grid barrier
constexpr size_t kMisiPlanDone = 36;     // u32 CTAs of the order kernel that finished
constexpr size_t kMisiTotals = 40;       // u64[2] elements of side A and of side B

// Technique hi: the entries are the slots of an open-addressing hash table of
// the values, twice as many as it can come to hold.
constexpr uint32_t kSlabMaxSlots = 1u << 21;
constexpr uint32_t kSlabMinSlots = 1u << 10;  // (slab_plan starts from it)
constexpr size_t kSlabKeyBytes = size_t(kSlabMaxSlots) * 4;
constexpr uint32_t kSlabEmpty = 0xffffffffu;  // an empty slot; that value has an entry of its own

// How a tile is counted: words per entry (0: the probe kernel counts) and, for
// technique hi, the table's slots.
struct SlabPlan {
    uint32_t words, slots, shift;  // slots = 2^(32 - shift)
    uint32_t vmin, span;  // the values lie in [vmin, vmin + span]
};

// rows: of the tile; vmin, vmax: its smallest and largest value; largest: the
// elements of its largest set; total: of its larger side.  A bitmap has an
// entry per value of the span and one that is always zero (values out of
// range, which only an unsorted set has, read it); a table of n slots has the
// zero entry n and entry n + 1 for the value that marks empty slots.
__host__ __device__ inline SlabPlan slab_plan(bool hash, uint32_t rows, uint32_t vmin, uint32_t vmax,
                                              uint64_t largest, uint64_t total) {
    SlabPlan pl = {0, 0, 0, vmin, vmax - vmin};
    if (rows < kSlabMinRows || vmax < vmin) return pl;  // (vmax < vmin: every set is empty)
    if (largest <= kSlabSmallSet && rows <= (hash ? kSlabSmallRowsHash : kSlabSmallRows)) return pl;
    uint64_t entries = uint64_t(pl.span) + 2;
    if (hash) {
        // distinct values at once: all of them, or a group's (whose rows end before half of the slots is full)
        const uint64_t distinct = total < uint64_t(pl.span) + 1 ? total : uint64_t(pl.span) + 1;
        pl.slots = kSlabMinSlots;
        pl.shift = 22;
        for (; pl.slots < kSlabMaxSlots && pl.slots < 2 * distinct; --pl.shift) pl.slots *= 2;
        if (pl.slots < 2 * distinct && largest > pl.slots / 2) return pl;
        entries = uint64_t(pl.slots) + 2;
    }
    uint32_t e = rows <= 128 ? 4u : rows <= 256 ? 8u : kSlabMaxWords;
    while (e >= kSlabMinWords && entries * e * 4 > kSlabBytes) e /= 2;
    if (e >= kSlabMinWords) pl.words = e;
    return pl;
}

struct SlabParams {
    const uint32_t* el;
    const uint64_t* off;
    uint32_t a_start, b_start, nA, nB;
    uint32_t self;
    uint64_t stride;
    const uint64_t* keys;  // sorted: side A [0, nA), side B [nA, nA + nB)
    const uint64_t* P;     // prefix sums of the sorted sizes: side A [0, nA], side B [nA + 1, nA + 1 + nB]
    const uint32_t* cs;    // first partner of every row in the other side's sorted list
    uint32_t* counts;
    unsigned char* header;
    uint32_t* table;
    uint32_t* slots;  // technique hi: the values in the slots
};

#ifdef __CUDACC__
// The plan of a tile, from the all-pairs header and the sorted prefix sums.
__device__ __forceinline__ SlabPlan slab_plan_of(bool hash, uint32_t nA, uint32_t nB, const unsigned char* header,
                                                 const uint64_t* P) {
    const uint64_t* PB = P + nA + 1;
    const uint64_t largestA = nA ? P[1] : 0, largestB = nB ? PB[1] : 0;
    const uint64_t totalA = nA ? P[nA] : 0, totalB = nB ? PB[nB] : 0;
    return slab_plan(hash, nA + nB, ~*reinterpret_cast<const uint32_t*>(header + kMisiValueMin),
                     *reinterpret_cast<const uint32_t*>(header + kMisiValueMax),
                     largestA > largestB ? largestA : largestB, totalA > totalB ? totalA : totalB);
}
#endif

// t: SI_TECH_BITMAP or SI_TECH_HI.
si_status misi_slab(const SlabParams& p, si_technique t, cudaStream_t stream);

}  // namespace si
