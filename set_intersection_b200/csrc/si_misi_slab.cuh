// si_misi_slab.cuh -- the value-major bit matrix of the all-pairs bitmap and
// hash techniques: what si_misi.cu (plan, fallback) and si_misi_slab.cu (the kernel)
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
// So do collections of small sets, where the matrix' clears and grid barriers and
// its cost per partner and group of rows are more than the probes: see
// slab_few_probes.
constexpr uint32_t kSlabSmallSet = 64;     // the probe kernel gives each lane a partner of up to this many elements
constexpr uint32_t kSlabLargeSet = 8192;  // it stages larger sets in chunks (hash), each with all their partners

// Words of the all-pairs header that the plan and both kernels use.
constexpr size_t kMisiTicket = 16;      // u32 ticket of the probe kernel
constexpr size_t kMisiValueMin = 20;    // u32 ~(smallest first value of a set), 0 when every set is empty
constexpr size_t kMisiValueMax = 24;    // u32 largest last value of a set
constexpr size_t kMisiSlabTicket = 28;  // u32 slices handed out in the current group
constexpr size_t kMisiSlabBarrier = 32;  // u32 arrivals at the grid barrier
constexpr size_t kMisiPlanDone = 36;     // u32 CTAs of the order kernel that finished
constexpr size_t kMisiTotals = 40;       // u64[2] elements of side A and of side B
constexpr size_t kMisiWork = 56;         // u64 partner elements of all rows: the probe kernel's probes

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

// What the plan kernels know of a tile.
struct SlabTile {
    uint32_t nA, nB;      // sets of the sides (nB = 0: one side against itself)
    uint32_t vmin, vmax;  // smallest and largest value
    uint64_t largest;     // elements of the largest set
    uint64_t total;       // elements of the larger side
    uint64_t work;        // partner elements of all rows
};

// Whether the probe kernel is the faster one for a tile that the matrix could
// count: by the mean probes of a pair, which bound the probe kernel's work from
// below however the sizes are spread.  words, slots: the matrix' entries and the
// table that hash would use.  Tiles of sets of 1..m elements, whole calls in us,
// probe kernel / matrix, values of a span of 2^20 unless given:
//   bitmap  200 sets: m = 16 39/54, 32 47/49     1000 sets: m = 2 122/149, 8 156/125
//           600 sets: m = 8 84/134, 32 97/98     4000 sets: m = 2 1417/681
//           span 2^22 (128 rows at a time), 1000 sets: m = 2 149/588, 8 311/337
//           two sides, 600 sets in all: m = 8 79/86, 16 87/78
//   hash    200 sets: m = 65 57/89, 100 81/67    1000 sets: m = 65 122/167, 100 163/154
//           600 sets: m = 65 82/141, 200 147/166 4000 sets: m = 8 763/953, 65 703/483
//           two sides, 600 sets: m = 65 80/86    1000 sets: m = 16 100/118, 65 116/94
//           32 sets: m = 1000 56/76, 4000 70/80; 64 sets: m = 100 62/61, 2000 66/89
// (sets of 1..m elements come to m / 3 probes a pair).  Four of 200 sets of 30000
// elements, the others of 3: hash 346/109.
__host__ __device__ inline bool slab_few_probes(bool hash, const SlabTile& t, uint32_t words, uint32_t slots) {
    const uint32_t rows = t.nA + t.nB;
    const bool self = t.nB == 0;
    const uint64_t pairs = self ? uint64_t(rows) * (rows - 1) / 2 : uint64_t(t.nA) * t.nB;
    if (t.largest <= kSlabSmallSet && rows <= (hash ? 1024 : 128)) return true;
    if (t.largest > kSlabLargeSet) return false;
    uint64_t mean;  // probes of a pair, at most
    if (hash) {
        if (rows < 128 && t.largest <= 2048 && (rows < 48 || t.largest > 512) && slots > 2048) return true;
        if (self) mean = rows > 4096 ? 5 : rows > 2048 ? 8 : rows > 512 && rows <= 768 ? 36 : 26;
        else mean = rows > 4096 ? 5 : rows > 768 ? 8 : 26;
    } else {
        if (rows <= 128) mean = t.vmax - t.vmin < 1u << 20 ? 20 : 8;  // (the probe kernel's bitmap has 2^20 values)
        else if (rows <= (self ? 768 : 640)) mean = self ? 6 : 4;
        else if (words == 4) mean = self ? (rows <= 1024 ? 4 : 3) : 2;
        else mean = (self && rows <= 1024) || (words == 8 && rows <= 2048) ? 2 : 0;
    }
    return t.work <= mean * pairs;
}

// A bitmap has an entry per value of the span and one that is always zero
// (values out of range, which only an unsorted set has, read it); a table of n
// slots has the zero entry n and entry n + 1 for the value that marks empty slots.
__host__ __device__ inline SlabPlan slab_plan(bool hash, const SlabTile& t) {
    const uint32_t rows = t.nA + t.nB;
    SlabPlan pl = {0, 0, 0, t.vmin, t.vmax - t.vmin};
    if (rows < kSlabMinRows || t.vmax < t.vmin) return pl;  // (vmax < vmin: every set is empty)
    uint64_t entries = uint64_t(pl.span) + 2;
    if (hash) {
        // distinct values at once: all of them, or a group's (whose rows end before half of the slots is full)
        const uint64_t distinct = t.total < uint64_t(pl.span) + 1 ? t.total : uint64_t(pl.span) + 1;
        pl.slots = kSlabMinSlots;
        pl.shift = 22;
        for (; pl.slots < kSlabMaxSlots && pl.slots < 2 * distinct; --pl.shift) pl.slots *= 2;
        if (pl.slots < 2 * distinct && t.largest > pl.slots / 2) return pl;
        entries = uint64_t(pl.slots) + 2;
    }
    uint32_t e = rows <= 128 ? 4u : rows <= 256 ? 8u : kSlabMaxWords;
    while (e >= kSlabMinWords && entries * e * 4 > kSlabBytes) e /= 2;
    if (e >= kSlabMinWords && !slab_few_probes(hash, t, e, pl.slots)) pl.words = e;
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
    return slab_plan(hash, {nA, nB, ~*reinterpret_cast<const uint32_t*>(header + kMisiValueMin),
                            *reinterpret_cast<const uint32_t*>(header + kMisiValueMax),
                            largestA > largestB ? largestA : largestB, totalA > totalB ? totalA : totalB,
                            *reinterpret_cast<const uint64_t*>(header + kMisiWork)});
}
#endif

// t: SI_TECH_BITMAP or SI_TECH_HI.
si_status misi_slab(const SlabParams& p, si_technique t, cudaStream_t stream);

}  // namespace si
