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

// Words of the all-pairs header that the plan and both kernels use.
constexpr size_t kMisiTicket = 16;      // u32 ticket of the probe kernel
constexpr size_t kMisiValueMin = 20;    // u32 ~(smallest first value of a set), 0 when every set is empty
constexpr size_t kMisiValueMax = 24;    // u32 largest last value of a set
constexpr size_t kMisiSlabTicket = 28;  // u32 slices handed out in the current group
constexpr size_t kMisiSlabBarrier = 32;  // u32 arrivals at the grid barrier
constexpr size_t kMisiPlanDone = 36;     // u32 CTAs of the order kernel that finished
constexpr size_t kMisiTotals = 40;       // u64[2] elements of side A and of side B

// Words per entry for a collection of `rows` rows whose values lie in
// [vmin, vmin + span], or 0 when the narrowest entries do not fit: then the
// probe kernel counts.  Entry span + 1 is always zero (values out of range,
// which only an unsorted set has, read it).
__host__ __device__ inline uint32_t slab_words(uint32_t rows, uint32_t span) {
    if (rows < kSlabMinRows) return 0;
    uint32_t e = rows <= 128 ? 4u : rows <= 256 ? 8u : kSlabMaxWords;
    while (e >= kSlabMinWords && (uint64_t(span) + 2) * e * 4 > kSlabBytes) e /= 2;
    return e >= kSlabMinWords ? e : 0u;
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
};

si_status misi_slab(const SlabParams& p, cudaStream_t stream);

}  // namespace si
