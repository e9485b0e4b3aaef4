// si_misi_slab.cu -- all pairs of a collection by bitmap or by hash, many rows
// at a time.
//
// The reference gives a block one set's bitmap or hash table and probes it
// with one partner after another (src/bitmap_dynamic.cu:279-319, src/hi.cu:
// 295-420): one probe per element and pair.  Here the bitmap of up to 512 rows
// (sets) is turned over: entry v of the matrix holds one bit per row, set when
// the row's set holds value v.  One 64-byte gather then probes an element of a
// partner against 512 rows at once, and the hits of all rows are summed in
// vertical counters (bit planes, one LOP3 sum and one LOP3 carry per adder for
// 32 rows).  Technique hi finds a value's entry by hashing: one open-addressing
// table holds the values of all the rows, a slot's entry their bits, so any
// range of values fits and an element costs one lookup for all the rows.
//
// One cooperative launch walks the row groups, largest sets first.  Per group:
//   build   every element of the group's rows sets its row's bit (red.or)
//   probe   the warps take slices of the partners' elements (a partner's cost
//           is its elements plus kSlabOver, the price of turning the planes
//           into counts), and count every whole partner against every row of
//           the group; a partner cut by a slice end is summed atomically
//   clear   the group's entries back to zero (its elements again, or the whole
//           matrix when that is less)
// with a grid barrier after each.  Rows are sorted by size, and a partner
// counts only against rows at least as large, so the elements read are the
// smaller sets', as in the probe kernel.
//
// Power-law collection (8192 sets, 45.6 M elements, 2^20 values), bitmap: the
// launch takes 1.79 ms where the probe kernel takes 35.2 ms (builds 0.38 ms,
// bound by the L2's atomics at 1.4e11 a second; probes 1.26 ms, bound by L2
// gathers in the first groups and by latency in the last; clears 0.15 ms).
// Hash, a cross tile of 1500 x 1500 of such sets: 0.94-1.0 ms against 8.05 ms.
// 64 sets of up to 512 elements: bitmap 46 us a call against 62, hash 60 and 62.
#include <algorithm>

#include "si_device.cuh"
#include "si_internal.h"
#include "si_misi_slab.cuh"
#include "si_stream.cuh"

namespace si {
namespace {

constexpr int kSlabThreads = 256;
constexpr int kSlabWarps = kSlabThreads / 32;
constexpr int kSlabCtasPerSm = 2;
constexpr uint32_t kSlabOver = 256;    // elements that cost about as much as one partner's plane sums and stores
constexpr uint32_t kSlabSlice = 4096;  // cost of a slice, at most: 13 planes hold a slice's counts
constexpr uint32_t kSlabSliceMin = 1024;
// A cross tile whose smaller side has at most this many row groups takes rows
// from that side alone, and all of the other side's sets as partners: more
// elements probed than with rows on both sides (where a partner counts against
// larger rows only), but one side's inserts and fewer groups.  Measured (rows
// on both sides -> one): 1 x 2000 sets 147-168 -> 80-95 us, 1500 x 1500 (3
// groups) 344 -> 235, 3000 x 3000 (6 groups) 706 -> 580 for sets of up to 16384
// elements, 440 -> 261 for sets of up to 32.
constexpr uint32_t kSlabAllGroups = 8;
constexpr uint32_t kBuildSlice = 1024;  // elements a warp inserts or clears at a time, at most
constexpr uint32_t kBuildSliceMin = 64;  // and at least: a warp walks its slice's rows one after another
constexpr int kPlanes = 13;
static_assert(kSlabSlice < (1u << kPlanes), "a slice's counts fit the planes");

struct GroupRows {
    uint64_t base[32 * kSlabMaxWords];  // see row_base
    uint32_t id[32 * kSlabMaxWords];    // local index of the row's set
    uint32_t cs[32 * kSlabMaxWords];
};

// Index of pair (i, j), i < j, of the triangular order is tri_base(n, i) + j.
__device__ __forceinline__ uint64_t tri_base(uint64_t n, uint64_t i) {
    return n * (n - 1) / 2 - (n - i) * (n - i - 1) / 2 - i - 1;
}

// All CTAs arrive and wait for each other; false when the wait gave up.
__device__ __forceinline__ bool grid_barrier(uint32_t* arrived, uint32_t target, uint32_t* err, uint32_t* s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(arrived, 1u);
        bool ok = true;
        WaitBudget budget;
        for (;;) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
            if (v >= target) break;
            if (budget.expired()) {
                record_error(err, SI_ERR_TIMEOUT, 41, target);
                ok = false;
                break;
            }
        }
        __threadfence();
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// Where a value's entry is.  Bitmap: at the value's offset in the span.  Hash:
// in the slot that linear probing finds it in.
template <bool kHash>
struct Entries {
    uint32_t* slots;
    uint32_t vmin, span, mask, shift;
    __device__ __forceinline__ explicit Entries(const SlabParams& p, const SlabPlan& pl)
        : slots(p.slots), vmin(pl.vmin), span(pl.span), mask(pl.slots - 1), shift(pl.shift) {}
    __device__ __forceinline__ uint32_t zero() const { return kHash ? mask + 1 : span + 1; }
    __device__ __forceinline__ uint32_t total() const { return kHash ? mask + 3 : span + 2; }
    __device__ __forceinline__ uint32_t slot(uint32_t v) const { return (v * 0x9e3779b1u) >> shift; }
    // What can be loaded ahead of find(): the value in v's first slot.
    __device__ __forceinline__ uint32_t first(uint32_t v) const { return kHash ? slots[slot(v)] : 0u; }
    // v's entry, the zero entry when it has none.
    __device__ __forceinline__ uint32_t find(uint32_t v, uint32_t k) const {
        if constexpr (!kHash) return min(v - vmin, span + 1);
        if (v == kSlabEmpty) return mask + 2;
        uint32_t h = slot(v);
        while (k != v) {
            if (k == kSlabEmpty) return mask + 1;
            h = (h + 1) & mask;
            k = slots[h];
        }
        return h;
    }
};

// The group's rows [r0, r1) of one side: every element sets (kSet) or zeroes
// its row's word in the matrix.  P: prefix sums of the side's sorted sizes.
// Values outside the span, which only an unsorted set has, are left out (the
// table's slots are as many as distinct values of the span could need).
template <int E, bool kHash, bool kSet>
__device__ __forceinline__ void group_elements(const SlabParams& p, const Entries<kHash>& en, const uint64_t* keys,
                                               const uint64_t* P, uint32_t start, uint32_t r0, uint32_t r1) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t e0 = P[r0], e1 = P[r1];
    const uint64_t nwarps = uint64_t(gridDim.x) * kSlabWarps;
    const uint64_t w = uint64_t(blockIdx.x) * kSlabWarps + (threadIdx.x >> 5);
    const uint64_t slice = max(uint64_t(kBuildSliceMin), min(uint64_t(kBuildSlice), (e1 - e0 + nwarps - 1) / nwarps));
    for (uint64_t lo = e0 + w * slice; lo < e1; lo += nwarps * slice) {
        const uint64_t hi = min(lo + slice, e1);
        uint32_t r = static_cast<uint32_t>(warp_first_true(r0, r1, [&](uint64_t q) { return P[q + 1] > lo; }));
        for (uint64_t e = lo; e < hi; ++r) {
            const uint64_t pr = P[r], pe = min(P[r + 1], hi);
            const uint32_t* x = p.el + p.off[start + static_cast<uint32_t>(keys[r] & 0xffffffffu)] + (e - pr);
            const uint32_t n = static_cast<uint32_t>(pe - e), bit = r - r0;
            constexpr uint32_t kLd = 8;  // loads in flight per lane
            for (uint32_t i = lane; i < n; i += 32 * kLd) {
                uint32_t o[kLd];
                bool on[kLd];
#pragma unroll
                for (uint32_t u = 0; u < kLd; ++u) {
                    const uint32_t v = i + 32 * u < n ? __ldg(x + i + 32 * u) : en.vmin - 1;
                    on[u] = i + 32 * u < n && v - en.vmin <= en.span;
                    o[u] = kHash ? v : v - en.vmin;
                }
                if constexpr (kHash) {
                    // every element's first slot is read, then claimed, before any goes on to its next
                    uint32_t h[kLd], k[kLd];
#pragma unroll
                    for (uint32_t u = 0; u < kLd; ++u) {
                        h[u] = en.slot(o[u]);
                        k[u] = on[u] ? __ldcg(en.slots + h[u]) : 0u;
                    }
#pragma unroll
                    for (uint32_t u = 0; u < kLd; ++u)
                        if (kSet && on[u] && k[u] == kSlabEmpty && o[u] != kSlabEmpty) {
                            k[u] = atomicCAS(en.slots + h[u], kSlabEmpty, o[u]);
                            if (k[u] == kSlabEmpty) k[u] = o[u];
                        }
#pragma unroll
                    for (uint32_t u = 0; u < kLd; ++u) {
                        while (on[u] && o[u] != kSlabEmpty && k[u] != o[u]) {
                            if (!kSet && k[u] == kSlabEmpty) break;
                            h[u] = (h[u] + 1) & en.mask;
                            k[u] = __ldcg(en.slots + h[u]);
                            if (kSet && k[u] == kSlabEmpty) {
                                k[u] = atomicCAS(en.slots + h[u], kSlabEmpty, o[u]);
                                if (k[u] == kSlabEmpty) k[u] = o[u];
                            }
                        }
                        o[u] = o[u] == kSlabEmpty ? en.mask + 2 : h[u];
                    }
                }
#pragma unroll
                for (uint32_t u = 0; u < kLd; ++u) {
                    if (!on[u]) continue;
                    uint32_t* word = p.table + uint64_t(o[u]) * E + (bit >> 5);
                    if constexpr (kSet)
                        asm volatile("red.global.or.b32 [%0], %1;" ::"l"(word), "r"(1u << (bit & 31)) : "memory");
                    else
                        *word = 0u;
                }
            }
            e = pe;
        }
    }
}

template <int E>
__device__ __forceinline__ void clear_table(const SlabParams& p, uint64_t entries) {
    uint4* t = reinterpret_cast<uint4*>(p.table);
    const uint64_t n = entries * (E / 4), stride = uint64_t(gridDim.x) * kSlabThreads;
    for (uint64_t i = uint64_t(blockIdx.x) * kSlabThreads + threadIdx.x; i < n; i += stride)
        t[i] = make_uint4(0u, 0u, 0u, 0u);
}

__device__ __forceinline__ void clear_slots(const SlabParams& p, uint32_t slots) {
    uint4* t = reinterpret_cast<uint4*>(p.slots);
    const uint32_t stride = gridDim.x * kSlabThreads;
    for (uint32_t i = blockIdx.x * kSlabThreads + threadIdx.x; i < slots / 4; i += stride)
        t[i] = make_uint4(kSlabEmpty, kSlabEmpty, kSlabEmpty, kSlabEmpty);
}

// (sum, carry) of three bits in every position.
__device__ __forceinline__ void csa(uint32_t& s, uint32_t& c, uint32_t a, uint32_t b, uint32_t d) {
    const uint32_t carry = (a & b) | (a & d) | (b & d);
    s = a ^ b ^ d;
    c = carry;
}

// Adds eight entries' words w to the planes.
template <int NP>
__device__ __forceinline__ void add8(uint32_t (&pl)[NP][4], int w, const uint4 (&x)[8]) {
    uint32_t s, t1, t2, t3, t4, f1, f2, c;
    csa(s, t1, pl[0][w], comp(x[0], w), comp(x[1], w));
    csa(s, t2, s, comp(x[2], w), comp(x[3], w));
    csa(s, t3, s, comp(x[4], w), comp(x[5], w));
    csa(pl[0][w], t4, s, comp(x[6], w), comp(x[7], w));
    csa(s, f1, pl[1][w], t1, t2);
    csa(pl[1][w], f2, s, t3, t4);
    csa(pl[2][w], c, pl[2][w], f1, f2);
#pragma unroll
    for (int j = 3; j < NP; ++j) {
        const uint32_t t = pl[j][w] & c;
        pl[j][w] ^= c;
        c = t;
    }
}

// Counts of partner elements y[0, n) against the group's rows.  The lanes of
// a warp share E / 4 lanes to an element (16 bytes of its entry each), 128 / E
// elements at a time, eight such steps to a round; a round's elements are
// loaded while the round before is summed.  sink(row, count) is called for
// every row of the group with a nonzero count, each row by one lane.
//
// On the power-law collection (8192 sets, 2^20 values) the gathers of the
// first group run at 8.7 TB/s of L2 traffic (336 us), all groups' probes take
// 1.23 ms.  Measured and dropped: gathers of half a round in flight while the
// other half is summed (1.67 ms), gathers staged by cp.async two and three
// rounds ahead (2.5 and 2.7 ms), 24 warps per SM at 80 registers (1.74 ms:
// spills), entries of 256 rows (1.72 against 1.59 ms) or of 128 rows, elements
// loaded two rounds ahead (no change).
template <int E, bool kHash, class Sink>
__device__ __forceinline__ void count_partner(const uint32_t* __restrict__ y, uint32_t n, const uint32_t* table,
                                              const Entries<kHash>& en, Sink sink) {
    constexpr int LPE = E / 4;        // lanes per element
    constexpr int NG = 32 / LPE;      // elements per step
    constexpr int kRound = 8 * NG;
    constexpr int kLoads = kRound / 32;
    // planes that hold a lane's counts of a slice: kSlabSlice / NG elements
    constexpr int NP = E == 16 ? 10 : E == 8 ? 9 : 8;
    static_assert(kSlabSlice / NG < (1 << NP), "a lane's counts fit its planes");
    const uint32_t lane = threadIdx.x & 31, q = lane & (LPE - 1), gi = lane / LPE;
    const uint4* t4 = reinterpret_cast<const uint4*>(table) + q;
    uint32_t pl[NP][4];
#pragma unroll
    for (int j = 0; j < NP; ++j)
#pragma unroll
        for (int w = 0; w < 4; ++w) pl[j][w] = 0u;
    // a round's elements, 32 to a load: as entries (bitmap), or as values of
    // which the first slots are read next (hash); past the end the zero entry
    uint32_t v[kLoads], k1[kLoads], next[kLoads];
    auto load = [&](uint32_t b, uint32_t (&r)[kLoads]) {
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const uint32_t i = b + 32 * k + lane;
            if constexpr (kHash) r[k] = i < n ? __ldg(y + i) : 0u;
            else r[k] = i < n ? en.find(__ldg(y + i), 0u) : en.zero();
        }
    };
    auto look = [&]() {
        if constexpr (kHash) {
#pragma unroll
            for (int k = 0; k < kLoads; ++k) k1[k] = en.first(v[k]);
        }
    };
    load(0, v);
    look();
    if constexpr (kHash) load(kRound, next);
    for (uint32_t b = 0; b < n; b += kRound) {
        uint4 x[8];
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const uint32_t o = !kHash ? v[k] : b + 32 * k + lane < n ? en.find(v[k], k1[k]) : en.zero();
#pragma unroll
            for (int st = 0; st < LPE; ++st) {  // 32 elements, one per lane: LPE steps of NG of them
                const uint32_t oe = LPE == 1 ? o : __shfl_sync(kFullMask, o, st * NG + gi);
                x[k * LPE + st] = t4[uint64_t(oe) * LPE];
            }
        }
        if constexpr (kHash) {  // the slots a round ahead, the elements two
#pragma unroll
            for (int k = 0; k < kLoads; ++k) v[k] = next[k];
            look();
            load(b + 2 * kRound, next);
        } else {
            load(b + kRound, v);
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) add8<NP>(pl, w, x);
    }
    // Sum the planes of the lane groups.  Rounds 1 and 2 (lanes 16, then 8
    // apart) each keep half of the words; the later ones keep the word and
    // leave the same sums in all the lanes that share it.
    uint32_t p2[NP + 1][2];
    {
        const bool up = lane & 16;
        uint32_t c[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < NP; ++j)
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const uint32_t mine = up ? pl[j][2 + w] : pl[j][w];
                const uint32_t give = up ? pl[j][w] : pl[j][2 + w];
                const uint32_t got = __shfl_xor_sync(kFullMask, give, 16);
                csa(p2[j][w], c[w], mine, got, c[w]);
            }
        p2[NP][0] = c[0];
        p2[NP][1] = c[1];
    }
    uint32_t pp[kPlanes];
    {
        const bool up = lane & 8;
        uint32_t c = 0u;
#pragma unroll
        for (int j = 0; j <= NP; ++j) {
            const uint32_t mine = up ? p2[j][1] : p2[j][0];
            const uint32_t give = up ? p2[j][0] : p2[j][1];
            const uint32_t got = __shfl_xor_sync(kFullMask, give, 8);
            csa(pp[j], c, mine, got, c);
        }
        pp[NP + 1] = c;
#pragma unroll
        for (int j = NP + 2; j < kPlanes; ++j) pp[j] = 0u;
    }
#pragma unroll
    for (int d = 4; d >= LPE; d >>= 1) {
        uint32_t c = 0u;
#pragma unroll
        for (int j = 0; j < kPlanes; ++j) {
            const uint32_t got = __shfl_xor_sync(kFullMask, pp[j], d);
            uint32_t s;
            csa(s, c, pp[j], got, c);
            pp[j] = s;
        }
    }
    // the lane's word of the entry, and its share of the word's rows: bits
    // s, s + 8, s + 16, s + 24 for every s = share, share + NS, ... below 8
    constexpr int NS = 8 / LPE;
    const uint32_t word = 4 * q + 2 * ((lane >> 4) & 1) + ((lane >> 3) & 1);
    const uint32_t share = gi & (NS - 1);
#pragma unroll
    for (int u = 0; u < 8 / NS; ++u) {
        const uint32_t s = share + u * NS;
        uint32_t lo = 0u, hi = 0u;  // counts of the four rows, a byte each
#pragma unroll
        for (int j = 0; j < 8; ++j) lo |= ((pp[j] >> s) & 0x01010101u) << j;
#pragma unroll
        for (int j = 8; j < kPlanes; ++j) hi |= ((pp[j] >> s) & 0x01010101u) << (j - 8);
        if ((lo | hi) == 0u) continue;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t cnt = ((lo >> (8 * t)) & 0xffu) | (((hi >> (8 * t)) & 0xffu) << 8);
            if (cnt) sink(32 * word + s + 8 * t, cnt);
        }
    }
}

template <int E, bool kHash>
__device__ void slab_run(const SlabParams& p, const SlabPlan& plan, GroupRows& rows, uint32_t* s_ok) {
    uint32_t* err = reinterpret_cast<uint32_t*>(p.header);
    uint32_t* ticket = reinterpret_cast<uint32_t*>(p.header + kMisiSlabTicket);
    uint32_t* arrived = reinterpret_cast<uint32_t*>(p.header + kMisiSlabBarrier);
    const uint32_t lane = threadIdx.x & 31;
    constexpr uint32_t R = 32 * E;
    const Entries<kHash> en(p, plan);
    // Hash: at most this many distinct values are in the slots at once.  With
    // fewer in the whole span the slots are never emptied; otherwise they are
    // when the groups since then could fill half of them.
    const uint64_t cap = plan.slots / 2;
    const bool bounded = !kHash || uint64_t(plan.span) + 1 <= cap;
    uint64_t held = 0;  // elements inserted since the slots were emptied
    uint32_t epoch = 0;
    clear_table<E>(p, en.total());
    if constexpr (kHash) clear_slots(p, plan.slots);
    if (!grid_barrier(arrived, gridDim.x * ++epoch, err, s_ok)) return;
    // Cross tile: with few groups on one side, only that side's sets are rows,
    // and all of the other side's sets partners
    auto groups = [&](uint32_t n, const uint64_t* P) {
        const uint64_t g = (uint64_t(n) + R - 1) / R, h = bounded || n == 0 ? 0 : (P[n] + cap - 1) / cap;
        return g > h ? g : h;
    };
    const uint64_t groupsA = groups(p.nA, p.P), groupsB = groups(p.nB, p.P + p.nA + 1);
    const bool all = !p.self && min(groupsA, groupsB) <= kSlabAllGroups;
    bool dirty = false;  // the last group's bits are in the matrix: its rows [q0, q1) of the side before or this one
    uint32_t q0 = 0, q1 = 0, q_start = 0;
    const uint64_t *Kq = nullptr, *Pq = nullptr;
    for (int side = 0; side < (p.self ? 1 : 2); ++side) {
        const bool rowA = side == 0;
        if (all && rowA != (groupsA <= groupsB)) continue;
        const uint32_t nrows = rowA ? p.nA : p.nB, row_start = rowA ? p.a_start : p.b_start;
        const uint64_t* Kr = rowA ? p.keys : p.keys + p.nA;
        const uint64_t* Pr = rowA ? p.P : p.P + p.nA + 1;
        const uint32_t* cs = rowA ? p.cs : p.cs + p.nA;
        const bool partnersA = p.self || !rowA;
        const uint32_t nt = partnersA ? p.nA : p.nB, t_start = partnersA ? p.a_start : p.b_start;
        const uint64_t* Kt = partnersA ? p.keys : p.keys + p.nA;
        const uint64_t* Pt = partnersA ? p.P : p.P + p.nA + 1;
        for (uint32_t r0 = 0, r1; r0 < nrows; r0 = r1) {
            r1 = min(r0 + R, nrows);
            if (!bounded) {  // the rows that fill half of the slots (one set does not)
                const uint64_t full = Pr[r0] + cap;
                r1 = static_cast<uint32_t>(warp_first_true(r0 + 1, r1 + 1, [&](uint64_t q) { return Pr[q] > full; })) - 1;
                r1 = max(r1, r0 + 1);
            }
            const uint32_t c0 = all ? 0u : cs[r0];
            // partner c takes [cost(c), cost(c + 1)): its elements, then kSlabOver
            auto cost = [&](uint64_t c) { return Pt[c] + uint64_t(kSlabOver) * c; };
            const uint64_t w0 = cost(c0), w1 = cost(nt);
            if (c0 >= nt || Pt[nt] == Pt[c0] || Pr[r1] == Pr[r0]) break;  // nor has any later group partners
            const uint64_t n_group = Pr[r1] - Pr[r0];
            const bool empty_slots = !bounded && held + n_group > cap;
            if (dirty) {  // back to zero: the group's words, unless the whole matrix is fewer stores
                if (!empty_slots && (Pq[q1] - Pq[q0]) * 24 < uint64_t(en.total()) * E) {
                    group_elements<E, kHash, false>(p, en, Kq, Pq, q_start, q0, q1);
                } else {
                    clear_table<E>(p, en.total());
                    if (empty_slots) clear_slots(p, plan.slots);
                }
                if (!grid_barrier(arrived, gridDim.x * ++epoch, err, s_ok)) return;
            }
            held = empty_slots ? n_group : held + n_group;
            group_elements<E, kHash, true>(p, en, Kr, Pr, row_start, r0, r1);
            dirty = true;
            q0 = r0;
            q1 = r1;
            q_start = row_start;
            Kq = Kr;
            Pq = Pr;
            if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
            for (uint32_t i = threadIdx.x; i < r1 - r0; i += kSlabThreads) {
                const uint32_t id = static_cast<uint32_t>(Kr[r0 + i] & 0xffffffffu);
                rows.id[i] = id;
                rows.cs[i] = all ? 0u : cs[r0 + i];
                rows.base[i] = p.self ? tri_base(p.stride, id) : rowA ? uint64_t(id) * p.stride : id;
            }
            if (!grid_barrier(arrived, gridDim.x * ++epoch, err, s_ok)) return;

            const uint64_t share = (w1 - w0) / (uint64_t(gridDim.x) * kSlabWarps * 4);
            const uint64_t slice = max(uint64_t(kSlabSliceMin), min(uint64_t(kSlabSlice), share));
            for (;;) {
                uint32_t tk = 0;
                if (lane == 0) tk = atomicAdd(ticket, 1u);
                tk = __shfl_sync(kFullMask, tk, 0);
                const uint64_t lo = w0 + tk * slice;
                if (lo >= w1) break;
                const uint64_t hi = min(lo + slice, w1);
                // the partner holding position lo: the last c with cost(c) <= lo
                uint32_t c = static_cast<uint32_t>(
                    warp_first_true(c0, nt + 1, [&](uint64_t k) { return cost(k) > lo; }) - 1);
                // 32 partners at a time: lane l loads the piece of partner c + l
                for (; c < nt; c += 32) {
                    const uint32_t cl = c + lane;
                    uint32_t n = 0, my_id = 0;
                    uint64_t y0 = 0;
                    bool in = cl < nt, whole = false;
                    if (in) {
                        const uint64_t pt = Pt[cl], pc = pt + uint64_t(kSlabOver) * cl, size = Pt[cl + 1] - pt;
                        in = pc < hi;
                        const uint64_t ys = lo > pc ? lo - pc : 0, ye = in ? min(size, hi - pc) : 0;
                        if (ys < ye) {  // else an empty set, or the overhead of a partner counted before
                            n = static_cast<uint32_t>(ye - ys);
                            whole = ys == 0 && ye == size;
                            my_id = static_cast<uint32_t>(Kt[cl] & 0xffffffffu);
                            y0 = p.off[t_start + my_id] + ys;
                        }
                    }
                    const uint32_t whole_mask = __ballot_sync(kFullMask, whole);
                    for (uint32_t todo = __ballot_sync(kFullMask, n != 0); todo; todo &= todo - 1) {
                        const int l = __ffs(todo) - 1;
                        const uint32_t yid = __shfl_sync(kFullMask, my_id, l);
                        const uint64_t ybase = p.self ? tri_base(p.stride, yid) : rowA ? yid : uint64_t(yid) * p.stride;
                        const bool y_whole = (whole_mask >> l) & 1u;
                        const uint32_t cy = c + l;
                        count_partner<E>(p.el + __shfl_sync(kFullMask, y0, l), __shfl_sync(kFullMask, n, l), p.table,
                                         en, [&](uint32_t row, uint32_t cnt) {
                                             if (row >= r1 - r0 || rows.cs[row] > cy) return;  // a row smaller than y
                                             const uint32_t id = rows.id[row];
                                             const uint64_t idx = !p.self     ? rows.base[row] + ybase
                                                                  : id < yid ? rows.base[row] + yid
                                                                             : ybase + id;
                                             if (y_whole) p.counts[idx] = cnt;
                                             else atomicAdd(p.counts + idx, cnt);
                                         });
                    }
                    if (!__all_sync(kFullMask, in)) break;
                }
            }
            if (!grid_barrier(arrived, gridDim.x * ++epoch, err, s_ok)) return;
        }
    }
}

template <bool kHash>
__global__ void __launch_bounds__(kSlabThreads, kSlabCtasPerSm) misi_slab_kernel(SlabParams p) {
    __shared__ GroupRows rows;
    __shared__ uint32_t s_ok;
    const SlabPlan plan = slab_plan_of(kHash, p.nA, p.nB, p.header, p.P);
    switch (plan.words) {
        case 16: slab_run<16, kHash>(p, plan, rows, &s_ok); break;
        case 8: slab_run<8, kHash>(p, plan, rows, &s_ok); break;
        case 4: slab_run<4, kHash>(p, plan, rows, &s_ok); break;
        default: break;
    }
}

}  // namespace

si_status misi_slab(const SlabParams& p, si_technique t, cudaStream_t stream) {
    const auto kernel = t == SI_TECH_HI ? misi_slab_kernel<true> : misi_slab_kernel<false>;
    int per_sm = 0;
    SI_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSlabThreads, 0));
    if (per_sm < 1) return SI_ERR_UNSUPPORTED;
    SlabParams prm = p;
    void* args[] = {&prm};
    PhaseTimer timer("misi_slab", stream);
    SI_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel),
                                            dim3(static_cast<unsigned>(sm_count() * per_sm)), dim3(kSlabThreads), args,
                                            0, stream));
    return SI_OK;
}

}  // namespace si
