// si_misi_dense.cu -- all-pairs intersection counts of a dense collection.
//
// Two techniques for the same result, counts[tri(k, a, b)] = |S_a ∩ S_b| for
// every a < b (triangular layout of include/util.hpp:68-70):
//
//  * mm (src/matrix_multiplication.cu): the reference builds a 0/1 FP32
//    incidence matrix on the host and runs cublasSgemm per tile pair
//    (:139-184).  Here the incidence matrix M (k x U, one row per set) is
//    built on the device as 0/1 INT8 or FP8-e4m3, and C = M * M^T runs on the
//    5th-generation tensor cores: tcgen05.mma kind::i8 (s32 accumulation) or
//    kind::f8f6f4 (f32 accumulation), operands staged by TMA in 128-byte
//    swizzled K-major tiles, accumulators in tensor memory, only the tiles
//    of the upper triangle computed, only pairs a < b written.  Exact: every
//    partial sum is an integer <= U < 2^24.
//  * bitmap_naive (src/bitmap_naive.cu): every set as a bitmap, then AND +
//    popcount for every pair.  The reference gives each pair a grid-stride
//    loop and an atomic (:167-181); here it is the plain register-tiled
//    CUDA-core kernel the tensor-core path is compared against.
#include <algorithm>
#include <cstring>
#include <cuda.h>

#include "si_device.cuh"
#include "si_internal.h"

namespace si {
namespace {

// --------------------------------------------------------- tile geometry --
// A pair of CTAs (one cluster, two SMs) computes a tile of 256 x 256 kN counts,
// kN = 1 or 2: each CTA holds 128 rows of A and 128 kN rows of B,
// tcgen05.mma.cta_group::2 multiplies the pair's A with the pair's B.  Shared
// memory is what bounds it.  Per 32 bytes of K and 128 clocks of MMA an SM
//   kN = 1: writes 8 KiB of operands and reads 12 (its A, and its half of B for
//           itself and for the other SM): 160 clocks of its 128 bytes a clock;
//   kN = 2: writes 6 and reads 10 (A is kept in the collector for the second
//           MMA): 128 clocks.
// One SM by itself with a 128 x 256 tile writes 12 and reads 12: 192 clocks.
// Measured on 16384 sets over 65536 values, in the share of the tensor pipe's
// peak: alone 68 % (5.47 ms), kN = 1 80 % (4.65 ms), kN = 2 90 % (4.16 ms).
constexpr int kTile = 256;         // rows (sets a) and columns (sets b) of a pair's tile
constexpr int kHalf = 128;         // rows of A, and of B, in each CTA = TMEM lanes
constexpr int kTileK = 128;        // bytes of K per stage (one 128-byte swizzle span)
constexpr int kMmaK = 32;          // K of one tcgen05.mma for 8-bit operands
constexpr int kBand = 8;           // row panels per rasterisation band
constexpr int kEpiWarps = 8;       // warp w reads TMEM lanes 32 (w % 4) .., columns 128 kN (w / 4) ..
constexpr int kTmaWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1;
constexpr int kGemmThreads = (kEpiWarps + 2) * 32;
constexpr uint32_t kOperandBytes = kHalf * kTileK;       // 16 KiB: a stage's A of one CTA, or B of one MMA
constexpr uint32_t kRingBytes = 12 * kOperandBytes;      // the stages: 6 (kN = 1) or 4 (kN = 2)
template <int kN>
constexpr uint32_t kStageBytes = (1 + kN) * kOperandBytes;
template <int kN>
constexpr uint32_t kStages = kRingBytes / kStageBytes<kN>;
constexpr uint32_t kBlockWords = 32 * 33;                // an epilogue warp's 32 x 32 counts, padded
constexpr size_t kGemmSmem = size_t(kRingBytes) + kEpiWarps * kBlockWords * 4 + 1024;  // + alignment slack
constexpr uint32_t kAccCols = kTile;  // one s32/f32 column per output column
constexpr uint32_t kTmemCols = 2 * kAccCols;  // kN = 1: one is read out while the other fills; kN = 2: the tile's two
constexpr uint32_t kSplitStages = 16;  // a part of a tile is at least this many stages of K

__host__ __device__ inline uint64_t tri_index(uint64_t n, uint64_t i, uint64_t j) {
    return (n * (n - 1) / 2) - (n - i) * ((n - i) - 1) / 2 + j - i - 1;
}

// Upper-triangle tiles: tile (i, j) covers rows [256 i, 256 i + 256) x columns
// [256 kN j, 256 kN (j + 1)) and is needed iff it holds a pair a < b, i.e.
// j >= i / kN; T row panels, J column panels.  Order: bands of kBand row panels;
// in a band, column panel by column panel, the band's row panels inside -- so
// the pairs running at the same time share a handful of panels in L2.
__host__ __device__ inline uint32_t band_tiles(uint32_t T, uint32_t J, uint32_t nN, uint32_t b) {
    uint32_t n = 0;
    for (uint32_t i = b * kBand; i < min((b + 1) * kBand, T); ++i) n += J - i / nN;
    return n;
}

__device__ inline void tile_of(uint32_t L, uint32_t T, uint32_t J, uint32_t nN, uint32_t& ti, uint32_t& tj) {
    uint32_t b = 0;
    for (;; ++b) {
        const uint32_t n = band_tiles(T, J, nN, b);
        if (L < n) break;
        L -= n;
    }
    const uint32_t i0 = b * kBand, i1 = min(i0 + kBand, T);
    // column panel j of the band holds the rows from i0 with i / nN <= j
    uint32_t j = i0 / nN;
    for (;; ++j) {
        const uint32_t cnt = min(i1, nN * (j + 1)) - i0;
        if (L < cnt) break;
        L -= cnt;
    }
    ti = i0 + L;
    tj = j;
}

// Who computes what.  Every pair takes whole tiles, as many as all pairs can;
// each of the tiles left over is cut along K into `cuts` parts for as many
// pairs, whose counts are added atomically into counts that the incidence
// kernel has zeroed.  Pairs with the same part of K run side by side, so they
// share panels in L2 (equal shares of the left-over tiles' stages, whatever tile
// they fall in, read them from HBM instead: 5000 sets over 65536 values took
// 669 us a call that way, 598 us this way).
struct Schedule {
    uint32_t T, J, nN;  // row panels, column panels, kN
    uint32_t tiles;
    uint32_t whole;     // tiles computed whole by all pairs (a multiple of the pairs)
    uint32_t stages;    // K stages of a tile
    uint32_t cuts;      // parts of each tile left over (1: it is whole too)
};

struct Work {
    uint32_t tile, k0, k1;  // stages [k0, k1) of a tile
};

// Item n of pair w's work; false when there is none.
__device__ __forceinline__ bool work_item(const Schedule& sc, uint32_t pairs, uint32_t w, uint32_t n, Work& out) {
    const uint32_t rounds = sc.whole / pairs, left = sc.tiles - sc.whole;
    if (n < rounds) {
        out = {w + n * pairs, 0, sc.stages};
        return true;
    }
    if (n > rounds || w >= left * sc.cuts) return false;
    const uint32_t part = w / left;
    out = {sc.whole + w % left, static_cast<uint32_t>(uint64_t(sc.stages) * part / sc.cuts),
           static_cast<uint32_t>(uint64_t(sc.stages) * (part + 1) / sc.cuts)};
    return true;
}

// ---------------------------------------------------------------- PTX ---
// The same shared-memory address in the cluster's CTA `rank`.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrives on an mbarrier of another CTA of the cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Bounded wait on a phase that warps of both CTAs complete.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, uint32_t* err, uint32_t site,
                                                  uint32_t info) {
    WaitBudget budget;
    do {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    } while (!budget.expired());
    record_error(err, SI_ERR_TIMEOUT, site, info);
    return false;
}

// A box of the matrix into this CTA's shared memory; bar (a cluster address)
// is a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
        "%3}], [%4];" ::"r"(smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// TMEM of both CTAs of a pair: a warp of each makes the call.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 128-byte swizzled, K-major operand tile: 8-row core groups of 1024 bytes
// (SBO = 1024), leading offset unused (1), descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t smem_desc_sw128(const void* base) {
    const uint64_t addr = smem_addr(base);
    uint64_t d = 0;
    d |= (addr >> 4) & 0x3fffull;             // start address
    d |= uint64_t(1) << 16;                   // leading byte offset (unused for swizzled K-major)
    d |= uint64_t(1024 >> 4) << 32;           // stride byte offset
    d |= uint64_t(1) << 46;                   // version
    d |= uint64_t(2) << 61;                   // SWIZZLE_128B
    return d;
}

// Instruction descriptor: D format, A/B formats, both K-major, N, M.
template <bool kFp8>
__host__ __device__ constexpr uint32_t instr_desc() {
    // kind::i8: D = s32 (2), A = B = unsigned 8-bit (0).  kind::f8f6f4: D = f32 (1), A = B = E4M3 (0).
    return (kFp8 ? (1u << 4) : (2u << 4)) | (uint32_t(kTile >> 3) << 17) | (uint32_t(kTile >> 4) << 24);
}

// kA: 0 = A is used once, 1 = keep A in the collector, 2 = take it from there
// (the next MMA's A is the same / the last one's was).
template <bool kFp8, int kA>
__device__ __forceinline__ void mma_issue(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
    constexpr uint32_t idesc = instr_desc<kFp8>();
#define SI_MMA(kind, collector)                                                                                   \
    asm volatile("{\n\t.reg .pred p;\n\t"                                                                        \
                 "setp.ne.b32 p, %4, 0;\n\t"                                                                     \
                 "tcgen05.mma.cta_group::2.kind::" kind ".collector::a::" collector " [%0], %1, %2, %3, p;\n\t}" \
                 ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)                                     \
                 : "memory")
    if constexpr (kFp8) {
        if constexpr (kA == 0) SI_MMA("f8f6f4", "discard");
        if constexpr (kA == 1) SI_MMA("f8f6f4", "fill");
        if constexpr (kA == 2) SI_MMA("f8f6f4", "lastuse");
    } else {
        if constexpr (kA == 0) SI_MMA("i8", "discard");
        if constexpr (kA == 1) SI_MMA("i8", "fill");
        if constexpr (kA == 2) SI_MMA("i8", "lastuse");
    }
#undef SI_MMA
}

// Arrives on `bar` in both CTAs of the pair once every tcgen05.mma issued so
// far by this thread is done.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_addr(bar)),
        "h"(static_cast<uint16_t>(3))
        : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ------------------------------------------------------ incidence build --
// One CTA per row of M: the row is assembled in shared memory 32 KiB of
// columns at a time (zeros, then a `one` byte at every element of the set
// inside the chunk) and written out with 16-byte stores; rows >= k are all
// zero.  The set is read once, in order: each chunk's loop stops at the first
// element past the chunk, which is where the next chunk starts.
constexpr uint32_t kChunk = 32768;
constexpr uint32_t kZeroBlocks = 32;  // blocks per cut tile, ahead of the rows' blocks
static_assert(kTile == 256, "a thread zeroes a column of 256");
__global__ void __launch_bounds__(256) build_incidence_kernel(const uint32_t* __restrict__ elements,
                                                              const uint64_t* __restrict__ offsets, uint32_t k,
                                                              uint8_t* __restrict__ M, uint64_t row_bytes,
                                                              uint32_t universe, uint8_t one, uint32_t* err,
                                                              Schedule sc,
                                                              uint32_t* __restrict__ counts) {
    __shared__ __align__(16) uint8_t chunk[kChunk];
    __shared__ unsigned long long s_next;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t zero_blocks = sc.cuts > 1 ? (sc.tiles - sc.whole) * kZeroBlocks : 0u;
    if (blockIdx.x < zero_blocks) {  // zero a cut tile's counts, which its parts add into
        constexpr uint32_t kRows = kTile / kZeroBlocks;
        uint32_t ti, tj;
        tile_of(sc.whole + blockIdx.x / kZeroBlocks, sc.T, sc.J, sc.nN, ti, tj);
        const uint64_t a0 = uint64_t(ti) * kTile + blockIdx.x % kZeroBlocks * kRows;
        for (uint32_t u = 0; u < sc.nN; ++u) {
            const uint64_t b = (uint64_t(tj) * sc.nN + u) * kTile + threadIdx.x;
#pragma unroll
            for (uint32_t r = 0; r < kRows; ++r)
                if (a0 + r < b && b < k) counts[tri_index(k, a0 + r, b)] = 0u;
        }
        return;
    }
    const uint32_t row = blockIdx.x - zero_blocks;
    uint4* c4 = reinterpret_cast<uint4*>(chunk);
    uint64_t lo = 0, e = 0;
    if (row < k) {
        lo = offsets[row];
        e = offsets[row + 1];
    }
    for (uint64_t c0 = 0; c0 < row_bytes; c0 += kChunk) {
        const uint64_t rem = row_bytes - c0;
        const uint32_t n16 = static_cast<uint32_t>((rem < kChunk ? rem : kChunk) / 16);
        for (uint32_t x = threadIdx.x; x < n16; x += blockDim.x) c4[x] = make_uint4(0, 0, 0, 0);
        if (threadIdx.x == 0) s_next = e;
        __syncthreads();
        for (uint64_t x = lo + threadIdx.x; x < e; x += blockDim.x) {
            const uint64_t v = __ldg(elements + x);
            if (v >= c0 + kChunk) {  // this thread's first element past the chunk
                atomicMin(&s_next, static_cast<unsigned long long>(x));
                break;
            }
            if (v < c0 || v > universe) { record_error(err, SI_ERR_INVALID_INPUT, 20, row); continue; }
            chunk[v - c0] = one;
        }
        __syncthreads();
        uint4* dst = reinterpret_cast<uint4*>(M + static_cast<uint64_t>(row) * row_bytes + c0);
        for (uint32_t x = threadIdx.x; x < n16; x += blockDim.x) dst[x] = c4[x];
        lo = s_next;
        __syncthreads();  // the chunk and s_next are rewritten for the next columns
    }
}

// ----------------------------------------------------- tensor-core GEMM --
// Persistent pairs.  Per CTA: warp 8 loads its halves of A and B, stage by
// stage, onto the leader CTA's barrier; warp 9 of the leader (rank 0) issues
// the MMAs of the pair; warps 0..7 read the finished accumulator out while the
// next tile fills the other one.
template <bool kFp8, int kN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap map, uint32_t k, const Schedule sc,
                   uint32_t* __restrict__ counts, uint32_t* err) {
    extern __shared__ uint8_t dsmem[];
    // operand stages must start on 1024-byte boundaries (swizzle atoms)
    uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dsmem) + 1023) & ~uintptr_t(1023));
    uint32_t* blocks = reinterpret_cast<uint32_t*>(stages + kRingBytes);
    constexpr uint32_t nStages = kStages<kN>, stageBytes = kStageBytes<kN>;
    constexpr uint32_t nAcc = 2 / kN;  // accumulators
    // full: the leader's, both CTAs' bytes of a stage; empty: each CTA's, the
    // MMAs have read the stage; acc_full: each CTA's, an accumulator is done;
    // acc_empty: the leader's, all epilogue warps of the pair have read it
    __shared__ __align__(8) uint64_t full[nStages], empty[nStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t s_tmem;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank(), pair = blockIdx.x / 2, pairs = gridDim.x / 2;

    if (tid == 0) {
        for (uint32_t s = 0; s < nStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 2 * kEpiWarps);
        }
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(&s_tmem, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers and TMEM are ready
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the matrix, and the zeroed counts

    if (warp == kTmaWarp) {
        if (lane == 0) {
            uint32_t g = 0;  // stages loaded so far
            bool ok = true;
            Work wk;
            for (uint32_t n = 0; ok && work_item(sc, pairs, pair, n, wk); ++n) {
                uint32_t ti, tj;
                tile_of(wk.tile, sc.T, sc.J, sc.nN, ti, tj);
                const int ya = static_cast<int>(ti * kTile + rank * kHalf);
                const int yb = static_cast<int>(tj * kTile * kN + rank * kHalf);
                for (uint32_t ks = wk.k0; ks < wk.k1; ++ks, ++g) {
                    const uint32_t s = g % nStages, round = g / nStages;
                    ok = mbar_wait_bounded(&empty[s], (round & 1) ^ 1, err, 21, ks);
                    if (!ok) break;
                    uint8_t* sa = stages + s * stageBytes;
                    const uint32_t bar = cluster_addr(&full[s], 0);
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * stageBytes);
                    tma_load_2d(sa, &map, static_cast<int>(ks * kTileK), ya, bar);
#pragma unroll
                    for (int h = 0; h < kN; ++h)
                        tma_load_2d(sa + (1 + h) * kOperandBytes, &map, static_cast<int>(ks * kTileK), yb + h * kTile, bar);
                }
            }
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        if (rank == 0 && lane == 0) {
            uint32_t g = 0;
            bool ok = true;
            Work wk;
            for (uint32_t n = 0; ok && work_item(sc, pairs, pair, n, wk); ++n) {
                const uint32_t acc = n % nAcc;
                ok = mbar_wait_cluster(&acc_empty[acc], ((n / nAcc) & 1) ^ 1, err, 25, n);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + acc * kAccCols;
                for (uint32_t ks = wk.k0; ks < wk.k1; ++ks, ++g) {
                    const uint32_t s = g % nStages, round = g / nStages;
                    ok = mbar_wait_bounded(&full[s], round & 1, err, 22, ks);
                    if (!ok) break;
                    tc_fence_after();
                    const uint8_t* sa = stages + s * stageBytes;
                    const uint64_t da = smem_desc_sw128(sa), db = smem_desc_sw128(sa + kOperandBytes);
#pragma unroll
                    for (int kk = 0; kk < kTileK / kMmaK; ++kk) {
                        // advance 32 bytes along K inside the swizzle span: +2 in the 16-byte address field
                        const uint32_t more = ks != wk.k0 || kk != 0;
                        mma_issue<kFp8, kN == 1 ? 0 : 1>(d, da + 2 * kk, db + 2 * kk, more);
                        if constexpr (kN == 2)
                            mma_issue<kFp8, 2>(d + kAccCols, da + 2 * kk, db + kOperandBytes / 16 + 2 * kk, more);
                    }
                    mma_commit(&empty[s]);  // the stage is free once these MMAs have read it
                }
                if (ok) mma_commit(&acc_full[acc]);
            }
        }
        __syncwarp();
    } else {
        uint32_t* blk = blocks + warp * kBlockWords;
        Work wk;
        for (uint32_t n = 0; work_item(sc, pairs, pair, n, wk); ++n) {
            const uint32_t acc = n % nAcc;
            // warp-uniform: the TMEM loads below are .sync.aligned
            if (!__all_sync(kFullMask, mbar_wait_bounded(&acc_full[acc], (n / nAcc) & 1, err, 23, n))) break;
            tc_fence_after();
            uint32_t ti, tj;
            tile_of(wk.tile, sc.T, sc.J, sc.nN, ti, tj);
            const bool whole = sc.cuts == 1 || wk.tile < sc.whole;
            const uint64_t a_first = uint64_t(ti) * kTile + rank * kHalf + (warp & 3) * 32;
            const uint64_t b_first = uint64_t(tj) * kTile * kN + (warp >> 2) * kHalf * kN;
            // TMEM lane l holds row a_first + l.  Each 32 x 32 block of counts
            // goes through a padded shared tile, so that each store writes 32
            // consecutive counts of one row; the index of (a, b) moves by
            // k - a - 2 from one row to the next.
            const uint32_t t0 =
                tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + acc * kAccCols + (warp >> 2) * kHalf * kN;
            const uint32_t rows = a_first < k ? static_cast<uint32_t>(min(uint64_t(32), k - a_first)) : 0u;
#pragma unroll 1
            for (int c = 0; c < kHalf * kN; c += 32) {
                const uint64_t b0 = b_first + c, b = b0 + lane;
                if (rows == 0 || b0 >= k || b0 + 31 <= a_first) continue;  // outside, or below the diagonal
                uint32_t v[32];
                tmem_ld32(t0 + static_cast<uint32_t>(c), v);
#pragma unroll
                for (int x = 0; x < 32; ++x)
                    blk[lane * 33 + x] = kFp8 ? static_cast<uint32_t>(__uint_as_float(v[x])) : v[x];
                __syncwarp();
                uint32_t* out = counts + (tri_index(k, a_first, a_first + 1) + (b - a_first - 1));
                uint64_t step = k - a_first - 2;
                // lane's rows: those before b, none when b is past the sets
                const uint32_t n = b >= k ? 0u : b <= a_first ? 0u : static_cast<uint32_t>(min(uint64_t(rows), b - a_first));
                if (whole) {
#pragma unroll 8
                    for (uint32_t r = 0; r < 32; ++r) {
                        if (r < n) *out = blk[r * 33 + lane];
                        out += step--;
                    }
                } else {
#pragma unroll 8
                    for (uint32_t r = 0; r < 32; ++r) {
                        const uint32_t x = blk[r * 33 + lane];
                        if (r < n && x) atomicAdd(out, x);
                        out += step--;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[acc], 0));
        }
        __syncwarp();
    }
    // A wait that gave up ends its role; the others' waits then give up in
    // turn, seconds after the last copy was issued.
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // neither CTA leaves while the other may still signal it or read its operands
    if (warp == kMmaWarp) tmem_dealloc(tmem, kTmemCols);
}

// ------------------------------------------- plain AND-popcount (CUDA cores) --
// Bitmaps: one row of W 32-bit words per set (bit v of set a: word v/32, bit v%32).
__global__ void __launch_bounds__(256) build_bitmaps_kernel(const uint32_t* __restrict__ elements,
                                                            const uint64_t* __restrict__ offsets, uint32_t k,
                                                            uint32_t* __restrict__ bits, uint32_t W, uint32_t universe,
                                                            uint32_t* err) {
    extern __shared__ uint32_t row[];
    const uint32_t a = blockIdx.x;
    for (uint32_t w = threadIdx.x; w < W; w += blockDim.x) row[w] = 0u;
    __syncthreads();
    if (a < k) {
        for (uint64_t x = offsets[a] + threadIdx.x; x < offsets[a + 1]; x += blockDim.x) {
            const uint32_t v = __ldg(elements + x);
            if (v > universe) { record_error(err, SI_ERR_INVALID_INPUT, 24, a); continue; }
            atomicOr(row + (v >> 5), 1u << (v & 31));
        }
    }
    __syncthreads();
    for (uint32_t w = threadIdx.x; w < W; w += blockDim.x) bits[static_cast<uint64_t>(a) * W + w] = row[w];
}

// 128 x 128 pair tiles, 256 threads, 8 x 8 pairs per thread (rows ty + 16i,
// columns tx + 16j, so a warp's shared loads hit distinct banks or broadcast);
// K staged 16 words at a time through shared memory (double-buffered).  Only
// tiles with a < b.
constexpr int kPopTile = 128, kPopK = 16, kPopThreads = 256;
__global__ void __launch_bounds__(kPopThreads) popcount_gemm_kernel(const uint32_t* __restrict__ bits, uint32_t k,
                                                                    uint32_t W, uint32_t T,
                                                                    uint32_t* __restrict__ counts) {
    // linear upper-triangle tile index -> (ti <= tj)
    uint32_t L = blockIdx.x, ti = 0;
    while (L >= T - ti) { L -= T - ti; ++ti; }
    const uint32_t tj = ti + L;
    __shared__ uint32_t sa[2][kPopK][kPopTile + 1], sb[2][kPopK][kPopTile + 1];
    const int tid = threadIdx.x;
    const int ty = tid / 16, tx = tid % 16;  // 16 x 16 threads, 8 x 8 each
    uint32_t acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0u;
    const uint64_t rowA0 = static_cast<uint64_t>(ti) * kPopTile, rowB0 = static_cast<uint64_t>(tj) * kPopTile;
    auto load = [&](int buf, uint32_t w0) {
        for (int x = tid; x < kPopTile * kPopK; x += kPopThreads) {
            const int r = x / kPopK, c = x % kPopK;
            const uint64_t ra = rowA0 + r, rb = rowB0 + r;
            sa[buf][c][r] = (ra < k && w0 + c < W) ? __ldg(bits + ra * W + w0 + c) : 0u;
            sb[buf][c][r] = (rb < k && w0 + c < W) ? __ldg(bits + rb * W + w0 + c) : 0u;
        }
    };
    load(0, 0);
    __syncthreads();
    const uint32_t nk = (W + kPopK - 1) / kPopK;
    for (uint32_t kb = 0; kb < nk; ++kb) {
        const int buf = kb & 1;
        if (kb + 1 < nk) load(buf ^ 1, (kb + 1) * kPopK);
#pragma unroll 4
        for (int c = 0; c < kPopK; ++c) {
            uint32_t x[8], y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = sa[buf][c][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = sb[buf][c][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] += __popc(x[i] & y[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint64_t a = rowA0 + ty + 16 * i;
        if (a >= k) continue;
        const uint64_t rowbase = tri_index(k, a, a + 1) - (a + 1);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint64_t b = rowB0 + tx + 16 * j;
            if (b > a && b < k) counts[rowbase + b] = acc[i][j];
        }
    }
}

// ---------------------------------------------------------------- host --
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

struct DenseLayout {
    uint32_t k_pad = 0;       // rows of M (multiple of 256)
    uint64_t row_bytes = 0;   // columns of M: universe + 1 rounded up to kTileK
    uint32_t W = 0;           // bitmap words per set
    size_t off_matrix = 0, total = 0;
};
constexpr size_t kDenseHeader = 256;  // error words

Schedule make_schedule(uint32_t T, uint32_t stages, uint32_t nN, uint32_t pairs) {
    Schedule sc;
    sc.T = T;
    sc.J = (T + nN - 1) / nN;
    sc.nN = nN;
    sc.stages = stages;
    uint64_t tiles = 0;
    for (uint32_t i = 0; i < T; ++i) tiles += sc.J - i / nN;
    sc.tiles = tiles > 0x7fffffffull ? 0xffffffffu : static_cast<uint32_t>(tiles);
    sc.whole = sc.tiles / pairs * pairs;
    const uint32_t left = sc.tiles - sc.whole;
    sc.cuts = left ? std::max(1u, std::min(pairs / left, stages / kSplitStages)) : 1u;
    return sc;
}

// Time of a schedule in units of one stage's MMAs at the tensor pipe's peak
// (512 clocks).  A stage of the narrow tile takes 1.25 units, of the wide one,
// twice the work, 2.1; a round's read-out that the next tile does not hide (the
// wide tile's accumulators fill TMEM, so all of it) 18 and 60, and half as much
// again where the parts of a cut tile are added atomically.  Fitted to 1000 ..
// 16384 sets over 2000 .. 65536 values; the wide tile is taken from 5000 sets
// over 40009 values on (376 -> 367 us; 16384 over 65536 4.94 -> 4.45 ms), not for
// 5000 over 10000 (113 us against 139) or 3001 over 40009 (166 against 227).
double schedule_cost(const Schedule& sc, uint32_t pairs) {
    const double stage = (sc.nN == 2 ? 2.1 : 1.25) * sc.stages, out = sc.nN == 2 ? 60 : 18;
    double t = (sc.whole / pairs) * (stage + out);
    if (sc.tiles > sc.whole) t += stage / sc.cuts + (sc.cuts > 1 ? 1.5 * out : out);
    return t;
}

DenseLayout dense_layout(uint32_t k, uint32_t universe, si_technique t) {
    DenseLayout L;
    const uint64_t U = static_cast<uint64_t>(universe) + 1;  // values 0..universe
    L.off_matrix = kDenseHeader;
    if (t == SI_TECH_BITMAP_NAIVE) {
        L.W = static_cast<uint32_t>((U + 31) / 32);
        L.total = L.off_matrix + static_cast<uint64_t>(k) * L.W * 4;
    } else {
        L.k_pad = (k + kTile - 1) / kTile * kTile;
        L.row_bytes = (U + kTileK - 1) / kTileK * kTileK;
        L.total = L.off_matrix + static_cast<uint64_t>(L.k_pad) * L.row_bytes;
    }
    return L;
}

}  // namespace

size_t dense_workspace_size(uint32_t k, uint32_t universe, si_technique t) {
    return dense_layout(k, universe, t).total;
}

si_status misi_dense(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, uint32_t universe,
                     si_technique t, int fp8, uint32_t* d_counts, void* ws, size_t ws_bytes, cudaStream_t stream) {
    const DenseLayout L = dense_layout(k, universe, t);
    if (ws_bytes < L.total) return SI_ERR_WORKSPACE_TOO_SMALL;
    unsigned char* w = static_cast<unsigned char*>(ws);
    uint32_t* err = reinterpret_cast<uint32_t*>(w);
    SI_CUDA_TRY(cudaMemsetAsync(w, 0, kDenseHeader, stream));
    if (k < 2) return SI_OK;

    if (t == SI_TECH_BITMAP_NAIVE) {
        uint32_t* bits = reinterpret_cast<uint32_t*>(w + L.off_matrix);
        const size_t row_smem = static_cast<size_t>(L.W) * 4;
        if (row_smem > 200 * 1024) return SI_ERR_UNSUPPORTED;  // universe above ~6.5M values
        SI_CUDA_TRY(cudaFuncSetAttribute(build_bitmaps_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(row_smem)));
        {
            PhaseTimer timer("naive_bitmaps", stream);
            build_bitmaps_kernel<<<k, 256, row_smem, stream>>>(d_elements, d_offsets, k, bits, L.W, universe, err);
        }
        SI_LAUNCH_CHECK("build_bitmaps_kernel");
        const uint32_t T = (k + kPopTile - 1) / kPopTile;
        const uint64_t ntiles = static_cast<uint64_t>(T) * (T + 1) / 2;
        if (ntiles > 0x7fffffffull) return SI_ERR_UNSUPPORTED;
        PhaseTimer timer("naive_popcount", stream);
        popcount_gemm_kernel<<<static_cast<unsigned>(ntiles), kPopThreads, 0, stream>>>(bits, k, L.W, T, d_counts);
        SI_LAUNCH_CHECK("popcount_gemm_kernel");
        return SI_OK;
    }

    // ---- mm on tensor cores ----
    uint8_t* M = reinterpret_cast<uint8_t*>(w + L.off_matrix);
    const uint32_t pairs_max = std::max(1, sm_count() / 2);
    const uint32_t nks = static_cast<uint32_t>(L.row_bytes / kTileK);
    Schedule sc = make_schedule(L.k_pad / kTile, nks, 1, pairs_max);
    const Schedule wide = make_schedule(L.k_pad / kTile, nks, 2, pairs_max);
    if (schedule_cost(wide, pairs_max) < schedule_cost(sc, pairs_max)) sc = wide;
    if (sc.tiles > 0x7fffffffu) return SI_ERR_UNSUPPORTED;
    auto kern = sc.nN == 2 ? (fp8 ? tc_gemm_kernel<true, 2> : tc_gemm_kernel<false, 2>)
                           : (fp8 ? tc_gemm_kernel<true, 1> : tc_gemm_kernel<false, 1>);
    SI_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kGemmSmem)));
    const uint32_t left = sc.tiles - sc.whole;
    const uint32_t pairs = sc.whole ? pairs_max : left * sc.cuts;
    const uint32_t zero_blocks = sc.cuts > 1 ? left * kZeroBlocks : 0u;
    {
        PhaseTimer timer("mm_incidence", stream);
        build_incidence_kernel<<<L.k_pad + zero_blocks, 256, 0, stream>>>(
            d_elements, d_offsets, k, M, L.row_bytes, universe, fp8 ? uint8_t(0x38) : uint8_t(1),  // 1.0 in e4m3 = 0x38
            err, sc, d_counts);
    }
    SI_LAUNCH_CHECK("build_incidence_kernel");

    EncodeTiledFn enc = encode_tiled();
    if (!enc) return cuda_fail(cudaErrorNotSupported, "cuTensorMapEncodeTiled unavailable");
    CUtensorMap map;
    const cuuint64_t gdim[2] = {L.row_bytes, L.k_pad};
    const cuuint64_t gstride[1] = {L.row_bytes};
    const cuuint32_t estride[2] = {1, 1};
    const cuuint32_t box[2] = {kTileK, kHalf};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, M, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cuda_fail(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");

    PhaseTimer timer("mm_gemm", stream);
    const si_status st = launch_dependent(kern, dim3(2 * pairs), dim3(kGemmThreads), kGemmSmem, stream, map, k, sc,
                                          d_counts, err);
    if (st != SI_OK) return st;
    SI_LAUNCH_CHECK("tc_gemm_kernel");
    return SI_OK;
}

}  // namespace si
