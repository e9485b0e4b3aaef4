// si_internal.h -- host-side interfaces between the C-ABI layer (si_api.cu)
// and the per-technique launchers.  Not installed; C++ only.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "si.h"

namespace si {

// Records a CUDA error text for si_last_error_string and returns SI_ERR_CUDA.
si_status cuda_fail(cudaError_t e, const char* what);

#define SI_CUDA_TRY(expr)                                                 \
    do {                                                                  \
        cudaError_t si_e_ = (expr);                                       \
        if (si_e_ != cudaSuccess) return ::si::cuda_fail(si_e_, #expr);   \
    } while (0)

#define SI_LAUNCH_CHECK(what)                                             \
    do {                                                                  \
        cudaError_t si_e_ = cudaGetLastError();                           \
        if (si_e_ != cudaSuccess) return ::si::cuda_fail(si_e_, what);    \
    } while (0)

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Number of SMs of the current device (cached per device).
int sm_count();

// Launches `kernel` with programmatic stream serialization: it may start while
// the previous kernel on the stream finishes, and must execute
// griddepcontrol.wait before it reads that kernel's results (or writes what
// that kernel still reads).  It reads them by plain or L2 loads: __ldg, or
// const __restrict__ on the parameter, would promise that nobody writes them
// while it runs, and let the compiler move the loads above the wait.
template <class Kernel, class... Args>
si_status launch_dependent(Kernel kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SI_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
    return SI_OK;
}

// Named phase timing on the launching stream (the engine's counterpart of the
// reference's DeviceTimer, include/device_timer.cuh:20-78).  When enabled via
// si_timer_enable, PhaseTimer records a cudaEvent pair around a launch.
class PhaseTimer {
public:
    PhaseTimer(const char* name, cudaStream_t stream);
    ~PhaseTimer();
    PhaseTimer(const PhaseTimer&) = delete;
    PhaseTimer& operator=(const PhaseTimer&) = delete;
private:
    int slot_;
    cudaStream_t stream_;
};

// ---- one pair ----
// Intersect path (si_sisi_ip.cu).
constexpr uint64_t kIpOneTile = 192 * 27;  // a tile of ip: elements of both sets that one CTA merges
constexpr uint64_t kObsOneChunk = 256;     // obs: elements of the smaller set that one CTA searches
size_t ip_workspace_size(uint64_t nA, uint64_t nB);
si_status ip_sisi(const uint32_t* dA, uint64_t nA, const uint32_t* dB, uint64_t nB, uint64_t* d_count,
                  uint32_t* d_out, uint64_t out_cap, void* ws, size_t ws_bytes, cudaStream_t stream);
// The stream engine of si_sisi_bitmap.cu: window bitmaps (technique bitmap)
// or, with hash set, window hash tables (technique hi) on the same ranges.
size_t bm_workspace_size(uint64_t nA, uint64_t nB);
si_status bm_sisi(const uint32_t* dA, uint64_t nA, const uint32_t* dB, uint64_t nB, uint64_t* d_count,
                  uint32_t* d_out, uint64_t out_cap, void* ws, size_t ws_bytes, cudaStream_t stream,
                  bool hash = false);
// What SI_TECH_AUTO runs for a pair.  Device time with elements out (counted
// only), us:
//                       ip           bitmap       obs
//   2^20 x 2^20           17 (8)       36 (25)      25 (21)
//   2^23 x 2^23           43 (23)      45 (31)      159 (138)
//   2^24 x 2^24           77           63
//   2^17, 1/16 of it      8.7 (5.0)                 6.6 (5.2)
//   2^17, 1/32            8.7 (5.0)                 6.7 (5.6)
//   2^20, 1/16            11.0 (6.0)                7.3 (6.1)
//   2^22, 1/8             17.7 (9.5)   25.7 (16.7)  17.1 (14.2)
//   2^22, 1/16            17.1 (9.1)   24.6 (16.5)  12.0 (10.0)
//   2^22, 1/32            16.4 (8.9)   23.2 (16.4)  9.1 (7.7)
//   2^24, 1/16            36 (20)      37 (27)      28 (24)
//   2^24, 1/32            36 (19)      37 (27)      19 (16)
//   2^27, 1/16            204 (130)    155 (115)    210 (185)
//   2^27, 1/32            192 (122)    147 (111)    139 (125)
//   2^27, 1/64            187 (117)    141 (108)    110 (101)
// (uniform values).  A pair of one merge tile is one launch of ip: 3.8 us against
// 4.2 and more.  Only counted, pairs up to 1.25 x 2^20 elements are merged too:
// over six distributions (uniform, powers, clusters at twelve scales, runs of
// 512, fractal) the larger set's 2^18, 2^20 and 3 x 2^19 elements take ip 5.1, 5.6
// and 6.1 us, obs 5.8, 6.0 and 6.1, the worst distribution 1.4, 1.4 and 1.2 times
// ip; not so when one CTA can search and count (up to 256 elements, 3.0-4.3 us).
// With elements out no distribution at these ratios takes obs longer than ip.
inline si_technique sisi_auto(uint64_t nA, uint64_t nB, bool elements) {
    const uint64_t small = nA < nB ? nA : nB, large = nA < nB ? nB : nA, total = nA + nB;
    const uint64_t ratio = elements && total <= (1ull << 25) ? 16 : total <= (1ull << 27) ? 32 : 64;
    if (total > (elements || small <= kObsOneChunk ? kIpOneTile : 5ull << 18) && small <= large / ratio) return SI_TECH_OBS;
    return total <= (1ull << 24) ? SI_TECH_IP : SI_TECH_BITMAP;
}
size_t obs_workspace_size(uint64_t nA, uint64_t nB);
si_status obs_sisi(const uint32_t* dA, uint64_t nA, const uint32_t* dB, uint64_t nB, uint64_t* d_count,
                   uint32_t* d_out, void* ws, size_t ws_bytes, cudaStream_t stream);

// ---- all pairs of a dense collection (si_misi_dense.cu) ----
// t: SI_TECH_MM (tensor cores; fp8 selects FP8-e4m3 operands instead of INT8)
// or SI_TECH_BITMAP_NAIVE (plain AND-popcount on CUDA cores).
size_t misi_workspace_size(si_set_range A, si_set_range B, si_technique t);
si_status misi_tile(const uint32_t* d_elements, const uint64_t* d_offsets, si_technique t, si_set_range A,
                    si_set_range B, uint64_t stride, uint32_t* d_counts, void* ws, size_t ws_bytes,
                    cudaStream_t stream);
size_t batch_workspace_size(uint64_t npairs);
si_status batch_count(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, const uint32_t* d_pairs,
                      uint64_t npairs, si_technique t, const uint8_t* table, uint32_t* d_counts, void* ws,
                      size_t ws_bytes, cudaStream_t stream);
si_status batch_tune(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, const uint32_t* d_pairs,
                     uint64_t npairs, uint32_t sample, uint32_t* d_counts, void* ws, size_t ws_bytes,
                     cudaStream_t stream, uint8_t* table_out);
size_t degree_workspace_size();
si_status degree_stats(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, uint64_t n_elements,
                       uint64_t slots, uint32_t* d_inv, uint64_t* d_set_sum, void* ws, size_t ws_bytes,
                       cudaStream_t stream);
// The dense path's range: MM needs every count exact in f32 (universe < 2^24);
// BITMAP_NAIVE builds one set's bitmap in shared memory (<= 200 KiB).
inline bool dense_supported(uint32_t universe, si_technique t) {
    if (t == SI_TECH_MM) return universe < (1u << 24);
    return (static_cast<uint64_t>(universe) + 32) / 32 * 4 <= 200 * 1024;
}
size_t dense_workspace_size(uint32_t k, uint32_t universe, si_technique t);
si_status misi_dense(const uint32_t* d_elements, const uint64_t* d_offsets, uint32_t k, uint32_t universe,
                     si_technique t, int fp8, uint32_t* d_counts, void* ws, size_t ws_bytes, cudaStream_t stream);

// ---- sortedness check (si_api.cu) ----
si_status validate_sorted(const uint32_t* d_x, uint64_t n, uint32_t* d_flag, cudaStream_t stream);

}  // namespace si
