// Brute-force matcher internals shared by the translation units that launch it
// (bf_match.cu, bf_match_noalloc.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>
#include "../../include/rsfm_b200.h"

namespace rsfm_b200 {
namespace bf {

// Tasks per matcher launch: the launch parameters hold this many tasks by value, as the
// reference's launcher does (bruteForceMatchIMMA.cu:626-633, std::array<Task, 16>).
constexpr int kMaxTasksPerLaunch = 16;

// Argument checks of every brute-force entry point: null pointers, 16-byte descriptor and 8-byte
// result alignment, and the per-task size limit (RSFM_ERR_CAPACITY above 0x7FFFFF00 rows).
int validate(const rsfm_sift_bf_task* tasks, size_t n);

// Results of up to kMaxTasksPerLaunch tasks, as the kernel that initialises them gets them.
struct InitParams {
    unsigned long long* bestA[kMaxTasksPerLaunch];
    unsigned long long* bestB[kMaxTasksPerLaunch];
    uint32_t* secondA[kMaxTasksPerLaunch];  // null entries: no second-best output
    uint32_t nA[kMaxTasksPerLaunch], nB[kMaxTasksPerLaunch];
};
inline InitParams init_params(const rsfm_sift_bf_task* tasks, size_t n, uint32_t* const* second) {
    InitParams ip{};
    for (size_t t = 0; t < n; ++t) {
        ip.bestA[t] = reinterpret_cast<unsigned long long*>(tasks[t].bestMatchA);
        ip.bestB[t] = reinterpret_cast<unsigned long long*>(tasks[t].bestMatchB);
        ip.secondA[t] = second ? second[t] : nullptr;
        ip.nA[t] = tasks[t].nbDescA;
        ip.nB[t] = tasks[t].nbDescB;
    }
    return ip;
}

// Init + matcher + index resolution (+ flags when `flags` is non-null, which needs `second`) for
// n <= kMaxTasksPerLaunch tasks on `stream`; second[t] is task t's per-row second-best output
// (nbDescA entries), `second` may be null. initialised: the results already hold ~0 on `stream`.
int launch_chunk(const rsfm_sift_bf_task* tasks, size_t n, uint32_t* const* second, uint32_t* const* flags,
                 uint32_t ratioNum, uint32_t ratioDen, cudaStream_t stream, bool initialised = false);

}  // namespace bf
}  // namespace rsfm_b200
