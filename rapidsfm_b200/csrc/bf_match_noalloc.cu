// Allocation-free variant of rsfm_bf_match (no reference counterpart): a call allocates no device
// memory, for callers that must not allocate (a scheduler thread that runs under a fixed memory
// budget, or code that may not touch the allocator while other work is in flight). A call whose
// tasks hold more than kNoAllocMaxRows = 1 Mi query rows in total returns RSFM_ERR_CAPACITY before
// enqueuing anything.
#include "bf_internal.h"
#include "common.h"

namespace rsfm_b200 {
namespace noalloc {
constexpr size_t kNoAllocMaxRows = size_t(1) << 20;
}  // namespace noalloc
}  // namespace rsfm_b200

using namespace rsfm_b200;

extern "C" int rsfm_bf_match_noalloc(const rsfm_sift_bf_task* tasks, size_t nbTasks, cudaStream_t stream) {
    launch_count_reset();
    // The same argument checks as rsfm_bf_match, then the limit on the total query rows, which callers may
    // rely on (rsfm_bf_match itself allocates nothing and has no such limit).
    int st = bf::validate(tasks, nbTasks);
    if (st != RSFM_OK) return st;
    size_t total = 0;
    for (size_t t = 0; t < nbTasks; ++t) total += tasks[t].nbDescA;
    if (total > noalloc::kNoAllocMaxRows) return RSFM_ERR_CAPACITY;
    return rsfm_bf_match(tasks, nbTasks, stream);
}
