// Brute-force SIFT matcher for B200 (sm_100a): tcgen05 int8 UMMA with TMEM accumulators,
// TMA-staged descriptor tiles and a fused bidirectional top-1 / top-2 epilogue. No distance
// matrix is written to memory.
//
// Semantics follow RapidSFM's brute-force matcher (paths relative to its source tree):
//   distance d(i,j) = |a_i|^2 + |b_j|^2 - 2 a_i.b_j         bruteForceMatchIMMA.cu:209-258 (finishAcc)
//   per A row: lexicographic min of (d, j); per B column: lexicographic min of (d, i)
//                                                         bruteForceMatch.cuh:110-187, 191-261
//   results initialised to {~0u, ~0u}                      bruteForceMatch.cuh:166-169, 293-305
//   squared norms                                          bruteForceMatchIMMA.cu:704-731
// Extension (no reference counterpart): per A row the second-smallest distance, used by the
// ratio test; flags for the ratio test and the cross-check.
//
// Every value that the epilogue compares leaves the tensor cores finished: an accumulator holds
//   tile       (lane = A row i, column = B column j)   2 a_i.b_j - (|b_j|^2 - cB)
//   transpose  (lane = B column j, column = A row i)   2 a_i.b_j - (|a_i|^2 - cA)
// (cA, cB: norms of the unit's first row and column), i.e. the distance up to a constant of the
// lane. The factor 2 comes from A tiles doubled in shared memory (bytes <= 127; a unit with a larger
// byte keeps its bytes and issues every product twice), the norms from one more K = 32 step: a
// constant operand [1, 127 x 15][1, 127 x 15] times per-descriptor s8 digits. A norm that the
// digits do not reach, and rows or columns past the end, leave a residual that the epilogue adds
// (slices that have one are flagged).
//
// The epilogue keeps, per lane, only maxima of 16-column chunks: one key (value << 8 | chunk
// code) per chunk, the best (and for the second-best output the two best) in registers. Results
// are published as (distance, first index of the chunk), the minimum over chunks being the
// lexicographic (distance, chunk) minimum; bf_resolve_kernel then finds the index inside the winning
// chunk, and the second-best inside it, from 16 exact distances.
//
// What bounds it: the tensor pipe. At 32768 x 32768 the two products take 2 x 5 K steps of 128
// cycles per 128 x 256 values = 145 us on 148 SMs; a call with norms at hand takes 230 us there (at 16384
// the tensor pipe is busy for 60 % of the matcher's cycles). Keys formed on the CUDA cores instead (two
// multiply-adds and a trigger per distance, the design before this one) took 362 us at 53 % issue.
// Where every unit holds a byte above 127, 9 K steps instead of 5, 260 us: 302 us at 32768 x 32768.
//
// Work decomposition. A "unit" is a block of 256 A rows times up to 16 blocks of 256 B columns.
// Persistent CTAs take units round-robin. Per CTA (768 threads):
//   warp 0      UMMA issuer (one thread; warp 1 owns the TMEM allocation, 2 and 3 are idle): per B
//               block the tiles of both 128-row halves and the transposes of both 128-column
//               halves, each M = 128, N = 256, into two pairs of accumulators (128 TMEM columns
//               each) in turn
//   warps 4-7   TMA loads (A rows of a unit into two slots: the next unit's load and are prepared
//               during this one; B blocks into three stages), doubling of the A rows, digits,
//               residuals, norms, unit description
//   warps 8-23  epilogue: warpgroup g reads accumulator g, warp q of it TMEM lanes 32q..
#include "bf_internal.h"
#include "common.h"
#include "sm100.cuh"
#include <algorithm>
#include <climits>
#include <vector>

namespace rsfm_b200 {
namespace bf {

using namespace sm100;

constexpr uint32_t kUnitRows = 256;      // A rows per unit (two 128-lane tiles)
constexpr uint32_t kBlockCols = 256;     // B columns per block (two 128-lane transposes)
constexpr uint32_t kChunk = 16;          // values per key
constexpr int kBStages = 3;
constexpr int kASlots = 2;
constexpr uint32_t kPrepThreads = 128;
constexpr uint32_t kEpiWarps = 16;
constexpr uint32_t kThreads = 32 * (4 + kEpiWarps) + kPrepThreads;
constexpr uint32_t kTileBytes = 256 * 128;
constexpr uint32_t kDigitBytes = 256 * 32;
constexpr int32_t kNoValue = -(1 << 23);  // below every 2ab - |x|^2 (> -128 * 255^2)

struct alignas(64) TaskDev {
    CUtensorMap tmA;
    CUtensorMap tmB;
    const uint4* descA;
    const uint4* descB;
    const uint32_t* sqrA;
    const uint32_t* sqrB;
    unsigned long long* bestA;  // rsfm_best_match viewed as (distance << 32 | index)
    unsigned long long* bestB;
    uint32_t* secondA;  // null: no second-best output
    uint32_t* flagsA;   // null: no flags
    uint32_t nA, nB;
    uint32_t rowBlocks;
    uint32_t unitBegin;   // first unit, first group of 4 results to resolve, first group of 32 rows:
    uint32_t groupBegin;  // each in the order of the tasks
    uint32_t rowGroupBegin;
};

// Launch parameters, with room for kTasks tasks: one (also for plans, whose tasks are in global memory)
// or kMaxTasksPerLaunch. A launch copies its parameters: 7 KB for sixteen tasks cost a call of one
// pair about 2 us of host time a launch.
struct ParamsBase {
    const TaskDev* gtasks;  // when non-null: any number of tasks, in global memory
    uint32_t nTasks;
    uint32_t totalUnits;
    uint32_t totalGroups, totalRowGroups;  // totalRowGroups: 0 without flags
    uint32_t ratioNum, ratioDen;
    uint32_t unitBlocks;  // 256-column blocks per unit (<= 32: the chunk code holds 8 * 32 values)
    uint32_t* err;
};
template <int kTasks>
struct Params : ParamsBase {
    TaskDev tasks[kTasks];
};

struct Unit {
    uint32_t r0, c0, rows, cols;
};

template <int N>
__device__ __forceinline__ const TaskDev& task_of(const Params<N>& P, uint32_t t) {
    return P.gtasks ? P.gtasks[t] : P.tasks[t];
}

// Unit u of task t, where t enters as the task of an earlier unit of this CTA (units are taken in
// increasing order, so the search only moves forward).
template <int N>
__device__ __forceinline__ Unit decode_unit(const Params<N>& P, uint32_t u, uint32_t& t) {
    while (t + 1 < P.nTasks && task_of(P, t + 1).unitBegin <= u) ++t;
    const TaskDev& T = task_of(P, t);
    const uint32_t local = u - T.unitBegin;
    const uint32_t cr = local / T.rowBlocks;
    Unit U;
    U.r0 = (local - cr * T.rowBlocks) * kUnitRows;
    U.c0 = cr * kBlockCols * P.unitBlocks;
    U.rows = min(T.nA - U.r0, kUnitRows);
    U.cols = min(T.nB - U.c0, kBlockCols * P.unitBlocks);
    return U;
}

// What the issuer and the epilogue need to know about the unit in an A slot.
struct UnitInfo {
    unsigned long long* bestA;
    unsigned long long* bestB;
    uint32_t* secondA;
    uint32_t r0, c0, rows, cols;
    uint32_t cA, cB;  // norms of the first row and column
    uint32_t big;     // some A byte exceeds 127: not doubled, products issued twice
};

struct Smem {
    // A rows and B blocks: 128-byte rows, 128-byte swizzle (1024-byte atoms)
    uint8_t a[kASlots][kTileBytes];
    uint8_t b[kBStages][kTileBytes];
    // norm digits: 32-byte rows, 32-byte swizzle (256-byte atoms)
    uint8_t digA[kASlots][kDigitBytes];
    uint8_t digB[kBStages][kDigitBytes];
    uint8_t ones[128 * 32];
    int32_t resA[kASlots][256];
    int32_t resB[kBStages][256];
    uint32_t nrmA[kASlots][256];
    uint32_t nrmB[kBStages][256];
    uint32_t flagA[kASlots][4];  // per 64-row slice: nonzero when some residual is
    uint32_t flagB[kBStages][4];
    UnitInfo info[kASlots];
    uint32_t bigWarp[4];
    uint64_t aRaw[kASlots], aReady[kASlots], aEpi[kASlots];
    uint64_t bReady[kBStages], bEpi[kBStages];
    uint64_t accFull[2], accEmpty[2];  // per pair of accumulators
    uint64_t mmaDone;
    uint32_t tmemBase;
};

// Programmatic dependent launch: the kernels of a call start while the one before them still runs (its
// blocks all started), and wait here for its results. Small calls are launch after launch: 600 x 600
// without norms 21.3 us as one cooperative launch behind the initialisation, 19.4 as three ordinary
// launches, 13.6 this way. A no-op in an ordinary launch.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void named_bar(uint32_t id, uint32_t n) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// s8 digits of w for the constant operand (row r of a 32-byte swizzled tile): d0 + 127 Q, Q spread
// over 30 digits; |w| <= 127 * 3810 + 63 is exact. Returns what is left.
__device__ __forceinline__ int32_t store_digits(uint8_t* tile, uint32_t r, int32_t w) {
    constexpr int32_t kQmax = 30 * 127;
    int32_t Q = __float2int_rn(float(w) * (1.f / 127.f));
    int32_t d0 = w - 127 * Q, left = 0;
    uint32_t dg[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (uint32_t(Q + 127) <= 254u) {  // one digit holds Q: norms within 16 K of each other
        dg[0] = (uint32_t(Q) & 255u) << 8;
    } else {
        Q = max(-kQmax, min(kQmax, Q));
        d0 = max(-127, min(127, w - 127 * Q));
        left = w - d0 - 127 * Q;
#pragma unroll
        for (int k = 1; k < 32; ++k) {
            if (k == 16) continue;  // the other weight-1 slot stays 0
            const int32_t v = max(-127, min(127, Q));
            dg[k >> 2] |= (uint32_t(v) & 255u) << (8 * (k & 3));
            Q -= v;
        }
    }
    dg[0] |= uint32_t(d0) & 255u;
    const uint32_t swap = ((r >> 2) & 1u) << 4;
    uint8_t* row = tile + 32u * r;
    *reinterpret_cast<uint4*>(row + swap) = make_uint4(dg[0], dg[1], dg[2], dg[3]);
    *reinterpret_cast<uint4*>(row + (16u ^ swap)) = make_uint4(dg[4], dg[5], dg[6], dg[7]);
    return left;
}

// Maxima of the two 16-value chunks of x, as four chains (a chain of eight 3-input maxima is
// latency-bound).
__device__ __forceinline__ void chunk_max(const uint32_t (&x)[32], int32_t& m0, int32_t& m1) {
    int32_t m[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) m[c] = __vimax3_s32(int32_t(x[8 * c]), int32_t(x[8 * c + 1]), int32_t(x[8 * c + 2]));
#pragma unroll
    for (int k = 3; k < 7; k += 2)
#pragma unroll
        for (int c = 0; c < 4; ++c) m[c] = __vimax3_s32(m[c], int32_t(x[8 * c + k]), int32_t(x[8 * c + k + 1]));
    m0 = __vimax3_s32(max(m[0], int32_t(x[7])), m[1], int32_t(x[15]));
    m1 = __vimax3_s32(max(m[2], int32_t(x[23])), m[3], int32_t(x[31]));
}

__device__ __forceinline__ void add_residuals(uint32_t (&x)[32], const int32_t* res) {
    const int4* r4 = reinterpret_cast<const int4*>(res);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int4 r = r4[k];
        x[4 * k] += uint32_t(r.x);
        x[4 * k + 1] += uint32_t(r.y);
        x[4 * k + 2] += uint32_t(r.z);
        x[4 * k + 3] += uint32_t(r.w);
    }
}

// ---------------------------------------------------------------- index inside the winning chunk
// The matcher leaves (distance, first index of a 16-descriptor chunk) per row and per column; eight
// lanes per result compute the chunk's 16 exact distances (each lane 16 bytes of every descriptor:
// one cache line per descriptor) and keep the first index at that distance. A row's other distances
// complete its second-best. Bound by L2 reads, 2 KiB per result: 134 MB for
// 32768 x 32768; chunks of 32 values would save the matcher 4 of 48 operations per 64 values and
// double these reads.

// Exact distances of q to the 16 descriptors of `set` from j0 on: lane l8 of the eight ends up with
// candidates 2 * l8 and 2 * l8 + 1 (~0u past the end, or without `has`).
__device__ __forceinline__ void chunk_distances(const uint4* __restrict__ q, uint32_t normQ,
                                                const uint4* __restrict__ set, const uint32_t* __restrict__ sqrSet,
                                                uint32_t nSet, uint32_t j0, bool has, uint32_t l8,
                                                uint32_t (&dist)[2]) {
    uint32_t dot[kChunk];
    uint4 qv = make_uint4(0, 0, 0, 0), tv[kChunk];
    if (has) qv = __ldg(&q[l8]);
#pragma unroll
    for (uint32_t k = 0; k < kChunk; ++k) {
        tv[k] = make_uint4(0, 0, 0, 0);
        if (has && j0 + k < nSet) tv[k] = __ldg(&set[size_t(j0 + k) * 8 + l8]);
    }
    uint32_t nv[2] = {0, 0};
#pragma unroll
    for (uint32_t e = 0; e < 2; ++e)
        if (has && j0 + 2 * l8 + e < nSet) nv[e] = __ldg(&sqrSet[j0 + 2 * l8 + e]);
#pragma unroll
    for (uint32_t k = 0; k < kChunk; ++k) {
        uint32_t a = __dp4a(qv.x, tv[k].x, 0u);
        a = __dp4a(qv.y, tv[k].y, a);
        a = __dp4a(qv.z, tv[k].z, a);
        dot[k] = __dp4a(qv.w, tv[k].w, a);
    }
#pragma unroll
    for (uint32_t w = 8; w >= 2; w >>= 1) {  // halve the candidates, add the partner's half
        const uint32_t o = w >> 1;           // lane distance 4, 2, 1
        const bool hi = (l8 & o) != 0u;
#pragma unroll
        for (uint32_t k = 0; k < w; ++k) {
            const uint32_t mine = hi ? dot[k + w] : dot[k], theirs = hi ? dot[k] : dot[k + w];
            dot[k] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
        }
    }
#pragma unroll
    for (uint32_t e = 0; e < 2; ++e) dist[e] = has && j0 + 2 * l8 + e < nSet ? normQ + nv[e] - 2u * dot[e] : ~0u;
}

// Last task whose `begin` is at or before w (tasks without any share their successor's).
template <int N>
__device__ __forceinline__ uint32_t task_at(const Params<N>& P, uint32_t TaskDev::*begin, uint32_t w) {
    uint32_t t = 0, hi = P.nTasks - 1u;
    while (t < hi) {
        const uint32_t mid = (t + hi + 1u) >> 1;
        if (task_of(P, mid).*begin <= w) t = mid; else hi = mid - 1u;
    }
    return t;
}

// Every warp takes a run of consecutive groups of four results (columns of B, then rows of A), eight
// lanes a result.
//
// kFlags: it sets the rows' flags too. A row's cross-check bit needs the final index of its match's column, which another warp may not have
// written yet. It is decided from either state: the column's distance must be the row's; then its
// index is the row itself (also as a chunk's first index: no earlier row of that chunk), or another
// row, or the first index of the row's own chunk - and in that last case the row is the column's match
// exactly if no earlier row of the chunk is as close. The alternatives: a launch of its own for the
// flags, which is better where there are many results (small_results); a grid-wide barrier (one
// cooperative launch for matching, resolution and flags), which needs all its blocks resident at once:
// a green context or a long kernel on another stream does not give that (and 600 x 600, one call alone
// with all outputs, took 74 us, against 68 as three launches).
template <int N, bool kFlags>
__global__ void __launch_bounds__(256) bf_resolve_kernel(const __grid_constant__ Params<N> P) {
    const uint32_t lane = threadIdx.x & 31u, l8 = lane & 7u;
    const uint32_t warps = gridDim.x * 8u;
    const uint32_t run = (P.totalGroups + warps - 1u) / warps;
    const uint32_t first = (blockIdx.x * 8u + (threadIdx.x >> 5)) * run;
    if (first >= P.totalGroups) return;
    const uint32_t end = min(P.totalGroups, first + run);
    uint32_t t = task_at(P, &TaskDev::groupBegin, first);
    grid_dep_wait();
    for (uint32_t w = first; w < end; ++w) {
        while (t + 1 < P.nTasks && task_of(P, t + 1).groupBegin <= w) ++t;
        const TaskDev& T = task_of(P, t);
        const uint64_t x = uint64_t(w - T.groupBegin) * 4u + (lane >> 3);
        const bool col = x < T.nB, row = !col && x < uint64_t(T.nA) + T.nB;
        const uint32_t i = col ? uint32_t(x) : row ? uint32_t(x - T.nB) : 0u;
        unsigned long long* best = (col ? T.bestB : T.bestA) + i;
        const unsigned long long bst = col || row ? __ldcg(best) : ~0ull;
        const uint32_t j0 = uint32_t(bst), d = uint32_t(bst >> 32);
        const bool has = j0 != ~0u;
        uint32_t dist[2];
        chunk_distances((col ? T.descB : T.descA) + size_t(i) * 8, has ? __ldg((col ? T.sqrB : T.sqrA) + i) : 0u,
                        col ? T.descA : T.descB, col ? T.sqrA : T.sqrB, col ? T.nA : T.nB, j0, has, l8, dist);
        uint32_t at = ~0u, s = ~0u;
#pragma unroll
        for (int e = 1; e >= 0; --e)
            if (has && dist[e] == d && dist[e] != ~0u) at = j0 + 2 * l8 + e;
#pragma unroll
        for (uint32_t o = 1; o < 8; o <<= 1) at = min(at, __shfl_xor_sync(0xffffffffu, at, o));
        if (has && l8 == 0 && at != ~0u) __stcg(best, (static_cast<unsigned long long>(d) << 32) | at);
        if (!__any_sync(0xffffffffu, row && T.secondA)) continue;
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (j0 + 2 * l8 + e != at) s = min(s, dist[e]);
#pragma unroll
        for (uint32_t o = 1; o < 8; o <<= 1) s = min(s, __shfl_xor_sync(0xffffffffu, s, o));
        if (row && l8 == 0) {
            const uint32_t old = __ldcg(&T.secondA[i]);
            if (s < old) T.secondA[i] = s;
            s = min(s, old);
        }
        if (!kFlags) continue;
        const uint32_t j = at != ~0u ? at : j0, c0 = i & ~(kChunk - 1u);
        unsigned long long cb = row && j < T.nB ? __ldcg(&T.bestB[j]) : ~0ull;
        cb = __shfl_sync(0xffffffffu, cb, int(lane & 24u));  // one state of it for the eight lanes
        const bool near = row && has && uint32_t(cb >> 32) == d;
        bool mutual = near && uint32_t(cb) == i;
        const bool open = near && !mutual && uint32_t(cb) == c0;
        if (__any_sync(0xffffffffu, open)) {
            chunk_distances(T.descB + size_t(open ? j : 0u) * 8, open ? __ldg(&T.sqrB[j]) : 0u, T.descA, T.sqrA, T.nA, c0,
                            open, l8, dist);
            const bool closer = (c0 + 2 * l8 < i && dist[0] == d) || (c0 + 2 * l8 + 1 < i && dist[1] == d);
            const uint32_t any = __ballot_sync(0xffffffffu, open && closer);
            if (open) mutual = ((any >> (lane & 24u)) & 0xFFu) == 0u;
        }
        if (row && l8 == 0) {
            uint32_t f = mutual ? 2u : 0u;
            if (has && uint64_t(P.ratioDen) * d < uint64_t(P.ratioNum) * s) f |= 1u;
            T.flagsA[i] = f;
        }
    }
}

// The flags as a launch of their own: bit0 ratio test, bit1 cross-check. Every warp takes a run of
// 32-row groups.
template <int N>
__global__ void __launch_bounds__(256) bf_flags_kernel(const __grid_constant__ Params<N> P) {
    const uint32_t lane = threadIdx.x & 31u, warps = gridDim.x * 8u;
    const uint32_t run = (P.totalRowGroups + warps - 1u) / warps;
    const uint32_t first = (blockIdx.x * 8u + (threadIdx.x >> 5)) * run;
    if (first >= P.totalRowGroups) return;
    const uint32_t end = min(P.totalRowGroups, first + run);
    uint32_t t = task_at(P, &TaskDev::rowGroupBegin, first);
    for (uint32_t w = first; w < end; ++w) {
        while (t + 1 < P.nTasks && task_of(P, t + 1).rowGroupBegin <= w) ++t;
        const TaskDev& T = task_of(P, t);
        const uint32_t i = (w - T.rowGroupBegin) * 32u + lane;
        if (i >= T.nA) continue;
        const unsigned long long bm = __ldcg(&T.bestA[i]);
        const uint32_t j = uint32_t(bm & 0xFFFFFFFFu), d = uint32_t(bm >> 32);
        uint32_t f = 0;
        if (j != ~0u) {
            if (uint64_t(P.ratioDen) * d < uint64_t(P.ratioNum) * __ldcg(&T.secondA[i])) f |= 1u;
            if (j < T.nB && uint32_t(__ldcg(&T.bestB[j]) & 0xFFFFFFFFu) == i) f |= 2u;
        }
        T.flagsA[i] = f;
    }
}

// kSecond: the second-best distances are wanted too.
template <bool kSecond, int N>
__global__ void __launch_bounds__(kThreads, 1) bf_match_kernel(const __grid_constant__ Params<N> P) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem& S = smem_aligned_1024<Smem>(smem_raw);
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    grid_dep_launch();

    if (threadIdx.x == 0) {
        for (int s = 0; s < kASlots; ++s) {
            S.info[s].rows = S.info[s].cols = 0;  // a timed-out wait must find nothing to write
            mbar_init(&S.aRaw[s], 1);
            mbar_init(&S.aReady[s], kPrepThreads);
            mbar_init(&S.aEpi[s], kEpiWarps);
        }
        for (int s = 0; s < kBStages; ++s) {
            mbar_init(&S.bReady[s], kPrepThreads);  // (and the bytes of the TMA load)
            mbar_init(&S.bEpi[s], kEpiWarps);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(&S.accFull[s], 1);
            mbar_init(&S.accEmpty[s], kEpiWarps / 2);
        }
        mbar_init(&S.mmaDone, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(&S.tmemBase, 512);
        tmem_relinquish();
    }
    if (threadIdx.x >= 128 && threadIdx.x < 384) {  // 128 x 32 bytes; both 16-byte chunks alike
        reinterpret_cast<uint4*>(S.ones)[threadIdx.x - 128] =
            make_uint4(0x7F7F7F01u, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmemBase;
    uint32_t* err = P.err;

    // Registers: every one of the 768 threads has 80. Handing some of the issuer's and the preparation's
    // to the epilogue (setmaxnreg, 88 or 96 there) ended in spills or moves: 251 to 287 us at
    // 32768 x 32768 against 224.
    if (warp < 4) {
        // ------------------------------------------------------------ UMMA issuer
        // One thread, so that products complete in order (with two or four issuers their UMMAs take
        // turns, all accumulators fill at the same time and the epilogue runs in bursts: 294 and
        // 335 us at 32768 x 32768); N = 256, because N = 128 reads 128 bytes of shared memory a
        // cycle, all there is.
        if (warp == 0 && elect_one()) {
            const uint32_t idesc = idesc_u8u8_s32(128, 256), idescN = idesc | (1u << 7) | (1u << 10);  // s8 digits
            constexpr uint32_t kHalf = 128u * 128u >> 4;  // descriptor step of 128 rows
            const uint64_t ones = umma_desc_k_sw32(smem_u32(S.ones));
            uint32_t stage = 0, bPhase = 0, use0 = 1, use1 = 1, k = 0;
            for (uint32_t u = blockIdx.x; u < P.totalUnits; u += gridDim.x, ++k) {
                const uint32_t slot = k & 1u;
                mbar_wait(&S.aReady[slot], (k >> 1) & 1u, err, kDevTimeoutTmaFull);
                const uint32_t cols = S.info[slot].cols, big = S.info[slot].big;
                const bool two = S.info[slot].rows > 128u;
                const uint64_t aDesc = umma_desc_k_sw128(smem_u32(S.a[slot]));
                const uint64_t aDig = umma_desc_k_sw32(smem_u32(S.digA[slot]));
                // a pair of accumulators: lanes x columns (4 K steps of 32 bytes = +2 in the
                // start-address field), then the norms
                auto product = [&](uint32_t pair, uint32_t& use, uint64_t lanes, uint64_t columns, uint64_t digits) {
                    mbar_wait(&S.accEmpty[pair], use, err, kDevTimeoutAccEmpty);
                    use ^= 1u;
                    tc_fence_after();
                    const uint32_t d = tmem + pair * 256u;
#pragma unroll
                    for (uint32_t s = 0; s < 4; ++s) umma_i8(d, lanes + 2u * s, columns + 2u * s, idesc, s);
                    if (big) {
#pragma unroll
                        for (uint32_t s = 0; s < 4; ++s) umma_i8(d, lanes + 2u * s, columns + 2u * s, idesc, 1u);
                    }
                    umma_i8(d, ones, digits, idescN, 1u);
                    umma_commit(&S.accFull[pair]);
                };
                for (uint32_t c = 0; c < cols; c += kBlockCols) {
                    mbar_wait(&S.bReady[stage], bPhase, err, kDevTimeoutTmaFull);
                    tc_fence_after();
                    const uint64_t bDesc = umma_desc_k_sw128(smem_u32(S.b[stage]));
                    const uint64_t bDig = umma_desc_k_sw32(smem_u32(S.digB[stage]));
                    product(0, use0, aDesc, bDesc, bDig);
                    if (two) product(1, use1, aDesc + kHalf, bDesc, bDig);
                    product(0, use0, bDesc, aDesc, aDig);
                    if (cols - c > 128u) product(1, use1, bDesc + kHalf, aDesc, aDig);
                    if (++stage == uint32_t(kBStages)) { stage = 0; bPhase ^= 1u; }
                }
            }
            // Drain: every product issued above is complete once this has arrived.
            umma_commit(&S.mmaDone);
            mbar_wait(&S.mmaDone, 0, err, kDevTimeoutOther);
        }
    } else if (warp < 8) {
        // ------------------------------------------------------------ loads and preparation
        const uint32_t pt = threadIdx.x - 128u, pw = warp - 4u;
        const uint32_t row0 = 64u * pw + lane;  // this thread's rows: row0, row0 + 32 (slice pw)
        uint32_t stage = 0, bPhase = 0, k = 0, t = 0;
        // 256 norms -> digits, residuals, norms, flags
        auto digits = [&](const uint32_t (&nv)[2], uint32_t valid, uint32_t centre, uint8_t* tile, int32_t* res,
                          uint32_t* nrm, uint32_t* flag) {
            int32_t any = 0;
#pragma unroll
            for (uint32_t m = 0; m < 2; ++m) {
                const uint32_t r = row0 + 32u * m;
                const bool in = r < valid;
                int32_t left = store_digits(tile, r, in ? int32_t(centre - nv[m]) : 0);
                if (!in) left = int32_t(centre) + kNoValue;  // the descriptor reads as zero
                res[r] = left;
                nrm[r] = nv[m];
                any |= left;
            }
            const uint32_t f = __any_sync(0xffffffffu, any != 0);
            if (lane == 0) flag[pw] = f;
        };
        // norms [first, first + valid) of the slice, 0 past the end
        auto norms = [&](uint32_t (&nv)[2], const uint32_t* sqr, uint32_t first, uint32_t valid) {
#pragma unroll
            for (uint32_t m = 0; m < 2; ++m) nv[m] = row0 + 32u * m < valid ? __ldg(&sqr[first + row0 + 32u * m]) : 0u;
        };
        // One thread issues the TMA loads; the stage or slot is free when the epilogue is done with
        // its last use (which implies the products that read it are complete).
        auto loadB = [&](const CUtensorMap* tm, uint32_t c, uint32_t st) {
            mbar_expect_tx(&S.bReady[st], kTileBytes);
            tma_load_2d(S.b[st], tm, &S.bReady[st], 0, int32_t(c));
        };
        auto loadA = [&](uint32_t u, uint32_t kk) {
            uint32_t tn = t;
            const Unit U = decode_unit(P, u, tn);
            mbar_wait(&S.aEpi[kk & 1u], ((kk >> 1) & 1u) ^ 1u, err, kDevTimeoutTmaEmpty);
            mbar_arrive_expect_tx(&S.aRaw[kk & 1u], kTileBytes);
            tma_load_2d(S.a[kk & 1u], &task_of(P, tn).tmA, &S.aRaw[kk & 1u], 0, int32_t(U.r0));
        };
        auto prepA = [&](uint32_t u, uint32_t kk) {
            const Unit U = decode_unit(P, u, t);
            const TaskDev& T = task_of(P, t);
            const uint32_t slot = kk & 1u, ph = (kk >> 1) & 1u;
            uint32_t nv[2];
            norms(nv, T.sqrA, U.r0, U.rows);
            const uint32_t cA = __ldg(&T.sqrA[U.r0]), cB = __ldg(&T.sqrB[U.c0]);
            mbar_wait(&S.aEpi[slot], ph ^ 1u, err, kDevTimeoutTmaEmpty);
            digits(nv, U.rows, cA, S.digA[slot], S.resA[slot], S.nrmA[slot], S.flagA[slot]);
            mbar_wait(&S.aRaw[slot], ph, err, kDevTimeoutTmaFull);
            uint4* a4 = reinterpret_cast<uint4*>(S.a[slot]);
            uint32_t any = 0;
#pragma unroll 4
            for (uint32_t x = pt; x < kTileBytes / 16; x += kPrepThreads) {
                const uint4 v = a4[x];
                any |= v.x | v.y | v.z | v.w;
            }
            any = __any_sync(0xffffffffu, (any & 0x80808080u) != 0u);
            if (lane == 0) S.bigWarp[pw] = any;
            named_bar(2, kPrepThreads);
            const uint32_t big = S.bigWarp[0] | S.bigWarp[1] | S.bigWarp[2] | S.bigWarp[3];
            if (!big) {
#pragma unroll 4
                for (uint32_t x = pt; x < kTileBytes / 16; x += kPrepThreads) {
                    uint4 v = a4[x];
                    v.x <<= 1;  // bytes <= 127: no carry into the next byte
                    v.y <<= 1;
                    v.z <<= 1;
                    v.w <<= 1;
                    a4[x] = v;
                }
            }
            if (pt == 0) {
                UnitInfo& I = S.info[slot];
                I.bestA = T.bestA;
                I.bestB = T.bestB;
                I.secondA = T.secondA;
                I.r0 = U.r0;
                I.c0 = U.c0;
                I.rows = U.rows;
                I.cols = U.cols;
                I.cA = cA;
                I.cB = cB;
                I.big = big;
            }
            fence_proxy_async_smem();
            mbar_arrive(&S.aReady[slot]);
            named_bar(2, kPrepThreads);  // bigWarp may be rewritten
        };
        uint32_t u = blockIdx.x;
        uint32_t ahead = 0;  // blocks of the current unit whose loads are already under way
        if (u < P.totalUnits) {
            const Unit U = decode_unit(P, u, t);
            ahead = min((U.cols + kBlockCols - 1) / kBlockCols, uint32_t(kBStages));
            if (pt == 0) {
                loadA(u, 0);
                for (uint32_t b = 0; b < ahead; ++b) loadB(&task_of(P, t).tmB, U.c0 + kBlockCols * b, b);
            }
            prepA(u, 0);
        }
        for (; u < P.totalUnits; u += gridDim.x, ++k, ahead = 0) {
            uint32_t tb = t;
            const Unit U = decode_unit(P, u, tb);
            const uint32_t* sqrB = task_of(P, tb).sqrB;
            const CUtensorMap* tmB = &task_of(P, tb).tmB;
            const uint32_t cB = __ldg(&sqrB[U.c0]);
            const uint32_t nb = (U.cols + kBlockCols - 1) / kBlockCols;
            const bool more = u + gridDim.x < P.totalUnits;
            uint32_t nv[2], next[2];
            norms(nv, sqrB, U.c0, U.cols);
            for (uint32_t b = 0; b < nb; ++b) {
                const uint32_t done = kBlockCols * (b + 1);
                norms(next, sqrB, U.c0 + done, done < U.cols ? U.cols - done : 0u);
                mbar_wait(&S.bEpi[stage], bPhase ^ 1u, err, kDevTimeoutTmaEmpty);
                if (pt == 0 && b >= ahead) loadB(tmB, U.c0 + done - kBlockCols, stage);
                digits(nv, U.cols - (done - kBlockCols), cB, S.digB[stage], S.resB[stage], S.nrmB[stage], S.flagB[stage]);
                nv[0] = next[0];
                nv[1] = next[1];
                fence_proxy_async_smem();
                mbar_arrive(&S.bReady[stage]);
                if (++stage == uint32_t(kBStages)) { stage = 0; bPhase ^= 1u; }
                // The next unit's rows: their slot is free from this unit's block 3 on (block 0 is done
                // then, so the unit before is), and they have a block's time to arrive.
                if (more && b == min(nb - 1, 3u) && pt == 0) loadA(u + gridDim.x, k + 1);
                if (more && b == min(nb - 1, 4u)) prepA(u + gridDim.x, k + 1);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        // Warpgroup g owns accumulator g: per block the tile (row half g / 2, column half g % 2) and
        // the transpose (column half g / 2, row half g % 2).
        const uint32_t g = (warp - 8u) >> 2, q = warp & 3u;  // q: TMEM lane quarter
        const uint32_t outer = 128u * (g >> 1), inner = 128u * (g & 1u);
        const uint32_t mine = outer + 32u * q + lane;  // this thread's row (tile) or column (transpose)
        const uint32_t taddr = tmem + ((32u * q) << 16) + 128u * g;
        uint32_t accPhase = 0, stage = 0, bPhase = 0, k = 0;
        grid_dep_wait();  // the results are initialised (nothing above reads or writes them)
        // The accumulator's eight 16-value chunks as keys (value << 8) + base - chunk, handed to
        // `take` in pairs.
        auto chunks = [&](const int32_t* res, uint32_t base, auto&& take) {
            mbar_wait(&S.accFull[g >> 1], accPhase, err, kDevTimeoutAccFull);
            accPhase ^= 1u;
            tc_fence_after();
#pragma unroll 4
            for (uint32_t part = 0; part < 4; ++part) {
                uint32_t x[32];
                tmem_ld16(taddr + 32u * part, *reinterpret_cast<uint32_t(*)[16]>(&x[0]));
                tmem_ld16(taddr + 32u * part + 16u, *reinterpret_cast<uint32_t(*)[16]>(&x[16]));
                tmem_wait_ld();
                if (part == 3) {  // the accumulator is read: hand it back
                    tc_fence_before();
                    if (lane == 0) mbar_arrive(&S.accEmpty[g >> 1]);
                }
                if (res) add_residuals(x, res + 32u * part);
                int32_t m0, m1;
                chunk_max(x, m0, m1);
                take(int32_t((uint32_t(m0) << 8) + (base - 2u * part)), int32_t((uint32_t(m1) << 8) + (base - 2u * part - 1u)));
            }
        };
        for (uint32_t u = blockIdx.x; u < P.totalUnits; u += gridDim.x, ++k) {
            const uint32_t slot = k & 1u;
            mbar_wait(&S.aReady[slot], (k >> 1) & 1u, err, kDevTimeoutAccFull);
            const UnitInfo& I = S.info[slot];
            // (read from shared memory where it is used: registers are short here)
            // residuals of the rows (transposes), if the row half has any
            const bool resA = (S.flagA[slot][inner >> 6] | S.flagA[slot][(inner >> 6) + 1]) != 0u;
            // keys: (value - centre) << 8 | code, the code falling with the chunk's position
            uint32_t baseR = 255u - (I.cB << 8);
            const uint32_t baseC = 255u - (I.cA << 8);
            int32_t l1 = INT_MIN, l2 = INT_MIN;  // the row's best chunk and (kSecond) the next
            uint32_t thrA = ~0u;  // row distances from here on change nothing
            for (uint32_t c = 0; c < I.cols; c += kBlockCols, baseR -= 8u) {
                mbar_wait(&S.bReady[stage], bPhase, err, kDevTimeoutAccFull);
                // A column's value below thr cannot change its result, which only falls (a tie can:
                // the lower index wins). Loaded here, used after the tile.
                int32_t thr = INT_MAX;
                if (mine < I.cols - c) {
                    const uint32_t d = __ldcg(reinterpret_cast<const uint32_t*>(&I.bestB[I.c0 + c + mine]) + 1);
                    thr = max(int32_t(S.nrmB[stage][mine] - min(d, 1u << 24)), kNoValue + 1);
                }
                if (I.cols - c <= kBlockCols && mine < I.rows) {  // last block: the row's results by now
                    thrA = __ldcg(reinterpret_cast<const uint32_t*>(&I.bestA[I.r0 + mine]) + 1);
                    thrA = min(thrA, ~1u) + 1u;
                    if (kSecond) thrA = max(thrA, __ldcg(&I.secondA[I.r0 + mine]));
                }
                if (outer < I.rows) {
                    const bool any = (S.flagB[stage][inner >> 6] | S.flagB[stage][(inner >> 6) + 1]) != 0u;
                    chunks(any ? &S.resB[stage][inner] : nullptr, baseR, [&](int32_t k0, int32_t k1) {
                        if (kSecond) {
                            const int32_t hi = max(k0, k1);
                            l2 = __vimax3_s32(l2, min(k0, k1), min(l1, hi));
                            l1 = max(l1, hi);
                        } else {
                            l1 = __vimax3_s32(l1, k0, k1);
                        }
                    });
                }
                if (outer < I.cols - c) {
                    int32_t best = INT_MIN;
                    chunks(resA ? &S.resA[slot][inner] : nullptr, baseC, [&](int32_t k0, int32_t k1) {
                        best = __vimax3_s32(best, k0, k1);
                    });
                    if ((best >> 8) >= thr) {
                        const uint32_t d = S.nrmB[stage][mine] - uint32_t(best >> 8);
                        const uint32_t i = I.r0 + inner + kChunk * (255u - (uint32_t(best) & 255u));
                        red_min_u64(&I.bestB[I.c0 + c + mine], (static_cast<unsigned long long>(d) << 32) | i);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.bEpi[stage]);
                if (++stage == uint32_t(kBStages)) { stage = 0; bPhase ^= 1u; }
            }
            // ---- the unit's rows: best chunk of this column half, merged by atomics with the others
            if (mine < I.rows && (l1 >> 8) != kNoValue) {
                const uint32_t na = S.nrmA[slot][mine];
                const uint32_t d1 = na - uint32_t(l1 >> 8);
                const uint32_t idx = 255u - (uint32_t(l1) & 255u);
                const unsigned long long key = (static_cast<unsigned long long>(d1) << 32) |
                                               (I.c0 + kBlockCols * (idx >> 3) + inner + kChunk * (idx & 7u));
                if (d1 < thrA) {
                    if (kSecond) {
                        const unsigned long long old = atomicMin(&I.bestA[I.r0 + mine], key);
                        uint32_t s = max(uint32_t(old >> 32), d1);
                        if ((l2 >> 8) != kNoValue) s = min(s, na - uint32_t(l2 >> 8));
                        red_min_u32(&I.secondA[I.r0 + mine], s);
                    } else {
                        red_min_u64(&I.bestA[I.r0 + mine], key);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.aEpi[slot]);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// Initialise results: bestA/bestB = {~0u, ~0u}, secondA = ~0u.
__global__ void bf_init_kernel(const __grid_constant__ InitParams P) {
    const uint32_t t = blockIdx.y;
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    grid_dep_launch();
    if (x < P.nA[t]) {
        P.bestA[t][x] = ~0ull;
        if (P.secondA[t]) P.secondA[t][x] = ~0u;
    }
    if (x < P.nB[t]) P.bestB[t][x] = ~0ull;
}

// ---------------------------------------------------------------- squared norms
// One warp per 4 descriptors: 8 lanes x 16 bytes per descriptor (coalesced 128-bit loads).
__global__ void sqr_norm_kernel(uint32_t* __restrict__ out, const uint4* __restrict__ desc, uint32_t n) {
    const uint64_t gid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t i = gid >> 3;
    const uint32_t part = uint32_t(gid) & 7u;
    uint32_t acc = 0;
    if (i < n) {
        const uint4 v = __ldg(&desc[size_t(i) * 8 + part]);
        acc = __dp4a(v.x, v.x, acc);
        acc = __dp4a(v.y, v.y, acc);
        acc = __dp4a(v.z, v.z, acc);
        acc = __dp4a(v.w, v.w, acc);
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    if (i < n && part == 0) out[i] = acc;
}

// 256-column blocks per unit. A CTA spends about 1.4 us of tensor time on a block (four products)
// and about 0.9 us more on a unit when the next unit's rows are not ready in time (units of fewer
// than four blocks) or 0.15 us when they are; the launch lasts as long as the CTA with the most
// units. The shape with the shortest estimate is taken, the longer unit on a tie (fewer row publishes).
static uint32_t choose_unit_blocks(const std::vector<std::pair<uint32_t, uint32_t>>& sizes, int nsm) {
    uint32_t pick = 1;
    double best = 0;
    for (uint32_t ub : {16u, 8u, 4u, 2u, 1u}) {
        uint64_t units = 0, blocks = 0;
        for (auto& s : sizes) {
            const uint64_t rb = (s.first + kUnitRows - 1) / kUnitRows;
            const uint64_t nb = (s.second + kBlockCols - 1) / kBlockCols;
            units += rb * ((nb + ub - 1) / ub);
            blocks += rb * nb;
        }
        if (units == 0) return 1;
        const uint64_t waves = (units + uint64_t(nsm) - 1) / uint64_t(nsm);
        const double perUnit = 1.4 * double(blocks) / double(units) + (ub >= 4 ? 0.15 : 0.9);
        const double est = double(waves) * perUnit;
        if (best == 0 || est < 0.98 * best) {
            best = est;
            pick = ub;
        }
    }
    return pick;
}

template <bool kSecond, int N>
static int ensure_attr() {
    return set_max_dynamic_smem(reinterpret_cast<const void*>(bf_match_kernel<kSecond, N>), sizeof(Smem) + 1024);
}

// `early`: start while the kernel before on the stream still runs.
template <class P>
static int launch(void (*kernel)(P), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t stream, bool early,
                  const P& params) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    RSFM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, params));
    launch_count_add(1);
    return RSFM_OK;
}

// Up to four groups of results for each warp that fits on the device (4 blocks of 8 per SM), the
// resolution starts while the matcher still runs, and sets the flags. Beyond, an early start leaves it
// the matcher's small L1 and the flags' look-ups come while most columns are open; us with all outputs,
// this way against waiting and a launch for the flags: 32768 x 32768 (16 K groups) 247.4 and 251.2, plan
// of 16 pairs (26 K) 89.7 and 88.4, of 40 (100 K) 394 and 374, of 512 (2.3 M) 11860 and 11300.
static bool small_results(const ParamsBase& P, int nsm) { return P.totalGroups <= uint32_t(nsm) * 128u; }

// The matcher and what follows it. afterInit: the kernel before on the stream is this call's
// initialisation (which waits for all before it, so the matcher may read its inputs at once).
template <bool kSecond, int N>
static int launch_match(const Params<N>& P, int nsm, cudaStream_t stream, bool afterInit) {
    if (P.totalUnits > 0) {
        int st = ensure_attr<kSecond, N>();
        if (st == RSFM_OK)
            st = launch(bf_match_kernel<kSecond, N>, std::min<uint32_t>(P.totalUnits, uint32_t(nsm)), kThreads,
                        sizeof(Smem) + 1024, stream, afterInit, P);
        if (st != RSFM_OK) return st;
    }
    if (P.totalGroups == 0) return RSFM_OK;
    const uint32_t grid = std::min<uint32_t>((P.totalGroups + 7) / 8, uint32_t(nsm) * 64u);
    const bool small = small_results(P, nsm), flags = P.totalRowGroups > 0;
    if (small)
        return launch(flags ? bf_resolve_kernel<N, true> : bf_resolve_kernel<N, false>, grid, 256, 0, stream,
                      P.totalUnits > 0, P);
    const int st = launch(bf_resolve_kernel<N, false>, grid, 256, 0, stream, false, P);
    if (st != RSFM_OK || !flags) return st;
    return launch(bf_flags_kernel<N>, std::min<uint32_t>((P.totalRowGroups + 7) / 8, uint32_t(nsm) * 64u), 256, 0, stream,
                  false, P);
}

// Fills a task's device description and counts it into P's totals. Empty sides get no units, and of
// the results only rows with flags need a look.
static int fill_task(TaskDev* T, const rsfm_sift_bf_task& in, uint32_t* second, uint32_t* flags, ParamsBase* P) {
    T->nA = in.nbDescA;
    T->nB = in.nbDescB;
    T->descA = static_cast<const uint4*>(in.descA);
    T->descB = static_cast<const uint4*>(in.descB);
    T->sqrA = in.sqrNormDescA;
    T->sqrB = in.sqrNormDescB;
    T->bestA = reinterpret_cast<unsigned long long*>(in.bestMatchA);
    T->bestB = reinterpret_cast<unsigned long long*>(in.bestMatchB);
    T->secondA = second;
    T->flagsA = flags;
    T->unitBegin = P->totalUnits;
    T->groupBegin = P->totalGroups;
    T->rowBlocks = 1;
    T->rowGroupBegin = P->totalRowGroups;
    if (flags) P->totalRowGroups += (T->nA + 31) / 32;
    if (T->nA > 0 && (T->nB > 0 || flags)) P->totalGroups += uint32_t((uint64_t(T->nA) + T->nB + 3) / 4);
    if (T->nA == 0 || T->nB == 0) return RSFM_OK;
    int st = encode_desc_tmap(&T->tmA, in.descA, T->nA, kUnitRows);
    if (st == RSFM_OK) st = encode_desc_tmap(&T->tmB, in.descB, T->nB, kBlockCols);
    if (st != RSFM_OK) return st;
    T->rowBlocks = (T->nA + kUnitRows - 1) / kUnitRows;
    const uint32_t unitCols = kBlockCols * P->unitBlocks;
    P->totalUnits += T->rowBlocks * ((T->nB + unitCols - 1) / unitCols);
    return RSFM_OK;
}

template <int N>
static int launch_tasks(const rsfm_sift_bf_task* tasks, size_t n, uint32_t* const* second, uint32_t* const* flags,
                        uint32_t ratioNum, uint32_t ratioDen, cudaStream_t stream, bool initialised) {
    const int nsm = sm_count();
    if (nsm <= 0) return RSFM_ERR_CUDA;

    const InitParams ip = init_params(tasks, n, second);
    uint32_t maxN = 0;
    std::vector<std::pair<uint32_t, uint32_t>> sizes;
    for (size_t t = 0; t < n; ++t) {
        maxN = std::max(maxN, std::max(tasks[t].nbDescA, tasks[t].nbDescB));
        sizes.emplace_back(tasks[t].nbDescA, tasks[t].nbDescB);
    }
    if (maxN > 0 && !initialised) {
        dim3 g((maxN + 255) / 256, uint32_t(n));
        bf_init_kernel<<<g, 256, 0, stream>>>(ip);
        RSFM_CUDA_TRY(cudaGetLastError());
        launch_count_add(1);
    }

    Params<N> P;
    memset(static_cast<void*>(&P), 0, sizeof(P));
    P.unitBlocks = choose_unit_blocks(sizes, nsm);
    P.ratioNum = ratioNum;
    P.ratioDen = ratioDen;
    for (size_t t = 0; t < n; ++t) {
        const int st = fill_task(&P.tasks[t], tasks[t], ip.secondA[t], flags ? flags[t] : nullptr, &P);
        if (st != RSFM_OK) return st;
    }
    P.nTasks = uint32_t(n);
    P.err = device_error_word();
    if (!P.err) return RSFM_ERR_CUDA;
    if (P.totalUnits > 0 || P.totalGroups > 0) {
        // the bracket of rsfm_profile_* holds all that produces the results, initialisation apart
        void* tok = nullptr;
        const bool prof = profile_begin(stream, &tok);
        const int st = second ? launch_match<true, N>(P, nsm, stream, !initialised)
                              : launch_match<false, N>(P, nsm, stream, !initialised);
        if (st != RSFM_OK) return st;
        if (prof) profile_end(stream, tok);
    }
    return RSFM_OK;
}

int launch_chunk(const rsfm_sift_bf_task* tasks, size_t n, uint32_t* const* second, uint32_t* const* flags,
                 uint32_t ratioNum, uint32_t ratioDen, cudaStream_t stream, bool initialised) {
    return n == 1 ? launch_tasks<1>(tasks, n, second, flags, ratioNum, ratioDen, stream, initialised)
                  : launch_tasks<kMaxTasksPerLaunch>(tasks, n, second, flags, ratioNum, ratioDen, stream, initialised);
}

// ---------------------------------------------------------------- batched plans
// A plan holds the tasks of a whole batch (any count) in device memory, so the matcher runs as
// one persistent launch over all (task, row block, column range) units; init and match
// are captured once in a CUDA graph and replayed.
__global__ void plan_init_kernel(const TaskDev* __restrict__ tasks) {
    grid_dep_launch();
    const TaskDev& T = tasks[blockIdx.y];
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < max(T.nA, T.nB); x += gridDim.x * blockDim.x) {
        if (x < T.nA) {
            T.bestA[x] = ~0ull;
            T.secondA[x] = ~0u;
        }
        if (x < T.nB) T.bestB[x] = ~0ull;
    }
}
}  // namespace bf
}  // namespace rsfm_b200

struct rsfm_bf_plan {
    rsfm_b200::bf::TaskDev* dTasks = nullptr;
    rsfm_b200::bf::Params<1> P;
    uint32_t nTasks = 0;
    uint32_t blocksX = 1;
    int nsm = 0;
    cudaStream_t capture = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint32_t launches = 0;  // kernels in the graph
};

namespace rsfm_b200 {
namespace bf {

static int plan_enqueue(rsfm_bf_plan* pl, cudaStream_t s) {
    launch_count_add(1);
    plan_init_kernel<<<dim3(pl->blocksX, pl->nTasks), 256, 0, s>>>(pl->dTasks);
    RSFM_CUDA_TRY(cudaGetLastError());
    return launch_match<true, 1>(pl->P, pl->nsm, s, true);
}

int validate(const rsfm_sift_bf_task* tasks, size_t n) {
    if (n > 0 && !tasks) return RSFM_ERR_INVALID_ARG;
    for (size_t t = 0; t < n; ++t) {
        const rsfm_sift_bf_task& T = tasks[t];
        if (T.nbDescA > 0 && (!T.descA || !T.bestMatchA || !T.sqrNormDescA)) return RSFM_ERR_INVALID_ARG;
        if (T.nbDescB > 0 && (!T.descB || !T.bestMatchB || !T.sqrNormDescB)) return RSFM_ERR_INVALID_ARG;
        if ((reinterpret_cast<uintptr_t>(T.descA) & 15u) || (reinterpret_cast<uintptr_t>(T.descB) & 15u))
            return RSFM_ERR_INVALID_ARG;
        if ((reinterpret_cast<uintptr_t>(T.bestMatchA) & 7u) || (reinterpret_cast<uintptr_t>(T.bestMatchB) & 7u))
            return RSFM_ERR_INVALID_ARG;
        // Row offsets within a unit are kept in 32 bits and TMA rows are int32 coordinates.
        if (T.nbDescA > 0x7FFFFF00u || T.nbDescB > 0x7FFFFF00u) return RSFM_ERR_CAPACITY;
    }
    return RSFM_OK;
}

}  // namespace bf
}  // namespace rsfm_b200

using namespace rsfm_b200;

extern "C" int rsfm_precomp_sift_sqr_norm(uint32_t* sqrNorm, const void* desc, uint32_t nbDesc, cudaStream_t stream) {
    launch_count_reset();
    if (nbDesc == 0) return RSFM_OK;
    if (!sqrNorm || !desc || (reinterpret_cast<uintptr_t>(desc) & 15u)) return RSFM_ERR_INVALID_ARG;
    const uint64_t threads = uint64_t(nbDesc) * 8;
    const uint32_t grid = uint32_t((threads + 255) / 256);
    bf::sqr_norm_kernel<<<grid, 256, 0, stream>>>(sqrNorm, static_cast<const uint4*>(desc), nbDesc);
    RSFM_CUDA_TRY(cudaGetLastError());
    launch_count_add(1);
    return RSFM_OK;
}

extern "C" int rsfm_bf_match_ext(const rsfm_sift_bf_task* tasks, size_t nbTasks, uint32_t* const* secondDistA,
                                 uint32_t* const* flagsA, uint32_t ratioNum, uint32_t ratioDen, cudaStream_t stream) {
    launch_count_reset();
    int st = bf::validate(tasks, nbTasks);
    if (st != RSFM_OK) return st;
    if (nbTasks > 0 && (!secondDistA || !flagsA)) return RSFM_ERR_INVALID_ARG;
    for (size_t t = 0; t < nbTasks; ++t)
        if (tasks[t].nbDescA > 0 && (!secondDistA[t] || !flagsA[t])) return RSFM_ERR_INVALID_ARG;
    for (size_t i = 0; i < nbTasks; i += bf::kMaxTasksPerLaunch) {
        const size_t n = std::min<size_t>(bf::kMaxTasksPerLaunch, nbTasks - i);
        st = bf::launch_chunk(tasks + i, n, secondDistA + i, flagsA + i, ratioNum, ratioDen, stream);
        if (st != RSFM_OK) return st;
    }
    return RSFM_OK;
}

extern "C" int rsfm_bf_match(const rsfm_sift_bf_task* tasks, size_t nbTasks, cudaStream_t stream) {
    launch_count_reset();
    int st = bf::validate(tasks, nbTasks);
    if (st != RSFM_OK) return st;
    if (nbTasks == 0) return RSFM_OK;
    for (size_t i = 0; i < nbTasks; i += bf::kMaxTasksPerLaunch) {
        const size_t n = std::min<size_t>(bf::kMaxTasksPerLaunch, nbTasks - i);
        st = bf::launch_chunk(tasks + i, n, nullptr, nullptr, 0, 1, stream);
        if (st != RSFM_OK) return st;
    }
    return RSFM_OK;
}

extern "C" int rsfm_bf_plan_create(const rsfm_sift_bf_task* tasks, size_t nbTasks, uint32_t* const* secondDistA,
                                   uint32_t* const* flagsA, uint32_t ratioNum, uint32_t ratioDen,
                                   const rsfm_bf_plan_options* opts, rsfm_bf_plan** out) {
    launch_count_reset();
    if (!out || nbTasks == 0 || nbTasks > 65535 || !secondDistA || !flagsA) return RSFM_ERR_INVALID_ARG;
    int st = bf::validate(tasks, nbTasks);
    if (st != RSFM_OK) return st;
    for (size_t t = 0; t < nbTasks; ++t)
        if (tasks[t].nbDescA > 0 && (!secondDistA[t] || !flagsA[t])) return RSFM_ERR_INVALID_ARG;
    const int nsm = sm_count();
    if (nsm <= 0) return RSFM_ERR_CUDA;
    auto* pl = new rsfm_bf_plan();
    memset(static_cast<void*>(&pl->P), 0, sizeof(pl->P));
    std::vector<std::pair<uint32_t, uint32_t>> sizes;
    uint32_t maxN = 1;
    for (size_t t = 0; t < nbTasks; ++t) {
        sizes.emplace_back(tasks[t].nbDescA, tasks[t].nbDescB);
        maxN = std::max(maxN, std::max(tasks[t].nbDescA, tasks[t].nbDescB));
    }
    // The options give a unit as rowTiles x colBlocks tiles of 128 x 128; units here are 256 rows
    // high, so the same area is taken as 256-column blocks.
    uint32_t ub = bf::choose_unit_blocks(sizes, nsm);
    if (opts && (opts->rowTiles || opts->colBlocks)) {
        const uint32_t rt = opts->rowTiles ? std::min<uint32_t>(opts->rowTiles, 8) : 8;
        const uint32_t cb = opts->colBlocks ? std::min<uint32_t>(opts->colBlocks, 8) : 8;
        ub = std::max<uint32_t>(1, rt * cb / 4);
    }
    // Unit order: pairs in the given order, or largest pairs first (their units are spread over
    // every CTA before the small pairs fill the tail).
    std::vector<size_t> order(nbTasks);
    for (size_t t = 0; t < nbTasks; ++t) order[t] = t;
    if (opts && opts->schedule == 1)
        std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) {
            return uint64_t(tasks[x].nbDescA) * tasks[x].nbDescB > uint64_t(tasks[y].nbDescA) * tasks[y].nbDescB;
        });
    std::vector<bf::TaskDev> host(nbTasks);
    pl->P.unitBlocks = ub;
    for (size_t o = 0; o < nbTasks; ++o) {
        const size_t t = order[o];
        bf::TaskDev& T = host[o];
        memset(&T, 0, sizeof(T));
        if ((st = bf::fill_task(&T, tasks[t], secondDistA[t], flagsA[t], &pl->P)) != RSFM_OK) {
            delete pl;
            return st;
        }
    }
    if (cudaMalloc(reinterpret_cast<void**>(&pl->dTasks), sizeof(bf::TaskDev) * nbTasks) != cudaSuccess ||
        cudaMemcpy(pl->dTasks, host.data(), sizeof(bf::TaskDev) * nbTasks, cudaMemcpyHostToDevice) != cudaSuccess) {
        rsfm_bf_plan_destroy(pl);
        return RSFM_ERR_CUDA;
    }
    pl->nTasks = uint32_t(nbTasks);
    pl->P.gtasks = pl->dTasks;
    pl->P.nTasks = uint32_t(nbTasks);
    pl->P.ratioNum = ratioNum;
    pl->P.ratioDen = ratioDen;
    pl->P.err = device_error_word();
    pl->nsm = nsm;
    pl->blocksX = std::min<uint32_t>((maxN + 255) / 256, 64);
    const bool useGraph = !opts || opts->useGraph;
    if (useGraph) {
        // Set kernel attributes outside the capture, then record the launches once.
        st = bf::ensure_attr<true, 1>();
        if (st != RSFM_OK) {
            rsfm_bf_plan_destroy(pl);
            return st;
        }
        if (cudaStreamCreateWithFlags(&pl->capture, cudaStreamNonBlocking) != cudaSuccess ||
            cudaStreamBeginCapture(pl->capture, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            rsfm_bf_plan_destroy(pl);
            return RSFM_ERR_CUDA;
        }
        launch_count_reset();
        st = bf::plan_enqueue(pl, pl->capture);
        pl->launches = rsfm_last_launch_count();
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(pl->capture, &g);
        pl->graph = g;
        if (st != RSFM_OK || e != cudaSuccess ||
            cudaGraphInstantiate(&pl->exec, pl->graph, 0) != cudaSuccess) {
            rsfm_bf_plan_destroy(pl);
            return st != RSFM_OK ? st : RSFM_ERR_CUDA;
        }
    }
    *out = pl;
    return RSFM_OK;
}

extern "C" int rsfm_bf_plan_launch(rsfm_bf_plan* plan, cudaStream_t stream) {
    launch_count_reset();
    if (!plan) return RSFM_ERR_INVALID_ARG;
    // (bracketed here and not in plan_enqueue: an event recorded while capturing cannot be read)
    void* tok = nullptr;
    const bool prof = profile_begin(stream, &tok);
    if (plan->exec) {
        RSFM_CUDA_TRY(cudaGraphLaunch(plan->exec, stream));
        launch_count_add(plan->launches);
    } else {
        const int st = bf::plan_enqueue(plan, stream);
        if (st != RSFM_OK) return st;
    }
    if (prof) profile_end(stream, tok);
    return RSFM_OK;
}

extern "C" int rsfm_bf_plan_destroy(rsfm_bf_plan* plan) {
    if (!plan) return RSFM_OK;
    if (plan->exec) cudaGraphExecDestroy(plan->exec);
    if (plan->graph) cudaGraphDestroy(plan->graph);
    if (plan->capture) cudaStreamDestroy(plan->capture);
    if (plan->dTasks) cudaFree(plan->dTasks);
    delete plan;
    return RSFM_OK;
}
