// Shared-memory layout of the finalize's warp shape (rerank.cu), in plain host
// arithmetic.
#pragma once

#ifdef __CUDACC__
#define SSG_HD __host__ __device__
#else
#define SSG_HD
#endif

namespace ssg {

constexpr int kDimStep = 32;               // dimensions staged per step
constexpr int kRowStride = kDimStep + 4;   // floats: 16-byte rows, float4 reads of 8 lanes on distinct banks
constexpr int kWarpKeys = 8;               // keys per lane in the warp shape (256 in all)
constexpr int kWarpStages = 3;

// A warp's shared memory, in 8-byte keys: the ring of need + 1 staged rows and,
// before it is used, the keys gathered from the query's lists.  Up to
// 32 * kWarpKeys gathered keys are taken into registers as they stand, so that
// many always fit (the rings of 1, 2 and 3 rows are 108, 162 and 216 keys).
// Even: every warp's memory is 16-byte aligned.
SSG_HD constexpr int warp_room(int need) {
    const int ring = kWarpStages * (need + 1) * kRowStride / 2;
    return ring > 32 * kWarpKeys ? ring : 32 * kWarpKeys;
}

}  // namespace ssg
