// kernels_flatten.h — launch interface of the flattening kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/lyon_gpu.h"

namespace lg {

struct FlattenArgs {
    const uint8_t* verbs;
    const float* points;
    const uint32_t* verb_offsets;
    const uint32_t* point_offsets;
    uint32_t num_paths;
    float tolerance;
    uint32_t* counts;          // one per verb (count pass)
    uint32_t* firsts;          // one per verb: its first point (count pass; null: not wanted), or
                               // FLATTEN_NO_POINTS
    const uint64_t* offsets;   // exclusive scan of counts (point pass)
    float* out_points;         // point pass output
};

constexpr uint32_t FLATTEN_NO_POINTS = 0;  // (a path's first point is its Begin's)

cudaError_t launch_flatten_counts(const FlattenArgs& a, int num_sms, cudaStream_t s);
// Points of the verbs [0, num_verbs) that the count pass gave a first point.
cudaError_t launch_flatten_points(const FlattenArgs& a, uint32_t num_verbs, int num_sms,
                                  cudaStream_t s);

}  // namespace lg
