// Host-side interface of the few-row linear projections.
#pragma once
#include "common.cuh"

namespace tops {
namespace skinny {
int linear(const tops_skinny_linear_params& p, cudaStream_t st);
}  // namespace skinny
}  // namespace tops
