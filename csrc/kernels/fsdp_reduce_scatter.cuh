// The reduce-scatter behind nangila_predres_launch (mode 2).
#pragma once
#include <cuda_runtime.h>

#include "nangila_kernels.h"

namespace nangila {
cudaError_t launch_reduce_scatter(const NangilaPredResParams& p, cudaStream_t stream);
}  // namespace nangila
