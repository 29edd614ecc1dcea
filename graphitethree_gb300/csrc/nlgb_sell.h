// nlgb_sell.h -- row-sorted sliced layout of a matrix for the phase kernels
// (nlgb_sell.cu).
#pragma once
#include <cuda_runtime.h>

#include "nlgb_core.cuh"
#include "nlgb_internal.h"

namespace nlgb {

// The kernel that replaces k_spmv_pq for this view, or null.
const void* sell_pq_kernel(const SysView& v);
// y = A x with a layout of A (sell_prepare).
cudaError_t sell_spmv64(const DeviceCRS& A, const SellView& m, const double* x, double* y, cudaStream_t s);

}  // namespace nlgb
