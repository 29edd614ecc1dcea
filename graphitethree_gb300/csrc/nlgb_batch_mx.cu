// nlgb_batch_mx.cu -- the batched kernel with mixed systems (a translation unit
// of its own: see nlgb_batch.cuh).
#include "nlgb_batch.cuh"

namespace nlgb {
const void* batch_kernel_mixed() { return (const void*)k_batch<true>; }
}  // namespace nlgb
