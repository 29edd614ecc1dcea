// nlgb_persist_f64.cu -- instances of the persistent PCG kernel (one
// translation unit per precision, so that they compile in parallel).
#include "nlgb_persist.cuh"

namespace nlgb {
const void* persist_kernel_f64(int tpr, bool cluster, int nc) {
  return cluster ? kernel_of<kPersistDouble, true>(tpr, nc) : kernel_of<kPersistDouble, false>(tpr, nc);
}
}  // namespace nlgb
