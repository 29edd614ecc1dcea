// nlgb_persist_mx.cu -- instances of the persistent PCG kernel (one
// translation unit per precision, so that they compile in parallel).
#include "nlgb_persist.cuh"

namespace nlgb {
const void* persist_kernel_mx(int tpr, bool cluster, int nc) {
  return cluster ? kernel_of<kPersistMixed, true>(tpr, nc) : kernel_of<kPersistMixed, false>(tpr, nc);
}
}  // namespace nlgb
