// nlgb_persist_df.cu -- instances of the persistent PCG kernel (one
// translation unit per precision, so that they compile in parallel).
#include "nlgb_persist.cuh"

namespace nlgb {
const void* persist_kernel_df(int tpr, bool cluster, int nc) {
  return cluster ? kernel_of<kPersistDf, true>(tpr, nc) : kernel_of<kPersistDf, false>(tpr, nc);
}
}  // namespace nlgb
