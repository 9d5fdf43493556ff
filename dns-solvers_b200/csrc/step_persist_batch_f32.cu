// The persistent time-loop kernel (step_persist.cuh) of a batch, FP32 storage.
#include "step_persist.cuh"

namespace dnslbm {
DNSLBM_PERSIST_UNIT(float, false, batch_f32)
}  // namespace dnslbm
