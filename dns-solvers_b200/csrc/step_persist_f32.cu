// The persistent time-loop kernel (step_persist.cuh) of one channel, FP32 storage.
#include "step_persist.cuh"

namespace dnslbm {
DNSLBM_PERSIST_UNIT(float, true, f32)
}  // namespace dnslbm
