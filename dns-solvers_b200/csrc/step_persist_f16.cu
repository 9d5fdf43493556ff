// The persistent time-loop kernel (step_persist.cuh) of one channel, FP16 storage.
#include "step_persist.cuh"

namespace dnslbm {
DNSLBM_PERSIST_UNIT(__half, true, f16)
}  // namespace dnslbm
