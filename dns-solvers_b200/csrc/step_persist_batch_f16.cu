// The persistent time-loop kernel (step_persist.cuh) of a batch, FP16 storage.
#include "step_persist.cuh"

namespace dnslbm {
DNSLBM_PERSIST_UNIT(__half, false, batch_f16)
}  // namespace dnslbm
