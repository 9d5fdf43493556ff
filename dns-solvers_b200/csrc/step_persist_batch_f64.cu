// The persistent time-loop kernel (step_persist.cuh) of a batch, FP64 (compiled with -fmad=false: the collision keeps the reference's rounding).
#include "step_persist.cuh"

namespace dnslbm {
DNSLBM_PERSIST_UNIT(double, false, batch_f64)
}  // namespace dnslbm
