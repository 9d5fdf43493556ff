// The persistent time-loop kernel (step_persist.cuh) of one channel, FP64 (compiled with -fmad=false: the collision keeps the reference's rounding).
#include "step_persist.cuh"

namespace dnslbm {
DNSLBM_PERSIST_UNIT(double, true, f64)
}  // namespace dnslbm
