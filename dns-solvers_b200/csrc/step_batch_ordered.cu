// FP32 / FP16 instantiations of the batch kernel whose sums go by items
// (step_batch_ordered.cuh).
#include "step_batch_ordered.cuh"

namespace dnslbm {

int ordered_batch_occupancy(int precision, int threads, size_t smem, size_t cap)
{
    return precision == 32 ? ordered::persist_occupancy<float>(threads, smem, cap)
                           : ordered::persist_occupancy<__half>(threads, smem, cap);
}

cudaError_t launch_ordered_batch(int precision, const ordered::PersistArgs &a, int grid, int threads, size_t smem,
                                 cudaStream_t s)
{
    return precision == 32 ? ordered::launch_persist<float>(a, grid, threads, smem, s)
                           : ordered::launch_persist<__half>(a, grid, threads, smem, s);
}

}  // namespace dnslbm
