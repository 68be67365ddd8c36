// The slot-map step of 16^3 blocks, FP16-shifted storage.
#include "lbm_map.cuh"

namespace octlb_gpu {
template cudaError_t launch_map_n<__half, 16>(const StepArgs&, const NearTables&, bool, bool, int, cudaStream_t);
}  // namespace octlb_gpu
