// The slot-map step of 8^3 blocks, FP32 storage.
#include "lbm_map.cuh"

namespace octlb_gpu {
template cudaError_t launch_map_n<float, 8>(const StepArgs&, const NearTables&, bool, bool, int, cudaStream_t);
}  // namespace octlb_gpu
