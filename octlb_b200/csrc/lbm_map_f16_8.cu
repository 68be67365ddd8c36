// The slot-map step of 8^3 blocks, FP16-shifted storage.
#include "lbm_map.cuh"

namespace octlb_gpu {
template cudaError_t launch_map_n<__half, 8>(const StepArgs&, const NearTables&, bool, bool, int, cudaStream_t);
}  // namespace octlb_gpu
