// The slot-map step's dispatch (the kernel: lbm_map.cuh).
#include "octlb_internal.h"

namespace octlb_gpu {

template <typename T, int N>
cudaError_t launch_map_n(const StepArgs&, const NearTables&, bool, bool, int, cudaStream_t);

// Slot-map step: n = 8 or 16 (the (n+2)^3 map of a block), 32-bit population
// offsets.
bool map_step_eligible(int n, long long nslots) { return (n == 8 || n == 16) && nslots * kQ < (1LL << 32); }

// CTAs of a BGK step's launch.
int map_step_ctas(const StepArgs& a, const NearTables& nt, bool links) {
  return (links ? (nt.n + 3) / 4 : 0) + a.nblk * (a.n * a.n * a.n / 256) + (a.n_open + 127) / 128;
}

// One step of a level; cm: its collide.
template <typename T>
cudaError_t launch_step_map(const StepArgs& a, const NearTables& nt, bool links, bool flags, int cm, cudaStream_t s) {
  if (a.nitems == 0) return cudaSuccess;
  const cudaError_t e =
      a.n == 8 ? launch_map_n<T, 8>(a, nt, links, flags, cm, s) : launch_map_n<T, 16>(a, nt, links, flags, cm, s);
  return e != cudaSuccess ? e : cudaGetLastError();
}
template cudaError_t launch_step_map<float>(const StepArgs&, const NearTables&, bool, bool, int, cudaStream_t);
template cudaError_t launch_step_map<__half>(const StepArgs&, const NearTables&, bool, bool, int, cudaStream_t);

}  // namespace octlb_gpu
