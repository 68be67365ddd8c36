// Parts of the level step shared by the step kernels (lbm_kernels.cu,
// lbm_map.cuh): solid-cell copies, halo items of open blocks, near-wall cells.
#ifndef OCTLB_LBM_STEP_CUH_
#define OCTLB_LBM_STEP_CUH_

#include "lbm_device.cuh"

namespace octlb_gpu {
namespace {

// The 19 populations of cell t copied unchanged; all loads are issued
// before the first store (for all the compiler knows, a store to row i may
// alias the load from row i + 1, which would cost a round trip each).
template <typename T>
__device__ __forceinline__ void copy_cell(const T* src, T* dst, long long qs, uint32_t t) {
  T v[kQ];
#pragma unroll
  for (int i = 0; i < kQ; ++i) v[i] = src[i * qs + t];
#pragma unroll
  for (int i = 0; i < kQ; ++i) dst[i * qs + t] = v[i];
}

// Torus-streamed halo population of an open block (block_lattice.h:70-89),
// item k: copied without collision.
template <typename T>
__device__ __forceinline__ void rotate_item(const StepArgs& a, uint32_t k) {
  if (k >= static_cast<uint32_t>(a.n_open)) return;
  long long d, sl;
  int i;
  const bool fill = rotate_slots(a, k, d, sl, i);
  pdl_wait();
  const T* src = static_cast<const T*>(a.src);
  T* dst = static_cast<T*>(a.dst);
  if (fill) Store<T>::st(dst + i * a.qs + d, pull_value(a, src, i, sl), a.scale);
  else dst[i * a.qs + d] = src[i * a.qs + sl];
}

// Cells flagged kFlagNear (links stream rule): the per-cell link rule of
// block_lattice.cpp:613-672 with every table lookup done on the host --
// direction i reads population i at nt.slot[i] and, where the rule applies,
// reflects own[opp(i)] (half-way bounce-back, reflect-on-pull at the block
// edge) or interpolates with Bouzidi (bouzidi_pull.h:8-26), then adds the
// moving-wall term.  Then the same save / collide / store as k_step.  One
// warp per cell, lane i on direction i; the collision gathers the 19 values
// so every lane computes the moments exactly as bgk() does.
template <typename T, int CM = kCollBgk>
__device__ __forceinline__ float near_cell(const StepArgs& a, const NearTables& nt, int k, int lane, float dr = 0.f) {
  if (k >= nt.n) return 0.f;
  const T* src = static_cast<const T*>(a.src);
  T* dst = static_cast<T*>(a.dst);
  const LaneDir d = lane_dir(lane);
  const uint32_t t = static_cast<uint32_t>(nt.cells[k]);
  const uint32_t mask = nt.mask[k];
  const uint8_t fl = a.flags[t];
  const int sl = d.act ? nt.slot[k * kQ + lane] : 0;
  const float q = d.act ? nt.q[k * kQ + lane] : 1.f, add = d.act ? nt.add[k * kQ + lane] : 0.f;
  pdl_wait();
  const float val = d.act ? pull_value(a, src, lane, sl) : 0.f;
  const float own = d.act ? LD(src, a.qs, lane, t, a.inv_scale) : 0.f;
  const float own_opp = __shfl_sync(0xffffffffu, own, d.opp);
  float f = val;
  if (d.act && ((mask >> lane) & 1u)) f = (q < 1.0f ? bouzidi(own_opp, val, own, q) : own_opp) + add;
  if ((fl & kFlagSave) && d.act) a.save_buf[static_cast<long long>(a.save_idx[t]) * kQ + lane] = f;
  float dh = 0.f;
  if constexpr (CM != kCollNone) {
    if ((fl & kKindMask) == kBulk) {
      float fa[kQ];
      gather_lanes(f, fa);
      if constexpr (CM == kCollConstRho) {
        f = bgk_lane_const_rho(d, lane, fa, f, a.omega, dr, dh);
        if (fl & kFlagProlong) dh = 0.f;
      } else {
        f = bgk_lane<false>(d, lane, fa, f, a.omega);
      }
    }
  }
  if (d.act) Store<T>::st(dst + lane * a.qs + t, f, a.scale);
  return dh;
}

}  // namespace
}  // namespace octlb_gpu

#endif  // OCTLB_LBM_STEP_CUH_
