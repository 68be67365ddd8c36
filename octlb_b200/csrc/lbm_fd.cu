// Finite-difference domain boundary conditions on the device: the post-stream
// reconstruction of velocity- and pressure-Dirichlet cells (Skordos
// InterpolatedVelocity, ApplyInterpolatedVelocityBoundaryCells,
// interpolated_velocity.h:951-1037: plane :571-636, edge :687-752, corner
// :638-685, the BoundaryLatticeView reads :213-445) and their Dirichlet
// collide (BcDispatcher::collide's velocity arm, bc_dispatcher.h:55-72 with
// BoundaryCellStatisticRho, interpolated_velocity.h:815-884).
//
// After a level step the state buffer holds, for a boundary cell, its
// post-stream populations f (the step leaves non-kBulk cells uncollided) and,
// for a fluid cell, its post-collision populations, whose velocity is the
// post-stream one (the collide keeps rho u).  The reference rewrites the
// boundary cells in place in (ix, iy, iz) order; a cell's stencil reads the
// densities of boundary cells one and two cells inward, rewritten or not by
// that order.  Edge cells read plane cells and corners read edge cells, so the
// pass runs as three launches -- planes, edges, corners -- each writing the
// rewritten populations to its own rows and reading an earlier phase's row
// where the reference's walk would have rewritten the cell already (one warp
// per cell, lane = population, every read of the stencil loaded at once).  A fourth
// launch collides the rewritten cells (velocity cells at the prescribed
// velocity, the next step's time; pressure cells are not collided) into the
// state buffer.  Every read a cell makes is resolved on the host into a table
// (FdCell): which slot or row, the velocity source (fluid populations, the
// prescribed velocity of a boundary cell, the overlap padding at rest, or a
// mirror image with flipped normal components), the density source.
// Arithmetic FP32; storage FP32 or FP16-shifted.
//
// The launches are small and each waits for the one before, so they are
// programmatic: every kernel lets its dependents start at once, and reads its
// records (constant tables, two dependent reads) before it waits for its
// predecessor, so what remains of a launch on the critical path is one read of
// the state, the arithmetic and one write.  cavity3d's 31^3 step: 43.8 us in
// plain stream order with a launch for the average and a store per step, 32.2 us now.
#include "lbm_device.cuh"

namespace octlb_gpu {

namespace {

constexpr int kFdThreads = 128;

// PolynomialStartScale: 10 x^3 - 15 x^4 + 6 x^5, x = t / t_end clamped to [0, 1].
__device__ __forceinline__ float ramp(float t, float t_end) {
  if (t_end <= 0.f) return 1.f;
  const float x = fminf(fmaxf(t / t_end, 0.f), 1.f);
  return x * x * x * (10.f + x * (-15.f + 6.f * x));
}

// The prescribed velocity b.xyz ramped over b.w steps.
__device__ __forceinline__ void prescribed(const float4& b, float t, float u[3]) {
  const float r = ramp(t, b.w);
  u[0] = r * b.x;
  u[1] = r * b.y;
  u[2] = r * b.z;
}

template <typename T>
__device__ __forceinline__ void load_pops(const T* state, long long qs, long long slot, float inv_s, float f[kQ]) {
#pragma unroll
  for (int i = 0; i < kQ; ++i) f[i] = Store<T>::ld(state + i * qs + slot, inv_s);
}

__device__ __forceinline__ float sum_pops(const float f[kQ]) {
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < kQ; ++i) s += f[i];
  return s;
}

// velocityBMRho: (2 sum_{c_d = o} f + sum_{c_d = 0} f + 1) / (1 + o u_d).
__device__ __forceinline__ float bm_rho(const float f[kQ], int d, int o, const float u[3]) {
  float out = 0.f, wall = 0.f;
#pragma unroll
  for (int i = 0; i < kQ; ++i) {
    const int c = d == 0 ? cx(i) : (d == 1 ? cy(i) : cz(i));
    if (c == 0) wall += f[i];
    else if (c == o) out += f[i];
  }
  return (2.f * out + wall + 1.f) / (1.f + o * u[d]);
}

// Shifted second-order equilibrium, rho w (1 + 3 cu + 4.5 cu^2 - 1.5 u^2) - w.
__device__ __forceinline__ float feq_i(int i, float rho, const float u[3], float usq) {
  const float cu = cx(i) * u[0] + cy(i) * u[1] + cz(i) * u[2];
  return rho * wf(i) * (1.f + 3.f * cu + 4.5f * cu * cu - 1.5f * usq) - wf(i);
}

// Gradient along `axis` by the one-sided second-order stencil
// -n (-3 u0 + 4 u1 - u2) / 2 (u1, u2 one and two cells inward).
__device__ __forceinline__ void normal_grad(const float u0[3], const float u1[3], const float u2[3], int n,
                                            float g[3]) {
#pragma unroll
  for (int b = 0; b < 3; ++b) g[b] = -n * (-3.f * u0[b] + 4.f * u1[b] - u2[b]) * 0.5f;
}

// Direction components and weight of a population index known only at run
// time (one lane per population), from bit masks of the D3Q19 table.
__host__ __device__ constexpr uint32_t fd_mask(int axis, int sign) {
  uint32_t m = 0;
  for (int i = 0; i < kQ; ++i)
    if ((axis == 0 ? cx(i) : axis == 1 ? cy(i) : cz(i)) == sign) m |= 1u << i;
  return m;
}
constexpr uint32_t kFdPx = fd_mask(0, 1), kFdNx = fd_mask(0, -1), kFdPy = fd_mask(1, 1), kFdNy = fd_mask(1, -1),
                   kFdPz = fd_mask(2, 1), kFdNz = fd_mask(2, -1);
__device__ __forceinline__ int c_rt(int axis, int i) {
  const uint32_t pos = axis == 0 ? kFdPx : (axis == 1 ? kFdPy : kFdPz);
  const uint32_t neg = axis == 0 ? kFdNx : (axis == 1 ? kFdNy : kFdNz);
  return static_cast<int>((pos >> i) & 1u) - static_cast<int>((neg >> i) & 1u);
}
__device__ __forceinline__ float w_rt(const int c[3]) {
  const int m = (c[0] != 0) + (c[1] != 0) + (c[2] != 0);
  return m == 0 ? 1.0f / 3.0f : (m == 1 ? 1.0f / 18.0f : 1.0f / 36.0f);
}
// One boundary cell of role ROLE (1 plane, 2 edge, 3 corner) per warp,
// lane i holding population i of every cell the stencil reads: all of them
// are loaded up front (independent loads, one memory latency), the moments
// and densities summed over the warp.  Rewritten populations feq(rho, u) +
// f_neq(Pi), Pi = -rho / (3 omega) (du + du^T), into the cell's row of fnew.
// (The corners in the last CTA of the edges' launch, in place of their own, cost
// 8 us per step more: its rounds read their records with nothing to hide them.)
template <typename T, int ROLE>
__global__ void __launch_bounds__(kFdThreads)
k_fd_reconstruct(const T* state, long long qs, float inv_s, const FdCell* cells, const int* list, int n,
                 float* fnew, const double* time, double time_shift, float omega, const float* cr_shift) {
  pdl_trigger();
  const int w = static_cast<int>((blockIdx.x * kFdThreads + threadIdx.x) >> 5);
  if (w >= n) return;  // whole warps
  const int lane = threadIdx.x & 31;
  const bool act = lane < kQ;
  const int i = act ? lane : 0;
  const int ci[3] = {c_rt(0, i), c_rt(1, i), c_rt(2, i)};
  // the cell's record, staged in shared memory before the predecessor's end
  __shared__ __align__(16) unsigned char rec[kFdThreads / 32][(sizeof(FdCell) + 15) / 16 * 16];
  const int row = list[w];
  {
    static_assert(sizeof(FdCell) % 8 == 0, "copied in 8-byte words");
    const unsigned long long* from = reinterpret_cast<const unsigned long long*>(cells + row);
    unsigned long long* to = reinterpret_cast<unsigned long long*>(rec[threadIdx.x >> 5]);
    for (int k = lane; k < static_cast<int>(sizeof(FdCell) / 8); k += 32) to[k] = from[k];
    __syncwarp();
  }
  const FdCell& cell = *reinterpret_cast<const FdCell*>(rec[threadIdx.x >> 5]);
  // ... and the prescribed velocities its reads name (before the ramp), a lane
  // each: read where they are used, they were up to 13 memory latencies in a row
  __shared__ float4 pres_s[kFdThreads / 32][13];
  float4* pres = pres_s[threadIdx.x >> 5];
  if (lane < 13) {
    int from = -1;
    if (lane < 7) {
      if (cell.u[lane].code == kFdPrescribed) from = static_cast<int>(cell.u[lane].idx);
    } else if (ROLE > 1 && lane - 7 < (ROLE == 2 ? 4 : 6)) {
      const FdRRead& r = cell.r[lane - 7];
      if (r.code == kFdRhoBmPre || r.code == kFdRhoBmNew) from = r.urow;
    }
    if (from >= 0) {
      const FdCell& c = cells[from];
      pres[lane] = make_float4(c.u_base[0], c.u_base[1], c.u_base[2], c.ramp_end);
    }
  }
  __syncwarp();
  pdl_wait();
  const float t = static_cast<float>(*time + time_shift);
  constexpr int nr = ROLE == 2 ? 4 : (ROLE == 3 ? 6 : 0);
  const bool own = ROLE == 1 && cell.kind != kPressureDirichlet;
  // Every value the warp sums, one population per lane: of each velocity read
  // its density and momentum, of each density read (and a plane cell's own
  // populations) the plain sum, or velocityBMRho's outgoing and wall sums.
  constexpr int nv = 28 + 2 * nr + (ROLE == 1 ? 2 : 0);
  float v[nv];
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const FdURead& r = cell.u[j];
    v[4 * j] = act && r.code == kFdFluid ? Store<T>::ld(state + i * qs + r.idx, inv_s) : 0.f;
  }
#pragma unroll
  for (int j = 0; j < nr; ++j) {
    const FdRRead& r = cell.r[j];
    float x = 0.f;
    if (act && r.code != kFdRhoConst)
      x = r.code == kFdRhoSumPre || r.code == kFdRhoBmPre ? Store<T>::ld(state + i * qs + r.idx, inv_s)
                                                          : fnew[r.idx * kQ + i];
    v[28 + 2 * j] = x;
  }
  if constexpr (ROLE == 1) v[28] = act && own ? Store<T>::ld(state + i * qs + cell.slot, inv_s) : 0.f;
  const float shift = cr_shift ? *cr_shift : 0.f;
#pragma unroll
  for (int j = 0; j < 7; ++j)
#pragma unroll
    for (int a = 0; a < 3; ++a) v[4 * j + 1 + a] = ci[a] * v[4 * j];
  auto split = [&](int k, int d, int o) {  // velocityBMRho's sums of v[k]
    const int c = d == 0 ? ci[0] : (d == 1 ? ci[1] : ci[2]);
    const float x = v[k];
    v[k] = c == o ? x : 0.f;
    v[k + 1] = c == 0 ? x : 0.f;
  };
#pragma unroll
  for (int j = 0; j < nr; ++j) {
    const FdRRead& r = cell.r[j];
    v[28 + 2 * j + 1] = 0.f;
    if (r.code == kFdRhoBmPre || r.code == kFdRhoBmNew) split(28 + 2 * j, r.d, r.o);
  }
  if constexpr (ROLE == 1) split(28, cell.d, cell.o);
  // All sums together, step by step of the butterfly: their shuffles are
  // independent (one sum after the other left a warp waiting 5 shuffles per
  // sum, 40 sums in a row: 7 us per launch).
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < nv; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  // the seven velocities
  float uu[7][3];
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const FdURead& r = cell.u[j];
    const float k = 1.f / (1.f + v[4 * j]);
#pragma unroll
    for (int a = 0; a < 3; ++a) uu[j][a] = r.code == kFdFluid ? v[4 * j + 1 + a] * k : 0.f;
    if (r.code == kFdPrescribed) prescribed(pres[j], t, uu[j]);
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (r.flip >> a & 1) uu[j][a] = -uu[j][a];
  }
  auto bm = [&](int k, int d, int o, const float u[3]) {
    const float ud = d == 0 ? u[0] : (d == 1 ? u[1] : u[2]);
    return (2.f * v[k] + v[k + 1] + 1.f) / (1.f + o * ud);
  };
  float rr[nr > 0 ? nr : 1];
#pragma unroll
  for (int j = 0; j < nr; ++j) {
    const FdRRead& r = cell.r[j];
    if (r.code == kFdRhoConst) {
      rr[j] = r.val;
    } else if (r.code == kFdRhoSumPre || r.code == kFdRhoSumNew) {
      // a kBulk cell's stored density under ConstRhoBGK carries the 1 -
      // average_rho its level's last collide added, if that collide came
      // after the level's stream (urow = 1 marks a kBulk cell)
      rr[j] = 1.f + v[28 + 2 * j] - (r.code == kFdRhoSumPre && r.urow == 1 ? shift : 0.f);
    } else {
      float u[3];
      prescribed(pres[7 + j], t, u);
      rr[j] = bm(28 + 2 * j, r.d, r.o, u);
    }
  }
  float du[3][3];
  float rho;
  if constexpr (ROLE == 1) {
    const int d = cell.d, o = cell.o;
    rho = cell.kind == kPressureDirichlet ? cell.rho_target : bm(28, d, o, uu[0]);
    float gn[3];
    normal_grad(uu[0], uu[1], uu[2], o, gn);
    const int t0 = d == 0 ? 1 : 0;  // the lower of the two tangential axes
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
        du[a][b] = a == d ? gn[b] : (a == t0 ? (uu[3][b] - uu[4][b]) * 0.5f : (uu[5][b] - uu[6][b]) * 0.5f);
  } else if constexpr (ROLE == 2) {
    const int p = cell.ax[0], d1 = cell.ax[1];
    float gp[3], g1[3], g2[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) gp[b] = (uu[1][b] - uu[2][b]) * 0.5f;
    normal_grad(uu[0], uu[3], uu[4], cell.nrm[0], g1);
    normal_grad(uu[0], uu[5], uu[6], cell.nrm[1], g2);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) du[a][b] = a == p ? gp[b] : (a == d1 ? g1[b] : g2[b]);
    rho = 2.f / 3.f * (rr[0] + rr[1]) - 1.f / 6.f * (rr[2] + rr[3]);
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) normal_grad(uu[0], uu[1 + 2 * a], uu[2 + 2 * a], cell.nrm[a], du[a]);
    rho = 4.f / 9.f * (rr[0] + rr[1] + rr[2]) - 1.f / 9.f * (rr[3] + rr[4] + rr[5]);
  }
  if (!act) return;
  const float s = -rho / 3.f / omega;
  const float pi[6] = {2.f * du[0][0] * s, (du[0][1] + du[1][0]) * s, (du[0][2] + du[2][0]) * s,
                       2.f * du[1][1] * s, (du[1][2] + du[2][1]) * s, 2.f * du[2][2] * s};
  const float* u = uu[0];
  const float usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
  const float c3[3] = {static_cast<float>(ci[0]), static_cast<float>(ci[1]), static_cast<float>(ci[2])};
  // f_neq from the symmetric stress (lbm.h:248-270): sum over a <= b of
  // (c_a c_b - delta_ab / 3) (x2 off the diagonal) Pi_ab, times w 9 / 2
  float q = 0.f;
  int m = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b, ++m) {
      float qq = c3[a] * c3[b] - (a == b ? 1.f / 3.f : 0.f);
      if (a != b) qq *= 2.f;
      q += qq * pi[m];
    }
  const float wi = w_rt(ci);
  const float cu = c3[0] * u[0] + c3[1] * u[1] + c3[2] * u[2];
  const float feq = rho * wi * (1.f + 3.f * cu + 4.5f * cu * cu - 1.5f * usq) - wi;
  fnew[static_cast<long long>(row) * kQ + i] = feq + q * wi * 4.5f;
}

// The collide of the boundary cells into the state buffer, at the start of
// their level's step: velocity cells f (1 - omega) + omega feq(rho,
// u_presc(t)), rho = velocityBMRho on plane cells and 1 + sum f on edges and
// corners; bounce-back cells the full-way swap of their streamed state (kept
// in their row); pressure cells unchanged.  Source: the rows (the last
// pass's, or the initial state's), or the state itself when fnew is null.
//
// ConstRhoBGK: each CTA's sum of the velocity cells' collide densities goes to
// up.bpart, and the last CTA to finish forms the average the step's collide
// uses (k_cr_update's sums in its order: 256 strided sums, then the shuffle
// trees), which saves that launch.
struct FdCrUpdate {
  double* bpart;              // null: no statistics
  unsigned int* done;
  double* avg;
  const double* part;
  int nparts;
  long long count, bcount;
  float* shift;
};
template <typename T>
__global__ void __launch_bounds__(kFdThreads)
k_fd_collide(T* state, long long qs, float scale, float inv_s, const FdCell* cells, int n, float* fnew,
             const double* time, double time_shift, float omega, const FdCrUpdate up) {
  pdl_trigger();
  const int row = blockIdx.x * kFdThreads + threadIdx.x;
  const FdCell& cell = cells[row < n ? row : 0];
  const int role = cell.role, kind = cell.kind, cd = cell.d, co = cell.o;
  const long long slot = cell.slot;
  const float ub[3] = {cell.u_base[0], cell.u_base[1], cell.u_base[2]}, ramp_end = cell.ramp_end;
  pdl_wait();
  double stat = 0.0;  // ConstRhoBGK statistics: the velocity cell's collide density
  if (row < n) {
  float f[kQ];
  if (role == 0) {
    // a bounce-back cell (the dispatcher's kBounceBack arm, bc_dispatcher.h:
    // 55-67): its streamed populations are its row (the state after the
    // step), then the full-way swap f_i <- f_opp(i)
    load_pops(state, qs, slot, inv_s, f);
    float g[kQ];
#pragma unroll
    for (int i = 0; i < kQ; ++i) {
      if (fnew) fnew[static_cast<long long>(row) * kQ + i] = f[i];
      g[i] = f[i];
    }
#pragma unroll
    for (int i = 0; i < kQ; ++i) f[i] = g[opp(i)];
  } else if (fnew) {
#pragma unroll
    for (int i = 0; i < kQ; ++i) f[i] = fnew[static_cast<long long>(row) * kQ + i];
  } else {
    load_pops(state, qs, slot, inv_s, f);
  }
  if (kind == kVelocityDirichlet) {
    const float r = ramp(static_cast<float>(*time + time_shift), ramp_end);
    const float u[3] = {r * ub[0], r * ub[1], r * ub[2]};
    const float rho = role == 1 ? bm_rho(f, cd, co, u) : 1.f + sum_pops(f);
    stat = rho;
    const float usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
#pragma unroll
    for (int i = 0; i < kQ; ++i) f[i] = f[i] * (1.f - omega) + omega * feq_i(i, rho, u, usq);
  }
#pragma unroll
  for (int i = 0; i < kQ; ++i) Store<T>::st(state + i * qs + slot, f[i], scale);
  }
  if (!up.bpart) return;
  // this CTA's sum, in a fixed order
  for (int o = 16; o > 0; o >>= 1) stat += __shfl_down_sync(0xffffffffu, stat, o);
  __shared__ double ws[kThreads / 32][2];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) ws[warp][0] = stat;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int w = 0; w < kFdThreads / 32; ++w) sum += ws[w][0];
    up.bpart[blockIdx.x] = sum;
    __threadfence();
    last = atomicInc(up.done, gridDim.x - 1) == gridDim.x - 1;  // wraps to 0 for the next launch
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  for (int h = 0; h < kThreads / kFdThreads; ++h) {  // k_cr_update's thread h * kFdThreads + threadIdx.x
    double v[2] = {0.0, 0.0};
    for (int p = h * kFdThreads + threadIdx.x; p < up.nparts; p += kThreads) v[0] += __ldcg(up.part + p);
    for (int p = h * kFdThreads + threadIdx.x; p < static_cast<int>(gridDim.x); p += kThreads) v[1] += __ldcg(up.bpart + p);
    for (int k = 0; k < 2; ++k) {
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
      if (lane == 0) ws[h * (kFdThreads / 32) + warp][k] = v[k];
    }
  }
  __syncthreads();
  if (warp == 0) {
    double v[2];
    for (int k = 0; k < 2; ++k) {
      v[k] = lane < kThreads / 32 ? ws[lane][k] : 0.0;
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    }
    if (lane == 0) {
      cr_average(up.avg, v[0], up.count, v[1], up.bcount);
      if (up.shift) *up.shift = static_cast<float>(1.0 - *up.avg);
    }
  }
}

__global__ void k_fd_tick(double* time) {
  pdl_wait();
  *time += 1.0;
}

// The pass's rewritten rows into the state (velocity and pressure cells; the
// bounce-back cells keep their streamed populations until their collide).
template <typename T>
__global__ void __launch_bounds__(kFdThreads)
k_fd_store(T* state, long long qs, float scale, const FdCell* cells, int n, const float* fnew, double* tick, double ticks) {
  pdl_trigger();
  const int row = blockIdx.x * kFdThreads + threadIdx.x;
  const int role = row < n ? cells[row].role : 0;
  const long long slot = row < n ? cells[row].slot : 0;
  pdl_wait();
  // the boundary clock's tick, where this is the step's last pass (no kernel
  // of the pass reads the clock after the reconstruction)
  if (tick && row == 0) *tick += ticks;
  if (role == 0) return;
  float f[kQ];  // loads before stores (they may alias for all the compiler knows)
#pragma unroll
  for (int i = 0; i < kQ; ++i) f[i] = fnew[static_cast<long long>(row) * kQ + i];
#pragma unroll
  for (int i = 0; i < kQ; ++i) Store<T>::st(state + i * qs + slot, f[i], scale);
}

// The Dirichlet cells' populations before their collide (the initial state)
// into their rows: what the reference holds for them after a step.
template <typename T>
__global__ void __launch_bounds__(kFdThreads)
k_fd_rows_from_state(const T* state, long long qs, float inv_s, const FdCell* cells, int n, float* fnew) {
  const int row = blockIdx.x * kFdThreads + threadIdx.x;
  if (row >= n) return;
#pragma unroll
  for (int i = 0; i < kQ; ++i)
    fnew[static_cast<long long>(row) * kQ + i] = Store<T>::ld(state + i * qs + cells[row].slot, inv_s);
}

// rho and u of the Dirichlet cells from their rows (the populations after the
// pass, before the next collide -- the reference's state after the step),
// over the fields the gather wrote; the bounce-back cells' fields are the
// gathered ones (their streamed state).
__global__ void __launch_bounds__(kFdThreads)
k_fd_fields(const FdCell* cells, int n, const float* fnew, const BlockRun run, FastDiv div_n3, double* rho, double* u) {
  const int row = blockIdx.x * kFdThreads + threadIdx.x;
  if (row >= n || cells[row].role == 0) return;
  double dr = 0, jx = 0, jy = 0, jz = 0;
#pragma unroll
  for (int i = 0; i < kQ; ++i) {
    const double v = fnew[static_cast<long long>(row) * kQ + i];
    dr += v; jx += cx(i) * v; jy += cy(i) * v; jz += cz(i) * v;
  }
  const double r = 1.0 + dr;
  // the cell in the host arrays, as k_gather placed it
  const long long s = host_cell(run, div_n3, static_cast<uint32_t>(cells[row].slot));
  if (s < 0) return;
  rho[s] = r;
  u[3 * s] = jx / r;
  u[3 * s + 1] = jy / r;
  u[3 * s + 2] = jz / r;
}

inline unsigned fd_grid(int n) { return static_cast<unsigned>((n + kFdThreads - 1) / kFdThreads); }

}  // namespace

unsigned fd_collide_parts(int n) { return fd_grid(n); }

template <typename T>
cudaError_t launch_fd_reconstruct(const void* state, long long qs, float inv_s, const FdCell* cells, const int* list,
                                  int role, int n, float* fnew, const double* time, double time_shift, float omega,
                                  const float* cr_shift, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const unsigned grid = static_cast<unsigned>((static_cast<long long>(n) * 32 + kFdThreads - 1) / kFdThreads);
  auto* k = role == 1 ? k_fd_reconstruct<T, 1> : (role == 2 ? k_fd_reconstruct<T, 2> : k_fd_reconstruct<T, 3>);
  const cudaError_t e = launch_chain(k, dim3(grid), dim3(kFdThreads), 0, s, static_cast<const T*>(state), qs, inv_s, cells,
                                     list, n, fnew, time, time_shift, omega, cr_shift);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <typename T>
cudaError_t launch_fd_collide(void* state, long long qs, float scale, float inv_s, const FdCell* cells, int n,
                              float* fnew, const double* time, double time_shift, float omega, double* bpart,
                              unsigned int* done, double* avg, const double* part, int nparts, long long count,
                              long long bcount, float* shift, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const FdCrUpdate up{bpart, done, avg, part, nparts, count, bcount, shift};
  const cudaError_t e = launch_chain(k_fd_collide<T>, dim3(fd_grid(n)), dim3(kFdThreads), 0, s, static_cast<T*>(state), qs,
                                     scale, inv_s, cells, n, fnew, time, time_shift, omega, up);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <typename T>
cudaError_t launch_fd_rows_from_state(const void* state, long long qs, float inv_s, const FdCell* cells, int n,
                                     float* fnew, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_fd_rows_from_state<T><<<fd_grid(n), kFdThreads, 0, s>>>(static_cast<const T*>(state), qs, inv_s, cells, n, fnew);
  return cudaGetLastError();
}

cudaError_t launch_fd_fields(const FdCell* cells, int n, const float* fnew, const BlockRun& run, FastDiv div_n3, double* rho,
                             double* u, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_fd_fields<<<fd_grid(n), kFdThreads, 0, s>>>(cells, n, fnew, run, div_n3, rho, u);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_fd_store(void* state, long long qs, float scale, const FdCell* cells, int n, const float* fnew,
                            double* tick, double ticks, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const cudaError_t e = launch_chain(k_fd_store<T>, dim3(fd_grid(n)), dim3(kFdThreads), 0, s, static_cast<T*>(state), qs,
                                     scale, cells, n, fnew, tick, ticks);
  return e != cudaSuccess ? e : cudaGetLastError();
}
template cudaError_t launch_fd_store<float>(void*, long long, float, const FdCell*, int, const float*, double*,
                                           double, cudaStream_t);
template cudaError_t launch_fd_store<__half>(void*, long long, float, const FdCell*, int, const float*, double*,
                                            double, cudaStream_t);

cudaError_t launch_fd_tick(double* time, cudaStream_t s) {
  const cudaError_t e = launch_chain(k_fd_tick, dim3(1), dim3(1), 0, s, time);
  return e != cudaSuccess ? e : cudaGetLastError();
}

#define OCTLB_FD_INST(T)                                                                                      \
  template cudaError_t launch_fd_reconstruct<T>(const void*, long long, float, const FdCell*, const int*, int, int, \
                                                float*, const double*, double, float, const float*, cudaStream_t);          \
  template cudaError_t launch_fd_collide<T>(void*, long long, float, float, const FdCell*, int, float*,        \
                                            const double*, double, float, double*, unsigned int*, double*,     \
                                            const double*, int, long long, long long, float*, cudaStream_t);
template cudaError_t launch_fd_rows_from_state<float>(const void*, long long, float, const FdCell*, int, float*,
                                                     cudaStream_t);
template cudaError_t launch_fd_rows_from_state<__half>(const void*, long long, float, const FdCell*, int, float*,
                                                      cudaStream_t);
OCTLB_FD_INST(float)
OCTLB_FD_INST(__half)

}  // namespace octlb_gpu
