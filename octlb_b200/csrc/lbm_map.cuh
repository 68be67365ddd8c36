// Forest-level step with a per-block slot map (k_step_map).
//
// Every block has an (n+2)^3 map: padded position -> slot (own core, the
// neighbour core the same-level exchange copies, the source cell of an
// outflow ghost copy, the own halo page) or a bounce-back wall marker (-1 at
// rest, -(2 + k) moving), so a pull is one map read and one load with no
// per-direction branching at block faces.
//
// Two z-adjacent cells per thread.  Where the block's z rows are uniform
// (kBlkRows: every row of sources is n adjacent slots, or all wall), the pair
// reads one map entry per source row (8) and one per row beyond whose end it
// pulls (5, lanes at the row's ends only), and one aligned 2-element load per
// population; directions along z take the element of the neighbouring lane by
// a shuffle.  Other blocks read map and value per cell and direction.  The
// pair is collided with packed FP32 instructions, each half rounded as bgk()
// rounds, and stored with 2-element accesses.  A CTA takes 2 THREADS
// consecutive cells of a block.  Under the links rule the first CTAs of the
// launch take the near-wall cells (one warp each), and the last CTAs stream
// the open blocks' halo items.
//
// What bounds it: on small levels the chain row table -> load -> collide ->
// store of one wave; on large ones memory latency at 28 warps per SM (60 % of
// the DRAM peak at 128^3 cells, FP32).  Measured per step, before (one or two
// cells 256 apart per thread, a map read per pull, scalar collide: 735
// instructions per cell) and now (300): 128^3 cavity under ConstRhoBGK FP32
// 84.2 -> 63.8 us, FP16 75.9 -> 48.8 us; the finest level of the 512x128x128
// cylinder FP16 82.8 -> 55.4 us.  Tried and slower: persistent CTAs with whole
// blocks staged in shared memory by tensor copies (16 warps per SM, 128
// registers: the pulls' index arithmetic and the barriers cost what the copies
// saved; 77 us on that cavity FP32, and 1.4 times this kernel's time on levels
// of a few hundred blocks).
#ifndef OCTLB_LBM_MAP_CUH_
#define OCTLB_LBM_MAP_CUH_

#include <cmath>

#include "lbm_pair.cuh"
#include "lbm_step.cuh"

namespace octlb_gpu {
namespace {

// How stored values meet the collide: FP32 storage as it is; FP16 storage
// units with a power-of-two scale (every rounding falls where the unit-scale
// collide's does); FP16 with any other scale converted at load and store.
enum : int { kUnit = 0, kPow2 = 1, kConvert = 2 };

template <int SM>
__device__ __forceinline__ float ld1(const float* p, float) { return *p; }
template <int SM>
__device__ __forceinline__ float ld1(const __half* p, float inv) {
  const float v = __half2float(*p);
  return SM == kConvert ? v * inv : v;
}
template <int SM>
__device__ __forceinline__ u64 ld2(const float* p, float) { return *reinterpret_cast<const u64*>(p); }
template <int SM>
__device__ __forceinline__ u64 ld2(const __half* p, float inv) {
  const float2 w = __half22float2(*reinterpret_cast<const __half2*>(p));
  return SM == kConvert ? pk(w.x * inv, w.y * inv) : pk(w.x, w.y);
}
template <int SM>
__device__ __forceinline__ void st2(float* p, u64 v, float) { *reinterpret_cast<u64*>(p) = v; }
template <int SM>
__device__ __forceinline__ void st2(__half* p, u64 v, float scale) {
  float a, b;
  upk(v, a, b);
  if (SM == kConvert) { a *= scale; b *= scale; }
  *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b);
}
template <int SM>
__device__ __forceinline__ void st1(float* p, float v, float) { *p = v; }
template <int SM>
__device__ __forceinline__ void st1(__half* p, float v, float scale) { *p = __float2half_rn(SM == kConvert ? v * scale : v); }

// The five (c_x, c_y) of the directions with c_z != 0, and those directions.
__host__ __device__ constexpr int combo_x(int c) { return c == 1 ? 1 : (c == 2 ? -1 : 0); }
__host__ __device__ constexpr int combo_y(int c) { return c == 3 ? 1 : (c == 4 ? -1 : 0); }
__host__ __device__ constexpr int combo_up(int c) {
  constexpr int t[5] = {12, 15, 7, 17, 9};
  return t[c];
}
__host__ __device__ constexpr int combo_dn(int c) {
  constexpr int t[5] = {3, 16, 6, 18, 8};
  return t[c];
}

// Two adjacent stored values as loaded.  shift_up: the pair one cell up the
// row, (value of z - 1, value of z), z - 1 from the previous lane's pair, or h
// in the row's first lane; shift_down: (z + 1, z + 2).
template <typename T> struct RawPairOf;
template <> struct RawPairOf<float> { using type = float2; };
template <> struct RawPairOf<__half> { using type = uint32_t; };
template <typename T> using RawPair = typename RawPairOf<T>::type;
__device__ __forceinline__ float2 shift_up(float2 v, float h, bool first, bool wall) {
  const float a = __shfl_up_sync(0xffffffffu, v.y, 1);
  return make_float2(first ? h : (wall ? v.x : a), wall ? v.y : v.x);
}
__device__ __forceinline__ float2 shift_down(float2 v, float h, bool last, bool wall) {
  const float b = __shfl_down_sync(0xffffffffu, v.x, 1);
  return make_float2(wall ? v.x : v.y, last ? h : (wall ? v.y : b));
}
__device__ __forceinline__ uint32_t shift_up(uint32_t v, __half h, bool first, bool wall) {
  const uint32_t a = __shfl_up_sync(0xffffffffu, v, 1) >> 16;
  const uint32_t lo = first ? static_cast<uint32_t>(__half_as_ushort(h)) : (wall ? v & 0xffffu : a);
  return lo | (wall ? v & 0xffff0000u : v << 16);
}
__device__ __forceinline__ uint32_t shift_down(uint32_t v, __half h, bool last, bool wall) {
  const uint32_t b = __shfl_down_sync(0xffffffffu, v, 1) << 16;
  const uint32_t hi = last ? static_cast<uint32_t>(__half_as_ushort(h)) << 16 : (wall ? v & 0xffff0000u : b);
  return hi | (wall ? v & 0xffffu : v >> 16);
}
template <int SM>
__device__ __forceinline__ u64 raw2(float2 v, float) { return pk(v.x, v.y); }
template <int SM>
__device__ __forceinline__ u64 raw2(uint32_t v, float inv) {
  const float2 w = __half22float2(*reinterpret_cast<const __half2*>(&v));
  return SM == kConvert ? pk(w.x * inv, w.y * inv) : pk(w.x, w.y);
}

// CM: kCollBgk, kCollConstRho (at average density *cr_avg, with per near-cell
// and core CTA the sum of rho - 1 over its collided kBulk cells in
// cr_part[blockIdx.x]; the halo-item CTAs after them write none), or
// kCollNone.
template <typename T, int N, int SM, bool LINKS, bool FLAGS, int CM, int THREADS, int WARPS>
__global__ void __launch_bounds__(THREADS, WARPS * 32 / THREADS) k_step_map(const StepArgs a, const NearTables nt) {
  constexpr uint32_t kN3 = N * N * N, kParts = kN3 / (2 * THREADS);
  constexpr int kNp = N + 2;
  constexpr uint32_t kWarps = THREADS / 32;
  __shared__ float sdh[CM == kCollConstRho ? 2 * THREADS : 1];
  __shared__ double sws[2][kThreads / 32];
  static_assert(CM != kCollConstRho || THREADS == kThreads, "the statistics take whole 512-cell CTAs");
  constexpr uint32_t kStat = LINKS ? 2 : 1;  // statistics values per core CTA
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t near_ctas = LINKS ? (static_cast<uint32_t>(nt.n) + kWarps - 1) / kWarps : 0;
  const uint32_t core_ctas = static_cast<uint32_t>(a.nblk) * kParts;
  if (LINKS && blockIdx.x < near_ctas) {
    const int k = static_cast<int>(blockIdx.x * kWarps + warp);
    if constexpr (CM == kCollConstRho) {
      pdl_wait();
      const float dr = static_cast<float>(1.0 - *a.cr_avg);
      const float dh = near_cell<T, kCollConstRho>(a, nt, k, static_cast<int>(lane), dr);
      double v[1] = {lane == 0 ? static_cast<double>(dh) : 0.0};
      block_reduce<1>(v);
      if (tid == 0) a.cr_part[blockIdx.x] = v[0];
      if (blockIdx.x == 0)
        for (int p = static_cast<int>(near_ctas + core_ctas * kStat + tid); p < a.cr_total; p += THREADS) a.cr_part[p] = 0.0;
    } else {
      near_cell<T, CM>(a, nt, k, static_cast<int>(lane));
    }
    return;
  }
  const uint32_t bid = blockIdx.x - near_ctas;
  if (bid >= core_ctas) {
    rotate_item<T>(a, (bid - core_ctas) * THREADS + tid);
    return;
  }
  const uint32_t b = bid / kParts, tl = (bid % kParts) * (2 * THREADS) + 2 * tid;
  const uint32_t t = b * kN3 + tl;
  const uint32_t x = tl / (N * N), y = (tl / N) % N, z = tl % N;
  const int* gm = a.slot_map + static_cast<long long>(b) * (kNp * kNp * kNp) + ((x + 1) * kNp + y + 1) * kNp + z + 1;
  const uint8_t info = a.blk_info[b];  // uniform over the CTA
  const uint32_t fl = FLAGS ? *reinterpret_cast<const uint16_t*>(a.flags + t) : 0;
  const T* src = static_cast<const T*>(a.src);
  T* dst = static_cast<T*>(a.dst);
  const uint32_t qs = static_cast<uint32_t>(a.qs);
  const float inv = a.inv_scale;
  u64 f[kQ];
  // marker-aware offset of cell t's pull of direction i from map value m
  auto offset = [&](int i, int m, uint32_t tc) {
    const uint32_t own = i <= 9 ? tc + 9 * qs : tc - 9 * qs;  // opposite row (mod 2^32)
    return static_cast<uint32_t>(i) * qs + (m < 0 ? own : static_cast<uint32_t>(m));
  };
  const float wscale = SM == kPow2 ? a.scale : 1.f;
  // the moving-wall term (markers < -1)
  auto wall_term = [&](int i, int second, float v) {
    const int m = __ldg(gm + second - (cx(i) * kNp * kNp + cy(i) * kNp + cz(i)));
    return m < -1 ? v + a.wall_add[(-m - 2) * kQ + i] * wscale : v;
  };
  // one cell's pull on its own
  auto pulled = [&](int i, int second) {
    const int m = __ldg(gm + second - (cx(i) * kNp * kNp + cy(i) * kNp + cz(i)));
    const float v = ld1<SM>(src + offset(i, m, t + second), inv);
    return (info & kBlkMoving) ? wall_term(i, second, v) : v;
  };
  // Uniform rows: row[cx][cy], the slot of the first cell of the pair's source
  // row (or its marker: the whole row is wall), and hz[combo], the one position
  // beyond the row that a lane at the row's ends needs (z - 1 for the first
  // pair of the row, z + 2 for the last).  The block's row table holds the
  // slots of Z = 1, 0 and n + 1 of every (X, Y), so a warp's rows are a few
  // consecutive entries.  Read before the block's kind is known: one latency
  // instead of two.
  constexpr int kRow = kNp * kNp;
  const bool zlo = z == 0, zhi = z == N - 2;
  const int* rm = a.row_map + b * (3u * kRow) + (x + 1) * kNp + y + 1;
  int row[3][3], hz[5];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q < 3; ++q)
      row[p][q] = p == 1 && q == 1 ? 0 : __ldg(rm - ((p - 1) * kNp + (q - 1)));
#pragma unroll
  for (int c = 0; c < 5; ++c)
    hz[c] = zlo || zhi ? __ldg(rm + (zlo ? kRow : 2 * kRow) - (combo_x(c) * kNp + combo_y(c))) : 0;
  if (info & kBlkRows) {
    pdl_wait();
    // a wall row is the cells' own opposite row, 9 planes up or down (mod 2^32)
    const uint32_t up9 = t + 9 * qs, dn9 = t - 9 * qs;
    RawPair<T> v[kQ];
    T h[5];
#pragma unroll
    for (int i = 0; i < kQ; ++i) {
      const int m = row[cx(i) + 1][cy(i) + 1];
      const uint32_t at = cx(i) == 0 && cy(i) == 0 ? t : (m < 0 ? (i <= 9 ? up9 : dn9) : static_cast<uint32_t>(m) + z);
      v[i] = *reinterpret_cast<const RawPair<T>*>(src + (static_cast<uint32_t>(i) * qs + at));
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      // population combo_up(c) (c_z = 1) for the first pair, combo_dn(c) for the last
      const uint32_t i = zlo ? combo_up(c) : combo_dn(c), o = zlo ? opp(combo_up(c)) : opp(combo_dn(c));
      const uint32_t off = hz[c] >= 0 ? i * qs + static_cast<uint32_t>(hz[c]) : o * qs + t + (zlo ? 0u : 1u);
      if (zlo || zhi) h[c] = src[off];
    }
#pragma unroll
    for (int i = 0; i < kQ; ++i)
      if (cz(i) == 0) f[i] = raw2<SM>(v[i], inv);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const bool wall = c > 0 && row[combo_x(c) + 1][combo_y(c) + 1] < 0;
      const RawPair<T> up = v[combo_up(c)], dn = v[combo_dn(c)];
      // a wall row: the cells' own values, not shifted; else one cell along z
      // through the neighbouring lane
      f[combo_up(c)] = raw2<SM>(shift_up(up, h[c], zlo, wall), inv);
      f[combo_dn(c)] = raw2<SM>(shift_down(dn, h[c], zhi, wall), inv);
    }
    if (info & kBlkMoving) {
      // wall term k = -marker - 2 (the table is read again: in L1, and no
      // registers held)
#pragma unroll
      for (int i = 1; i < kQ; ++i) {
        int m0, m1;
        row_wall_marks(cx(i) || cy(i), rm - (cx(i) * kNp + cy(i)), kRow, cz(i), static_cast<int>(z), N, m0, m1);
        float u, v;
        upk(f[i], u, v);
        if (cz(i) == 0) {  // both cells or neither: two loads at once (cylinder 256x64x64: 163 -> 161 us per call)
          if (m0 < -1) {
            u += a.wall_add[(-m0 - 2) * kQ + i] * wscale;
            v += a.wall_add[(-m0 - 1) * kQ + i] * wscale;
          }
        } else {
          if (m0 < -1) u += a.wall_add[(-m0 - 2) * kQ + i] * wscale;
          if (m1 < -1) v += a.wall_add[(-m1 - 2) * kQ + i] * wscale;
        }
        f[i] = pk(u, v);
      }
    }
  } else {
    int m[kQ][2];
#pragma unroll
    for (int i = 1; i < kQ; ++i) {
      const int off = -(cx(i) * kNp * kNp + cy(i) * kNp + cz(i));
      m[i][0] = __ldg(gm + off);
      m[i][1] = __ldg(gm + off + 1);
    }
    pdl_wait();
    f[0] = ld2<SM>(src + t, inv);
#pragma unroll
    for (int i = 1; i < kQ; ++i)
      f[i] = pk(ld1<SM>(src + offset(i, m[i][0], t), inv), ld1<SM>(src + offset(i, m[i][1], t + 1), inv));
    if (info & kBlkMoving) {
#pragma unroll
      for (int i = 1; i < kQ; ++i) {
        float u, v;
        upk(f[i], u, v);
        f[i] = pk(wall_term(i, 0, u), wall_term(i, 1, v));
      }
    }
  }
  const uint32_t fa = fl & 0xffu, fb = fl >> 8;
  bool bulk0 = true, bulk1 = true, go0 = true, go1 = true;
  if constexpr (LINKS) {
    go0 = (fa & kKindMask) != kSolid && !(fa & kFlagNear);
    go1 = (fb & kKindMask) != kSolid && !(fb & kFlagNear);
  }
  if constexpr (FLAGS) {
    if (fl & (kFlagSave | kFlagSave << 8)) {
      const float w = SM == kPow2 ? inv : 1.f;
      const bool s0 = (fa & kFlagSave) && go0, s1 = (fb & kFlagSave) && go1;
      float* sv0 = s0 ? a.save_buf + static_cast<long long>(a.save_idx[t]) * kQ : nullptr;
      float* sv1 = s1 ? a.save_buf + static_cast<long long>(a.save_idx[t + 1]) * kQ : nullptr;
#pragma unroll
      for (int i = 0; i < kQ; ++i) {
        float u, v;
        upk(f[i], u, v);
        if (s0) sv0[i] = u * w;
        if (s1) sv1[i] = v * w;
      }
    }
    bulk0 = (fa & kKindMask) == kBulk;
    bulk1 = (fb & kKindMask) == kBulk;
  }
  float d0 = 0.f, d1 = 0.f;
  if constexpr (CM != kCollNone) {
    float dr = 0.f;
    if constexpr (CM == kCollConstRho) dr = static_cast<float>(1.0 - *a.cr_avg);
    if (bulk0 && bulk1) {
      collide2<CM, SM == kPow2>(f, a.omega, a.scale, inv, dr, d0, d1);
    } else if (bulk0 || bulk1) {
      // one cell of the pair keeps its pulled populations
      collide2<CM, SM == kPow2>(f, a.omega, a.scale, inv, dr, d0, d1);
      const int second = bulk0 ? 1 : 0;
#pragma unroll
      for (int i = 0; i < kQ; ++i) {
        const float raw = pulled(i, second);
        float u, v;
        upk(f[i], u, v);
        f[i] = second ? pk(u, raw) : pk(raw, v);
      }
      (bulk0 ? d1 : d0) = 0.f;
    }
  }
  if (go0 && go1) {
#pragma unroll
    for (int i = 0; i < kQ; ++i) st2<SM>(dst + (static_cast<uint32_t>(i) * qs + t), f[i], a.scale);
  } else {
    // a solid cell keeps its populations (neither streamed nor collided,
    // block_lattice.cpp:581-583); a near-wall cell is near_cell's
#pragma unroll
    for (int i = 0; i < kQ; ++i) {
      T* oi = dst + (static_cast<uint32_t>(i) * qs + t);
      float u, v;
      upk(f[i], u, v);
      if (go0) st1<SM>(oi, u, a.scale);
      if (go1) st1<SM>(oi + 1, v, a.scale);
    }
    if ((fa & kKindMask) == kSolid) copy_cell(src, dst, a.qs, t);
    if ((fb & kKindMask) == kSolid) copy_cell(src, dst, a.qs, t + 1);
  }
  if constexpr (CM == kCollConstRho) {
    // The CTA's sum of rho - 1 in a fixed order, by block_reduce's shuffle tree
    // over 256 values: the cells c and c + 256 paired, or (links rule) each half
    // on its own.
    // (A prolongation's target and a near-wall cell are counted where their
    // collide is.)
    if (!go0 || (FLAGS && (fa & kFlagProlong))) d0 = 0.f;
    if (!go1 || (FLAGS && (fb & kFlagProlong))) d1 = 0.f;
    *reinterpret_cast<float2*>(&sdh[2 * tid]) = make_float2(d0, d1);
    __syncthreads();
#pragma unroll
    for (uint32_t h = 0; h < kStat; ++h) {
      double v = static_cast<double>(kStat == 1 ? sdh[tid] + sdh[tid + THREADS] : sdh[tid + h * THREADS]);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) sws[h][warp] = v;
    }
    __syncthreads();
    if (warp < kStat) {
      double v = lane < kWarps ? sws[warp][lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) a.cr_part[near_ctas + bid * kStat + warp] = v;
    }
    if (blockIdx.x == 0)
      for (int p = static_cast<int>(near_ctas + core_ctas * kStat + tid); p < a.cr_total; p += THREADS) a.cr_part[p] = 0.0;
  }
}

template <typename T, int N, int SM, int CM, int WARPS>
cudaError_t launch_map_w(const StepArgs& a, const NearTables& nt, bool links, bool flags, dim3 g, cudaStream_t s) {
  constexpr int kT = CM == kCollConstRho ? kThreads : 128;
  if (links) return launch_chain(k_step_map<T, N, SM, true, true, CM, kT, WARPS>, g, dim3(kT), 0, s, a, nt);
  if (flags) return launch_chain(k_step_map<T, N, SM, false, true, CM, kT, WARPS>, g, dim3(kT), 0, s, a, nt);
  return launch_chain(k_step_map<T, N, SM, false, false, CM, kT, WARPS>, g, dim3(kT), 0, s, a, nt);
}
template <typename T, int N, int SM, int CM>
cudaError_t launch_map(const StepArgs& a, const NearTables& nt, bool links, bool flags, cudaStream_t s) {
  // 128-thread CTAs (256 cells): small levels spread over more SMs and the last
  // wave is shorter.  The ConstRhoBGK statistics take 256-thread ones.
  constexpr int kT = CM == kCollConstRho ? kThreads : 128;
  const uint32_t parts = N * N * N / (2 * kT);
  const uint32_t near_ctas = links ? (static_cast<uint32_t>(nt.n) + kT / 32 - 1) / (kT / 32) : 0;
  const dim3 g(near_ctas + static_cast<uint32_t>(a.nblk) * parts + (static_cast<uint32_t>(a.n_open) + kT - 1) / kT);
  // 32 warps per SM (64 registers, the loads in two batches, 40 - 150 bytes of
  // spill) win where the CTAs fill more than one wave of the 20-warp form (2.1M
  // cells FP32: 63.8 us against 74.6); that form issues every load at once and
  // wins where they do not (32^3 cells: 4.1 us per step against 5.1).  It holds
  // five 128-thread CTAs per SM, and two of the statistics' 256-thread ones (16
  // warps): ConstRhoBGK on 324 - 360 blocks of 8^3, 7.7 us per step with 32 warps
  // against 9.4 - 9.8 FP32, 7.2 - 7.3 against 7.8 - 8.0 FP16; on 288 - 294 blocks
  // 6.7 - 6.9 and 5.8 - 6.0 us with the 20-warp form.
  constexpr uint32_t kResident = 20 * 32 / kT;
  const bool wide = g.x <= kResident * static_cast<uint32_t>(a.sms);
  if constexpr (SM != kConvert)
    if (wide) return launch_map_w<T, N, SM, CM, 20>(a, nt, links, flags, g, s);
  return launch_map_w<T, N, SM, CM, 32>(a, nt, links, flags, g, s);
}
template <typename T, int N, int SM>
cudaError_t launch_map_cm(const StepArgs& a, const NearTables& nt, bool links, bool flags, int cm, cudaStream_t s) {
  if (cm == kCollConstRho) return launch_map<T, N, SM, kCollConstRho>(a, nt, links, flags, s);
  if (cm == kCollNone) return launch_map<T, N, SM, kCollNone>(a, nt, links, flags, s);
  return launch_map<T, N, SM, kCollBgk>(a, nt, links, flags, s);
}
}  // namespace

// One step of a level of N^3 blocks; cm: its collide.  Every storage type and
// block edge is a source file of its own (lbm_map_*.cu): a process loads a
// file's kernels together, on its first launch of one of them (all in one file:
// 18 ms of a program's first advance_one).
template <typename T, int N>
cudaError_t launch_map_n(const StepArgs& a, const NearTables& nt, bool links, bool flags, int cm, cudaStream_t s) {
  if constexpr (sizeof(T) == 4) return launch_map_cm<T, N, kUnit>(a, nt, links, flags, cm, s);
  int ex = 0;
  if (std::frexp(a.scale, &ex) == 0.5f && ex > -60 && ex < 60) return launch_map_cm<T, N, kPow2>(a, nt, links, flags, cm, s);
  return launch_map_cm<T, N, kConvert>(a, nt, links, flags, cm, s);
}

}  // namespace octlb_gpu

#endif  // OCTLB_LBM_MAP_CUH_
