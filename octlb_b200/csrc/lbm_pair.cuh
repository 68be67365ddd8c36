// A pair of cells in packed FP32 (f32x2) registers: the arithmetic and the
// collide of the slot-map step, which holds two cells per thread.
#ifndef OCTLB_LBM_PAIR_CUH_
#define OCTLB_LBM_PAIR_CUH_

#include "lbm_common.cuh"

namespace octlb_gpu {
namespace {

using u64 = unsigned long long;

// Packed FP32 pairs: each half is the scalar operation, round to nearest.
__device__ __forceinline__ u64 pk(float a, float b) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ u64 pk1(float a) { return pk(a, a); }
__device__ __forceinline__ void upk(u64 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Moments of a pair in storage units, in moments()' order: dh = sum f, j.
__device__ __forceinline__ void moments2(const u64 (&f)[kQ], u64& dh, u64& jx, u64& jy, u64& jz) {
  const u64 m1 = pk1(-1.0f);
  auto sub = [&](u64 a, u64 b) { return fma2(b, m1, a); };
  const u64 d10 = sub(f[10], f[1]), d11 = sub(f[11], f[2]), d12 = sub(f[12], f[3]);
  const u64 d13 = sub(f[13], f[4]), d14 = sub(f[14], f[5]), d15 = sub(f[15], f[6]);
  const u64 d16 = sub(f[16], f[7]), d17 = sub(f[17], f[8]), d18 = sub(f[18], f[9]);
  jx = add2(add2(add2(d10, d13), add2(d14, d15)), d16);
  jy = add2(sub(add2(d11, d13), d14), add2(d17, d18));
  jz = add2(sub(add2(d12, d15), d16), sub(d17, d18));
  const u64 s1 = add2(add2(add2(f[1], f[10]), add2(f[2], f[11])), add2(f[3], f[12]));
  const u64 s2 = add2(add2(add2(f[4], f[13]), add2(f[5], f[14])), add2(add2(f[6], f[15]), add2(f[7], f[16])));
  const u64 s3 = add2(add2(f[8], f[17]), add2(f[9], f[18]));
  dh = add2(f[0], add2(s1, add2(s2, s3)));
}

// c_i . u of the positive direction i = 10..18 (its opposite is the exact
// negative).
template <int I>
__device__ __forceinline__ u64 cu_pos(u64 ux, u64 uy, u64 uz) {
  const u64 m1 = pk1(-1.0f);
  if constexpr (I == 10) return ux;
  else if constexpr (I == 11) return uy;
  else if constexpr (I == 12) return uz;
  else if constexpr (I == 13) return add2(ux, uy);
  else if constexpr (I == 14) return fma2(uy, m1, ux);
  else if constexpr (I == 15) return add2(ux, uz);
  else if constexpr (I == 16) return fma2(uz, m1, ux);
  else if constexpr (I == 17) return add2(uy, uz);
  else return fma2(uz, m1, uy);
}

// The pair's collide in storage units h = s (f - w), s a power of two (1 for
// FP32 storage): bgk<false>() of each cell.  Opposite directions share
// c . u; with q = 4.5 A cu -+ 3 A, t = c0 + cu q, the relaxation
// f + omega (w t - f) is formed as f - omega (f - w t): the same roundings.
// kCollConstRho adds dr w_i P_i as bgk_const_rho() (d0, d1: rho - 1).
template <int CM, bool SCALED>
__device__ __forceinline__ void collide2(u64 (&f)[kQ], float omega, float s, float inv_s, float dr, float& d0, float& d1) {
  u64 dh, jx, jy, jz;
  moments2(f, dh, jx, jy, jz);
  float h0, h1;
  upk(dh, h0, h1);
  if constexpr (SCALED) { h0 *= inv_s; h1 *= inv_s; }
  const float r0 = 1.0f + h0, r1 = 1.0f + h1;
  float k0 = __frcp_rn(r0), k1 = __frcp_rn(r1);
  if constexpr (SCALED) { k0 *= inv_s; k1 *= inv_s; }
  const u64 k = pk(k0, k1);
  const u64 ux = mul2(jx, k), uy = mul2(jy, k), uz = mul2(jz, k);
  const u64 usq = fma2(uz, uz, fma2(ux, ux, mul2(uy, uy)));
  u64 A = pk(r0, r1);  // s rho
  if constexpr (SCALED) A = mul2(A, pk1(s));
  const u64 no = pk1(-omega);
  constexpr float nw[3] = {-1.0f / 3.0f, -1.0f / 18.0f, -1.0f / 36.0f};
  if constexpr (CM == kCollConstRho) {
    d0 = h0;
    d1 = h1;
    const u64 nu15 = mul2(pk1(-1.5f), usq);  // P_0 - 1
    u64 d = pk(r0 > 1e-12f ? dr : 0.0f, r1 > 1e-12f ? dr : 0.0f);
    if constexpr (SCALED) d = mul2(d, pk1(s));
    const u64 one = pk1(1.0f), c45 = pk1(4.5f), c3 = pk1(3.0f), n3 = pk1(-3.0f);
    auto relax = [&](int i, u64 q) {
      const int w = i == 0 ? 0 : ((cx(i) != 0) + (cy(i) != 0) + (cz(i) != 0) == 1 ? 1 : 2);
      const u64 t = fma2(A, q, dh);
      const u64 g = fma2(no, fma2(pk1(nw[w]), t, f[i]), f[i]);
      f[i] = fma2(mul2(pk1(-nw[w]), d), add2(one, q), g);
    };
    relax(0, nu15);
    auto both = [&](int i, u64 cu) {
      relax(i, fma2(cu, fma2(c45, cu, c3), nu15));
      relax(i - 9, fma2(cu, fma2(c45, cu, n3), nu15));
    };
    both(10, cu_pos<10>(ux, uy, uz)); both(11, cu_pos<11>(ux, uy, uz)); both(12, cu_pos<12>(ux, uy, uz));
    both(13, cu_pos<13>(ux, uy, uz)); both(14, cu_pos<14>(ux, uy, uz)); both(15, cu_pos<15>(ux, uy, uz));
    both(16, cu_pos<16>(ux, uy, uz)); both(17, cu_pos<17>(ux, uy, uz)); both(18, cu_pos<18>(ux, uy, uz));
  } else {
    const u64 a3 = mul2(pk1(3.0f), A), n3 = mul2(pk1(-3.0f), A), b45 = mul2(pk1(4.5f), A);
    const u64 c0 = fma2(mul2(pk1(-1.5f), A), usq, dh);
    auto relax = [&](int i, u64 t) {
      const int w = i == 0 ? 0 : ((cx(i) != 0) + (cy(i) != 0) + (cz(i) != 0) == 1 ? 1 : 2);
      f[i] = fma2(no, fma2(pk1(nw[w]), t, f[i]), f[i]);
    };
    relax(0, c0);
    auto both = [&](int i, u64 cu) {
      relax(i, fma2(cu, fma2(b45, cu, a3), c0));
      relax(i - 9, fma2(cu, fma2(b45, cu, n3), c0));
    };
    both(10, cu_pos<10>(ux, uy, uz)); both(11, cu_pos<11>(ux, uy, uz)); both(12, cu_pos<12>(ux, uy, uz));
    both(13, cu_pos<13>(ux, uy, uz)); both(14, cu_pos<14>(ux, uy, uz)); both(15, cu_pos<15>(ux, uy, uz));
    both(16, cu_pos<16>(ux, uy, uz)); both(17, cu_pos<17>(ux, uy, uz)); both(18, cu_pos<18>(ux, uy, uz));
  }
}

}  // namespace
}  // namespace octlb_gpu

#endif  // OCTLB_LBM_PAIR_CUH_
