// FP32 macro step and MRT collision on one node or on two nodes at once.
//
// Blackwell's packed FP32 instructions (add / mul / fma .rn.f32x2) do two
// independent FP32 operations per issued instruction.  The step is bound by
// issue slots as soon as its bytes come from L2 (about 490 instructions per
// node, 69 % of the issue slots at 256^3, 75 % with 16-bit storage), so a
// thread works on two neighbouring nodes, one per half of each pair.
//
// The operator is mrt_collide_dev's (kernels_common.cuh).  Every operation
// here is one rounding that the source states (intrinsics or PTX, nothing
// left to contraction), so one node and two nodes give the same bits, in
// every kernel that includes this file.
#pragma once

#include "kernels_common.cuh"

namespace lbm {

// Two FP32 values in a 64-bit register pair.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 make_f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 split_f2(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}

template <typename V>
struct VecOf;
template <>
struct VecOf<float> {
  static constexpr int kNodes = 1;
  static __device__ __forceinline__ float splat(float x) { return x; }
};
template <>
struct VecOf<F2> {
  static constexpr int kNodes = 2;
  static __device__ __forceinline__ F2 splat(float x) { return make_f2(x, x); }
};

__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vrcp(float a) { return __frcp_rn(a); }
__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// a - b as a + (-1) b: one rounding, of the same value
__device__ __forceinline__ F2 vsub(F2 a, F2 b) { return vfma(b, make_f2(-1.f, -1.f), a); }
__device__ __forceinline__ F2 vrcp(F2 a) {
  const float2 s = split_f2(a);
  return make_f2(__frcp_rn(s.x), __frcp_rn(s.y));
}
__device__ __forceinline__ float vneg(float a) { return -a; }
// acc + c v for a compile-time integer c
template <typename V>
__device__ __forceinline__ V vterm(int c, V v, V acc) {
  if (c == 1) return vadd(acc, v);
  if (c == -1) return vsub(acc, v);
  return vfma(VecOf<V>::splat((float)c), v, acc);
}
// c v
template <typename V>
__device__ __forceinline__ V vscale(int c, V v) {
  return c == 1 ? v : vmul(VecOf<V>::splat((float)c), v);
}

// rho, u of the deviations f (macro_dev's sums, in its order).
template <typename V>
__device__ __forceinline__ void macro_vec(const V (&f)[kQ], float hgx, float hgy, float hgz, V& drho, V& rho, V& ux,
                                          V& uy, V& uz) {
  using O = VecOf<V>;
  V s[9], d[9];
#pragma unroll
  for (int i = 0; i < 9; i++) {
    s[i] = vadd(f[pair_q(i)], f[opp(pair_q(i))]);
    d[i] = vsub(f[pair_q(i)], f[opp(pair_q(i))]);
  }
  drho = vadd(f[0], vadd(vadd(vadd(vadd(s[0], s[1]), s[2]), vadd(vadd(s[3], s[4]), vadd(s[5], s[6]))),
                         vadd(s[7], s[8])));
  V jx = d[0], jy = d[1], jz = d[2];
#pragma unroll
  for (int i = 3; i < 9; i++) {
    if (cx(pair_q(i)) != 0) jx = vterm(cx(pair_q(i)), d[i], jx);
    if (cy(pair_q(i)) != 0) jy = vterm(cy(pair_q(i)), d[i], jy);
    if (cz(pair_q(i)) != 0) jz = vterm(cz(pair_q(i)), d[i], jz);
  }
  rho = vadd(O::splat(1.f), drho);
  const V inv = vrcp(rho);
  ux = vmul(vadd(jx, O::splat(hgx)), inv);
  uy = vmul(vadd(jy, O::splat(hgy)), inv);
  uz = vmul(vadd(jz, O::splat(hgz)), inv);
}

}  // namespace lbm
