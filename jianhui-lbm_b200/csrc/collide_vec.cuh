// FP32 macro step and MRT collision on one node or on two nodes at once.
//
// Blackwell's packed FP32 instructions (add / mul / fma .rn.f32x2) do two
// independent FP32 operations per issued instruction.  The step is bound by
// issue slots as soon as its bytes come from L2 (one node per thread: 665
// instructions per node through the table and 540 on its own slots, 69 % of the
// issue slots at 256^3, 75 % with 16-bit storage), so a
// thread works on two neighbouring nodes, one per half of each pair.
//
// The operator is mrt_collide_dev's (kernels_common.cuh).  Every operation
// here is one rounding that the source states (intrinsics or PTX, nothing
// left to contraction), so one node and two nodes give the same bits, in
// every kernel that includes this file.
#pragma once

#include <utility>

#include "kernels_common.cuh"

namespace lbm {

// f(0), ..., f(N - 1) with compile-time indices (integral constants): the
// coefficients below select their instructions with if constexpr, which an
// unrolled loop over constexpr functions was not reduced to.
template <typename F, int... I>
__device__ __forceinline__ void static_for_(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_(f, std::make_integer_sequence<int, N>{});
}

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

__device__ __forceinline__ float lane(float v, int) { return v; }
__device__ __forceinline__ float lane(F2 v, int j) { return j == 0 ? split_f2(v).x : split_f2(v).y; }

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
__device__ __forceinline__ F2 vneg(F2 a) { return vmul(a, make_f2(-1.f, -1.f)); }
// acc + C v; with FIRST, C v
template <int C, bool FIRST, typename V>
__device__ __forceinline__ V vterm(V v, V acc) {
  if constexpr (FIRST && C == 1)
    return v;
  else if constexpr (FIRST)
    return vmul(VecOf<V>::splat((float)C), v);
  else if constexpr (C == 1)
    return vadd(acc, v);
  else if constexpr (C == -1)
    return vsub(acc, v);
  else
    return vfma(VecOf<V>::splat((float)C), v, acc);
}
// Whether term i of row k (over the pairs) is its first; whether moment k is
// the first of its parity in the sum of pair i.
__host__ __device__ constexpr bool first_pair(int k, int i) {
  for (int j = 0; j < i; j++)
    if (mcoef(k, pair_q(j)) != 0) return false;
  return true;
}
__host__ __device__ constexpr bool first_moment(int k, int q) {
  for (int j = 1; j < k; j++)
    if (even_moment(j) == even_moment(k) && mcoef(j, q) != 0) return false;
  return true;
}

// Populations of one node, or of the nodes p and p + 1 of a row (p even).
// both: node p + 1 is the launch's; else its slot may be another kernel's (the
// face kernel's beside the step kernel) and is left alone, the first node's
// value standing in for it.
template <Store K>
__device__ __forceinline__ void load_row(const typename Traits<K>::T* p, float inv_scale, bool, float& v) {
  v = load_pop_rw<K>(p, inv_scale);
}
template <Store K>
__device__ __forceinline__ void load_row(const typename Traits<K>::T* p, float inv_scale, bool both, F2& v) {
  if (!both) {
    const float first = load_pop_rw<K>(p, inv_scale);
    v = make_f2(first, first);
  } else if constexpr (K == Store::F16) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(p));
    v = vmul(make_f2(a.x, a.y), make_f2(inv_scale, inv_scale));
  } else {
    v.v = *reinterpret_cast<const unsigned long long*>(p);
  }
}
template <Store K>
__device__ __forceinline__ void store_row(typename Traits<K>::T* p, float v, float scale, bool) {
  store_pop<K>(p, v, scale);
}
// both: the second node is stored too
template <Store K>
__device__ __forceinline__ void store_row(typename Traits<K>::T* p, F2 v, float scale, bool both) {
  const float2 a = split_f2(v);
  if (!both) {
    store_pop<K>(p, a.x, scale);
  } else if constexpr (K == Store::F16) {
    const float2 b = split_f2(vmul(v, make_f2(scale, scale)));
    *reinterpret_cast<__half2*>(p) = __floats2half2_rn(b.x, b.y);
  } else {
    *reinterpret_cast<unsigned long long*>(p) = v.v;
  }
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
  static_for<6>([&](auto i_) {
    constexpr int i = decltype(i_)::value + 3, q = pair_q(i);
    if constexpr (cx(q) != 0) jx = vterm<cx(q), false>(d[i], jx);
    if constexpr (cy(q) != 0) jy = vterm<cy(q), false>(d[i], jy);
    if constexpr (cz(q) != 0) jz = vterm<cz(q), false>(d[i], jz);
  });
  rho = vadd(O::splat(1.f), drho);
  const V inv = vrcp(rho);
  ux = vmul(vadd(jx, O::splat(hgx)), inv);
  uy = vmul(vadd(jy, O::splat(hgy)), inv);
  uz = vmul(vadd(jz, O::splat(hgz)), inv);
}

// 1 / |row K|^2
template <int K>
constexpr float kInvNorm = (float)(1.0 / mnorm(K));

// Scalars of the collision that are the same for every node.
struct CollideScalars {
  float gx, gy, gz;       // force
  float nsv, nso;         // -s_v, -s_o
  float hv, hv38;         // 1 - s_v/2, 38 (1 - s_v/2)
  float nhv11, nhv5;      // -11 (1 - s_v/2), -(1 - s_v/2)/2
  float nhoc;             // -(2/3) (1 - s_o/2)
};
__device__ __forceinline__ CollideScalars collide_scalars(float gx, float gy, float gz, float sv, float so) {
  CollideScalars c;
  c.gx = gx;
  c.gy = gy;
  c.gz = gz;
  c.nsv = -sv;
  c.nso = -so;
  c.hv = __fmaf_rn(-0.5f, sv, 1.f);
  c.hv38 = __fmul_rn(c.hv, 38.f);
  c.nhv11 = -__fmul_rn(c.hv, 11.f);
  c.nhv5 = -__fmul_rn(c.hv, 0.5f);
  c.nhoc = -__fmul_rn(__fmaf_rn(-0.5f, so, 1.f), (float)(2.0 / 3.0));
  return c;
}

// MRT collision with Guo forcing of the deviations f, in place; the operator
// and the closed forms of mrt_collide_dev.  POOL: the node pool's rounding, which
// rounds the force term's product of moment 2 and fuses the relaxation's, and
// fuses the first product of the cross terms of moments 13 to 15; the
// single-domain steps do both the other way round.  A solve in 16-bit storage
// stops by noise of this size, so each keeps its own bits.
template <typename V, bool POOL = false>
__device__ __forceinline__ void collide_vec(V (&f)[kQ], V drho, V rho, V ux, V uy, V uz, const CollideScalars& c) {
  using O = VecOf<V>;
  auto S = [](float x) { return O::splat(x); };
  V m[kQ];
  {
    V s[9], d[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
      s[i] = vadd(f[pair_q(i)], f[opp(pair_q(i))]);
      d[i] = vsub(f[pair_q(i)], f[opp(pair_q(i))]);
    }
    static_for<kQ>([&](auto k_) {
      constexpr int k = decltype(k_)::value;
      if constexpr (k == 1 || k == 2) {  // the rows with an f_0 term
        V acc = vterm<mcoef(k, 0), false>(f[0], vterm<mcoef(k, 1), true>(s[0], f[0]));
        static_for<8>([&](auto i_) {
          constexpr int i = decltype(i_)::value + 1;
          acc = vterm<mcoef(k, pair_q(i)), false>(s[i], acc);
        });
        m[k] = acc;
      } else if constexpr (k != 0 && k != 3 && k != 5 && k != 7) {  // not conserved
        V acc{};
        static_for<9>([&](auto i_) {
          constexpr int i = decltype(i_)::value, co = mcoef(k, pair_q(i));
          if constexpr (co != 0) acc = vterm<co, first_pair(k, i)>(even_moment(k) ? s[i] : d[i], acc);
        });
        m[k] = acc;
      }
    });
  }
  const V nux = vneg(ux), nuy = vneg(uy), nuz = vneg(uz);
  const V gx = S(c.gx), gy = S(c.gy), gz = S(c.gz);
  const V usq = vfma(uz, uz, vfma(ux, ux, vmul(uy, uy)));
  const V ug = vfma(uz, gz, vfma(ux, gx, vmul(uy, gy)));
  const V nsv = S(c.nsv), nso = S(c.nso), hv = S(c.hv);
  auto cross = [](V x, V y, V px, V py) {  // x py + y px
    if constexpr (POOL)
      return vfma(x, py, vmul(y, px));
    else
      return vfma(y, px, vmul(x, py));
  };
  // a_k = [ -S_k (m_k - m_eq,k) + (1 - S_k/2) (M G)_k ] / |row k|^2
  V a[kQ];
  a[1] = vmul(vfma(S(c.hv38), ug, vmul(nsv, vsub(m[1], vfma(vmul(S(19.f), rho), usq, vmul(S(-11.f), drho))))),
              S(kInvNorm<1>));
  const V x2 = vsub(m[2], vfma(S(3.f), drho, vmul(vmul(S(-5.5f), rho), usq)));
  if constexpr (POOL)
    a[2] = vmul(vfma(nsv, x2, vmul(S(c.nhv11), ug)), S(kInvNorm<2>));
  else
    a[2] = vmul(vfma(S(c.nhv11), ug, vmul(nsv, x2)), S(kInvNorm<2>));
  a[3] = S(__fmul_rn(c.gx, kInvNorm<3>));
  a[5] = S(__fmul_rn(c.gy, kInvNorm<5>));
  a[7] = S(__fmul_rn(c.gz, kInvNorm<7>));
  const V r23 = vmul(S((float)(2.0 / 3.0)), rho);
  a[4] = vmul(vfma(nso, vfma(r23, ux, m[4]), S(__fmul_rn(c.nhoc, c.gx))), S(kInvNorm<4>));
  a[6] = vmul(vfma(nso, vfma(r23, uy, m[6]), S(__fmul_rn(c.nhoc, c.gy))), S(kInvNorm<6>));
  a[8] = vmul(vfma(nso, vfma(r23, uz, m[8]), S(__fmul_rn(c.nhoc, c.gz))), S(kInvNorm<8>));
  const V ux2 = vadd(ux, ux);
  const V p9 = vmul(rho, vfma(nuz, uz, vfma(ux2, ux, vmul(nuy, uy))));
  const V f9h = vfma(nuz, gz, vfma(ux2, gx, vmul(nuy, gy)));
  const V f9 = vadd(f9h, f9h);
  a[9] = vmul(vfma(hv, f9, vmul(nsv, vsub(m[9], p9))), S(kInvNorm<9>));
  a[10] = vmul(vfma(nsv, vfma(S(0.5f), p9, m[10]), vmul(S(c.nhv5), f9)), S(kInvNorm<10>));
  const V p11 = vmul(rho, vfma(nuz, uz, vmul(uy, uy)));
  const V f11h = vfma(nuz, gz, vmul(uy, gy));
  const V f11 = vadd(f11h, f11h);
  const V x11 = vfma(hv, f11, vmul(nsv, vsub(m[11], p11)));  // a_11 |row 11|^2: its product is part of the sums below
  a[12] = vmul(vfma(nsv, vfma(S(0.5f), p11, m[12]), vmul(S(c.nhv5), f11)), S(kInvNorm<12>));
  const V nrx = vmul(rho, nux), nry = vmul(rho, nuy);
  a[13] = vmul(vfma(hv, cross(ux, uy, gx, gy), vmul(nsv, vfma(nrx, uy, m[13]))), S(kInvNorm<13>));
  a[14] = vmul(vfma(hv, cross(uy, uz, gy, gz), vmul(nsv, vfma(nry, uz, m[14]))), S(kInvNorm<14>));
  a[15] = vmul(vfma(hv, cross(ux, uz, gx, gz), vmul(nsv, vfma(nrx, uz, m[15]))), S(kInvNorm<15>));
  a[16] = vmul(vmul(nso, m[16]), S(kInvNorm<16>));
  a[17] = vmul(vmul(nso, m[17]), S(kInvNorm<17>));
  a[18] = vmul(vmul(nso, m[18]), S(kInvNorm<18>));

  // f*_q = f_q + sum_k M_kq a_k, split into even/odd parts per opposite pair
  f[0] = vadd(f[0], vterm<mcoef(2, 0), false>(a[2], vterm<mcoef(1, 0), true>(a[1], a[1])));
  static_for<9>([&](auto i_) {
    constexpr int q = pair_q(decltype(i_)::value);
    V ev{}, od{};
    static_for<kQ>([&](auto k_) {
      constexpr int k = decltype(k_)::value, co = mcoef(k, q);
      constexpr bool first = first_moment(k, q);
      if constexpr (k == 0 || co == 0) {
      } else if constexpr (k == 11) {
        ev = vfma(x11, S(co * kInvNorm<11>), ev);
      } else if constexpr (even_moment(k)) {
        ev = vterm<co, first>(a[k], ev);
      } else if constexpr ((k == 5 || k == 7) && !first) {
        od = vfma(k == 5 ? gy : gz, S(co * kInvNorm<k>), od);
      } else {
        od = vterm<co, first>(a[k], od);
      }
    });
    f[q] = vadd(f[q], vadd(ev, od));
    f[opp(q)] = vadd(f[opp(q)], vsub(ev, od));
  });
}

}  // namespace lbm
