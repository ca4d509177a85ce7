// Drag + lift and the corner weights of two faces at once, as the two lanes
// of packed f32x2 arithmetic (pair.cuh).  Every lane gives the bits of
// physics.cuh's face_total_force and face_corner_weight for its face
// (tests/test_gpu_math.py checks this).
#pragma once

#include "pair.cuh"

namespace fgb {

// Drag + lift of a face (D), and what its corner angles are made of: the
// cross product's magnitude y and the dot products x0, x1 of corners 0 and 1
// (springy_mesh.rs:629-654, 134-172), as face_total_force and
// face_corner_weight compute them.  nwind: the wind negated.  (Every dot
// product kept rounded, the drag and the lift apart, took 22 packed
// operations more per face: 53.2 us a step of the 1024 x 1024 cloth, 51.6
// with this.)
struct FacePair {
  V3x2 D;
  f2 y, x0, x1;
};
template <bool FAST>
__device__ __forceinline__ FacePair face_pair(V3x2 x0, V3x2 x1, V3x2 x2, V3x2 v0, V3x2 v1, V3x2 v2, V3x2 nwind,
                                              f2 neg_cd, f2 neg_lift, f2 one, uint32_t& far) {
  const V3x2 sum = add3(add3(v0, v1), v2);
  const f2 r3 = dup2(kRcp3);
  const V3x2 rv{fma2(sum.x, r3, nwind.x), fma2(sum.y, r3, nwind.y), fma2(sum.z, r3, nwind.z)};
  const V3x2 e1 = sub3(x1, x0), e2 = sub3(x2, x0), e3 = sub3(x1, x2);
  const V3x2 cr = cross3(e1, e2, one);
  f2 mag, inv;
  root_and_rcp<FAST>(fdot3(cr, cr), mag, inv, far);
  const V3x2 n = scale3(inv, cr), nr = cross3(n, rv, one);
  const f2 eff = mul2(mul2(mag, dup2(0.5f)), abs2(fdot3(n, rv)));
  const f2 m2 = root_or_zero<FAST>(fdot3(nr, nr), far);
  return {scale3(mul2(eff, fma2(neg_lift, m2, neg_cd)), rv), mag, fdot3(e2, e1), fdot3(e1, e3)};
}

// The shares of corners 0 and 1 of N faces: angle times RN(1/pi).  Corner
// 2's share is the rest, face_last_share.
template <bool FAST, int N>
__device__ __forceinline__ void face_shares(const FacePair (&f)[N], f2 one, f2 (&w0)[N], f2 (&w1)[N], uint32_t& far) {
  f2 y[2 * N], x[2 * N], a[2 * N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    y[2 * j] = y[2 * j + 1] = f[j].y;
    x[2 * j] = f[j].x0;
    x[2 * j + 1] = f[j].x1;
  }
  if (FAST) {
    if (!x_ok(x)) far = 0xffffffffu;
    angles_fast2<2 * N>(y, x, one, a);
  } else {
#pragma unroll 1
    for (int j = 0; j < 2 * N; ++j) {
      const float2 yj = upk(y[j]), xj = upk(x[j]);
      a[j] = pk(angle_pos(yj.x, xj.x), angle_pos(yj.y, xj.y));
    }
  }
  const f2 rpi = dup2(kRcpPi);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    w0[j] = mul2(a[2 * j], rpi);
    w1[j] = mul2(a[2 * j + 1], rpi);
  }
}

// (1 - w0) - w1, the products behind w0 and w1 kept rounded
__device__ __forceinline__ f2 face_last_share(f2 w0, f2 w1, f2 mone) {
  return fma2(w1, mone, fma2(w0, mone, dup2(1.0f)));
}

// The same with both lanes' results as scalars: D and w0, then w1 and w2 (the
// form the tests compare with the scalar functions).
__device__ __forceinline__ void face_terms2(V3x2 x0, V3x2 x1, V3x2 x2, V3x2 v0, V3x2 v1, V3x2 v2, V3x2 wind,
                                            float neg_cd, float neg_lift, float one_rt, float4& DwA, float2& wA,
                                            float4& DwB, float2& wB) {
  const f2 one = dup2(one_rt);
  const V3x2 nwind{neg2(wind.x), neg2(wind.y), neg2(wind.z)};
  uint32_t far = 0;
  FacePair f[1] = {face_pair<true>(x0, x1, x2, v0, v1, v2, nwind, dup2(neg_cd), dup2(neg_lift), one, far)};
  f2 w0[1], w1[1];
  face_shares<true>(f, one, w0, w1, far);
  if (far > kRootSpan) {
    f[0] = face_pair<false>(x0, x1, x2, v0, v1, v2, nwind, dup2(neg_cd), dup2(neg_lift), one, far);
    face_shares<false>(f, one, w0, w1, far);
  }
  const float2 dx = upk(f[0].D.x), dy = upk(f[0].D.y), dz = upk(f[0].D.z), u0 = upk(w0[0]), u1 = upk(w1[0]),
               u2 = upk(face_last_share(w0[0], w1[0], neg2(one)));
  DwA = make_float4(dx.x, dy.x, dz.x, u0.x);
  DwB = make_float4(dx.y, dy.y, dz.y, u0.y);
  wA = make_float2(u1.x, u2.x);
  wB = make_float2(u1.y, u2.y);
}

}  // namespace fgb
