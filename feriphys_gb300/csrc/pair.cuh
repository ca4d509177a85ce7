// Two vertices (or two faces) at a time: 3-vectors whose components are the
// two lanes of packed f32x2 registers (angle.cuh: f2).  Every lane rounds as
// the scalar instruction does, so a packed sequence gives the bits of the
// scalar one; a sum with a product operand is an fma with the run-time unit
// multiplier `one` (angle.cuh says why).
//
// The packed operations run at the scalar ones' flop rate on this part
// (measured: 115 lane operations per clock and SM for add, mul and fma, packed
// or not), so what they save is issue slots: one for two lanes.
#pragma once

#include "angle.cuh"
#include "devmath.cuh"
#include "fastdiv.cuh"

namespace fgb {

struct V3x2 {
  f2 x, y, z;
};
__device__ __forceinline__ V3x2 pk3(V3<float> a, V3<float> b) { return {pk(a.x, b.x), pk(a.y, b.y), pk(a.z, b.z)}; }
__device__ __forceinline__ V3x2 add3(V3x2 a, V3x2 b) { return {add2(a.x, b.x), add2(a.y, b.y), add2(a.z, b.z)}; }
__device__ __forceinline__ V3x2 sub3(V3x2 a, V3x2 b) { return {sub2(a.x, b.x), sub2(a.y, b.y), sub2(a.z, b.z)}; }
// s * v (operator*(T, V3): s * v.x, ...) and v * s: the same products
__device__ __forceinline__ V3x2 scale3(f2 s, V3x2 v) { return {mul2(s, v.x), mul2(s, v.y), mul2(s, v.z)}; }
// F + p for a product p kept rounded (one = 1), F - p with one = -1
__device__ __forceinline__ V3x2 add_p3(V3x2 F, V3x2 p, f2 one) {
  return {fma2(p.x, one, F.x), fma2(p.y, one, F.y), fma2(p.z, one, F.z)};
}
// (x x' + y y') + z z', every sum of products an fma with the unit `one`
// (angle.cuh: add_p2), so each product and each sum is rounded once
__device__ __forceinline__ f2 dot3(V3x2 a, V3x2 b, f2 one) {
  return add_p2(mul2(a.z, b.z), add_p2(mul2(a.x, b.x), mul2(a.y, b.y), one), one);
}
// devmath.cuh's fdot and cross in both lanes
__device__ __forceinline__ f2 fdot3(V3x2 a, V3x2 b) { return fma2(a.z, b.z, fma2(a.y, b.y, mul2(a.x, b.x))); }
__device__ __forceinline__ V3x2 cross3(V3x2 a, V3x2 b, f2 one) {
  return {rsub_p2(mul2(a.z, b.y), mul2(a.y, b.z), one), rsub_p2(mul2(a.x, b.z), mul2(a.z, b.x), one),
          rsub_p2(mul2(a.y, b.x), mul2(a.x, b.y), one)};
}

// lane 0 of a where l0, lane 1 of a where l1, the rest of b
__device__ __forceinline__ f2 lanes(bool l0, bool l1, f2 a, f2 b) {
  const float2 u = upk(a), v = upk(b);
  return pk(l0 ? u.x : v.x, l1 ? u.y : v.y);
}
__device__ __forceinline__ V3x2 lanes3(bool l0, bool l1, V3x2 a, V3x2 b) {
  return {lanes(l0, l1, a.x, b.x), lanes(l0, l1, a.y, b.y), lanes(l0, l1, a.z, b.z)};
}
__device__ __forceinline__ V3<float> lane3(V3x2 v, int l) {
  const float2 x = upk(v.x), y = upk(v.y), z = upk(v.z);
  return l ? V3<float>{x.y, y.y, z.y} : V3<float>{x.x, y.x, z.x};
}

// rcp_of_root (fastdiv.cuh) in both lanes: 1 / magnitude with the bits of 1/x
__device__ __forceinline__ f2 rcp_of_root2(f2 x) {
  const float2 u = upk(x);
  const f2 y0 = pk(rcp_approx_ftz(u.x), rcp_approx_ftz(u.y));
  const f2 e = fma2(neg2(x), y0, dup2(1.0f));
  const float2 y1 = upk(fma2(y0, e, y0)), z = upk(y0);
  return pk(y1.x != y1.x ? z.x : y1.x, y1.y != y1.y ? z.y : y1.y);
}

// The square root of both lanes, exactly the IEEE one, for 2^-100 <= x <=
// 2^100 (root_range): g = x y and h = y / 2 from the hardware's approximate
// y = 1/sqrt(x), then one step of Newton's iteration for the root of g^2 = x,
// g + (x - g^2) / (2 sqrt(x)) = g + h (x - g g), with the residual and the sum
// fused.  Before its last rounding the result is off by about 2^-44 relative;
// that it then rounds to sqrtf(x) for every float of that range is established
// by exhaustion (tests/test_gpu_pair.py).  Four packed operations and two
// approximations for two roots, and no branch.
constexpr uint32_t kRootLo = 0x0d800000u, kRootSpan = 0x71800000u - 0x0d800000u;  // 2^-100 .. 2^100
__device__ __forceinline__ float rsqrt_approx_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ f2 root_fast2(f2 x) {
  const float2 u = upk(x);
  const f2 y = pk(rsqrt_approx_ftz(u.x), rsqrt_approx_ftz(u.y));
  const f2 g = mul2(x, y), h = mul2(y, dup2(0.5f));
  return fma2(fma2(mul2(g, dup2(-1.0f)), g, x), h, g);
}
// 1/s for a root s of root_fast2's range, the bits of 1/s (fastdiv.cuh: rcp_rn_fast)
__device__ __forceinline__ f2 rcp_root_fast2(f2 s) {
  const float2 u = upk(s);
  const f2 y = pk(rcp_approx_ftz(u.x), rcp_approx_ftz(u.y));
  const f2 e = fma2(mul2(s, dup2(-1.0f)), y, dup2(1.0f));
  return fma2(y, e, y);
}
// the larger of `far` and how far a lane of x lies above 2^-100 (a value
// below it, negative or NaN wraps to a huge one): in range while the result
// is at most kRootSpan
__device__ __forceinline__ uint32_t root_range(f2 x, uint32_t far) {
  return max(far, max(uint32_t(x) - kRootLo, uint32_t(x >> 32) - kRootLo));
}

// Root and reciprocal root of x = |v|^2 as a thread's terms need them: FAST
// takes the sequences above and records in `far` whether every operand was in
// their range; the caller, once at its end, redoes its terms with FAST =
// false when one was not (a degenerate strut or face, extreme or non-finite
// numbers).  One check instead of one per root keeps the terms one straight
// run of instructions that the compiler can interleave.
template <bool FAST>
__device__ __forceinline__ void root_and_rcp(f2 x, f2& mag, f2& inv, uint32_t& far) {
  if (FAST) {
    far = root_range(x, far);
    mag = root_fast2(x);
    inv = rcp_root_fast2(mag);
  } else {
    const float2 u = upk(x);
    mag = pk(sqrtf(u.x), sqrtf(u.y));
    inv = rcp_of_root2(mag);
  }
}
// The root alone; zero lanes stay on the fast path (the approximation is
// taken of 2^-100 instead, and the root of a zero comes out as zero).
template <bool FAST>
__device__ __forceinline__ f2 root_or_zero(f2 x, uint32_t& far) {
  const float2 u = upk(x);
  if (!FAST) return pk(sqrtf(u.x), sqrtf(u.y));
  const uint32_t b0 = __float_as_uint(u.x), b1 = __float_as_uint(u.y);
  far = max(far, max((b0 == 0u ? kRootLo : b0) - kRootLo, (b1 == 0u ? kRootLo : b1) - kRootLo));
  const float lo = __uint_as_float(kRootLo);
  const f2 y = pk(rsqrt_approx_ftz(fmaxf(u.x, lo)), rsqrt_approx_ftz(fmaxf(u.y, lo)));
  const f2 g = mul2(x, y), h = mul2(y, dup2(0.5f));
  return fma2(fma2(mul2(g, dup2(-1.0f)), g, x), h, g);
}

}  // namespace fgb
