// Grid-stencil step for meshes with Cloth::new's topology (cloth.rs:20-113).
//
// The neighbourhood of every vertex is implicit in (row, col): no index
// lists are read.  Strut constants live in per-row records of 32 columns
// (grid_order.h: param_rec).  The force terms are summed in the exact
// order of the reference's scatter loops (strut ids ascending, then face ids
// ascending -- checked on the host against the real ids before this kernel is
// chosen), so the result is bit-identical to the general gather.
#include <type_traits>

#include "chain_launch.cuh"
#include "cp_async.cuh"
#include "face_pair.cuh"
#include "fastdiv.cuh"
#include "grid_order.h"
#include "kernels.h"
#include "per_device.h"
#include "physics.cuh"

namespace fgb {

namespace {

using namespace grid;

__device__ __forceinline__ void strut_ends(int kind, int owner, int C, int& a, int& b) {
  switch (kind) {
    case KH: a = owner; b = owner + 1; break;
    case KV: a = owner; b = owner + C; break;
    case KS: a = owner + 1; b = owner + C; break;
    case KBH: a = owner; b = owner + 2; break;
    default: a = owner; b = owner + 2 * C; break;
  }
}

__global__ void __launch_bounds__(256) k_step_grid_v1(int R, int C, const float* __restrict__ params,
                                                      const float4* __restrict__ pos,
                                                      const float4* __restrict__ vel,
                                                      const float4* __restrict__ force_in,
                                                      float4* __restrict__ pos_out, float4* __restrict__ vel_out,
                                                      StepConsts c) {
  const int n = R * C;
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const float4 P4 = pos[v], V4 = vel[v];
  if (V4.w != 0.0f) {
    pos_out[v] = P4;
    vel_out[v] = V4;
    return;
  }
  const int r = v / C, cc = v - r * C;
  const V3<float> P = xyz<float>(P4), V = xyz<float>(V4);
  V3<float> F{c.force0[0], c.force0[1], c.force0[2]};
  if (force_in) F = xyz<float>(force_in[v]) + F;
  for (int j = 0; j < N_SLOTS; ++j) {
    const SlotDesc d = slot_desc(slot_at(j, r, cc, R, C));
    const int ro = r + d.dr, co = cc + d.dc;
    if (!owned_exists(d.kind, ro, co, R, C)) continue;
    const int owner = ro * C + co;
    int a, b;
    strut_ends(d.kind, owner, C, a, b);
    const float k = params[param_at(d.kind, 0, ro, co, C)];
    const float cdmp = params[param_at(d.kind, 1, ro, co, C)];
    const float L = params[param_at(d.kind, 2, ro, co, C)];
    V3<float> sf, df;
    if (d.role == 0) {
      strut_forces<float>(P, xyz<float>(pos[b]), V, xyz<float>(vel[b]), k, cdmp, L, sf, df);
      F = F + sf;
      F = F + df;
    } else {
      strut_forces<float>(xyz<float>(pos[a]), P, xyz<float>(vel[a]), V, k, cdmp, L, sf, df);
      F = F + (-1.0f * sf);
      F = F + (-1.0f * df);
    }
  }
  const V3<float> wind{c.wind[0], c.wind[1], c.wind[2]};
  for (int s = 0; s < N_FACE_SLOTS; ++s) {
    const FaceDesc fd = face_desc(s);
    const int qr = r + fd.dr, qc = cc + fd.dc;
    if (!quad_exists(qr, qc, R, C)) continue;
    const int q = qr * C + qc;
    int i0, i1, i2;
    if (fd.is_b) { i0 = q + 1; i1 = q + C + 1; i2 = q + C; }
    else { i0 = q + 1; i1 = q + C; i2 = q; }
    const V3<float> x0 = xyz<float>(pos[i0]), x1 = xyz<float>(pos[i1]), x2 = xyz<float>(pos[i2]);
    const V3<float> v0 = xyz<float>(vel[i0]), v1 = xyz<float>(vel[i1]), v2 = xyz<float>(vel[i2]);
    const V3<float> total = face_total_force<float>(x0, x1, x2, v0, v1, v2, wind, c.neg_drag, c.neg_lift);
    F = F + face_corner_weight<float>(x0, x1, x2, fd.corner) * total;
  }
  V3<float> np, nv, nF;
  const float m = P4.w;
  integrate_point<float>(c.integration, c.dt, P, V, F, m, np, nv, nF);
  collide_point<float>(static_cast<const ObsFace*>(c.obstacle_faces), c.n_obstacle_faces, P, V, F, m, np, nv, c);
  pos_out[v] = make4<float>(np, m);
  vel_out[v] = make4<float>(nv, V4.w);
  const bool bad = !(finite3(np) && finite3(nv));
  if (__any_sync(__activemask(), bad) && bad && c.flags) atomicOr(c.flags, 1u);
}


// ---------------------------------------------------------------------------
// Tiled kernel.  A CTA owns a tile of 32 x TH vertices and works on vertex
// pairs: columns c and c + 16 of a tile row are the two lanes of packed f32x2
// arithmetic (pair.cuh), so one instruction does a strut, a face or a sum for
// two vertices.  The step is bound by the instructions it issues (the
// reference's f32 arithmetic, operation by operation), not by memory or by
// the arithmetic units, and the packed form needs about half of them: the
// lanes are paired once, while the state is staged, and never repacked.
// Measured against one vertex per thread (faces packed only): 1024 x 1024
// cloth over a plane 57.4 -> 53.8 us a step (43.9 -> 27.7 million warp
// instructions), 256 cloths of 16..128 vertices a side 133.6 -> 98.7 us (48.1
// and 93.5 now, with the face terms fused and launches chained).
//
// The tile and a halo of two vertices (binding struts reach that far) are
// staged in shared memory as pairs; every strut and face touching the tile is
// computed once, and each thread then gathers its two vertices' terms in the
// reference's order.  In the halo columns left of the tile, lane 1 repeats a
// column of lane 0 (the packed instruction is issued for lane 0 anyway).

constexpr int kTileW = 32;          // tiles are 32 columns wide
constexpr int kPairW = kTileW / 2;  // pair columns of a tile row
constexpr int kHalo = 32;           // helper threads: one warp computes the tile's halo struts and faces

template <int TH>
struct Tile {
  static constexpr int NMAIN = kPairW * TH, NT = NMAIN + kHalo;
  // row strides: odd multiples of 16 bytes apart, so that a column of slots (the
  // helper's reads and writes left of the tile) meets no bank twice
  static constexpr int EC = kPairW + 4, EW = EC + 1, EH = TH + 4, NE = EW * EH;  // staged pairs, origin (-2, -2)
  // strut slots by owner pair, all kinds with the row stride OW (columns -2..15);
  // rows: KH and KBH 0.., KV and KS -1.., KBV -2..
  static constexpr int OW = kPairW + 3;
  static constexpr int NS = OW * (5 * TH + 4);
  static constexpr int QW = kPairW + 1, NQ = QW * (TH + 1);  // quads, origin (-1, -1)
  // staged pair: position and velocity 48 B; strut: unit vector, s1, s2 40 B;
  // quad: two faces' force and two shares each, 80 B
  static constexpr size_t SMEM = size_t(NE) * 48 + size_t(NS) * 40 + size_t(NQ) * 80;
  // resident CTAs per SM the launch bounds ask for (shared memory 33, 58, 83
  // KB).  Four CTAs of 8 rows would fit in 57 KB and 96 registers: 59.4 us a
  // step of the 1024 x 1024 cloth against 55.4 with three (of an earlier
  // form), the rest of the L1 then being too small for the loads in flight.
  static constexpr int MIN_CTAS = TH <= 4 ? 5 : (TH <= 8 ? 3 : 2);
  // slot of the strut of `kind` owned by tile-relative pair (r, pc)
  static __device__ __forceinline__ int slot(int kind, int r, int pc) {
    const int first = kind == KH ? 0 : (kind == KV ? TH : (kind == KS ? 2 * TH + 1 : (kind == KBH ? 3 * TH + 2 : 4 * TH + 2)));
    const int up = kind == KH || kind == KBH ? 0 : (kind == KBV ? 2 : 1);
    return (first + up + r) * OW + pc + 2;
  }
  static __device__ __forceinline__ int staged(int r, int pc) { return (r + 2) * EW + pc + 2; }
  static __device__ __forceinline__ int quad(int r, int pc) { return (r + 1) * QW + pc + 1; }
};

// 16 bytes of shared memory as two f32x2
struct __align__(16) F2x2 {
  f2 a, b;
};

// The staged state: {x, y}, {z, vx}, {vy, vz} of a pair.
template <int TH>
struct StagedState {
  F2x2* xy;
  F2x2* zu;
  F2x2* vw;
  __device__ __forceinline__ explicit StagedState(unsigned char* smem) {
    xy = reinterpret_cast<F2x2*>(smem);
    zu = xy + Tile<TH>::NE;
    vw = zu + Tile<TH>::NE;
  }
  __device__ __forceinline__ void get(int i, V3x2& p, V3x2& v) const {
    const F2x2 a = xy[i], b = zu[i], c = vw[i];
    p = {a.a, a.b, b.a};
    v = {b.b, c.a, c.b};
  }
  __device__ __forceinline__ void put(int i, float4 p0, float4 p1, float4 v0, float4 v1) const {
    xy[i] = {pk(p0.x, p1.x), pk(p0.y, p1.y)};
    zu[i] = {pk(p0.z, p1.z), pk(v0.x, v1.x)};
    vw[i] = {pk(v0.y, v1.y), pk(v0.z, v1.z)};
  }
};

// Struts of the compact form: unit vector u and the spring and damper scalars
// s1 = k (|d| - L), s2 = c (dv . u); the forces are s1 u and s2 u, which a
// gathering thread forms itself (the same products, so the same bits).
template <int TH>
struct StrutTerms {
  F2x2* uxy;
  F2x2* uz_s1;
  f2* s2;
  __device__ __forceinline__ explicit StrutTerms(unsigned char* smem) {
    uxy = reinterpret_cast<F2x2*>(smem + size_t(Tile<TH>::NE) * 48);
    uz_s1 = uxy + Tile<TH>::NS;
    s2 = reinterpret_cast<f2*>(uz_s1 + Tile<TH>::NS);
  }
};

// Faces A = (i+1, i+C, i) and B = (i+1, i+C+1, i+C) of a quad with origin i:
// force D, shares w0 and w1 (the third is the rest of the unit share).
template <int TH>
struct QuadTerms {
  F2x2* dxy;  // face B's entries NQ after face A's, here and below
  f2* dz;
  f2* w0;
  f2* w1;
  __device__ __forceinline__ explicit QuadTerms(unsigned char* smem) {
    dxy = reinterpret_cast<F2x2*>(smem + size_t(Tile<TH>::NE) * 48 + size_t(Tile<TH>::NS) * 40);
    dz = reinterpret_cast<f2*>(dxy + 2 * Tile<TH>::NQ);
    w0 = dz + 2 * Tile<TH>::NQ;
    w1 = w0 + 2 * Tile<TH>::NQ;
  }
};

// A vertex pair's staged state.
struct PairState {
  V3x2 p, v;
};
template <int TH>
__device__ __forceinline__ PairState pair_at(const StagedState<TH>& state, int i) {
  PairState a;
  state.get(i, a.p, a.v);
  return a;
}

// A position whose components' magnitudes sum to a finite number and a velocity
// and wind whose sum to less than 2^61; false for a NaN.  (One test for the three;
// apart they took 0.15 us more a step of a 1024 x 1024 cloth.)
__device__ __forceinline__ float length1(V3<float> v) { return fabsf(v.x) + fabsf(v.y) + fabsf(v.z); }
__device__ __forceinline__ bool mild(V3<float> p, V3<float> v, float wind1) {
  return isfinite(__fmaf_rn(length1(v) + wind1, 0x1p67f, length1(p)));
}

// Where a boundary tile's staged points outside the cloth are put: far away, at
// rest and no two in the same place.  A strut that does not exist then has
// some finite length, its constants are zero, and so are its forces; a quad
// that does not exist has finite terms and a zero drag and lift coefficient.
// Adding a zero of either sign leaves a force sum as it is (no sum is ever -0:
// it starts from 0 + gravity), so the terms and their sums need no look at
// what exists, and boundary and interior tiles run the same instructions.  A
// boundary tile with a staged state that is not `mild` takes the slow form of
// its terms, which does look: there a zero constant does not always make a zero
// force, since a term may overflow before it is multiplied by it.  (Lengths and
// cross products are 2^50 at most, root_range; times a mild relative velocity
// they stay below 2^113.)
// (With a second, checked form of the whole tile beside the unchecked one the
// two did not fit the instruction cache: 256 cloths of 16..128 vertices a
// side, which mix both, took 115 instead of 105 us a step.)
__device__ __forceinline__ float4 outside_pos(int sr, int sc) {
  return make_float4(65536.0f + 1024.0f * float(sc), 1024.0f * float(sr), 0.0f, 1.0f);
}

// The terms of one strut in both lanes, from staged pairs a to b with
// constants k, c, L.  FAST = false (root_and_rcp) also covers what outside_pos
// does not, points that coincide and non-finite states: struts that do not
// exist (bits 0, 1 of `absent`) get zeros whatever came out.
template <bool FAST, int TH>
__device__ __forceinline__ void strut_pair(const StrutTerms<TH>& out, int o, const PairState& a, const PairState& b,
                                           f2 k, f2 c, f2 L, unsigned absent, f2 one, uint32_t& far) {
  const V3x2 d = sub3(b.p, a.p);
  f2 mag, inv;
  root_and_rcp<FAST>(dot3(d, d, one), mag, inv, far);
  V3x2 u = scale3(inv, d);
  f2 s1 = mul2(k, sub2(mag, L)), s2 = mul2(c, dot3(sub3(b.v, a.v), u, one));
  if (!FAST) {
    u = lanes3(absent & 1u, absent & 2u, V3x2{0, 0, 0}, u);
    s1 = lanes(absent & 1u, absent & 2u, 0, s1);
    s2 = lanes(absent & 1u, absent & 2u, 0, s2);
  }
  out.uxy[o] = {u.x, u.y};
  out.uz_s1[o] = {u.z, s1};
  out.s2[o] = s2;
}

// Both faces of a pair of quads with the corners 00, 01, 10, 11.  neg_cd and
// neg_lift are zero in the lanes whose quad does not exist; with FAST = false
// those lanes (has0, has1 false) store a zero force whatever came out.
// Returns root_and_rcp's range verdict.
template <bool FAST, int TH>
__device__ __forceinline__ uint32_t quad_pair(const QuadTerms<TH>& out, int q, const PairState& s00,
                                              const PairState& s01, const PairState& s10, const PairState& s11,
                                              f2 neg_cd, f2 neg_lift, bool has0, bool has1, V3x2 nwind, f2 one) {
  constexpr int NQ = Tile<TH>::NQ;
  uint32_t far = 0;
  // face A = (01, 10, 00), face B = (01, 11, 10)
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const PairState &s1 = k ? s11 : s10, &s2 = k ? s10 : s00;
    const FacePair f[1] = {
        face_pair<FAST>(s01.p, s1.p, s2.p, s01.v, s1.v, s2.v, nwind, neg_cd, neg_lift, one, far)};
    f2 w0[1], w1[1];
    face_shares<FAST>(f, one, w0, w1, far);
    V3x2 D = f[0].D;
    if (!FAST) {
      D = lanes3(has0, has1, D, V3x2{0, 0, 0});
      w0[0] = lanes(has0, has1, w0[0], 0);
      w1[0] = lanes(has0, has1, w1[0], 0);
    }
    out.dxy[q + k * NQ] = {D.x, D.y};
    out.dz[q + k * NQ] = D.z;
    out.w0[q + k * NQ] = w0[0];
    out.w1[q + k * NQ] = w1[0];
  }
  return far;
}

// F / m of both lanes, the bits of physics.cuh's div_mass (Markstein's
// division by a known reciprocal, fastdiv.cuh).  The fast path takes masses
// in [2^-30, 2^30] and force components that are +0 or of magnitude
// [2^-70, 2^60]: then every quotient lies in [2^-100, 2^90], inside the
// range the theorem needs, without a look at the quotient itself (a force
// sum is never -0, see strut_pairs).
static __device__ __noinline__ V3x2 div_cold2(V3x2 F, f2 m) {
  const float2 mm = upk(m);
  return pk3(lane3(F, 0) / mm.x, lane3(F, 1) / mm.y);
}
__device__ __forceinline__ V3x2 div_mass2(V3x2 F, f2 m) {
  constexpr uint32_t lo = 0x1c800000u, span = 0x5d800000u - 0x1c800000u;   // 2^-70 .. 2^60
  constexpr uint32_t mlo = 0x30800000u, mspan = 0x4e800000u - 0x30800000u;  // 2^-30 .. 2^30, positive
  auto lane_ok = [&](uint32_t b) { return b == 0u || (b & 0x7fffffffu) - lo <= span; };
  auto ok2 = [&](f2 a) { return lane_ok(uint32_t(a)) && lane_ok(uint32_t(a >> 32)); };
  if (uint32_t(m) - mlo <= mspan && uint32_t(m >> 32) - mlo <= mspan && ok2(F.x) && ok2(F.y) && ok2(F.z)) {
    const float2 mm = upk(m);
    const f2 y = pk(rcp_rn_fast(mm.x), rcp_rn_fast(mm.y)), nm = mul2(m, dup2(-1.0f));
    auto div = [&](f2 a) {
      const f2 q = mul2(a, y);
      return fma2(fma2(nm, q, a), y, q);
    };
    return {div(F.x), div(F.y), div(F.z)};
  }
  return div_cold2(F, m);
}

// physics.cuh's integrate_point for both lanes, the same operations.  In the
// reference's "RK4" (state.rs:86-106) every stage divides the same F by the
// same m (F + 0 h = F for a sum that is never -0, m + 0 h = m), so its four
// accelerations are one.
__device__ __forceinline__ void integrate_pair(const StepConsts& c, V3x2 p, V3x2 v, V3x2 F, f2 m, f2 one, V3x2& np,
                                               V3x2& nv) {
  const V3x2 a = div_mass2(F, m);
  const f2 h = dup2(c.dt);
  if (c.integration == 0) {
    np = add_p3(p, scale3(h, v), one);
    nv = add_p3(v, scale3(h, a), one);
  } else {
    const f2 hh = dup2(c.dt * 0.5f), h6 = dup2(c.dt / 6.0f), h3 = dup2(c.dt / 3.0f);
    const V3x2 v2 = add_p3(v, scale3(hh, a), one), v4 = add_p3(v, scale3(h, a), one);
    const V3x2 t3 = scale3(h3, v2), a3 = scale3(h3, a), a6 = scale3(h6, a);
    const V3x2 sv = add_p3(add_p3(add_p3(t3, scale3(h6, v), one), t3, one), scale3(h6, v4), one);
    const V3x2 sa = add_p3(add_p3(add_p3(a3, a6, one), a3, one), a6, one);
    np = add3(p, sv);
    nv = add3(v, sa);
  }
}

// The whole search for one lane, out of line: moves the cells cannot answer.
static __device__ __noinline__ void collide_lane(V3<float> P, V3<float> V, V3<float> F, float m, V3<float>& np,
                                                 V3<float>& nv, const StepConsts& c) {
  collide_point<float>(static_cast<const ObsFace*>(c.obstacle_faces), c.n_obstacle_faces, P, V, F, m, np, nv, c);
}

// Collision query and response of a pair's moves from P to np (collide_point
// for both lanes, the same hits and the same arithmetic).  finite: 0 in a lane
// whose ends are finite; live0, live1: lanes that collide at all.
//
// Each move's box (query_slack's margin and a little more: a larger box only
// adds candidates) is tested against the few boxes in the launch constants;
// most pairs meet none and are done.  For a box it meets, the move's cell
// lists every face of that obstacle the move can hit, provided the cell,
// grown by its slack, holds the box (whichever cell rounding picks); the two
// lanes' cells, lists and faces are fetched together, so that a pair in
// contact pays the chain of loads once (157 x 211 cloth settling on a floor:
// 12.9 us a step with one lane's search after the other's, 10.7 with this).
// What the cells cannot answer -- a box that does not fit its cell, an
// obstacle without cells, a non-finite end -- goes through the whole search.
__device__ __forceinline__ void collide_pair(const StepConsts& c, V3x2 P, V3x2 V, V3x2 F, float m0, float m1,
                                             float2 finite, bool live0, bool live1, V3x2& np, V3x2& nv) {
  if (c.n_obstacle_faces == 0) return;
  bool full[2] = {live0 && (!c.accel.enabled || finite.x != 0.0f), live1 && (!c.accel.enabled || finite.y != 0.0f)};
  const bool live[2] = {live0 && !full[0], live1 && !full[1]};
  float lo[2][3], hi[2][3];
  {
    const f2 o3[3] = {P.x, P.y, P.z}, n3[3] = {np.x, np.y, np.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float2 o = upk(o3[d]), n = upk(n3[d]);
      const f2 ns = fma2(pk(fmaxf(fabsf(o.x), fabsf(n.x)), fmaxf(fabsf(o.y), fabsf(n.y))), dup2(-3.0002e-5f),
                         dup2(-2e-30f));
      const float2 l = upk(add2(pk(fminf(o.x, n.x), fminf(o.y, n.y)), ns));
      const float2 h = upk(sub2(pk(fmaxf(o.x, n.x), fmaxf(o.y, n.y)), ns));
      lo[0][d] = l.x;
      lo[1][d] = l.y;
      hi[0][d] = h.x;
      hi[1][d] = h.y;
    }
  }
  unsigned met = 0;  // bit 2 k + l: lane l meets box k
#pragma unroll
  for (int k = 0; k < kObsBoxes; ++k) {
    if (k >= c.accel.n_boxes) break;
    const ObsBox& b = c.accel.box[k];
#pragma unroll
    for (int l = 0; l < 2; ++l)
      if (live[l] & (hi[l][0] >= b.lo[0]) & (lo[l][0] <= b.hi[0]) & (hi[l][1] >= b.lo[1]) & (lo[l][1] <= b.hi[1]) &
          (hi[l][2] >= b.lo[2]) & (lo[l][2] <= b.hi[2]))
        met |= 1u << (2 * k + l);
  }
  if (!(met != 0 || full[0] || full[1])) return;
  const ObsFace* faces = static_cast<const ObsFace*>(c.obstacle_faces);
  const float dtd = c.dt_duration;
  int hit[2] = {-1, -1};
  float d_old[2] = {0.0f, 0.0f}, d_new[2] = {0.0f, 0.0f};
#pragma unroll 1
  for (int k = 0; (met >> (2 * k)) != 0; ++k) {
    const ObsBox& b = c.accel.box[k];
    int at[2] = {0, 0}, end[2] = {0, 0};  // the lanes' candidates, ascending
#pragma unroll
    for (int l = 0; l < 2; ++l) {
      if (((met >> (2 * k + l)) & 1u) == 0 || hit[l] >= 0 || full[l]) continue;
      int idx[3];
      bool fits = b.n[0] > 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int i = max(min(int(floorf((0.5f * (lo[l][d] + hi[l][d]) - b.lo[d]) * b.inv[d])), b.n[d] - 1), 0);
        fits = fits & (lo[l][d] >= b.lo[d] + float(i) * b.cell[d] - b.slack) &
               (hi[l][d] <= b.lo[d] + float(i + 1) * b.cell[d] + b.slack);
        idx[d] = i;
      }
      full[l] = !fits;
      if (fits) {
        const int* off = c.accel.cell_off + b.off_base + (idx[0] * b.n[1] + idx[1]) * b.n[2] + idx[2];
        at[l] = __ldg(off);
        end[l] = __ldg(off + 1);
      }
    }
#pragma unroll 1
    while (at[0] < end[0] || at[1] < end[1]) {
      int f[2];
#pragma unroll
      for (int l = 0; l < 2; ++l) f[l] = at[l] < end[l] ? __ldg(c.accel.cell_faces + at[l]++) : -1;
#pragma unroll
      for (int l = 0; l < 2; ++l)
        if (f[l] >= 0 && face_hit<float>(faces + f[l], lane3(P, l), lane3(np, l), dtd, d_old[l], d_new[l])) {
          hit[l] = f[l];
          end[l] = at[l];
        }
    }
  }
  V3<float> npl[2] = {lane3(np, 0), lane3(np, 1)}, nvl[2] = {lane3(nv, 0), lane3(nv, 1)};
#pragma unroll
  for (int l = 0; l < 2; ++l) {
    if (full[l] && hit[l] < 0)
      collide_lane(lane3(P, l), lane3(V, l), lane3(F, l), l ? m1 : m0, npl[l], nvl[l], c);
    else if (hit[l] >= 0)
      collision_response<float>(faces + hit[l], d_old[l], d_new[l], lane3(P, l), lane3(V, l), lane3(F, l), l ? m1 : m0,
                                c.dt, c.restitution, c.friction, npl[l], nvl[l]);
  }
  np = pk3(npl[0], npl[1]);
  nv = pk3(nvl[0], nvl[1]);
}

// Tiles split into an interior rectangle [bx0, bx1] x [by0, by1] (every
// neighbour of every tile vertex exists: no checks) and the ring of boundary
// tiles around it.
struct TileSplit {
  int tx, ty;          // tiles per row / column
  int bx0, bx1, by0, by1;  // interior rectangle (empty when bx1 < bx0 or by1 < by0)
};

__host__ __device__ __forceinline__ void ring_tile(const TileSplit& t, int k, int& bx, int& by) {
  const bool has_interior = t.bx1 >= t.bx0 && t.by1 >= t.by0;
  if (!has_interior) {
    bx = k % t.tx;
    by = k / t.tx;
    return;
  }
  const int top = t.by0 * t.tx;
  if (k < top) {
    bx = k % t.tx;
    by = k / t.tx;
    return;
  }
  k -= top;
  const int bottom = (t.ty - 1 - t.by1) * t.tx;
  if (k < bottom) {
    bx = k % t.tx;
    by = t.by1 + 1 + k / t.tx;
    return;
  }
  k -= bottom;
  const int per_row = t.bx0 + (t.tx - 1 - t.bx1);
  by = t.by0 + k / per_row;
  const int j = k % per_row;
  bx = j < t.bx0 ? j : t.bx1 + 1 + (j - t.bx0);
}

// Tile of CTA b of the single-cloth kernel: the first n_ring CTAs take the
// ring tiles in ring_tile's order, the rest the interior rectangle row by
// row.  Returns whether the tile is an interior one.
__host__ __device__ __forceinline__ bool grid_tile(const TileSplit& t, int n_ring, int b, int& bx, int& by) {
  if (b < n_ring) {
    ring_tile(t, b, bx, by);
    return false;
  }
  const int k = b - n_ring, nbx = t.bx1 - t.bx0 + 1;
  bx = t.bx0 + k % nbx;
  by = t.by0 + k / nbx;
  return true;
}

// One tile of one cloth; edge: some neighbour of a tile vertex may not exist.
// BATCH: the state is read past the L1, whose few KB beside the shared memory
// are then the many cloths' constants' alone (256 cloths of 16..128 vertices a
// side: 95.0 us a step with it in the L1, 93.9 past it; one cloth, 1024 x 1024,
// the other way round: 47.6 and 47.9).
template <int TH, bool BATCH>
__device__ __forceinline__ void tile_step(int bx, int by, bool edge, int R, int C, const float* __restrict__ params,
                                          const float4* pos, const float4* vel,
                                          const float4* force_in, float4* __restrict__ pos_out,
                                          float4* __restrict__ vel_out, const StepConsts& c, V3<float> wind,
                                          unsigned* flags) {
  using T = Tile<TH>;
  extern __shared__ __align__(128) unsigned char s_dyn[];
  const StagedState<TH> state(s_dyn);
  const StrutTerms<TH> strut(s_dyn);
  const QuadTerms<TH> quads(s_dyn);
  const int c0 = bx * kTileW, r0 = by * TH;
  const int tid = threadIdx.x;
  const f2 one = dup2(c.one), mone = dup2(-c.one);
  const V3x2 nwind{dup2(-wind.x), dup2(-wind.y), dup2(-wind.z)};

  const int lr = tid / kPairW, lc = tid % kPairW;  // main threads: this thread's pair of vertices
  const int h = tid - T::NMAIN;                    // helper lane
  // The helper warp's strut of round j: in the rows above the tile two rounds
  // of natural pairs, left of it pairs whose lanes lie in different blocks.
  auto halo_job = [&](int j, int& kind, int& jr, int& jc) {
    if (j == 0) {
      kind = KBV; jr = h < 16 ? -2 : -1; jc = h & 15;
    } else if (j == 1) {
      kind = h < 16 ? KV : KS; jr = -1; jc = h & 15;
    } else if (j == 2) {
      kind = h < TH ? KH : (h <= 2 * TH ? KS : -1);
      jr = h < TH ? h : (h < 2 * TH ? h - TH : -1);
      jc = -1;
    } else {
      kind = h < 2 * TH ? KBH : -1;
      jr = h < TH ? h : h - TH;
      jc = h < TH ? -2 : -1;
    }
  };

  // ---- copy the strut constants into the slots their struts' terms will take
  // (k and c in uxy, L in s2; each thread copies for the struts it computes)
  const int rec_row = ((C + 31) / 32) * kParamRec;
  const float* rec0 = params + param_rec(0, c0, C) + size_t(r0) * rec_row;
  const uint32_t a_uxy = uint32_t(__cvta_generic_to_shared(strut.uxy)), a_s2 = uint32_t(__cvta_generic_to_shared(strut.s2));
  auto copy_main = [&]() {
    const bool row = r0 + lr < R;
    const float* rec = rec0 + (row ? lr * rec_row : 0) + 4 * lc;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const int o = T::slot(j, lr, lc);
      cp_async16(a_uxy + 16 * o, rec + 64 * j, row);
      cp_async8(a_s2 + 8 * o, rec - 2 * lc + 320 + 32 * j, row);
    }
  };
  auto copy_halo = [&]() {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int kind, jr, jc;
      halo_job(j, kind, jr, jc);
      if (kind < 0) continue;
      const int o = T::slot(kind, jr, jc);
      const bool row = unsigned(r0 + jr) < unsigned(R);
      const float* rec = rec0 + (row ? jr * rec_row : 0);
      const int left = kind == KH ? 0 : (kind == KS ? 1 : (jc == -2 ? 2 : 3));
      cp_async16(a_uxy + 16 * o, rec + (jc >= 0 ? 64 * kind + 4 * jc : kParamLeft + 4 * left), row);
      cp_async8(a_s2 + 8 * o, rec + (jc >= 0 ? 320 + 32 * kind + 2 * jc : kParamLeft + 16 + 2 * left), row);
    }
  };
  if (tid < T::NMAIN)
    copy_main();
  else
    copy_halo();

  // what was read so far (constants, tables) no step writes
  chain_wait();
  chain_next();

  // ---- stage the state as pairs: whole rows of EC pairs a round, so a thread
  // keeps its column
  const float wind1 = length1(wind);
  bool slow = false;  // an edge tile that looks at what exists
  {
    constexpr int RPR = T::NT / T::EC, ROUNDS = (T::EH + RPR - 1) / RPR;
    const int sr = tid / T::EC, sc = tid - sr * T::EC;
    float4 P[ROUNDS][2], V[ROUNDS][2];
    const int first = (r0 - 2 + sr) * C + c0 - 2 + sc;
    auto state_at = [](const float4* p) { return BATCH ? __ldcg(p) : *p; };
    const float4* src_p = pos + first;
    const float4* src_v = vel + first;
    if (edge) {
#pragma unroll
      for (int k = 0; k < ROUNDS; ++k) {
        const int row = sr + k * RPR;
        const bool mine = sr < RPR && row < T::EH && unsigned(r0 - 2 + row) < unsigned(R);
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          const bool ok = mine && unsigned(c0 - 2 + sc + l * kPairW) < unsigned(C);
          P[k][l] = outside_pos(row, sc + l * kPairW);
          V[k][l] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (ok) {
            P[k][l] = state_at(src_p + (k * RPR * C + l * kPairW));
            V[k][l] = state_at(src_v + (k * RPR * C + l * kPairW));
          }
          slow |= !mild(xyz<float>(P[k][l]), xyz<float>(V[k][l]), wind1);
        }
      }
    } else {
#pragma unroll
      for (int k = 0; k < ROUNDS; ++k)
        if (sr < RPR && sr + k * RPR < T::EH)
#pragma unroll
          for (int l = 0; l < 2; ++l) {
            P[k][l] = state_at(src_p + (k * RPR * C + l * kPairW));
            V[k][l] = state_at(src_v + (k * RPR * C + l * kPairW));
          }
    }
#pragma unroll
    for (int k = 0; k < ROUNDS; ++k)
      if (sr < RPR && sr + k * RPR < T::EH)
        state.put((sr + k * RPR) * T::EW + sc, P[k][0], P[k][1], V[k][0], V[k][1]);
  }
  cp_async_wait_all();  // this thread's own copies: it is their only reader
  if (edge)
    slow = __syncthreads_or(slow);
  else
    __syncthreads();

  const int r = r0 + lr, col = c0 + lc, v0 = r * C + col, v1 = v0 + kPairW;
  const bool in0 = tid < T::NMAIN && r < R && col < C, in1 = tid < T::NMAIN && r < R && col + kPairW < C;
  float m0 = 1.0f, m1 = 1.0f, pin0 = 0.0f, pin1 = 0.0f;
  auto absent = [&](int kind, int rr, int cc) {
    return (owned_exists(kind, r0 + rr, c0 + cc, R, C) ? 0u : 1u) |
           (owned_exists(kind, r0 + rr, c0 + cc + kPairW, R, C) ? 0u : 2u);
  };
  PairState s00, s01, s10, s11;  // the corners of this thread's quad pair
  // The struts a thread computes: a main thread's own five, a helper's four.
  // Return root_and_rcp's range verdict.
  auto main_struts = [&](auto fast) -> uint32_t {
    constexpr bool FAST = decltype(fast)::value;
    uint32_t far = 0;
    const int e = T::staged(lr, lc);
    auto strut_to = [&](int kind, const PairState& a, const PairState& b) {
      const int o = T::slot(kind, lr, lc);
      const F2x2 kc = strut.uxy[o];
      strut_pair<FAST>(strut, o, a, b, kc.a, kc.b, strut.s2[o], FAST ? 0u : absent(kind, lr, lc), one, far);
    };
    s00 = pair_at(state, e);
    strut_to(KBH, s00, pair_at(state, e + 2));
    strut_to(KBV, s00, pair_at(state, e + 2 * T::EW));
    s01 = pair_at(state, e + 1);
    s10 = pair_at(state, e + T::EW);
    strut_to(KH, s00, s01);
    strut_to(KV, s00, s10);
    strut_to(KS, s01, s10);
    return far;
  };
  auto halo_struts = [&](auto fast) -> uint32_t {
    constexpr bool FAST = decltype(fast)::value;
    uint32_t far = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int kind, jr, jc;
      halo_job(j, kind, jr, jc);
      if (kind < 0) continue;
      const int e = T::staged(jr, jc), o = T::slot(kind, jr, jc);
      const int ia = kind == KS ? e + 1 : e;
      const int ib = kind == KH ? e + 1 : (kind == KBH ? e + 2 : (kind == KBV ? e + 2 * T::EW : e + T::EW));
      const F2x2 kc = strut.uxy[o];
      strut_pair<FAST>(strut, o, pair_at(state, ia), pair_at(state, ib), kc.a, kc.b, strut.s2[o],
                       FAST ? 0u : absent(kind, jr, jc), one, far);
    }
    return far;
  };
  uint32_t far;
  if (tid < T::NMAIN) {
    far = main_struts(std::true_type{});
    if (__builtin_expect(slow || far > kRootSpan, 0)) {  // the constants' slots hold the terms by now: copy them again
      copy_main();
      cp_async_wait_all();
      main_struts(std::false_type{});
    }
    // mass and pin flag of the pair, needed after the gather
    if (in0) {
      m0 = pos[v0].w;
      pin0 = vel[v0].w;
    }
    if (in1) {
      m1 = pos[v1].w;
      pin1 = vel[v1].w;
    }
  } else {
    far = halo_struts(std::true_type{});
    if (__builtin_expect(slow || far > kRootSpan, 0)) {
      copy_halo();
      cp_async_wait_all();
      halo_struts(std::false_type{});
    }
  }
  {
    // one quad pair a thread: a main thread's own, a helper's above or left of the tile
    const bool main = tid < T::NMAIN;
    const int qr = main ? lr : (h < T::QW ? -1 : h - T::QW), qc = main ? lc : (h < T::QW ? h - 1 : -1);
    if (main || h < T::QW + TH) {
      const int e = T::staged(qr, qc), q = T::quad(qr, qc);
      if (!main) {
        s00 = pair_at(state, e);
        s01 = pair_at(state, e + 1);
        s10 = pair_at(state, e + T::EW);
      }
      s11 = pair_at(state, e + T::EW + 1);
      bool has0 = true, has1 = true;
      f2 neg_cd = dup2(c.neg_drag), neg_lift = dup2(c.neg_lift);
      if (edge) {
        has0 = quad_exists(r0 + qr, c0 + qc, R, C);
        has1 = quad_exists(r0 + qr, c0 + qc + kPairW, R, C);
        neg_cd = lanes(has0, has1, neg_cd, 0);
        neg_lift = lanes(has0, has1, neg_lift, 0);
      }
      far = quad_pair<true>(quads, q, s00, s01, s10, s11, neg_cd, neg_lift, has0, has1, nwind, one);
      if (__builtin_expect(slow || far > kRootSpan, 0))
        quad_pair<false>(quads, q, pair_at(state, e), pair_at(state, e + 1), pair_at(state, e + T::EW),
                         pair_at(state, e + T::EW + 1), neg_cd, neg_lift, has0, has1, nwind, one);
    }
  }
  __syncthreads();
  if (in0 || in1) {
    // ---- gather in the reference's summation order (grid_order.h)
    V3x2 F = pk3(V3<float>{c.force0[0], c.force0[1], c.force0[2]}, V3<float>{c.force0[0], c.force0[1], c.force0[2]});
    if (force_in) {
      const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      F = add3(pk3(xyz<float>(in0 ? force_in[v0] : zero4), xyz<float>(in1 ? force_in[v1] : zero4)), F);
    }
    struct Term {
      V3x2 u;
      f2 s1, s2;
    };
    auto load = [&](int kind, int rr, int cc) {
      const int o = T::slot(kind, rr, cc);
      const F2x2 a = strut.uxy[o], b = strut.uz_s1[o];
      return Term{{a.a, a.b, b.a}, b.b, strut.s2[o]};
    };
    // role 0 adds the strut's forces, role 1 (sign = -1) subtracts them: F - s u == F + (-s) u exactly
    auto add = [&](const Term& t, f2 sign) {
      F = add_p3(F, scale3(t.s1, t.u), sign);
      F = add_p3(F, scale3(t.s2, t.u), sign);
    };
    add(load(KS, lr - 1, lc), mone);  // SH_UP
    {
      Term vt = load(KV, lr - 1, lc), sh = load(KS, lr, lc - 1), hz = load(KH, lr, lc - 1);
      // the last column's upward vertical comes after its shear and horizontal (grid_order.h: slot_at)
      const bool mid = edge && r >= 1 && r <= R - 2;
      const bool late0 = mid && col == C - 1, late1 = mid && col + kPairW == C - 1;
      if (late0 || late1) {
        auto neg = [&](Term& t) { t.s1 = neg2(t.s1); t.s2 = neg2(t.s2); };
        neg(vt);
        neg(hz);
        auto pick = [&](const Term& a, const Term& b) {  // a in late lanes, b in the others
          return Term{lanes3(late0, late1, a.u, b.u), lanes(late0, late1, a.s1, b.s1), lanes(late0, late1, a.s2, b.s2)};
        };
        add(pick(sh, vt), one);
        add(pick(hz, sh), one);
        add(pick(vt, hz), one);
      } else {
        add(vt, mone);  // VT_UP
        add(sh, one);   // SH_LEFT
        add(hz, mone);  // HZ_LEFT
      }
    }
    add(load(KV, lr, lc), one);        // VT_DOWN
    add(load(KH, lr, lc), one);        // HZ_RIGHT
    add(load(KBV, lr - 2, lc), mone);  // BV_UP
    add(load(KBH, lr, lc - 2), mone);  // BH_LEFT
    add(load(KBH, lr, lc), one);       // BH_RIGHT
    add(load(KBV, lr, lc), one);       // BV_DOWN
#pragma unroll
    for (int s = 0; s < N_FACE_SLOTS; ++s) {
      const FaceDesc fd = face_desc(s);
      const int q = T::quad(lr + fd.dr, lc + fd.dc) + fd.is_b * T::NQ;
      const F2x2 dxy = quads.dxy[q];
      const f2 w = fd.corner == 0   ? quads.w0[q]
                   : fd.corner == 1 ? quads.w1[q]
                                    : face_last_share(quads.w0[q], quads.w1[q], mone);
      F = add_p3(F, scale3(w, V3x2{dxy.a, dxy.b, quads.dz[q]}), one);
    }

    // ---- integrate, collide, write
    V3x2 P, V, np, nv;
    state.get(T::staged(lr, lc), P, V);
    integrate_pair(c, P, V, F, pk(m0, m1), one, np, nv);
    // 0 in a lane whose numbers are all finite, NaN otherwise: the move's ends
    const f2 z = dup2(0.0f);
    const f2 ends = fma2(P.z, z, fma2(P.y, z, fma2(P.x, z, fma2(np.z, z, fma2(np.y, z, mul2(np.x, z))))));
    const bool free0 = in0 && pin0 == 0.0f, free1 = in1 && pin1 == 0.0f;
    collide_pair(c, P, V, F, m0, m1, upk(ends), free0, free1, np, nv);
    // the new state
    const float2 after = upk(fma2(nv.z, z, fma2(nv.y, z, fma2(nv.x, z, fma2(np.z, z, fma2(np.y, z, mul2(np.x, z)))))));
    if (((free0 && after.x != 0.0f) || (free1 && after.y != 0.0f)) && flags) atomicOr(flags, 1u);
    // pinned: update_points restores the old point
    if (!(free0 && free1)) {
      np = lanes3(free0, free1, np, P);
      nv = lanes3(free0, free1, nv, V);
    }
    if (in0) {
      pos_out[v0] = make4<float>(lane3(np, 0), m0);
      vel_out[v0] = make4<float>(lane3(nv, 0), pin0);
    }
    if (in1) {
      pos_out[v1] = make4<float>(lane3(np, 1), m1);
      vel_out[v1] = make4<float>(lane3(nv, 1), pin1);
    }
  }
}

// One launch for all tiles: the boundary ring first (its tiles are slower
// and then overlap the interior ones instead of running as a lone wave).
template <int TH>
__global__ void __launch_bounds__(Tile<TH>::NT, Tile<TH>::MIN_CTAS)
    k_step_grid_tiled(int R, int C, TileSplit split, int n_ring, const float* __restrict__ params,
                      const float4* pos, const float4* vel,
                      const float4* force_in, float4* __restrict__ pos_out,
                      float4* __restrict__ vel_out, const __grid_constant__ StepConsts c) {
  int bx, by;
  const V3<float> wind{c.wind[0], c.wind[1], c.wind[2]};
  const bool inner = grid_tile(split, n_ring, blockIdx.x, bx, by);
  tile_step<TH, false>(bx, by, !inner, R, C, params, pos, vel, force_in, pos_out, vel_out, c, wind, c.flags);
}

// Many cloths in one launch, one CTA per work item {cloth, tile x, tile y,
// interior} of a list packed on the host (largest cloths first, each cloth's
// boundary tiles before its interior ones; CTAs start in list order).
// Persistent CTAs that loop over items were slower: what does not depend on
// the tile was kept in registers from tile to tile and 530 bytes a thread
// spilled (256 cloths of 16..128 vertices a side: 146 against 119 us a step).
// n_work_dev: null, or the number of items in device memory (at most the
// grid's size).
template <int TH>
__global__ void __launch_bounds__(Tile<TH>::NT, Tile<TH>::MIN_CTAS)
    k_step_batched(const ClothDesc* __restrict__ cloths, const int4* __restrict__ work, int parity,
                   const __grid_constant__ StepConsts c, const int* __restrict__ n_work_dev) {
  if (n_work_dev && int(blockIdx.x) >= *n_work_dev) return;
  const int4 w = __ldg(work + blockIdx.x);
  const ClothDesc& d = cloths[w.x];
  if (d.skip) return;  // masked out: uniform over the CTA
  const V3<float> wind{d.wind[0], d.wind[1], d.wind[2]};
  tile_step<TH, true>(w.y, w.z, w.w == 0, d.rows, d.cols, d.params, d.pos[parity], d.vel[parity], d.force_in,
                d.pos[parity ^ 1], d.vel[parity ^ 1], c, wind, d.flags);
}

// Ring / interior split of an R x C cloth's 32 x th tiles.  Interior tiles
// have every neighbour of every vertex inside the cloth:
// c0 >= 2, c0 + 32 <= C - 2, r0 >= 2, r0 + th <= R - 2.
TileSplit split_tiles(int rows, int cols, int th) {
  TileSplit t;
  t.tx = (cols + kTileW - 1) / kTileW;
  t.ty = (rows + th - 1) / th;
  t.bx0 = 1;
  t.bx1 = cols >= kTileW + 4 ? (cols - 2 - kTileW) / kTileW : 0;
  t.by0 = 1;
  t.by1 = rows >= th + 4 ? (rows - 2 - th) / th : 0;
  return t;
}

template <int TH>
cudaError_t prime_tiled() {
  cudaError_t e = cudaFuncSetAttribute(k_step_batched<TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(Tile<TH>::SMEM));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_step_grid_tiled<TH>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Tile<TH>::SMEM));
  return e;
}

template <int TH>
int batched_ctas_per_sm_t() {
  int n = 0;
  if (prime_tiled<TH>() != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_step_batched<TH>, Tile<TH>::NT, Tile<TH>::SMEM) !=
          cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return n > 0 ? n : 1;
}

template <int TH>
void launch_batched_t(int grid, const ClothDesc* cloths, const int4* work, int parity, const StepConsts& c,
                      cudaStream_t s, const int* n_work_dev, bool chained) {
  chain_launch(k_step_batched<TH>, grid, Tile<TH>::NT, Tile<TH>::SMEM, s, chained, cloths, work, parity, c, n_work_dev);
}

}  // namespace

bool batch_tile_height_ok(int th) { return th == 4 || th == 8 || th == 12; }

void batch_tiles(int cloth, int rows, int cols, int th, int* out4, int* n_ring, int* n_interior) {
  const TileSplit t = split_tiles(rows, cols, th);
  const bool has_interior = t.bx1 >= t.bx0 && t.by1 >= t.by0;
  const int ni = has_interior ? (t.bx1 - t.bx0 + 1) * (t.by1 - t.by0 + 1) : 0;
  const int nr = t.tx * t.ty - ni;
  *n_ring = nr;
  *n_interior = ni;
  if (!out4) return;
  int k = 0;
  for (int by = 0; by < t.ty; ++by)  // ring tiles first
    for (int bx = 0; bx < t.tx; ++bx) {
      const bool inner = has_interior && bx >= t.bx0 && bx <= t.bx1 && by >= t.by0 && by <= t.by1;
      if (inner) continue;
      out4[4 * k] = cloth; out4[4 * k + 1] = bx; out4[4 * k + 2] = by; out4[4 * k + 3] = 0;
      ++k;
    }
  for (int by = t.by0; has_interior && by <= t.by1; ++by)
    for (int bx = t.bx0; bx <= t.bx1; ++bx) {
      out4[4 * k] = cloth; out4[4 * k + 1] = bx; out4[4 * k + 2] = by; out4[4 * k + 3] = 1;
      ++k;
    }
}

int grid_tiles(int rows, int cols, int th, int* out3) {
  const TileSplit t = split_tiles(rows, cols, th);
  const bool has_interior = t.bx1 >= t.bx0 && t.by1 >= t.by0;
  const int n_interior = has_interior ? (t.bx1 - t.bx0 + 1) * (t.by1 - t.by0 + 1) : 0;
  const int n_ring = t.tx * t.ty - n_interior;
  for (int b = 0; out3 && b < n_ring + n_interior; ++b)  // blockIdx.x b of k_step_grid_tiled
    out3[3 * b + 2] = grid_tile(t, n_ring, b, out3[3 * b], out3[3 * b + 1]) ? 1 : 0;
  return n_ring + n_interior;
}

cudaError_t prime_step_kernels() {
  // the attribute is per function and per device: set once on each device used
  static PerDeviceOnce once;
  return once.run([] {
    cudaError_t e = prime_tiled<4>();
    if (e == cudaSuccess) e = prime_tiled<8>();
    if (e == cudaSuccess) e = prime_tiled<12>();
    return e;
  });
}

int batched_ctas_per_sm(int th) {
  switch (th) {
    case 4: return batched_ctas_per_sm_t<4>();
    case 12: return batched_ctas_per_sm_t<12>();
    default: return batched_ctas_per_sm_t<8>();
  }
}

cudaError_t launch_step_batched(const ClothDesc* cloths, const int4* work, int n_work, int parity,
                                const StepConsts& c, cudaStream_t s, bool chained, const int* n_work_dev, int th) {
  if (n_work <= 0) return cudaSuccess;
  if (!batch_tile_height_ok(th)) return cudaErrorInvalidValue;
  const cudaError_t ea = prime_step_kernels();
  if (ea != cudaSuccess) return ea;
  switch (th) {
    case 4: launch_batched_t<4>(n_work, cloths, work, parity, c, s, n_work_dev, chained); break;
    case 12: launch_batched_t<12>(n_work, cloths, work, parity, c, s, n_work_dev, chained); break;
    default: launch_batched_t<8>(n_work, cloths, work, parity, c, s, n_work_dev, chained); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_step_grid(const GridTopo& g, const float4* pos, const float4* vel, const float4* force_in,
                             float4* pos_out, float4* vel_out, const StepConsts& c, cudaStream_t s, bool chained) {
  const int n = g.rows * g.cols;
  if (n <= 0) return cudaSuccess;
  if (g.variant == 1) {
    k_step_grid_v1<<<(n + 255) / 256, 256, 0, s>>>(g.rows, g.cols, g.params, pos, vel, force_in, pos_out, vel_out,
                                                   c);
  } else {
    const cudaError_t ea = prime_step_kernels();
    if (ea != cudaSuccess) return ea;
    // 8-row tiles, or 4-row ones where there would be no more 8-row tiles than
    // SMs: a tile's latency is the step's then, and the shorter tile has less
    // (us a step with 8 rows and with 4: 20 x 20 3.82 and 3.53, 64 x 64 4.15 and
    // 3.78, 157 x 211 4.46 and 4.45; 190 x 200, 168 tiles of 8 rows, 4.73 and
    // 4.98, 256 x 256 5.8 and 6.1, 1024 x 1024 48 and 56)
    const auto launch = [&](auto kernel, int th, int threads, size_t smem) {
      const TileSplit t = split_tiles(g.rows, g.cols, th);
      const bool has_interior = t.bx1 >= t.bx0 && t.by1 >= t.by0;
      const int n_interior = has_interior ? (t.bx1 - t.bx0 + 1) * (t.by1 - t.by0 + 1) : 0;
      const int n_ring = t.tx * t.ty - n_interior;
      chain_launch(kernel, n_ring + n_interior, threads, smem, s, chained, g.rows, g.cols, t, n_ring, g.params, pos, vel,
                   force_in, pos_out, vel_out, c);
    };
    const long long tiles8 = (long long)((g.cols + kTileW - 1) / kTileW) * ((g.rows + 7) / 8);
    if (tiles8 <= sm_count())
      launch(k_step_grid_tiled<4>, 4, Tile<4>::NT, Tile<4>::SMEM);
    else
      launch(k_step_grid_tiled<8>, 8, Tile<8>::NT, Tile<8>::SMEM);
  }
  return cudaGetLastError();
}

}  // namespace fgb
