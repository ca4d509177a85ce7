// General-mesh step: a deterministic vertex-centric gather over CSR
// incidence lists (no float atomics).
//
// The reference accumulates forces by scattering over struts in strut order
// (springy_mesh.rs:533-551) and then over faces in face order (629-654).  For
// one vertex, its accumulator therefore receives: gravity, then for each
// incident strut in increasing strut index its spring term and its damper
// term, then for each incident face in increasing face index its corner
// share.  The incidence lists here are sorted exactly that way, so each
// vertex sums the same terms in the same order as the reference and the
// result is bit-identical (with -fmad=false) except in the face weights
// (physics.cuh: face_corner_weight; in f32 their corner angles differ from
// the reference's by rounding).
//
// Layout (one entry per incidence):
//   strut_off[v]..strut_off[v+1]  ->  strut_inc[e] = {other vertex, strut<<1 | role}
//                                     role 0: v is the strut's first vertex a, 1: its second b
//   strut_kcl[s]                  =   {stiffness, damping, rest length, 0}
//   face_off[v]..face_off[v+1]    ->  face_inc[e] = face<<2 | corner
//   face_vtx[f]                   =   {v0, v1, v2, 0}
// State: pos[v] = {x, y, z, mass}, vel[v] = {vx, vy, vz, pinned ? 1 : 0}.
//
// The compact forms (FORM 1 and 2; built by mesh_build.cpp's build_compact)
// carry the same lists in fewer bytes, which is what bounds this kernel's
// DRAM traffic: one word per strut incidence (the other vertex as an offset
// from v, the role, and the strut's rank among its first vertex's struts;
// 32 bits in form 1, 16 in form 2 when every offset and rank is small), the
// strut constants as three float arrays in owner order (struts grouped by
// first vertex, ascending id within a group: v's role-0 incidences take v's
// group in order, a role-1 incidence takes entry `rank` of its other
// vertex's group), and one 16-bit word per face incidence (the corner, and
// where the face's other two vertices sit in v's strut list): 2 or 4 bytes
// plus 12 / 2 per strut incidence and 2 per face incidence, instead of
// 8 + 16 and 4 + 16.  The terms and their order are the same, so are the
// bits.
#include "chain_launch.cuh"
#include "kernels.h"
#include "physics.cuh"

namespace fgb {

namespace {

// One strut term added to F, and one face term, in the reference's order.
template <class T>
__device__ __forceinline__ void add_strut(V3<T>& F, V3<T> P, V3<T> V, V3<T> Po, V3<T> Vo, int role, float k,
                                          float cd, float L) {
  V3<T> sf, df;
  if (role == 0) {
    strut_forces<T>(P, Po, V, Vo, T(k), T(cd), T(L), sf, df);
    F = F + sf;
    F = F + df;
  } else {
    strut_forces<T>(Po, P, Vo, V, T(k), T(cd), T(L), sf, df);
    F = F + (T(-1) * sf);
    F = F + (T(-1) * df);
  }
}
template <class T>
__device__ __forceinline__ V3<T> face_term(int i0, int i1, int i2, int corner, const Vec4<T>* pos,
                                           const Vec4<T>* vel, V3<T> wind, const StepConsts& c) {
  const V3<T> x0 = xyz<T>(pos[i0]), x1 = xyz<T>(pos[i1]), x2 = xyz<T>(pos[i2]);
  const V3<T> v0 = xyz<T>(vel[i0]), v1 = xyz<T>(vel[i1]), v2 = xyz<T>(vel[i2]);
  const V3<T> total = face_total_force<T>(x0, x1, x2, v0, v1, v2, wind, T(c.neg_drag), T(c.neg_lift));
  return face_corner_weight<T>(x0, x1, x2, corner) * total;
}

// A strut word of form 1 (32 bits) or 2 (16 bits; a role-0 word has no rank
// and a 15-bit offset): other-vertex offset, rank, role.
template <int FORM>
__device__ __forceinline__ void strut_word(const GeneralTopo& t, int e, int& off, int& rank, int& role) {
  if (FORM == 2) {
    const uint32_t w = __ldg(t.strut_word16 + e);
    role = int(w & 1u);
    off = int(int16_t(uint16_t(w))) >> (role ? 4 : 1);
    rank = int((w >> 1) & 7u);  // meaningful for role 1 only
  } else {
    const uint32_t w = __ldg(t.strut_word + e);
    off = int(w) >> 6;
    rank = int((w >> 1) & 31u);
    role = int(w & 1u);
  }
}

// Strut terms of vertex v added to F in strut order.
template <class T, int FORM>
__device__ __forceinline__ V3<T> gather_struts(int v, V3<T> P, V3<T> V, V3<T> F, const Vec4<T>* pos,
                                               const Vec4<T>* vel, const GeneralTopo& t) {
  const int s_beg = t.strut_off[v], s_end = t.strut_off[v + 1];
  if constexpr (FORM != 0) {
    int own = t.own_off[v];  // owner position of v's next role-0 strut
    for (int e = s_beg; e < s_end; ++e) {
      int off, rank, role;
      strut_word<FORM>(t, e, off, rank, role);
      const int o = v + off;
      const int i = role ? __ldg(t.own_off + o) + rank : own++;
      add_strut<T>(F, P, V, xyz<T>(pos[o]), xyz<T>(vel[o]), role, __ldg(t.sk + i), __ldg(t.sc + i),
                   __ldg(t.sl + i));
    }
  } else {
    for (int e = s_beg; e < s_end; ++e) {
      const int2 inc = t.strut_inc[e];
      const float4 kcl = t.strut_kcl[inc.y >> 1];
      add_strut<T>(F, P, V, xyz<T>(pos[inc.x]), xyz<T>(vel[inc.x]), inc.y & 1, kcl.x, kcl.y, kcl.z);
    }
  }
  return F;
}

// The share of v in its face incidence e (s_beg: v's first strut incidence).
template <class T, int FORM>
__device__ __forceinline__ V3<T> face_share(int v, int e, int s_beg, const Vec4<T>* pos,
                                            const Vec4<T>* vel, const GeneralTopo& t, V3<T> wind,
                                            const StepConsts& c) {
  if constexpr (FORM != 0) {
    const uint32_t h = __ldg(t.face_word + e);
    const int corner = int(h & 3u);
    int o1, o2, rk, rl;
    strut_word<FORM>(t, s_beg + int((h >> 2) & 127u), o1, rk, rl);
    strut_word<FORM>(t, s_beg + int(h >> 9), o2, rk, rl);
    const int u1 = v + o1, u2 = v + o2;
    const int i0 = corner == 0 ? v : u1, i1 = corner == 0 ? u1 : (corner == 1 ? v : u2), i2 = corner == 2 ? v : u2;
    return face_term<T>(i0, i1, i2, corner, pos, vel, wind, c);
  } else {
    const int fc = t.face_inc[e];
    const int4 fv = t.face_vtx[fc >> 2];
    return face_term<T>(fv.x, fv.y, fv.z, fc & 3, pos, vel, wind, c);
  }
}

template <class T, int FORM>
__device__ __forceinline__ V3<T> gather_forces(int v, V3<T> P, V3<T> V, V3<T> F, const Vec4<T>* pos,
                                               const Vec4<T>* vel, const GeneralTopo& t,
                                               const StepConsts& c) {
  const V3<T> wind{T(c.wind[0]), T(c.wind[1]), T(c.wind[2])};
  F = gather_struts<T, FORM>(v, P, V, F, pos, vel, t);
  const int s_beg = t.strut_off[v], f_beg = t.face_off[v], f_end = t.face_off[v + 1];
  for (int e = f_beg; e < f_end; ++e) F = F + face_share<T, FORM>(v, e, s_beg, pos, vel, t, wind, c);
  return F;
}

__device__ __forceinline__ void flag_nonfinite(bool bad, unsigned* flags) {
  if (__any_sync(__activemask(), bad) && bad && flags) atomicOr(flags, 1u);
}

// Fused Simulation::step for one mesh (accumulate -> integrate -> collide ->
// pin restore -> clear), one thread per vertex.  The f32 form asks for 4
// blocks of 256 per SM (at most 64 registers: the gather is latency-bound, so
// resident warps count).  FP64 comes here, over the plain lists, on path 4 and
// without room for k_terms64's scratch; bound by the FP64 units (one warp instruction takes one of them 64
// cycles), it takes single-warp blocks so that a mesh reaches as many of them
// as it has warps (90 x 61 tube: 123 us a step with blocks of 256, 64 with 32).
template <class T> constexpr int kStepBlock = sizeof(T) == 4 ? 256 : 32;
template <class T, int FORM>
__global__ void __launch_bounds__(kStepBlock<T>, sizeof(T) == 4 ? 4 : 1)
    k_step_general(int n, const Vec4<T>* pos, const Vec4<T>* vel,
                   const Vec4<T>* force_in, Vec4<T>* __restrict__ pos_out, Vec4<T>* __restrict__ vel_out,
                   GeneralTopo t, StepConsts c) {
  chain_wait();
  chain_next();
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const Vec4<T> P4 = pos[v];
  const Vec4<T> V4 = vel[v];
  if (V4.w != T(0)) {  // pinned: update_points restores the old point (springy_mesh.rs:492-496)
    pos_out[v] = P4;
    vel_out[v] = V4;
    return;
  }
  const V3<T> P = xyz<T>(P4), V = xyz<T>(V4);
  const T m = P4.w;
  V3<T> F;
  if (force_in) {
    const V3<T> g{T(c.force0[0]), T(c.force0[1]), T(c.force0[2])};
    F = xyz<T>(force_in[v]) + g;
  } else {
    F = V3<T>{T(c.force0[0]), T(c.force0[1]), T(c.force0[2])};
  }
  F = gather_forces<T, FORM>(v, P, V, F, pos, vel, t, c);
  V3<T> np, nv, nF;
  integrate_point<T>(c.integration, T(c.dt), P, V, F, m, np, nv, nF);
  collide_point<T>(static_cast<const ObsFace*>(c.obstacle_faces), c.n_obstacle_faces, P, V, F, m, np, nv, c);
  pos_out[v] = make4<T>(np, m);
  vel_out[v] = make4<T>(nv, V4.w);
  flag_nonfinite(!(finite3(np) && finite3(nv)), c.flags);
}

// The same step with a vertex's terms spread over the warps of a block: 32
// vertices a block, warp 0 sums their struts, the NF other warps compute their
// face shares (warp 1 + j the faces j, j + NF, ...) into shared memory, and
// warp 0 adds those in face order, integrates and collides.  The same terms in
// the same order, so the same bits as k_step_general; a vertex's chain of
// terms is what a step of a small or slow mesh waits for (see the launch).
constexpr int kSplitFaceWarps = 3, kSplitFacesEach = 2;

template <int FORM>
__global__ void __launch_bounds__(32 * (kSplitFaceWarps + 1))
    k_step_split(int n, const float4* pos, const float4* vel, const float4* force_in,
                 float4* __restrict__ pos_out, float4* __restrict__ vel_out,
                 GeneralTopo t, StepConsts c) {
  using T = float;
  constexpr int NF = kSplitFaceWarps, SLOTS = NF * kSplitFacesEach;
  __shared__ T share[SLOTS][3][32];
  __shared__ int s_rounds;
  const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
  const int v = blockIdx.x * 32 + lane;
  const bool vertex = v < n;
  chain_wait();
  chain_next();
  const Vec4<T> V4 = vertex ? vel[v] : make4<T>(V3<T>{T(0), T(0), T(0)}, T(1));
  const bool free = vertex && V4.w == T(0);  // pinned: update_points restores the old point
  const int f_beg = free ? t.face_off[v] : 0, f_end = free ? t.face_off[v + 1] : 0;
  if (role == 0) {
    const int most = __reduce_max_sync(0xffffffffu, f_end - f_beg);
    if (lane == 0) s_rounds = (most + SLOTS - 1) / SLOTS;
  }
  Vec4<T> P4 = V4;
  V3<T> F{T(0), T(0), T(0)};
  if (role == 0) {
    if (vertex) P4 = pos[v];
    if (free) {
      const V3<T> g{T(c.force0[0]), T(c.force0[1]), T(c.force0[2])};
      F = force_in ? xyz<T>(force_in[v]) + g : g;
      F = gather_struts<T, FORM>(v, xyz<T>(P4), xyz<T>(V4), F, pos, vel, t);
    }
  }
  auto shares = [&](int round) {
    const V3<T> wind{T(c.wind[0]), T(c.wind[1]), T(c.wind[2])};
    const int s_beg = free ? t.strut_off[v] : 0;
#pragma unroll 1
    for (int j = role - 1; j < SLOTS; j += NF) {
      const int e = f_beg + round * SLOTS + j;
      if (e >= f_end) break;
      const V3<T> w = face_share<T, FORM>(v, e, s_beg, pos, vel, t, wind, c);
      share[j][0][lane] = w.x;
      share[j][1][lane] = w.y;
      share[j][2][lane] = w.z;
    }
  };
  if (role > 0) shares(0);
  __syncthreads();
  for (int round = 0; round < s_rounds; ++round) {
    if (round > 0) {
      if (role > 0) shares(round);
      __syncthreads();
    }
    if (role == 0)
      for (int j = 0; j < SLOTS && f_beg + round * SLOTS + j < f_end; ++j)
        F = F + V3<T>{share[j][0][lane], share[j][1][lane], share[j][2][lane]};
    if (round + 1 < s_rounds) __syncthreads();
  }
  if (role != 0 || !vertex) return;
  if (!free) {
    pos_out[v] = P4;
    vel_out[v] = V4;
    return;
  }
  const V3<T> P = xyz<T>(P4), V = xyz<T>(V4);
  const T m = P4.w;
  V3<T> np, nv, nF;
  integrate_point<T>(c.integration, T(c.dt), P, V, F, m, np, nv, nF);
  collide_point<T>(static_cast<const ObsFace*>(c.obstacle_faces), c.n_obstacle_faces, P, V, F, m, np, nv, c);
  pos_out[v] = make4<T>(np, m);
  vel_out[v] = make4<T>(nv, V4.w);
  flag_nonfinite(!(finite3(np) && finite3(nv)), c.flags);
}

// FP64 in two launches: every strut's and every face's terms once
// (k_terms64), then per vertex their sum in the same order, the integration
// and the collisions (k_gather64).  The same values, so the same bits as
// k_step_general, which evaluates a strut twice, a face's force three times
// and its cross product six times: the FP64 units bound this step (see
// kStepBlock), and the terms' 96 bytes a strut and face written and read cost
// little beside them.  Blocks of the terms are single warps, the long ones
// first, so that a small mesh reaches every unit.  A face has four threads
// (its force, and each corner's share, which needs the cross product again) up
// to kWholeFaces and one beyond, where the units are full (us a step, four and
// one: 10,700 faces 17.5 and 18.0, 41,800 39.3 and 66.2, 47,800 43.5 and
// 66.4, 59,700 58.5 and 60.9, 71,800 66 and 75, 89,700 78 and 76, 119,600 104 and
// 92, 239,400 197 and 172).
constexpr int kWholeFaces = 65536;

template <int ROLES>
__global__ void __launch_bounds__(32) k_terms64(const Dbl4* pos, const Dbl4* vel, GeneralTopo t, StepConsts c) {
  const int nbf = (t.n_faces + 31) / 32, role = nbf > 0 ? min(int(blockIdx.x) / nbf, ROLES) : ROLES;
  if (role < ROLES) {
    const int f = (int(blockIdx.x) - role * nbf) * 32 + int(threadIdx.x);
    const int4 w = t.face_vtx[min(f, t.n_faces - 1)];
    chain_wait();
    chain_next();
    if (f >= t.n_faces) return;
    const V3<double> x0 = xyz<double>(pos[w.x]), x1 = xyz<double>(pos[w.y]), x2 = xyz<double>(pos[w.z]);
    double* out = t.face_term + 6 * size_t(f);
    if (ROLES == 1)
      for (int k = 0; k < 3; ++k) out[3 + k] = face_corner_weight<double>(x0, x1, x2, k);
    else if (role < 3)
      out[3 + role] = face_corner_weight<double>(x0, x1, x2, role);
    if (role == ROLES - 1) {
      const V3<double> D = face_total_force<double>(
          x0, x1, x2, xyz<double>(vel[w.x]), xyz<double>(vel[w.y]), xyz<double>(vel[w.z]),
          V3<double>{double(c.wind[0]), double(c.wind[1]), double(c.wind[2])}, double(c.neg_drag), double(c.neg_lift));
      out[0] = D.x;
      out[1] = D.y;
      out[2] = D.z;
    }
    return;
  }
  const int e = (int(blockIdx.x) - ROLES * nbf) * 32 + int(threadIdx.x);
  const int i = min(e, t.n_struts - 1);
  const uint32_t a = t.strut_ab[i], b = t.strut_ab[t.n_struts + i];
  const float4 kcl = t.strut_kcl[i];
  chain_wait();
  chain_next();
  if (e >= t.n_struts) return;
  V3<double> sf, df;
  strut_forces<double>(xyz<double>(pos[a]), xyz<double>(pos[b]), xyz<double>(vel[a]), xyz<double>(vel[b]),
                       double(kcl.x), double(kcl.y), double(kcl.z), sf, df);
  double2* out = reinterpret_cast<double2*>(t.strut_term + 6 * size_t(e));
  out[0] = make_double2(sf.x, sf.y);
  out[1] = make_double2(sf.z, df.x);
  out[2] = make_double2(df.y, df.z);
}

// The sums and the integration are the same for each component, so a vertex
// has three threads, in three warps; only the collisions, where there are
// obstacles, take one.  At most 112 registers, six blocks an SM: the unfused
// collision search takes 118 if it may (90 x 61 tube: 20.1 us a step, 17.7 so;
// other sizes within 2%).
__global__ void __maxnreg__(112) k_gather64(int n, const double* pos, const double* vel, const double* force_in,
                                                 double* pos_out, double* vel_out, GeneralTopo t, StepConsts c) {
  __shared__ double sh[9][32];
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  const int v = blockIdx.x * 32 + lane;
  const bool vertex = v < n;
  const int s_beg = vertex ? t.strut_off[v] : 0, s_end = vertex ? t.strut_off[v + 1] : 0;
  const int f_beg = vertex ? t.face_off[v] : 0, f_end = vertex ? t.face_off[v + 1] : 0;
  chain_wait();
  chain_next();
  const size_t at = 4 * size_t(vertex ? v : 0);
  const double m = pos[at + 3], pin = vel[at + 3], p = pos[at + k], w = vel[at + k];
  const bool free = vertex && pin == 0.0;  // pinned: update_points restores the old point (springy_mesh.rs:492-496)
  double F = double(c.force0[k]);
  if (force_in) F = force_in[at + k] + F;
  if (free) {
#pragma unroll 2
    for (int e = s_beg; e < s_end; ++e) {
      const int s = t.strut_inc[e].y;
      const double* q = t.strut_term + 6 * size_t(s >> 1) + k;
      const long long sign = (long long)(s & 1) << 63;  // the second point's: times -1
      F = F + __longlong_as_double(__double_as_longlong(q[0]) ^ sign);
      F = F + __longlong_as_double(__double_as_longlong(q[3]) ^ sign);
    }
#pragma unroll 2
    for (int e = f_beg; e < f_end; ++e) {
      const int f = t.face_inc[e];
      const double* q = t.face_term + 6 * size_t(f >> 2);
      F = F + q[3 + (f & 3)] * q[k];
    }
  }
  V3<double> np, nv, nF;
  integrate_point<double>(c.integration, double(c.dt), V3<double>{p, 0.0, 0.0}, V3<double>{w, 0.0, 0.0},
                          V3<double>{F, 0.0, 0.0}, m, np, nv, nF);
  if (c.n_obstacle_faces > 0) {
    sh[k][lane] = F;
    sh[3 + k][lane] = np.x;
    sh[6 + k][lane] = nv.x;
    __syncthreads();
    if (k == 0 && free) {
      const V3<double> P{p, pos[at + 1], pos[at + 2]}, V{w, vel[at + 1], vel[at + 2]};
      V3<double> n3{sh[3][lane], sh[4][lane], sh[5][lane]}, v3{sh[6][lane], sh[7][lane], sh[8][lane]};
      collide_point<double>(static_cast<const ObsFace*>(c.obstacle_faces), c.n_obstacle_faces, P, V,
                            V3<double>{sh[0][lane], sh[1][lane], sh[2][lane]}, m, n3, v3, c);
      sh[3][lane] = n3.x; sh[4][lane] = n3.y; sh[5][lane] = n3.z;
      sh[6][lane] = v3.x; sh[7][lane] = v3.y; sh[8][lane] = v3.z;
    }
    __syncthreads();
    np.x = sh[3 + k][lane];
    nv.x = sh[6 + k][lane];
  }
  if (!vertex) return;
  pos_out[at + k] = free ? np.x : p;
  vel_out[at + k] = free ? nv.x : w;
  if (k == 0) {
    pos_out[at + 3] = m;
    vel_out[at + 3] = pin;
  }
  if (free) flag_nonfinite(!(isfinite(np.x) && isfinite(nv.x)), c.flags);
}

// accumulate_forces: force[v] = force[v] + gravity + struts + faces; pins -> 0.
template <class T, int FORM>
__global__ void __launch_bounds__(256) k_accumulate(int n, const Vec4<T>* __restrict__ pos,
                                                    const Vec4<T>* __restrict__ vel, Vec4<T>* __restrict__ force,
                                                    GeneralTopo t, StepConsts c) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const Vec4<T> V4 = vel[v];
  const V3<T> g{T(c.force0[0]), T(c.force0[1]), T(c.force0[2])};
  V3<T> F = xyz<T>(force[v]) + g;
  F = gather_forces<T, FORM>(v, xyz<T>(pos[v]), xyz<T>(V4), F, pos, vel, t, c);
  if (V4.w != T(0)) F = V3<T>{T(0), T(0), T(0)};
  force[v] = make4<T>(F, T(0));
}

// State::euler_step / rk4_step into the staging points.
template <class T>
__global__ void __launch_bounds__(256) k_integrate(int n, int integration, T h, const Vec4<T>* __restrict__ pos,
                                                   const Vec4<T>* __restrict__ vel,
                                                   const Vec4<T>* __restrict__ force, Vec4<T>* __restrict__ spos,
                                                   Vec4<T>* __restrict__ svel, Vec4<T>* __restrict__ sforce) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const Vec4<T> P4 = pos[v], V4 = vel[v];
  V3<T> np, nv, nF;
  const T m = P4.w;
  integrate_point<T>(integration, h, xyz<T>(P4), xyz<T>(V4), xyz<T>(force[v]), m, np, nv, nF);
  spos[v] = make4<T>(np, m + T(0) * h);
  svel[v] = make4<T>(nv, V4.w);
  sforce[v] = make4<T>(nF, T(0));
}

// update_points with the staged points: collide, then restore pins.
template <class T>
__global__ void __launch_bounds__(256) k_update(int n, Vec4<T>* __restrict__ pos, Vec4<T>* __restrict__ vel,
                                                Vec4<T>* __restrict__ force, const Vec4<T>* __restrict__ spos,
                                                const Vec4<T>* __restrict__ svel,
                                                const Vec4<T>* __restrict__ sforce, StepConsts c) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const Vec4<T> P4 = pos[v], V4 = vel[v];
  if (V4.w != T(0)) return;  // pinned: keep the old point
  const Vec4<T> nP4 = spos[v], nV4 = svel[v];
  V3<T> np = xyz<T>(nP4), nv = xyz<T>(nV4);
  collide_point<T>(static_cast<const ObsFace*>(c.obstacle_faces), c.n_obstacle_faces, xyz<T>(P4), xyz<T>(V4),
                   xyz<T>(force[v]), P4.w, np, nv, c);
  pos[v] = make4<T>(np, nP4.w);
  vel[v] = make4<T>(nv, V4.w);
  force[v] = sforce[v];
}

template <class T>
__global__ void k_zero4(int n, Vec4<T>* __restrict__ a) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) a[v] = make4<T>(V3<T>{T(0), T(0), T(0)}, T(0));
}

inline int blocks_for(int n, int bs) { return (n + bs - 1) / bs; }

}  // namespace

template <class T>
cudaError_t launch_step_general(int n, const void* pos, const void* vel, const void* force_in, void* pos_out,
                                void* vel_out, const GeneralTopo& t, const StepConsts& c, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const auto run = [&](auto kernel, int blocks, int threads) {
    chain_launch(kernel, blocks, threads, 0, s, true, n, static_cast<const Vec4<T>*>(pos),
                 static_cast<const Vec4<T>*>(vel), static_cast<const Vec4<T>*>(force_in),
                 static_cast<Vec4<T>*>(pos_out), static_cast<Vec4<T>*>(vel_out), t, c);
  };
  if constexpr (sizeof(T) == 8) {
    // (90 x 61 tube: 29.4 us a step in one launch, 17.6 in two; 12 x 10: 24 and 11.4; 300 x 200: 161 and 92.4)
    if (t.strut_term && t.face_term) {
      const bool whole = t.n_faces > kWholeFaces;
      const int terms = (whole ? 1 : 4) * blocks_for(t.n_faces, 32) + blocks_for(t.n_struts, 32);
      if (terms > 0) {
        const cudaError_t e = chain_launch(whole ? k_terms64<1> : k_terms64<4>, terms, 32, 0, s, true,
                                           static_cast<const Dbl4*>(pos), static_cast<const Dbl4*>(vel), t, c);
        if (e != cudaSuccess) return e;
      }
      return chain_launch(k_gather64, blocks_for(n, 32), 96, 0, s, true, n,
                          static_cast<const double*>(pos), static_cast<const double*>(vel),
                          static_cast<const double*>(force_in), static_cast<double*>(pos_out),
                          static_cast<double*>(vel_out), t, c);
    }
  }
  // f32: up to this many vertices a step takes as long as one vertex's chain
  // of terms, which the split kernel shortens; beyond, its shared-memory exchange
  // only costs (tubes, us a step, one thread per vertex and split: 120 vertices
  // 7.8 and 5.6, 8,000 7.9 and 6.4, 32,600 8.4 and 6.5, 32,768 7.8 and 6.6; 37,500
  // 8.4 and 10.6, 60,000 9.6 and 11.6, 100,800 13.8 and 16.4).
  constexpr int kSplitMost = 32768;
  if constexpr (sizeof(T) == 8)
    run(k_step_general<double, 0>, blocks_for(n, kStepBlock<T>), kStepBlock<T>);
  else if (n <= kSplitMost)
    run(t.form == 2 ? k_step_split<2> : (t.form == 1 ? k_step_split<1> : k_step_split<0>), blocks_for(n, 32),
        32 * (kSplitFaceWarps + 1));
  else
    run(t.form == 2 ? k_step_general<T, 2> : (t.form == 1 ? k_step_general<T, 1> : k_step_general<T, 0>),
        blocks_for(n, kStepBlock<T>), kStepBlock<T>);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_accumulate(int n, const void* pos, const void* vel, void* force, const GeneralTopo& t,
                              const StepConsts& c, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  auto k = t.form == 2 ? k_accumulate<T, 2> : (t.form == 1 ? k_accumulate<T, 1> : k_accumulate<T, 0>);
  k<<<blocks_for(n, 256), 256, 0, s>>>(n, static_cast<const Vec4<T>*>(pos), static_cast<const Vec4<T>*>(vel),
                                       static_cast<Vec4<T>*>(force), t, c);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_integrate(int n, int integration, float h, const void* pos, const void* vel, const void* force,
                             void* spos, void* svel, void* sforce, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_integrate<T><<<blocks_for(n, 256), 256, 0, s>>>(
      n, integration, T(h), static_cast<const Vec4<T>*>(pos), static_cast<const Vec4<T>*>(vel),
      static_cast<const Vec4<T>*>(force), static_cast<Vec4<T>*>(spos), static_cast<Vec4<T>*>(svel),
      static_cast<Vec4<T>*>(sforce));
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_update(int n, void* pos, void* vel, void* force, const void* spos, const void* svel,
                          const void* sforce, const StepConsts& c, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_update<T><<<blocks_for(n, 256), 256, 0, s>>>(n, static_cast<Vec4<T>*>(pos), static_cast<Vec4<T>*>(vel),
                                                 static_cast<Vec4<T>*>(force), static_cast<const Vec4<T>*>(spos),
                                                 static_cast<const Vec4<T>*>(svel),
                                                 static_cast<const Vec4<T>*>(sforce), c);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_zero4(int n, void* a, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_zero4<T><<<blocks_for(n, 256), 256, 0, s>>>(n, static_cast<Vec4<T>*>(a));
  return cudaGetLastError();
}

#define FGB_INSTANTIATE(T)                                                                                        \
  template cudaError_t launch_step_general<T>(int, const void*, const void*, const void*, void*, void*,          \
                                              const GeneralTopo&, const StepConsts&, cudaStream_t);                     \
  template cudaError_t launch_accumulate<T>(int, const void*, const void*, void*, const GeneralTopo&,            \
                                            const StepConsts&, cudaStream_t);                                     \
  template cudaError_t launch_integrate<T>(int, int, float, const void*, const void*, const void*, void*, void*, \
                                           void*, cudaStream_t);                                                  \
  template cudaError_t launch_update<T>(int, void*, void*, void*, const void*, const void*, const void*,         \
                                        const StepConsts&, cudaStream_t);                                         \
  template cudaError_t launch_zero4<T>(int, void*, cudaStream_t);
FGB_INSTANTIATE(float)
FGB_INSTANTIATE(double)

}  // namespace fgb
