// gdem_adjoint.cu -- gradients of a trajectory loss for calibration: a
// hand-written adjoint of the DEM step for spheres in a walled box.
//
// Forward model (one step, spheres, h = dt / 2; the production FP64 step in
// exact arithmetic: for a sphere the body-frame SSP-RK3 update rotated back
// to the space frame is w + T h / I):
//   vh = v_n + F_n h / m,  wh = w_n + T_n h / I,  x_{n+1} = x_n + vh dt,
//   (F, T, history)_{n+1} = Phi(x_{n+1}, vh, wh, history_n; kn, en, muc),
//   v_{n+1} = vh + F_{n+1} h / m,  w_{n+1} = wh + T_{n+1} h / I,
// with Phi the sphere-sphere and sphere-wall contact geometry and the Hooke /
// HookeMemory law of gdem_adjoint_law.cuh (tangential spring carried from
// step to step), and (F, T)_0 = Phi(x_0, v_0, w_0) with the cumulative spring
// then zeroed (Grains.cpp:168-173).
//
// Loss: L = sum_i |x_i(N) - x*_i|^2 + |v_i(N) - v*_i|^2.
//
// Reverse sweep: the transposed leapfrog per particle, and per contact the
// transposed Jacobian of Phi applied to the adjoints of its outputs, by the
// chain rule through the law in reverse order (gdem_adjoint_vjp.cuh).  States
// are recomputed from checkpoints taken every K steps.  A forward run on
// Dual<3> numbers seeded on (kn, en, muc) gives the forward-mode gradient
// that checks the parameter part of the adjoint.
//
// Pair search: a linked-cell grid over the domain box (cells at least the
// largest contact distance wide, coordinates outside the box clamped into the
// edge cells) is rebuilt at every force evaluation; each particle collects
// the partners of its 27 cells whose centres pass the contact-distance test
// and takes them in ascending index, the order of an all-pairs loop, so the
// sums and lists do not depend on the grid.
//
// Scope: spheres (any number of classes), box walls, Hooke / HookeMemory
// without rolling resistance, non-periodic domains.  kt and the other law
// parameters come from the XML; kn, en and muc of every contact model are
// replaced by the calibrated values.  MotionError and grid checks are not
// made here (the forward model of a calibration is the step's own).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/grains_b200.h"
#include "gdem_adjoint_vjp.cuh"
#include "gdem_setup.h"

namespace gdem {
namespace {

constexpr int kAdjCap = 32;      // contacts per particle
constexpr int kAdjWalls = 8;     // walls
// Lanes that share one particle's contacts.  A step of a calibration box is
// the latency of one particle's serial work (4,096 particles are one warp per
// multiprocessor): its cells, its contacts and its walls each go one to a
// lane.  8 lanes cover the walls and most particles' contacts in one pass.
constexpr int kAdjLanes = 8;
constexpr int kAdjBlock = 128;

struct AdjCheck : std::runtime_error {
  using std::runtime_error::runtime_error;
};
#define ACK(call)                                                                    \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess) throw AdjCheck(std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Per-class and per-wall constants on the device.
struct AdjTables {
  const TypeDesc* types;
  const WallDesc* walls;
  const ModelDesc* models;
  int nwalls;
  double dt;
};

template <typename T>
__device__ __forceinline__ V3<T> ldv(const T* p, size_t i) {
  return v3(p[3 * i], p[3 * i + 1], p[3 * i + 2]);
}
template <typename T>
__device__ __forceinline__ void stv(T* p, size_t i, V3<T> a) {
  p[3 * i] = a.x; p[3 * i + 1] = a.y; p[3 * i + 2] = a.z;
}
__device__ __forceinline__ V3<double> ldd(const double* p, size_t i) {
  return v3(p[3 * i], p[3 * i + 1], p[3 * i + 2]);
}
template <typename T>
__device__ __forceinline__ V3<T> promote(V3<double> a) {
  return v3(Scal<T>::make(a.x), Scal<T>::make(a.y), Scal<T>::make(a.z));
}

__device__ __forceinline__ ModelDesc const& modelOf(AdjTables const& A, int ma, int mb) {
  return A.models[ma * kMaxMat + mb];
}

// Slot of partner u in particle t's list (of the previous step), or -1.
template <typename L>
__device__ __forceinline__ int findSlotT(L const& lists, int t, int u) {
  const int np = lists.npart[t];
  for (int k = 0; k < np; ++k)
    if (lists.partner[(size_t)t * kAdjCap + k] == u) return k;
  return -1;
}

// Outputs of one pair contact (a = lower index, b = higher index): the force
// and torque it adds to a and to b, the new spring and normal.
template <typename T>
struct PairY {
  V3<T> fa, ta, fb, tb, kd, pn;
  bool contact;
};
template <typename T>
struct PairIn {
  V3<T> xa, xb, va, vb, wa, wb, kd, pn;
  T kn, en, muc;
};

template <typename T>
__device__ __forceinline__ PairY<T> pairContact(AdjTables const& A, PairIn<T> const& in,
                                                TypeDesc const& ta, TypeDesc const& tb,
                                                bool existed) {
  PairY<T> y;
  V3<T> pc, pen;
  y.contact = sphereSphereG(in.xa, ta.radius, in.xb, tb.radius, pc, pen);
  if (!y.contact) return y;
  ModelDesc const& m = modelOf(A, ta.mat, tb.mat);
  LawOut<T> o = contactLaw(m, A.dt, in.kn, in.en, in.muc, pc, pen, in.xa, in.va, in.wa, ta.mass,
                           in.xb, in.vb, in.wb, tb.mass, existed, in.kd, in.pn);
  y.fa = o.f;
  y.ta = vcross(pc - in.xa, o.f);
  y.fb = -o.f;
  y.tb = vcross(pc - in.xb, -o.f);
  y.kd = o.kd;
  y.pn = o.pn;
  return y;
}

template <typename T>
struct WallY {
  V3<T> f, t, kd, pn;
  bool contact;
};
template <typename T>
struct WallIn {
  V3<T> x, v, w, kd, pn;
  T kn, en, muc;
};

template <typename T>
__device__ __forceinline__ WallY<T> wallContact(AdjTables const& A, WallIn<T> const& in,
                                                TypeDesc const& tp, WallDesc const& wd,
                                                bool existed) {
  WallY<T> y;
  V3<T> pc, pen;
  y.contact = sphereWallG(in.x, tp.radius, wd, pc, pen);
  if (!y.contact) return y;
  ModelDesc const& m = modelOf(A, tp.mat, wd.mat);
  const V3<T> zero = vconst<T>(0., 0., 0.);
  LawOut<T> o = contactLaw(m, A.dt, in.kn, in.en, in.muc, pc, pen, in.x, in.v, in.w, tp.mass,
                           vconst<T>(wd.centre[0], wd.centre[1], wd.centre[2]), zero, zero, 1.e20,
                           existed, in.kd, in.pn);
  y.f = o.f;
  y.t = vcross(pc - in.x, o.f);
  y.kd = o.kd;
  y.pn = o.pn;
  return y;
}

template <typename T>
struct ListsT {
  int* partner;
  int* npart;
  T* kd;
  T* pn;
  int* wflag;
  T* wkd;
  T* wpn;
};

// ---------------------------------------------------------- pair search --
// The linked-cell grid of the forward model: cell (i, j, k) has key
// (k nb1 + j) nb0 + i; start[c] .. start[c + 1] index its particles in items.
struct AdjGrid {
  double org[3], inv_edge[3];
  int nb[3];
  int ncells;
  const int* cell;    // cell key of each particle
  const int* start;   // ncells + 1 offsets
  const int* items;   // particles in cell order
};

__device__ __forceinline__ int adjCellIndex(AdjGrid const& g, int d, double x) {
  const double f = floor((x - g.org[d]) * g.inv_edge[d]);
  return f < 0. ? 0 : (f >= (double)g.nb[d] ? g.nb[d] - 1 : (int)f);
}

template <typename T>
__device__ __forceinline__ void adjBin(AdjGrid const& g, int t, V3<T> x, int* cell, int* count) {
  const int i = adjCellIndex(g, 0, val(x.x)), j = adjCellIndex(g, 1, val(x.y)),
            k = adjCellIndex(g, 2, val(x.z));
  const int c = (k * g.nb[1] + j) * g.nb[0] + i;
  cell[t] = c;
  atomicAdd(&count[c], 1);
}

template <typename T>
__global__ void k_adj_bin(int n, AdjGrid g, const T* x, int* cell, int* count) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) adjBin(g, t, ldv(x, t), cell, count);
}

// Exclusive scan of the cell counts by one block of 1024 threads, 4,096
// cells at a time (a calibration box has about that many, so one pass);
// start[ncells] receives the total, cursor a copy of the starts (k_adj_place
// counts it up), and the counts are cleared for the next evaluation.
__global__ void __launch_bounds__(1024) k_adj_scan(int ncells, int* count, int* start,
                                                   int* cursor) {
  constexpr int kPer = 4;
  __shared__ int warp_sum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int carry = 0;
  for (int base = 0; base < ncells; base += 1024 * kPer) {
    const int i0 = base + kPer * threadIdx.x;
    int v[kPer], sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      v[j] = i0 + j < ncells ? count[i0 + j] : 0;
      sum += v[j];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int y = warp_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int z = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += z;
      }
      warp_sum[lane] = y;
    }
    __syncthreads();
    int at = carry + (wid > 0 ? warp_sum[wid - 1] : 0) + x - sum;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (i0 + j < ncells) {
        start[i0 + j] = at;
        cursor[i0 + j] = at;
        count[i0 + j] = 0;
      }
      at += v[j];
    }
    carry += warp_sum[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) start[ncells] = carry;
}

__global__ void k_adj_place(int n, const int* cell, int* cursor, int* items) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) items[atomicAdd(&cursor[cell[t]], 1)] = t;
}

// The value of v on lane src of the particle's lanes.
__device__ __forceinline__ double laneOf(unsigned mask, double v, int src) {
  return __shfl_sync(mask, v, src, kAdjLanes);
}
template <int N>
__device__ __forceinline__ Dual<N> laneOf(unsigned mask, Dual<N> v, int src) {
  v.v = laneOf(mask, v.v, src);
#pragma unroll
  for (int k = 0; k < N; ++k) v.d[k] = laneOf(mask, v.d[k], src);
  return v;
}
template <typename T>
__device__ __forceinline__ V3<T> laneOf(unsigned mask, V3<T> v, int src) {
  return v3(laneOf(mask, v.x, src), laneOf(mask, v.y, src), laneOf(mask, v.z, src));
}

// ------------------------------------------------------------- forward --
// Contact forces and the new contact lists at one step.  vel/omg are the
// velocities the law sees (half-step ones, or the initial ones at the
// leapfrog start).  zero_spring: the leapfrog start zeroes the cumulative
// spring after the evaluation.  kAdjLanes lanes per particle: the 27 cells,
// then the contacts, then the walls are shared out; the partners are taken in
// ascending index and the forces added in that order, whatever the lanes'
// order of finding them.
template <typename T>
__global__ void __launch_bounds__(kAdjBlock)
    k_fwd_forces(int n, AdjTables A, AdjGrid G, const int* type, const T* x, const T* vel,
                 const T* omg, ListsT<T> prev, int has_prev, ListsT<T> cur, T* F, T* Tq, T kn,
                 T en, T muc, int zero_spring, int* overflow) {
  constexpr int kGroups = kAdjBlock / kAdjLanes;
  __shared__ int found_s[kGroups][kAdjCap], cand_s[kGroups][kAdjCap], count_s[kGroups];
  const int grp = threadIdx.x / kAdjLanes, lane = threadIdx.x % kAdjLanes;
  const unsigned mask = ((1u << kAdjLanes) - 1u) << (threadIdx.x & 31 & ~(kAdjLanes - 1));
  const int t = blockIdx.x * kGroups + grp;
  if (t >= n) return;   // (the particle's lanes together)
  TypeDesc const& tp = A.types[type[t]];
  const V3<T> xt = ldv(x, t);
  V3<T> Ft = vconst<T>(tp.weight[0], tp.weight[1], tp.weight[2]);
  V3<T> Tt = vconst<T>(0., 0., 0.);
  const V3<T> zero = vconst<T>(0., 0., 0.);
  // partners whose centres pass the contact-distance test, from the 27
  // cells around t's
  if (lane == 0) count_s[grp] = 0;
  __syncwarp(mask);
  {
    const int c = G.cell[t];
    const int ci = c % G.nb[0], cj = (c / G.nb[0]) % G.nb[1], ck = c / (G.nb[0] * G.nb[1]);
    for (int q = lane; q < 27; q += kAdjLanes) {
      const int i3 = ci + q % 3 - 1, j3 = cj + (q / 3) % 3 - 1, k3 = ck + q / 9 - 1;
      if (i3 < 0 || i3 >= G.nb[0] || j3 < 0 || j3 >= G.nb[1] || k3 < 0 || k3 >= G.nb[2]) continue;
      const int cc = (k3 * G.nb[1] + j3) * G.nb[0] + i3;
      for (int e = G.start[cc]; e < G.start[cc + 1]; ++e) {
        const int u = G.items[e];
        if (u == t) continue;
        TypeDesc const& tu = A.types[type[u]];
        const V3<T> xu = ldv(x, u);
        const double dx = val(xu.x) - val(xt.x), dy = val(xu.y) - val(xt.y),
                     dz = val(xu.z) - val(xt.z);
        const double R = (tp.radius + tu.radius) * (1. + 1.e-9);
        if (dx * dx + dy * dy + dz * dz >= R * R) continue;
        const int at = atomicAdd(&count_s[grp], 1);
        if (at < kAdjCap) found_s[grp][at] = u;
        else atomicOr(overflow, 1);
      }
    }
  }
  __syncwarp(mask);
  const int nc = min(count_s[grp], kAdjCap);
  for (int i = lane; i < nc; i += kAdjLanes) {
    const int u = found_s[grp][i];
    int rank = 0;
    for (int j = 0; j < nc; ++j) rank += found_s[grp][j] < u;
    cand_s[grp][rank] = u;
  }
  __syncwarp(mask);
  int k = 0;
  for (int q0 = 0; q0 < nc; q0 += kAdjLanes) {
    V3<T> f = zero, tq = zero, kd, pn;
    int u = 0;
    bool hit = false;
    if (q0 + lane < nc) {
      u = cand_s[grp][q0 + lane];
      const int a = t < u ? t : u, b = t < u ? u : t;
      const int j = has_prev ? findSlotT(prev, t, u) : -1;
      const bool existed = j >= 0;
      PairIn<T> in;
      in.xa = ldv(x, a); in.xb = ldv(x, b);
      in.va = ldv(vel, a); in.vb = ldv(vel, b);
      in.wa = ldv(omg, a); in.wb = ldv(omg, b);
      in.kd = existed ? ldv(prev.kd, (size_t)t * kAdjCap + j) : zero;
      in.pn = existed ? ldv(prev.pn, (size_t)t * kAdjCap + j) : zero;
      in.kn = kn; in.en = en; in.muc = muc;
      const PairY<T> y = pairContact(A, in, A.types[type[a]], A.types[type[b]], existed);
      hit = y.contact;
      if (hit) {
        f = t == a ? y.fa : y.fb;
        tq = t == a ? y.ta : y.tb;
        kd = y.kd;
        pn = y.pn;
      }
    }
    unsigned hits = __ballot_sync(mask, hit) >> (threadIdx.x & 31 & ~(kAdjLanes - 1));
    if (hit) {
      const size_t sl = (size_t)t * kAdjCap + k + __popc(hits & ((1u << lane) - 1u));
      cur.partner[sl] = u;
      stv(cur.kd, sl, zero_spring ? zero : kd);
      stv(cur.pn, sl, pn);
    }
    k += __popc(hits & ((1u << kAdjLanes) - 1u));
    for (hits &= (1u << kAdjLanes) - 1u; hits; hits &= hits - 1u) {
      const int src = __ffs(hits) - 1;
      Ft = Ft + laneOf(mask, f, src);
      Tt = Tt + laneOf(mask, tq, src);
    }
  }
  if (lane == 0) cur.npart[t] = k;
  static_assert(kAdjWalls <= kAdjLanes, "one wall per lane");
  {
    V3<T> f = zero, tq = zero;
    bool hit = false;
    if (lane < A.nwalls) {
      WallDesc const& wd = A.walls[lane];
      const size_t sl = (size_t)t * kAdjWalls + lane;
      const bool existed = has_prev && prev.wflag[sl];
      WallIn<T> in;
      in.x = xt; in.v = ldv(vel, t); in.w = ldv(omg, t);
      in.kd = existed ? ldv(prev.wkd, sl) : zero;
      in.pn = existed ? ldv(prev.wpn, sl) : zero;
      in.kn = kn; in.en = en; in.muc = muc;
      const WallY<T> y = wallContact(A, in, tp, wd, existed);
      hit = y.contact;
      cur.wflag[sl] = hit ? 1 : 0;
      if (hit) {
        f = y.f;
        tq = y.t;
        stv(cur.wkd, sl, zero_spring ? zero : y.kd);
        stv(cur.wpn, sl, y.pn);
      }
    }
    unsigned hits = __ballot_sync(mask, hit) >> (threadIdx.x & 31 & ~(kAdjLanes - 1));
    for (hits &= (1u << kAdjLanes) - 1u; hits; hits &= hits - 1u) {
      const int src = __ffs(hits) - 1;
      Ft = Ft + laneOf(mask, f, src);
      Tt = Tt + laneOf(mask, tq, src);
    }
  }
  if (lane == 0) {
    stv(F, t, Ft);
    stv(Tq, t, Tt);
  }
}

// Closing kick (unless v, w are the step's full velocities already): v = vh +
// F h / m, w = wh + T h / I.
template <typename T>
__device__ __forceinline__ void closeKick(AdjTables const& A, TypeDesc const& tp, int closed, V3<T> F,
                                          V3<T> Tq, V3<T>& v, V3<T>& w) {
  if (closed) return;
  const double h = 0.5 * A.dt;
  v = v + vscale(F, Scal<T>::make(h / tp.mass));
  w = w + vscale(Tq, Scal<T>::make(h / tp.inertia[0]));
}

// The closing kick of the step before (closeKick on vi, wi), then this step's
// opening kick + drift: vh = v + F h / m, wh = w + T h / I, x' = x + vh dt;
// the particle is counted into its cell on the way.
template <typename T>
__global__ void k_fwd_move(int n, AdjTables A, AdjGrid G, const int* type, int closed, const T* x,
                           const T* vi, const T* wi, const T* F, const T* Tq, T* xo, T* vh, T* wh,
                           int* cell, int* count) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  TypeDesc const& tp = A.types[type[t]];
  const double h = 0.5 * A.dt;
  const V3<T> f = ldv(F, t), tq = ldv(Tq, t);
  V3<T> v = ldv(vi, t), w = ldv(wi, t);
  closeKick(A, tp, closed, f, tq, v, w);
  const V3<T> vv = v + vscale(f, Scal<T>::make(h / tp.mass));
  const V3<T> ww = w + vscale(tq, Scal<T>::make(h / tp.inertia[0]));
  stv(vh, t, vv);
  stv(wh, t, ww);
  const V3<T> xn = ldv(x, t) + vscale(vv, Scal<T>::make(A.dt));
  stv(xo, t, xn);
  adjBin(G, t, xn, cell, count);
}

// The full state after a step (closeKick on vi, wi), into its own arrays.
template <typename T>
__global__ void k_fwd_state(int n, AdjTables A, const int* type, int closed, const T* x,
                            const T* vi, const T* wi, const T* F, const T* Tq, T* xo, T* vo, T* wo,
                            T* Fo, T* To) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const V3<T> f = ldv(F, t), tq = ldv(Tq, t);
  V3<T> v = ldv(vi, t), w = ldv(wi, t);
  closeKick(A, A.types[type[t]], closed, f, tq, v, w);
  stv(xo, t, ldv(x, t));
  stv(vo, t, v);
  stv(wo, t, w);
  stv(Fo, t, f);
  stv(To, t, tq);
}

// The used part of one step's contact lists, kAdjLanes lanes per particle.
template <typename T>
__global__ void __launch_bounds__(kAdjBlock) k_copy_lists(int n, ListsT<T> dst, ListsT<T> src) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = i / kAdjLanes, lane = i % kAdjLanes;
  if (t >= n) return;
  const int np = src.npart[t];
  if (lane == 0) dst.npart[t] = np;
  for (int k = lane; k < np; k += kAdjLanes) {
    const size_t sl = (size_t)t * kAdjCap + k;
    dst.partner[sl] = src.partner[sl];
    stv(dst.kd, sl, ldv(src.kd, sl));
    stv(dst.pn, sl, ldv(src.pn, sl));
  }
  const size_t ws = (size_t)t * kAdjWalls + lane;
  const int wf = src.wflag[ws];
  dst.wflag[ws] = wf;
  if (wf) {
    stv(dst.wkd, ws, ldv(src.wkd, ws));
    stv(dst.wpn, ws, ldv(src.wpn, ws));
  }
}

// Per-particle squared error of positions and velocities.
template <typename T>
__global__ void k_fwd_loss(int n, const T* x, const T* v, const double* tx, const double* tv,
                           T* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const V3<T> dx = ldv(x, t) - promote<T>(ldd(tx, t));
  const V3<T> dv = ldv(v, t) - promote<T>(ldd(tv, t));
  out[t] = vdot(dx, dx) + vdot(dv, dv);
}

// ------------------------------------------------------------- reverse --
// Adjoints of the particles' x, v, w, F, T after a step (or, at the leapfrog
// start, of its inputs), 3 per particle each.
struct AdjState {
  double *x, *v, *w, *F, *T;
};
// Adjoints of one step's contact history, in the layout of its lists; only
// the entries of the lists in use are meaningful.
struct AdjHist {
  double *kd, *pn, *wkd, *wpn;
};

// One step, transposed: the closing kick, the contact forces and the opening
// kick + drift, from the adjoints at step s (in) to those at s - 1 (out);
// start: the leapfrog start's evaluation alone (no kicks; the spring it left
// was zeroed).  Per contact the adjoints of t's own inputs come from one
// sweep of contactBar, once from either side; the history's go to the slots
// of step s - 1 that supplied it, and kn, en, muc's to the lower index.
// kAdjLanes lanes per particle, one contact or wall each, summed over the
// lanes in a fixed tree.
__global__ void __launch_bounds__(kAdjBlock)
    k_bwd_step(int n, AdjTables A, const int* type, const double* x, const double* vel,
               const double* omg, ListsT<double> prev, int has_prev, ListsT<double> cur,
               AdjState in, AdjState out, AdjHist h_in, AdjHist h_out, double* lp, double kn,
               double en, double muc, int start) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = i / kAdjLanes, lane = i % kAdjLanes;
  const unsigned mask = ((1u << kAdjLanes) - 1u) << (threadIdx.x & 31 & ~(kAdjLanes - 1));
  if (t >= n) return;   // (the particle's lanes together)
  TypeDesc const& tp = A.types[type[t]];
  const double h = 0.5 * A.dt;
  const W3 zero = w3zero();
  // adjoint of the force and torque of particle p: the closing kick's share added
  auto forceBar = [&](int p, TypeDesc const& q, W3& f, W3& tq) {
    f = ldd(in.F, p);
    tq = ldd(in.T, p);
    if (!start) {
      f = f + (h / q.mass) * ldd(in.v, p);
      tq = tq + (h / q.inertia[0]) * ldd(in.w, p);
    }
  };
  W3 lFt, lTt;
  forceBar(t, tp, lFt, lTt);
  const W3 xt = ldd(x, t), vt = ldd(vel, t), wt = ldd(omg, t);
  W3 gx = zero, gv = zero, gw = zero, gp = zero;
  // the history adjoints of step s - 1 start from zero
  if (has_prev) {
    const int pp = prev.npart[t];
    for (int k = lane; k < pp; k += kAdjLanes) {
      stv(h_out.kd, (size_t)t * kAdjCap + k, zero);
      stv(h_out.pn, (size_t)t * kAdjCap + k, zero);
    }
    stv(h_out.wkd, (size_t)t * kAdjWalls + lane, zero);
    stv(h_out.wpn, (size_t)t * kAdjWalls + lane, zero);
  }
  __syncwarp(mask);
  const int np = cur.npart[t];
  for (int k = lane; k < np; k += kAdjLanes) {
    const size_t sl = (size_t)t * kAdjCap + k;
    const int u = cur.partner[sl];
    TypeDesc const& tu = A.types[type[u]];
    const int j = has_prev ? findSlotT(prev, t, u) : -1;
    const bool existed = j >= 0;
    const size_t pj = (size_t)t * kAdjCap + (j >= 0 ? j : 0);
    const bool mine = t < u;   // t is the law's first body
    const W3 xu = ldd(x, u);
    W3 lFu, lTu;
    forceBar(u, tu, lFu, lTu);
    LawArgs a, g;
    W3 pen;
    const W3 xa = mine ? xt : xu, xb = mine ? xu : xt;
    const double ra = mine ? tp.radius : tu.radius, rb = mine ? tu.radius : tp.radius;
    if (!sphereSphereG(xa, ra, xb, rb, a.pc, pen)) continue;
    a.pen = pen;
    const W3 vu = ldd(vel, u), wu = ldd(omg, u);
    a.x0 = xa; a.v0 = mine ? vt : vu; a.w0 = mine ? wt : wu;
    a.x1 = xb; a.v1 = mine ? vu : vt; a.w1 = mine ? wu : wt;
    a.kd = existed ? ldd(prev.kd, pj) : zero;
    a.pn = existed ? ldd(prev.pn, pj) : zero;
    a.kn = kn; a.en = en; a.muc = muc;
    ModelDesc const& m = mine ? modelOf(A, tp.mat, tu.mat) : modelOf(A, tu.mat, tp.mat);
    contactBar(m, A.dt, a, mine ? tp.mass : tu.mass, mine ? tu.mass : tp.mass, existed,
               mine ? lFt : lFu, mine ? lTt : lTu, mine ? lFu : lFt, mine ? lTu : lTt,
               start ? zero : ldd(h_in.kd, sl), ldd(h_in.pn, sl), g);
    sphereSphereBar(xa, ra, xb, rb, g.pc, g.pen, g.x0, g.x1);
    acc(gx, mine ? g.x0 : g.x1);
    acc(gv, mine ? g.v0 : g.v1);
    acc(gw, mine ? g.w0 : g.w1);
    if (mine) acc(gp, v3(g.kn, g.en, g.muc));
    if (existed && m.memory) {
      stv(h_out.kd, pj, g.kd);
      stv(h_out.pn, pj, g.pn);
    }
  }
  if (lane < A.nwalls && cur.wflag[(size_t)t * kAdjWalls + lane]) {
    const size_t sl = (size_t)t * kAdjWalls + lane;
    WallDesc const& wd = A.walls[lane];
    const bool existed = has_prev && prev.wflag[sl];
    ModelDesc const& m = modelOf(A, tp.mat, wd.mat);
    LawArgs a, g;
    W3 pen;
    if (sphereWallG(xt, tp.radius, wd, a.pc, pen)) {
      a.pen = pen;
      a.x0 = xt; a.v0 = vt; a.w0 = wt;
      a.x1 = v3(wd.centre[0], wd.centre[1], wd.centre[2]);
      a.v1 = zero; a.w1 = zero;
      a.kd = existed ? ldd(prev.wkd, sl) : zero;
      a.pn = existed ? ldd(prev.wpn, sl) : zero;
      a.kn = kn; a.en = en; a.muc = muc;
      contactBar(m, A.dt, a, tp.mass, 1.e20, existed, lFt, lTt, zero, zero,
                 start ? zero : ldd(h_in.wkd, sl), ldd(h_in.wpn, sl), g);
      sphereWallBar(xt, tp.radius, wd, g.pc, g.pen, g.x0);
      acc(gx, g.x0);
      acc(gv, g.v0);
      acc(gw, g.w0);
      acc(gp, v3(g.kn, g.en, g.muc));
      if (existed && m.memory) {
        stv(h_out.wkd, sl, g.kd);
        stv(h_out.wpn, sl, g.pn);
      }
    }
  }
  __syncwarp(mask);
#pragma unroll
  for (int o = kAdjLanes / 2; o > 0; o >>= 1) {
    auto add = [&](W3& q) {
      q = q + v3(__shfl_xor_sync(mask, q.x, o, kAdjLanes), __shfl_xor_sync(mask, q.y, o, kAdjLanes),
                 __shfl_xor_sync(mask, q.z, o, kAdjLanes));
    };
    add(gx); add(gv); add(gw); add(gp);
  }
  if (lane != 0) return;
  stv(lp, t, ldd(lp, t) + gp);
  if (start) {
    stv(out.v, t, ldd(in.v, t) + gv);
    return;
  }
  // opening kick + drift, transposed
  const W3 lx = ldd(in.x, t) + gx;
  const W3 lv = ldd(in.v, t) + gv + A.dt * lx, lw = ldd(in.w, t) + gw;
  stv(out.x, t, lx);
  stv(out.v, t, lv);
  stv(out.w, t, lw);
  stv(out.F, t, (h / tp.mass) * lv);
  stv(out.T, t, (h / tp.inertia[0]) * lw);
}

__global__ void k_bwd_seed(int n, const double* x, const double* v, const double* tx,
                           const double* tv, double* lx, double* lv) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  for (int d = 0; d < 3; ++d) {
    lx[3 * t + d] = 2. * (x[3 * t + d] - tx[3 * t + d]);
    lv[3 * t + d] = 2. * (v[3 * t + d] - tv[3 * t + d]);
  }
}

}  // namespace
}  // namespace gdem

// ------------------------------------------------------------------ host --
namespace gdem {
namespace {

template <typename T>
__global__ void k_promote(int n3, const double* a, T* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) out[i] = Scal<T>::make(a[i]);
}

inline int nblk(int n) { return (n + 127) / 128; }

// Sets the first derivative slot of one element to 1 (forward-mode seed).
template <typename T>
__global__ void k_seed(T* a, int i) {
  a[i].d[0] = 1.;
}
template <>
__global__ void k_seed<double>(double*, int) {}

struct AdjointSystem {
  AdjointSetup setup;
  AdjTables A{};
  int n = 0;
  int* d_type = nullptr;
  double *d_x0 = nullptr, *d_v0 = nullptr, *d_w0 = nullptr;
  int* d_overflow = nullptr;
  AdjGrid G{};
  int *d_cell = nullptr, *d_count = nullptr, *d_cursor = nullptr, *d_start = nullptr,
      *d_items = nullptr;
  std::vector<void*> allocs;
  // A run's working memory: blocks handed out in order, kept for the next run
  // up to kKeepBytes in all and given back with the system.  (A run of the
  // calibration case needs some 500 arrays; allocating and freeing them took
  // longer than its kernels.)
  struct Block {
    char* p;
    size_t size, used;
  };
  std::vector<Block> work;
  static constexpr size_t kKeepBytes = size_t(1) << 30, kBlockBytes = size_t(32) << 20;
  cudaStream_t st = nullptr;

  ~AdjointSystem() {
    for (void* p : allocs) cudaFree(p);
    for (auto const& b : work) cudaFree(b.p);
    if (st) cudaStreamDestroy(st);
  }
  template <typename T>
  T* scratch(size_t count) {
    const size_t bytes = (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
    for (auto& b : work)
      if (b.size - b.used >= bytes) {
        T* p = reinterpret_cast<T*>(b.p + b.used);
        b.used += bytes;
        return p;
      }
    Block b{nullptr, std::max(bytes, kBlockBytes), bytes};
    if (cudaMalloc(&b.p, b.size) != cudaSuccess) {
      // (a block larger than the array asked for may not fit any more)
      cudaGetLastError();
      b.size = bytes;
      ACK(cudaMalloc(&b.p, b.size));
    }
    work.push_back(b);
    return reinterpret_cast<T*>(b.p);
  }
  template <typename T>
  T* alloc(size_t count) {
    void* p = nullptr;
    ACK(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
    allocs.push_back(p);
    return static_cast<T*>(p);
  }
  template <typename T>
  ListsT<T> allocLists() {
    ListsT<T> L;
    L.partner = scratch<int>((size_t)n * kAdjCap);
    L.npart = scratch<int>(n);
    L.kd = scratch<T>((size_t)n * kAdjCap * 3);
    L.pn = scratch<T>((size_t)n * kAdjCap * 3);
    L.wflag = scratch<int>((size_t)n * kAdjWalls);
    L.wkd = scratch<T>((size_t)n * kAdjWalls * 3);
    L.wpn = scratch<T>((size_t)n * kAdjWalls * 3);
    // (k_fwd_forces writes the flags of the walls there are)
    ACK(cudaMemsetAsync(L.wflag, 0, (size_t)n * kAdjWalls * sizeof(int), st));
    return L;
  }
  template <typename T>
  void copyLists(ListsT<T> const& dst, ListsT<T> const& src) {
    k_copy_lists<T><<<laneBlocks(), kAdjBlock, 0, st>>>(n, dst, src);
  }
  // blocks of a kernel with kAdjLanes lanes per particle
  int laneBlocks() const { return (int)(((long long)n * kAdjLanes + kAdjBlock - 1) / kAdjBlock); }

  void create(std::string const& xml) {
    readAdjointSetup(xml, setup);
    for (auto const& t : setup.types)
      if (t.shape != 0) throw std::runtime_error("the adjoint handles spheres only");
    for (int d = 0; d < 3; ++d)
      if (setup.periodic[d]) throw std::runtime_error("the adjoint handles non-periodic domains only");
    if ((int)setup.walls.size() > kAdjWalls) throw std::runtime_error("the adjoint handles at most 8 walls");
    for (auto const& m : setup.models)
      if (m.valid && m.rolling) throw std::runtime_error("the adjoint has no rolling resistance");
    ACK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    TypeDesc* dt = alloc<TypeDesc>(setup.types.size());
    WallDesc* dw = alloc<WallDesc>(setup.walls.size());
    ModelDesc* dm = alloc<ModelDesc>(kMaxMat * kMaxMat);
    ACK(cudaMemcpy(dt, setup.types.data(), setup.types.size() * sizeof(TypeDesc), cudaMemcpyHostToDevice));
    if (!setup.walls.empty())
      ACK(cudaMemcpy(dw, setup.walls.data(), setup.walls.size() * sizeof(WallDesc), cudaMemcpyHostToDevice));
    ACK(cudaMemcpy(dm, setup.models, sizeof(setup.models), cudaMemcpyHostToDevice));
    A.types = dt; A.walls = dw; A.models = dm;
    A.nwalls = (int)setup.walls.size();
    A.dt = setup.dt;
    d_overflow = alloc<int>(1);
    // pair-search grid: cells at least the largest contact distance wide,
    // at most 2^22 of them
    double rmax = 0.;
    for (auto const& t : setup.types) rmax = std::max(rmax, t.radius);
    const double emin = 2. * rmax * (1. + 1.e-6);
    for (int d = 0; d < 3; ++d) {
      const double L = setup.maxc[d] - setup.origin[d];
      G.nb[d] = (L > 0. && emin > 0.) ? std::max(1, (int)std::min(std::floor(L / emin), 1.e6)) : 1;
      G.org[d] = setup.origin[d];
    }
    while ((long long)G.nb[0] * G.nb[1] * G.nb[2] > (1ll << 22)) {
      int dm = 0;
      for (int d = 1; d < 3; ++d)
        if (G.nb[d] > G.nb[dm]) dm = d;
      G.nb[dm] = (G.nb[dm] + 1) / 2;
    }
    for (int d = 0; d < 3; ++d) {
      const double L = setup.maxc[d] - setup.origin[d];
      G.inv_edge[d] = L > 0. ? G.nb[d] / L : 0.;
    }
    G.ncells = G.nb[0] * G.nb[1] * G.nb[2];
    d_count = alloc<int>(G.ncells);
    d_cursor = alloc<int>(G.ncells);
    ACK(cudaMemset(d_count, 0, (size_t)G.ncells * sizeof(int)));
    d_start = alloc<int>((size_t)G.ncells + 1);
    G.start = d_start;
  }

  void setParticles(int64_t nn, const int* type, const double* x0, const double* v0,
                    const double* w0) {
    if (nn <= 0 || nn > (1 << 24)) throw std::runtime_error("particle count out of range");
    if (d_type) throw std::runtime_error("particles already set");
    n = (int)nn;
    for (int64_t i = 0; i < nn; ++i)
      if (type[i] < 0 || type[i] >= (int)setup.types.size())
        throw std::runtime_error("particle type out of range");
    d_type = alloc<int>(n);
    d_x0 = alloc<double>(3 * (size_t)n);
    d_v0 = alloc<double>(3 * (size_t)n);
    d_w0 = alloc<double>(3 * (size_t)n);
    d_cell = alloc<int>(n);
    d_items = alloc<int>(n);
    G.cell = d_cell;
    G.items = d_items;
    ACK(cudaMemcpy(d_type, type, n * sizeof(int), cudaMemcpyHostToDevice));
    ACK(cudaMemcpy(d_x0, x0, 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
    ACK(cudaMemcpy(d_v0, v0, 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
    if (w0) ACK(cudaMemcpy(d_w0, w0, 3 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
    else ACK(cudaMemset(d_w0, 0, 3 * (size_t)n * sizeof(double)));
  }

  // Takes the working memory back at the end of a run; what is beyond
  // kKeepBytes is freed.
  struct Scope {
    AdjointSystem* sys;
    explicit Scope(AdjointSystem* s) : sys(s) {}
    ~Scope() {
      if (sys->st) cudaStreamSynchronize(sys->st);
      size_t kept = 0;
      std::vector<Block> keep;
      for (auto& b : sys->work) {
        if (kept + b.size <= kKeepBytes) {
          kept += b.size;
          b.used = 0;
          keep.push_back(b);
        } else {
          cudaFree(b.p);
        }
      }
      sys->work.swap(keep);
    }
  };

  void checkOverflow() {
    int ov = 0;
    ACK(cudaMemcpyAsync(&ov, d_overflow, sizeof(int), cudaMemcpyDeviceToHost, st));
    ACK(cudaStreamSynchronize(st));
    if (ov) throw std::runtime_error("a particle has more than 32 contacts");
  }

  // State of one step of the forward model.
  template <typename T>
  struct State {
    T *x, *v, *w, *F, *Tq;
  };
  template <typename T>
  State<T> allocState() {
    State<T> S;
    for (T** p : {&S.x, &S.v, &S.w, &S.F, &S.Tq}) *p = scratch<T>(3 * (size_t)n);
    return S;
  }
  // Where the forward run is: positions, the velocities (closed: after the
  // step's closing kick, else the half-step ones), forces and torques.
  template <typename T>
  struct Point {
    const T *x, *v, *w;
    int closed;
    T *F, *Tq;
  };

  // Contact forces at positions x, whose cells are counted.
  template <typename T>
  void forces(const T* x, const T* vel, const T* omg, ListsT<T> const& prev, int has_prev,
              ListsT<T> const& cur, T* F, T* Tq, T kn, T en, T muc, int zero_spring) {
    k_adj_scan<<<1, 1024, 0, st>>>(G.ncells, d_count, d_start, d_cursor);
    k_adj_place<<<nblk(n), 128, 0, st>>>(n, d_cell, d_cursor, d_items);
    k_fwd_forces<T><<<laneBlocks(), kAdjBlock, 0, st>>>(n, A, G, d_type, x, vel, omg, prev,
                                                        has_prev, cur, F, Tq, kn, en, muc,
                                                        zero_spring, d_overflow);
  }

  // Leapfrog start: forces at (x0, v0, w0) with no history, spring zeroed.
  template <typename T>
  Point<T> start(State<T> const& S, ListsT<T> const& L, T kn, T en, T muc, int seed_v0 = -1) {
    const int n3 = 3 * n;
    // (a run that failed part way may have left counts behind)
    ACK(cudaMemsetAsync(d_count, 0, (size_t)G.ncells * sizeof(int), st));
    k_promote<T><<<nblk(n3), 128, 0, st>>>(n3, d_x0, S.x);
    k_promote<T><<<nblk(n3), 128, 0, st>>>(n3, d_v0, S.v);
    if (seed_v0 >= 0) k_seed<T><<<1, 1, 0, st>>>(S.v, seed_v0);
    k_promote<T><<<nblk(n3), 128, 0, st>>>(n3, d_w0, S.w);
    k_adj_bin<T><<<nblk(n), 128, 0, st>>>(n, G, S.x, d_cell, d_count);
    forces<T>(S.x, S.v, S.w, L, 0, L, S.F, S.Tq, kn, en, muc, 1);
    ACK(cudaGetLastError());
    return {S.x, S.v, S.w, 1, S.F, S.Tq};
  }
  // One step from P: move into (xs, vh, wh), then the forces there with
  // history prev -> cur; P becomes the new point, before its closing kick.
  template <typename T>
  void advance(Point<T>& P, T* xs, T* vh, T* wh, ListsT<T> const& prev, ListsT<T> const& cur,
               T kn, T en, T muc) {
    k_fwd_move<T><<<nblk(n), 128, 0, st>>>(n, A, G, d_type, P.closed, P.x, P.v, P.w, P.F, P.Tq, xs,
                                           vh, wh, d_cell, d_count);
    forces<T>(xs, vh, wh, prev, 1, cur, P.F, P.Tq, kn, en, muc, 0);
    ACK(cudaGetLastError());
    P.x = xs; P.v = vh; P.w = wh; P.closed = 0;
  }
  // The full state at P into S.
  template <typename T>
  void stateOf(Point<T> const& P, State<T> const& S) {
    k_fwd_state<T><<<nblk(n), 128, 0, st>>>(n, A, d_type, P.closed, P.x, P.v, P.w, P.F, P.Tq, S.x,
                                            S.v, S.w, S.F, S.Tq);
  }
  // Targets to the device (x, then v).
  double* targets(const double* tx, const double* tv) {
    const size_t n3 = 3 * (size_t)n;
    double* d = scratch<double>(2 * n3);
    ACK(cudaMemcpyAsync(d, tx, n3 * sizeof(double), cudaMemcpyHostToDevice, st));
    ACK(cudaMemcpyAsync(d + n3, tv, n3 * sizeof(double), cudaMemcpyHostToDevice, st));
    return d;
  }
  template <typename T>
  void lossOf(State<T> const& S, const double* dt, std::vector<T>& per) {
    T* out = scratch<T>(n);
    k_fwd_loss<T><<<nblk(n), 128, 0, st>>>(n, S.x, S.v, dt, dt + 3 * (size_t)n, out);
    per.resize(n);
    ACK(cudaMemcpyAsync(per.data(), out, n * sizeof(T), cudaMemcpyDeviceToHost, st));
    ACK(cudaStreamSynchronize(st));
  }
  // Two sets of the arrays a step moves into, used alternately.
  template <typename T>
  struct Pair {
    T *x[2], *v[2], *w[2];
  };
  template <typename T>
  Pair<T> allocPair() {
    Pair<T> b;
    for (int k = 0; k < 2; ++k)
      for (T** p : {&b.x[k], &b.v[k], &b.w[k]}) *p = scratch<T>(3 * (size_t)n);
    return b;
  }

  // Forward run (and, with gradients requested, the reverse sweep) in FP64.
  void run(int nsteps, int K, const double* p, const double* tx, const double* tv, double* loss,
           double* x_out, double* v_out, double* dLdp, double* dLdv0) {
    if (nsteps < 1 || K < 1) throw std::runtime_error("nsteps and the checkpoint interval must be >= 1");
    if (!d_type) throw std::runtime_error("set the particles first");
    Scope scope(this);
    const bool grads = dLdp || dLdv0;
    if ((grads || loss) && (!tx || !tv)) throw std::runtime_error("the loss needs target x and v");
    const double kn = p[0], en = p[1], muc = p[2];
    const size_t n3 = 3 * (size_t)n;
    ACK(cudaMemsetAsync(d_overflow, 0, sizeof(int), st));
    State<double> S = allocState<double>();
    Pair<double> B = allocPair<double>();
    ListsT<double> L[2] = {allocLists<double>(), allocLists<double>()};
    const int nseg = (nsteps + K - 1) / K;
    std::vector<State<double>> ck;
    std::vector<ListsT<double>> ckL;
    Point<double> P = start(S, L[0], kn, en, muc);
    auto checkpoint = [&](ListsT<double> const& lists) {
      ck.push_back(allocState<double>()); ckL.push_back(allocLists<double>());
      stateOf(P, ck.back()); copyLists(ckL.back(), lists);
    };
    if (grads) checkpoint(L[0]);
    for (int s = 1; s <= nsteps; ++s) {
      advance(P, B.x[s & 1], B.v[s & 1], B.w[s & 1], L[(s - 1) & 1], L[s & 1], kn, en, muc);
      if (grads && s % K == 0 && s < nsteps) checkpoint(L[s & 1]);
    }
    State<double> E = allocState<double>();
    stateOf(P, E);
    checkOverflow();
    if (x_out) ACK(cudaMemcpy(x_out, E.x, n3 * sizeof(double), cudaMemcpyDeviceToHost));
    if (v_out) ACK(cudaMemcpy(v_out, E.v, n3 * sizeof(double), cudaMemcpyDeviceToHost));
    double* target = nullptr;
    if (tx && tv) {
      target = targets(tx, tv);
      std::vector<double> per;
      lossOf(E, target, per);
      double Ls = 0.;
      for (double a : per) Ls += a;
      if (loss) *loss = Ls;
    }
    if (!grads) return;
    // ------------------------------------------------------ reverse sweep
    AdjState adj[2];
    AdjHist hist[2];
    const size_t nh = (size_t)n * kAdjCap * 3, nwh = (size_t)n * kAdjWalls * 3;
    for (int k = 0; k < 2; ++k) {
      for (double** a : {&adj[k].x, &adj[k].v, &adj[k].w, &adj[k].F, &adj[k].T})
        *a = scratch<double>(n3);
      hist[k].kd = scratch<double>(nh); hist[k].pn = scratch<double>(nh);
      hist[k].wkd = scratch<double>(nwh); hist[k].wpn = scratch<double>(nwh);
    }
    double* lp = scratch<double>(n3);
    // after the last step nothing depends on its history, w, F or T
    for (double* z : {hist[0].kd, hist[0].pn}) ACK(cudaMemsetAsync(z, 0, nh * sizeof(double), st));
    for (double* z : {hist[0].wkd, hist[0].wpn}) ACK(cudaMemsetAsync(z, 0, nwh * sizeof(double), st));
    for (double* z : {adj[0].w, adj[0].F, adj[0].T, lp}) ACK(cudaMemsetAsync(z, 0, n3 * sizeof(double), st));
    k_bwd_seed<<<nblk(n), 128, 0, st>>>(n, E.x, E.v, target, target + n3, adj[0].x, adj[0].v);
    // per-step storage of one segment
    const int len = std::min(K, nsteps);
    std::vector<double*> Xs(len + 1), Vh(len + 1), Wh(len + 1);
    std::vector<ListsT<double>> Ls(len + 1);
    for (int k = 1; k <= len; ++k) {
      Xs[k] = scratch<double>(n3); Vh[k] = scratch<double>(n3); Wh[k] = scratch<double>(n3);
      Ls[k] = allocLists<double>();
    }
    int cur = 0;
    for (int seg = nseg - 1; seg >= 0; --seg) {
      const int c = seg * K, e = std::min(c + K, nsteps);
      Ls[0] = ckL[seg];
      // (the step's forces overwrite F, T: those of a checkpoint are not needed again)
      Point<double> R{ck[seg].x, ck[seg].v, ck[seg].w, 1, ck[seg].F, ck[seg].Tq};
      for (int s = c + 1; s <= e; ++s)
        advance(R, Xs[s - c], Vh[s - c], Wh[s - c], Ls[s - c - 1], Ls[s - c], kn, en, muc);
      for (int s = e; s >= c + 1; --s) {
        k_bwd_step<<<laneBlocks(), kAdjBlock, 0, st>>>(
            n, A, d_type, Xs[s - c], Vh[s - c], Wh[s - c], Ls[s - c - 1], 1, Ls[s - c], adj[cur],
            adj[cur ^ 1], hist[cur], hist[cur ^ 1], lp, kn, en, muc, 0);
        ACK(cudaGetLastError());
        cur ^= 1;
      }
    }
    // leapfrog start: forces at (x0, v0, w0), the spring it leaves is zeroed
    k_bwd_step<<<laneBlocks(), kAdjBlock, 0, st>>>(n, A, d_type, d_x0, d_v0, d_w0, ckL[0], 0, ckL[0],
                                                   adj[cur], adj[cur ^ 1], hist[cur], hist[cur ^ 1],
                                                   lp, kn, en, muc, 1);
    ACK(cudaGetLastError());
    std::vector<double> hp(n3);
    if (dLdv0) ACK(cudaMemcpyAsync(dLdv0, adj[cur ^ 1].v, n3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    ACK(cudaMemcpyAsync(hp.data(), lp, n3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    ACK(cudaStreamSynchronize(st));
    checkOverflow();
    if (dLdp) {
      dLdp[0] = dLdp[1] = dLdp[2] = 0.;
      for (int t = 0; t < n; ++t)
        for (int d = 0; d < 3; ++d) dLdp[d] += hp[3 * (size_t)t + d];
    }
  }

  // Forward-mode derivative of the loss: the whole forward run on Dual<3>
  // numbers seeded on (kn, en, muc), or, with seed_particle >= 0, on the one
  // initial velocity component (seed_particle, seed_component) in slot 0.
  void forwardDual(int nsteps, const double* p, const double* tx, const double* tv,
                   double* loss, double* dLdp, int seed_particle, int seed_component) {
    using D = Dual<3>;
    if (nsteps < 1) throw std::runtime_error("nsteps must be >= 1");
    if (!tx || !tv) throw std::runtime_error("the loss needs target x and v");
    if (!d_type) throw std::runtime_error("set the particles first");
    Scope scope(this);
    ACK(cudaMemsetAsync(d_overflow, 0, sizeof(int), st));
    D kn = dconst<3>(p[0]), en = dconst<3>(p[1]), muc = dconst<3>(p[2]);
    const bool seed_v = seed_particle >= 0;
    if (seed_v && (seed_particle >= n || seed_component < 0 || seed_component > 2))
      throw std::runtime_error("seed out of range");
    if (!seed_v) { kn.d[0] = 1.; en.d[1] = 1.; muc.d[2] = 1.; }
    State<D> S = allocState<D>();
    Pair<D> B = allocPair<D>();
    ListsT<D> L[2] = {allocLists<D>(), allocLists<D>()};
    Point<D> P = start(S, L[0], kn, en, muc, seed_v ? 3 * seed_particle + seed_component : -1);
    for (int s = 1; s <= nsteps; ++s)
      advance(P, B.x[s & 1], B.v[s & 1], B.w[s & 1], L[(s - 1) & 1], L[s & 1], kn, en, muc);
    State<D> E = allocState<D>();
    stateOf(P, E);
    checkOverflow();
    std::vector<D> per;
    lossOf(E, targets(tx, tv), per);
    double Lv = 0., g[3] = {0., 0., 0.};
    for (auto const& a : per) {
      Lv += a.v;
      for (int d = 0; d < 3; ++d) g[d] += a.d[d];
    }
    if (loss) *loss = Lv;
    if (dLdp) {
      if (seed_v) dLdp[0] = g[0];
      else for (int d = 0; d < 3; ++d) dLdp[d] = g[d];
    }
  }
};

}  // namespace
}  // namespace gdem

// ----------------------------------------------------------------- C ABI --
using namespace gdem;

namespace {
template <typename F>
int adjGuarded(F&& f) {
  try {
    f();
    return GDEM_OK;
  } catch (AdjCheck const& e) {
    setLastError(e.what());
    return GDEM_ERR_CUDA;
  } catch (std::exception const& e) {
    setLastError(e.what());
    return GDEM_ERR_INVALID;
  }
}
AdjointSystem* adj(gdem_adjoint_handle h) { return reinterpret_cast<AdjointSystem*>(h); }
}  // namespace

extern "C" {

int gdem_adjoint_create(const char* xml_path, gdem_adjoint_handle* out) {
  return adjGuarded([&] {
    if (!xml_path || !out) throw std::runtime_error("invalid arguments");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
      throw AdjCheck("no CUDA device: the adjoint has no CPU fallback");
    auto s = std::make_unique<AdjointSystem>();
    s->create(xml_path);
    *out = reinterpret_cast<gdem_adjoint_handle>(s.release());
  });
}

int gdem_adjoint_set_particles(gdem_adjoint_handle h, int64_t n, const int* type,
                               const double* x0, const double* v0, const double* w0) {
  return adjGuarded([&] {
    if (!h || !type || !x0 || !v0) throw std::runtime_error("invalid arguments");
    adj(h)->setParticles(n, type, x0, v0, w0);
  });
}

int gdem_adjoint_run(gdem_adjoint_handle h, int nsteps, int checkpoint_every,
                     const double* params, const double* target_x, const double* target_v,
                     double* loss, double* x_out, double* v_out, double* dL_dparams,
                     double* dL_dv0) {
  return adjGuarded([&] {
    if (!h || !params) throw std::runtime_error("invalid arguments");
    adj(h)->run(nsteps, checkpoint_every, params, target_x, target_v, loss, x_out, v_out,
                dL_dparams, dL_dv0);
  });
}

int gdem_adjoint_forward_dual(gdem_adjoint_handle h, int nsteps, const double* params,
                              const double* target_x, const double* target_v,
                              int seed_particle, int seed_component, double* loss,
                              double* dL_dseed) {
  return adjGuarded([&] {
    if (!h || !params) throw std::runtime_error("invalid arguments");
    adj(h)->forwardDual(nsteps, params, target_x, target_v, loss, dL_dseed, seed_particle,
                        seed_component);
  });
}

void gdem_adjoint_destroy(gdem_adjoint_handle h) { delete adj(h); }

}  // extern "C"
