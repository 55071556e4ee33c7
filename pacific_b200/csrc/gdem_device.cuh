// gdem_device.cuh -- device-side state and helpers for the Grains3D DEM step.
#pragma once
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include "gdem_types.h"

namespace gdem {

// Contact memory.  It lives beside what uses it: per pair of the compact pair
// list and per (particle, wall) of the wall list (MemView), where the
// pair kernel's lanes read and write it in list order.  Values are as seen
// from the lower-ID body (or the particle, for a wall); the other body's view
// is the negation, as in the reference where p1 holds (-kdelta, -normal,
// -spring) (HookeMemoryContactForceModel.cpp:191-192).  An entry carries the
// evaluation that last wrote it: the plain step uses it when that is the
// evaluation before, so entries not touched in a step disappear, which is what
// Component::updateContactMap (Component.cpp:583-595) does; the coupled step
// uses it whenever it was ever written.
//
// HistTable carries the memory across what changes the lists (a rebuild, a
// new state, a larger allocation) and in and out of the library: open
// addressing with linear probing, keyed on the unordered particle pair or on
// (particle, wall).  The plain step's table is emptied before the lists are
// saved into it; the coupled step's keeps the entries of every pair that ever
// touched.  (The table used to be read and written by every evaluation, at
// random places of two tables: 1M spheres 5 of the pair kernel's 24 us, a
// packed bed two thirds of its memory traffic.)
//
// Key layout: bits 27-53 the lower particle ID, bits 0-26 the higher particle
// ID or, for a wall, 2^27 - 1 - wall index; kEmptyKey in a free slot.
constexpr int kMaxIdBits = 27;
constexpr unsigned long long kEmptyKey = 0xFFFFFFFFFFFFFFFFull;

struct HistTable {
  unsigned long long* keys;
  void* vals;            // 9 values per slot (kdelta, prev normal, spring torque)
  int log2cap;
};

__host__ __device__ inline unsigned long long pairKey(int ida, int idb) {
  return ((unsigned long long)(uint32_t)ida << kMaxIdBits) | (uint32_t)idb;
}
__host__ __device__ inline unsigned long long wallKey(int id, int wall) {
  return ((unsigned long long)(uint32_t)id << kMaxIdBits) |
         (uint32_t)((1 << kMaxIdBits) - 1 - wall);
}
__host__ __device__ inline uint32_t hashSlot(unsigned long long k, int log2cap) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return (uint32_t)(k & ((1ull << log2cap) - 1));
}
// Slot holding key, or -1.
__device__ inline int histFind(HistTable const& t, unsigned long long key) {
  const uint32_t mask = (1u << t.log2cap) - 1;
  uint32_t s = hashSlot(key, t.log2cap);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const unsigned long long k = t.keys[s];
    if (k == key) return (int)s;
    if (k == kEmptyKey) return -1;
    s = (s + 1) & mask;
  }
  return -1;
}
// The slot of key, claimed if need be (one writer per key at a time); -1 when
// the table is full.
__device__ inline int histInsert(HistTable const& t, unsigned long long key) {
  const uint32_t mask = (1u << t.log2cap) - 1;
  uint32_t s = hashSlot(key, t.log2cap);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    unsigned long long cur = t.keys[s];
    if (cur == kEmptyKey) cur = atomicCAS(&t.keys[s], kEmptyKey, key);
    if (cur == kEmptyKey || cur == key) return (int)s;
    s = (s + 1) & mask;
  }
  return -1;
}

// Contact memory in list order: n entries in planes of vectors, so that
// neighbouring entries' loads coalesce.  FP32: (kdelta, evaluation),
// (normal, spring x), (spring y, z); FP64: five pairs of doubles in the same
// order.  The last plane (spring y, z) only matters with rolling resistance.
struct MemView {
  void* p;
  long long n;
};
constexpr size_t kMemBytes32 = 40, kMemBytes64 = 80;
__device__ __forceinline__ int memLoad(MemView m, long long i, float* v, bool spring) {
  const float4* A = static_cast<const float4*>(m.p);
  const float4 a = A[i], b = A[m.n + i];
  v[0] = a.x; v[1] = a.y; v[2] = a.z;
  v[3] = b.x; v[4] = b.y; v[5] = b.z; v[6] = b.w;
  if (spring) {
    const float2 c = reinterpret_cast<const float2*>(A + 2 * m.n)[i];
    v[7] = c.x; v[8] = c.y;
  }
  return __float_as_int(a.w);
}
__device__ __forceinline__ void memStore(MemView m, long long i, const float* v, int evaluation,
                                         bool spring) {
  float4* A = static_cast<float4*>(m.p);
  A[i] = make_float4(v[0], v[1], v[2], __int_as_float(evaluation));
  A[m.n + i] = make_float4(v[3], v[4], v[5], v[6]);
  if (spring) reinterpret_cast<float2*>(A + 2 * m.n)[i] = make_float2(v[7], v[8]);
}
__device__ __forceinline__ int memLoad(MemView m, long long i, double* v, bool spring) {
  const double2* A = static_cast<const double2*>(m.p);
  const double2 a = A[i], b = A[m.n + i], c = A[2 * m.n + i], d = A[3 * m.n + i];
  v[0] = a.x; v[1] = a.y; v[2] = b.x;
  v[3] = c.x; v[4] = c.y; v[5] = d.x; v[6] = d.y;
  if (spring) {
    const double2 e = A[4 * m.n + i];
    v[7] = e.x; v[8] = e.y;
  }
  return (int)__double_as_longlong(b.y);
}
__device__ __forceinline__ void memStore(MemView m, long long i, const double* v, int evaluation,
                                         bool spring) {
  double2* A = static_cast<double2*>(m.p);
  A[i] = make_double2(v[0], v[1]);
  A[m.n + i] = make_double2(v[2], __longlong_as_double((long long)evaluation));
  A[2 * m.n + i] = make_double2(v[3], v[4]);
  A[3 * m.n + i] = make_double2(v[5], v[6]);
  if (spring) A[4 * m.n + i] = make_double2(v[7], v[8]);
}
// The evaluation that last wrote entry i (-1: none), and marking it so.
__device__ __forceinline__ int memEvaluation(MemView m, long long i, float) {
  return __float_as_int(static_cast<const float4*>(m.p)[i].w);
}
__device__ __forceinline__ int memEvaluation(MemView m, long long i, double) {
  return (int)__double_as_longlong(static_cast<const double2*>(m.p)[m.n + i].y);
}
__device__ __forceinline__ void memForget(MemView m, long long i, float) {
  static_cast<float4*>(m.p)[i].w = __int_as_float(kNeverWritten);
}
__device__ __forceinline__ void memForget(MemView m, long long i, double) {
  static_cast<double2*>(m.p)[m.n + i].y = __longlong_as_double((long long)kNeverWritten);
}

// Overlap statistics of the contacts over the evaluations since the last
// reset (AppCollision::addToContactsFeatures, Base/src/AppCollision.cpp:
// 159-179): the sum and the count of |overlap| over the contacts (pairs and
// walls, each once per evaluation), the largest |overlap| (its FP64 bits:
// non-negative doubles order like their bit patterns) and the evaluation
// counter at which it was first reached.
struct ContactStats {
  double sum;
  unsigned long long count;
  unsigned long long max_bits;
  long long max_epoch;
};

// Whole device state of one batch of instances.  Per-particle arrays are in
// the current sorted (cell) order; component d of particle s of an n-vector
// field lives at [d * cap + s] (structure of arrays).
struct DevState {
  int n;                  // particles
  int cap;                // allocated particles (component stride)
  int ncells;             // total cell keys of all instances (pair-list grids)
  int ninst;
  double dt;
  int* id; int* type; int* inst;
  double* x; double* v; double* w; double* wbf; double* q; double* F; double* T;
  // wbf_state: w_bf is integrated (FP64 mode, or convex bodies present);
  // otherwise (FP32-split, spheres only) w is the angular state and w_bf is
  // derived on output as q* w q
  int wbf_state;
  double* basis;          // 9 per particle, non-spherical shapes only
  // second buffers: a step reads x, v, w, w_bf, q, basis and writes x2 ...;
  // a pair-list rebuild permutes everything into them and copies back
  int* id2; int* type2; int* inst2;
  double* x2; double* v2; double* w2; double* wbf2; double* q2; double* basis2;
  double* F2; double* T2;
  // pair-list validity: the FP32 position at the last rebuild (the posf
  // value written then; displacement = posf - posf0) and the periodic wraps
  // since then (signed bytes x, y, z)
  float4* posf0; int* wrap; int* wrap2;
  int* ctl;               // control words (CtlWords)
  // binning
  int* skey;              // cell key in the old order
  int* rank;              // arrival rank within the cell
  int* cell_count; int* cell_start; int* order;
  int* scan_tmp;
  // compact copies for the contact kernels (sorted order)
  double4* pos64;         // x, y, z, radius
  double4* vel64;         // v, mass
  double4* omg64;         // w (space frame), equivalent radius
  float4* offh;           // FP32 cell-relative offset; FP32 radius
  int4* cellc;            // pair-list cell i, j, k and instance at the last rebuild
  // skin pair list, compressed rows: the entries of slot t are
  // pairs[pair_off[t] .. pair_off[t] + npairs[t]), pair_off the exclusive
  // scan of npairs; pair_cap entries are allocated (kCtlEntries holds the
  // total of the last rebuild)
  int* pairs; int* npairs; int* pair_off;
  int pair_cap;
  // candidates found by the counting pass of a rebuild, kCandKept per particle
  // ([k * cap + t]; the download staging, free during a step)
  int* cand;
  int* pair_scan_tmp;     // tile sums of the pair-count scan
  double* hydro;          // coupled runs: hydrodynamic force and torque by particle ID (6 each), or null
  int2* upairs;           // compact pair list: (slot, entry) of every upper entry, ctl[kCtlPairs] of them
  int* epos;              // per compact pair: position of the pair in its two rows, e_t | e_u << 16
  // compact-list indices of the pairs kept by the filter: ctl[kCtlKept] from
  // the front and, in FP32-split with non-spherical classes, the pairs not in
  // contact at the last evaluation, ctl[kCtlKeptCold], from slot pair_cap / 2
  // downwards
  int* kept;
  int* kept2;             // the cold pairs k_pairsep32 left undecided, ctl[kCtlKept2]
  // per list entry: this evaluation's force and torque on the row's particle
  // from that pair (written by the pair kernel for a contact, tagged with the
  // evaluation counter), summed in row order by the leapfrog kernel
  void* share;
  // wall list (rebuilt with the pair list): a slot per (particle, wall) that
  // can come near one another before the next rebuild, a particle's slots
  // together and in wall order; each particle's first slot and number of
  // slots; per slot the contact memory and this evaluation's share
  int2* wlist; int2* wrow;
  int wall_cap;           // slots allocated
  void* wshare;           // kWallShare vectors per slot
  int* nact;              // flag words, two buffers of cap (contactFlags)
  float4* posf;           // FP32 continuous position since the last rebuild + circumscribed radius
  // this evaluation's wall items, ctl[kCtlWork]: slots of the wall list
  // (spheres) or, with non-spherical classes, the first slots of its particles
  int* work;
  int nsm;                // multiprocessors of the device (persistent grids)
  int forces_bps;         // blocks per multiprocessor of the pair kernel's persistent grid (0: the default)
  double* pair_delta;     // diagnostics: overlap of each entry (+inf: no contact)
  double* wall_delta;     // diagnostics: overlap with each wall slot
  double* pair_force;     // diagnostics: contact force on the lower ID (3 per entry)
  unsigned long long* gjk_counts;   // convex: GJK calls, iterations, most iterations of a call
  unsigned long long* law_counts;   // FP32-split: contacts evaluated, re-evaluated in FP64
  ContactStats* cstats;   // overlap statistics over all evaluations
  double* wall_force;     // diagnostics: wall contact force on the particle (3 per slot)
  int diag;
  MemView pmem, wmem;     // contact memory of the pair list and of the wall list
  HistTable hist;         // the memory across rebuilds
  int prune;              // memory of ended contacts is dropped (the plain step)
  int* status;
  GridDesc const* grids;  // reference linked-cell grids (cell reports, periodic wrap)
  GridDesc const* bgrids; // pair-list grids: cells at least 2 rmax + skin wide
  TypeDesc const* types; ModelDesc const* models;
  WallDesc const* walls;
  const double* poly_verts;   // polyhedron vertices of all classes (x, y, z)
  const int* poly_adj_off;    // vertex graph of the polyhedra: per global vertex, its first neighbour
  const int* poly_adj;        // neighbours (vertex indices within their polyhedron)
  // current polyhedron vertex of each particle (Polyhedron::m_curr_vertex),
  // its permutation buffer, and the record this evaluation's GJK calls leave
  // (0: none; else priority << 16 | vertex, see recordVertex)
  int* curv; int* curv2; int* curv_next;
  int max_walls;          // walls of the largest instance
  int any_convex;         // some class is not a sphere (GJK narrow phase)
  int any_poly;           // some class is a polyhedron (carried support vertices)
  int any_walls;          // some instance has walls
  float filt_margin_max;  // largest contact-filter margin of the instances
  int filter_qblocks;     // contact filter: blocks for the pairs (0: from the particle count)
  int filter_wblocks;     // and for the wall list
};

// ----------------------------------------------------------- FP64 helpers --
struct d3 { double x, y, z; };
__device__ __forceinline__ d3 mk(double a, double b, double c) { d3 r; r.x = a; r.y = b; r.z = c; return r; }
__device__ __forceinline__ d3 operator+(d3 a, d3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ d3 operator-(d3 a) { return mk(-a.x, -a.y, -a.z); }
__device__ __forceinline__ d3 operator*(d3 a, double s) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ d3 operator*(double s, d3 a) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ d3 operator/(d3 a, double s) { return mk(a.x / s, a.y / s, a.z / s); }
__device__ __forceinline__ double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// Vector3::operator^ (Geometry/src/Vector3.cpp:114-119)
__device__ __forceinline__ d3 cross(d3 a, d3 b) {
  return mk(a.y * b.z - a.z * b.y, -a.x * b.z + a.z * b.x, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double norm(d3 a) { return sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
__device__ __forceinline__ d3 ld3(const double* p, int cap, int s) {
  return mk(p[s], p[cap + s], p[2 * cap + s]);
}
__device__ __forceinline__ void st3(double* p, int cap, int s, d3 a) {
  p[s] = a.x; p[cap + s] = a.y; p[2 * cap + s] = a.z;
}

struct dq { d3 v; double w; };
__device__ __forceinline__ dq qmk(d3 v, double w) { dq q; q.v = v; q.w = w; return q; }
__device__ __forceinline__ dq conj(dq q) { return qmk(-q.v, q.w); }
// Quaternion::operator* (Geometry/src/Quaternion.cpp:442-448)
__device__ __forceinline__ dq qmul(dq a, dq b) {
  double t = (a.w * b.w) - dot(a.v, b.v);
  d3 vt = (cross(a.v, b.v) + (a.w * b.v)) + (b.w * a.v);
  return qmk(vt, t);
}
// operator,(Vector3, Quaternion) = q.multLeftVec(lhs) (Quaternion.cpp:93-98)
__device__ __forceinline__ dq vecq(d3 l, dq q) {
  double t = dot(-l, q.v);
  d3 vt = cross(l, q.v) + (l * q.w);
  return qmk(vt, t);
}
// Quaternion::multToVector3 (Quaternion.cpp:108-113)
__device__ __forceinline__ d3 multToVector3(dq a, dq r) {
  return (cross(a.v, r.v) + (a.w * r.v)) + (r.w * a.v);
}
// Quaternion::setRotFromTwoVectors (Quaternion.cpp:263-288)
__device__ __forceinline__ dq rotFromTwoVectors(d3 u, d3 v) {
  double nn = sqrt(dot(u, u) * dot(v, v));
  double real = nn + dot(u, v);
  d3 vect;
  if (real < 1.e-6 * nn) {
    real = 0.;
    vect = fabs(u.x) > fabs(u.z) ? mk(-u.y, u.x, 0.) : mk(0., -u.z, u.y);
  } else {
    vect = cross(u, v);
  }
  double nq = sqrt(vect.x * vect.x + vect.y * vect.y + vect.z * vect.z + real * real);
  double s = 1. / nq;
  return qmk(vect * s, real * s);
}
// Quaternion::rotateVector (Quaternion.cpp:293-299)
__device__ __forceinline__ d3 rotateVector(dq q, d3 v) {
  double nv = norm(q.v);
  return ((q.w * q.w - nv * nv) * v + (2. * dot(v, q.v)) * q.v) + (2. * q.w) * cross(q.v, v);
}

__device__ __forceinline__ void raise(int* status, int bits) { atomicOr(status, bits); }

// 16-byte words of a wall share: force with the evaluation tag, torque of the
// lever arm with a rolling flag, rolling torque.
constexpr int kWallShare32 = 3, kWallShare64 = 6;

// Pairs of the compact list whose entries are allocated.
__device__ __forceinline__ int listedPairs(DevState const& S) {
  return (int)min((long long)S.ctl[kCtlPairs], S.pmem.n);
}
__device__ __forceinline__ int listedWalls(DevState const& S) {
  return min(S.ctl[kCtlWallSlots], S.wall_cap);
}
__device__ __forceinline__ bool remembered(DevState const& S, int e, int now) {
  return memoryHolds(S.prune, e, now);
}

// Cell of a neighbour offset (di, dj, dk) around (i, j, k) of grid g, with
// the periodic minimum-image wrap.  Returns the global cell key or -1, and the
// image shift (in units of the period) of the particles found there.
__device__ __forceinline__ int neighbourKey(GridDesc const& g, int i, int j, int k,
                                            int di, int dj, int dk, int* sh) {
  int c[3] = {i + di, j + dj, k + dk};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    sh[d] = 0;
    if (g.periodic[d]) {
      int nin = g.nb[d] - 2;
      if (c[d] < 1) { c[d] += nin; sh[d] = -1; }
      else if (c[d] > nin) { c[d] -= nin; sh[d] = 1; }
    } else if (c[d] < 0 || c[d] >= g.nb[d]) {
      return -1;
    }
  }
  return g.cell_offset + c[1] * g.nb[2] * g.nb[0] + c[2] * g.nb[0] + c[0];
}

// Enumerates the particles of the 27 cells around cell cc (i, j, k, inst),
// row by row: for each of the 9 (dj, dk) rows the cells i-1, i, i+1 are
// consecutive in the cell numbering, so their particles are one contiguous
// slot range [cell_start[i-1], cell_start[i+2]); the cell of a candidate
// within the row follows from two boundaries.  In a periodic x direction the
// two extra layers are empty and the wrapped neighbour cell is visited
// separately.  fn(u, dcx, dj, dk, shx, shy, shz) receives the candidate slot,
// its cell offset and the periodic image shift (in periods); the centre
// particle itself is included.
template <typename Fn>
__device__ __forceinline__ void forEachCandidate(const int* __restrict__ cs, GridDesc const& g,
                                                 int4 cc, Fn&& fn) {
  const int nbx = g.nb[0];
  for (int dj = -1; dj <= 1; ++dj) {
    int jj = cc.y + dj, shy = 0;
    if (g.periodic[1]) {
      int nin = g.nb[1] - 2;
      if (jj < 1) { jj += nin; shy = -1; } else if (jj > nin) { jj -= nin; shy = 1; }
    } else if (jj < 0 || jj >= g.nb[1]) {
      continue;
    }
    for (int dk = -1; dk <= 1; ++dk) {
      int kk = cc.z + dk, shz = 0;
      if (g.periodic[2]) {
        int nin = g.nb[2] - 2;
        if (kk < 1) { kk += nin; shz = -1; } else if (kk > nin) { kk -= nin; shz = 1; }
      } else if (kk < 0 || kk >= g.nb[2]) {
        continue;
      }
      const int row = g.cell_offset + jj * g.nb[2] * nbx + kk * nbx;
      int ilo = cc.x - 1, ihi = cc.x + 1;
      if (!g.periodic[0]) { ilo = max(ilo, 0); ihi = min(ihi, nbx - 1); }
      const int b0 = cs[row + ilo], b1 = cs[row + cc.x], b2 = cs[row + cc.x + 1],
                b3 = cs[row + ihi + 1];
#pragma unroll 4
      for (int u = b0; u < b3; ++u) fn(u, u < b1 ? -1 : (u < b2 ? 0 : 1), dj, dk, 0, shy, shz);
      if (g.periodic[0]) {
        const int nin = nbx - 2;
        if (cc.x == 1) {
          const int e0 = cs[row + nin], e1 = cs[row + nin + 1];
          for (int u = e0; u < e1; ++u) fn(u, -1, dj, dk, -1, shy, shz);
        }
        if (cc.x == nin) {
          const int e0 = cs[row + 1], e1 = cs[row + 2];
          for (int u = e0; u < e1; ++u) fn(u, 1, dj, dk, 1, shy, shz);
        }
      }
    }
  }
}

// Orders a particle's list entries by partner ID, the partners with a
// higher ID than the particle's own (idt) first, and returns how many those
// are.  The reduction order of its forces then does not depend on the cells
// at the last rebuild (nor on when the list was rebuilt), and the contact
// filter tests each pair once, from the lower ID's "upper" entries.
__device__ __forceinline__ int sortEntriesUpperFirst(int* seg, int cnt, const int* id, int idt) {
  auto key = [&](int e) {
    const int idu = id[e & ((1 << 27) - 1)];
    return idu > idt ? idu : (1 << 30) | idu;
  };
  int nup = 0;
  for (int i = 0; i < cnt; ++i) {
    const int e = seg[i];
    const int ke = key(e);
    if (ke < (1 << 30)) ++nup;
    int j = i - 1;
    while (j >= 0 && key(seg[j]) > ke) {
      seg[j + 1] = seg[j];
      --j;
    }
    seg[j + 1] = e;
  }
  return nup;
}

// The same for a row of at most kSortKept entries given by load(k), in
// registers: each entry goes to its rank.  (The insertion sort above reads IDs
// and entries from memory at every comparison.)
constexpr int kSortKept = 12;
template <typename Load>
__device__ __forceinline__ int rankEntriesUpperFirst(int* seg, int cnt, const int* id, int idt,
                                                     Load&& load) {
  int e[kSortKept], key[kSortKept];
  int nup = 0;
#pragma unroll
  for (int k = 0; k < kSortKept; ++k) {
    key[k] = INT_MAX;
    if (k < cnt) e[k] = load(k);
  }
#pragma unroll
  for (int k = 0; k < kSortKept; ++k) {
    if (k < cnt) {
      const int idu = id[e[k] & ((1 << 27) - 1)];
      key[k] = idu > idt ? idu : (1 << 30) | idu;
      nup += idu > idt ? 1 : 0;
    }
  }
#pragma unroll
  for (int k = 0; k < kSortKept; ++k) {
    int rank = 0;
#pragma unroll
    for (int j = 0; j < kSortKept; ++j)
      rank += (key[j] < key[k] || (j < k && key[j] == key[k])) ? 1 : 0;
    if (k < cnt) seg[rank] = e[k];
  }
  return nup;
}

// Candidates per particle the counting pass keeps for the filling one (of the
// 44 ints the staging has room for): a longer row is searched again.
constexpr int kCandKept = 44;

// Row length of a particle with cnt candidates: at most kRowMax (an entry's
// position in its row is kept in 16 bits); more raises kErrPairsFull.
__device__ __forceinline__ int rowLength(DevState const& S, int cnt) {
  if (cnt > kRowMax) {
    raise(S.status, kErrPairsFull);
    return kRowMax;
  }
  return cnt;
}
// Whether slot t's row, placed by the scan of the row lengths, lies inside
// the allocation of the pair list; with one that does not the evaluation is
// put off until the host has enlarged it.
__device__ __forceinline__ bool rowFits(DevState const& S, int t) {
  const int off = S.pair_off[t];   // negative when the scan's total overflowed
  if (off >= 0 && (long long)off + S.npairs[t] <= (long long)S.pair_cap) return true;
  S.npairs[t] = 0;
  S.ctl[kCtlNeed] = kPutOff;
  return false;
}

// Appends the first nu entries of slot t's row (seg) to the compact pair
// list (one atomic per warp), with each entry's position in the row.  Every
// lane of the warp calls it; valid lanes only contribute.
__device__ __forceinline__ void appendUpperPairs(DevState const& S, int t, const int* seg, int nu) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int incl = nu;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += y;
  }
  const int total = __shfl_sync(full, incl, 31);
  if (!total) return;
  int base = 0;
  if (lane == 31) base = atomicAdd(&S.ctl[kCtlPairs], total);
  base = __shfl_sync(full, base, 31);
  const long long cap = (long long)S.pair_cap / 2 + 1;
  if (base + (long long)total > cap) {
    if (lane == 0) S.ctl[kCtlNeed] = kPutOff;
    return;
  }
  const int first = base + incl - nu;
  for (int e = 0; e < nu; ++e) {
    S.upairs[first + e] = make_int2(t, seg[e]);
    S.epos[first + e] = e;
  }
}

// Programmatic dependent launch (sm_90 and later): a kernel launched with
// the programmatic-serialization attribute (launchAfterPrevious) may start
// while the previous kernel of its stream still runs.  pdlWait() returns once
// that kernel has completed and its writes are visible (at once for a kernel
// launched without the attribute); pdlTrigger() lets the next kernel start
// early.  Everything a kernel reads that its predecessor writes, and all its
// writes, come after its pdlWait().
__device__ __forceinline__ void pdlWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdlTrigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Which of n items the lanes of a warp take: `lanes` consecutive ones per warp
// (lane < lanes), from first on, every stride.  No more items than the grid
// has warps go one to a warp instead of filling the first few: an item is a
// chain of dependent latencies, and lanes on different branches of it take
// turns (200 packed spheres, 680 items: step 43.2 -> 35.5 us).  A few lanes
// per warp for more items cost more than they gave (7,777 spheres 35.4 ->
// 39.5 us, the 1M gas's pair kernel 20.9 -> 24.2 us): every warp on every
// multiprocessor fetches the whole law's instructions.
struct WarpItems {
  int lanes, first, stride;
};
__device__ __forceinline__ WarpItems warpItems(int n) {
  const int warps = (int)(gridDim.x * blockDim.x) >> 5;
  const int warp = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lanes = n <= warps ? 1 : 32;
  return {lanes, warp * lanes, warps * lanes};
}

// Contact-filter flags of the current force evaluation: two buffers used
// alternately, the leapfrog kernel of one evaluation clearing the other's, so
// that no kernel needs to clear flags that other warps may still be setting.
__device__ __forceinline__ int* contactFlags(DevState const& S, int which = 0) {
  return S.nact + (size_t)(((unsigned)S.ctl[kCtlEpoch] + (unsigned)which) & 1u) * S.cap;
}

// Code of a periodic image shift (in periods, each -1, 0 or 1) in 0..26.
__device__ __forceinline__ int shiftCode(int sx, int sy, int sz) {
  return (sx + 1) + 3 * (sy + 1) + 9 * (sz + 1);
}

// Code of a stencil offset in 0..26 and back.
__device__ __forceinline__ int offCode(int di, int dj, int dk) { return (di + 1) + 3 * (dk + 1) + 9 * (dj + 1); }
__device__ __forceinline__ void offDecode(int c, int* di, int* dj, int* dk) {
  *di = c % 3 - 1; *dk = (c / 3) % 3 - 1; *dj = c / 9 - 1;
}

}  // namespace gdem
