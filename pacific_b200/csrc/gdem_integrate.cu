// gdem_integrate.cu -- leapfrog move and pair-list rebuild kernels.
//
// Compiled with -fmad=false: positions, velocities and cell indices are FP64
// and follow the reference's expression order, so cell assignments are
// bit-identical to Cell::GetCell on the same state.
//
// A step is (host side, gdem_host.cu): k_decide, then -- only when some
// particle has moved more than half the pair-list skin since the last
// rebuild -- the rebuild below, then k_filter, the force kernel
// (gdem_contact64.cu / gdem_contact32.cu) and k_move.
//
//   k_decide    turns the rebuild request of the previous step into this
//               step's decision (and the CUDA-graph condition), and counts
//               the force evaluation (tag of shares and contact memory).
//   k_bin       pair-list cell of each particle and the cell histogram.
//   scan/place/cellsort
//               counting sort of particles on their cell key: a one-digit
//               radix sort whose digit is the cell key, made stable by
//               ordering each cell's entries by particle ID; it yields the
//               cell start/end tables.
//   k_permute / k_copyback
//               the whole state into cell order (through the second
//               buffers), with the compact copies the pair search reads.
//   k_pairs_*   (gdem_contact64/32.cu) the rows of the skin pair list:
//               counted, placed by a scan of the counts, written; k_link
//               then records where each pair of the compact list sits in
//               its partner's row, and k_wall_rows lists the (particle, wall)
//               pairs within the skin.
//   k_mem_*     the contact memory from the old lists through its table into
//               the new ones.
//   k_filter    lists the pairs of the skin list whose bounding spheres
//               overlap now, and the wall-list slots that are near, and marks
//               their particles as candidates; the pair kernel (gdem_contact64/32.cu)
//               evaluates them exactly and writes each contact's two shares
//               into the partners' rows.
//   k_move      the leapfrog of each particle in place: its force and torque
//               as the weight plus its shares in row order, then the closing
//               kick of the step that ends and the opening kick + drift of
//               the next (SecondOrderLeapFrog::Move / advanceVelocity,
//               ParticleKinematics::Move).
// Rebuild kernels take a gate: with a non-null gate they return at once
// unless this step rebuilds (plain launches); inside the graph's conditional
// node they run ungated.
#include <algorithm>

#include "gdem_kernels.cuh"
#include "gdem_motion.cuh"

namespace gdem {

namespace {

__device__ __forceinline__ bool gatedOff(const int* gate) { return gate && !*gate; }

// Most rounds of 32 pairs a warp of the contact filter takes per append.
constexpr int kFilterRounds = 8;

__global__ void k_decide(DevState S, cudaGraphConditionalHandle h, int use_handle) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int need = S.ctl[kCtlNeed];
  S.ctl[kCtlActive] = need;
  S.ctl[kCtlNeed] = 0;
  S.ctl[kCtlEpoch] += 1;
  S.ctl[kCtlWork] = 0;
  // the filter's rounds per append, from the last evaluation's kept pairs
  const long long kept = (long long)S.ctl[kCtlKept] + S.ctl[kCtlKeptCold];
  S.ctl[kCtlRounds] = 8 * kept > S.ctl[kCtlPairs] ? kFilterRounds : 1;
  S.ctl[kCtlKept] = 0;
  S.ctl[kCtlKeptCold] = 0;
  S.ctl[kCtlKept2] = 0;
  S.ctl[kCtlRebuilds] += need ? 1 : 0;
  if (use_handle) cudaGraphSetConditional(h, need ? 1u : 0u);
}

// Pair-list cell key of x (clamped into the grid; outside it raises
// kErrOutOfGrid like the reference's SimulationError).
__device__ __forceinline__ int buildKey(GridDesc const& bg, d3 x, int* status) {
  const double xs[3] = {x.x, x.y, x.z};
  int id[3];
  bool valid = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    id[d] = (int)floor((xs[d] - bg.lc_origin[d]) / bg.edge[d]);
    if (id[d] < 0 || id[d] >= bg.nb[d]) {
      valid = false;
      id[d] = min(max(id[d], 0), bg.nb[d] - 1);
    }
  }
  if (!valid) raise(status, kErrOutOfGrid);
  return bg.cell_offset + id[1] * bg.nb[2] * bg.nb[0] + id[2] * bg.nb[0] + id[0];
}

__global__ void k_bin(DevState S, const int* gate) {
  if (gatedOff(gate)) return;
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  // the lists are empty until the pair search and k_wall_rows fill them (their
  // memory has been saved)
  if (s == 0) {
    S.ctl[kCtlPairs] = 0;
    S.ctl[kCtlWallSlots] = 0;
  }
  if (s >= S.n) return;
  const int key = buildKey(S.bgrids[S.inst[s]], ld3(S.x, S.cap, s), S.status);
  S.skey[s] = key;
  S.rank[s] = atomicAdd(&S.cell_count[key], 1);
}

// ------------------------------------------------------------------ scan --
// Exclusive scan of cell counts, three phases over 1024-element tiles.
constexpr int kScanTile = 1024;

__device__ __forceinline__ int blockExclusiveScan(int v, int* smem, int& total) {
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    int y = lane < nw ? smem[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    smem[lane] = y;
  }
  __syncthreads();
  int before = wid > 0 ? smem[wid - 1] : 0;
  total = smem[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before + x - v;
}

__global__ void k_scan_tiles(const int* in, int* out, int* tile_sums, int n, const int* gate) {
  if (gatedOff(gate)) return;
  __shared__ int smem[32];
  int i = blockIdx.x * kScanTile + threadIdx.x;
  int v = i < n ? in[i] : 0;
  int total;
  int ex = blockExclusiveScan(v, smem, total);
  if (i < n) out[i] = ex;
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Scans the tile sums in place with one block, looping over chunks.
__global__ void k_scan_sums(int* sums, int ntiles, const int* gate) {
  if (gatedOff(gate)) return;
  __shared__ int smem[32];
  int carry = 0;
  for (int base = 0; base < ntiles; base += kScanTile) {
    int i = base + threadIdx.x;
    int v = i < ntiles ? sums[i] : 0;
    int total;
    int ex = blockExclusiveScan(v, smem, total);
    if (i < ntiles) sums[i] = ex + carry;
    carry += total;
    __syncthreads();
  }
}

// Adds the tile offsets; out[n] receives the total so that cell c spans
// [out[c], out[c + 1]).
__global__ void k_scan_add(int* out, const int* tile_sums, const int* in, int n,
                           const int* gate, int* ctl) {
  if (gatedOff(gate)) return;
  int i = blockIdx.x * kScanTile + threadIdx.x;
  if (i < n) {
    int v = out[i] + tile_sums[blockIdx.x];
    out[i] = v;
    if (i == n - 1) {
      // (a total beyond 2^31 - 1 wraps negative: the rows then do not fit)
      const int total = v + in[i];
      out[n] = total;
      if (ctl) {
        ctl[kCtlEntries] = total;
        atomicMax(&ctl[kCtlEntriesMax], total < 0 ? INT_MAX : total);
      }
    }
  }
}

__global__ void k_place(DevState S, const int* gate) {
  if (gatedOff(gate)) return;
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S.n) return;
  S.order[S.cell_start[S.skey[s]] + S.rank[s]] = s;
}

// Orders each cell's entries by particle ID, so the permutation does not
// depend on the arrival order of the atomic histogram.  It also resets the
// cell histogram for the next rebuild (every count has been consumed by the
// scan at this point).
__global__ void k_cellsort(DevState S, const int* gate) {
  if (gatedOff(gate)) return;
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= S.ncells) return;
  int b = S.cell_start[c];
  int cnt = S.cell_start[c + 1] - b;
  S.cell_count[c] = 0;
  if (cnt < 2) return;
  for (int i = 1; i < cnt; ++i) {
    int e = S.order[b + i];
    int ide = S.id[e];
    int j = i - 1;
    while (j >= 0 && S.id[S.order[b + j]] > ide) {
      S.order[b + j + 1] = S.order[b + j];
      --j;
    }
    S.order[b + j + 1] = e;
  }
}

// Gathers the state into cell order (second buffers) and writes the compact
// arrays of the pair search: the cell, the FP64 position + radius (FP64
// mode) or the FP32 offset from the cell's lower corner + radius (FP32-split).
// forces: F, T too (before the first step of a call; a rebuild inside a call
// comes between their last use and the last evaluation's, which writes them).
__global__ void k_permute(DevState S, const int* gate, int forces) {
  if (gatedOff(gate)) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  const int cap = S.cap;
  const int s = S.order[t];
  const int ty = S.type[s], in = S.inst[s];
  S.id2[t] = S.id[s]; S.type2[t] = ty; S.inst2[t] = in;
  const d3 x = ld3(S.x, cap, s);
  st3(S.x2, cap, t, x);
  st3(S.v2, cap, t, ld3(S.v, cap, s));
  st3(S.w2, cap, t, ld3(S.w, cap, s));
  if (S.wbf_state) st3(S.wbf2, cap, t, ld3(S.wbf, cap, s));
  if (forces) {
    st3(S.F2, cap, t, ld3(S.F, cap, s));
    st3(S.T2, cap, t, ld3(S.T, cap, s));
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) S.q2[k * cap + t] = S.q[k * cap + s];
  if (S.basis) {
#pragma unroll
    for (int k = 0; k < 9; ++k) S.basis2[k * cap + t] = S.basis[k * cap + s];
  }
  if (S.curv) S.curv2[t] = S.curv[s];
  GridDesc const& bg = S.bgrids[in];
  const int c = S.skey[s] - bg.cell_offset;
  const int ci = c % bg.nb[0];
  const int ck = (c / bg.nb[0]) % bg.nb[2];
  const int cj = c / (bg.nb[0] * bg.nb[2]);
  S.cellc[t] = make_int4(ci, cj, ck, in);
  TypeDesc const& tp = S.types[ty];
  if (S.pos64) S.pos64[t] = make_double4(x.x, x.y, x.z, tp.radius);
  if (S.offh) {
    S.offh[t] = make_float4((float)(x.x - (bg.lc_origin[0] + ci * bg.edge[0])),
                            (float)(x.y - (bg.lc_origin[1] + cj * bg.edge[1])),
                            (float)(x.z - (bg.lc_origin[2] + ck * bg.edge[2])), tp.r_f);
  }
}

// Second buffers back into the current ones; the wraps since the rebuild
// start again from zero and the FP32 position becomes the rebuild's.
__global__ void k_copyback(DevState S, const int* gate, int forces) {
  if (gatedOff(gate)) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  const int cap = S.cap;
  S.id[t] = S.id2[t]; S.type[t] = S.type2[t]; S.inst[t] = S.inst2[t];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const size_t k = (size_t)d * cap + t;
    S.x[k] = S.x2[k]; S.v[k] = S.v2[k]; S.w[k] = S.w2[k];
    if (S.wbf_state) S.wbf[k] = S.wbf2[k];
    if (forces) { S.F[k] = S.F2[k]; S.T[k] = S.T2[k]; }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) S.q[k * cap + t] = S.q2[k * cap + t];
  if (S.basis) {
#pragma unroll
    for (int k = 0; k < 9; ++k) S.basis[k * cap + t] = S.basis2[k * cap + t];
  }
  if (S.curv) S.curv[t] = S.curv2[t];
  S.wrap[t] = 0;
  const d3 x = ld3(S.x, cap, t);
  const float4 p = make_float4((float)x.x, (float)x.y, (float)x.z,
                               (float)S.types[S.type[t]].radius);
  S.posf[t] = p;
  S.posf0[t] = p;
}

// Force and torque of particle t in this evaluation: its weight plus the
// shares the pair kernel wrote into its row, in row order, then its wall
// share.  The entry bits of the flag word name the shares of the first
// kMaskEntries entries, so their loads are issued together, two at a time
// (a particle rarely has more contacts, and larger batches spill);
// entries beyond (kFarEntry) are found by their evaluation tags.  FP32-split
// (kFast): FP32 shares summed in FP32; FP64: FP64 shares summed in FP64 onto
// the weight.
template <bool kFast>
__device__ __forceinline__ void sumShares(DevState const& S, int t, TypeDesc const& tp,
                                          unsigned na, int off, int tag, d3& F, d3& T) {
  constexpr int kBatch = 2;
  if constexpr (kFast) {
    float fx = 0.f, fy = 0.f, fz = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
    const float4* sh = static_cast<const float4*>(S.share) + 2 * (size_t)off;
    unsigned m = na & kEntryBits;
    while (m) {
      float4 a[kBatch], b[kBatch];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (m) {
          const int e = __ffs(m) - 1;
          m &= m - 1u;
          a[j] = sh[2 * e];
          b[j] = sh[2 * e + 1];
          cnt = j + 1;
        }
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (j < cnt) {
          fx += a[j].x; fy += a[j].y; fz += a[j].z;
          tx += b[j].x; ty += b[j].y; tz += b[j].z;
        }
      }
    }
    if (na & kFarEntry) {
      const int np = S.npairs[t];
      for (int e = kMaskEntries; e < np; ++e) {
        const float4 a = sh[2 * e];
        if (__float_as_int(a.w) != tag) continue;
        const float4 b = sh[2 * e + 1];
        fx += a.x; fy += a.y; fz += a.z;
        tx += b.x; ty += b.y; tz += b.z;
      }
    }
    if (na & kNearWall) {
      // the walls' own sum first, in wall order
      const int2 row = S.wrow[t];
      const float4* ws = static_cast<const float4*>(S.wshare) +
                         (size_t)kWallShare32 * row.x;
      float wx = 0.f, wy = 0.f, wz = 0.f, ux = 0.f, uy = 0.f, uz = 0.f;
      for (int k = 0; k < row.y; ++k, ws += kWallShare32) {
        const float4 a = ws[0];
        if (__float_as_int(a.w) != tag) continue;
        const float4 b = ws[1];
        wx += a.x; wy += a.y; wz += a.z;
        ux += b.x; uy += b.y; uz += b.z;
        if (b.w != 0.f) {
          const float4 c = ws[2];
          ux += c.x; uy += c.y; uz += c.z;
        }
      }
      fx += wx; fy += wy; fz += wz;
      tx += ux; ty += uy; tz += uz;
    }
    F = mk(tp.weight[0] + (double)fx, tp.weight[1] + (double)fy, tp.weight[2] + (double)fz);
    T = mk((double)tx, (double)ty, (double)tz);
  } else {
    F = mk(tp.weight[0], tp.weight[1], tp.weight[2]);
    T = mk(0., 0., 0.);
    const double2* sh = static_cast<const double2*>(S.share) + 4 * (size_t)off;
    unsigned m = na & kEntryBits;
    while (m) {
      double2 a[kBatch], b[kBatch], c[kBatch], d[kBatch];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (m) {
          const int e = __ffs(m) - 1;
          m &= m - 1u;
          a[j] = sh[4 * e]; b[j] = sh[4 * e + 1]; c[j] = sh[4 * e + 2]; d[j] = sh[4 * e + 3];
          cnt = j + 1;
        }
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (j < cnt) {
          F = F + mk(a[j].y, b[j].x, b[j].y);
          T = T + mk(c[j].x, c[j].y, d[j].x);
        }
      }
    }
    if (na & kFarEntry) {
      const int np = S.npairs[t];
      for (int e = kMaskEntries; e < np; ++e) {
        const double2 a = sh[4 * e];
        if ((int)__double_as_longlong(a.x) != tag) continue;
        const double2 b = sh[4 * e + 1], c = sh[4 * e + 2], d = sh[4 * e + 3];
        F = F + mk(a.y, b.x, b.y);
        T = T + mk(c.x, c.y, d.x);
      }
    }
    if (na & kNearWall) {
      const int2 row = S.wrow[t];
      const double2* ws = static_cast<const double2*>(S.wshare) +
                          (size_t)kWallShare64 * row.x;
      d3 Fw = mk(0., 0., 0.), Tw = mk(0., 0., 0.);
      for (int k = 0; k < row.y; ++k, ws += kWallShare64) {
        const double2 a = ws[0];
        if ((int)__double_as_longlong(a.x) != tag) continue;
        const double2 b = ws[1], c = ws[2], d = ws[3];
        Fw = Fw + mk(a.y, b.x, b.y);
        Tw = Tw + mk(c.x, c.y, d.x);
        if (d.y != 0.) {
          const double2 e = ws[4], f = ws[5];
          Tw = Tw + mk(e.x, e.y, f.x);
        }
      }
      F = F + Fw;
      T = T + Tw;
    }
  }
}

// Threads per block of k_move.
template <bool kFast, bool kBasis>
constexpr int kMoveBlock() { return kBasis ? 256 : 128; }

// Leapfrog of each particle.  Launch bounds, by the whole step: the kernel
// starts while the pair kernel runs, so its own time is not all that counts.
// FP32-split spheres: 128-thread blocks, eight per multiprocessor at 64
// registers (1M: faster than 256-thread blocks at three, four or five; bound by
// the latency of its loads).  FP64 spheres: six at 80 registers; 256,000 gas
// spheres step 50.7 us, with five 52.0, with seven 52.7, 60,000 packed 63.9,
// 65.0 and 66.4, although alone the kernel is as fast or faster with five (23.1
// and 23.1 us, 18.6 and 17.4).  With an orientation matrix: two 256-thread
// blocks, an instantiation of its own in both modes (a convex FP64 pour's move
// 21.5 -> 13.8 us).
//
// With kStepSum the force and torque of this evaluation: the weight for a
// particle the contact filter did not mark as a
// candidate, else the weight plus its shares (sumShares); without it, the
// stored F, T (the opening kick of a call continues from the last evaluation
// of the previous one).  Then the closing kick of the step that ends
// (flags & kStepClose) and the opening kick + drift of the next
// (flags & kStepMove); kStepStoreFT writes F, T back (the last evaluation of
// a call, and the leapfrog start, which only stores them).  Per particle
// only, so it runs in place (the launcher aliases the second buffers to the
// current ones).
//
// The kernel starts while the pair kernel still runs (programmatic launch:
// the pair kernel triggers after its own wait, so the filter has completed
// and its candidate marks are final).  A particle that is not a candidate
// takes no share and is not read by the pair kernel, so its leapfrog runs at
// once; a candidate waits for the pair kernel before it reads its shares.
template <bool kFast, bool kBasis>
__global__ void __launch_bounds__(kMoveBlock<kFast, kBasis>(), kBasis ? 2 : (kFast ? 8 : 6))
    k_move(DevState S, int flags) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  TypeDesc const& tp = S.types[S.type[t]];
  MoveIn m;
  loadMoveIn<kFast, kBasis>(S, t, m);   // nothing the contact kernels write
  const bool sum = (flags & kStepSum) != 0;
  // (asked after the state's loads are on their way; before them it cost 0.6 %
  // of a step)
  if (sum && S.ctl[kCtlNeed] == kPutOff) return;
  d3 F, T;
  bool candidate = false;
  if (sum) {
    int* fl = contactFlags(S);
    candidate = ((unsigned)fl[t] & kCandidate) != 0u;
    if (!candidate) {
      F = mk(tp.weight[0], tp.weight[1], tp.weight[2]);
      T = mk(0., 0., 0.);
    } else {
      // the row of t (written by the last rebuild, before the filter)
      const int off = S.pair_off[t];
      pdlWait();
      sumShares<kFast>(S, t, tp, (unsigned)fl[t], off, S.ctl[kCtlEpoch], F, T);
    }
    if (flags & kStepStoreFT) { st3(S.F, S.cap, t, F); st3(S.T, S.cap, t, T); }
  } else {
    pdlWait();
    F = ld3(S.F, S.cap, t);
    T = ld3(S.T, S.cap, t);
  }
  if (S.hydro) {
    // coupled run: the fluid's force and torque, added after the contacts as
    // the PRSHydroFT application does (it runs after the collision one)
    const double* hy = S.hydro + 6 * (size_t)S.id[t];
    F = F + mk(hy[0], hy[1], hy[2]);
    T = T + mk(hy[3], hy[4], hy[5]);
  }
  if (flags & (kStepClose | kStepMove))
    advanceParticle<kFast, kBasis>(S, t, tp, F, T, (flags & kStepClose) != 0,
                                   (flags & kStepMove) != 0, m);
  // the next evaluation's flag words start clear (no other kernel touches
  // that buffer until the next contact filter)
  contactFlags(S, 1)[t] = 0;
  if (candidate && S.curv_next) {
    // the polyhedron vertex this evaluation's GJK calls left (recordVertex;
    // only candidates take part in GJK calls)
    const int r = S.curv_next[t];
    if (r) {
      S.curv[t] = r & 0xFFFF;
      S.curv_next[t] = 0;
    }
  }
}

// Appends the kept pairs of a warp's rounds to a list that grows upwards
// (dir 1) or downwards (dir -1) from list[0] and marks their partners: lane j
// holds the ballot of round j in mine (0 beyond the rounds), round j's pairs
// are first + step j + lane.  The flag words are clear (the last leapfrog
// kernel left them so) and only this kernel writes them until the pair kernel
// starts, always this value: a plain store marks a candidate whoever else
// does.  Every lane of the warp calls it.
__device__ __forceinline__ void appendRounds(DevState const& S, int* flags, int* list, int dir,
                                             int* count, unsigned mine, int first, int step) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int c = __popc(mine);
  const int total = __reduce_add_sync(full, c);
  if (!total) return;
  int incl = c;
#pragma unroll
  for (int o = 1; o < kFilterRounds; o <<= 1) {
    const int y = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += y;
  }
  int base = 0;
  if (lane == 0) base = atomicAdd(count, total);
  base = __shfl_sync(full, base, 0);
  for (unsigned some = __ballot_sync(full, c != 0); some; some &= some - 1u) {
    const int j = __ffs(some) - 1;
    const unsigned m = __shfl_sync(full, mine, j);
    const int at = base + __shfl_sync(full, incl - c, j) + __popc(m & ((1u << lane) - 1u));
    if (m >> lane & 1u) {
      const int i = first + step * j + lane;
      const int2 pr = S.upairs[i];
      list[(long long)dir * at] = i;
      flags[pr.x] = (int)kCandidate;
      flags[(unsigned)pr.y & ((1u << 27) - 1u)] = (int)kCandidate;
    }
  }
}

// Whether particle t (posf: its FP32 continuous position) comes within the
// margin (plus reach) of wall k of its instance: its contacts with that wall
// can only come about then.  q: the centre wrapped back into the box.
struct WallProbe {
  float q[3], R;
};
__device__ __forceinline__ WallProbe wallProbe(DevState const& S, int t, GridDesc const& bg,
                                               float reach) {
  const float4 pt = S.posf[t];
  const int wt = S.wrap[t];
  return {{pt.x - (float)wrapGet(wt, 0) * bg.Lf[0], pt.y - (float)wrapGet(wt, 1) * bg.Lf[1],
           pt.z - (float)wrapGet(wt, 2) * bg.Lf[2]},
          pt.w + bg.filt_margin + reach};
}
// images: a wall whose nearest periodic image is near too (the particle can
// leave through one face of the box and come in at the other).
__device__ __forceinline__ bool nearWall(GridDesc const& bg, WallDesc const& wd, WallProbe const& p,
                                         bool images) {
  float d2 = 0.f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float c = p.q[d] - (float)wd.centre[d];
    if (images && bg.periodic[d]) c -= bg.Lf[d] * rintf(c / bg.Lf[d]);
    const float o = fabsf(c) - (float)wd.extent[d];
    if (o > 0.f) d2 += o * o;
  }
  return d2 <= p.R * p.R;
}

// The wall list: the walls, or periodic images of them, within the skin of each
// particle; it can reach no others before the next rebuild (part of a rebuild,
// after k_copyback).
__global__ void k_wall_rows(DevState S, const int* gate) {
  if (gatedOff(gate)) return;
  const unsigned full = 0xffffffffu;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int count = 0, begin = 0, nw = 0;
  WallProbe p{};
  GridDesc const* bg = nullptr;
  if (t < S.n) {
    bg = &S.bgrids[S.inst[t]];
    begin = bg->wall_begin;
    nw = bg->wall_count;
    p = wallProbe(S, t, *bg, bg->skin_f);
    for (int k = 0; k < nw; ++k) count += nearWall(*bg, S.walls[begin + k], p, true);
  }
  int incl = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += y;
  }
  int base = 0;
  if (lane == 31 && incl) base = atomicAdd(S.ctl + kCtlWallSlots, incl);
  int slot = __shfl_sync(full, base, 31) + incl - count;
  if (t >= S.n) return;
  S.wrow[t] = make_int2(slot, count);
  if (!count) return;
  if (slot > S.wall_cap - count) {
    S.ctl[kCtlNeed] = kPutOff;
    return;
  }
  for (int k = 0; k < nw; ++k)
    if (nearWall(*bg, S.walls[begin + k], p, true)) S.wlist[slot++] = make_int2(t, k);
}

// This evaluation's wall items: for spheres every near slot of the wall list,
// else the first slots of the particles near any wall (their walls are taken
// in turn: a polyhedron's support vertex runs through them).
__device__ __forceinline__ void filterWalls(DevState const& S, int* flags, int nblocks) {
  const int lane = threadIdx.x & 31;
  const int ns = listedWalls(S);
  for (int s0 = (int)(blockIdx.x * blockDim.x + threadIdx.x) & ~31; s0 < ns;
       s0 += nblocks * blockDim.x) {   // warp-uniform
    const int slot = s0 + lane;
    bool near = false;
    if (slot < ns) {
      const int2 e = S.wlist[slot];
      int last = slot;
      if (S.any_convex) {
        const int2 row = S.wrow[e.x];
        last = row.x == slot ? slot + row.y - 1 : slot - 1;
      }
      GridDesc const& bg = S.bgrids[S.inst[e.x]];
      const WallProbe p = wallProbe(S, e.x, bg, 0.f);
      for (int s = slot; s <= last && !near; ++s)
        near = nearWall(bg, S.walls[bg.wall_begin + (s == slot ? e.y : S.wlist[s].y)], p, false);
      if (near) flags[e.x] = (int)kCandidate;
    }
    const unsigned m = __ballot_sync(0xffffffffu, near);
    if (!m) continue;
    int at = 0;
    if (lane == 0) at = atomicAdd(S.ctl + kCtlWork, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (near) S.work[at] = slot;
  }
}

// Contact filter.  One lane per pair of the compact pair list (each pair
// once, from its lower ID): the FP32 bounding-sphere test, a superset of the
// contacts; the kept pairs are listed for the pair kernel, which decides each
// exactly, and both partners marked as candidates.  With walls, the first
// pblocks blocks take the wall list (filterWalls).  A warp tests `rounds`
// rounds of 32 pairs, then appends all it kept with one atomic: where the last
// evaluation kept more than an eighth of the pairs (a packed bed, colliding
// convex bodies) up to kFilterRounds of them, else one, whose append then
// overlaps the other warps' loads.  A grid-stride loop covers any count (known
// on the device only).
// What bounds it: in a gas (few pairs kept) the latency of the position
// gathers (1M spheres: 20.9 us with 1 round, 23.1 with 8); in a bed the marks
// and the appends, which were two atomics per kept pair and one per 32 pairs
// on a single counter (250,000 packed spheres, 737,000 pairs kept: 32.9 us
// then, 31.3 with plain marks and 1 round, 22.5 with 8 rounds; 16.7 since the
// walls are tested for the wall list only).
// kSplit: FP32-split with non-spherical classes (the kept pairs in two lists).
template <bool kSplit>
__global__ void __launch_bounds__(256, 8) k_filter(DevState S, int pblocks) {
  pdlTrigger();   // the pair kernel may be scheduled; it waits for this one
  const int lane = threadIdx.x & 31;
  int* flags = contactFlags(S);
  if ((int)blockIdx.x < pblocks) {
    filterWalls(S, flags, pblocks);
    return;
  }
  const int np = listedPairs(S);
  const long long wq = ((long long)((int)blockIdx.x - pblocks) * blockDim.x + threadIdx.x) >> 5;
  const long long nwq = ((long long)(gridDim.x - pblocks) * blockDim.x) >> 5;
  // (all warp-uniform) round j of a warp is the grid's j-th sweep over the list
  const long long sweep = 32 * nwq;
  const int rounds = (int)min((long long)S.ctl[kCtlRounds], (np + sweep - 1) / sweep);
  for (long long c0 = 32 * wq; c0 < np; c0 += sweep * rounds) {
    unsigned mine = 0, mine_cold = 0;
    for (int j = 0; j < rounds; ++j) {
      const long long c = c0 + sweep * j + lane;
      bool keep = false, hot = false;
      if (c < np) {
        const int2 pr = S.upairs[c];
        const int t = pr.x, u = (int)((unsigned)pr.y & ((1u << 27) - 1u));
        const float4 pa = S.posf[t], pb = S.posf[u];
        // the largest margin of the instances (a superset of the contacts);
        // the period only for an entry with an image shift (code 13 is
        // none), which needs the instance's grid
        const unsigned code = (unsigned)pr.y >> 27;
        float sx = 0.f, sy = 0.f, sz = 0.f;
        if (code != 13u) {
          GridDesc const& bg = S.bgrids[S.inst[t]];
          sx = (float)((int)(code % 3u) - 1) * bg.Lf[0];
          sy = (float)((int)((code / 3u) % 3u) - 1) * bg.Lf[1];
          sz = (float)((int)(code / 9u) - 1) * bg.Lf[2];
        }
        const float dx = (pb.x - pa.x) + sx;
        const float dy = (pb.y - pa.y) + sy;
        const float dz = (pb.z - pa.z) + sz;
        const float R = pa.w + pb.w + S.filt_margin_max;
        keep = dx * dx + dy * dy + dz * dz <= R * R;
        if constexpr (kSplit) {
          // a pair in contact at the last evaluation (its share on t's side
          // carries that evaluation's tag) goes to the front of the list, the
          // others to the back, so the pair kernel runs the full
          // closest-point searches and laws of the likely contacts in warps
          // of their own and the searches that stop early in others
          // (measured: 3 % off the convex pour's FP32-split step; the FP64
          // step, whose searches all run to their end, was 1 % slower with
          // it).  A guess that a rebuild made stale only reorders.
          if (keep) {
            const long long e = (long long)S.pair_off[t] + (S.epos[c] & 0xFFFF);
            hot = __float_as_int(static_cast<const float4*>(S.share)[2 * e].w) ==
                  S.ctl[kCtlEpoch] - 1;
          }
        } else {
          hot = keep;
        }
      }
      const unsigned mh = __ballot_sync(0xffffffffu, hot);
      if (lane == j) mine = mh;
      if constexpr (kSplit) {
        const unsigned mc = __ballot_sync(0xffffffffu, keep && !hot);
        if (lane == j) mine_cold = mc;
      }
    }
    appendRounds(S, flags, S.kept, 1, S.ctl + kCtlKept, mine, (int)c0, (int)sweep);
    if constexpr (kSplit)
      appendRounds(S, flags, S.kept + (S.pair_cap / 2), -1, S.ctl + kCtlKeptCold, mine_cold,
                   (int)c0, (int)sweep);
  }
}

// Where each pair of the compact list sits in its partner's row: the entry of
// the lower-ID slot t in the row of u (rows are symmetric: the pair search
// decides both directions with the same expression).  0xFFFF when absent (a
// row cut off at kRowMax).  Grid-stride over the pairs, whose count is known on
// the device only; not where the list is incomplete for lack of room.
__global__ void __launch_bounds__(256) k_link(DevState S, const int* gate) {
  if (gatedOff(gate) || S.ctl[kCtlNeed] == kPutOff) return;
  const int np = listedPairs(S);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x) {
    const int2 pr = S.upairs[k];
    const int t = pr.x;
    const int u = (int)((unsigned)pr.y & ((1u << 27) - 1u));
    const int nu = S.npairs[u];
    const int* row = S.pairs + S.pair_off[u];
    int eu = 0xFFFF;
    for (int e = 0; e < nu; ++e)
      if ((int)((unsigned)row[e] & ((1u << 27) - 1u)) == t) { eu = e; break; }
    S.epos[k] = (S.epos[k] & 0xFFFF) | (eu << 16);
  }
}

// Diagnostics: every entry and wall slot starts at +inf (no contact); the
// pair kernel records the pairs it evaluates.
__global__ void k_diag_prefill(DevState S) {
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const long long ne = S.ctl[kCtlEntries] < 0 ? 0 : min(S.ctl[kCtlEntries], S.pair_cap);
  const long long nw = (long long)S.n * S.max_walls;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ne + nw; i += stride) {
    if (i < ne) S.pair_delta[i] = inf;
    else S.wall_delta[i - ne] = inf;
  }
}

// Scatter of sorted-order state into ID order (for download).
__global__ void k_scatter_by_id(DevState S, double* out_x, double* out_v, double* out_w,
                                double* out_wbf, double* out_q, double* out_F, double* out_T,
                                int id_base) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  const int cap = S.cap, n = S.n;
  int i = S.id[t] - id_base;
  if (i < 0 || i >= n) return;
  if (out_wbf && !S.wbf_state) {
    // q* w q (ParticleKinematics.cpp:220-221), the body-frame image of the state w
    const dq qq = qmk(mk(S.q[t], S.q[cap + t], S.q[2 * cap + t]), S.q[3 * cap + t]);
    const d3 wb = multToVector3(conj(qq), vecq(ld3(S.w, cap, t), qq));
    out_wbf[3 * i] = wb.x; out_wbf[3 * i + 1] = wb.y; out_wbf[3 * i + 2] = wb.z;
    out_wbf = nullptr;
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (out_x) out_x[3 * i + d] = S.x[d * cap + t];
    if (out_v) out_v[3 * i + d] = S.v[d * cap + t];
    if (out_w) out_w[3 * i + d] = S.w[d * cap + t];
    if (out_wbf) out_wbf[3 * i + d] = S.wbf[d * cap + t];
    if (out_F) out_F[3 * i + d] = S.F[d * cap + t];
    if (out_T) out_T[3 * i + d] = S.T[d * cap + t];
  }
  if (out_q) {
#pragma unroll
    for (int k = 0; k < 4; ++k) out_q[4 * i + k] = S.q[k * cap + t];
  }
}

// Orientation matrices (row-major, 9 per particle) into ID order.
__global__ void k_basis_by_id(DevState S, double* out, int id_base) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  int i = S.id[t] - id_base;
  if (i < 0 || i >= S.n) return;
#pragma unroll
  for (int k = 0; k < 9; ++k) out[9 * (size_t)i + k] = S.basis[k * S.cap + t];
}

// Reference-grid cell (Cell::GetCell) of each particle, by ID.
__global__ void k_cells_by_id(DevState S, int* ijk, int id_base) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  int i = S.id[t] - id_base;
  if (i < 0 || i >= S.n) return;
  GridDesc const& g = S.grids[S.inst[t]];
  const d3 x = ld3(S.x, S.cap, t);
  const double xs[3] = {x.x, x.y, x.z};
#pragma unroll
  for (int d = 0; d < 3; ++d) ijk[3 * i + d] = (int)floor((xs[d] - g.lc_origin[d]) / g.edge[d]);
}

// Coordination number of each particle at the last force evaluation, by ID:
// the listed partners and the walls whose overlap recorded by that
// evaluation is negative.  The reference counts the distinct components a
// particle touched in its force computation (Particle::
// addContactingComponentID, Component/src/Particle.cpp:1702-1706, called by
// Particle::InterAction and SimpleObstacle::InterAction for each contact of
// negative overlap, Particle.cpp:530-543, SimpleObstacle.cpp:262-270); the
// pair list holds each partner once and each wall has one slot.
__global__ void k_coordination_by_id(DevState S, int* out, int id_base) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  int i = S.id[t] - id_base;
  if (i < 0 || i >= S.n) return;
  const int np = S.npairs[t];
  const double* pd = S.pair_delta + S.pair_off[t];
  int c = 0;
  for (int e = 0; e < np; ++e) c += pd[e] < 0. ? 1 : 0;
  const int nw = S.grids[S.inst[t]].wall_count;
  const double* wd = S.wall_delta + (size_t)t * S.max_walls;
  for (int k = 0; k < nw; ++k) c += wd[k] < 0. ? 1 : 0;
  out[i] = c;
}

// Contact memory between the lists and the table.  Entries 0 .. pairs - 1 are
// the compact pair list's, then come the wall list's.
__device__ __forceinline__ void memEntry(DevState const& S, int np, long long i, MemView& m,
                                         long long& at, unsigned long long& key) {
  if (i < np) {
    const int2 pr = S.upairs[i];
    m = S.pmem;
    at = i;
    key = pairKey(S.id[pr.x], S.id[(unsigned)pr.y & ((1u << 27) - 1u)]);
    return;
  }
  m = S.wmem;
  at = i - np;
  const int2 e = S.wlist[at];
  key = wallKey(S.id[e.x], e.y);
}

// Frees the table's slots before the lists' memory is saved (the plain step).
__global__ void k_mem_clear(DevState S, const int* gate) {
  if (gatedOff(gate) || !S.ctl[kCtlMemory]) return;
  const size_t cap = size_t(1) << S.hist.log2cap;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap;
       i += (size_t)gridDim.x * blockDim.x)
    S.hist.keys[i] = kEmptyKey;
}

// The memory that evaluation now (the counter less back) left in the lists, or
// any there (the coupled step), into the table.
template <typename T>
__global__ void k_mem_save(DevState S, const int* gate, int back) {
  if (gatedOff(gate) || !S.ctl[kCtlMemory]) return;
  const int now = S.ctl[kCtlEpoch] - back;
  const int np = listedPairs(S);
  const long long ne = np + listedWalls(S);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ne;
       i += (long long)gridDim.x * blockDim.x) {
    MemView m;
    long long at;
    unsigned long long key;
    memEntry(S, np, i, m, at, key);
    if (!remembered(S, memEvaluation(m, at, T()), now + 1)) continue;
    T v[9];
    memLoad(m, at, v, true);
    const int s = histInsert(S.hist, key);
    if (s < 0) { raise(S.status, kErrHashFull); continue; }
    T* d = static_cast<T*>(S.hist.vals) + 9 * (size_t)s;
#pragma unroll
    for (int k = 0; k < 9; ++k) d[k] = v[k];
  }
}

// The table's memory into the new lists, as left by the last evaluation; from
// here on the lists hold it.  The last kernel of a rebuild: where a list ran
// short it puts the evaluation off instead (kPutOff).
template <typename T>
__global__ void k_mem_load(DevState S, const int* gate) {
  if (gatedOff(gate)) return;
  const int last = S.ctl[kCtlEpoch] - 1;
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool off = S.ctl[kCtlNeed] == kPutOff;
  const int np = listedPairs(S);
  const long long ne = np + listedWalls(S);
  if (i0 == 0) {
    S.ctl[kCtlMemory] = off ? 0 : 1;
    S.ctl[kCtlWallSlotsMax] = max(S.ctl[kCtlWallSlotsMax], S.ctl[kCtlWallSlots]);
    if (off) {
      // (the table keeps the memory)
      S.ctl[kCtlPairs] = 0;
      S.ctl[kCtlWallSlots] = 0;
      S.ctl[kCtlEpoch] -= 1;
      S.ctl[kCtlRebuilds] -= 1;
    }
  }
  if (off) return;
  for (long long i = i0; i < ne; i += (long long)gridDim.x * blockDim.x) {
    MemView m;
    long long at;
    unsigned long long key;
    memEntry(S, np, i, m, at, key);
    const int s = histFind(S.hist, key);
    if (s < 0) { memForget(m, at, T()); continue; }
    const T* d = static_cast<const T*>(S.hist.vals) + 9 * (size_t)s;
    T v[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = d[k];
    memStore(m, at, v, last, true);
  }
}

// Zeroes the cumulative tangential and rolling memories of every contact of
// the last evaluation (Component::setContactMapCumulativeFeaturesToZero,
// Component.cpp:842-851), in the lists and, in the coupled step, of the pairs
// the table keeps.
template <typename V>
__global__ void k_mem_zero_cumulative(DevState S) {
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int now = S.ctl[kCtlEpoch];
  const int np = listedPairs(S);
  const long long ne = np + listedWalls(S);
  for (long long i = i0; i < ne; i += stride) {
    MemView m = i < np ? S.pmem : S.wmem;
    const long long at = i < np ? i : i - np;
    const int e = memEvaluation(m, at, V());
    if (!remembered(S, e, now + 1)) continue;
    V v[9];
    memLoad(m, at, v, true);
    v[0] = v[1] = v[2] = v[6] = v[7] = v[8] = 0;
    memStore(m, at, v, e, true);
  }
  if (S.prune) return;
  for (long long i = i0; i < (1ll << S.hist.log2cap); i += stride) {
    if (S.hist.keys[i] == kEmptyKey) continue;
    V* v = static_cast<V*>(S.hist.vals) + 9 * (size_t)i;
    v[0] = v[1] = v[2] = v[6] = v[7] = v[8] = 0;
  }
}

// Orientation matrix of the quaternion q (x, y, z, w) with the expression
// order of Matrix::setRotation (Geometry/src/Matrix.cpp:114-127).
__device__ __forceinline__ void basisOfQuaternion(const double* q, double* m) {
  const double x = q[0], y = q[1], z = q[2], w4 = q[3];
  const double s = 2.0 / (x * x + y * y + z * z + w4 * w4);
  const double xs = x * s, ys = y * s, zs = z * s;
  const double wx = w4 * xs, wy = w4 * ys, wz = w4 * zs;
  const double xx = x * xs, xy = x * ys, xz = x * zs, yy = y * ys, yz = y * zs, zz = z * zs;
  m[0] = 1.0 - (yy + zz); m[1] = xy - wz; m[2] = xz + wy;
  m[3] = xy + wz; m[4] = 1.0 - (xx + zz); m[5] = yz - wx;
  m[6] = xz - wy; m[7] = yz + wx; m[8] = 1.0 - (xx + yy);
}

// An inserted particle (Grains::insertParticle, Base/src/Grains.cpp:
// 2063-2139) written into slot p.slot, after the others: position,
// velocities, quaternion and its orientation matrix (or the given one), the
// body-frame angular velocity q* w q, its weight as force and a zero torque
// (Particle::InitializeForce(true)), the start vertex of a new polyhedron,
// no displacement, wraps or contact marks.  The host asks for a pair-list
// rebuild before the next force evaluation.
__global__ void k_append_particle(DevState S, NewParticle p) {
  if (threadIdx.x || blockIdx.x) return;
  const int cap = S.cap, i = p.slot;
  TypeDesc const& tp = S.types[p.type];
  S.id[i] = p.id;
  S.type[i] = p.type;
  S.inst[i] = 0;
  const d3 x = mk(p.x[0], p.x[1], p.x[2]), w = mk(p.w[0], p.w[1], p.w[2]);
  st3(S.x, cap, i, x);
  st3(S.v, cap, i, mk(p.v[0], p.v[1], p.v[2]));
  st3(S.w, cap, i, w);
#pragma unroll
  for (int k = 0; k < 4; ++k) S.q[k * cap + i] = p.q[k];
  if (S.basis) {
    double m[9];
    if (p.has_basis) {
      for (int k = 0; k < 9; ++k) m[k] = p.basis[k];
    } else {
      basisOfQuaternion(p.q, m);
    }
    for (int k = 0; k < 9; ++k) S.basis[k * cap + i] = m[k];
  }
  const dq qq = qmk(mk(p.q[0], p.q[1], p.q[2]), p.q[3]);
  st3(S.wbf, cap, i, multToVector3(conj(qq), vecq(w, qq)));
  st3(S.F, cap, i, mk(tp.weight[0], tp.weight[1], tp.weight[2]));
  st3(S.T, cap, i, mk(0., 0., 0.));
  S.wrap[i] = 0;
  if (S.curv) {
    S.curv[i] = tp.poly_start;
    S.curv_next[i] = 0;
  }
  S.nact[i] = 0;
  S.nact[cap + i] = 0;
  const float4 pf = make_float4((float)x.x, (float)x.y, (float)x.z, (float)tp.radius);
  S.posf[i] = pf;
  S.posf0[i] = pf;
}

// Loads host-layout state (AoS, by particle ID, staged in device memory)
// into the SoA arrays, in ID order.
__global__ void k_load_state(DevState S, const double* x, const double* v, const double* w,
                             const double* wbf, const double* q, const double* F,
                             const double* T, const int* type_by_id, const int* inst_by_id) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.n) return;
  const int cap = S.cap;
  S.id[i] = i;
  S.type[i] = type_by_id[i];
  S.inst[i] = inst_by_id[i];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    S.x[d * cap + i] = x[3 * i + d];
    S.v[d * cap + i] = v[3 * i + d];
    S.w[d * cap + i] = w[3 * i + d];
    if (wbf) S.wbf[d * cap + i] = wbf[3 * i + d];
    if (F) S.F[d * cap + i] = F[3 * i + d];
    if (T) S.T[d * cap + i] = T[3 * i + d];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) S.q[k * cap + i] = q[4 * i + k];
  if (S.basis) {
    // gdem_upload_basis may replace it
    double m[9];
    basisOfQuaternion(q + 4 * i, m);
#pragma unroll
    for (int k = 0; k < 9; ++k) S.basis[k * cap + i] = m[k];
  }
  // the host requests a pair-list rebuild after a load, which sets posf and
  // posf0 from these positions
  S.wrap[i] = 0;
  // a new (or reloaded) polyhedron starts its support search where
  // Polyhedron::BuildPolyhedron leaves it
  if (S.curv) S.curv[i] = S.types[type_by_id[i]].poly_start;
  if (!wbf) {
    // q* (w, q) (ParticleKinematics.cpp:220-221)
    dq qq = qmk(mk(q[4 * i], q[4 * i + 1], q[4 * i + 2]), q[4 * i + 3]);
    d3 wb = multToVector3(conj(qq), vecq(mk(w[3 * i], w[3 * i + 1], w[3 * i + 2]), qq));
    st3(S.wbf, cap, i, wb);
  }
}

// GrainsCoupledWithFluid::updateParticlesVelocity (Fluid/src/
// GrainsCoupledWithFluid.cpp:1126-1180): velocities and space-frame angular
// velocities by particle ID (AoS), the body-frame one rebuilt as q* w q.
__global__ void k_set_velocities(DevState S, const double* v, const double* w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.n) return;
  const int cap = S.cap, i = S.id[t];
  const d3 vi = mk(v[3 * i], v[3 * i + 1], v[3 * i + 2]);
  const d3 wi = mk(w[3 * i], w[3 * i + 1], w[3 * i + 2]);
  st3(S.v, cap, t, vi);
  st3(S.w, cap, t, wi);
  if (S.wbf_state) {
    const dq qq = qmk(mk(S.q[t], S.q[cap + t], S.q[2 * cap + t]), S.q[3 * cap + t]);
    st3(S.wbf, cap, t, multToVector3(conj(qq), vecq(wi, qq)));
  }
}

// AllComponents::ComputeMaxMeanVelocity (Component/src/AllComponents.cpp:
// 1781-1811): block partial max and sum of |v|, reduced in a fixed order.
__global__ void k_vstats_partial(DevState S, double* part) {
  __shared__ double smax[256], ssum[256];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  double vit = 0.;
  if (i < S.n) vit = norm(ld3(S.v, S.cap, i));
  smax[threadIdx.x] = vit;
  ssum[threadIdx.x] = vit;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + o]);
      ssum[threadIdx.x] += ssum[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { part[2 * blockIdx.x] = smax[0]; part[2 * blockIdx.x + 1] = ssum[0]; }
}
__global__ void k_vstats_final(const double* part, int nparts, int n, double* out) {
  __shared__ double smax[256], ssum[256];
  double m = 0., s = 0.;
  for (int k = threadIdx.x; k < nparts; k += blockDim.x) { m = fmax(m, part[2 * k]); s += part[2 * k + 1]; }
  smax[threadIdx.x] = m;
  ssum[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + o]);
      ssum[threadIdx.x] += ssum[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { out[0] = smax[0]; out[1] = n > 0 ? ssum[0] / n : 0.; }
}

// Sum of the pair-list segment lengths and count of the contact-memory table's
// entries (the host saves the lists into it first).
__global__ void k_pair_counts(DevState S, unsigned long long* out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long e = 0, c = 0;
  if (i < S.n) e = (unsigned long long)S.npairs[i];
  const long long cap = 1ll << S.hist.log2cap;
  for (long long k = i; k < cap; k += gridDim.x * blockDim.x) c += S.hist.keys[k] != kEmptyKey;
  for (int o = 16; o > 0; o >>= 1) {
    e += __shfl_down_sync(0xffffffffu, e, o);
    c += __shfl_down_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) { atomicAdd(&out[0], e); atomicAdd(&out[1], c); }
}

}  // namespace

inline int blocks(int n, int b) { return (n + b - 1) / b; }

void launch_decide(DevState const& S, cudaGraphConditionalHandle h, int use_handle,
                   cudaStream_t st) {
  k_decide<<<1, 32, 0, st>>>(S, h, use_handle);
}
void launch_bin(DevState const& S, const int* gate, cudaStream_t st) {
  if (S.n) k_bin<<<blocks(S.n, 256), 256, 0, st>>>(S, gate);
}
void launch_scan(DevState const& S, const int* gate, cudaStream_t st) {
  int ntiles = blocks(S.ncells, kScanTile);
  k_scan_tiles<<<ntiles, kScanTile, 0, st>>>(S.cell_count, S.cell_start, S.scan_tmp, S.ncells, gate);
  k_scan_sums<<<1, kScanTile, 0, st>>>(S.scan_tmp, ntiles, gate);
  k_scan_add<<<ntiles, kScanTile, 0, st>>>(S.cell_start, S.scan_tmp, S.cell_count, S.ncells, gate,
                                           nullptr);
}
void launch_row_scan(DevState const& S, const int* gate, cudaStream_t st) {
  if (!S.n) return;
  int ntiles = blocks(S.n, kScanTile);
  k_scan_tiles<<<ntiles, kScanTile, 0, st>>>(S.npairs, S.pair_off, S.pair_scan_tmp, S.n, gate);
  k_scan_sums<<<1, kScanTile, 0, st>>>(S.pair_scan_tmp, ntiles, gate);
  k_scan_add<<<ntiles, kScanTile, 0, st>>>(S.pair_off, S.pair_scan_tmp, S.npairs, S.n, gate, S.ctl);
}
int filterBlocks(long long pairs, int nsm) {
  const long long full = (pairs + 2047) / 2048, one = (pairs + 255) / 256;
  return (int)std::max(1ll, std::max(full, std::min(one, 4ll * nsm)));
}
int wallBlocks(long long slots, int n) {
  return std::max(blocks(n, 2048), (int)(5 * slots / 1024) + 1);
}
void launch_filter(DevState const& S, cudaStream_t st) {
  if (!S.n) return;
  const int pblocks =
      S.any_walls ? (S.filter_wblocks > 0 ? S.filter_wblocks : wallBlocks(0, S.n)) : 0;
  // about 4 pairs per particle until the leapfrog start has counted them
  const int qblocks = S.filter_qblocks > 0 ? S.filter_qblocks : filterBlocks(4ll * S.n, S.nsm);
  if (S.any_convex && !S.pos64) k_filter<true><<<pblocks + qblocks, 256, 0, st>>>(S, pblocks);
  else k_filter<false><<<pblocks + qblocks, 256, 0, st>>>(S, pblocks);
}
void launch_wall_rows(DevState const& S, const int* gate, cudaStream_t st) {
  if (S.n && S.any_walls) k_wall_rows<<<blocks(S.n, 256), 256, 0, st>>>(S, gate);
}
void launch_link(DevState const& S, const int* gate, cudaStream_t st) {
  if (S.n) k_link<<<4 * S.nsm, 256, 0, st>>>(S, gate);
}
void launch_diag_prefill(DevState const& S, cudaStream_t st) {
  if (S.n && S.pair_delta) k_diag_prefill<<<8 * S.nsm, 256, 0, st>>>(S);
}
void launch_place(DevState const& S, const int* gate, cudaStream_t st) {
  if (S.n) k_place<<<blocks(S.n, 256), 256, 0, st>>>(S, gate);
}
void launch_cellsort(DevState const& S, const int* gate, cudaStream_t st) {
  k_cellsort<<<blocks(S.ncells, 256), 256, 0, st>>>(S, gate);
}
void launch_permute(DevState const& S, const int* gate, int forces, cudaStream_t st) {
  if (S.n) k_permute<<<blocks(S.n, 256), 256, 0, st>>>(S, gate, forces);
}
void launch_copyback(DevState const& S, const int* gate, int forces, cudaStream_t st) {
  if (S.n) k_copyback<<<blocks(S.n, 256), 256, 0, st>>>(S, gate, forces);
}
void launch_move(DevState const& S, int flags, int fast, cudaStream_t st) {
  if (!S.n) return;
  DevState M = S;   // in place: the "next" buffers are the current ones
  M.x2 = S.x; M.v2 = S.v; M.w2 = S.w; M.wbf2 = S.wbf; M.q2 = S.q; M.basis2 = S.basis;
  M.wrap2 = S.wrap;
  const int nb = blocks(S.n, 256);
  if (!fast && S.basis) launchAfterPrevious(k_move<false, true>, nb, 256, st, M, flags);
  else if (!fast) launchAfterPrevious(k_move<false, false>, blocks(S.n, kMoveBlock<false, false>()), kMoveBlock<false, false>(), st, M, flags);
  else if (S.basis) launchAfterPrevious(k_move<true, true>, nb, 256, st, M, flags);
  else launchAfterPrevious(k_move<true, false>, blocks(S.n, kMoveBlock<true, false>()), kMoveBlock<true, false>(), st, M, flags);
}
void launch_append_particle(DevState const& S, NewParticle const& p, cudaStream_t st) {
  k_append_particle<<<1, 32, 0, st>>>(S, p);
}
void launch_mem_clear(DevState const& S, const int* gate, cudaStream_t st) {
  k_mem_clear<<<8 * S.nsm, 256, 0, st>>>(S, gate);
}
void launch_mem_save(DevState const& S, const int* gate, int back, int fp64, cudaStream_t st) {
  if (fp64) k_mem_save<double><<<8 * S.nsm, 256, 0, st>>>(S, gate, back);
  else k_mem_save<float><<<8 * S.nsm, 256, 0, st>>>(S, gate, back);
}
void launch_mem_load(DevState const& S, const int* gate, int fp64, cudaStream_t st) {
  if (fp64) k_mem_load<double><<<8 * S.nsm, 256, 0, st>>>(S, gate);
  else k_mem_load<float><<<8 * S.nsm, 256, 0, st>>>(S, gate);
}
void launch_mem_zero_cumulative(DevState const& S, int fp64, cudaStream_t st) {
  if (fp64) k_mem_zero_cumulative<double><<<8 * S.nsm, 256, 0, st>>>(S);
  else k_mem_zero_cumulative<float><<<8 * S.nsm, 256, 0, st>>>(S);
}
void launch_pair_counts(DevState const& S, unsigned long long* out, cudaStream_t st) {
  cudaMemsetAsync(out, 0, 2 * sizeof(unsigned long long), st);
  k_pair_counts<<<blocks(std::max(S.n, 1), 256), 256, 0, st>>>(S, out);
}
void launch_load_state(DevState const& S, const double* x, const double* v, const double* w,
                       const double* wbf, const double* q, const double* F, const double* T,
                       const int* type_by_id, const int* inst_by_id, cudaStream_t st) {
  if (S.n) k_load_state<<<blocks(S.n, 256), 256, 0, st>>>(S, x, v, w, wbf, q, F, T, type_by_id, inst_by_id);
}
void launch_set_velocities(DevState const& S, const double* v, const double* w, cudaStream_t st) {
  if (S.n) k_set_velocities<<<blocks(S.n, 256), 256, 0, st>>>(S, v, w);
}
void launch_vstats(DevState const& S, double* part, double* out, cudaStream_t st) {
  int nb = blocks(S.n, 256);
  if (nb) k_vstats_partial<<<nb, 256, 0, st>>>(S, part);   // (none: an empty system)
  k_vstats_final<<<1, 256, 0, st>>>(part, nb, S.n, out);
}
void launch_scatter_by_id(DevState const& S, double* x, double* v, double* w, double* wbf,
                          double* q, double* F, double* T, int id_base, cudaStream_t st) {
  if (S.n) k_scatter_by_id<<<blocks(S.n, 256), 256, 0, st>>>(S, x, v, w, wbf, q, F, T, id_base);
}
void launch_basis_by_id(DevState const& S, double* out, int id_base, cudaStream_t st) {
  if (S.n && S.basis) k_basis_by_id<<<blocks(S.n, 256), 256, 0, st>>>(S, out, id_base);
}
void launch_cells_by_id(DevState const& S, int* ijk, int id_base, cudaStream_t st) {
  if (S.n) k_cells_by_id<<<blocks(S.n, 256), 256, 0, st>>>(S, ijk, id_base);
}
void launch_coordination_by_id(DevState const& S, int* out, int id_base, cudaStream_t st) {
  if (S.n) k_coordination_by_id<<<blocks(S.n, 256), 256, 0, st>>>(S, out, id_base);
}
}  // namespace gdem
