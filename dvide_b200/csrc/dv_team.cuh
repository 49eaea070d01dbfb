// dv_team.cuh -- teams: the CTAs of a persistent solve kernel that work on one
// scene together, from its setup to its update, and leave it only when it is
// solved.
//
// A scene's passes are separated by barriers.  With one barrier for the whole
// grid every scene of a batch waits for every other in every pass, and all
// scenes' vectors stream through L2 between two visits.  A team has a barrier
// of its own and keeps to one scene, so scenes run at their own pace, a scene's
// vectors stay in L2 while it iterates, and the CTAs that a finished scene
// frees take the next one.
//
// The plan (k_team_plan) lists the scenes by size, largest first, and gives
// each a run of slots, one per member.  A CTA takes the next slot by one atomic.
// Slots are handed out in order, so only the team formed last can lack
// members; it waits for CTAs of earlier teams, which have all theirs and
// finish.  A team is at most the grid, and the grid is co-resident.
#pragma once

#include "dv_solve.cuh"
#include "dv_tiles.h"

namespace dv {

namespace {

// What a member knows of its team and its share of the scene (shared memory,
// written by thread 0).
struct Team {
  int s;            // scene
  int rank, m;      // this CTA's place among the team's m members
  int c0, nc;       // contacts [c0, c0 + nc)
  int t0, ntc, nt;  // first tile; contact tiles; with the bilateral rows' tiles
  int w0, w1;       // this member's bodies
  int gsize;
  TileShare share;
  int fail;
  unsigned target;  // arrivals that open the next barrier
  unsigned* bar;
};

// The member's walks over the contact tiles, and over all tiles (dv_tiles.h).
__device__ inline int contact_tile(const Team& t, int i) { return share_tile(t.share, t.ntc, i); }
__device__ inline int team_tile(const Team& t, int i) { return scene_tile(t.share, t.ntc, t.nt, i); }

__device__ inline void red_add_release(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ inline void red_add(unsigned* p, unsigned v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Barrier of a team.  Arrivals are counted without a result (the counter only
// rises: barrier k opens at k m), so a member waits for one trip to L2 and the
// polls after it.  False after a time limit or another CTA's.  The first
// barrier of a team (`joining`) may wait for members that are still busy with
// earlier scenes: there the limit starts again while any team makes progress.
// `other` is run by all threads between the arrival and the polls.
struct Nothing {
  __device__ void operator()() const {}
};
template <class K, class Fn = Nothing>
__device__ inline bool team_sync(const K& a, Team& t, bool joining = false, Fn other = Fn{}) {
  __syncthreads();
  if (threadIdx.x == 0) {
    if (a.nseg > 1 && t.rank == 0) red_add(&a.ew->progress, 1u);
    if (t.m > 1) red_add_release(t.bar, 1u);
  }
  other();
  if (threadIdx.x == 0 && t.m > 1) {
    t.target += (unsigned)t.m;
    const unsigned target = t.target;
    unsigned polls = 0, seen = 0;
    uint64_t t0 = 0;
    while ((int)(ld_acquire(t.bar) - target) < 0) {
      if (joining) __nanosleep(200);
      if ((++polls & 1023u) == 0u) {
        if (ld_acquire(&a.ew->err) & (kErrBarrierTimeout | kErrCopyTimeout)) {
          t.fail = 1;
          break;
        }
        const uint64_t now = global_ns();
        if (t0 == 0) t0 = now;
        if (joining) {
          const unsigned p = ld_acquire(&a.ew->progress);
          if (p != seen) t0 = now;
          seen = p;
        }
        if (now - t0 > a.ew->wait_limit_ns) {
          atomicOr(&a.ew->err, kErrBarrierTimeout);
          t.fail = 1;
          break;
        }
      }
    }
  }
  __syncthreads();
  return t.fail == 0;
}

// Takes the next slot of the plan; false when there is none left.  One scene
// needs no plan: its team is the first m CTAs, and the first of them clears the
// scene's error bits, as the plan does for the others: in a launch that works,
// so the mark that a failed collision detection leaves on its scene stays.
template <class K>
__device__ inline bool join_team(const K& a, Team& t, int* slot_seen) {
  __syncthreads();  // the last scene's reads of the team are done
  if (threadIdx.x == 0) {
    int s = -1, rank = 0, m = 0;
    if (a.nseg == 1) {
      m = *slot_seen ? 0 : team_size(a.sst[0].nt, a.nb, 1, gridDim.x);
      rank = blockIdx.x;
      if (rank == 0 && m > 0 && !a.refine) a.sst[0].err = 0u;
      if (rank < m && (a.seg[0].active != 0) && (!a.refine || a.sst[0].ctl.refined)) s = 0;
    } else {
      const unsigned slot = atomicAdd(&a.ew->ticket, 1u);
      if (slot < (unsigned)__ldcg(&a.ew->nslots)) {
        const int2 e = __ldcg(a.slots + slot);
        s = e.x;
        rank = e.y;
        m = __ldcg(&a.sst[s].members);
      }
    }
    *slot_seen = 1;
    t.s = s;
    if (s >= 0) {
      const SegState& X = a.sst[s];
      const SegParams& P = a.seg[s];
      t.rank = rank;
      t.m = m;
      t.c0 = X.c0;
      t.nc = X.nc;
      t.t0 = X.t0;
      t.nt = X.nt;
      t.ntc = (X.nc + kTileItems - 1) / kTileItems;
      const int n = P.b1 - P.b0;
      const int per = ((n + m - 1) / m + 31) & ~31;
      t.w0 = P.b0 + min(n, rank * per);
      t.w1 = P.b0 + min(n, (rank + 1) * per);
      t.gsize = X.gsize;
      t.share = TileShare{rank, m, a.chunk, a.contiguous};
      t.fail = 0;
      t.target = 0;
      t.bar = a.team_bar + (size_t)s * kTeamBarStride;
    }
  }
  __syncthreads();
  return t.s >= 0;
}

// Phases of a one-scene engine, timed by its first member between barriers (in
// shared memory).
struct PhaseTimer {
  unsigned long long last, ns[8];
  unsigned count[8];
  __device__ void start() {
    last = global_ns();
    for (int i = 0; i < 8; ++i) {
      ns[i] = 0;
      count[i] = 0;
    }
  }
  template <class K>
  __device__ void mark(const K& a, int phase) {
    if (a.nseg == 1 && blockIdx.x == 0 && threadIdx.x == 0) {
      const unsigned long long now = global_ns();
      ns[phase] += now - last;
      count[phase] += 1;
      last = now;
    }
  }
  template <class K>
  __device__ void store(const K& a) const {
    if (a.nseg == 1 && blockIdx.x == 0 && threadIdx.x == 0) {
      for (int i = 0; i < 8; ++i) {
        a.ew->phase_ns[i] += ns[i];
        a.ew->phase_count[i] += count[i];
      }
    }
  }
};

// Folds the eight quantities of a warp's lanes together, each in the order of
// warp_fold (strides 16, 8, 4, 2, 1; addition commutes, so which of two lanes
// adds does not matter).  At each of the first three strides a lane hands half
// of its quantities to its partner and keeps the other half: 9 exchanges for
// the eight instead of 40.  Lane l returns quantity l / 4; with kMax the last
// one is a maximum.
template <bool kMax>
__device__ __forceinline__ double warp_fold8(const double (&v)[8]) {
  const int lane = threadIdx.x & 31;
  const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
  const bool last = kMax && u16 && u8 && u4;
  double r[4], s[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double keep = u16 ? v[i + 4] : v[i];
    const double x = __shfl_xor_sync(0xffffffffu, u16 ? v[i] : v[i + 4], 16);
    r[i] = (kMax && i == 3 && u16) ? fmax(keep, x) : keep + x;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double keep = u8 ? r[i + 2] : r[i];
    const double x = __shfl_xor_sync(0xffffffffu, u8 ? r[i] : r[i + 2], 8);
    s[i] = (kMax && i == 1 && u16 && u8) ? fmax(keep, x) : keep + x;
  }
  const double keep = u4 ? s[1] : s[0];
  double x = __shfl_xor_sync(0xffffffffu, u4 ? s[0] : s[1], 4);
  double t = last ? fmax(keep, x) : keep + x;
  x = __shfl_xor_sync(0xffffffffu, t, 2);
  t = last ? fmax(t, x) : t + x;
  x = __shfl_xor_sync(0xffffffffu, t, 1);
  return last ? fmax(t, x) : t + x;
}

// The warps' folds of the tiles a member has finished, until fold_tiles_out
// completes them: warps go on to the next tile without a CTA barrier.
constexpr int kParkSlots = 8;
struct ParkBuf {
  double w[kParkSlots][8][kWarps];  // [slot][quantity][warp]
  int tile[kParkSlots];
};

template <bool kMax>
__device__ __forceinline__ void park8(ParkBuf& B, int slot, int tile, const double (&v)[8]) {
  const int lane = threadIdx.x & 31;
  const double t = warp_fold8<kMax>(v);
  if ((lane & 3) == 0) B.w[slot][lane >> 2][threadIdx.x >> 5] = t;
  if (threadIdx.x == 0) B.tile[slot] = tile;
}

// Completes the 8-warp tree of the n parked tiles' quantities into
// part[quantity][tile].
template <bool kMax, int kT>
__device__ inline void fold_parked8(ParkBuf& B, double* part, int tcap, int n) {
  __syncthreads();
  for (int i = threadIdx.x; i < n * 8; i += kT) {
    const int slot = i >> 3, q = i & 7;
    const double* w = B.w[slot][q];
    double r;
    if (kMax && q == 7)
      r = fmax(fmax(fmax(w[0], w[4]), fmax(w[2], w[6])), fmax(fmax(w[1], w[5]), fmax(w[3], w[7])));
    else
      r = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
    part[(size_t)q * tcap + B.tile[slot]] = r;
  }
  __syncthreads();
}

// Folds a scene's tile partials (in a fixed order: slot j sums tiles
// j, j + 256, ..., then the 256-slot tree), NS sums and, with kMax, a maximum
// in plane 7, into out[].  Every member of a team calls it after the pass's
// barrier and runs the scene's controller on its own copy of the scalars: the
// partials cross L2 once more per member, and the result needs no second trip
// through a word that one CTA writes and the others wait for.
// In a CTA of two groups of 256 threads the second one folds quantities 4 to 7.
template <int Q0, int Q1, int NS, bool kMax>
__device__ __forceinline__ void sum_tiles(const double* part, int tcap, int nt, int tid, double (&v)[8]) {
  constexpr int U = 4;
  for (int t = tid; t < nt; t += U * kThreads) {
    double x[8][U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int at = t + u * kThreads;
#pragma unroll
      for (int q = Q0; q < Q1; ++q)
        if (q < NS || (kMax && q == 7)) x[q][u] = at < nt ? __ldcg(part + (size_t)q * tcap + at) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (t + u * kThreads < nt) {
#pragma unroll
        for (int q = Q0; q < Q1; ++q) {
          if (q < NS) v[q] = v[q] + x[q][u];
          if (kMax && q == 7) v[q] = fmax(v[q], x[q][u]);
        }
      }
    }
  }
}
template <int NS, bool kMax, int kGroups>
__device__ __noinline__ void fold_team(const double* part, int tcap, int nt, double* scratch,
                                       double* out) {
  const int tid = threadIdx.x & (kThreads - 1);
  const bool second = kGroups == 2 && threadIdx.x >= kThreads;
  double v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = 0.0;
  if (kGroups == 1) sum_tiles<0, 8, NS, kMax>(part, tcap, nt, tid, v);
  else if (second) sum_tiles<4, 8, NS, kMax>(part, tcap, nt, tid, v);
  else sum_tiles<0, 4, NS, kMax>(part, tcap, nt, tid, v);
  const int lane = threadIdx.x & 31, warp = tid >> 5;
  const double f = warp_fold8<kMax>(v);  // of a group, its own quantities
  if ((lane & 3) == 0 && (kGroups == 1 || (lane >= 16) == second)) scratch[(lane >> 2) * 8 + warp] = f;
  __syncthreads();
  if (threadIdx.x < 8) {
    const double* w = scratch + threadIdx.x * 8;
    double r;
    if (kMax && threadIdx.x == 7)
      r = fmax(fmax(fmax(w[0], w[4]), fmax(w[2], w[6])), fmax(fmax(w[1], w[5]), fmax(w[3], w[7])));
    else
      r = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
    out[threadIdx.x] = r;
  }
  __syncwarp();  // warp 0 runs the controller
}

// A tile of a CTA of two groups: each thread of the second group hands its
// values of the tile's second 256 items to its partner, which adds them to
// those of the first 256 -- a thread's own order -- and parks the tile.  Four
// warps, two of each group, meet at a named barrier; of the two buffers one is
// still being read when the next tile's values go to the other.
struct PairBuf {
  double x[2][8][kThreads];
};
template <int NQ, bool kMax>
__device__ __forceinline__ void park_pair8(ParkBuf& B, PairBuf& X, int& flip, int slot, int tile, double (&acc)[8]) {
  const int tid = threadIdx.x & (kThreads - 1);
  const int id = 1 + (tid >> 6);
  double (*x)[kThreads] = X.x[flip];
  flip ^= 1;
  if (threadIdx.x >= kThreads) {
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q < NQ || (kMax && q == 7)) x[q][tid] = acc[q];
    asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory");
  } else {
    asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory");
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (q < NQ) acc[q] = acc[q] + x[q][tid];
      if (kMax && q == 7) acc[q] = fmax(acc[q], x[q][tid]);
    }
    park8<kMax>(B, slot, tile, acc);
  }
}

// The heads and first eight incidence entries of a member's first bodies, one
// per thread, kept for all body passes of a solve: they do not change, and
// reading them is two trips to L2 that the gathers of q wait for.
template <int kT>
struct BodyCache {
  double mi[kT];
  int s[kT], e[kT];
  uint32_t c[8][kT];
};
template <class K, int kT>
__device__ inline void fill_body_cache(const K& a, const Team& t, BodyCache<kT>& k) {
  const int b = t.w0 + threadIdx.x;
  BodyHead h{0.0, 0, 0};
  if (b < t.w1) h = body_head(a, b);
  k.mi[threadIdx.x] = h.mi;
  k.s[threadIdx.x] = h.s;
  k.e[threadIdx.x] = h.e;
#pragma unroll
  for (int j = 0; j < 8; ++j) k.c[j][threadIdx.x] = (h.s + j < h.e) ? __ldg(a.inc + h.s + j) : 0u;
}

// Body pass of a member: w_b = minv_b (D^T x)_b for its bodies.  Past the kept
// ones, heads load two rounds ahead and each body's first eight incidence
// entries one round ahead, while the current round gathers.
template <class T, bool kAR, int kT>
__device__ inline void team_body_pass(const KArgs<T>& a, const Team& t, const BodyCache<kT>& k,
                                      typename Vec4<T>::type* w, const typename Vec4<T>::type* q) {
  const int e = t.w1;
  int b = t.w0 + threadIdx.x;
  if (b >= e) return;
  BodyHead h{k.mi[threadIdx.x], k.s[threadIdx.x], k.e[threadIdx.x]}, hn{0.0, 0, 0};
  if (b + kT < e) hn = body_head(a, b + kT);
  uint32_t c[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) c[j] = k.c[j][threadIdx.x];
  for (; b < e; b += kT) {
    const int bnn = b + 2 * kT;
    BodyHead hnn{0.0, 0, 0};
    if (bnn < e) hnn = body_head(a, bnn);
    uint32_t cn[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) cn[j] = (hn.s + j < hn.e) ? __ldg(a.inc + hn.s + j) : 0u;
    body_w<T, kAR>(a, w, q, b, h, c);
    h = hn;
    hn = hnn;
#pragma unroll
    for (int j = 0; j < 8; ++j) c[j] = cn[j];
  }
}

}  // namespace

}  // namespace dv
