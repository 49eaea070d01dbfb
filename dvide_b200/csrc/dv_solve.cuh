// dv_solve.cuh -- device machinery shared by the persistent solve kernels
// (APGD in dv_apgd.cu, PGJ in dv_pgj.cu, PGS in dv_pgs.cu): kernel arguments,
// the tangent frame and the matrix-free products with the frame, the ordered
// tile reductions, the body gather, bilateral rows, and the per-warp staging
// of bulk asynchronous copies.  Every wait has a time limit.
#pragma once

#include <stdio.h>
#include <stdlib.h>

#include "dv_internal.cuh"

namespace dv {

namespace {

constexpr int kWarps = kThreads / 32;
constexpr int kMaxWarps = 16;  // warps of the largest CTA that has stages
constexpr int kSub = kThreads;  // contacts per sub-tile

// Phases timed between barriers (EngineWords::phase_ns).
enum Phase : int {
  kPhaseSetup = 0,     // k, r, Lipschitz estimate
  kPhaseStep = 1,      // gamma_new = P(y - t g): first iteration or backtrack
  kPhaseBody = 3,      // body gather w = Minv D^T q
  kPhaseProduct = 4,   // N gamma_new, objective, residual, look-ahead step
  kPhaseFinal = 5,     // gamma = gamma_hat, update
};

template <class T> struct Vec4;
template <> struct Vec4<double> { using type = double4; };
template <> struct Vec4<float> { using type = float4; };

template <class T>
struct KArgs {
  int nb, nseg;
  int solve_only;     // 1: the solve without the update (v, p, f_contact, clock untouched)
  int refine;         // 1: FP64 refinement of the solves a mixed-precision launch marked
  int tcap;           // plane stride of the partials
  int chunk, contiguous;
  size_t S;           // plane stride of contact arrays
  size_t WS;          // plane stride of the warm-start arena
  double4* p4;
  double4* v4;
  double4* k4;
  const double4* __restrict__ f4;
  double4* fc4;
  double4* wd;        // body vector, double4 (setup); reinterpreted as Vec4<T> in iterations
  const double* __restrict__ minv;
  const uint32_t* __restrict__ ida;
  const uint32_t* __restrict__ idb;
  const double* __restrict__ F;
  const double* __restrict__ gap;
  T* r;
  T* fr;              // PGJ, PGS: frame words (FrameWords), 3 planes, written by the setup pass
  T* blk;             // APGD: the contacts' constants in blocks of 32 (the same memory)
  const int* __restrict__ inc_start;
  const uint32_t* __restrict__ inc;
  T* G[5];            // APGD: iterate blocks (3 planes of 32, then the product's 3); PGJ, PGS: planes
  double4* qd;        // contact vector q, double4 (final pass); Vec4<T> in iterations
  double* gamma;
  uint32_t* wid;      // matched warm start: B of the pair per warm slot (segment-relative)
  int* ws;            // matched warm start: per body, first warm slot of its A-contacts
  int* wc;            // ... and their count
  const int* __restrict__ cbase;     // this step's contact offsets (unpadded) per body
  const int* __restrict__ cnt_cont;  // this step's contacts with A = body
  int* body_count;    // PGS: contacts of each body that the sweep has updated (scratch)
  double* part;
  const SegParams* __restrict__ seg;
  SegState* sst;
  EngineWords* ew;
  const int2* slots;       // the plan of the teams: (scene, rank) per slot
  unsigned* team_bar;      // arrivals of each scene's team, kTeamBarStride words apart
  // bilateral DOF rows (nbil = 0: none; FP64 iterates only)
  int nbil;
  const int2* __restrict__ bil_off;
  const double4* __restrict__ bil_info;
  const int* __restrict__ bil_inc_start;
  const uint32_t* __restrict__ bil_inc;
  T* bG[5];            // iterates of the rows (the contacts' G[k] slot k)
  T* bNG[5];           // their products
  T* br;               // Schur vector of the rows
  T* bq;               // the rows' share of the body gather (the contacts' q)
  double* bil_gam;     // warm start / solution of the rows
  double* bil_b;       // b of the rows (for the CCP violation)
  double* seg_time;    // System::time of each segment at the step's start
  // APGD anti-relaxation (the kAR kernel): r_n and ar planes (current, next;
  // stride S), v = Minv (k + D^T x) of the iterate under test
  double* ar_r0;
  double* ar_v;
  double4* v_ar;
};

template <class T>
struct Frame {
  T n0, n1, n2, u0, u1, u2, v0, v1, v2;
};

// The FP64 frame of a normal in the scene's mode.
__device__ inline Frame<double> frame_d(double n0, double n1, double n2, bool exact) {
  d3 u, v;
  frame_from_normal(mk3(n0, n1, n2), &u, &v, exact);
  Frame<double> f;
  f.n0 = n0; f.n1 = n1; f.n2 = n2;
  f.u0 = u.x; f.u1 = u.y; f.u2 = u.z;
  f.v0 = v.x; f.v1 = v.y; f.v2 = v.z;
  return f;
}

// What a frame cannot cheaply be rebuilt without, per contact: u has one zero
// component by construction (System.cu:753-762), so its other two and the
// reciprocal length of n x u give the frame back with twelve multiplications,
// in the same order as frame_from_normal (the same bits), where rebuilding it
// from the normal alone takes a division, two square roots and two reciprocals
// in one dependent chain.
template <class T>
struct FrameWords {
  T a, b;  // u_x, and u_z (or u_y when n is along y)
  T iv;    // 1 / |n x u|
};

__device__ inline FrameWords<double> frame_words(double n0, double n1, double n2, bool exact) {
  const bool along = n2 == 0 && n0 == 0;
  d3 r;
  if (n2 != 0) r = mk3(1, 0, -n0 / n2);
  else if (n0 != 0) r = mk3(-n2 / n0, 0, 1);
  else r = mk3(1, -n0 / n1, 0);
  const d3 u = scale3(r, inv_length3x(r, exact));
  FrameWords<double> w;
  w.a = u.x;
  w.b = along ? u.y : u.z;
  w.iv = inv_length3x(cross3(mk3(n0, n1, n2), u), exact);
  return w;
}
// System.cu:753-762 in float arithmetic (mixed path; it has no exact mode).
__device__ inline FrameWords<float> frame_words(float n0, float n1, float n2, bool) {
  const bool along = n2 == 0.0f && n0 == 0.0f;
  float ux, uy, uz;
  if (n2 != 0.0f) {
    ux = 1.0f; uy = 0.0f; uz = __fdiv_rn(-n0, n2);
  } else if (n0 != 0.0f) {
    ux = __fdiv_rn(-n2, n0); uy = 0.0f; uz = 1.0f;
  } else {
    ux = 1.0f; uy = __fdiv_rn(-n0, n1); uz = 0.0f;
  }
  const float iu = __fdiv_rn(1.0f, __fsqrt_rn(ux * ux + uy * uy + uz * uz));
  ux *= iu; uy *= iu; uz *= iu;
  const float vx = n1 * uz - n2 * uy, vy = n2 * ux - n0 * uz, vz = n0 * uy - n1 * ux;
  FrameWords<float> w;
  w.a = ux;
  w.b = along ? uy : uz;
  w.iv = __fdiv_rn(1.0f, __fsqrt_rn(vx * vx + vy * vy + vz * vz));
  return w;
}

template <class T>
__device__ inline Frame<T> make_frame(T n0, T n1, T n2, const FrameWords<T>& w) {
  const bool along = n2 == T(0) && n0 == T(0);
  Frame<T> f;
  f.n0 = n0; f.n1 = n1; f.n2 = n2;
  f.u0 = w.a;
  f.u1 = along ? w.b : T(0);
  f.u2 = along ? T(0) : w.b;
  f.v0 = (n1 * f.u2 - n2 * f.u1) * w.iv;
  f.v1 = (n2 * f.u0 - n0 * f.u2) * w.iv;
  f.v2 = (n0 * f.u1 - n1 * f.u0) * w.iv;
  return f;
}

// The frame of contact c from the normal and the words that a solve's setup
// pass left in the fr planes.
template <class T>
__device__ inline Frame<T> load_frame(const KArgs<T>& a, int c) {
  const FrameWords<T> w{a.fr[c], a.fr[a.S + c], a.fr[2 * a.S + c]};
  return make_frame<T>((T)__ldg(a.F + c), (T)__ldg(a.F + a.S + c), (T)__ldg(a.F + 2 * a.S + c), w);
}

// Setup: forms the words of contact c, keeps them and returns the frame.
template <class T>
__device__ inline Frame<T> start_frame(const KArgs<T>& a, int c, bool exact) {
  const T n0 = (T)__ldg(a.F + c), n1 = (T)__ldg(a.F + a.S + c), n2 = (T)__ldg(a.F + 2 * a.S + c);
  const FrameWords<T> w = frame_words(n0, n1, n2, exact);
  a.fr[c] = w.a;
  a.fr[a.S + c] = w.b;
  a.fr[2 * a.S + c] = w.iv;
  return make_frame<T>(n0, n1, n2, w);
}

template <class T>
__device__ inline Frame<double> load_frame_fp64(const KArgs<T>& a, int c, bool exact) {
  return frame_d(__ldg(a.F + c), __ldg(a.F + a.S + c), __ldg(a.F + 2 * a.S + c), exact);
}

// Stores of the vectors a pass writes and the next pass reads at once (q for
// the body pass, w for the contact pass's gathers), with an L2 evict-last
// priority: each contact pass streams more contact data than L2 holds, and
// without the hint these lines are the first to go.  A hint, not a value
// change.
__device__ inline uint64_t l2_evict_last_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ inline void store_keep(double4* addr, const double4& v) {
  const uint64_t pol = l2_evict_last_policy();
  asm volatile("st.global.L2::cache_hint.v4.f64 [%0], {%1, %2, %3, %4}, %5;" ::"l"(addr),
               "d"(v.x), "d"(v.y), "d"(v.z), "d"(v.w), "l"(pol)
               : "memory");
}
__device__ inline void store_keep(float4* addr, const float4& v) {
  const uint64_t pol = l2_evict_last_policy();
  asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(addr),
               "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "l"(pol)
               : "memory");
}
// One 4-vector by one load (32 bytes in FP64: a sector, where two 16-byte
// loads would each ask for it).
__device__ inline double4 load_vec(const double4* p) {
  double4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
               : "l"(p));
  return v;
}
__device__ inline float4 load_vec(const float4* p) { return *p; }

// q = F x : q_k = (n_k x0 + u_k x1) + v_k x2
template <class T, class V>
__device__ inline V f_times(const Frame<T>& f, T x0, T x1, T x2) {
  V q;
  q.x = (f.n0 * x0 + f.u0 * x1) + f.v0 * x2;
  q.y = (f.n1 * x0 + f.u1 * x1) + f.v1 * x2;
  q.z = (f.n2 * x0 + f.u2 * x1) + f.v2 * x2;
  q.w = T(0);
  return q;
}

// (F^T d)_row = (f_x d_x + f_y d_y) + f_z d_z with d = w_A - w_B
template <class T, class V>
__device__ inline void ft_times(const Frame<T>& f, V wa, V wb, T* o0, T* o1, T* o2) {
  T d0 = wa.x - wb.x, d1 = wa.y - wb.y, d2 = wa.z - wb.z;
  *o0 = (f.n0 * d0 + f.n1 * d1) + f.n2 * d2;
  *o1 = (f.u0 * d0 + f.u1 * d1) + f.u2 * d2;
  *o2 = (f.v0 * d0 + f.v1 * d1) + f.v2 * d2;
}

// Dot products of the reductions, always in FP64.
template <class A, class B>
__device__ inline double dot3i(A a0, A a1, A a2, B b0, B b1, B b2) {
  return ((double)a0 * (double)b0 + (double)a1 * (double)b1) + (double)a2 * (double)b2;
}

// Folds a scene's tile maxima, planes 0 to NM - 1 of its nt tiles from t0 on, to
// thread 0.  Four tiles' loads per plane are in flight at once.
template <int NM, class K>
__device__ inline void fold_tile_maxima(const K& a, int t0, int nt, double (&out)[NM], double* scratch) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* p = a.part + t0;
  double mx[NM];
#pragma unroll
  for (int q = 0; q < NM; ++q) mx[q] = 0.0;
  int t = threadIdx.x;
  for (; t + (U - 1) * kThreads < nt; t += U * kThreads) {
    double x[NM][U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int q = 0; q < NM; ++q) x[q][u] = __ldcg(p + (size_t)q * a.tcap + t + u * kThreads);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int q = 0; q < NM; ++q) mx[q] = fmax(mx[q], x[q][u]);
    }
  }
  for (; t < nt; t += kThreads) {
#pragma unroll
    for (int q = 0; q < NM; ++q) mx[q] = fmax(mx[q], __ldcg(p + (size_t)q * a.tcap + t));
  }
#pragma unroll
  for (int q = 0; q < NM; ++q) mx[q] = warp_max(mx[q]);
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NM; ++q) scratch[q * kWarps + warp] = mx[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NM; ++q) {
      double w = lane < kWarps ? scratch[q * kWarps + lane] : 0.0;
#pragma unroll
      for (int off = kWarps / 2; off >= 1; off >>= 1) w = fmax(w, __shfl_down_sync(0xffffffffu, w, off));
      out[q] = w;
    }
  }
  __syncthreads();
}

// Deferred tile folds: the warps park their maxima of a tile and go on to the
// next; fold_parked_max() completes the parked tiles.
constexpr int kMaxDefer = 8, kMaxima = 3;
struct DeferBuf {
  double w[kMaxDefer][kMaxima][kWarps];  // [slot][quantity][warp]
  int tile[kMaxDefer];
};

// ---- maxima reductions of PGJ and PGS (only maxima: no summation order) ----
// max_c -min(0, scale * x_n - |x_t|), a NaN term counting 0 (PGJ.cu:112-142, PGS.cu:335-365)
__device__ inline double pgj_feasible(double xn, double xt1, double xt2, double scale) {
  double v = scale * xn - sqrt(xt1 * xt1 + xt2 * xt2);
  if (v != v) v = 0.0;
  return -fmin(0.0, v);
}

// Per-tile maxima: each warp folds (exact, order-free) and parks them; the
// CTA completes the 8-warp fold later and writes planes 0..NQ-1.
template <int NQ>
__device__ inline void park_max(DeferBuf& B, int slot, int tile, const double (&m)[NQ]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const double v = warp_max(m[q]);
    if (lane == 0) B.w[slot][q][warp] = v;
  }
  if (threadIdx.x == 0) B.tile[slot] = tile;
}

template <int NQ, class K>
__device__ inline void fold_parked_max(const K& a, DeferBuf& B, int n) {
  __syncthreads();
  for (int i = threadIdx.x; i < n * NQ; i += kThreads) {
    const int slot = i / NQ, q = i - slot * NQ;
    const double* w = B.w[slot][q];
    double r = w[0];
    for (int k = 1; k < kWarps; ++k) r = fmax(r, w[k]);
    a.part[(size_t)q * a.tcap + B.tile[slot]] = r;
  }
  __threadfence();
  __syncthreads();
}

// Eight incidence entries c[0, n) of a body's run (n <= 8): their q gathered
// together, then added to (ax, ay, az) in order, -q for a B side.
template <class T, class V>
__device__ inline void add_q8(const V* q, const uint32_t* c, int n, T& ax, T& ay, T& az) {
  V qq[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j < n) {
      qq[j] = load_vec(q + (c[j] & 0x7fffffffu));
    } else {
      qq[j].x = T(0); qq[j].y = T(0); qq[j].z = T(0); qq[j].w = T(0);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j < n) {
      if (c[j] & 0x80000000u) {
        ax = ax - qq[j].x; ay = ay - qq[j].y; az = az - qq[j].z;
      } else {
        ax = ax + qq[j].x; ay = ay + qq[j].y; az = az + qq[j].z;
      }
    }
  }
}

// Sum of -q over B-side contacts, then +q over A-side contacts, ascending
// contact order (the flat incidence list).  Sixteen incidence entries are
// read at once (a settled body has about seven contacts, often more than
// eight), their q in two groups of eight; the additions stay in order.
template <class T, class V, class K>
__device__ inline V gather_q(const K& a, const V* q, int s, int e) {
  T ax = T(0), ay = T(0), az = T(0);
  for (int i = s; i < e; i += 16) {
    uint32_t c[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) c[j] = (i + j < e) ? __ldg(a.inc + i + j) : 0u;
    add_q8<T, V>(q, c, e - i, ax, ay, az);
    if (i + 8 < e) add_q8<T, V>(q, c + 8, e - i - 8, ax, ay, az);
  }
  V r;
  r.x = ax; r.y = ay; r.z = az; r.w = T(0);
  return r;
}

// gather_q with the run's first eight entries already loaded (c0; zero past
// the run): entries 8..15 load alongside the first group's q.  The same sums
// in the same order.
template <class T, class V, class K>
__device__ inline V gather_q_pre(const K& a, const V* q, int s, int e, const uint32_t* c0) {
  T ax = T(0), ay = T(0), az = T(0);
  uint32_t c1[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) c1[j] = (s + 8 + j < e) ? __ldg(a.inc + s + 8 + j) : 0u;
  add_q8<T, V>(q, c0, e - s, ax, ay, az);
  if (s + 8 < e) add_q8<T, V>(q, c1, e - s - 8, ax, ay, az);
  for (int i = s + 16; i < e; i += 16) {
    uint32_t c[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) c[j] = (i + j < e) ? __ldg(a.inc + i + j) : 0u;
    add_q8<T, V>(q, c, e - i, ax, ay, az);
    if (i + 8 < e) add_q8<T, V>(q, c + 8, e - i - 8, ax, ay, az);
  }
  V r;
  r.x = ax; r.y = ay; r.z = az; r.w = T(0);
  return r;
}

template <class T, class V, class K>
__device__ inline V gather_q(const K& a, const V* q, int b) {
  return gather_q<T, V>(a, q, __ldg(a.inc_start + b), __ldg(a.inc_start + b + 1));
}

// Bilateral DOF rows.  Tile t of a segment with contacts [0, nc) and tiles
// starting at t0 is a tile of its rows when it lies past the contact tiles;
// returns the tile's first row (segment-relative), else -1.
__device__ inline int bil_tile_k0(int t, int t0, int nc) {
  const int ntc = (nc + kTileItems - 1) / kTileItems;
  return (t - t0) >= ntc ? (t - t0 - ntc) * kTileItems : -1;
}

// Row i of D w (System.cu:622-638): w[A] - w[B], or w[A] for one DOF.  o holds
// the DOFs' element offsets (4 body + axis) into a 4-wide body vector.
template <class T>
__device__ inline T bil_dw(int2 o, const T* w) {
  const T wa = w[o.x];
  return o.y >= 0 ? wa - w[o.y] : wa;
}

// The rows' part of (D^T x)_b, added after the contacts' part: +x_i at DOF A,
// -x_i at DOF B, ascending rows.  x is written inside the kernel (read through L2).
template <class T, class V>
__device__ inline void add_bilateral(const int* __restrict__ start, const uint32_t* __restrict__ inc,
                                     const T* x, int b, V& s) {
  const int e0 = __ldg(start + b), e1 = __ldg(start + b + 1);
  for (int e = e0; e < e1; ++e) {
    const uint32_t code = __ldg(inc + e);
    const T v = __ldcg(x + (code >> 3));
    const int k = (code >> 1) & 3;
    if (code & 1u) {
      if (k == 0) s.x = s.x - v; else if (k == 1) s.y = s.y - v; else s.z = s.z - v;
    } else {
      if (k == 0) s.x = s.x + v; else if (k == 1) s.y = s.y + v; else s.z = s.z + v;
    }
  }
}

// A solver error of segment s; with stop_on_seg_err it also stops the steps
// that follow (every kernel checks EngineWords::err first).
template <class K>
__device__ inline void seg_error(const K& a, int s, unsigned bit) {
  atomicOr(&a.sst[s].err, bit);
  if (a.ew->stop_on_seg_err) atomicOr(&a.ew->err, bit);
}

// The words a body's gather starts from, its inverse mass and the bounds of its
// incidence run, loaded together so that they cost one memory round trip.
struct BodyHead {
  double mi;
  int s, e;
};

template <class K>
__device__ inline BodyHead body_head(const K& a, int b) {
  BodyHead h;
  h.mi = __ldg(a.minv + b);
  h.s = __ldg(a.inc_start + b);
  h.e = __ldg(a.inc_start + b + 1);
  return h;
}

// w_b = minv_b * (D^T x)_b of one body; fixed bodies keep w = 0.
// kAR: also v = Minv (k + D^T x) for the anti-relaxation (APGD.cu:338-340;
// 0 for fixed bodies, whose v enters only as squares).
// c0 holds the body's first eight incidence entries, loaded a round ahead by the
// body pass (zero past its run).
template <class T, bool kAR>
__device__ inline void body_w(const KArgs<T>& a, typename Vec4<T>::type* w,
                              const typename Vec4<T>::type* q, int b, const BodyHead& h,
                              const uint32_t* c0) {
  using V = typename Vec4<T>::type;
  const double mi = h.mi;
  if (mi != 0.0) {
    V s = gather_q_pre<T, V>(a, q, h.s, h.e, c0);
    if (a.nbil) add_bilateral<T, V>(a.bil_inc_start, a.bil_inc, a.bq, b, s);
    T m = (T)mi;
    V o;
    o.x = m * s.x; o.y = m * s.y; o.z = m * s.z; o.w = T(0);
    store_keep(w + b, o);
    if (kAR) {
      const double4 k = a.k4[b];
      a.v_ar[b] = make_double4(mi * (k.x + (double)s.x), mi * (k.y + (double)s.y),
                               mi * (k.z + (double)s.z), 0.0);
    }
  } else if (kAR) {
    a.v_ar[b] = make_double4(0.0, 0.0, 0.0, 0.0);
  } else if (sizeof(T) != sizeof(double)) {
    // the FP32 view of w overlays the FP64 setup values: store the zero
    V o;
    o.x = T(0); o.y = T(0); o.z = T(0); o.w = T(0);
    store_keep(w + b, o);
  }
}

// Members of a team: one per `per` contact tiles or 256 * per bodies, as many
// as the grid has at most.
__device__ inline int team_size(int nt, int nb, int per, int grid) {
  const int m = max((nt + per - 1) / per, (nb + kThreads * per - 1) / (kThreads * per));
  return max(1, min(m, grid));
}

// A buffer holding none of the iterates in use (5 buffers, at most 4 in use).
__device__ inline int free_slot(int a, int b, int c, int d) {
  for (int i = 0; i < 5; ++i)
    if (i != a && i != b && i != c && i != d) return i;
  return 0;
}

// ---------------------------------------------------------------------------
// Shared-memory staging of the contact pass, per warp.  A CTA walks its
// sub-tiles (256 consecutive contacts, kItemsPerThread per reduction tile) in
// order; warp w owns contacts [32w, 32w+32) of each sub-tile and two stages of
// its own.  While the warp works on one, its lane 0 has already issued the
// bulk copies of the next sub-tile into the other, completed on the warp's own
// mbarrier, so warps never wait for each other except at the reductions.
// A segment's contacts start on a multiple of 256, so every copy starts on a
// 128-byte boundary.
// ---------------------------------------------------------------------------
struct Staging {
  unsigned char* base;  // warp w, stage s at base + (2w + s) * stage_bytes
  unsigned stage_bytes;
  uint64_t* bar;        // mbarrier of warp w, stage s: bar[2w + s]
  unsigned phase;       // bit s: parity the next wait on this warp's stage s expects
};

// Per warp, bit s: copies issued into stage s and not yet seen complete; one
// byte per warp after the mbarriers (lane 0 writes it).
__device__ inline volatile unsigned char* stage_pending(const Staging& st) {
  return reinterpret_cast<volatile unsigned char*>(st.bar + 2 * kMaxWarps) + (threadIdx.x >> 5);
}
__device__ inline void mark_stage_issued(const Staging& st, int s) {
  if ((threadIdx.x & 31) == 0) *stage_pending(st) |= (unsigned char)(1u << s);
}

// Waits for the phase of parity `parity` of an mbarrier to complete; false
// after `*limit_ns` (read only if the first test fails).
__device__ inline bool bounded_mbar_wait(uint64_t* bar, unsigned parity,
                                         const unsigned long long* limit_ns) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    const uint64_t limit = *limit_ns;
    const uint64_t t0 = global_ns();
    while (!(ok = mbar_try_wait(bar, parity))) {
      if (global_ns() - t0 > limit) break;
    }
  }
  return ok;
}

// Bounded wait on this warp's stage s.
__device__ inline bool bounded_stage_wait(Staging& st, int s, const unsigned long long* limit_ns) {
  const int w = threadIdx.x >> 5;
  const unsigned par = (st.phase >> s) & 1u;
  uint64_t* bar = st.bar + 2 * w + s;
  const bool ok = bounded_mbar_wait(bar, par, limit_ns);
  if (ok) {
    st.phase ^= (1u << s);
    if ((threadIdx.x & 31) == 0) *stage_pending(st) &= (unsigned char)~(1u << s);
  }
  return ok;
}

// Waits for this warp's stage s; false after a timeout (error recorded, the
// stage left pending for drain_warp_stages).
template <class K>
__device__ inline bool wait_warp_stage(const K& a, Staging& st, int s) {
  const bool ok = bounded_stage_wait(st, s, &a.ew->wait_limit_ns);
  if (!ok && (threadIdx.x & 31) == 0) atomicOr(&a.ew->err, kErrCopyTimeout);
  __syncwarp();
  return ok;
}

// Before a CTA leaves the kernel early: waits once more, again with a time
// limit, for the copies this warp still has in flight into its stages.
__device__ __noinline__ void drain_warp_stages(Staging st, const unsigned long long* limit_ns) {
  __syncwarp();
  const unsigned pend = __shfl_sync(0xffffffffu, (unsigned)*stage_pending(st), 0);
  for (int s = 0; s < 2; ++s)
    if ((pend >> s) & 1u) bounded_stage_wait(st, s, limit_ns);
  __syncwarp();
}

// Kernel arguments of the solve kernels for an engine and a launch shape.
template <class T>
KArgs<T> make_kargs(SceneDev& sd, const SolveConfig& cfg) {
  KArgs<T> a;
  a.nb = sd.nb;
  a.nseg = sd.nseg;
  a.solve_only = 0;
  a.refine = 0;
  a.tcap = sd.tcap;
  a.chunk = cfg.chunk > 0 ? cfg.chunk : 1;
  a.contiguous = cfg.contiguous;
  a.S = sd.ccap;
  a.WS = sd.wtotal;
  a.p4 = sd.p4;
  a.v4 = sd.v4;
  a.k4 = sd.k4;
  a.f4 = sd.f4;
  a.fc4 = sd.fc4;
  a.wd = sd.w4;
  a.minv = sd.minv;
  a.ida = sd.ida;
  a.idb = sd.idb;
  a.F = sd.F;
  a.gap = sd.gap;
  a.r = reinterpret_cast<T*>(sd.r);
  a.fr = a.blk = reinterpret_cast<T*>(sd.blk);
  a.inc_start = sd.inc_start;
  a.inc = sd.inc;
  for (int k = 0; k < 5; ++k) a.G[k] = reinterpret_cast<T*>(sd.G[k]);
  a.qd = sd.q;
  a.gamma = sd.gamma;
  a.wid = sd.wid;
  a.ws = sd.ws;
  a.wc = sd.wc;
  a.cbase = sd.cbase;
  a.cnt_cont = sd.cnt_cont;
  a.body_count = sd.cnt_cand;
  a.part = sd.part;
  a.seg = sd.seg;
  a.sst = sd.sst;
  a.ew = sd.ew;
  a.slots = sd.slots;
  a.team_bar = sd.team_bar;
  a.nbil = sizeof(T) == sizeof(double) ? sd.nbil : 0;
  a.bil_off = sd.bil_off;
  a.bil_info = sd.bil_info;
  a.bil_inc_start = sd.bil_inc_start;
  a.bil_inc = sd.bil_inc;
  T* bw = a.nbil ? reinterpret_cast<T*>(sd.bil_work) : nullptr;
  const size_t nbl = (size_t)sd.nbil;
  for (int k = 0; k < 5; ++k) {
    a.bG[k] = bw ? bw + k * nbl : nullptr;
    a.bNG[k] = bw ? bw + (5 + k) * nbl : nullptr;
  }
  a.br = bw ? bw + 10 * nbl : nullptr;
  a.bq = bw ? bw + 11 * nbl : nullptr;
  a.bil_gam = sd.bil_gam;
  a.bil_b = sd.bil_b;
  a.seg_time = sd.seg_time;
  a.ar_r0 = sd.ar_r0;
  a.ar_v = sd.ar_v;
  a.v_ar = sd.v_ar;
  return a;
}

}  // namespace

}  // namespace dv
