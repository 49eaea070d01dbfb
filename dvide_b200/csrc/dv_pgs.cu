// dv_pgs.cu -- the time step with the PGS solver (System(6), PGS.cu:367-459)
// for every segment of an engine, as one persistent cooperative kernel per
// step: applied impulse, Schur vector, PGS iterations, update.  FP64 only.
//
// PGS: gamma starts at (1, 0, 0) per contact (:372, no warm start), the body
// velocities at v = Minv D^T gamma + Minv k (:376-379), B_c as in PGJ
// (buildB_PGS, :272-304), and each iteration is a Gauss-Seidel sweep over the
// contacts in their order (updateImpulseVector_CPU, :143-224): per contact
//   gamma_hat = P(gamma - omega B (D_c^T v + b_c))     (omega 0.3)
//   gamma     = lambda gamma_hat + (1 - lambda) gamma  (lambda 2/3)
//   v_A += minv_A F delta,  v_B -= minv_B F delta,  delta = lambda (gamma_hat - gamma_old)
// followed by the residual max(feasibleX(gamma), feasibleY(N gamma + r),
// max_c |(N gamma + r)_c . gamma_c|) (:402-426).
//
// A sweep is sequential by definition: every update reads the velocities the
// previous ones wrote.  But an update reads and writes two bodies only, so it
// depends on the last earlier contact of either body and on no other: contacts
// whose earlier neighbours are done can be updated together, with the same
// values as one after another.  One CTA of a scene's team sweeps, 256 contacts
// at a time in their order, one per thread, in rounds: each body counts its
// contacts done, and a contact goes when it is next for both of its bodies.
// A window of a pile takes about a dozen rounds.  A fixed body's velocity stays
// what it is (its inverse mass is zero), so its contacts need not wait for each
// other -- unless a product with that zero is not a number: then the sweep
// starts again with the fixed bodies' order kept too.  One thread sweeping in
// order took 1.8 us per contact, the time of its dependent loads and of one
// cone projection.
//
// The sweep writes q = F gamma as it goes, which leaves the residual's Schur
// product to the parallel body and contact passes.  The working velocities
// live in v4, which the update at the end of the step overwrites, as the
// reference's sweep overwrites System::v.
#include <string.h>

#include <algorithm>
#include <vector>

#include "dv_team.cuh"

namespace dv {

namespace {

constexpr double kPgsOmega = 0.3;
constexpr double kPgsLambda = 2.0 / 3.0;
constexpr int kPgsChunk = 32768;  // contacts between two barriers: keeps the others' wait short

// Scalars of a solve, one copy per member.
struct PgsSolve {
  double residual;
  int k, cur, iterations, sweeps, done;
};

// After a residual pass (thread 0): m holds the maxima of feasibleX(gamma),
// feasibleY(N gamma + r) and |(N gamma + r) . gamma|.
__device__ inline void pgs_ctl(PgsSolve& C, const double* m, const SegParams& P) {
  const int k = C.k;
  const double residual = fmax(fmax(m[0], m[1]), m[2]);
  C.residual = residual;
  if (residual < P.tol) {
    C.done = 1;
    C.iterations = k;
  } else if (k + 1 >= P.max_iter) {
    C.done = 1;
    C.iterations = P.max_iter;
  }
  C.sweeps = k + 1;
  if (!C.done) C.k = k + 1;
}

// Contacts [from, to) of the scene, from gamma in Gc to gamma in Gn, by one CTA
// (all its threads).  `strict`: fixed bodies' contacts one after another too.
// Returns, in every thread, whether a fixed body's velocity would have changed
// (only without `strict`).  Every round updates at least the first contact that
// is left, so none of a window waits for more rounds than the window has contacts;
// one that does, because the counts and the incidence disagree, gives up, and the
// sweep ends with an error.
enum PgsSweep : int { kSweepDone = 0, kSweepOdd = 1, kSweepStalled = 2 };
__device__ PgsSweep pgs_sweep(const KArgs<double>& a, const Team& tm, const SegParams& P, const double* Gc,
                          double* Gn, const Cone<double>& cone, int from, int to, bool strict) {
  __shared__ int s_stalled;
  if (threadIdx.x == 0) s_stalled = 0;
  const size_t S = a.S;
  const double h = P.h;
  const double* Bc = a.G[4];
  const int2* place = reinterpret_cast<const int2*>(a.G[3]);  // c among A's and B's contacts
  double4* v = a.v4;
  double4* q = a.qd;
  int* done_of = a.body_count;
  bool odd = false;
  for (int k0 = from; k0 < to; k0 += kThreads) {
    const int k = k0 + threadIdx.x;
    const int c = tm.c0 + k;
    bool todo = k < to;
    uint32_t ia = 0, ib = 0;
    Frame<double> f{};
    double ob = 0, bn = 0, mia = 0, mib = 0, o0 = 0, o1 = 0, o2 = 0;
    int2 at = make_int2(0, 0);
    if (todo) {
      ia = __ldg(a.ida + c);
      ib = __ldg(a.idb + c);
      f = load_frame<double>(a, c);
      ob = kPgsOmega * Bc[c];
      bn = __ldg(a.gap + c) / h;
      mia = __ldg(a.minv + ia);
      mib = __ldg(a.minv + ib);
      o0 = Gc[0 * S + c];
      o1 = Gc[1 * S + c];
      o2 = Gc[2 * S + c];
      at = place[c];
    }
    const bool wait_a = strict || mia != 0.0, wait_b = strict || mib != 0.0;
    int waited = 0;
    while (__syncthreads_or(todo)) {
      const bool go = todo && (!wait_a || done_of[ia] == at.x) && (!wait_b || done_of[ib] == at.y);
      __syncthreads();  // every thread has read the counts
      if (!go) {
        if (++waited > kThreads && todo) {
          todo = false;
          s_stalled = 1;
        }
        continue;
      }
      const double4 va = v[ia], vb = v[ib];
      double g0 = o0 - ob * (f.n0 * va.x + f.n1 * va.y + f.n2 * va.z - f.n0 * vb.x - f.n1 * vb.y -
                             f.n2 * vb.z + bn);
      double g1 = o1 - ob * (f.u0 * va.x + f.u1 * va.y + f.u2 * va.z - f.u0 * vb.x - f.u1 * vb.y -
                             f.u2 * vb.z);
      double g2 = o2 - ob * (f.v0 * va.x + f.v1 * va.y + f.v2 * va.z - f.v0 * vb.x - f.v1 * vb.y -
                             f.v2 * vb.z);
      project_cone<double>(g0, g1, g2, cone);
      const double la = kPgsLambda, lb = 1.0 - kPgsLambda;
      const double y0 = la * g0 + lb * o0, y1 = la * g1 + lb * o1, y2 = la * g2 + lb * o2;
      Gn[0 * S + c] = y0;
      Gn[1 * S + c] = y1;
      Gn[2 * S + c] = y2;
      const double d0 = la * (g0 - o0), d1 = la * (g1 - o1), d2 = la * (g2 - o2);
      const double ex = f.n0 * d0 + f.u0 * d1 + f.v0 * d2;
      const double ey = f.n1 * d0 + f.u1 * d1 + f.v1 * d2;
      const double ez = f.n2 * d0 + f.u2 * d1 + f.v2 * d2;
      const double4 na = make_double4(va.x + mia * ex, va.y + mia * ey, va.z + mia * ez, 0.0);
      // a contact's bodies differ
      const double4 nb = make_double4(vb.x - mib * ex, vb.y - mib * ey, vb.z - mib * ez, 0.0);
      if (wait_a) {
        v[ia] = na;
        done_of[ia] = at.x + 1;
      } else {
        odd |= !(na.x == va.x && na.y == va.y && na.z == va.z);
      }
      if (wait_b) {
        v[ib] = nb;
        done_of[ib] = at.y + 1;
      } else {
        odd |= !(nb.x == vb.x && nb.y == vb.y && nb.z == vb.z);
      }
      q[c] = f_times<double, double4>(f, y0, y1, y2);
      todo = false;
    }
  }
  odd = __syncthreads_or(odd);
  if (s_stalled && threadIdx.x == 0) atomicOr(&a.ew->err, kErrBarrierTimeout);
  return s_stalled ? kSweepStalled : odd ? kSweepOdd : kSweepDone;
}

__global__ void __launch_bounds__(kThreads, 2) k_pgs_solve(KArgs<double> a) {
  __shared__ double scratch[kMaxima * kWarps];
  __shared__ DeferBuf s_def;
  __shared__ Team tm;
  __shared__ BodyCache<kThreads> bodies;
  __shared__ PhaseTimer timer;
  __shared__ PgsSolve C;
  __shared__ int s_seen;
  const size_t S = a.S;
  if (threadIdx.x == 0) {
    s_seen = 0;
    timer.start();
  }
  __syncthreads();
  if (ld_acquire(&a.ew->err)) return;
  auto sync = [&](int phase, bool joining = false) {
    const bool ok = team_sync(a, tm, joining);
    timer.mark(a, phase);
    return ok;
  };

  while (join_team(a, tm, &s_seen)) {
    const int s = tm.s;
    const SegParams& P = a.seg[s];
    const int nc = tm.nc, c0 = tm.c0;
    double4* wv = a.wd;
    double4* qv = a.qd;
    double* Bc = a.G[4];                                      // per-contact B (plane 0)
    int2* place = reinterpret_cast<int2*>(a.G[3]);            // c among A's and B's contacts
    double4* v_kept = a.wd;   // the free bodies' v at the sweep's start (w is formed after it)
    const bool live = nc > 0;
    if (threadIdx.x == 0) {
      C.residual = 0.0;
      C.k = C.cur = C.iterations = C.sweeps = 0;
      C.done = (live && P.max_iter > 0) ? 0 : 1;
    }

    // ---- applied impulse: k = m v + h f; w = minv k
    for (int b = tm.w0 + threadIdx.x; b < tm.w1; b += kThreads) {
      const double h = P.h;
      double mi = __ldg(a.minv + b);
      double m = mi;
      if (m) m = 1.0 / m;
      double4 v = a.v4[b], f = a.f4[b];
      double4 k = make_double4(h * f.x + m * v.x, h * f.y + m * v.y, h * f.z + m * v.z, 0.0);
      a.k4[b] = k;
      a.wd[b] = make_double4(mi * k.x, mi * k.y, mi * k.z, 0.0);
    }

    if (live) {
      fill_body_cache(a, tm, bodies);
      if (!sync(kPhaseSetup, true)) return;
      // ---- r = D (Minv k) + b; gamma_0 = (1, 0, 0) -> G[0]; B; q = F gamma_0
      const int shift = a.sst[s].delta;
      for (int i = 0;; ++i) {
        const int t = team_tile(tm, i);
        if (t < 0) break;
        const double h = P.h;
        for (int m = 0; m < kItemsPerThread; ++m) {
          const int k = t * kTileItems + m * kThreads + threadIdx.x;
          if (k < nc) {
            const int c = c0 + k;
            Frame<double> fd = start_frame<double>(a, c, P.exact != 0);
            const uint32_t ia = __ldg(a.ida + c), ib = __ldg(a.idb + c);
            double4 wa = a.wd[ia], wb = a.wd[ib];
            double d0, d1, d2;
            ft_times<double, double4>(fd, wa, wb, &d0, &d1, &d2);
            double bn = __ldg(a.gap + c) / h;
            a.r[0 * S + c] = bn + d0;
            a.r[1 * S + c] = 0.0 + d1;
            a.r[2 * S + c] = 0.0 + d2;
            a.G[0][0 * S + c] = 1.0;
            a.G[0][1 * S + c] = 0.0;
            a.G[0][2 * S + c] = 0.0;
            // buildB_PGS: the nine frame entries squared and summed in row order n, u, v
            double sum = fd.n0 * fd.n0;
            sum = sum + fd.n1 * fd.n1;
            sum = sum + fd.n2 * fd.n2;
            sum = sum + fd.u0 * fd.u0;
            sum = sum + fd.u1 * fd.u1;
            sum = sum + fd.u2 * fd.u2;
            sum = sum + fd.v0 * fd.v0;
            sum = sum + fd.v1 * fd.v1;
            sum = sum + fd.v2 * fd.v2;
            const double mia = __ldg(a.minv + ia), mib = __ldg(a.minv + ib);
            Bc[c] = 3.0 / ((mia + mib) * sum);
            // a body's contacts in their order: those where it is B (ascending,
            // at the head of its incidence run), then those where it is A
            const int sa = __ldg(a.inc_start + ia), na = __ldg(a.cnt_cont + ia);
            const int nb_a = __ldg(a.inc_start + ia + 1) - sa - na;
            const int sb = __ldg(a.inc_start + ib);
            int lo = 0, hi = __ldg(a.inc_start + ib + 1) - sb - __ldg(a.cnt_cont + ib);
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              if ((__ldg(a.inc + sb + mid) & 0x7fffffffu) < (uint32_t)c) lo = mid + 1;
              else hi = mid;
            }
            place[c] = make_int2(nb_a + (c - (__ldg(a.cbase + ia) + shift)), lo);
            store_keep(qv + c, f_times<double, double4>(fd, 1.0, 0.0, 0.0));
          }
        }
      }
      const Cone<double> cone = make_cone<double>(P.mu);
      const double mu = P.mu, imu = 1.0 / P.mu;
      if (!sync(kPhaseSetup)) return;

      // ---- v = Minv (D^T gamma_0) + Minv k (PGS.cu:376-379: two products, then
      // the sum), for a scene that iterates
      if (!C.done) {
        for (int b = tm.w0 + threadIdx.x; b < tm.w1; b += kThreads) {
          const double mi = __ldg(a.minv + b);
          const double4 fc = gather_q<double, double4>(a, qv, b);
          const double4 k = a.k4[b];
          const double4 t = make_double4(mi * k.x, mi * k.y, mi * k.z, 0.0);
          a.v4[b] = make_double4(t.x + mi * fc.x, t.y + mi * fc.y, t.z + mi * fc.z, 0.0);
        }
        if (!sync(kPhaseSetup)) return;
      }

      // ---- iterations: a sweep by the first member, then the residual: one body
      // pass (w of q = F gamma) and one contact pass
      while (!C.done) {
        const double* Gc = a.G[C.cur];
        double* Gn = a.G[C.cur ^ 1];
        for (int strict = 0;; strict = 1) {
          bool odd = false;
          if (tm.rank == 0) {
            for (int b = P.b0 + threadIdx.x; b < P.b1; b += kThreads) {
              a.body_count[b] = 0;
              if (__ldg(a.minv + b) == 0.0) continue;
              if (strict) a.v4[b] = v_kept[b];
              else v_kept[b] = a.v4[b];
            }
            __syncthreads();
          }
          for (int from = 0; from < nc; from += kPgsChunk) {
            if (tm.rank == 0) {
              const int to = min(nc, from + kPgsChunk);
              const PgsSweep r = pgs_sweep(a, tm, P, Gc, Gn, cone, from, to, strict != 0);
              if (r == kSweepStalled) return;
              odd |= r == kSweepOdd;
              // a strict sweep leaves the word alone: members that are slow to
              // leave the barrier may still read it
              if (to == nc && !strict && threadIdx.x == 0) a.sst[s].ctl.mode = odd ? 1 : 0;
            }
            if (!sync(kPhaseStep)) return;
          }
          if (strict || __ldcg(&a.sst[s].ctl.mode) == 0) break;
        }
        team_body_pass<double, false>(a, tm, bodies, wv, qv);
        if (!sync(kPhaseBody)) return;
        int nslot = 0;
        for (int i = 0;; ++i) {
          const int t = team_tile(tm, i);
          if (t < 0) break;
          double mx[3] = {0.0, 0.0, 0.0};
          for (int m = 0; m < kItemsPerThread; ++m) {
            const int k = t * kTileItems + m * kThreads + threadIdx.x;
            if (k < nc) {
              const int c = c0 + k;
              double4 wa = load_vec(wv + __ldg(a.ida + c)), wb = load_vec(wv + __ldg(a.idb + c));
              Frame<double> f = load_frame<double>(a, c);
              double N0, N1, N2;
              ft_times<double, double4>(f, wa, wb, &N0, &N1, &N2);
              const double x0 = Gn[0 * S + c], x1 = Gn[1 * S + c], x2 = Gn[2 * S + c];
              const double g0 = a.r[0 * S + c] + N0, g1 = a.r[1 * S + c] + N1,
                           g2 = a.r[2 * S + c] + N2;
              mx[0] = fmax(mx[0], pgj_feasible(x0, x1, x2, mu));
              mx[1] = fmax(mx[1], pgj_feasible(g0, g1, g2, imu));
              const double d = (g0 * x0 + g1 * x1) + g2 * x2;
              mx[2] = fmax(mx[2], fabs(d));
            }
          }
          park_max<3>(s_def, nslot, tm.t0 + t, mx);
          if (++nslot == kMaxDefer) {
            fold_parked_max<3>(a, s_def, nslot);
            nslot = 0;
          }
        }
        fold_parked_max<3>(a, s_def, nslot);
        if (!sync(kPhaseProduct)) return;
        double mm[kMaxima];
        fold_tile_maxima(a, tm.t0, tm.nt, mm, scratch);
        if (threadIdx.x == 0) {
          C.cur ^= 1;
          pgs_ctl(C, mm, P);
        }
        __syncthreads();
      }

      // ---- gamma -> warm-start region (System::gamma_d); q = F gamma (FP64)
      const double* src = a.G[C.cur];
      for (int i = 0;; ++i) {
        const int t = team_tile(tm, i);
        if (t < 0) break;
        for (int m = 0; m < kItemsPerThread; ++m) {
          const int k = t * kTileItems + m * kThreads + threadIdx.x;
          if (k < nc) {
            const int c = c0 + k;
            const double x0 = src[0 * S + c], x1 = src[1 * S + c], x2 = src[2 * S + c];
            const size_t wi = (size_t)P.wbase + k;
            a.gamma[0 * a.WS + wi] = x0;
            a.gamma[1 * a.WS + wi] = x1;
            a.gamma[2 * a.WS + wi] = x2;
            Frame<double> f = load_frame<double>(a, c);
            a.qd[c] = f_times<double, double4>(f, x0, x1, x2);
          }
        }
      }
      if (!sync(kPhaseFinal)) return;
    }

    // ---- f_c = D^T gamma; v = Minv (k + f_c); f_contact = f_c / h; p += h v
    for (int b = tm.w0 + threadIdx.x; b < tm.w1 && !a.solve_only; b += kThreads) {
      const double h = P.h;
      double4 k = a.k4[b];
      double mi = __ldg(a.minv + b);
      double4 v, fcv;
      if (nc > 0) {
        double4 fc = gather_q<double, double4>(a, a.qd, b);
        v = make_double4(mi * (k.x + fc.x), mi * (k.y + fc.y), mi * (k.z + fc.z), 0.0);
        const double invh = 1.0 / h;
        fcv = make_double4(invh * fc.x, invh * fc.y, invh * fc.z, 0.0);
      } else {
        v = make_double4(mi * k.x, mi * k.y, mi * k.z, 0.0);
        fcv = make_double4(0.0, 0.0, 0.0, 0.0);
      }
      a.v4[b] = v;
      a.fc4[b] = fcv;
      double4 p = a.p4[b];
      a.p4[b] = make_double4(h * v.x + p.x, h * v.y + p.y, h * v.z + p.z, 0.0);
    }
    if (tm.rank == 0 && threadIdx.x == 0) {
      SegState& X = a.sst[s];
      SolveResult& D = X.ctl;
      D.iterations = C.iterations;
      D.sweeps = C.sweeps;
      D.residual = C.residual;
      D.backtracks = 0;
      D.objective = 0.0;
      D.refined = 0;
      D.refine_it = 0;
      if (nc > 0) X.gsize = nc;
    }
  }
  timer.store(a);
}

// A sweep over a chain of contacts (contact c between bodies c and c + 1), with
// the contacts' places among their bodies' as they are, or one further on: then
// no contact is ever next.
constexpr int kStallBodies = 64;
__global__ void __launch_bounds__(kThreads) k_selftest_sweep(KArgs<double> a, int* out) {
  __shared__ Team tm;
  if (threadIdx.x == 0) tm.c0 = 0;
  __syncthreads();
  const Cone<double> cone = make_cone<double>(0.5);
  const PgsSweep r = pgs_sweep(a, tm, a.seg[0], a.G[0], a.G[1], cone, 0, kStallBodies - 1, false);
  if (threadIdx.x == 0) *out = r == kSweepStalled;
}

}  // namespace

}  // namespace dv

extern "C" {

DV_API int dv_selftest_stalled_sweep(int32_t further, int32_t* stalled, uint32_t* error_bits) {
  using namespace dv;
  constexpr int S = kStallBodies;
  // planes of S doubles: v and q (4 each), the five iterates, F, frame words (3
  // each), gap, minv, ids, counts
  enum { kV = 0, kQ = 4, kG = 8, kF = 23, kFr = 26, kGap = 29, kMinv, kIds, kCount, kPlanes };
  std::vector<double> h((size_t)kPlanes * S, 0.0);
  uint32_t* ids = reinterpret_cast<uint32_t*>(h.data() + kIds * S);
  int2* place = reinterpret_cast<int2*>(h.data() + (kG + 9) * S);
  for (int i = 0; i < S; ++i) {
    h[kMinv * S + i] = 1.0;
    h[(kF + 2) * S + i] = h[kFr * S + i] = h[(kFr + 2) * S + i] = 1.0;
    ids[i] = (uint32_t)i;
    ids[S + i] = (uint32_t)std::min(i + 1, S - 1);
    place[i] = make_int2((i > 0 ? 1 : 0) + (further ? 1 : 0), further ? 1 : 0);
  }
  SegParams P{};
  P.h = 1.0;
  P.mu = 0.5;
  EngineWords words{};
  struct Block {
    double* w;
    SegParams* seg;
    EngineWords* ew;
    int* out;
  } b{nullptr, nullptr, nullptr, nullptr};
  int r = -1;
  auto run = [&]() -> int {
    DV_CUDA_TRY(cudaMalloc(&b.w, h.size() * sizeof(double)));
    DV_CUDA_TRY(cudaMalloc(&b.seg, sizeof(P)));
    DV_CUDA_TRY(cudaMalloc(&b.ew, sizeof(words)));
    DV_CUDA_TRY(cudaMalloc(&b.out, sizeof(int)));
    DV_CUDA_TRY(cudaMemcpy(b.w, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    DV_CUDA_TRY(cudaMemcpy(b.seg, &P, sizeof(P), cudaMemcpyHostToDevice));
    DV_CUDA_TRY(cudaMemcpy(b.ew, &words, sizeof(words), cudaMemcpyHostToDevice));
    KArgs<double> a;
    memset((void*)&a, 0, sizeof(a));
    a.S = S;
    a.v4 = reinterpret_cast<double4*>(b.w + kV * S);
    a.qd = reinterpret_cast<double4*>(b.w + kQ * S);
    for (int k = 0; k < 5; ++k) a.G[k] = b.w + (kG + 3 * k) * S;
    a.F = b.w + kF * S;
    a.fr = b.w + kFr * S;
    a.gap = b.w + kGap * S;
    a.minv = b.w + kMinv * S;
    a.ida = reinterpret_cast<const uint32_t*>(b.w + kIds * S);
    a.idb = a.ida + S;
    a.body_count = reinterpret_cast<int*>(b.w + kCount * S);
    a.seg = b.seg;
    a.ew = b.ew;
    k_selftest_sweep<<<1, kThreads>>>(a, b.out);
    DV_CUDA_TRY(cudaGetLastError());
    DV_CUDA_TRY(cudaDeviceSynchronize());
    DV_CUDA_TRY(cudaMemcpy(&r, b.out, sizeof(int), cudaMemcpyDeviceToHost));
    DV_CUDA_TRY(cudaMemcpy(&words, b.ew, sizeof(words), cudaMemcpyDeviceToHost));
    return DV_OK;
  };
  const int rc = run();
  cudaFree(b.w);
  cudaFree(b.seg);
  cudaFree(b.ew);
  cudaFree(b.out);
  if (rc != DV_OK) return rc;
  if (stalled) *stalled = r;
  if (error_bits) *error_bits = words.err;
  return DV_OK;
}

}  // extern "C"

namespace dv {

void launch_pgs_solve(SceneDev& sd, const SolveConfig& cfg, cudaStream_t st, int64_t* launches,
                      bool solve_only) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pgs_solve, kThreads, 0);
  const int grid = std::min(cfg.grid, sms * std::max(per_sm, 1));
  KArgs<double> a = make_kargs<double>(sd, cfg);
  a.solve_only = solve_only ? 1 : 0;
  plan_teams(sd, grid, false, st, launches);
  void* params[] = {&a};
  cudaLaunchCooperativeKernel((const void*)k_pgs_solve, grid, kThreads, params, 0, st);
  ++*launches;
}

}  // namespace dv
