// dv_pgj.cu -- the time step with the PGJ solver (System(5), PGJ.cu:152-224)
// for every segment of an engine, as one persistent cooperative kernel per
// step: applied impulse, Schur vector, PGJ iterations, update.
//
// PGJ: gamma starts at (1, 0, 0) per contact (PGJ.cu:170, no warm start),
// B_c = 3 / ((minv_A + minv_B) |F_c|^2) (buildB, :73-89), and each iteration
//   gamma_hat = P(gamma - omega B (N gamma + r))
//   gamma     = lambda gamma_hat + (1 - lambda) gamma       (omega 0.3, lambda 2/3)
// stops when max(feasibleX, feasibleY, max_c |(N gamma + r)_c . gamma_c|) of
// the new gamma is below the tolerance (:188-214).  N of the new iterate
// serves its residual and the next iteration, so an iteration is one body
// pass and one contact pass: the contact pass forms N gamma_k, the residual
// terms of gamma_k and the step to gamma_{k+1} (its feasibleX and q = F
// gamma_{k+1}); the scene's controller then decides on gamma_k.  Only maxima
// are reduced, so the result does not depend on any summation order.
//
// A team of CTAs solves a scene (dv_team.cuh); every member folds the maxima
// and runs the controller on its own copy of the scalars.
#include <algorithm>

#include "dv_team.cuh"

namespace dv {

namespace {

constexpr double kPgjOmega = 0.3;
constexpr double kPgjLambda = 2.0 / 3.0;

// Scalars of a solve, one copy per member: gamma_k is in G[cur], the next
// iterate goes to G[cur ^ 1].
struct PgjSolve {
  double fx, residual;  // feasibleX of the iterate computed last
  double m[3];
  int k, cur, iterations, sweeps, done;
};

// After a contact pass (thread 0): m holds the maxima of feasibleX of the new
// iterate, and of feasibleY and res3 of the current one.
__device__ inline void pgj_ctl(PgjSolve& C, const double* m, const SegParams& P) {
  const int k = C.k;
  if (k >= 1) {
    const double residual = fmax(fmax(C.fx, m[1]), m[2]);
    C.residual = residual;
    if (residual < P.tol) {
      C.done = 1;
      C.iterations = k - 1;
    } else if (k >= P.max_iter) {
      C.done = 1;
      C.iterations = P.max_iter;
    }
  }
  if (!C.done) {
    C.fx = m[0];
    C.cur ^= 1;
    C.k = k + 1;
    C.sweeps += 1;
  }
}

template <class T>
__global__ void __launch_bounds__(kThreads, 2) k_pgj_solve(KArgs<T> a) {
  using V = typename Vec4<T>::type;
  __shared__ double scratch[kMaxima * kWarps];
  __shared__ DeferBuf s_def;
  __shared__ Team tm;
  __shared__ BodyCache<kThreads> bodies;
  __shared__ PhaseTimer timer;
  __shared__ PgjSolve C;
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
    // in FP32 the iterations' w and q lie over the scene's own FP64 ones
    V* wv = reinterpret_cast<V*>(a.wd + P.b0) - P.b0;
    V* qv = reinterpret_cast<V*>(a.qd + c0) - c0;
    T* Bc = a.G[4];  // per-contact B (plane 0)
    const bool live = nc > 0;
    if (threadIdx.x == 0) {
      C.fx = C.residual = 0.0;
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
      for (int i = 0;; ++i) {
        const int t = team_tile(tm, i);
        if (t < 0) break;
        const double h = P.h;
        for (int m = 0; m < kItemsPerThread; ++m) {
          const int k = t * kTileItems + m * kThreads + threadIdx.x;
          if (k < nc) {
            const int c = c0 + k;
            Frame<double> fd = load_frame_fp64(a, c, P.exact != 0);
            const uint32_t ia = __ldg(a.ida + c), ib = __ldg(a.idb + c);
            double4 wa = a.wd[ia], wb = a.wd[ib];
            double d0, d1, d2;
            ft_times<double, double4>(fd, wa, wb, &d0, &d1, &d2);
            double bn = __ldg(a.gap + c) / h;
            a.r[0 * S + c] = (T)(bn + d0);
            a.r[1 * S + c] = (T)(0.0 + d1);
            a.r[2 * S + c] = (T)(0.0 + d2);
            a.G[0][0 * S + c] = T(1);
            a.G[0][1 * S + c] = T(0);
            a.G[0][2 * S + c] = T(0);
            // buildB: the nine frame entries squared and summed in row order n, u, v
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
            Bc[c] = (T)(3.0 / ((mia + mib) * sum));
            Frame<T> f = start_frame<T>(a, c, P.exact != 0);
            store_keep(qv + c, f_times<T, V>(f, T(1), T(0), T(0)));
          }
        }
      }
      const Cone<T> cone = make_cone<T>((T)P.mu);
      const double mud = P.mu, imu = 1.0 / mud;
      if (!sync(kPhaseSetup)) return;

      // ---- iterations: one body pass (w of q = F gamma_k) and one contact pass
      // (N gamma_k, residual terms of gamma_k, step to gamma_{k+1}) each
      while (!C.done) {
        team_body_pass<T, false>(a, tm, bodies, wv, qv);
        if (!sync(kPhaseBody)) return;
        int nslot = 0;
        const int kk = C.k;
        const T* Gc = a.G[C.cur];
        T* Gn = a.G[C.cur ^ 1];
        for (int i = 0;; ++i) {
          const int t = team_tile(tm, i);
          if (t < 0) break;
          double mx[3] = {0.0, 0.0, 0.0};
          for (int m = 0; m < kItemsPerThread; ++m) {
            const int k = t * kTileItems + m * kThreads + threadIdx.x;
            if (k < nc) {
              const int c = c0 + k;
              V wa = load_vec(wv + __ldg(a.ida + c)), wb = load_vec(wv + __ldg(a.idb + c));
              Frame<T> f = load_frame<T>(a, c);
              T N0, N1, N2;
              ft_times<T, V>(f, wa, wb, &N0, &N1, &N2);
              const T x0 = Gc[0 * S + c], x1 = Gc[1 * S + c], x2 = Gc[2 * S + c];
              const T r0 = a.r[0 * S + c], r1 = a.r[1 * S + c], r2 = a.r[2 * S + c];
              const T g0 = N0 + r0, g1 = N1 + r1, g2 = N2 + r2;
              if (kk >= 1) {
                const double d = ((double)g0 * (double)x0 + (double)g1 * (double)x1) +
                                 (double)g2 * (double)x2;
                mx[2] = fmax(mx[2], fabs(d));
                mx[1] = fmax(mx[1], pgj_feasible(g0, g1, g2, imu));
              }
              // gamma_hat = gamma + (-omega) (B (N gamma + r)), projected
              const T b = Bc[c];
              const T om = (T)(-kPgjOmega);
              T h0 = x0 + om * (b * g0), h1 = x1 + om * (b * g1), h2 = x2 + om * (b * g2);
              project_cone<T>(h0, h1, h2, cone);
              const T la = (T)kPgjLambda, lb = (T)(1.0 - kPgjLambda);
              const T y0 = la * h0 + lb * x0, y1 = la * h1 + lb * x1, y2 = la * h2 + lb * x2;
              Gn[0 * S + c] = y0; Gn[1 * S + c] = y1; Gn[2 * S + c] = y2;
              mx[0] = fmax(mx[0], pgj_feasible(y0, y1, y2, mud));
              store_keep(qv + c, f_times<T, V>(f, y0, y1, y2));
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
        if (threadIdx.x == 0) pgj_ctl(C, mm, P);
        __syncthreads();
      }

      // ---- gamma -> warm-start region; q = F gamma (FP64)
      const T* src = a.G[C.cur];
      for (int i = 0;; ++i) {
        const int t = team_tile(tm, i);
        if (t < 0) break;
        for (int m = 0; m < kItemsPerThread; ++m) {
          const int k = t * kTileItems + m * kThreads + threadIdx.x;
          if (k < nc) {
            const int c = c0 + k;
            const double x0 = (double)src[0 * S + c], x1 = (double)src[1 * S + c],
                         x2 = (double)src[2 * S + c];
            const size_t wi = (size_t)P.wbase + k;
            a.gamma[0 * a.WS + wi] = x0;
            a.gamma[1 * a.WS + wi] = x1;
            a.gamma[2 * a.WS + wi] = x2;
            Frame<double> f = load_frame_fp64(a, c, P.exact != 0);
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

template <class T>
void launch_typed(SceneDev& sd, const SolveConfig& cfg, cudaStream_t st, int64_t* launches,
                  bool solve_only) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pgj_solve<T>, kThreads, 0);
  const int grid = std::min(cfg.grid, sms * std::max(per_sm, 1));
  KArgs<T> a = make_kargs<T>(sd, cfg);
  a.solve_only = solve_only ? 1 : 0;
  plan_teams(sd, grid, false, st, launches);
  void* params[] = {&a};
  cudaLaunchCooperativeKernel((const void*)k_pgj_solve<T>, grid, kThreads, params, 0, st);
  ++*launches;
}

}  // namespace

void launch_pgj_solve(SceneDev& sd, const SolveConfig& cfg, cudaStream_t st, int64_t* launches,
                      bool solve_only) {
  if (sd.precision == DV_PREC_MIXED) launch_typed<float>(sd, cfg, st, launches, solve_only);
  else launch_typed<double>(sd, cfg, st, launches, solve_only);
}

}  // namespace dv
