// dv_apgd.cu -- the time step after collision detection, for every segment
// (scene) of an engine, as ONE persistent cooperative kernel per step:
//
//   applied impulse k = M v + h f             System.cu:1411-1417, 1502-1514
//   Schur vector r = D Minv k + b             System.cu:1516-1524, 1561-1580
//   APGD solve (all iterations)               APGD.cu:164-361
//   v = Minv (k + D^T gamma), p += h v        System.cu:570-583
//
// The reference runs each BLAS-1 call, SpMV and projection as its own launch
// and brings every dot/nrm2/nrmmax back to the host (APGD.cu:227-350).  Here a
// team of CTAs (dv_team.cuh) takes a scene and runs all of it.  The scalar
// control (step size, Lipschitz backtracking, restart, best iterate,
// convergence) runs on the device: after a pass's barrier every member folds
// the scene's per-tile partial sums in a fixed order and executes the control
// logic on its own copy of the scalars, in shared memory.
//
// Matrix-free N x = D Minv D^T x (D's block of contact c is [+F_c^T | -F_c^T],
// F_c = [n u v]):
//   contact pass: q_c = F_c x_c (written by the pass that produced x_c)
//   body pass:    w_b = minv_b * (sum of -q_c over contacts where b is B,
//                 then +q_c where b is A, ascending contact order; no atomics)
//   contact pass: (N x)_c = F_c^T (w_A - w_B), fused with the APGD vector
//                 updates, the cone projection and the reductions.
//
// One Schur product per iteration.  The reference evaluates N y_k with its own
// product (APGD.cu:229, 239) and N gamma_new twice more (:237, :276).  Since
// y_k = (1 + b) gamma_k - b gamma_{k-1} (APGD.cu:273) or gamma_k after a
// restart (:315), N y_k is formed here from the stored products of the two
// previous iterates; N gamma_new is computed once and serves the objective and
// the residual.  Iterates and their products rotate through five buffers, so
// y, g and gamma_hat are never copied.  The CPU oracle evaluates the same
// sequence (apgd_solve_fused), and bit-for-bit the same arithmetic.
//
// Precision: the kernel is a template on the iterate type T.  T = double is
// the FP64 path (bit-exact against the oracle).  T = float is the mixed path:
// frames, Jacobian and N gamma products, iterates and the cone projection in
// FP32; the Schur vector r (computed in FP64, stored in FP32), the objective
// and Lipschitz-test sums, the residual, the final D^T gamma and the
// integration in FP64.
//
// What the passes read per contact lies in blocks of 32 contacts, one warp's
// share: the constants of a solve (normal, frame words, r, body ids) in one
// block, each iterate with its product in another.  A warp brings its next 32
// contacts with three bulk copies of 0.4 to 2.5 KB.  As separate planes they
// were twenty copies of 256 bytes, and the copy engine's rate per copy (about
// 30 cycles), not the bytes, set the pass's time: 52 us in FP64 and 51 us in
// FP32 on 741,000 contacts.
//
// Work is split in tiles of 512 contacts (2 per thread).  Every wait has a
// time limit.
#include <algorithm>
#include <atomic>

#include "dv_team.cuh"

namespace dv {

namespace {

// A solve's scalar state (APGD.cu:208-223, 266-332), one copy per member in
// shared memory, and what the passes take from it.  Iterates live in five
// rotating buffers: cur = gamma_k, prev = gamma_{k-1}, nw = target of
// gamma_new, best = gamma_hat (-1 before the first accepted iterate), nw2 the
// next iterate computed ahead.
struct Solve {
  double L, theta_new;
  double obj1, obj2, obj2_base, residual, objective, objN;
  double gdiff, ginv, gneg, L0;        // gd, 1 / gd, -(1 / gd)
  double step_ya, step_ym, step_nt;    // step pass: 1 + yb, -yb, -t
  double prod_ya, prod_ym, prod_nt;    // look-ahead: 1 + b, -b, -(1 / (0.9 L))
  // the scalars after the product pass, formed ahead: after an accepted iterate
  // (a_) and after a failed test (f_)
  double a_theta, a_theta_new, a_beta, a_L, a_t, a_nt, f_L, f_t, f_nt;
  Cone<double> cone;
  Cone<float> conef;
  double sums[8];
  int a_nw2_kept, a_nw2_best;  // the next look-ahead's buffer: gamma_hat kept, or gamma_new
  int k, restart, cur, prev, nw, nw2, best, yr, first, step;
  int backtracks, sweeps, iterations, rsel, since_best, done;
  unsigned err;
};

template <class T> __device__ inline const Cone<T>& cone_of(const Solve& c);
template <> __device__ inline const Cone<double>& cone_of<double>(const Solve& c) { return c.cone; }
template <> __device__ inline const Cone<float>& cone_of<float>(const Solve& c) { return c.conef; }

// Mixed precision with refinement: the FP32 phase of a solve ends when its
// best residual has not improved for this many accepted iterations.
constexpr int kStallIterations = 50;

// ---- controllers (thread 0 of every member, after fold_team) ----

__device__ __noinline__ void ctl_lipschitz(Solve& C, const SegParams& P, int nc, int cap,
                                           bool mixed) {
  const double L = sqrt(C.sums[0]) / C.L0;
  C.L = L;
  const double th = 1.0;
  const double tn = (-(th * th) + th * sqrt(th * th + 4.0)) / 2.0;
  C.theta_new = tn;
  const double beta = th * (1.0 - th) / (th * th + tn);
  C.step_ya = 1.0;  // y_0 = gamma_0
  C.step_ym = -0.0;
  C.step_nt = -(1.0 / L);
  C.prod_ya = 1.0 + beta;
  C.prod_ym = -beta;
  C.prod_nt = -(1.0 / (0.9 * L));
  C.residual = 10e30;
  C.objective = 0.0;
  // APGD.cu:92: 1 / (contacts + bilateral rows)^2
  const double ncd = (double)(nc + P.nbil);
  const double gd = 1.0 / (ncd * ncd);
  C.gdiff = gd;
  C.ginv = 1.0 / gd;
  C.gneg = -1.0 / gd;
  C.k = 0;
  C.step = 1;
  C.iterations = 0;
  C.sweeps = 0;
  C.restart = 0;
  C.cur = 0;
  C.prev = -1;
  C.nw = 1;
  C.best = -1;
  C.nw2 = free_slot(1, 0, -1, -1);
  C.yr = 1;
  C.first = 1;
  C.backtracks = 0;
  C.obj1 = 0.0;
  C.obj2 = 0.0;
  C.obj2_base = 0.0;
  C.rsel = 0;
  C.objN = 0.0;
  C.since_best = 0;
  C.done = cap <= 0 ? 1 : 0;
  C.cone = make_cone<double>(P.mu);
  if (mixed) C.conef = make_cone<float>((float)P.mu);
}

__device__ __noinline__ void ctl_step(Solve& C) {
  double ob = C.obj2_base;
  if (C.first) {
    ob = 0.5 * C.sums[3] + C.sums[4];
    C.obj2_base = ob;
  }
  const double nr = sqrt(C.sums[1]);
  C.obj2 = ob + (C.sums[0] + 0.5 * C.L * (nr * nr));
  C.restart = (C.sums[2] > 0) ? 1 : 0;
  C.first = 0;
  C.step = 0;
}

// Formed by one thread while the barrier before the product pass waits: every
// value that does not depend on the pass's sums (a square root and four
// divisions in a row otherwise stand between the sums and the next pass).
__device__ __noinline__ void ctl_ahead(Solve& C) {
  const double th = C.restart ? 1.0 : C.theta_new;
  const double tn = (-(th * th) + th * sqrt(th * th + 4.0)) / 2.0;
  C.a_theta = th;
  C.a_theta_new = tn;
  C.a_beta = th * (1.0 - th) / (th * th + tn);
  const double aL = 0.9 * C.L, fL = 2.0 * C.L;
  C.a_L = aL;
  C.a_t = 1.0 / aL;
  C.a_nt = -(1.0 / (0.9 * aL));
  C.f_L = fL;
  C.f_t = 1.0 / fL;
  C.f_nt = -(1.0 / (0.9 * fL));
  C.a_nw2_kept = free_slot(C.nw2, C.nw, C.cur, C.best);
  C.a_nw2_best = free_slot(C.nw2, C.nw, C.cur, C.nw);
}

__device__ __noinline__ void ctl_product(Solve& C, const SegParams& P, int cap, bool mixed, bool ar) {
  const double obj1 = 0.5 * C.sums[0] + C.sums[1];
  const double res = C.sums[7];
  C.obj1 = obj1;
  int k = C.k;
  bool finished = false;
  // APGD.cu:240: obj1 >= obj2 means the step was too long.  With FP32
  // iterates both objectives carry rounding of order 1e-7 |f|; a difference
  // within that noise is not a failed test (else L doubles on noise alone).
  const double obj2 = C.obj2;
  const bool fail = mixed ? (obj1 - obj2 >= 1e-6 * (fabs(obj1) + fabs(obj2))) : (obj1 >= obj2);
  if (fail) {
    // (10)-(14): double L and retry the projection
    if (C.backtracks >= P.max_bt) {
      C.err |= kErrBacktrackCap;
      finished = true;
    } else {
      C.backtracks += 1;
      C.L = C.f_L;
      C.step_nt = -C.f_t;
      C.prod_nt = C.f_nt;
      C.step = 1;
    }
  } else {
    C.sweeps += 1;
    C.since_best += 1;
    bool better = false;
    if (res < C.residual) {
      C.residual = res;
      C.objective = obj1;
      if (ar) C.objN = 0.5 * C.sums[0];
      C.best = C.nw;
      C.since_best = 0;
      better = true;
    }
    if (C.residual < P.tol) {
      finished = true;
    } else if (mixed && P.refine > 0 && C.since_best >= kStallIterations) {
      // FP32 iterates no longer improve: the FP64 refinement continues
      // from gamma_hat
      finished = true;
    } else {
      // APGD.cu:335-345 after this iteration: r moves to the plane the
      // product pass wrote for the look-ahead
      if (ar) C.rsel ^= 1;
      // y of the next step pass is this pass's look-ahead y
      C.step_ya = C.prod_ya;
      C.step_ym = C.prod_ym;
      C.yr = C.restart;
      C.L = C.a_L;
      C.step_nt = -C.a_t;
      C.prod_nt = C.a_nt;
      C.prev = C.cur;
      C.cur = C.nw;
      C.nw = C.nw2;
      C.nw2 = better ? C.a_nw2_best : C.a_nw2_kept;
      k += 1;
      C.k = k;
      if (k >= cap) {
        finished = true;
      } else {
        C.theta_new = C.a_theta_new;
        C.prod_ya = 1.0 + C.a_beta;
        C.prod_ym = -C.a_beta;
        // the look-ahead step is now iteration k's step
        const double ob = 0.5 * C.sums[5] + C.sums[6];
        C.obj2_base = ob;
        const double nr = sqrt(C.sums[3]);
        C.obj2 = ob + (C.sums[2] + 0.5 * C.L * (nr * nr));
        C.restart = (C.sums[4] > 0) ? 1 : 0;
      }
    }
  }
  if (finished) {
    C.iterations = k;
    C.done = 1;
  }
}

// ---- blocks of 32 contacts ----
// Constant block: 9 planes of 32 (normal, frame words, r), then the 32 ids A
// and the 32 ids B.  Iterate block: 3 planes of the iterate, 3 of its product.
template <class T> struct Block {
  static constexpr int kIds = 9 * 32;                               // in T
  static constexpr int kConst = kIds + 256 / (int)sizeof(T);
  static constexpr unsigned kConstBytes = kConst * sizeof(T);
  static constexpr unsigned kHalfBytes = 3 * 32 * sizeof(T);        // an iterate or a product
  // a warp's stage: constants, gamma_new, gamma_k with its product
  static constexpr unsigned kStageBytes = kConstBytes + 3 * kHalfBytes;
};

template <class T>
__device__ inline T* const_at(const KArgs<T>& a, int c) {
  return a.blk + (size_t)(c >> 5) * Block<T>::kConst + (c & 31);
}
constexpr int kIterBlock = 6 * 32;
template <class T>
__device__ inline T* iter_at(T* x, int c) {
  return x + (size_t)(c >> 5) * kIterBlock + (c & 31);
}
template <class T>
__device__ inline Frame<T> block_frame(const T* p) {
  return make_frame<T>(p[0], p[32], p[64], FrameWords<T>{p[96], p[128], p[160]});
}
template <class T>
__device__ inline uint2 block_ids(const KArgs<T>& a, int c) {
  const uint32_t* p =
      reinterpret_cast<const uint32_t*>(a.blk + (size_t)(c >> 5) * Block<T>::kConst + Block<T>::kIds) +
      (c & 31);
  return make_uint2(p[0], p[32]);
}

// The arrays of one bilateral tile in the product pass.
template <class T>
struct BilRows {
  const int2* off;
  const T* w;          // body vector (4 per body)
  const T* Gc;         // gamma_k
  const T* Gn;         // gamma_new
  T* G2;               // the look-ahead iterate
  const T* NGc;
  T* NGn;
  const T* r;
  T* q;
};

// Product pass on rows [r0, r0 + min(n, 512)): N gamma_new, the objective and
// residual items, the look-ahead step, without the cone projection; the sums
// into acc.  Called after the contact tiles (where
// it adds no registers to the contact loops).  Returns whether a residual
// item of this thread was NaN.
template <class T, int kGroups>
__device__ inline bool bil_product_tile(BilRows<T> R, const Solve& C, int r0, int n,
                                        bool has_contacts, double (&acc)[8]) {
  const T ya = (T)C.prod_ya, ym = (T)C.prod_ym, nt2 = (T)C.prod_nt;
  bool bad = false;
  for (int m = kGroups == 2 ? (int)(threadIdx.x >> 8) : 0; m < kItemsPerThread; m += kGroups) {
    const int k = m * kThreads + (threadIdx.x & (kThreads - 1));
    if (k < n) {
      const int r = r0 + k;
      const T N0 = bil_dw<T>(__ldg(R.off + r), R.w);
      R.NGn[r] = N0;
      const T x0 = R.Gn[r], rr = R.r[r];
      acc[0] = acc[0] + (double)x0 * (double)N0;
      acc[1] = acc[1] + (double)x0 * (double)rr;
      // APGD.cu:90-102 on a row: no projection; without contacts the
      // residual is |N x + r| (the reference skips both axpby)
      double T0 = (double)rr + (double)N0;
      if (has_contacts) {
        const double X0 = x0;
        T0 = X0 + (-C.gdiff) * T0;
        T0 = C.ginv * X0 + C.gneg * T0;
      }
      const double m0 = fabs(T0);
      bad |= (m0 != m0);
      acc[7] = fmax(acc[7], m0);
      T y0, M0;
      if (C.restart) {
        y0 = x0;
        M0 = N0;
      } else {
        y0 = ya * x0 + ym * R.Gc[r];
        M0 = ya * N0 + ym * R.NGc[r];
      }
      const T g0 = M0 + rr;
      const T z0 = y0 + nt2 * g0;
      R.G2[r] = z0;
      R.q[r] = z0;
      const T t0 = z0 + T(-1) * y0, s0 = z0 + T(-1) * x0;
      acc[2] = acc[2] + (double)g0 * (double)t0;
      acc[3] = acc[3] + (double)t0 * (double)t0;
      acc[4] = acc[4] + (double)g0 * (double)s0;
      acc[5] = acc[5] + (double)y0 * (double)M0;
      acc[6] = acc[6] + (double)y0 * (double)rr;
    }
  }
  return bad;
}

// The end of a tile: its partials into slot `slot`.
template <int kGroups, int NQ, bool kMax>
__device__ __forceinline__ void park_group(ParkBuf& park, PairBuf& pair, int& flip, int slot, int tile,
                                           double (&acc)[8]) {
  if constexpr (kGroups == 2) park_pair8<NQ, kMax>(park, pair, flip, slot, tile, acc);
  else park8<kMax>(park, slot, tile, acc);
}

// kGroups 2: CTAs of 512 threads, one per SM, whose second group of 256 takes
// the second sub-tile of every tile: a scene with a tile per member waits for
// the contact arithmetic once a pass instead of twice.  kGroups 1: CTAs of 256
// threads, kMinB per SM, which hide each other's waits where there is work for
// all of them.
// kAR: APGD's anti-relaxation (APGD.cu:335-345), FP64 one-scene engines.
template <class T, int kGroups, int kMinB, bool kAR>
__global__ void __launch_bounds__(kThreads* kGroups, kMinB) k_step_solve(KArgs<T> a) {
  using V = typename Vec4<T>::type;
  using B = Block<T>;
  constexpr bool kMixed = sizeof(T) != sizeof(double);
  constexpr int kT = kThreads * kGroups;
  __shared__ double scratch[64];
  __shared__ Solve C;
  __shared__ Team tm;
  __shared__ BodyCache<kT> bodies;
  __shared__ ParkBuf park;
  __shared__ PhaseTimer timer;
  __shared__ int s_seen, s_copy_fail;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  const size_t S = a.S;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // this thread's sub-tile of a tile (kGroups 2) and its place in it
  const int group = kGroups == 2 ? (int)(threadIdx.x >> 8) : 0;
  const int tid = threadIdx.x & (kThreads - 1), gwarp = tid >> 5;
  Staging stg;
  stg.base = dyn_smem;
  stg.stage_bytes = B::kStageBytes;
  stg.bar = reinterpret_cast<uint64_t*>(dyn_smem + (size_t)kWarps * kGroups * 2 * B::kStageBytes);
  PairBuf& pair = *reinterpret_cast<PairBuf*>(stg.bar + 2 * kMaxWarps + kMaxWarps / 8);
  int flip = 0;
  stg.phase = 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * kWarps * kGroups; ++i) mbar_init(stg.bar + i, 1);
    for (int w = 0; w < kMaxWarps; ++w) reinterpret_cast<unsigned char*>(stg.bar + 2 * kMaxWarps)[w] = 0;
    fence_mbar_init();
    s_seen = 0;
    s_copy_fail = 0;
    timer.start();
  }
  __syncthreads();
  if (ld_acquire(&a.ew->err)) return;  // an error of collision detection: nothing to do

  // a warp's sub-tile j: of the member's tile tile_of(j) its part sub_of(j)
  auto tile_of = [](int j) { return kGroups == 2 ? j : j >> 1; };
  auto sub_of = [&](int j) { return kGroups == 2 ? group : j & 1; };
  // a phase ends at a barrier
  auto sync = [&](int phase, bool joining = false) {
    const bool ok = team_sync(a, tm, joining);
    timer.mark(a, phase);
    return ok;
  };

  while (join_team(a, tm, &s_seen)) {
    const int s = tm.s;
    const SegParams& P = a.seg[s];
    const int nc = tm.nc, c0 = tm.c0;
    // the iterations' w and q: in FP32 they lie over the scene's own FP64 ones
    // (setup and update), not over another scene's
    V* wv = reinterpret_cast<V*>(a.wd + P.b0) - P.b0;
    V* qv = reinterpret_cast<V*>(a.qd + c0) - c0;
    double* part = a.part + tm.t0;
    int parity = 0;  // the partials' planes of this pass (a member may be a pass ahead)
    auto planes = [&]() { return part + (size_t)parity * 8 * a.tcap; };
    const bool live = nc > 0 || P.nbil > 0;  // System.cu:560: a solve runs with contacts or rows
    const int cap = a.refine ? P.refine : P.max_iter;
    int it_lo = 0, bt_lo = 0, sw_lo = 0;
    if (a.refine && threadIdx.x == 0) {
      const SolveResult& D = a.sst[s].ctl;
      it_lo = D.iterations;
      bt_lo = D.backtracks;
      sw_lo = D.sweeps;
    }
    if (threadIdx.x == 0) {
      C.err = 0u;
      C.done = 1;
      C.iterations = C.sweeps = C.backtracks = 0;
      C.residual = C.objective = 0.0;
      C.best = -1;
      C.rsel = 0;
    }

    // ---- applied impulse: k = m v + h f (m = 1/minv, 0 for fixed); w = minv k
    for (int b = tm.w0 + threadIdx.x; b < tm.w1; b += kT) {
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

      // ---- r = D (Minv k) + b; gamma_0 -> G[0]; e = gamma_0 - gamma_hat_0 (= gamma_0 - 1)
      {
        int nslot = 0;
        for (int i = 0;; ++i) {
          const int t = team_tile(tm, i);
          if (t < 0) break;
          const int k0 = t * kTileItems, gsize = tm.gsize;
          const double h = P.h;
          double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
          const int kb = a.nbil ? bil_tile_k0(t, 0, nc) : -1;
          if (kb >= 0) {
            // bilateral rows: b = violation / h (System.cu:1526-1544) at the
            // step's start time, r = b + (D Minv k)_row, gamma_0, e = gamma_0 - 1
            const double* pd = reinterpret_cast<const double*>(a.p4);
            const double* wdv = reinterpret_cast<const double*>(a.wd);
            const double tmv = a.seg_time[s];
            for (int m = group; m < kItemsPerThread; m += kGroups) {
              const int k = kb + m * kThreads + tid;
              if (k < P.nbil) {
                const int i2 = P.bil0 + k;
                const int2 o = __ldg(a.bil_off + i2);
                const double4 inf = a.bil_info[i2];  // velocity, start time, p0
                double velocity = inf.x;
                if (tmv < inf.y) velocity = 0;
                const double pa = pd[o.x];
                const double viol = o.y >= 0 ? pa - pd[o.y] - velocity * (tmv - inf.y)
                                             : pa - inf.z - velocity * (tmv - inf.y);
                const double bb = viol / h;
                a.bil_b[i2] = bb;
                a.br[i2] = (T)(bb + bil_dw<double>(o, wdv));
                // warm start: the row's last impulse.  Without it the reference's
                // initialiser writes (1, 0, 0) over flat entries [0, 3 nc) with
                // the rows first (APGD.cu:114-120, 200): row k takes 1 if k is a
                // multiple of 3, 0 otherwise, and keeps its last impulse from 3 nc on.
                double g = a.bil_gam[i2];
                if (!P.warm && k < 3 * nc) g = (k % 3 == 0) ? 1.0 : 0.0;
                const T x0 = (T)g;
                a.bG[0][i2] = x0;
                const T e0 = x0 + T(-1);
                acc[0] = acc[0] + (double)e0 * (double)e0;
                a.bq[i2] = e0;
              }
            }
          }
          for (int m = group; m < kItemsPerThread && kb < 0; m += kGroups) {
            int k = k0 + m * kThreads + tid;
            if (k < nc) {
              const int c = c0 + k;
              const uint32_t ia = __ldg(a.ida + c), ib = __ldg(a.idb + c);
              double4 wa = a.wd[ia], wb = a.wd[ib];
              const double n0 = __ldg(a.F + c), n1 = __ldg(a.F + S + c), n2 = __ldg(a.F + 2 * S + c);
              const FrameWords<double> fw = frame_words(n0, n1, n2, P.exact != 0);
              const Frame<double> fd = make_frame<double>(n0, n1, n2, fw);
              double d0, d1, d2;
              ft_times<double, double4>(fd, wa, wb, &d0, &d1, &d2);
              double bn = __ldg(a.gap + c) / h;
              const T r0 = (T)(bn + d0), r1 = (T)(0.0 + d1), r2 = (T)(0.0 + d2);
              a.r[0 * S + c] = r0;
              a.r[1 * S + c] = r1;
              a.r[2 * S + c] = r2;
              if (kAR) {
                // r_n and the anti-relaxation vector (0 at the start, APGD.cu:196)
                a.ar_r0[c] = bn + d0;
                a.ar_v[c] = 0.0;
              }
              double g0, g1, g2;
              // refinement: positional, from the FP32 phase's gamma_hat of this step
              const int warm = a.refine ? 1 : P.warm;
              if (warm == 2) {
                // matched: the impulse the same (A, B) pair had at the last solve;
                // A's earlier contacts are sorted by B, so a binary search finds it
                const uint32_t bl = ib - (uint32_t)P.b0;
                int lo = a.ws[ia], hi = lo + a.wc[ia];
                if (hi > gsize) hi = gsize;
                while (lo < hi) {
                  const int mid = (lo + hi) >> 1;
                  if (a.wid[(size_t)P.wbase + mid] < bl) lo = mid + 1;
                  else hi = mid;
                }
                g0 = 0.0; g1 = 0.0; g2 = 0.0;
                if (lo < gsize && lo < a.ws[ia] + a.wc[ia] && a.wid[(size_t)P.wbase + lo] == bl) {
                  const size_t wj = (size_t)P.wbase + lo;
                  g0 = a.gamma[0 * a.WS + wj];
                  g1 = a.gamma[1 * a.WS + wj];
                  g2 = a.gamma[2 * a.WS + wj];
                }
              } else if (warm) {
                const size_t wi = (size_t)P.wbase + k;
                g0 = k < gsize ? a.gamma[0 * a.WS + wi] : 0.0;
                g1 = k < gsize ? a.gamma[1 * a.WS + wi] : 0.0;
                g2 = k < gsize ? a.gamma[2 * a.WS + wi] : 0.0;
              } else if (P.nbil == 0) {
                g0 = 1.0; g1 = 0.0; g2 = 0.0;
              } else {
                // the initialiser's (1, 0, 0) pattern over flat entries [0, 3 nc)
                // of a vector whose first nbil entries are the bilateral rows;
                // flat entries from 3 nc on keep what the resize kept
                const long long f = (long long)P.nbil + 3LL * k, lim = 3LL * nc;
                const size_t wi = (size_t)P.wbase + k;
                double gg[3];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                  gg[d] = (f + d < lim) ? (((f + d) % 3 == 0) ? 1.0 : 0.0)
                                        : (k < gsize ? a.gamma[d * a.WS + wi] : 0.0);
                g0 = gg[0]; g1 = gg[1]; g2 = gg[2];
              }
              const T x0 = (T)g0, x1 = (T)g1, x2 = (T)g2;
              T* gi = iter_at(a.G[0], c);
              gi[0] = x0; gi[32] = x1; gi[64] = x2;
              const T e0 = x0 + T(-1), e1 = x1 + T(-1), e2 = x2 + T(-1);
              acc[0] = acc[0] + dot3i(e0, e1, e2, e0, e1, e2);
              // the contact's constants
              T* p = const_at(a, c);
              Frame<T> f;
              if (kMixed) {
                const T m0 = (T)n0, m1 = (T)n1, m2 = (T)n2;
                const FrameWords<T> w = frame_words(m0, m1, m2, false);
                f = make_frame<T>(m0, m1, m2, w);
                p[96] = w.a; p[128] = w.b; p[160] = w.iv;
              } else {
                f = make_frame<T>((T)n0, (T)n1, (T)n2, FrameWords<T>{(T)fw.a, (T)fw.b, (T)fw.iv});
                p[96] = (T)fw.a; p[128] = (T)fw.b; p[160] = (T)fw.iv;
              }
              p[0] = f.n0; p[32] = f.n1; p[64] = f.n2;
              p[192] = r0; p[224] = r1; p[256] = r2;
              uint32_t* pi = reinterpret_cast<uint32_t*>(a.blk + (size_t)(c >> 5) * B::kConst + B::kIds) +
                             (c & 31);
              pi[0] = ia;
              pi[32] = ib;
              store_keep(qv + c, f_times<T, V>(f, e0, e1, e2));
            }
          }
          park_group<kGroups, 1, false>(park, pair, flip, nslot, t, acc);
          if (++nslot == kParkSlots) {
            fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
            nslot = 0;
          }
        }
        fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
      }
      if (!sync(kPhaseSetup)) return;
      fold_team<1, false, kGroups>(planes(), a.tcap, tm.nt, scratch, C.sums);
      if (threadIdx.x == 0) C.L0 = sqrt(C.sums[0]);
      parity ^= 1;
      team_body_pass<T, kAR>(a, tm, bodies, wv, qv);
      if (!sync(kPhaseSetup)) return;

      // ---- L = ||N e|| / ||e||; q = F gamma_0 for the first N y
      {
        int nslot = 0;
        for (int i = 0;; ++i) {
          const int t = team_tile(tm, i);
          if (t < 0) break;
          const int k0 = t * kTileItems;
          double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
          const int kb = a.nbil ? bil_tile_k0(t, 0, nc) : -1;
          if (kb >= 0) {
            // bilateral rows: (N e)_row; q = gamma_0 for the first N y
            const T* wt = reinterpret_cast<const T*>(wv);
            for (int m = group; m < kItemsPerThread; m += kGroups) {
              const int k = kb + m * kThreads + tid;
              if (k < P.nbil) {
                const int i2 = P.bil0 + k;
                const T n0 = bil_dw<T>(__ldg(a.bil_off + i2), wt);
                acc[0] = acc[0] + (double)n0 * (double)n0;
                a.bq[i2] = a.bG[0][i2];
              }
            }
          }
          for (int m = group; m < kItemsPerThread && kb < 0; m += kGroups) {
            int k = k0 + m * kThreads + tid;
            if (k < nc) {
              const int c = c0 + k;
              const Frame<T> f = block_frame<T>(const_at(a, c));
              const uint2 id = block_ids(a, c);
              V wa = load_vec(wv + id.x), wb = load_vec(wv + id.y);
              T n0, n1, n2;
              ft_times<T, V>(f, wa, wb, &n0, &n1, &n2);
              acc[0] = acc[0] + dot3i(n0, n1, n2, n0, n1, n2);
              const T* gi = iter_at(a.G[0], c);
              store_keep(qv + c, f_times<T, V>(f, gi[0], gi[32], gi[64]));
            }
          }
          park_group<kGroups, 1, false>(park, pair, flip, nslot, t, acc);
          if (++nslot == kParkSlots) {
            fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
            nslot = 0;
          }
        }
        fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
      }
      if (!sync(kPhaseSetup)) return;
      fold_team<1, false, kGroups>(planes(), a.tcap, tm.nt, scratch, C.sums);
      if (threadIdx.x == 0) ctl_lipschitz(C, P, nc, cap, kMixed);
      parity ^= 1;
      team_body_pass<T, kAR>(a, tm, bodies, wv, qv);
      if (!sync(kPhaseSetup)) return;

      // ---- APGD iterations (APGD.cu:227-350)
      //
      // Each iteration is one body pass (w = Minv D^T q of gamma_new) and one
      // contact pass that computes N gamma_new, the objective and the residual of
      // iteration k, and -- assuming the Lipschitz test accepts gamma_new -- the
      // whole step of iteration k+1 (y, N y, g, gamma_new = P(y - t g), q).  When
      // the test fails (backtracking) the look-ahead is discarded and a step pass
      // recomputes gamma_new with the doubled L; the arithmetic of every value is
      // the same either way.  A scene's first step is a step pass too (N y_0
      // is a product: w of gamma_0).
      while (!C.done) {
        if (C.step) {
          int nslot = 0;
          const int cur = C.cur, prev = C.prev, first = C.first, yr = C.yr;
          const T ya = (T)C.step_ya, ym = (T)C.step_ym, nt_ = (T)C.step_nt;
          T* Xc = a.G[cur];
          const T* Xp = a.G[prev < 0 ? cur : prev];
          T* Xn = a.G[C.nw];
          // A member of several tiles brings the constants and gamma_k with its
          // product through the stages; of gamma_{k-1}, and with one tile of all
          // (nothing would hide the copies), the lines of the next sub-tile go to L2.
          const bool staged = tm.ntc > tm.m;
          auto bring = [&](int j) {
            const int t = contact_tile(tm, tile_of(j));
            const int kw = t * kTileItems + sub_of(j) * kSub + gwarp * 32;
            if (t < 0 || kw >= nc) return;
            const size_t blk = (size_t)(c0 + kw) >> 5;
            const auto lines = [&](const T* p, unsigned bytes) {
              if (lane * 128u < bytes) prefetch_l2(reinterpret_cast<const unsigned char*>(p) + lane * 128);
            };
            if (!yr) lines(Xp + blk * kIterBlock, 2 * B::kHalfBytes);
            if (!staged) {
              lines(a.blk + blk * B::kConst, B::kConstBytes);
              lines(Xc + blk * kIterBlock, 2 * B::kHalfBytes);
            } else if (lane == 0) {
              const int sidx = j & 1;
              unsigned char* dst = stg.base + (size_t)(2 * warp + sidx) * B::kStageBytes;
              uint64_t* bar = stg.bar + 2 * warp + sidx;
              mark_stage_issued(stg, sidx);
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              mbar_arrive_expect_tx(bar, B::kConstBytes + 2u * B::kHalfBytes);
              bulk_g2s(dst, a.blk + blk * B::kConst, B::kConstBytes, bar);
              bulk_g2s(dst + B::kConstBytes, Xc + blk * kIterBlock, 2 * B::kHalfBytes, bar);
            }
          };
          if (staged) {
            asm volatile("fence.proxy.async;" ::: "memory");
            __syncwarp();
            bring(0);
          }
          bring(1);
          bool failed = false;
          int j = 0;  // sub-tile of this member
          for (int i = 0;; ++i) {
            const int t = team_tile(tm, i);
            if (t < 0) break;
            const int k0 = t * kTileItems;
            double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            const int kb = a.nbil ? bil_tile_k0(t, 0, nc) : -1;
            if (kb >= 0) {
              // bilateral rows: the same step without the cone projection
              const T* wt = reinterpret_cast<const T*>(wv);
              const T* bGc = a.bG[cur];
              const T* bGp = a.bG[prev < 0 ? cur : prev];
              T* bNGc = a.bNG[cur];
              const T* bNGp = a.bNG[prev < 0 ? cur : prev];
              T* bGn = a.bG[C.nw];
              for (int m = group; m < kItemsPerThread; m += kGroups) {
                const int k = kb + m * kThreads + tid;
                if (k < P.nbil) {
                  const int i2 = P.bil0 + k;
                  const T c0v = bGc[i2];
                  T y0, N0;
                  if (yr) y0 = c0v;
                  else y0 = ya * c0v + ym * bGp[i2];
                  if (first) {
                    N0 = bil_dw<T>(__ldg(a.bil_off + i2), wt);
                    bNGc[i2] = N0;
                  } else if (yr) {
                    N0 = bNGc[i2];
                  } else {
                    N0 = ya * bNGc[i2] + ym * bNGp[i2];
                  }
                  const T r0 = a.br[i2];
                  const T g0 = N0 + r0;
                  const T x0 = y0 + nt_ * g0;
                  bGn[i2] = x0;
                  a.bq[i2] = x0;
                  const T t0 = x0 + T(-1) * y0, s0 = x0 + T(-1) * c0v;
                  acc[0] = acc[0] + (double)g0 * (double)t0;
                  acc[1] = acc[1] + (double)t0 * (double)t0;
                  acc[2] = acc[2] + (double)g0 * (double)s0;
                  if (first) {
                    acc[3] = acc[3] + (double)y0 * (double)N0;
                    acc[4] = acc[4] + (double)y0 * (double)r0;
                  }
                }
              }
            }
            for (int m = group; m < kItemsPerThread && kb < 0; m += kGroups, ++j) {
              const int sidx = j & 1;
              if (j > 0 && !failed) {
                __syncwarp();  // the warp's reads of the other stage are done
                bring(j + 1);
              }
              const int kw = k0 + m * kSub + gwarp * 32;
              const int k = kw + lane;
              const int c = c0 + k;
              T p0 = T(0), p1 = T(0), p2 = T(0), q0 = T(0), q1 = T(0), q2 = T(0);
              if (k < nc && !yr) {
                const T* xp = iter_at(Xp, c);
                p0 = xp[0]; p1 = xp[32]; p2 = xp[64];
                q0 = xp[96]; q1 = xp[128]; q2 = xp[160];
              }
              if (staged && kw < nc && !failed && !wait_warp_stage(a, stg, sidx)) {
                failed = true;
                s_copy_fail = 1;
              }
              if (k < nc && !failed) {
                const T* p = const_at(a, c);
                const T* x = iter_at(Xc, c);
                if (staged) {
                  p = reinterpret_cast<const T*>(stg.base + (size_t)(2 * warp + sidx) * B::kStageBytes) + lane;
                  x = p + B::kConst;
                }
                const Frame<T> f = block_frame<T>(p);
                const T c0v = x[0], c1v = x[32], c2v = x[64];
                T y0, y1, y2, N0, N1, N2;
                if (yr) {
                  y0 = c0v; y1 = c1v; y2 = c2v;
                } else {
                  y0 = ya * c0v + ym * p0;
                  y1 = ya * c1v + ym * p1;
                  y2 = ya * c2v + ym * p2;
                }
                if (first) {
                  const uint2 id = block_ids(a, c);
                  V wa = load_vec(wv + id.x), wb = load_vec(wv + id.y);
                  ft_times<T, V>(f, wa, wb, &N0, &N1, &N2);
                  T* xc = iter_at(Xc, c);
                  xc[96] = N0; xc[128] = N1; xc[160] = N2;
                } else if (yr) {
                  N0 = x[96]; N1 = x[128]; N2 = x[160];
                } else {
                  N0 = ya * x[96] + ym * q0;
                  N1 = ya * x[128] + ym * q1;
                  N2 = ya * x[160] + ym * q2;
                }
                const T r0 = kAR ? (T)a.ar_r0[(size_t)C.rsel * S + c] : p[192];
                const T r1 = p[224], r2 = p[256];
                const T g0 = N0 + r0, g1 = N1 + r1, g2 = N2 + r2;
                T x0 = y0 + nt_ * g0, x1 = y1 + nt_ * g1, x2 = y2 + nt_ * g2;
                project_cone<T>(x0, x1, x2, cone_of<T>(C));
                T* xn = iter_at(Xn, c);
                xn[0] = x0; xn[32] = x1; xn[64] = x2;
                store_keep(qv + c, f_times<T, V>(f, x0, x1, x2));
                const T t0 = x0 + T(-1) * y0, t1 = x1 + T(-1) * y1, t2 = x2 + T(-1) * y2;
                const T s0 = x0 + T(-1) * c0v, s1 = x1 + T(-1) * c1v, s2 = x2 + T(-1) * c2v;
                acc[0] = acc[0] + dot3i(g0, g1, g2, t0, t1, t2);
                acc[1] = acc[1] + dot3i(t0, t1, t2, t0, t1, t2);
                acc[2] = acc[2] + dot3i(g0, g1, g2, s0, s1, s2);
                if (first) {
                  acc[3] = acc[3] + dot3i(y0, y1, y2, N0, N1, N2);
                  acc[4] = acc[4] + dot3i(y0, y1, y2, r0, r1, r2);
                }
              }
            }
            park_group<kGroups, 5, false>(park, pair, flip, nslot, t, acc);
            if (++nslot == kParkSlots) {
              fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
              nslot = 0;
            }
          }
          fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
          if (s_copy_fail) {
            drain_warp_stages(stg, &a.ew->wait_limit_ns);
            return;
          }
          if (!sync(kPhaseStep)) return;
          fold_team<5, false, kGroups>(planes(), a.tcap, tm.nt, scratch, C.sums);
          if (threadIdx.x == 0) ctl_step(C);
          parity ^= 1;
          __syncthreads();
        }

        // ---- the contact pass's sub-tiles of this member
        const int cur = C.cur, nw = C.nw, restart = C.restart;
        auto issue = [&](int j) {  // this warp's sub-tile j into stage j & 1
          const int t = contact_tile(tm, tile_of(j));
          const int kw = t * kTileItems + sub_of(j) * kSub + gwarp * 32;
          if (t >= 0 && kw < nc && lane == 0) {
            const int sidx = j & 1;
            const size_t blk = (size_t)(c0 + kw) >> 5;
            unsigned char* dst = stg.base + (size_t)(2 * warp + sidx) * B::kStageBytes;
            uint64_t* bar = stg.bar + 2 * warp + sidx;
            mark_stage_issued(stg, sidx);
            // gamma_k and N gamma_k only enter without a restart
            mbar_arrive_expect_tx(bar, B::kConstBytes + (restart ? 1u : 3u) * B::kHalfBytes);
            bulk_g2s(dst, a.blk + blk * B::kConst, B::kConstBytes, bar);
            bulk_g2s(dst + B::kConstBytes, a.G[nw] + blk * kIterBlock, B::kHalfBytes, bar);
            if (!restart)
              bulk_g2s(dst + B::kConstBytes + B::kHalfBytes, a.G[cur] + blk * kIterBlock,
                       2 * B::kHalfBytes, bar);
          }
        };
        team_body_pass<T, kAR>(a, tm, bodies, wv, qv);
        // while the barrier waits: the copies of the first two sub-tiles, and the
        // next controller's scalars.  This warp's earlier writes of the iterates,
        // and its reads of the stages, come before the copies (once for the pass:
        // a fence of global memory waits for the warp's stores).
        if (!team_sync(a, tm, false, [&]() {
              asm volatile("fence.proxy.async;" ::: "memory");
              __syncwarp();
              issue(0);
              issue(1);
              if (threadIdx.x == 32) ctl_ahead(C);
            })) {
          drain_warp_stages(stg, &a.ew->wait_limit_ns);
          return;
        }
        timer.mark(a, kPhaseBody);

        // N gamma_new, objective (APGD.cu:237-238), residual (:90-102); then the
        // next iteration's step assuming gamma_new is accepted (:266-273, 312-332)
        {
          int nslot = 0;
          double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
          bool bad = false, failed = false;
          T* Xn = a.G[nw];
          T* X2 = a.G[C.nw2];
          for (int j = 0;; ++j) {
            const int t = contact_tile(tm, tile_of(j));
            if (t < 0) break;
            const int sidx = j & 1, sub = sub_of(j);
            if (j && !failed) {
              __syncwarp();  // the warp's reads of stage sidx^1 are done
              if (lane == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              issue(j + 1);
            }
            const int kw = t * kTileItems + sub * kSub + gwarp * 32;
            if (kw < nc && !failed && !wait_warp_stage(a, stg, sidx)) {
              failed = true;
              s_copy_fail = 1;
            }
            const int k = kw + lane;
            if (k < nc && !failed) {
              const int c = c0 + k;
              const T* sd =
                  reinterpret_cast<const T*>(stg.base + (size_t)(2 * warp + sidx) * B::kStageBytes) + lane;
              const uint32_t* su = reinterpret_cast<const uint32_t*>(
                  stg.base + (size_t)(2 * warp + sidx) * B::kStageBytes + B::kIds * sizeof(T)) + lane;
              const uint32_t ia = su[0], ib = su[32];
              const V wa = load_vec(wv + ia), wb = load_vec(wv + ib);
              const Frame<T> f = block_frame<T>(sd);
              const T* sx = sd + B::kConst;
              T N0, N1, N2;
              ft_times<T, V>(f, wa, wb, &N0, &N1, &N2);
              T* xn = iter_at(Xn, c);
              xn[96] = N0; xn[128] = N1; xn[160] = N2;
              const T x0 = sx[0], x1 = sx[32], x2 = sx[64];
              T r0 = sd[192];
              const T r1 = sd[224], r2 = sd[256];
              if (kAR) r0 = (T)a.ar_r0[(size_t)C.rsel * S + c];
              acc[0] = acc[0] + dot3i(x0, x1, x2, N0, N1, N2);
              acc[1] = acc[1] + dot3i(x0, x1, x2, r0, r1, r2);
              {
                // residual, FP64 in both paths (gd = 1/nc^2 is far below float
                // resolution).  The mixed path takes it at the FP64 projection of
                // the FP32 iterate: the residual divides by gd, which would
                // otherwise magnify the iterate's float rounding off the cone.
                double X0 = x0, X1 = x1, X2v = x2;
                if (kMixed) project_cone<double>(X0, X1, X2v, C.cone);
                const double gd = C.gdiff, gA = C.ginv, gB = C.gneg;
                double T0 = (double)r0 + (double)N0, T1 = (double)r1 + (double)N1,
                       T2 = (double)r2 + (double)N2;
                T0 = X0 + (-gd) * T0; T1 = X1 + (-gd) * T1; T2 = X2v + (-gd) * T2;
                project_cone<double>(T0, T1, T2, C.cone);
                T0 = gA * X0 + gB * T0; T1 = gA * X1 + gB * T1; T2 = gA * X2v + gB * T2;
                double m0 = fabs(T0), m1 = fabs(T1), m2 = fabs(T2);
                bad |= (m0 != m0) || (m1 != m1) || (m2 != m2);
                acc[7] = fmax(acc[7], fmax(m0, fmax(m1, m2)));
              }
              // look-ahead step of iteration k+1: y = (1+b) x - b gamma_k, or x after a restart
              T y0, y1, y2, M0, M1, M2;
              if (restart) {
                y0 = x0; y1 = x1; y2 = x2;
                M0 = N0; M1 = N1; M2 = N2;
              } else {
                const T ya = (T)C.prod_ya, ym = (T)C.prod_ym;
                y0 = ya * x0 + ym * sx[96]; y1 = ya * x1 + ym * sx[128]; y2 = ya * x2 + ym * sx[160];
                M0 = ya * N0 + ym * sx[192];
                M1 = ya * N1 + ym * sx[224];
                M2 = ya * N2 + ym * sx[256];
              }
              T rn0 = r0;  // r_n of the next iteration
              if (kAR) {
                // APGD.cu:335-345 for gamma_new = x: v = Minv (k + D^T x) of the
                // body pass, s = (D v)_(u, v), ar = sqrt(s_u^2 + s_v^2) mu;
                // r_n' = ar + (-ar_old + r_n), into the next plane
                const double4 va = a.v_ar[ia], vb = a.v_ar[ib];
                const double d0 = va.x - vb.x, d1 = va.y - vb.y, d2 = va.z - vb.z;
                const double s_u = (f.u0 * d0 + f.u1 * d1) + f.u2 * d2;
                const double s_v = (f.v0 * d0 + f.v1 * d1) + f.v2 * d2;
                const double arn = sqrt(s_u * s_u + s_v * s_v) * C.cone.mu;
                const size_t cur_p = (size_t)C.rsel * S + c, nxt_p = (size_t)(C.rsel ^ 1) * S + c;
                const double rnn = arn + (-a.ar_v[cur_p] + (double)r0);
                a.ar_r0[nxt_p] = rnn;
                a.ar_v[nxt_p] = arn;
                rn0 = (T)rnn;
              }
              const T nt2 = (T)C.prod_nt;
              T g0 = M0 + rn0, g1 = M1 + r1, g2 = M2 + r2;
              T z0 = y0 + nt2 * g0, z1 = y1 + nt2 * g1, z2 = y2 + nt2 * g2;
              project_cone<T>(z0, z1, z2, cone_of<T>(C));
              T* x2p = iter_at(X2, c);
              x2p[0] = z0; x2p[32] = z1; x2p[64] = z2;
              store_keep(qv + c, f_times<T, V>(f, z0, z1, z2));
              T t0 = z0 + T(-1) * y0, t1 = z1 + T(-1) * y1, t2 = z2 + T(-1) * y2;
              T s0 = z0 + T(-1) * x0, s1 = z1 + T(-1) * x1, s2 = z2 + T(-1) * x2;
              acc[2] = acc[2] + dot3i(g0, g1, g2, t0, t1, t2);
              acc[3] = acc[3] + dot3i(t0, t1, t2, t0, t1, t2);
              acc[4] = acc[4] + dot3i(g0, g1, g2, s0, s1, s2);
              acc[5] = acc[5] + dot3i(y0, y1, y2, M0, M1, M2);
              acc[6] = acc[6] + dot3i(y0, y1, y2, rn0, r1, r2);
            }
            if (kGroups == 2 || sub == kItemsPerThread - 1) {
              if (__any_sync(0xffffffffu, bad) && lane == 0) seg_error(a, s, kErrNaN);
              park_group<kGroups, 7, true>(park, pair, flip, nslot, t, acc);
#pragma unroll
              for (int q = 0; q < 8; ++q) acc[q] = 0.0;
              bad = false;
              if (++nslot == kParkSlots) {
                fold_parked8<true, kT>(park, planes(), a.tcap, nslot);
                nslot = 0;
              }
            }
          }
          fold_parked8<true, kT>(park, planes(), a.tcap, nslot);
          if (s_copy_fail) {
            drain_warp_stages(stg, &a.ew->wait_limit_ns);
            return;
          }
          if (a.nbil) {
            // then the bilateral rows' tiles: N gamma_new, the objective and
            // residual items and the look-ahead step, without the cone projection
            nslot = 0;
            const T* wt = reinterpret_cast<const T*>(wv);
            for (int i = 0;; ++i) {
              const int t = team_tile(tm, i);
              if (t < 0) break;
              const int kb = bil_tile_k0(t, 0, nc);
              if (kb < 0) continue;
              BilRows<T> br_{a.bil_off, wt, a.bG[cur], a.bG[nw], a.bG[C.nw2], a.bNG[cur],
                             a.bNG[nw], a.br, a.bq};
              double racc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
              const bool bad2 =
                  bil_product_tile<T, kGroups>(br_, C, P.bil0 + kb, P.nbil - kb, nc > 0, racc);
              park_group<kGroups, 7, true>(park, pair, flip, nslot, t, racc);
              if (__any_sync(0xffffffffu, bad2) && lane == 0) seg_error(a, s, kErrNaN);
              if (++nslot == kParkSlots) {
                fold_parked8<true, kT>(park, planes(), a.tcap, nslot);
                nslot = 0;
              }
            }
            fold_parked8<true, kT>(park, planes(), a.tcap, nslot);
          }
        }
        if (!sync(kPhaseProduct)) return;
        fold_team<7, true, kGroups>(planes(), a.tcap, tm.nt, scratch, C.sums);
        if (threadIdx.x == 0) ctl_product(C, P, cap, kMixed, kAR);
        parity ^= 1;
        __syncthreads();
      }

      // ---- anti-relaxation: objectiveCCP = 1/2 gamma_hat' N gamma_hat + gamma_hat' r
      // with the last r (APGD.cu:353-354); the first term was kept when gamma_hat was
      // found, the second is folded over the tiles here (one scene)
      if (kAR) {
        int nslot = 0;
        const int best = C.best;
        for (int i = 0;; ++i) {
          const int t = team_tile(tm, i);
          if (t < 0) break;
          double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
          if (best >= 0) {
            for (int m = group; m < kItemsPerThread; m += kGroups) {
              const int k = t * kTileItems + m * kThreads + tid;
              if (k < nc) {
                const int c = c0 + k;
                const T* x = iter_at(a.G[best], c);
                const T* p = const_at(a, c);
                acc[0] = acc[0] + dot3i(x[0], x[32], x[64], a.ar_r0[(size_t)C.rsel * S + c],
                                        (double)p[224], (double)p[256]);
              }
            }
          }
          park_group<kGroups, 1, false>(park, pair, flip, nslot, t, acc);
          if (++nslot == kParkSlots) {
            fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
            nslot = 0;
          }
        }
        fold_parked8<false, kT>(park, planes(), a.tcap, nslot);
        if (!sync(kPhaseFinal)) return;
        fold_team<1, false, kGroups>(planes(), a.tcap, tm.nt, scratch, C.sums);
        if (threadIdx.x == 0 && best >= 0) C.objective = C.objN + C.sums[0];
        parity ^= 1;
        __syncthreads();
      }

      // ---- gamma = gamma_hat (APGD.cu:358) into the warm-start region; q = F gamma (FP64)
      {
        const int best = C.best;
        // a refinement whose FP64 phase accepted no iterate keeps the FP32
        // launch's gamma_hat; q is formed again (the setup wrote over it)
        const bool keep = a.refine && best < 0;
        const T* src = best >= 0 ? a.G[best] : nullptr;
        for (int i = 0;; ++i) {
          const int t = team_tile(tm, i);
          if (t < 0) break;
          const int kb = a.nbil ? bil_tile_k0(t, 0, nc) : -1;
          if (kb >= 0) {
            // the rows' gamma_hat (ones before the first accepted iterate)
            for (int m = group; m < kItemsPerThread; m += kGroups) {
              const int k = kb + m * kThreads + tid;
              if (k < P.nbil) {
                const int r = P.bil0 + k;
                a.bil_gam[r] = best >= 0 ? (double)a.bG[best][r] : 1.0;
              }
            }
            continue;
          }
          for (int m = group; m < kItemsPerThread; m += kGroups) {
            int k = t * kTileItems + m * kThreads + tid;
            if (k < nc) {
              const int c = c0 + k;
              double x0 = 1.0, x1 = 1.0, x2 = 1.0;
              const size_t wi = (size_t)P.wbase + k;
              if (keep) {
                x0 = a.gamma[0 * a.WS + wi]; x1 = a.gamma[1 * a.WS + wi]; x2 = a.gamma[2 * a.WS + wi];
              } else {
                if (src) {
                  const T* x = iter_at(src, c);
                  x0 = (double)x[0]; x1 = (double)x[32]; x2 = (double)x[64];
                }
                a.gamma[0 * a.WS + wi] = x0;
                a.gamma[1 * a.WS + wi] = x1;
                a.gamma[2 * a.WS + wi] = x2;
              }
              a.wid[wi] = __ldg(a.idb + c) - (uint32_t)P.b0;
              Frame<double> f;
              if (kMixed) f = load_frame_fp64(a, c, P.exact != 0);
              else {
                const T* p = const_at(a, c);
                f = make_frame<double>((double)p[0], (double)p[32], (double)p[64],
                                       FrameWords<double>{(double)p[96], (double)p[128], (double)p[160]});
              }
              a.qd[c] = f_times<double, double4>(f, x0, x1, x2);
            }
          }
        }
      }
      if (!sync(kPhaseFinal)) return;
    }

    // mixed precision: a solve that ended above the tolerance without an error
    // is refined in FP64 by the launch that follows, which also updates it
    const unsigned err = C.err | (live ? __ldcg(&a.sst[s].err) : 0u);
    const bool refine_next = kMixed && P.refine > 0 && live && err == 0u && !(C.residual < P.tol);

    // Where an error ends the call (plain scenes), one in the FP32 phase of a
    // solve with refinement leaves the scene as it was: the update is the FP64
    // phase's, which it does not get to.
    const bool stay = kMixed && P.refine > 0 && err != 0u && a.ew->stop_on_seg_err;

    // ---- f_c = D^T gamma; v = Minv (k + f_c); f_contact = f_c / h; p += h v.
    // Scenes with neither contacts nor bilateral rows: v = Minv k, f_contact = 0
    // (System.cu:577-581); the rows' impulses enter f_c like the contacts'.
    if (!a.solve_only && !refine_next && !stay) {
      for (int b = tm.w0 + threadIdx.x; b < tm.w1; b += kT) {
        const double h = P.h;
        double4 k = a.k4[b];
        double mi = __ldg(a.minv + b);
        double4 v, fcv;
        if (live) {
          double4 fc = gather_q<double, double4>(a, a.qd, b);
          if (a.nbil) add_bilateral<double, double4>(a.bil_inc_start, a.bil_inc, a.bil_gam, b, fc);
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
    }
    // matched warm start: where each body's A-contacts went in the warm region
    if (live) {
      const int shift = a.sst[s].delta - c0;
      for (int b = tm.w0 + threadIdx.x; b < tm.w1; b += kT) {
        a.ws[b] = a.cbase[b] + shift;
        a.wc[b] = a.cnt_cont[b];
      }
    }
    // the scene's results, and its warm-start length (System::gamma_d resize)
    if (tm.rank == 0 && threadIdx.x == 0) {
      SegState& X = a.sst[s];
      SolveResult& D = X.ctl;
      if (C.err) {
        X.err = err;
        if (a.ew->stop_on_seg_err) atomicOr(&a.ew->err, C.err);
      }
      D.iterations = C.iterations + it_lo;
      D.backtracks = C.backtracks + bt_lo;
      D.sweeps = C.sweeps + sw_lo;
      D.residual = C.residual;
      D.objective = C.objective;
      D.refine_it = a.refine ? C.iterations : 0;
      if (!a.refine) D.refined = refine_next ? 1 : 0;
      if (live) X.gsize = nc;
      // System::time += h (System.cu:584), read by the next step's rows
      if (a.nbil && !a.solve_only) a.seg_time[s] = a.seg_time[s] + P.h;
    }
  }
  timer.store(a);
}

// The scenes of one launch in teams (engines of several scenes): those that
// are active (in a refinement launch, those the FP32 launch marked), by size,
// largest first, each with one member per `per` tiles; slots[] lists (scene,
// rank) in that order.  One CTA.
__global__ void __launch_bounds__(1024) k_team_plan(int nseg, const SegParams* __restrict__ seg,
                                                    SegState* __restrict__ sst, int refine, int grid,
                                                    int2* __restrict__ slots, int slot_cap,
                                                    int* __restrict__ order,
                                                    unsigned* __restrict__ team_bar,
                                                    EngineWords* __restrict__ ew) {
  constexpr int kBins = 128;
  __shared__ int s_bin[kBins], s_tiles, s_warp[32], s_carry;
  if (ew->err) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kBins; i += 1024) s_bin[i] = 0;
  if (tid == 0) {
    s_tiles = 0;
    s_carry = 0;
  }
  __syncthreads();
  // bins of four per octave of the tiles, largest first
  auto bin_of = [](int nt) {
    if (nt < 4) return kBins - 1 - nt;
    const int e = 31 - __clz(nt);
    return kBins - 1 - (4 * (e - 1) + ((nt >> (e - 2)) & 3));
  };
  auto takes = [&](int s) { return seg[s].active && (!refine || sst[s].ctl.refined); };
  for (int s = tid; s < nseg; s += 1024) {
    if (!refine) sst[s].err = 0u;
    if (!takes(s)) continue;
    atomicAdd(&s_bin[bin_of(sst[s].nt)], 1);
    atomicAdd(&s_tiles, sst[s].nt);
  }
  __syncthreads();
  if (tid == 0) {
    int at = 0;
    for (int i = 0; i < kBins; ++i) {
      const int n = s_bin[i];
      s_bin[i] = at;
      at += n;
    }
    s_warp[0] = at;
  }
  __syncthreads();
  const int n = s_warp[0];
  // tiles per member: one while the grid has a CTA for each, then as many as
  // fill the grid, four at most (a team's barriers and folds cost about 8 us an
  // iteration, a tile about 5)
  const int per = max(1, min(kTeamTiles, (s_tiles + grid - 1) / grid));
  for (int s = tid; s < nseg; s += 1024) {
    if (!takes(s)) continue;
    order[atomicAdd(&s_bin[bin_of(sst[s].nt)], 1)] = s;
    sst[s].members = team_size(sst[s].nt, seg[s].b1 - seg[s].b0, per, grid);
    team_bar[(size_t)s * kTeamBarStride] = 0u;
  }
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int i = base + tid;
    const int s = i < n ? order[i] : -1;
    const int m = s >= 0 ? sst[s].members : 0;
    int x = m;
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    int before = s_carry, total = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += s_warp[w];
      total += s_warp[w];
    }
    const int at = before + x - m;
    for (int r = 0; r < m; ++r)
      if (at + r < slot_cap) slots[at + r] = make_int2(s, r);
    __syncthreads();
    if (tid == 0) s_carry += total;
    __syncthreads();
  }
  if (tid == 0) {
    ew->ticket = 0u;
    ew->nslots = min(s_carry, slot_cap);
  }
}

template <class T, int kGroups>
constexpr size_t solve_smem_bytes() {
  return (size_t)kWarps * kGroups * 2 * Block<T>::kStageBytes + (size_t)kMaxWarps * 2 * 8 + kMaxWarps +
         (kGroups == 2 ? sizeof(PairBuf) : 0);
}

// Co-resident CTAs of a form of the kernel on the current device, asked for once
// per device (a member of a team that never runs would be waited for).
template <class T, int G, int MB, bool AR>
int resident_ctas() {
  constexpr int kDevices = 64;
  static std::atomic<int> known[kDevices];
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  const bool keep = dev >= 0 && dev < kDevices;
  if (keep && known[dev].load(std::memory_order_relaxed)) return known[dev].load(std::memory_order_relaxed);
  const size_t smem = solve_smem_bytes<T, G>();
  const cudaError_t e = cudaFuncSetAttribute(
      k_step_solve<T, G, MB, AR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_step_solve<T, G, MB, AR>, kThreads * G, smem);
  const int n = sms * std::max(per_sm, 1);
  if (keep && e == cudaSuccess && per_sm > 0) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

template <class T, int G, int MB, bool AR = false>
void launch_typed(SceneDev& sd, const SolveConfig& cfg, cudaStream_t st, int64_t* launches,
                  bool solve_only, bool refine) {
  KArgs<T> a = make_kargs<T>(sd, cfg);
  a.solve_only = solve_only ? 1 : 0;
  a.refine = refine ? 1 : 0;
  const int grid = std::min(G == 2 ? std::max(1, cfg.grid / 2) : cfg.grid, resident_ctas<T, G, MB, AR>());
  plan_teams(sd, grid, refine, st, launches);
  void* params[] = {&a};
  cudaLaunchCooperativeKernel((const void*)k_step_solve<T, G, MB, AR>, grid, kThreads * G, params,
                              solve_smem_bytes<T, G>(), st);
  ++*launches;
}

// Which form of the kernel a launch takes (128 registers per thread in both):
// 512-thread CTAs for one scene of at most kPairBodies bodies, whose tiles are
// then at most about one per SM.  Solve per step in 512- and 256-thread CTAs:
// 1,000 spheres 1.63 and 1.73 ms, 20,011 mixed 8.16 and 8.95; 200,000 spheres
// 44 and 34 ms (their stages leave the body pass a sixth of the L1); 64 scenes
// 2.9 and 2.7 ms (their 160 tiles need a second wave).  Setup and one iteration
// near the line, FP64: 20,000 spheres 113 and 119 us, 30,000 131 and 139, 40,000
// 164 and 160.  A pile below the line that is dense enough for more tiles than SMs
// gains nothing or pays a little: 238 tiles 225 and 225 us, 517 tiles 25.7 and 23.1
// us per iteration.
template <class T, bool AR = false>
void launch_form(SceneDev& sd, const SolveConfig& cfg, cudaStream_t st, int64_t* launches,
                 bool solve_only, bool refine = false) {
  if (sd.nseg == 1 && sd.nb <= kPairBodies)
    launch_typed<T, 2, 1, AR>(sd, cfg, st, launches, solve_only, refine);
  else
    launch_typed<T, 1, 2, AR>(sd, cfg, st, launches, solve_only, refine);
}

}  // namespace

// Co-resident CTAs of the solve kernel for a precision and a register budget
// (blocks_per_sm 2: 128 registers per thread; 3: 80, FP32 iterates only).
int apgd_max_ctas(int precision, int blocks_per_sm) {
  if (precision == DV_PREC_MIXED)
    return blocks_per_sm == 3 ? resident_ctas<float, 1, 3, false>() : resident_ctas<float, 1, 2, false>();
  return resident_ctas<double, 1, 2, false>();
}

void plan_teams(SceneDev& sd, int grid, bool refine, cudaStream_t st, int64_t* launches) {
  if (sd.nseg > 1) {
    k_team_plan<<<1, 1024, 0, st>>>(sd.nseg, sd.seg, sd.sst, refine ? 1 : 0, grid, sd.slots,
                                    sd.slot_cap, sd.order, sd.team_bar, sd.ew);
    ++*launches;
  } else {
    cudaMemsetAsync(sd.team_bar, 0, sizeof(unsigned), st);
  }
}

void launch_step_solve(SceneDev& sd, const SolveConfig& cfg, cudaStream_t st, int64_t* launches,
                       bool solve_only) {
  if (sd.solver == DV_SOLVER_PGJ) {
    launch_pgj_solve(sd, cfg, st, launches, solve_only);
  } else if (sd.solver == DV_SOLVER_PGS) {
    launch_pgs_solve(sd, cfg, st, launches, solve_only);
  } else if (sd.precision == DV_PREC_MIXED) {
    // with refinement the FP32 launch leaves the update of the solves it marks
    // to an FP64 launch, which refines them first
    if (cfg.blocks_per_sm == 3) launch_typed<float, 1, 3>(sd, cfg, st, launches, solve_only, false);
    else launch_form<float>(sd, cfg, st, launches, solve_only);
    if (sd.refine_any) {
      SolveConfig c2 = cfg;
      c2.blocks_per_sm = 2;
      c2.grid = std::min(cfg.grid, std::max(1, sd.refine_grid));
      launch_form<double>(sd, c2, st, launches, solve_only, true);
    }
  } else if (sd.anti_relax) {
    launch_form<double, true>(sd, cfg, st, launches, solve_only);
  } else {
    launch_form<double>(sd, cfg, st, launches, solve_only);
  }
}

}  // namespace dv
