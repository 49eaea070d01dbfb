// dv_selftest.cu -- makes the solve kernels' bounded waits run out on
// purpose, without a fault: a team of two whose second member never arrives at
// its barrier, and an mbarrier that expects 16 bytes no copy will bring.  The
// waits are the ones the solve kernels use (team_sync, bounded_mbar_wait); each
// must end after the limit with its error bit set, and the context stays usable.
// The barrier that a team forms at starts its limit again while other teams make
// progress: a second CTA makes some for a while, and stops.
#include "dv_team.cuh"

#include "dvide.h"

namespace dv {

namespace {

struct WaitTestArgs {
  EngineWords* ew;
  unsigned* team_bar;
  int nseg;
};

__global__ void __launch_bounds__(kThreads) k_selftest_waits(WaitTestArgs a, int* out) {
  __shared__ __align__(8) uint64_t bar[1];
  __shared__ Team tm;
  if (threadIdx.x == 0) {
    // a team of two whose second member never arrives
    tm.rank = 0;
    tm.m = 2;
    tm.fail = 0;
    tm.target = 0;
    tm.bar = a.team_bar;
  }
  __syncthreads();
  const bool barrier_ok = team_sync(a, tm);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  bool copy_ok = true;
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) mbar_arrive_expect_tx(bar, 16u);  // no copy follows
    __syncwarp();
    copy_ok = __all_sync(0xffffffffu, bounded_mbar_wait(bar, 0u, &a.ew->wait_limit_ns));
  }
  if (threadIdx.x == 0) {
    if (!copy_ok) atomicOr(&a.ew->err, kErrCopyTimeout);
    out[0] = barrier_ok ? 0 : 1;
    out[1] = copy_ok ? 0 : 1;
  }
}

// CTA 0: a member of a team of two whose second one never joins.  CTA 1: another
// team, which passes `passes` barriers of its own, a quarter of the limit apart.
// ns: when the wait ended, and when the last progress was made.
__global__ void __launch_bounds__(kThreads) k_selftest_join(WaitTestArgs a, int passes, int* out,
                                                           unsigned long long* ns) {
  __shared__ Team tm;
  const uint64_t limit = a.ew->wait_limit_ns;
  if (threadIdx.x == 0) {
    tm.rank = blockIdx.x == 0 ? 1 : 0;  // the first member reports progress
    tm.m = blockIdx.x == 0 ? 2 : 1;
    tm.fail = 0;
    tm.target = 0;
    tm.bar = a.team_bar + blockIdx.x;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    const bool ok = team_sync(a, tm, true);
    if (threadIdx.x == 0) {
      *out = ok ? 0 : 1;
      ns[0] = global_ns();
    }
    return;
  }
  for (int i = 0; i < passes; ++i) {
    const uint64_t t0 = global_ns();
    while (global_ns() - t0 < limit / 4) __nanosleep(1000);
    team_sync(a, tm);
    if (threadIdx.x == 0) ns[1] = global_ns();
  }
}

}  // namespace

}  // namespace dv

using namespace dv;

DV_API int dv_selftest_bounded_waits(int32_t limit_ms, int32_t* barrier_timed_out,
                                     int32_t* copy_timed_out, uint32_t* error_bits) {
  if (limit_ms <= 0) return DV_ERR_ARG;
  EngineWords* ew = nullptr;
  int* out = nullptr;  // two results, then the barrier's counter
  if (cudaMalloc(&ew, sizeof(EngineWords)) != cudaSuccess) return DV_ERR_OOM;
  if (cudaMalloc(&out, 3 * sizeof(int)) != cudaSuccess) {
    cudaFree(ew);
    return DV_ERR_OOM;
  }
  EngineWords h;
  memset(&h, 0, sizeof(h));
  h.wait_limit_ns = (unsigned long long)limit_ms * 1000000ull;
  int host_out[3] = {-1, -1, 0};
  cudaMemcpy(ew, &h, sizeof(h), cudaMemcpyHostToDevice);
  cudaMemcpy(out, host_out, sizeof(host_out), cudaMemcpyHostToDevice);
  WaitTestArgs a{ew, reinterpret_cast<unsigned*>(out + 2), 1};
  k_selftest_waits<<<1, kThreads>>>(a, out);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(host_out, out, sizeof(host_out), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(&h, ew, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(out);
  cudaFree(ew);
  if (e != cudaSuccess) return dv_record_cuda_error(e, "dv_selftest_bounded_waits", __FILE__, __LINE__);
  if (barrier_timed_out) *barrier_timed_out = host_out[0];
  if (copy_timed_out) *copy_timed_out = host_out[1];
  if (error_bits) *error_bits = h.err;
  return DV_OK;
}

DV_API int dv_selftest_bounded_join(int32_t limit_ms, int32_t passes, int32_t* timed_out,
                                    double* ms_after_progress, uint32_t* error_bits) {
  if (limit_ms <= 0 || limit_ms > 500 || passes < 0 || passes > 100) return DV_ERR_ARG;
  struct Words {
    EngineWords ew;
    unsigned long long ns[2];
    unsigned bar[2];
    int out;
  };
  Words h{};
  h.ew.wait_limit_ns = (unsigned long long)limit_ms * 1000000ull;
  h.out = -1;
  Words* d = nullptr;
  if (cudaMalloc(&d, sizeof(Words)) != cudaSuccess) return DV_ERR_OOM;
  cudaError_t e = cudaMemcpy(d, &h, sizeof(h), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    // both CTAs run at once: the first sees the second's progress
    WaitTestArgs a{&d->ew, d->bar, 2};
    int* out = &d->out;
    unsigned long long* ns = d->ns;
    void* params[] = {&a, &passes, &out, &ns};
    e = cudaLaunchCooperativeKernel((const void*)k_selftest_join, 2, kThreads, params, 0, 0);
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return dv_record_cuda_error(e, "dv_selftest_bounded_join", __FILE__, __LINE__);
  if (timed_out) *timed_out = h.out;
  if (ms_after_progress) *ms_after_progress = passes ? ((double)h.ns[0] - (double)h.ns[1]) / 1e6 : 0.0;
  if (error_bits) *error_bits = h.ew.err;
  return DV_OK;
}
