// Self-test of the bounded device-side wait: a kernel that waits on a barrier nobody arrives on.
// It exercises the path every tensor-core kernel takes when a wait runs out (status word written,
// kernel returns, the context stays usable) without faulting or hanging anything.  It also leaves counts of arrived slices behind
// that are not zero, as a launch that gave up may; with these no slice would ever be found the last of its tile.
#include "internal.h"
#include "ptx.cuh"

namespace b200 {
namespace {

struct Bars {
  uint64_t never, over;         // nobody arrives; complete from the start
  volatile int abort;
};

__global__ void __launch_bounds__(128, 1) wait_selftest_kernel(int* status, unsigned int* arrivals, int narrivals, long long limit) {
  __shared__ Bars bars;
  if (threadIdx.x == 0) {
    mbar_init(&bars.never, 1);
    mbar_init(&bars.over, 1);
    bars.abort = 0;
    mbar_fence_init();
    mbar_arrive(&bars.over);
  }
  for (int i = threadIdx.x; i < narrivals; i += blockDim.x) arrivals[i] = 0xFFFFFFFFu;
  __syncthreads();
  const int warp = uniform_warp_index();
  bool ok;
  if (warp == 0) {
    ok = uniform_wait(&bars.never, 0, &bars, limit);                               // the issuers' wait
    if (!ok && elect_one()) report_status(status, kStatusTimeout);
  } else if (warp >= 2) {
    // epilogue warps that meet at a named barrier, one of whose waits run out and the other's do not: both walk through all items
    ok = true;
    for (int item = 0; item < 3; ++item) {
      wait_or_walk_on(ok, warp == 2 ? &bars.never : &bars.over, 0, &bars, threadIdx.x & 31, limit);
      named_barrier(1, 64);
    }
  } else {
    ok = warp_wait_or_abort(&bars.never, 0, &bars, threadIdx.x & 31, limit);       // the epilogue warps' wait
    if (!ok && (threadIdx.x & 31) == 0) report_status(status, kStatusTimeout);
  }
  __syncthreads();
  if (bars.abort) abort_grace(limit);
}

}  // namespace

cudaError_t launch_wait_selftest(int* status, unsigned int* arrivals, int narrivals, long long limit, cudaStream_t s) {
  wait_selftest_kernel<<<1, 128, 0, s>>>(status, arrivals, narrivals, limit);
  return cudaGetLastError();
}

}  // namespace b200
