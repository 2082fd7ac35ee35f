// Self-test of the failure path every tensor-core kernel of this library shares: a bounded mbarrier wait
// that runs out, the device status word it sets, warps of one role that leave together although the wait of
// only one of them ran out, loads in flight that are waited for, and a context that stays usable afterwards.  Nothing faults, traps or spins
// without bound: one warp waits, for at most the given time, on a barrier that nothing ever arrives at.
#include "tc_common.cuh"

namespace m2 {
__device__ __align__(16) const uint32_t selftest_words[4] = {1u, 2u, 3u, 4u};
__global__ void wait_timeout_kernel(unsigned long long limit_ns) {
  __shared__ uint64_t bar[6];
  __shared__ __align__(16) uint32_t landed[4];
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 6; ++i) tc::mbar_init(bar + i, 1);
    abort_flag = 0;
    tc::mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    tc::mbar_arrive(bar + 1);
    tc::mbar_expect_tx(bar + 2, 16);
    tc::bulk_load(landed, selftest_words, 16, bar + 2);
    tc::mbar_expect_tx(bar + 5, 16);                               // of a load that never lands
  }
  // the last warp's barrier never completes, the others' does
  const int last = threadIdx.x >= 96;
  bool ok = tc::mbar_wait_ns(bar + !last, 0, &abort_flag, tc::ST_TIMEOUT_TMA, limit_ns);
  ok = tc::group_and<1, 128>(ok);
  if (ok) atomicOr(&m2_dev_status_word, tc::ST_TIMEOUT_EPI);     // a warp that would go on
  if (threadIdx.x == 0) {
    // a ring of four stages of which two were loaded into: one load has landed, the other never will
    if (!tc::drain_loads(bar + 2, 3, tc::ring_parities(1, 0), limit_ns) || landed[0] + landed[3] != 5u) atomicOr(&m2_dev_status_word, tc::ST_TIMEOUT_EMPTY);
    if (tc::drain_loads(bar + 2, 4, 6u, limit_ns / 4)) atomicOr(&m2_dev_status_word, tc::ST_TIMEOUT_MMA);
  }
  __syncthreads();
}
}  // namespace m2

extern "C" int m2_selftest_wait_timeout(unsigned long long limit_ns, void* stream) {
  M2_REQUIRE(limit_ns > 0 && limit_ns <= 1000000000ull, M2_ERR_ARG,
             "m2_selftest_wait_timeout: limit must be between 1 ns and 1 s");
  m2::wait_timeout_kernel<<<1, 128, 0, static_cast<cudaStream_t>(stream)>>>(limit_ns);
  M2_LAUNCH_CHECK("wait_timeout_kernel");
  return M2_OK;
}
