// TEST-ONLY translation unit (built by tests/test_gpu_bounded_waits.py, never linked into the library).
// Makes the kernels' bounded waits run out on purpose, the one way a wait failure may be provoked on a
// shared GPU: a flag that nothing sets, a limit of one millisecond, and a status word the host reads.
// No trap, no bad address, no endless loop; the context stays usable.
#define MOE_WAIT_LIMIT_NS 1000000ull   // 1 ms instead of the library's 0.4 s
#include "gemm_common.cuh"

namespace {

// The decode kernel's grid barrier with a target ONE ABOVE the number of CTAs that arrive.
__global__ void grid_barrier_probe(unsigned int* word2, int* status, unsigned int tag) {
  if (threadIdx.x != 0) return;
  if (blockIdx.x == 0) moe::grid_barrier_init(word2, tag);
  if (!moe::grid_barrier_tag_wait(word2, tag)) {
    atomicOr(status, 0x100);
    return;
  }
  moe::grid_barrier_arrive(word2);
  if (!moe::grid_barrier_wait(word2, tag, gridDim.x + 1)) atomicOr(status, moe::kErrGemm1Timeout);
}

// The producer's form of that wait, by a warp whose lanes ask for different targets: lanes below `split` for the one
// arrival there is, the others for one more.  results[lane] = what the lane was told; no collective follows.
__global__ void grid_barrier_lanes_probe(unsigned int* word2, int* results, int split, unsigned int tag) {
  const int lane = static_cast<int>(threadIdx.x);
  if (lane == 0) {
    moe::grid_barrier_init(word2, tag);
    moe::grid_barrier_arrive(word2);
  }
  __syncwarp();
  results[lane] = moe::grid_barrier_wait_warp(word2, tag, lane < split ? 1u : 2u) ? 1 : 0;
}

// The pipeline's mbarrier wait (a whole warp waits) on a phase that no arrival or TMA transaction ever completes; a
// second warp sees the CTA-wide abort flag and leaves as well.  Both warps then elect a lane, as the kernels do behind
// a wait.
__global__ void mbarrier_probe(int* status) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    moe::mbar_init(moe::smem_u32(&bar), 1);
    moe::fence_mbar_init();
  }
  __syncthreads();
  if (!moe::mbar_wait(moe::smem_u32(&bar), 0, &abort_flag) && moe::elect_one()) atomicOr(status, moe::kErrGemm2Timeout);
  __syncthreads();
  if (abort_flag) moe::settle_after_abort();
  if (threadIdx.x == 0 && abort_flag) atomicOr(status, 0x200);
}

// The answer of a warp whose lanes see different phases: lanes below `split` wait on a barrier that is complete, the
// others on one that never is.  results[lane] = what the lane was told (0 / 1).  No collective follows, so lanes that
// were told different things would still all leave.
__global__ void mbarrier_lanes_probe(int* results, int split) {
  __shared__ uint64_t bar[2];
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < 2; ++i) moe::mbar_init(moe::smem_u32(&bar[i]), 1);
    moe::fence_mbar_init();
    moe::mbar_arrive(moe::smem_u32(&bar[0]));
  }
  __syncthreads();
  const int lane = static_cast<int>(threadIdx.x);
  results[lane] = moe::mbar_wait(moe::smem_u32(&bar[lane < split ? 0 : 1]), 0, &abort_flag) ? 1 : 0;
}

}  // namespace

// status_dev: one int, zeroed by the caller; word_dev: two uints (any contents).  Returns the cudaError_t.
extern "C" int moe_test_wait_timeouts(int* status_dev, unsigned int* word_dev, void* stream_v) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  grid_barrier_probe<<<4, 32, 0, stream>>>(word_dev, status_dev, 0x5EEDu);
  mbarrier_probe<<<1, 64, 0, stream>>>(status_dev);
  return static_cast<int>(cudaGetLastError());
}

// results_dev: 32 ints.  Lanes below `split` wait for something that has happened, the others for something that never does.
extern "C" int moe_test_mbarrier_lanes(int* results_dev, int split, void* stream_v) {
  mbarrier_lanes_probe<<<1, 32, 0, static_cast<cudaStream_t>(stream_v)>>>(results_dev, split);
  return static_cast<int>(cudaGetLastError());
}

// The same of the decode kernel's grid barrier; word_dev: two uints (any contents).
extern "C" int moe_test_grid_barrier_lanes(int* results_dev, unsigned int* word_dev, int split, void* stream_v) {
  grid_barrier_lanes_probe<<<1, 32, 0, static_cast<cudaStream_t>(stream_v)>>>(word_dev, results_dev, split, 0x5EEDu);
  return static_cast<int>(cudaGetLastError());
}
