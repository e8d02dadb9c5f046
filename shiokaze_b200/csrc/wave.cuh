// Device helpers shared by the wavefront kernels (solver.cu, mic_pencil.cu).
#pragma once
#include "common.cuh"

namespace shkz {

#define SPIN_LIMIT (1 << 21)   // polling rounds of a bounded wait, ~0.15 s with the back-off of the polling loops

// Deterministic finish of a grid reduction: every block writes its partial;
// the last block to arrive sums them in block order.
__device__ __forceinline__ bool last_block(unsigned *counter) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned ticket = atomicAdd(counter, 1u);
    s_last = (ticket == gridDim.x - 1);
  }
  __syncthreads();
  return s_last;
}

struct WaveSync {
  int slot;
  unsigned finished;
  int epoch;
  int error;         // 0, or the slot that gave up waiting + 1
  int spin_limit;    // polling rounds of a bounded wait (0: SPIN_LIMIT); set by the host
  int skip_publish;  // fault injection (0: off): wavefront slot k - 1 of a forward pencil sweep does not publish
};

// Rounds a bounded wait polls before it gives up.
__device__ __forceinline__ int spin_rounds(const WaveSync *ws) {
  const int v = *((volatile const int *)&ws->spin_limit);
  return v > 0 ? v : SPIN_LIMIT;
}

}  // namespace shkz
