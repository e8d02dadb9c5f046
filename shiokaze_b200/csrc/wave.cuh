// Device helpers shared by the wavefront kernels (solver.cu, mic_pencil.cu).
#pragma once
#include "common.cuh"

namespace shkz {

// polling rounds of a bounded wait: 0.5 s in the pencil sweeps (0.24 us a round, measured), of that order in the others
#define SPIN_LIMIT (1 << 21)

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

// Exclusive scan of n counts by one warp, 32 at a time; returns the total. (One
// thread adding them up waited for a load per entry: 60 us for a 512^3 grid's
// 256 block sums, a few us this way.)
__device__ __forceinline__ int warp_scan_counts(int *v, int n) {
  const int lane = threadIdx.x & 31;
  int acc = 0;
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    const int own = i < n ? v[i] : 0;
    int incl = own;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (i < n) v[i] = acc + incl - own;
    acc += __shfl_sync(0xffffffffu, incl, 31);
  }
  return acc;
}

// error words of the three wave-sync blocks (factor, forward, backward)
__device__ __forceinline__ bool any_wave_error(const void *waves) {
  const WaveSync *w = static_cast<const WaveSync *>(waves);
  int e = 0;
  if (w)
    for (int i = 0; i < 3; ++i) e |= *((volatile const int *)&w[i].error);
  return e != 0;
}

__device__ __forceinline__ void store_release_system(unsigned long long *p, unsigned long long v) {
  asm volatile("st.release.sys.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void store_release_system(unsigned *p, unsigned v) {
  asm volatile("st.release.sys.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One thread, after it has updated st: the host's view of the solve. Launches
// that find st->done set return before they report, so a host that has seen
// `done` may clear the word before it resumes the solve.
__device__ __forceinline__ void report_progress(const SolverState *st) {
  if (!st->mail) return;
  unsigned long long v = (unsigned)st->iter | (unsigned long long)(st->done & 0xff) << kProgressDone;
  if (any_wave_error(st->waves)) v |= kProgressWaveError;
  if (st->status < 0) v |= kProgressNan;
  asm volatile("st.relaxed.sys.global.b64 [%0], %1;" ::"l"(&st->mail->progress), "l"(v) : "memory");
}
// the same with the residual norm in front of it
__device__ __forceinline__ void report_progress_rmax(const SolverState *st) {
  if (!st->mail) return;
  *(volatile double *)&st->mail->rmax = st->rmax;
  __threadfence_system();
  report_progress(st);
}

}  // namespace shkz
