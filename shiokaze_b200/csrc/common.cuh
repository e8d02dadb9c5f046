// Shared definitions for the B200 pressure-projection kernels.
//
// Device layout ("tile pool"): the grid is cut into 8^3-cell tiles. Only
// tiles that contain at least one pressure unknown are kept; they are
// compacted into a pool of K tiles. Every per-cell solver array is stored
// pool-major, [K][512] floats, cell (ii,jj,kk) of a tile at ii + 8*jj + 64*kk
// (x fastest, like the reference's in-tile order, src/array/tiledarray3.cpp:806-808).
// A tile is 2 KB per FP32 field, so one CTA moves whole tiles with
// coalesced 16-byte accesses.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define SHKZ_T 8
#define SHKZ_TC 512          // cells per tile
#define SHKZ_LOG_T 3

namespace shkz {

// Neighbour slots in the per-tile neighbour table.
enum { NB_XM = 0, NB_XP = 1, NB_YM = 2, NB_YP = 3, NB_ZM = 4, NB_ZP = 5 };

struct Geometry {
  int nx, ny, nz;          // cells
  int bx, by, bz;          // tiles per axis
  long long ntiles;        // bx*by*bz
};

// What the kernels of a context tell the host while the stream runs: pinned
// host memory that the device writes and the host polls. A device-to-host copy
// and a stream synchronisation in its place left the GPU idle for 25-40 us each
// (64^3 dam break), against 5-8 us for a posted write and the next launch.
struct Mailbox {
  unsigned long long progress;  // PROGRESS_* of the solve loop
  double rmax;                  // ||r||_inf that belongs to it (k_update_xr only)
  double norms[4];              // k_residual64: ||r||inf, ||r||^2, ||b||inf, ||b||^2
  long long unknowns;           // k_pool_scan: unknowns, tiles and macro tiles that hold any
  int tiles, macro_tiles;
  int wave_error;               // a bounded wait gave up, as of the last k_residual64
  unsigned seq;                 // number of the last report of norms or counts
};
// progress: iterations completed (low 32 bits), SolverState::done, flags
constexpr int kProgressDone = 32;                        // 8 bits
constexpr unsigned long long kProgressWaveError = 1ull << 40;
constexpr unsigned long long kProgressNan = 1ull << 41;  // status < 0

// Device-resident solver scalars. Kernels read alpha/beta from here so the
// host never waits inside an iteration; once `done` is set the remaining
// launched iterations return at once.
struct SolverState {
  double rho;              // z.r of the current iterate
  double rho_new;
  double pq;               // p.Ap
  double alpha, beta;
  double rmax;             // ||r||_inf (recursive residual)
  double rmax0;            // ||b||_inf
  double r2;               // ||r||_2^2
  double tol_abs;          // tol * ||b||_inf
  double ru_threshold;     // request an FP64 residual replacement below this ||r||inf
  int iter;                // iterations completed
  int done;                // 1 = converged, 2 = max iterations, 3 = breakdown, 4 = replace residual
  int status;              // 0 ok, <0 error (wait timeout, NaN)
  int x_pending;           // the fused iteration's x += alpha p has not been applied yet
  Mailbox *mail;           // where the kernels report progress (null: nowhere)
  const void *waves;       // the context's wave-sync words, whose errors are reported with it
};

// A kernel launched by launch_overlapped may start while the kernel before it
// in the stream runs: it reads and writes global memory only after
// wait_for_previous, which returns once that kernel (and so, kernel by kernel,
// everything before it) is complete and its writes are visible.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Block-wide sum of one double; every thread gets the result.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *smem) {
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) smem[w] = v;
  __syncthreads();
  double s = 0.0;
  #pragma unroll
  for (int i = 0; i < NT / 32; ++i) s += smem[i];
  return s;
}

template <int NT>
__device__ __forceinline__ double block_max(double v, double *smem) {
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) smem[w] = v;
  __syncthreads();
  double s = 0.0;
  #pragma unroll
  for (int i = 0; i < NT / 32; ++i) s = fmax(s, smem[i]);
  return s;
}

// Launch of a kernel that begins with wait_for_previous. Its blocks take the
// place of the previous kernel's as those finish, instead of 2.5 us after the
// last one: a 64^3 dam break 2.41 -> 2.16 ms a projection, a 256^3 tank 65.8 ->
// 64.4. (With an explicit launch_dependents at the top of the iteration's
// kernels, 2.20 and 69: early blocks of the sweeps are in the stencil's way.)
// Such a kernel's pointer parameters are not __restrict__: the promise would
// cover the time before wait_for_previous returns, when the previous kernel is
// still writing what they point to, and let loads be moved above it.
template <class... P, class... A>
inline void launch_overlapped(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace shkz

#define SHKZ_CUDA_TRY(expr)                                       \
  do {                                                            \
    cudaError_t _e = (expr);                                      \
    if (_e != cudaSuccess) {                                      \
      shkz_set_cuda_error(_e, #expr, __FILE__, __LINE__);         \
      return SHKZ_B200_ERR_CUDA;                                  \
    }                                                             \
  } while (0)

void shkz_set_cuda_error(cudaError_t e, const char *expr, const char *file, int line);

// Number of kernels this library has launched (host-side count, all threads).
namespace shkz {
void count_launches(int n);
long long launches_so_far();
}
