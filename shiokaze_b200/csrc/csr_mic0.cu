// MIC(0) preconditioner for the generic CSR solver path (LinSolver=pcg_b200
// with B200.Preconditioner=mic0): the reference header's own factorisation
// and triangular solves (local/include/pcgsolver/pcg_solver.h:88-223) on the
// device, for any symmetric row-sorted CSR matrix.
//
// The lower factor L keeps A's lower pattern, stored by column as the header
// stores it (column i = row i's entries right of the diagonal). The
// factorisation is left-looking: column j takes the update of every column
// k < j with L(j,k) != 0, in increasing k, exactly the updates (and their
// order) the header's right-looking loop applies to it, then is finalised.
// Columns are grouped into levels (level(j) = 1 + the largest level of its
// k's). The factorisation and the triangular solves run column- or row-wise in
// one launch each: warps take chunks of up to 32 rows of one level from an
// atomic counter in level order (reverse order for the transpose solve), and
// a row waits for each row it depends on until the warp that owns that one has
// stored it. Each row's subtractions keep the header's order. Every product
// and sum is rounded on its own (no fused multiply-add), as the host code the
// header compiles to computes them.
//
// The pattern is analysed on the device when it is that of a symmetric matrix
// with sorted rows (k_pattern_*), else on the host with the same outcome
// for what the header reads. On the host it took 5 to 6 ms of a 48^3 7-point
// solve's 31, and a launch per level of the factorisation 2 ms.
#include "common.cuh"
#include "kernels.h"
#include "csr_mic0.h"

#include <algorithm>
#include <vector>

namespace shkz {

__global__ void k_csrmic_init(int nnzl, const int *__restrict__ src, int n, const int *__restrict__ dpos,
                              const double *__restrict__ data, double *val, double *invdiag, double *adiag) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nnzl; p += gridDim.x * blockDim.x) val[p] = data[src[p]];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double a = dpos[i] >= 0 ? data[dpos[i]] : 0.0;
    invdiag[i] = a;
    adiag[i] = a;
  }
}

// factor_modified_incomplete_cholesky0 (pcg_solver.h:122-189): all updates into
// column j, then its finalisation. Columns of one chunk are of one level and
// wait only for columns of earlier chunks, as in the triangular solves. What
// does not change is read before the wait and the columns' values after it all
// at once (past L1, where a line may predate them), four columns of four
// entries at a time. 142 levels of a 48^3 7-point system: 1.45 ms; 4.76 with
// the values read where the loops come to them, 2.06 with a launch a level.
constexpr int kFactorCols = 4, kFactorEntries = 4;

__device__ __forceinline__ int load_flag(const int *p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__global__ void __launch_bounds__(128) k_csrmic_factor(CsrMicDevice M, const int *__restrict__ cols,
                                                       const int *__restrict__ chunks, const int *__restrict__ nchunks,
                                                       double omega, double min_ratio, int *ready, unsigned *counter,
                                                       int *err, int limit, int skip) {
  const int lane = threadIdx.x & 31, total = *nchunks;
  while (true) {
    int chunk = 0;
    if (lane == 0) chunk = (int)atomicAdd(counter, 1u);
    chunk = __shfl_sync(0xffffffffu, chunk, 0);
    if (chunk >= total) return;
    const int first = chunks[chunk], count = chunks[chunk + 1] - first;
    if (lane >= count) continue;
    const int j = cols[first + lane];
    const int jb = M.colstart[j], je = M.colstart[j + 1];
    const int ab = M.a_ptr[j], ae = M.a_ptr[j + 1];
    const int q1 = M.lrow_start[j + 1];
    const double ad = M.adiag[j];
    double inv = M.invdiag[j];
    asm volatile("prefetch.global.L1 [%0];" ::"l"(M.a_idx + ab));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(M.rowindex + jb));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(M.val + jb));
    for (int q0 = M.lrow_start[j]; q0 < q1; q0 += kFactorCols) {
      int col[kFactorCols], kb[kFactorCols], ke[kFactorCols], ri[kFactorCols][kFactorEntries];
      const double *mp[kFactorCols];
      double kd[kFactorCols];
      #pragma unroll
      for (int u = 0; u < kFactorCols; ++u) {
        const bool has = q0 + u < q1;
        col[u] = has ? M.lrow_col[q0 + u] : -1;
        mp[u] = has ? M.val + M.lrow_pos[q0 + u] : M.val;
        kb[u] = has ? M.colstart[col[u]] : 0;
        ke[u] = has ? M.colstart[col[u] + 1] : 0;
        kd[u] = has ? M.adiag[col[u]] : 0.0;
        #pragma unroll
        for (int e = 0; e < kFactorEntries; ++e) ri[u][e] = kb[u] + e < ke[u] ? M.rowindex[kb[u] + e] : 0;
      }
      for (int it = 0;; ++it) {
        bool pending = false;
        #pragma unroll
        for (int u = 0; u < kFactorCols; ++u) pending |= col[u] >= 0 && load_flag(ready + col[u]) == 0;
        if (!pending) break;
        if (it >= limit) {
          atomicExch(err, 1);
          break;
        }
        __nanosleep(32);
      }
      __threadfence();  // the columns' values after their flags
      double mult[kFactorCols], v[kFactorCols][kFactorEntries];
      #pragma unroll
      for (int u = 0; u < kFactorCols; ++u) {
        mult[u] = col[u] >= 0 ? __ldcg(mp[u]) : 0.0;
        #pragma unroll
        for (int e = 0; e < kFactorEntries; ++e) v[u][e] = kb[u] + e < ke[u] ? __ldcg(M.val + kb[u] + e) : 0.0;
      }
      #pragma unroll
      for (int u = 0; u < kFactorCols; ++u) {
        if (col[u] < 0 || kd[u] == 0.0) continue;  // a null column eliminates nothing
        double missing = 0.0;
        int b = ab, c = jb;
        // column k's entries in order of their rows
        auto entry = [&](int ra, double va) {
          if (ra < j) {
            // dropped when A's row j does not have it (pcg_solver.h:140-155)
            while (b < ae && M.a_idx[b] < ra) ++b;
            if (b < ae && M.a_idx[b] != ra) missing = __dadd_rn(missing, va);
          } else if (ra == j) {
            inv = __dsub_rn(inv, __dmul_rn(mult[u], va));
          } else {
            // eliminate into column j's entries below the diagonal (pcg_solver.h:160-176)
            while (c < je && M.rowindex[c] < ra) ++c;
            if (c < je && M.rowindex[c] == ra) {
              M.val[c] = __dsub_rn(M.val[c], __dmul_rn(mult[u], va));
              ++c;
            } else {
              missing = __dadd_rn(missing, va);
            }
          }
        };
        #pragma unroll
        for (int e = 0; e < kFactorEntries; ++e)
          if (kb[u] + e < ke[u]) entry(ri[u][e], v[u][e]);
        for (int a = kb[u] + kFactorEntries; a < ke[u]; ++a) entry(M.rowindex[a], __ldcg(M.val + a));
        inv = __dsub_rn(inv, __dmul_rn(__dmul_rn(omega, mult[u]), missing));
      }
    }
    // finalise column j (pcg_solver.h:126-135)
    if (ad != 0.0) {
      inv = inv < __dmul_rn(min_ratio, ad) ? __ddiv_rn(1.0, __dsqrt_rn(ad)) : __ddiv_rn(1.0, __dsqrt_rn(inv));
      for (int p = jb; p < je; ++p) M.val[p] = __dmul_rn(M.val[p], inv);
    }
    M.invdiag[j] = inv;
    __threadfence();
    // fault injection (tests only): the column at level-order position skip
    // never says that it is done, so the waits on it run out
    if (first + lane != skip) asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(ready + j), "r"(1) : "memory");
  }
}

// Sync-free triangular solves. Output values start as a signalling-NaN
// pattern that no arithmetic produces; a 64-bit store of the final value is
// single-copy atomic, so the value is its own ready flag. A chunk holds rows
// of one level and waits only on rows of earlier chunks, which warps that are
// already running hold, so every wait ends; each is still bounded, and on
// expiry the row stores a quiet NaN (its dependants then finish at once and
// the solve's NaN check stops it) and sets the error word.
constexpr unsigned long long kPending = 0x7ff4000000000001ull;
constexpr int kSolveWarpsPerSm = 8;

__device__ __forceinline__ double poll_value(const double *p, int limit, int *err) {
  unsigned long long w;
  for (int it = 0;; ++it) {
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    if (w != kPending) return __longlong_as_double((long long)w);
    if (it >= limit) {
      atomicExch(err, 1);
      return __longlong_as_double(0x7ff8000000000000ll);
    }
    __nanosleep(32);
  }
}

__device__ __forceinline__ void store_value(double *p, double v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(__double_as_longlong(v)) : "memory");
}

// both solves' outputs to pending, both chunk counters to zero
__global__ void k_csrmic_pending(int n, double *t, double *z, unsigned *counters, const int *done) {
  if (done && *done) return;
  const double pend = __longlong_as_double((long long)kPending);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    t[i] = pend;
    z[i] = pend;
  }
  if (blockIdx.x == 0 && threadIdx.x < 2) counters[threadIdx.x] = 0;
}

__device__ __forceinline__ unsigned long long load_word(const double *p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}

// s - sum_q val[pos(q)] * x[col(q)] over q in [q0, q1), in q order. The first
// kDepBatch values are loaded together and re-polled together until none is
// pending, so a row waits about one L2 round trip once its dependencies are
// stored; any further ones are polled one by one.
constexpr int kDepBatch = 8;
template <class Col, class Pos>
__device__ __forceinline__ double row_update(double s, int q0, int q1, const double *x, const double *val, Col col,
                                             Pos pos, int limit, int *err) {
  // the entries' places and values first: nothing but the poll and the
  // arithmetic is then left between a dependency's store and this row's
  // (48^3 7-point system, 284 levels both ways: 580 -> 290 us an application,
  // 268 with the rows of a level in order)
  const double *at[kDepBatch];
  double v[kDepBatch];
  unsigned long long w[kDepBatch];
  #pragma unroll
  for (int k = 0; k < kDepBatch; ++k) {
    at[k] = q0 + k < q1 ? x + col(q0 + k) : nullptr;
    v[k] = q0 + k < q1 ? val[pos(q0 + k)] : 0.0;
  }
  #pragma unroll
  for (int k = 0; k < kDepBatch; ++k) w[k] = at[k] ? load_word(at[k]) : 0ull;
  for (int it = 0;; ++it) {
    bool pending = false;
    #pragma unroll
    for (int k = 0; k < kDepBatch; ++k) pending |= w[k] == kPending;
    if (!pending) break;
    if (it >= limit) {
      atomicExch(err, 1);
      #pragma unroll
      for (int k = 0; k < kDepBatch; ++k)
        if (w[k] == kPending) w[k] = 0x7ff8000000000000ull;
      break;
    }
    __nanosleep(32);
    #pragma unroll
    for (int k = 0; k < kDepBatch; ++k)
      if (w[k] == kPending) w[k] = load_word(at[k]);
  }
  #pragma unroll
  for (int k = 0; k < kDepBatch; ++k)
    if (at[k]) s = __dsub_rn(s, __dmul_rn(v[k], __longlong_as_double((long long)w[k])));
  for (int q = q0 + kDepBatch; q < q1; ++q) s = __dsub_rn(s, __dmul_rn(val[pos(q)], poll_value(x + col(q), limit, err)));
  return s;
}

// solve_lower (pcg_solver.h:195-209): y[r] = (b[r] - sum_k L(r,k) y[k]) * invdiag[r]
__global__ void __launch_bounds__(128) k_csrmic_lower_sf(CsrMicDevice M, const int *__restrict__ cols,
                                                         const int *__restrict__ chunks, const int *__restrict__ nchunks_p,
                                                         const double *__restrict__ b, double *y, unsigned *counter,
                                                         int *err, int limit, const int *done, int skip) {
  if (done && *done) return;
  const int lane = threadIdx.x & 31, nchunks = *nchunks_p;
  while (true) {
    int c = 0;
    if (lane == 0) c = (int)atomicAdd(counter, 1u);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= nchunks) return;
    const int first = chunks[c], count = chunks[c + 1] - first;
    if (lane < count) {
      const int r = cols[first + lane];
      const double inv = M.invdiag[r];
      const double s = row_update(
          b[r], M.lrow_start[r], M.lrow_start[r + 1], y, M.val, [&](int q) { return M.lrow_col[q]; },
          [&](int q) { return M.lrow_pos[q]; }, limit, err);
      // fault injection (tests only): the row at level-order position skip
      // never stores, so the waits on it run out
      if (first + lane != skip) store_value(y + r, __dmul_rn(s, inv));
    }
  }
}

// solve_lower_transpose_in_place (pcg_solver.h:211-223), out of place:
// z[i] = (t[i] - sum L(r,i) z[r]) * invdiag[i], chunks in reverse level order
__global__ void __launch_bounds__(128) k_csrmic_upper_sf(CsrMicDevice M, const int *__restrict__ cols,
                                                         const int *__restrict__ chunks, const int *__restrict__ nchunks_p,
                                                         const double *__restrict__ t, double *z, unsigned *counter,
                                                         int *err, int limit, const int *done) {
  if (done && *done) return;
  const int lane = threadIdx.x & 31, nchunks = *nchunks_p;
  while (true) {
    int c = 0;
    if (lane == 0) c = (int)atomicAdd(counter, 1u);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= nchunks) return;
    c = nchunks - 1 - c;
    const int first = chunks[c], count = chunks[c + 1] - first;
    if (lane < count) {
      const int i = cols[first + lane];
      const double inv = M.invdiag[i];
      const double s = row_update(
          t[i], M.colstart[i], M.colstart[i + 1], z, M.val, [&](int p) { return M.rowindex[p]; },
          [](int p) { return p; }, limit, err);
      store_value(z + i, __dmul_rn(s, inv));
    }
  }
}

static int solve_blocks() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms * kSolveWarpsPerSm / 4;
}

// ---------------------------------------------------------------------------
// Pattern analysis on the device. meta: 0 the pattern is not of the kind
// handled here, 1 levels, 2 entries of L, 3 chunks.
enum { META_REFUSED = 0, META_LEVELS = 1, META_ENTRIES = 2, META_CHUNKS = 3 };

// entries left and right of the diagonal, and the diagonal, of each row
__global__ void k_pattern_rows(int n, const int *__restrict__ ap, const int *__restrict__ ai, int *right, int *left,
                               int *dpos, int *meta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  int l = 0, r = 0, d = -1;
  if (i < n) {
    int last = -1;
    for (int p = ap[i]; p < ap[i + 1]; ++p) {
      const int k = ai[p];
      if (k <= last || k >= n) meta[META_REFUSED] = 1;
      last = k;
      l += k < i;
      r += k > i;
      if (k == i) d = p;
    }
    dpos[i] = d;
  }
  right[i] = r;
  left[i] = l;
}

// L by column and by row. Row j of L is A's row j left of the diagonal; where
// such an entry k sits in column k is found in A's row k, and if it always is
// and there are as many entries right of the diagonal, the pattern is symmetric.
__global__ void k_pattern_fill(int n, int room, const int *__restrict__ ap, const int *__restrict__ ai,
                               const int *__restrict__ dpos, const int *__restrict__ colstart,
                               const int *__restrict__ lrow_start, int *rowindex, int *src, int *lrow_col,
                               int *lrow_pos, int *meta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (i == 0) {
    meta[META_ENTRIES] = colstart[n];
    if (colstart[n] != lrow_start[n] || colstart[n] > room) meta[META_REFUSED] = 1;
  }
  if (meta[META_REFUSED] || colstart[n] > room || lrow_start[n] > room) return;
  const int l0 = lrow_start[i], l = lrow_start[i + 1] - l0, a0 = ap[i];
  for (int q = 0; q < l; ++q) {
    const int k = ai[a0 + q];
    // row k's entries right of its diagonal
    int lo = ap[k] + (lrow_start[k + 1] - lrow_start[k]) + (dpos[k] >= 0), hi = ap[k + 1];
    const int first = lo;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (ai[mid] < i) lo = mid + 1;
      else hi = mid;
    }
    if (lo >= ap[k + 1] || ai[lo] != i) meta[META_REFUSED] = 1;
    lrow_col[l0 + q] = k;
    lrow_pos[l0 + q] = colstart[k] + (lo - first);
  }
  const int r0 = colstart[i], r = colstart[i + 1] - r0, b0 = ap[i + 1] - r;
  for (int q = 0; q < r; ++q) {
    rowindex[r0 + q] = ai[b0 + q];
    src[r0 + q] = b0 + q;
  }
}

// Levels in one launch: warps take 32 rows at a time in order; a lane looks at
// what its row depends on without blocking the warp's other rows, on some of
// which it may depend. Rows are taken in order, so the lowest unfinished one
// can always finish.
__global__ void __launch_bounds__(128) k_pattern_levels(int n, const int *__restrict__ lrow_start,
                                                        const int *__restrict__ lrow_col, int *level, unsigned *counter,
                                                        int limit, int *meta) {
  if (meta[META_REFUSED]) return;
  const int lane = threadIdx.x & 31;
  while (true) {
    unsigned c = 0;
    if (lane == 0) c = atomicAdd(counter, 32u);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= (unsigned)n) return;
    const int j = (int)c + lane;
    bool open = j < n;
    int q = open ? lrow_start[j] : 0, l = 0;
    const int end = open ? lrow_start[j + 1] : 0;
    for (int it = 0; __any_sync(0xffffffffu, open); ++it) {
      if (!open) continue;
      while (q < end) {
        int v;
        asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(level + lrow_col[q]) : "memory");
        if (v < 0) break;
        l = max(l, v + 1);
        ++q;
      }
      if (q < end && it >= limit) {  // gave up: the host analyses the pattern
        meta[META_REFUSED] = 1;
        q = end;
      }
      if (q == end) {
        asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(level + j), "r"(l) : "memory");
        open = false;
      }
    }
  }
}

__global__ void k_pattern_histogram(int n, const int *__restrict__ level, int *count, int *meta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int l = -1;
  if (i < n && !meta[META_REFUSED]) {
    l = level[i];
    atomicAdd(&count[l], 1);
  }
  l = __reduce_max_sync(0xffffffffu, l);
  if ((threadIdx.x & 31) == 0 && l >= 0) atomicMax(&meta[META_LEVELS], l + 1);
}

// chunks of up to 32 rows of one level: how many, then where they start
__global__ void k_pattern_chunk_count(int n, const int *__restrict__ count, int *chunk) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l <= n) chunk[l] = (count[l] + 31) / 32;
}
__global__ void k_pattern_chunks(int n, const int *__restrict__ start, const int *__restrict__ chunk, int *chunks,
                                 int *meta) {
  const int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (l >= meta[META_LEVELS]) return;
  for (int c = chunk[l] + lane; c < chunk[l + 1]; c += 32) chunks[c] = start[l] + 32 * (c - chunk[l]);
  if (l == meta[META_LEVELS] - 1 && lane == 0) {
    chunks[chunk[l + 1]] = n;
    meta[META_CHUNKS] = chunk[l + 1];
  }
}
__global__ void k_pattern_order(int n, const int *__restrict__ level, int *cursor, int *cols, const int *meta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && !meta[META_REFUSED]) cols[atomicAdd(&cursor[level[i]], 1)] = i;
}

// Rows of a level in increasing order, as neighbours in a chunk then are in the
// arrays: one block a level, a bitonic network over up to kSortRows rows. The
// order inside a level changes no result; larger levels keep the one they
// have. 48^3 7-point system: a solve pair 268 us, 315 in order of arrival.
constexpr int kSortRows = 8192;
__global__ void __launch_bounds__(512) k_pattern_sort(int nlev, const int *__restrict__ end, int *cols) {
  __shared__ int v[kSortRows];
  for (int l = blockIdx.x; l < nlev; l += gridDim.x) {
    // the cursors of k_pattern_order stand at the levels' ends
    const int first = l > 0 ? end[l - 1] : 0, count = end[l] - first;
    if (count > kSortRows || count < 2) continue;
    int size = 2;
    while (size < count) size *= 2;
    for (int i = threadIdx.x; i < size; i += blockDim.x) v[i] = i < count ? cols[first + i] : INT32_MAX;
    for (int k = 2; k <= size; k *= 2)
      for (int d = k / 2; d > 0; d /= 2) {
        __syncthreads();
        for (int i = threadIdx.x; i < size / 2; i += blockDim.x) {
          const int a = 2 * i - (i & (d - 1)), b = a + d;
          const int x = v[a], y = v[b];
          if ((x > y) == ((a & k) == 0)) {
            v[a] = y;
            v[b] = x;
          }
        }
      }
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += blockDim.x) cols[first + i] = v[i];
    __syncthreads();
  }
}

CsrMic0::~CsrMic0() { release(); }

void CsrMic0::release() {
  if (arena) cudaFree(arena);
  arena = nullptr;
}

// One allocation for everything, with room for `entries` of L.
bool CsrMic0::allocate(long long entries) {
  release();
  size_t at = 0;
  auto place = [&](size_t bytes) {
    const size_t p = at;
    at += (bytes + 255) & ~(size_t)255;
    return p;
  };
  const size_t N = (size_t)n, H = (size_t)std::max(1ll, entries);
  const size_t o_val = place(8 * H), o_inv = place(8 * N), o_ad = place(8 * N), o_t = place(8 * N);
  const size_t o_col = place(4 * (N + 1)), o_row = place(4 * H), o_ls = place(4 * (N + 1)), o_lc = place(4 * H),
               o_lp = place(4 * H), o_src = place(4 * H), o_dp = place(4 * N), o_cols = place(4 * N),
               o_ch = place(4 * (N + 1)), o_ready = place(4 * N), o_cnt = place(4 * (N + 1)), o_cc = place(4 * (N + 1)),
               o_sums = place(4 * (scan_tile_count((long long)N + 1) + 1)), o_sync = place(64);
  if (cudaMalloc((void **)&arena, at) != cudaSuccess) {
    arena = nullptr;
    return false;
  }
  auto I = [&](size_t o) { return reinterpret_cast<int *>(arena + o); };
  auto D = [&](size_t o) { return reinterpret_cast<double *>(arena + o); };
  d_val = D(o_val); d_invdiag = D(o_inv); d_adiag = D(o_ad); d_t = D(o_t);
  d_colstart = I(o_col); d_rowindex = I(o_row); d_lrow_start = I(o_ls); d_lrow_col = I(o_lc); d_lrow_pos = I(o_lp);
  d_src = I(o_src); d_dpos = I(o_dp); d_cols = I(o_cols); d_chunks = I(o_ch); d_ready = I(o_ready);
  d_count = I(o_cnt); d_chunk = I(o_cc); d_sums = I(o_sums); d_sync = I(o_sync);
  return true;
}

int CsrMic0::build(int n_, long long nnz, const int *indptr, const int *indices, const int *d_indptr,
                   const int *d_indices, cudaStream_t s) {
  n = n_;
  a_ptr = d_indptr;
  a_idx = d_indices;
  const int rc = build_device(nnz, s);
  return rc == kNotSymmetric ? build_host(indptr, indices, s) : rc;
}

int CsrMic0::build_device(long long nnz, cudaStream_t s) {
  if (n >= INT32_MAX - 1024) return kNotSymmetric;
  const int room = (int)(nnz / 2);
  if (!allocate(room)) return SHKZ_B200_ERR_NOMEM;
  int *meta = d_sync + 4;
  if (cudaMemsetAsync(d_sync, 0, 64, s) != cudaSuccess || cudaMemsetAsync(d_ready, 0xff, sizeof(int) * (size_t)n, s) != cudaSuccess ||
      cudaMemsetAsync(d_count, 0, sizeof(int) * ((size_t)n + 1), s) != cudaSuccess)
    return SHKZ_B200_ERR_CUDA;
  const int rows = (n + 255) / 256, rows1 = n / 256 + 1;
  int *level = d_ready;  // the factorisation's flags later
  count_launches(8);
  k_pattern_rows<<<rows1, 256, 0, s>>>(n, a_ptr, a_idx, d_colstart, d_lrow_start, d_dpos, meta);
  launch_exclusive_scan(d_colstart, (long long)n + 1, d_sums, s);
  launch_exclusive_scan(d_lrow_start, (long long)n + 1, d_sums, s);
  k_pattern_fill<<<rows, 256, 0, s>>>(n, room, a_ptr, a_idx, d_dpos, d_colstart, d_lrow_start, d_rowindex, d_src,
                                      d_lrow_col, d_lrow_pos, meta);
  k_pattern_levels<<<solve_blocks(), 128, 0, s>>>(n, d_lrow_start, d_lrow_col, level,
                                                  reinterpret_cast<unsigned *>(d_sync), 1 << 22, meta);
  k_pattern_histogram<<<rows, 256, 0, s>>>(n, level, d_count, meta);
  k_pattern_chunk_count<<<rows1, 256, 0, s>>>(n, d_count, d_chunk);
  launch_exclusive_scan(d_count, (long long)n + 1, d_sums, s);
  launch_exclusive_scan(d_chunk, (long long)n + 1, d_sums, s);
  k_pattern_chunks<<<(int)(((long long)n * 32 + 255) / 256), 256, 0, s>>>(n, d_count, d_chunk, d_chunks, meta);
  k_pattern_order<<<rows, 256, 0, s>>>(n, level, d_count, d_cols, meta);
  int h[4];
  if (cudaMemcpyAsync(h, meta, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return SHKZ_B200_ERR_CUDA;
  if (h[META_REFUSED]) return kNotSymmetric;
  nlev = h[META_LEVELS];
  nnzl = h[META_ENTRIES];
  d_nchunks = meta + META_CHUNKS;
  count_launches(1);
  k_pattern_sort<<<std::min(nlev, 148 * 4), 512, 0, s>>>(nlev, d_count, d_cols);
  return cudaGetLastError() == cudaSuccess ? 0 : SHKZ_B200_ERR_CUDA;
}

int CsrMic0::build_host(const int *indptr, const int *indices, cudaStream_t s) {
  // pattern of L by column (row i right of the diagonal) and of the diagonal
  std::vector<int> colstart(n + 1), rowindex, src, dpos(n, -1);
  for (int i = 0; i < n; ++i) {
    colstart[i] = (int)rowindex.size();
    for (int p = indptr[i]; p < indptr[i + 1]; ++p) {
      if (indices[p] > i) {
        rowindex.push_back(indices[p]);
        src.push_back(p);
      } else if (indices[p] == i) {
        dpos[i] = p;
      }
    }
  }
  colstart[n] = (int)rowindex.size();
  nnzl = colstart[n];
  // L by row: for row j the columns k < j with L(j,k) != 0, increasing k, and
  // where L(j,k) sits in column k
  std::vector<int> lrow_start(n + 1, 0), lrow_col(nnzl), lrow_pos(nnzl);
  for (int p = 0; p < nnzl; ++p) ++lrow_start[rowindex[p] + 1];
  for (int j = 0; j < n; ++j) lrow_start[j + 1] += lrow_start[j];
  {
    std::vector<int> cur(lrow_start.begin(), lrow_start.end() - 1);
    for (int k = 0; k < n; ++k)
      for (int p = colstart[k]; p < colstart[k + 1]; ++p) {
        const int j = rowindex[p];
        lrow_col[cur[j]] = k;
        lrow_pos[cur[j]] = p;
        ++cur[j];
      }
  }
  // levels: a column (row) after every column it depends on
  std::vector<int> level(n, 0);
  nlev = 0;
  for (int j = 0; j < n; ++j) {
    int l = 0;
    for (int q = lrow_start[j]; q < lrow_start[j + 1]; ++q) l = std::max(l, level[lrow_col[q]] + 1);
    level[j] = l;
    nlev = std::max(nlev, l + 1);
  }
  std::vector<int> level_start(nlev + 1, 0);
  for (int j = 0; j < n; ++j) ++level_start[level[j] + 1];
  for (int l = 0; l < nlev; ++l) level_start[l + 1] += level_start[l];
  std::vector<int> cols(n);
  {
    std::vector<int> cur(level_start.begin(), level_start.end() - 1);
    for (int j = 0; j < n; ++j) cols[cur[level[j]]++] = j;
  }
  // chunks of up to 32 rows, never across a level boundary
  std::vector<int> chunks;
  for (int l = 0; l < nlev; ++l)
    for (int q = level_start[l]; q < level_start[l + 1]; q += 32) chunks.push_back(q);
  chunks.push_back(n);
  const int nchunks = (int)chunks.size() - 1;
  if (!allocate(nnzl)) return SHKZ_B200_ERR_NOMEM;
  int *meta = d_sync + 4;
  d_nchunks = meta + META_CHUNKS;
  auto upload = [&](int *d, const std::vector<int> &h) -> bool {
    return h.empty() || cudaMemcpyAsync(d, h.data(), sizeof(int) * h.size(), cudaMemcpyHostToDevice, s) == cudaSuccess;
  };
  bool ok = cudaMemsetAsync(d_sync, 0, 64, s) == cudaSuccess && upload(d_colstart, colstart) &&
            upload(d_rowindex, rowindex) && upload(d_lrow_start, lrow_start) && upload(d_lrow_col, lrow_col) &&
            upload(d_lrow_pos, lrow_pos) && upload(d_src, src) && upload(d_dpos, dpos) && upload(d_cols, cols) &&
            upload(d_chunks, chunks) &&
            cudaMemcpyAsync(meta + META_CHUNKS, &nchunks, sizeof(int), cudaMemcpyHostToDevice, s) == cudaSuccess;
  // the host vectors must outlive the asynchronous uploads
  if (cudaStreamSynchronize(s) != cudaSuccess) ok = false;
  return ok ? 0 : SHKZ_B200_ERR_CUDA;
}

CsrMicDevice CsrMic0::device() const {
  CsrMicDevice M;
  M.n = n;
  M.colstart = d_colstart;
  M.rowindex = d_rowindex;
  M.val = d_val;
  M.invdiag = d_invdiag;
  M.adiag = d_adiag;
  M.lrow_start = d_lrow_start;
  M.lrow_col = d_lrow_col;
  M.lrow_pos = d_lrow_pos;
  M.a_ptr = a_ptr;
  M.a_idx = a_idx;
  return M;
}

int CsrMic0::factor(const double *d_data, double omega, double min_ratio, cudaStream_t s) {
  count_launches(1);
  k_csrmic_init<<<std::min((std::max(nnzl, n) + 255) / 256, 148 * 8) + 1, 256, 0, s>>>(nnzl, d_src, n, d_dpos, d_data,
                                                                                       d_val, d_invdiag, d_adiag);
  if (cudaMemsetAsync(d_ready, 0, sizeof(int) * (size_t)n, s) != cudaSuccess ||
      cudaMemsetAsync(d_sync, 0, sizeof(int) * 4, s) != cudaSuccess)
    return SHKZ_B200_ERR_CUDA;
  count_launches(1);
  k_csrmic_factor<<<solve_blocks(), 128, 0, s>>>(device(), d_cols, d_chunks, d_nchunks, omega, min_ratio, d_ready,
                                                 reinterpret_cast<unsigned *>(d_sync) + 3, d_sync + 2, wait_limit,
                                                 skip_column);
  return cudaGetLastError() == cudaSuccess ? 0 : SHKZ_B200_ERR_CUDA;
}

int CsrMic0::apply(const double *r, double *z, cudaStream_t s, const int *done) {
  const CsrMicDevice M = device();
  const int blocks = solve_blocks();
  unsigned *counters = reinterpret_cast<unsigned *>(d_sync);
  int *err = d_sync + 2;
  count_launches(3);
  k_csrmic_pending<<<std::max(1, std::min((n + 255) / 256, 148 * 8)), 256, 0, s>>>(n, d_t, z, counters, done);
  k_csrmic_lower_sf<<<blocks, 128, 0, s>>>(M, d_cols, d_chunks, d_nchunks, r, d_t, counters, err, wait_limit, done,
                                           skip_pos);
  k_csrmic_upper_sf<<<blocks, 128, 0, s>>>(M, d_cols, d_chunks, d_nchunks, d_t, z, counters + 1, err, wait_limit,
                                           done);
  return cudaGetLastError() == cudaSuccess ? 0 : SHKZ_B200_ERR_CUDA;
}

int CsrMic0::wait_error(cudaStream_t s) const {
  if (!arena) return 0;
  int e = 0;
  if (cudaMemcpyAsync(&e, d_sync + 2, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return SHKZ_B200_ERR_CUDA;
  return e ? SHKZ_B200_ERR_TIMEOUT : 0;
}

}  // namespace shkz
