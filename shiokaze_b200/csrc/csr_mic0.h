// MIC(0) on a generic CSR matrix (csr_mic0.cu).
#pragma once
#include "common.cuh"
#include "../../include/shkz_b200.h"

#include <vector>

namespace shkz {

struct CsrMicDevice {
  int n;
  const int *colstart, *rowindex;                 // L by column: rows right of the diagonal
  double *val, *invdiag, *adiag;
  const int *lrow_start, *lrow_col, *lrow_pos;    // L by row: columns k < j and positions in column k
  const int *a_ptr, *a_idx;                       // A's pattern (CSR)
};

class CsrMic0 {
 public:
  ~CsrMic0();
  // Pattern analysis (0-based; on the device for sorted rows and a symmetric
  // pattern, else on the host); d_indptr/d_indices: the same pattern on the
  // device (kept by the caller).
  int build(int n, long long nnz, const int *indptr, const int *indices, const int *d_indptr, const int *d_indices,
            cudaStream_t s);
  // Factor the values of A (device, CSR order) with the header's parameters.
  int factor(const double *d_data, double omega, double min_ratio, cudaStream_t s);
  // z = (L L^T)^-1 r (z must not alias r); every launch returns at once
  // while *done != 0
  int apply(const double *r, double *z, cudaStream_t s, const int *done = nullptr);
  // SHKZ_B200_ERR_TIMEOUT when a wait of the factorisation or of a triangular
  // solve since it ran out
  int wait_error(cudaStream_t s) const;
  // polling rounds of each wait in the factorisation and the triangular solves
  void set_wait_limit(int limit) { wait_limit = limit; }
  // fault injection for tests: the forward solve's row at level-order
  // position pos (-1: none) never stores its value
  void set_fault_skip(int pos) { skip_pos = pos; }
  // the same for the factorisation: the column there never says it is done
  void set_fault_skip_column(int pos) { skip_column = pos; }
  int levels() const { return nlev; }

 private:
  static constexpr int kNotSymmetric = 1;
  void release();
  bool allocate(long long entries);
  int build_device(long long nnz, cudaStream_t s);
  int build_host(const int *indptr, const int *indices, cudaStream_t s);
  CsrMicDevice device() const;
  int n = 0, nnzl = 0, nlev = 0, wait_limit = 1 << 22, skip_pos = -1, skip_column = -1;
  char *arena = nullptr;  // holds all of the following
  int *d_colstart = nullptr, *d_rowindex = nullptr, *d_lrow_start = nullptr, *d_lrow_col = nullptr,
      *d_lrow_pos = nullptr, *d_src = nullptr, *d_dpos = nullptr, *d_cols = nullptr, *d_chunks = nullptr;
  int *d_ready = nullptr;  // levels, then the factorisation's flags
  int *d_count = nullptr, *d_chunk = nullptr, *d_sums = nullptr;  // scratch of the analysis
  int *d_sync = nullptr;  // two chunk counters, the wait error word, the factorisation's counter, the analysis' results
  int *d_nchunks = nullptr;
  double *d_val = nullptr, *d_invdiag = nullptr, *d_adiag = nullptr, *d_t = nullptr;
  const int *a_ptr = nullptr, *a_idx = nullptr;
};

}  // namespace shkz
