// dst_mma.h -- the DST-I passes of the FP64 Dirichlet solves as integer
// products on the tensor cores (dst_mma.cu).
#pragma once
#include "vpmg_internal.h"

namespace vpmg {

// Whether `lines` lines of n points each, in nc components, go as products; once:
// with tables made for this call alone.
bool dst_mma_wanted(int n, long long lines, int nc, bool once);
// Tables of a line length's sine matrix, for plans with p.n points.
size_t dst_mma_table_bytes(int n);
struct DstTable {
  unsigned char* T;
  int n;
  double factor;  // in [1, 2)
};
void dst_mma_setup();  // once per device, outside stream capture
void dst_mma_tables(const DstTable* t, int count, cudaStream_t s);  // up to three, one launch
// Passes: lines of n points; nc components (strides in doubles).  A wait that
// runs out of polls makes the outputs NaN and *status (if any) kErrWait.
struct DstWait {
  int polls;
  int* status;
};
struct DstBox {
  int dims[3], o[3], m[3];
};
void dst_mma_x_fwd(const unsigned char* T, int shift, int neg, const double* rhs, const double* sol, bool zero_bc,
                   double* out, const DstBox& b, double ihx2, double ihy2, double ihz2, int nc, size_t rcs, size_t scs,
                   size_t ocs, const DstWait& w, cudaStream_t s);
void dst_mma_y(const unsigned char* T, const double* in, double* out, int m0, int m1, int m2, int nc, size_t cs,
               const DstWait& w, cudaStream_t s);
void dst_mma_x_inv(const unsigned char* T, const double* in, double* sol, const DstBox& b, int nc, size_t ics,
                   size_t scs, const DstWait& w, cudaStream_t s);

}  // namespace vpmg
