// Residual and componentwise backward error of a sparse solve (internal to the library; used by the
// transient driver's checked solves, include/xyce_rf.h).
#pragma once

#include <cuda_runtime.h>

// A's CSR pattern (borrowed device arrays) and the plan of its long rows.
constexpr int kResidualStatus = 3;  // status words a check can bring along
struct XdResidual {
  int n = 0;
  const int *d_rowptr = nullptr, *d_colind = nullptr;
  int nlong = 0, nseg = 0;
  int *d_long = nullptr;                  // [nlong] long rows
  int *d_lseg = nullptr;                  // [nlong + 1] their segments
  int2 *d_seg = nullptr;                  // [nseg] entry range of each segment
  double *d_part = nullptr;               // [2 nseg] the segments' sums
  unsigned long long *d_acc = nullptr;    // {largest error, entries of x that are not finite, blocks done}
  double *h_out = nullptr;                // pinned: error, entries of x not finite, then status words
};

int xd_residual_init(XdResidual *r, int n, const int *rowptr, const int *d_rowptr, const int *d_colind);
void xd_residual_free(XdResidual *r);
// d_r = b - A x; h_out[0] = max_i |r_i| / max((|A| |x| + |b|)_i, 1e-300), 0 where r_i is 0 (NaN when any
// is), h_out[1] = the number of entries of x that are not finite, h_out[2 + q] = status[q] for q <
// nstatus (status may be null). Stream-ordered: h_out is the host's after the stream is synchronised.
int xd_residual_check(XdResidual *r, const double *d_vals, const double *d_b, const double *d_x, double *d_r,
                      const int *d_status, int nstatus, cudaStream_t st);
// d_x += d_d
int xd_residual_add(XdResidual *r, double *d_x, const double *d_d, cudaStream_t st);
