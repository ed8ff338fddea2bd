// The check after a sparse solve, in one launch: r = b - A x, the componentwise backward error and
// whether x is finite, written to pinned host memory. As separate products, absolute values,
// quotients and reductions it was about 25 launches and four synchronisations per Newton iteration,
// longer on the host than the factorization and the solves on the device: a step of the 20,000-MOSFET
// placed netlist (40,700 unknowns) took 3.5 ms with them and takes 2.5 ms with this (15 us of it).
//
// What bounds it is one pass over A's values and columns (a gather of x from L2). Eight lanes to a
// row, as the rows of circuit matrices have 3 to 12 entries; a supply node's row has an entry per
// device, so rows above kLongRow go to blocks of kSegment entries each, and the block that finishes
// last adds their sums in order. The largest error is taken over the bits of non-negative doubles
// (NaN above infinity above the rest), so the result does not depend on the order of the blocks.
#include "residual.h"

#include <algorithm>
#include <string>
#include <vector>

int xd_internal_fail(int code, const std::string &msg);

namespace {

constexpr int kBlock = 256;
constexpr int kLanes = 8;
constexpr int kLongRow = 128;
constexpr int kSegment = 1024;
static_assert(kSegment == 4 * kBlock, "a thread takes four entries of a segment");

__device__ __forceinline__ unsigned long long error_bits(double r, double den) {
  if (r == 0.0) return 0ull;
  const double d = den < 1e-300 ? 1e-300 : den;
  return (unsigned long long)__double_as_longlong(fabs(r) / d) & 0x7fffffffffffffffull;
}

__device__ __forceinline__ unsigned long long block_max(unsigned long long v, unsigned long long *red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[threadIdx.x & (kBlock / 32 - 1)];
#pragma unroll
  for (int off = kBlock / 64; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

__global__ void __launch_bounds__(kBlock) residual_check_kernel(XdResidual p, const double *__restrict__ vals,
                                                                const double *__restrict__ b,
                                                                const double *__restrict__ x, double *__restrict__ r,
                                                                const int *__restrict__ status, int nstatus) {
  __shared__ unsigned long long red[kBlock / 32];
  __shared__ double sums[2][kBlock / 32];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31;
  unsigned long long worst = 0;
  if ((int)blockIdx.x < p.nseg) {
    const int2 seg = p.d_seg[blockIdx.x];
    int col[4];
    double v[4], s = 0.0, a = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = seg.x + q * kBlock + tid;
      col[q] = k < seg.y ? p.d_colind[k] : -1;
      v[q] = k < seg.y ? vals[k] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (col[q] < 0) continue;
      const double t = v[q] * x[col[q]];
      s += t;
      a += fabs(t);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, off);
      a += __shfl_xor_sync(0xffffffffu, a, off);
    }
    if (lane == 0) {
      sums[0][tid >> 5] = s;
      sums[1][tid >> 5] = a;
    }
    __syncthreads();
    if (tid < 2) {
      double t = 0.0;
      for (int w = 0; w < kBlock / 32; ++w) t += sums[tid][w];
      p.d_part[2 * blockIdx.x + tid] = t;
    }
  } else {
    const int row = ((int)blockIdx.x - p.nseg) * (kBlock / kLanes) + tid / kLanes, sub = tid & (kLanes - 1);
    int k = 0, end = 0;
    if (row < p.n) {
      k = p.d_rowptr[row];
      end = p.d_rowptr[row + 1];
    }
    const bool mine = row < p.n && end - k <= kLongRow;
    double s = 0.0, a = 0.0;
    if (mine)
      for (k += sub; k < end; k += kLanes) {
        const double t = vals[k] * x[p.d_colind[k]];
        s += t;
        a += fabs(t);
      }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, off);
      a += __shfl_xor_sync(0xffffffffu, a, off);
    }
    if (sub == 0 && row < p.n) {
      if (!isfinite(x[row])) atomicAdd(&p.d_acc[1], 1ull);
      if (mine) {
        const double bi = b[row], ri = bi - s;
        r[row] = ri;
        worst = error_bits(ri, a + fabs(bi));
      }
    }
    worst = block_max(worst, red);
    if (tid == 0 && worst != 0) atomicMax(&p.d_acc[0], worst);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&p.d_acc[2], 1ull) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  worst = 0;
  for (int l = tid; l < p.nlong; l += kBlock) {
    const int row = p.d_long[l], q1 = p.d_lseg[l + 1];
    double s = 0.0, a = 0.0;
    for (int q = p.d_lseg[l]; q < q1; ++q) {
      s += __ldcg(p.d_part + 2 * q);
      a += __ldcg(p.d_part + 2 * q + 1);
    }
    const double bi = b[row], ri = bi - s;
    r[row] = ri;
    worst = max(worst, error_bits(ri, a + fabs(bi)));
  }
  worst = block_max(worst, red);
  if (tid == 0) {
    worst = max(worst, atomicAdd(&p.d_acc[0], 0ull));
    p.h_out[0] = __longlong_as_double((long long)worst);
    p.h_out[1] = (double)atomicAdd(&p.d_acc[1], 0ull);
    for (int q = 0; q < nstatus; ++q) p.h_out[2 + q] = (double)status[q];
    p.d_acc[0] = p.d_acc[1] = p.d_acc[2] = 0;
  }
}

__global__ void __launch_bounds__(kBlock) residual_add_kernel(int n, double *__restrict__ x,
                                                              const double *__restrict__ d) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i < n) x[i] = x[i] + d[i];
}

int fail(cudaError_t e, const char *where) {
  return xd_internal_fail(-3, std::string("CUDA error in ") + where + ": " + cudaGetErrorString(e));
}

}  // namespace

int xd_residual_init(XdResidual *r, int n, const int *rowptr, const int *d_rowptr, const int *d_colind) {
  r->n = n;
  r->d_rowptr = d_rowptr;
  r->d_colind = d_colind;
  std::vector<int> rows, lseg(1, 0);
  std::vector<int2> seg;
  for (int i = 0; i < n; ++i) {
    if (rowptr[i + 1] - rowptr[i] <= kLongRow) continue;
    rows.push_back(i);
    for (int k = rowptr[i]; k < rowptr[i + 1]; k += kSegment)
      seg.push_back(make_int2(k, std::min(rowptr[i + 1], k + kSegment)));
    lseg.push_back((int)seg.size());
  }
  r->nlong = (int)rows.size();
  r->nseg = (int)seg.size();
  const size_t nl = std::max<size_t>(1, rows.size()), ns = std::max<size_t>(1, seg.size());
  cudaError_t e;
  if ((e = cudaMalloc(&r->d_long, sizeof(int) * nl)) != cudaSuccess ||
      (e = cudaMalloc(&r->d_lseg, sizeof(int) * (nl + 1))) != cudaSuccess ||
      (e = cudaMalloc(&r->d_seg, sizeof(int2) * ns)) != cudaSuccess ||
      (e = cudaMalloc(&r->d_part, sizeof(double) * 2 * ns)) != cudaSuccess ||
      (e = cudaMalloc(&r->d_acc, sizeof(unsigned long long) * 3)) != cudaSuccess ||
      (e = cudaMemset(r->d_acc, 0, sizeof(unsigned long long) * 3)) != cudaSuccess ||
      (e = cudaMemcpy(r->d_long, rows.data(), sizeof(int) * rows.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(r->d_lseg, lseg.data(), sizeof(int) * lseg.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(r->d_seg, seg.data(), sizeof(int2) * seg.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaHostAlloc(&r->h_out, sizeof(double) * (2 + kResidualStatus), cudaHostAllocPortable)) != cudaSuccess) {
    xd_residual_free(r);
    return fail(e, "the residual check's set-up");
  }
  return 0;
}

void xd_residual_free(XdResidual *r) {
  cudaFree(r->d_long);
  cudaFree(r->d_lseg);
  cudaFree(r->d_seg);
  cudaFree(r->d_part);
  cudaFree(r->d_acc);
  if (r->h_out) cudaFreeHost(r->h_out);
  *r = XdResidual();
}

int xd_residual_check(XdResidual *r, const double *d_vals, const double *d_b, const double *d_x, double *d_r,
                      const int *d_status, int nstatus, cudaStream_t st) {
  const int rows = kBlock / kLanes, blocks = r->nseg + (r->n + rows - 1) / rows;
  residual_check_kernel<<<blocks, kBlock, 0, st>>>(*r, d_vals, d_b, d_x, d_r, d_status, d_status ? nstatus : 0);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : fail(e, "residual_check_kernel launch");
}

int xd_residual_add(XdResidual *r, double *d_x, const double *d_d, cudaStream_t st) {
  residual_add_kernel<<<(r->n + kBlock - 1) / kBlock, kBlock, 0, st>>>(r->n, d_x, d_d);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : fail(e, "residual_add_kernel launch");
}
