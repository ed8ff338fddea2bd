// Sparse LU refactorization over an elimination-tree plan (lutree.h).
//
// What bounds it is the longest chain of dependent pivots, not arithmetic or bytes: at 200k unknowns
// 12.6M updates (0.7 us of the FP64 pipe) and 15 MB of values, but 2,888 pivots in a row. On the
// B200: 1.16 ms per refactorization there, of which the chains 0.8 ms (0.28 us a pivot), the bottom
// subtrees 0.09 ms and their updates of top entries 0.03 ms; 0.31 ms at 41k unknowns. The level
// lists of lu.cu, a barrier and a round trip to global memory per level, take 7.32 and 1.40 ms.
#include <algorithm>
#include <cfloat>
#include <string>

#include "lu_updates.cuh"
#include "lutree.h"

int xd_internal_fail(int code, const std::string &msg);

namespace {

constexpr int kBottomThreads = 512;
constexpr int kSchurLanes = 8;        // threads per top destination
constexpr int kTopThreads = 256;
constexpr int kB = kBlockPivots;
constexpr int kLd = kB + 2;           // row stride of the block's L and U in shared memory: 16-byte reads without conflicts
constexpr int kSpinLimit = 1 << 24;   // polls of a chain's flag before the wait gives up

// The bottom subtrees: block g walks its own levels, one barrier per level (the schedule of lu.cu's
// lu_levels_block_kernel: a level's updates form their L factors on the spot, the divisions that
// store them follow during the next level). A level's pivot updates ancestors only, which sit in
// later levels of the same block or in the top part.
__global__ void __launch_bounds__(kBottomThreads) tree_bottom_kernel(
    const int *__restrict__ glev, const int *__restrict__ ldiv, const int *__restrict__ ldst,
    const int2 *__restrict__ div, const int4 *__restrict__ dst, const int4 *__restrict__ pairs, double *v) {
  const int l0 = glev[blockIdx.x], l1 = glev[blockIdx.x + 1], tid = threadIdx.x;
  int4 ds_next = make_int4(0, 0, 0, 0);
  int2 dv_next = make_int2(0, 0);
  int ub = ldst[l0], ue = l0 < l1 ? ldst[l0 + 1] : ub, db = ldiv[l0], de = db;
  if (ub + tid < ue) ds_next = dst[ub + tid];
  for (int l = l0; l < l1; ++l) {
    const int4 ds = ds_next;
    const int2 dv = dv_next;
    const int ne = l + 1 < l1 ? ldst[l + 2] : ue, nd = ldiv[l + 1];
    if (ue + tid < ne) ds_next = dst[ue + tid];
    if (de + tid < nd) dv_next = div[de + tid];
    if (ub + tid < ue) {
      lu_update_divide(ds, pairs, v);
      for (int d = ub + tid + kBottomThreads; d < ue; d += kBottomThreads) lu_update_divide(dst[d], pairs, v);
    }
    if (db + tid < de) {
      lu_divide(dv, v);
      for (int t = db + tid + kBottomThreads; t < de; t += kBottomThreads) lu_divide(div[t], v);
    }
    __syncthreads();
    ub = ue;
    ue = ne;
    db = de;
    de = nd;
  }
  if (db + tid < de) {
    lu_divide(dv_next, v);
    for (int t = db + tid + kBottomThreads; t < de; t += kBottomThreads) lu_divide(div[t], v);
  }
}

// The bottom pivots' updates of top entries, all at once: kSchurLanes threads per destination, fixed
// reduction order.
__global__ void __launch_bounds__(256) tree_schur_kernel(int nd, const int *__restrict__ sdst,
                                                         const int *__restrict__ sptr, const int2 *__restrict__ pairs,
                                                         double *v) {
  const int d = (blockIdx.x * 256 + threadIdx.x) / kSchurLanes, lane = threadIdx.x % kSchurLanes;
  double acc = 0.0;
  if (d < nd)
    for (int p = sptr[d] + lane, e = sptr[d + 1]; p < e; p += kSchurLanes) {
      const int2 lu = pairs[p];
      acc = fma(v[lu.x], v[lu.y], acc);
    }
#pragma unroll
  for (int o = kSchurLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (d < nd && lane == 0) v[sdst[d]] -= acc;
}

__device__ __forceinline__ void cp_async16(void *s, const void *g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(g) : "memory");
}

// 1 / x for normal x: the approximate reciprocal instruction and two Newton steps y += y (1 - x y),
// each squaring its relative error of 2^-20; branch-free, where the division operator's
// special-case branch would keep the compiler from overlapping a pivot's reciprocal with the
// block's other updates. Zero and subnormal pivots are reported by tree_finish_kernel.
__device__ __forceinline__ double reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// A frame's shared memory: the frame, two blocks' panels, the block's L and U, its diagonal part,
// two blocks' records and the slots of its pivots.
struct Frame {
  double *a, *ring, *sl, *su, *sd;
  int *rec;
  unsigned char *piv;
  static __host__ __device__ int ld(int F) { return F + 1; }
  static __host__ __device__ size_t bytes(int F) {
    return sizeof(double) * ((size_t)F * ld(F) + 2 * kB * 2 * F + 2 * F * kLd + kB * kB) + 2 * sizeof(int) * kBlockInts + F;
  }
  __device__ Frame(double *s, int F) {
    a = s;  // F is a multiple of 16, so every part starts on 16 bytes
    ring = a + F * ld(F);
    sl = ring + 2 * kB * 2 * F;
    su = sl + F * kLd;
    sd = su + F * kLd;
    rec = (int *)(sd + kB * kB);
    piv = (unsigned char *)(rec + 2 * kBlockInts);
  }
};

// The frame minus the block's rank-kB product over rows [0, R) and 16 * NB columns from c0: thread
// (tid / 16, tid % 16) takes every 16th row and column, two rows at a time. The pivots' own rows
// and columns become zero: their slots are free for the variables that enter next.
template <int NB>
__device__ __forceinline__ void rank_update(const Frame &f, int ld, int R, int c0, int tid) {
  const int tx = tid & 15, ty = tid >> 4;
  double u[NB][kB];
  bool cp[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int c = c0 + tx + 16 * b;
#pragma unroll
    for (int j = 0; j < kB; j += 2) {
      const double2 v = *(const double2 *)(f.su + c * kLd + j);
      u[b][j] = v.x;
      u[b][j + 1] = v.y;
    }
    cp[b] = f.piv[c];
  }
  for (int r = ty; r < R; r += 32) {
    const int r2 = min(r + 16, R - 1);
    double l[2][kB], a[2][NB];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int rr = h ? r2 : r;
#pragma unroll
      for (int j = 0; j < kB; j += 2) {
        const double2 v = *(const double2 *)(f.sl + rr * kLd + j);
        l[h][j] = -v.x;
        l[h][j + 1] = -v.y;
      }
#pragma unroll
      for (int b = 0; b < NB; ++b) a[h][b] = f.a[rr * ld + c0 + tx + 16 * b];
    }
    const bool p0 = f.piv[r], p1 = f.piv[r2];
#pragma unroll
    for (int j = 0; j < kB; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int b = 0; b < NB; ++b) a[h][b] = fma(l[h][j], u[b][j], a[h][b]);
#pragma unroll
    for (int b = 0; b < NB; ++b) f.a[r * ld + c0 + tx + 16 * b] = p0 || cp[b] ? 0.0 : a[0][b];
    if (r + 16 < R)
#pragma unroll
      for (int b = 0; b < NB; ++b) f.a[r2 * ld + c0 + tx + 16 * b] = p1 || cp[b] ? 0.0 : a[1][b];
  }
}

// The top pivots: one block per chain, kB pivots at a time. The frame holds, for every pair of
// variables in the chain's front, the sum of the updates so far; a pivot's own row and column (A's
// entries and the bottom's updates, its panel) are added when its block comes. Per block of pivots,
// with a barrier after each:
//   1. thread r of the first half takes row r's entries of the pivots' columns, thread c of the
//      second half column c's entries of their rows, and the last threads gather the kB x kB
//      diagonal part;
//   2. each of those threads factors the diagonal part in its own registers and eliminates its row
//      (column) along with it, so the block's pivots follow one another without a barrier or a
//      message: a pivot's reciprocal, a multiplication and an update are the serial chain;
//   3. all threads subtract the rank-kB product from the frame.
// A child chain leaves its remaining front in jbuf and its parent adds it at the block where the
// two paths meet. Chains are taken by ticket, children first, so a chain that waits only waits for
// blocks already running.
__global__ void __launch_bounds__(kTopThreads) tree_top_kernel(int F, const int *__restrict__ cptr,
                                                               const int *__restrict__ bptr,
                                                               const int *__restrict__ blocks,
                                                               const int *__restrict__ jchild,
                                                               const unsigned char *__restrict__ jmap, double *jbuf,
                                                               double *panels, int *ctl) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_chain;
  const Frame f(smem, F);
  const int ld = Frame::ld(F), tid = threadIdx.x;
  if (tid == 0) s_chain = atomicAdd(ctl + kTreeTicket, 1);
  for (int i = tid; i < F * ld; i += kTopThreads) f.a[i] = 0.0;
  for (int i = tid; i < F; i += kTopThreads) f.piv[i] = 0;
  __syncthreads();
  const int chain = s_chain, len = cptr[chain + 1] - cptr[chain], b0 = bptr[chain], nblk = bptr[chain + 1] - b0;
  panels += (size_t)cptr[chain] * 2 * F;
  auto fetch = [&](int t) {  // block t's panels and record
    if (t < nblk) {
      const int units = min(kB, len - t * kB) * F;
      double *to = f.ring + (t & 1) * kB * 2 * F;
      const double *from = panels + (size_t)t * kB * 2 * F;
      for (int i = tid; i < units; i += kTopThreads) cp_async16(to + 2 * i, from + 2 * i);
      if (tid < kBlockInts / 4)
        cp_async16(f.rec + (t & 1) * kBlockInts + 4 * tid, blocks + (size_t)(b0 + t) * kBlockInts + 4 * tid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  for (int t = 0; t < nblk; ++t) {
    const int nb = min(kB, len - t * kB);
    const double *pan = f.ring + (t & 1) * kB * 2 * F;
    const int *rec = f.rec + (t & 1) * kBlockInts;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    fetch(t + 1);
    const int R = rec[kB];
    for (int j = rec[kB + 1]; j < rec[kB + 2]; ++j) {
      const int child = jchild[j];
      if (tid == 0) {
        int w = 0;
        while (atomicAdd(ctl + kTreeFlags + child, 0) == 0 && ++w < kSpinLimit) __nanosleep(64);
        if (w == kSpinLimit) ctl[kTreeExpired] = 1;
        __threadfence();
      }
      __syncthreads();
      const unsigned char *map = jmap + (size_t)child * F;
      const double *from = jbuf + (size_t)child * F * F;
      for (int i = tid; i < R * R; i += kTopThreads) {
        const int r = i / R, c = i % R, rm = map[r], cm = map[c];
        if (rm != kJoinNone && cm != kJoinNone) f.a[r * ld + c] += __ldcg(from + rm * F + cm);
      }
      __syncthreads();
    }
    const int half = (R + 31) & ~31;
    const bool lside = tid < half, uside = !lside && tid < 2 * half;
    const int me = lside ? tid : tid - half, m = min(me, R - 1);
    double x[kB];
    if (lside || uside) {
      const double *base = lside ? f.a + m * ld : f.a + m, *pb = pan + (lside ? F + m : m);
      const int step = lside ? 1 : ld;
      double p[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const int s = rec[j];
        x[j] = base[(s & 0xff) * step];
        p[j] = pb[j * 2 * F];
      }
#pragma unroll
      for (int j = 0; j < kB; ++j) x[j] = j < nb && me < R ? x[j] + p[j] : 0.0;
    }
    if (tid >= kTopThreads - kB * kB) {
      const int i = (tid - (kTopThreads - kB * kB)) / kB, j = tid % kB;
      const int ti = rec[i] & 0xff, tj = rec[j] & 0xff;
      const double v = f.a[ti * ld + tj], w = pan[j >= i ? i * 2 * F + tj : j * 2 * F + F + ti];
      f.sd[i * kB + j] = i < nb && j < nb ? v + w : (i == j ? 1.0 : 0.0);
    }
    if (tid < nb) f.piv[rec[tid]] = 1;
    __syncthreads();
    if (lside || uside) {
      double d[kB][kB];
#pragma unroll
      for (int i = 0; i < kB; ++i)
#pragma unroll
        for (int j = 0; j < kB; j += 2) {
          const double2 v = *(const double2 *)&f.sd[i * kB + j];
          d[i][j] = v.x;
          d[i][j + 1] = v.y;
        }
      int mine = kB;  // this slot's pivot of the block: its row (column) ends there
#pragma unroll
      for (int j = 0; j < kB; ++j)
        if (rec[j] == me) mine = j;
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const double rp = reciprocal(d[j][j]);
#pragma unroll
        for (int i = j + 1; i < kB; ++i) d[i][j] *= rp;
        if (lside) {
          x[j] = j < mine ? x[j] * rp : 0.0;
#pragma unroll
          for (int i = j + 1; i < kB; ++i) x[i] = fma(-x[j], d[j][i], x[i]);
        } else {
          if (j > mine) x[j] = 0.0;
#pragma unroll
          for (int i = j + 1; i < kB; ++i) x[i] = fma(-d[i][j], x[j], x[i]);
        }
#pragma unroll
        for (int i = j + 1; i < kB; ++i)
#pragma unroll
          for (int c = j + 1; c < kB; ++c) d[i][c] = fma(-d[i][j], d[j][c], d[i][c]);
      }
      if (me < F) {  // zeros in the slots from R on, which the update reads up to a multiple of 16
        double *sx = (lside ? f.sl : f.su) + me * kLd;
#pragma unroll
        for (int j = 0; j < kB; j += 2) *(double2 *)(sx + j) = make_double2(x[j], x[j + 1]);
        double *to = panels + (size_t)t * kB * 2 * F + (lside ? F : 0) + me;
#pragma unroll
        for (int j = 0; j < kB; ++j)
          if (j < nb) to[j * 2 * F] = x[j];
      }
    }
    __syncthreads();
    for (int c0 = 0; c0 < R; c0 += 64) {
      const int nt = min(4, (R - c0 + 15) / 16);
      if (nt == 4)
        rank_update<4>(f, ld, R, c0, tid);
      else if (nt == 3)
        rank_update<3>(f, ld, R, c0, tid);
      else if (nt == 2)
        rank_update<2>(f, ld, R, c0, tid);
      else
        rank_update<1>(f, ld, R, c0, tid);
    }
    __syncthreads();
    if (tid < nb) f.piv[rec[tid]] = 0;
  }
  double *to = jbuf + (size_t)chain * F * F;
  for (int i = tid; i < F * F; i += kTopThreads) __stcg(to + i, f.a[(i / F) * ld + i % F]);
  __threadfence();
  __syncthreads();
  if (tid == 0) atomicExch(ctl + kTreeFlags + chain, 1);
}

// What follows the elimination: the top pivots' column entries outside their panels are divided,
// and zero pivots (of the top, subnormal ones too) reported: n - k for the first such k.
__global__ void tree_finish_kernel(int nt, const int2 *__restrict__ tdiv, int n, const int *__restrict__ diag, int p0,
                                   double *v, int *ctl) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nt) lu_divide(tdiv[k], v);
  if (k < n) {
    const double p = v[diag[k]];
    if (p == 0.0 || (diag[k] >= p0 && fabs(p) < DBL_MIN)) atomicMax(ctl + kTreeInfo, n - k);
  }
}

template <class D, class T>
cudaError_t upload(D **d, const std::vector<T> &h) {
  static_assert(sizeof(D) == sizeof(T), "device and host records match");
  cudaError_t e = cudaMalloc(d, std::max<size_t>(1, h.size()) * sizeof(T));
  if (e != cudaSuccess || h.empty()) return e;
  return cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
}

}  // namespace

int xd_tree_upload(XdTree *t, const XdTreePlan &p) {
  t->n = p.n;
  t->F = p.F;
  t->ntop = p.ntop;
  t->ngroups = p.ngroups;
  t->nchains = p.nchains;
  t->nsd = (int)p.sdst.size();
  t->ntdiv = (int)p.tdiv.size();
  t->p0 = p.p0;
  t->nv = p.nv;
  cudaError_t e;
  if ((e = cudaMalloc(&t->d_v, sizeof(double) * std::max<long long>(1, p.nv))) != cudaSuccess ||
      (e = upload(&t->d_diag, p.diag)) != cudaSuccess || (e = upload(&t->d_glev, p.glev)) != cudaSuccess ||
      (e = upload(&t->d_ldiv, p.ldiv)) != cudaSuccess || (e = upload(&t->d_ldst, p.ldst)) != cudaSuccess ||
      (e = upload(&t->d_div, p.div)) != cudaSuccess || (e = upload(&t->d_dst, p.dst)) != cudaSuccess ||
      (e = upload(&t->d_pairs, p.pairs)) != cudaSuccess || (e = upload(&t->d_sdst, p.sdst)) != cudaSuccess ||
      (e = upload(&t->d_sptr, p.sptr)) != cudaSuccess || (e = upload(&t->d_spairs, p.spairs)) != cudaSuccess ||
      (e = upload(&t->d_tdiv, p.tdiv)) != cudaSuccess || (e = upload(&t->d_cptr, p.cptr)) != cudaSuccess ||
      (e = upload(&t->d_bptr, p.bptr)) != cudaSuccess || (e = upload(&t->d_blocks, p.blocks)) != cudaSuccess ||
      (e = upload(&t->d_jchild, p.jchild)) != cudaSuccess || (e = upload(&t->d_jmap, p.jmap)) != cudaSuccess ||
      (e = cudaMalloc(&t->d_jbuf, sizeof(double) * std::max<size_t>(1, (size_t)p.nchains * p.F * p.F))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(tree_top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)Frame::bytes(kMaxFrame))) != cudaSuccess ||
      (e = cudaMalloc(&t->d_ctl, sizeof(int) * (kTreeFlags + p.nchains))) != cudaSuccess) {
    xd_tree_free(t);
    return xd_internal_fail(-3, std::string("LU set-up upload: ") + cudaGetErrorString(e));
  }
  t->on = true;
  return 0;
}

void xd_tree_free(XdTree *t) {
  for (void *p : {(void *)t->d_v, (void *)t->d_diag, (void *)t->d_glev, (void *)t->d_ldiv, (void *)t->d_ldst,
                  (void *)t->d_div, (void *)t->d_dst, (void *)t->d_pairs, (void *)t->d_sdst, (void *)t->d_sptr,
                  (void *)t->d_spairs, (void *)t->d_tdiv, (void *)t->d_cptr, (void *)t->d_bptr, (void *)t->d_blocks,
                  (void *)t->d_jchild, (void *)t->d_jmap, (void *)t->d_jbuf, (void *)t->d_ctl})
    cudaFree(p);
  *t = XdTree();
}

int xd_tree_factor(XdTree *t, cudaStream_t st) {
  if (t->ngroups > 0)
    tree_bottom_kernel<<<t->ngroups, kBottomThreads, 0, st>>>(t->d_glev, t->d_ldiv, t->d_ldst, t->d_div, t->d_dst,
                                                              t->d_pairs, t->d_v);
  if (t->nsd > 0) {
    const long long threads = (long long)t->nsd * kSchurLanes;
    tree_schur_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(t->nsd, t->d_sdst, t->d_sptr, t->d_spairs,
                                                                         t->d_v);
  }
  if (t->nchains > 0) {
    tree_top_kernel<<<t->nchains, kTopThreads, Frame::bytes(t->F), st>>>(
        t->F, t->d_cptr, t->d_bptr, t->d_blocks, t->d_jchild, t->d_jmap, t->d_jbuf, t->d_v + t->p0, t->d_ctl);
  }
  const int work = std::max(t->n, t->ntdiv);
  if (work > 0)
    tree_finish_kernel<<<(work + 255) / 256, 256, 0, st>>>(t->ntdiv, t->d_tdiv, t->n, t->d_diag, t->p0,
                                                             t->d_v, t->d_ctl);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return xd_internal_fail(-3, std::string("LU refactorization launch: ") + cudaGetErrorString(e));
  return 0;
}
