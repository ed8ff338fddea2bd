// Sparse LU refactorization and triangular solves over an elimination-tree plan (lutree.h).
//
// What bounds them is the longest chain of dependent pivots, not arithmetic or bytes: at 200k unknowns
// 12.6M updates (0.7 us of the FP64 pipe) and 27 MB of values, but 2,888 pivots in a row. On the
// B200, per refactorization there: 1.09 ms, of which the chains 0.95 ms (0.33 us a pivot), the bottom
// subtrees 0.09 ms and their updates of top entries 0.03 ms; per solve 0.63 ms: the chains 0.22 ms
// forward and 0.35 ms backward, the bottom subtrees 0.03 ms each way. At 41k unknowns 0.28 and 0.21
// ms. The level lists of lu.cu and sptrsv.cu, with a barrier and a round trip to global memory per
// level, take 7.32 and 7.25 ms, and 1.40 and 1.56 ms.
#include <algorithm>
#include <string>

#include "lu_updates.cuh"
#include "lutree.h"

int xd_internal_fail(int code, const std::string &msg);

namespace {

constexpr int kBottomThreads = 512;
constexpr int kBottomEntries = 13 * 1024;  // a group's entries in shared memory: two blocks to an SM
constexpr int kSchurLanes = 8;        // threads per top destination
constexpr int kSchurLong = 512;       // updates of a top destination that these take; more: a block
constexpr int kTopRowLong = 1024;     // entries of a top row that a warp sums; more: a block
constexpr int kTopThreads = 256;
constexpr int kB = kBlockPivots;
constexpr int kLd = kB + 2;           // row stride of the block's L and U in shared memory: 16-byte reads without conflicts
constexpr int kSpinLimit = 1 << 24;   // polls of a chain's flag before the wait gives up

// One destination's updates, its first two pairs already here (ds.w < 0 and more than one or two: the
// rest in batches, so that a batch waits for one round of loads).
__device__ __forceinline__ void bottom_update(int4 ds, int4 p0, int4 p1, const int4 *__restrict__ pairs, double *m) {
  double acc = m[ds.x];
  if (ds.w >= 0) {
    acc = acc - (m[ds.y] / m[ds.w]) * m[ds.z];
  } else {
    acc = acc - (m[p0.x] / m[p0.z]) * m[p0.y];
    if (ds.z > 1) acc = acc - (m[p1.x] / m[p1.z]) * m[p1.y];
    for (int p = ds.y + 2; p < ds.y + ds.z; p += 4) {
      int4 lu[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p + k < ds.y + ds.z) lu[k] = pairs[p + k];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p + k < ds.y + ds.z) acc = acc - (m[lu[k].x] / m[lu[k].z]) * m[lu[k].y];
    }
  }
  m[ds.x] = acc;
}

// The same by a warp, for a destination with many updates (a node that everything in its subtree hangs
// on: a refactorization with a hub of 6,000 leaves took 1,870 us with one thread on its pairs, and takes
// 153; with 25 hubs of 2,000, 1,200 and 140): strided, fixed tree.
__device__ __forceinline__ void bottom_update_long(int4 ds, const int4 *__restrict__ pairs, int lane, double *m) {
  double acc = 0.0;
#pragma unroll 4
  for (int p = ds.y + lane; p < ds.y + ds.z; p += 32) {
    const int4 lu = pairs[p];
    acc += (m[lu.x] / m[lu.z]) * m[lu.y];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) m[ds.x] -= acc;
}

// A block's levels, one barrier per level (the schedule of lu.cu's lu_levels_block_kernel: a level's
// updates form their L factors on the spot, the divisions that store them follow during the next
// level). A level's pivot updates ancestors only, which sit in later levels of the same block or in
// the top part. A level's lists are read two levels ahead, its first pairs one level ahead. LONG: the
// destinations from llong on take a warp each.
template <bool LONG>
__device__ __forceinline__ void bottom_levels(int l0, int l1, const int *__restrict__ ldiv,
                                              const int *__restrict__ ldst, const int *__restrict__ llong,
                                              const int2 *__restrict__ div,
                                              const int4 *__restrict__ dst, const int4 *__restrict__ pairs, double *m) {
  const int tid = threadIdx.x;
  const int4 none = make_int4(0, 0, 0, 0);
  auto short_end = [&](int l) { return LONG ? llong[l] : ldst[l + 1]; };
  auto list = [&](int l) {  // this thread's destination of level l
    if (l >= l1) return none;
    const int b = ldst[l] + tid;
    return b < short_end(l) ? dst[b] : none;
  };
  auto pair = [&](int4 ds, int k) { return ds.w < 0 && ds.z > k ? pairs[ds.y + k] : none; };
  int4 ds1 = list(l0), ds2 = list(l0 + 1), p0 = pair(ds1, 0), p1 = pair(ds1, 1);
  int2 dv_next = make_int2(0, 0);
  int ub = ldst[l0], ue = l0 < l1 ? short_end(l0) : ub, db = ldiv[l0], de = db;
  for (int l = l0; l < l1; ++l) {
    const int4 ds = ds1, q0 = p0, q1 = p1;
    const int2 dv = dv_next;
    const int ne = l + 1 < l1 ? short_end(l + 1) : ue, nd = ldiv[l + 1], nb = LONG ? ldst[l + 1] : ue;
    ds1 = ds2;
    ds2 = list(l + 2);
    p0 = pair(ds1, 0);
    p1 = pair(ds1, 1);
    if (de + tid < nd) dv_next = div[de + tid];
    if (ub + tid < ue) {
      bottom_update(ds, q0, q1, pairs, m);
      for (int d = ub + tid + kBottomThreads; d < ue; d += kBottomThreads) {
        const int4 more = dst[d];
        bottom_update(more, pair(more, 0), pair(more, 1), pairs, m);
      }
    }
    if (LONG)
      for (int d = ue + tid / 32; d < nb; d += kBottomThreads / 32) bottom_update_long(dst[d], pairs, tid % 32, m);
    if (db + tid < de) {
      lu_divide(dv, m);
      for (int t = db + tid + kBottomThreads; t < de; t += kBottomThreads) lu_divide(div[t], m);
    }
    __syncthreads();
    ub = nb;
    ue = ne;
    db = de;
    de = nd;
  }
  if (db + tid < de) {
    lu_divide(dv_next, m);
    for (int t = db + tid + kBottomThreads; t < de; t += kBottomThreads) lu_divide(div[t], m);
  }
}

// The bottom subtrees, a block each. What bounds a block is its levels one after the other: quotients,
// barriers and, in global memory, an L2 round trip of a level's operands. So the group's own entries
// (gpos: their places in V) come to shared memory first, the lists hold positions there, and the
// entries go back at the end: refactorization of 4,455 unknowns 149 -> 139 us, of 41k 288 -> 276, of
// 200k (where the chains wait) the same. A group with more than kBottomEntries entries (gptr: none of
// them) works in V itself: systems of millions of unknowns have such groups, and a single subtree can be
// one (the limit on subtrees counts updates, of which a hub of 6,000 leaves has 6,000 for 18,000 entries).
template <bool LONG>
__global__ void __launch_bounds__(kBottomThreads) tree_bottom_kernel(
    const int *__restrict__ glev, const int *__restrict__ ldiv, const int *__restrict__ ldst, const int *__restrict__ llong,
    const int2 *__restrict__ div, const int4 *__restrict__ dst, const int4 *__restrict__ pairs,
    const int *__restrict__ gptr, const int *__restrict__ gpos, double *v) {
  extern __shared__ double entries[];
  const int l0 = glev[blockIdx.x], l1 = glev[blockIdx.x + 1], e0 = gptr[blockIdx.x], ne = gptr[blockIdx.x + 1] - e0;
  if (ne == 0) {
    bottom_levels<LONG>(l0, l1, ldiv, ldst, llong, div, dst, pairs, v);
    return;
  }
  for (int i = threadIdx.x; i < ne; i += kBottomThreads) entries[i] = v[gpos[e0 + i]];
  __syncthreads();
  bottom_levels<LONG>(l0, l1, ldiv, ldst, llong, div, dst, pairs, entries);
  __syncthreads();
  for (int i = threadIdx.x; i < ne; i += kBottomThreads) v[gpos[e0 + i]] = entries[i];
}

// The sum of the threads' values over a block of 256, in thread 0, in a fixed order.
__device__ __forceinline__ double block_sum256(double acc, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = acc;
  __syncthreads();
  acc = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < 8; ++w) acc += red[w];
  __syncthreads();
  return acc;
}

// The bottom pivots' updates of top entries, all at once: kSchurLanes threads per destination, and the
// whole block for one with more than kSchurLong updates (LONG: there are such); fixed reduction order.
template <bool LONG>
__global__ void __launch_bounds__(256) tree_schur_kernel(int nd, const int *__restrict__ sdst,
                                                         const int *__restrict__ sptr, const int2 *__restrict__ pairs,
                                                         double *v) {
  const int d = (blockIdx.x * 256 + threadIdx.x) / kSchurLanes, lane = threadIdx.x % kSchurLanes;
  double acc = 0.0;
  const int b = d < nd ? sptr[d] : 0, e = d < nd ? sptr[d + 1] : 0;
  const bool many = LONG && e - b > kSchurLong;
  if (!many)
    for (int p = b + lane; p < e; p += kSchurLanes) {
      const int2 lu = pairs[p];
      acc = fma(v[lu.x], v[lu.y], acc);
    }
#pragma unroll
  for (int o = kSchurLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (d < nd && lane == 0 && !many) v[sdst[d]] -= acc;
  if (!LONG || !__syncthreads_or(many)) return;
  __shared__ double red[8];
  for (int q = blockIdx.x * (256 / kSchurLanes), qe = min(nd, q + 256 / kSchurLanes); q < qe; ++q) {
    const int qb = sptr[q], qn = sptr[q + 1];
    if (qn - qb <= kSchurLong) continue;
    acc = 0.0;
#pragma unroll 4
    for (int p = qb + threadIdx.x; p < qn; p += 256) {
      const int2 lu = pairs[p];
      acc = fma(v[lu.x], v[lu.y], acc);
    }
    acc = block_sum256(acc, red);
    if (threadIdx.x == 0) v[sdst[q]] -= acc;
  }
}

__device__ __forceinline__ void cp_async16(void *s, const void *g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(g) : "memory");
}

// 1 / x for ordinary x (below): the approximate reciprocal instruction and two Newton steps y += y (1 -
// x y), each squaring its relative error of 2^-20; branch-free, where the division operator's
// special-case branch would keep the compiler from overlapping a pivot's reciprocal with the
// block's other updates.
__device__ __forceinline__ double reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// Pivots whose reciprocal and its approximation are normal numbers. The others (subnormal, above 2^1021,
// zero, not finite) need the division: tree_finish_kernel reports them, and the caller then takes the
// matrix again with DIVIDE. The chains' kernels do not look for them on their way: a check per pivot
// and a way round it cost 46 us of the 1.79 ms of a refactorization and solve at 200k unknowns.
__device__ __forceinline__ bool ordinary(double p) { return fabs(p) >= 0x1p-1021 && fabs(p) <= 0x1p1021; }

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
template <bool DIVIDE>
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
  const size_t stride = xd_panel_size(F);
  panels += b0 * stride;
  auto fetch = [&](int t) {  // block t's panels and record
    if (t < nblk) {
      double *to = f.ring + (t & 1) * kB * 2 * F;
      const double *from = panels + t * stride;
      for (int i = tid; i < kB * F; i += kTopThreads) cp_async16(to + 2 * i, from + 2 * i);
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
      const double *base = lside ? f.a + m * ld : f.a + m, *pb = pan + (lside ? kB * F + m : m);
      const int step = lside ? 1 : ld;
      double p[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const int s = rec[j];
        x[j] = base[(s & 0xff) * step];
        p[j] = pb[j * F];
      }
#pragma unroll
      for (int j = 0; j < kB; ++j) x[j] = j < nb && me < R ? x[j] + p[j] : 0.0;
    }
    if (tid >= kTopThreads - kB * kB) {
      const int i = (tid - (kTopThreads - kB * kB)) / kB, j = tid % kB;
      const int ti = rec[i] & 0xff, tj = rec[j] & 0xff;
      const double v = f.a[ti * ld + tj], w = pan[j >= i ? i * F + tj : (kB + j) * F + ti];
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
        const double pv = d[j][j], rp = DIVIDE ? 0.0 : reciprocal(pv);
#pragma unroll
        for (int i = j + 1; i < kB; ++i) d[i][j] = DIVIDE ? d[i][j] / pv : d[i][j] * rp;
        if (lside) {
          x[j] = j >= mine ? 0.0 : DIVIDE ? x[j] / pv : x[j] * rp;
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
        double *to = panels + t * stride + (lside ? kB * F : 0) + me;
#pragma unroll
        for (int j = 0; j < kB; ++j)
          if (j < nb) to[j * F] = x[j];
      }
    }
    __syncthreads();
    if (tid >= kTopThreads - kB * kB) {  // the factored diagonal part, for the solves
      const int i = (tid - (kTopThreads - kB * kB)) / kB, j = tid % kB;
      const double *row = (j >= i ? f.su : f.sl) + (rec[max(i, j)] & 0xff) * kLd;
      double d = i == j ? 1.0 : 0.0;
      if (i < nb && j < nb) d = i != j ? row[min(i, j)] : DIVIDE ? row[i] : reciprocal(row[i]);
      panels[t * stride + 2 * kB * F + i * kB + j] = d;
    }
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

// What follows the elimination: the top pivots' column entries outside their panels are divided, zero
// pivots reported (n - k for the first such k), and whether a top pivot is not an ordinary one.
__global__ void tree_finish_kernel(int nt, const int2 *__restrict__ tdiv, int n, const int *__restrict__ diag, int p0,
                                   double *v, int *ctl) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nt) lu_divide(tdiv[k], v);
  if (k < n) {
    const double p = v[diag[k]];
    if (p == 0.0) atomicMax(ctl + kTreeInfo, n - k);
    if (diag[k] >= p0 && !ordinary(p)) ctl[kTreeOdd] = 1;
  }
}

// ---- solves --------------------------------------------------------------------------------------
// Forward: the bottom subtrees' rows level by level, the top rows' sums over bottom columns in one
// pass, then the chains; backward the other way round. As in the factorization, a chain's pivots
// are the serial part: a block per chain takes kB of them at a time, a thread per slot of the frame and
// one more warp that streams the panels in; every thread solves the block's small triangle redundantly
// in registers, so that consecutive pivots cost a multiply-add's latency.

constexpr int kSolveAhead = 4;        // blocks in flight in a chain's solve
constexpr int kPassRows = 24 * 1024;  // rows of a group whose values fit shared memory
constexpr int kTailChunk = 2048;      // entries a block sums of a row solved last
static_assert(kB == 8, "the backward solve's reduction is written for blocks of eight pivots");

__global__ void tree_rhs_kernel(int n, const int *__restrict__ bsrc, const double *__restrict__ b,
                                double *__restrict__ y) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x < n) y[x] = b[bsrc[x]];
}

// One bottom group's passes (XdPasses): s[row] from the row's sum over already solved s. The group's
// own solved values are kept in shared memory (the group's rows are [base, base + size); a group
// with more than kPassRows keeps them in s), and what does not depend on them - columns and values of
// a pass's first round, its rows and their right-hand sides, solved values of columns outside the
// group - is loaded a pass ahead, so a level waits for shared memory alone. Forward: s[row] =
// rhs[row] - sum, in place; backward: divided by the diagonal, and scattered to the solution. LONG:
// there are rows of several warps.
template <bool BACKWARD, bool LONG>
__global__ void __launch_bounds__(kPassThreads) tree_pass_kernel(const int *__restrict__ gptr,
                                                                 const int4 *__restrict__ pass,
                                                                 const int *__restrict__ rows,
                                                                 const int *__restrict__ col, int off0,
                                                                 const double *__restrict__ v,
                                                                 const double *__restrict__ vd, const double *rhs,
                                                                 double *s, const int *__restrict__ xdst, double *out,
                                                                 const int *__restrict__ grow) {
  extern __shared__ __align__(16) double smem[];
  __shared__ double red[kPassThreads / 32];
  const int tid = threadIdx.x, base = grow[blockIdx.x], size = grow[blockIdx.x + 1] - base;
  const bool fits = size <= kPassRows;
  double *loc = fits ? smem : s + base;
  auto own = [&](int c) { return (unsigned)(c - base) < (unsigned)size; };
  if (!BACKWARD && fits) {  // rows without entries keep their right-hand sides
    for (int i = tid; i < size; i += kPassThreads) smem[i] = rhs[base + i];
    __syncthreads();
  }
  // First what needs only the pass's record, two passes ahead; then what its column and row point to.
  struct First {
    int4 m;
    int x, c;
    double a;
  };
  struct Second {
    double b, d, sv;
    int to;
  };
  auto load_first = [&](int4 m) {
    First f;
    f.m = m;
    f.x = f.c = -1;
    f.a = 0.0;
    const int lg = m.y >> 16 & 0xff;
    if (tid < (m.y & 0xffff) << lg) {
      f.c = col[m.z - off0 + tid];
      f.a = v[m.z + tid];
      if ((tid & ((1 << lg) - 1)) == 0) f.x = rows[m.x + (tid >> lg)];
    }
    return f;
  };
  auto load_second = [&](const First &f) {
    Second q;
    q.b = q.sv = 0.0;
    q.d = 1.0;
    q.to = 0;
    if (f.c >= 0 && !own(f.c)) q.sv = s[f.c];
    if (f.x >= 0) {
      q.b = rhs[f.x];
      if (BACKWARD) {
        q.d = vd[f.x];
        q.to = xdst[f.x];
      }
    }
    return q;
  };
  const int p1 = gptr[blockIdx.x + 1];
  int p = gptr[blockIdx.x];
  if (p >= p1) return;
  auto record = [&](int q) { return q < p1 ? pass[q] : make_int4(0, 0, 0, 0); };
  int4 m2 = record(p + 1), m3 = record(p + 2);
  First f0 = load_first(record(p)), f1 = load_first(m2);
  Second q0 = load_second(f0);
  m2 = m3;
  m3 = record(p + 3);
  for (; p < p1; ++p) {
    const First f = f0;
    const Second q = q0;
    q0 = load_second(f1);
    f0 = f1;
    f1 = load_first(m2);
    m2 = m3;
    m3 = record(p + 4);
    const int lg = f.m.y >> 16 & 0xff, width = (f.m.y & 0xffff) << lg;
    double acc = f.c >= 0 ? f.a * (own(f.c) ? loc[f.c - base] : q.sv) : 0.0;
    if (tid < width)
      for (int k = 1; k < f.m.w; ++k) {
        const int at = f.m.z + k * width + tid, c = col[at - off0];
        if (c >= 0) acc += v[at] * (own(c) ? loc[c - base] : s[c]);
      }
    for (int o = LONG ? min(16, 1 << lg >> 1) : 1 << lg >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (LONG && lg > 5) {
      if (tid % 32 == 0) red[tid / 32] = acc;
      __syncthreads();
      if (f.x >= 0)
        for (int w = 1; w < 1 << (lg - 5); ++w) acc += red[tid / 32 + w];
      __syncthreads();
    }
    if (f.x >= 0) {
      const double r = BACKWARD ? (q.b - acc) / q.d : q.b - acc;
      s[f.x] = r;
      if (fits) smem[f.x - base] = r;
      if (BACKWARD) out[q.to] = r;
    }
    if (f.m.y >> 24) __syncthreads();
  }
}

// Rows [x0, n): the top rows' sums over columns outside their panels, a warp each, the block for a row of
// more than kTopRowLong entries (LONG: there are such).
template <bool LONG>
__global__ void __launch_bounds__(256) tree_top_rows_kernel(int x0, int n, const int *__restrict__ lptr,
                                                            const int *__restrict__ lcol, const double *v, double *y) {
  const int r = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x % 32, rows = n - x0;
  const int b = r < rows ? lptr[r] : 0, end = r < rows ? lptr[r + 1] : 0;
  const bool many = LONG && end - b > kTopRowLong;
  double acc = 0.0;
  if (!many)
    for (int e = b + lane; e < end; e += 32) acc += v[e] * y[lcol[e]];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0 && end > b && !many) y[x0 + r] -= acc;
  if (!LONG || !__syncthreads_or(many)) return;
  __shared__ double red[8];
  for (int q = blockIdx.x * 8, qe = min(rows, q + 8); q < qe; ++q) {
    const int qb = lptr[q], qn = lptr[q + 1];
    if (qn - qb <= kTopRowLong) continue;
    acc = 0.0;
#pragma unroll 4
    for (int e = qb + threadIdx.x; e < qn; e += 256) acc += v[e] * y[lcol[e]];
    acc = block_sum256(acc, red);
    if (threadIdx.x == 0) y[x0 + q] -= acc;
  }
}

__device__ __forceinline__ void cp_async8(void *s, const void *g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(g) : "memory");
}

// A chain's solve in shared memory: per block in flight its panel half, its diagonal part, its
// right-hand sides and its record; and what the threads exchange.
struct SolveSmem {
  double *ring, *diag, *rhs, *red;
  int *rec;
  static __host__ __device__ size_t bytes(int F) {
    return sizeof(double) * (kSolveAhead * (kB * F + kB * kB + kB) + 2 * kB * (kMaxFrame / 32)) +
           sizeof(int) * kSolveAhead * kBlockInts;
  }
  __device__ SolveSmem(double *s, int F) {
    ring = s;
    diag = ring + kSolveAhead * kB * F;
    rhs = diag + kSolveAhead * kB * kB;
    red = rhs + kSolveAhead * kB;
    rec = (int *)(red + 2 * kB * (kMaxFrame / 32));
  }
  // Block t (of nblk, records and panels from the chain's first) by one warp; half 0: U, 1: L.
  __device__ void fetch(int t, int nblk, int len, int F, int half, const double *panels, const int *blocks,
                        const double *y, int lane) const {
    if (t >= 0 && t < nblk) {
      const int q = t % kSolveAhead, nb = min(kB, len - t * kB);
      const double *from = panels + t * (size_t)xd_panel_size(F);
      for (int i = lane; i < kB * F / 2; i += 32) cp_async16(ring + q * kB * F + 2 * i, from + half * kB * F + 2 * i);
      cp_async16(diag + q * kB * kB + 2 * lane, from + 2 * kB * F + 2 * lane);
      if (lane < kBlockInts / 4) cp_async16(rec + q * kBlockInts + 4 * lane, blocks + (size_t)t * kBlockInts + 4 * lane);
      if (lane < nb) cp_async8(rhs + q * kB + lane, y + t * kB + lane);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
};

// Waits (one thread) for a chain's flag; false when the wait gave up.
__device__ __forceinline__ bool chain_wait(int *flag) {
  int w = 0;
  while (atomicAdd(flag, 0) == 0 && ++w < kSpinLimit) __nanosleep(32);
  __threadfence();
  return w < kSpinLimit;
}

// The value of the block's `mine`-th pivot from registers.
__device__ __forceinline__ double pick(const double (&v)[kB], int mine) {
  double x = v[0];
#pragma unroll
  for (int j = 1; j < kB; ++j) x = mine == j ? v[j] : x;
  return x;
}

// This slot's pivot of the block, or -1.
__device__ __forceinline__ int pivot_of(const int *rec, int r) {
  int m = -1;
#pragma unroll
  for (int j = 0; j < kB; ++j)
    if (rec[j] == r) m = j;
  return m;
}

// What a chain's solve has in its registers of a block: the diagonal part, this slot's panel entries
// and the right-hand sides.
struct BlockRegs {
  double d[kB][kB], pan[kB], rhs[kB];
  __device__ void load(const SolveSmem &s, int q, int F, int r, int nb) {
#pragma unroll
    for (int i = 0; i < kB; ++i)
#pragma unroll
      for (int j = 0; j < kB; j += 2) {
        const double2 t = *(const double2 *)(s.diag + q * kB * kB + i * kB + j);
        d[i][j] = t.x;
        d[i][j + 1] = t.y;
      }
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      pan[j] = r < F ? s.ring[(q * kB + j) * F + r] : 0.0;
      rhs[j] = j < nb ? s.rhs[q * kB + j] : 0.0;
    }
  }
};

// Forward chains: thread r holds slot r's sum (of L's entries times the solved values so far), the
// last warp streams the blocks in. Per block: the threads of the pivots' slots publish their sums,
// a barrier, and every thread solves the block's triangle and takes its entries times the block's
// values. ticket, flags: zeroed by the caller.
__global__ void __launch_bounds__(kMaxFrame + 32) tree_forward_chain_kernel(
    int F, const int *__restrict__ cptr, const int *__restrict__ bptr, const int *__restrict__ blocks,
    const int *__restrict__ jchild, const unsigned char *__restrict__ jmap, double *wbuf, const double *panels,
    double *y, int *ticket, int *flags) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_chain, s_ok;
  const SolveSmem s(smem, F);
  const int r = threadIdx.x, lane = r % 32;
  const bool feeder = r >= (int)blockDim.x - 32;
  if (r == 0) s_chain = atomicAdd(ticket, 1);
  __syncthreads();
  const int chain = s_chain, len = cptr[chain + 1] - cptr[chain], b0 = bptr[chain], nblk = bptr[chain + 1] - b0;
  panels += b0 * (size_t)xd_panel_size(F);
  blocks += (size_t)b0 * kBlockInts;
  y += cptr[chain];
  if (feeder) {
    for (int t = 0; t < kSolveAhead - 1; ++t) s.fetch(t, nblk, len, F, 1, panels, blocks, y, lane);
    asm volatile("cp.async.wait_group %0;" ::"n"(kSolveAhead - 2) : "memory");
  }
  __syncthreads();
  double w = 0.0;
  for (int t = 0; t < nblk; ++t) {
    const int q = t % kSolveAhead, nb = min(kB, len - t * kB);
    const int *rec = s.rec + q * kBlockInts;
    double *red = s.red + (t & 1) * kB;
    for (int j = rec[kB + 1]; j < rec[kB + 2]; ++j) {
      const int child = jchild[j];
      if (r == 0) s_ok = chain_wait(flags + child);
      __syncthreads();
      if (r < F) {
        const int m = jmap[(size_t)child * F + r];
        if (m != kJoinNone) w += s_ok ? __ldcg(wbuf + (size_t)child * F + m) : __longlong_as_double(-1LL);
      }
      __syncthreads();
    }
    BlockRegs g;
    int mine = -1;
    if (!feeder) {
      mine = pivot_of(rec, r);
      if (mine >= 0) {
        red[mine] = w;
        w = 0.0;
      }
      g.load(s, q, F, r, nb);
    } else {
      asm volatile("cp.async.wait_group %0;" ::"n"(kSolveAhead - 3) : "memory");
    }
    __syncthreads();
    if (feeder) {
      s.fetch(t + kSolveAhead - 1, nblk, len, F, 1, panels, blocks, y, lane);
    } else {
      double v[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) v[j] = j < nb ? g.rhs[j] + red[j] : 0.0;
#pragma unroll
      for (int j = 0; j < kB; ++j)
#pragma unroll
        for (int i = j + 1; i < kB; ++i) v[i] = i < nb ? fma(-g.d[i][j], v[j], v[i]) : 0.0;
      double w2 = 0.0;
#pragma unroll
      for (int j = 0; j < kB; j += 2) {
        w = fma(-g.pan[j], v[j], w);
        w2 = fma(-g.pan[j + 1], v[j + 1], w2);
      }
      w += w2;
      if (mine >= 0) {
        w = 0.0;
        y[t * kB + mine] = pick(v, mine);
      }
    }
  }
  if (r < F) __stcg(wbuf + (size_t)chain * F + r, w);
  __threadfence();
  __syncthreads();
  if (r == 0) atomicExch(flags + chain, 1);
}

// Backward chains, parents first: thread r holds the solved value of slot r's variable. Per block:
// the pivots' row sums over the front, reduced within warps by shuffles and across them through
// shared memory, then the block's triangle.
template <bool DIVIDE>
__global__ void __launch_bounds__(kMaxFrame + 32) tree_backward_chain_kernel(
    int nchains, int F, const int *__restrict__ cptr, const int *__restrict__ bptr, const int *__restrict__ blocks,
    const int *__restrict__ jchild, const int *__restrict__ border, const double *panels, const double *y, int x0,
    double *x, const int *__restrict__ xdst, double *out, int *ticket, int *flags, const int *__restrict__ joined) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_chain, s_ok;
  const SolveSmem s(smem, F);
  const int r = threadIdx.x, lane = r % 32, warps = (int)blockDim.x / 32 - 1;
  const bool feeder = r >= (int)blockDim.x - 32;
  if (r == 0) {
    s_chain = nchains - 1 - atomicAdd(ticket, 1);
    s_ok = joined[s_chain] ? chain_wait(flags + s_chain) : 1;
  }
  __syncthreads();
  const int chain = s_chain, p0 = cptr[chain], len = cptr[chain + 1] - p0, b0 = bptr[chain];
  const int nblk = bptr[chain + 1] - b0;
  panels += b0 * (size_t)xd_panel_size(F);
  blocks += (size_t)b0 * kBlockInts;
  y += x0 + p0;
  if (feeder) {
    for (int t = nblk - 1; t > nblk - kSolveAhead; --t) s.fetch(t, nblk, len, F, 0, panels, blocks, y, lane);
    asm volatile("cp.async.wait_group %0;" ::"n"(kSolveAhead - 2) : "memory");
  }
  double w = 0.0;
  if (r < F) {
    const int at = border[(size_t)chain * F + r];
    if (at >= 0) w = s_ok ? __ldcg(x + at) : __longlong_as_double(-1LL);
  }
  __syncthreads();
  for (int t = nblk - 1; t >= 0; --t) {
    const int q = t % kSolveAhead, nb = min(kB, len - t * kB);
    const int *rec = s.rec + q * kBlockInts;
    const int j0 = rec[kB + 1], j1 = rec[kB + 2];
    double *red = s.red + (t & 1) * kB * (kMaxFrame / 32);
    BlockRegs g;
    int mine = -1;
    if (!feeder) {
      mine = pivot_of(rec, r);
      if (mine >= 0) w = 0.0;  // the pivots' own slots: not solved yet
      g.load(s, q, F, r, nb);
      double acc[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) acc[j] = j < nb ? g.pan[j] * w : 0.0;
      // Eight sums over 32 lanes: halve the values held while halving the lanes they come from.
#pragma unroll
      for (int h = 4; h > 0; h >>= 1) {
        const int bit = h * 4;
        const bool up = lane & bit;
#pragma unroll
        for (int j = 0; j < h; ++j) {
          const double keep = up ? acc[j + h] : acc[j], give = up ? acc[j] : acc[j + h];
          acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
        }
      }
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
      if ((lane & 3) == 0) red[r / 32 * kB + (lane >> 4 & 1) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1)] = acc[0];
    } else {
      asm volatile("cp.async.wait_group %0;" ::"n"(kSolveAhead - 3) : "memory");
    }
    __syncthreads();
    if (feeder) {
      s.fetch(t - kSolveAhead + 1, nblk, len, F, 0, panels, blocks, y, lane);
    } else {
      double v[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) v[j] = g.rhs[j] - red[j];
      for (int k = 1; k < warps; ++k)
#pragma unroll
        for (int j = 0; j < kB; ++j) v[j] -= red[k * kB + j];
#pragma unroll
      for (int j = kB - 1; j >= 0; --j) {
        v[j] = j >= nb ? 0.0 : DIVIDE ? v[j] / g.d[j][j] : v[j] * g.d[j][j];
#pragma unroll
        for (int i = 0; i < j; ++i) v[i] = fma(-g.d[i][j], v[j], v[i]);
      }
      if (mine >= 0) {
        w = pick(v, mine);
        const int at = x0 + p0 + t * kB + mine, to = xdst[at];
        __stcg(x + at, w);
        if (to >= 0) out[to] = w;
      }
    }
    if (j0 < j1) {  // child chains start from here
      __threadfence();
      __syncthreads();
      for (int j = j0 + r; j < j1; j += blockDim.x) atomicExch(flags + jchild[j], 1);
    }
  }
}

// Rows solved last (nobody reads their values, and one may hold an entry for every device of a
// supply): a block per kTailChunk entries; the block that finishes a row's last chunk adds the
// chunks' sums in order. A top row has its panel's part in xs already.
__global__ void __launch_bounds__(256) tree_tail_kernel(const int4 *__restrict__ chunk, const int4 *__restrict__ tail,
                                                        int nbot, const int *__restrict__ tcol, const double *vt,
                                                        const double *v, const double *y, const double *xs,
                                                        const int *__restrict__ xdst, double *part, int *done,
                                                        double *out) {
  __shared__ double red[8];
  const int lane = threadIdx.x % 32;
  const int4 c = chunk[blockIdx.x], row = tail[c.x];
  double acc = 0.0;
  for (int e = c.y + threadIdx.x; e < c.z; e += 256) acc += vt[e] * xs[tcol[e]];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) red[threadIdx.x / 32] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    acc = 0.0;
    for (int w = 0; w < 8; ++w) acc += red[w];
    if (row.w > 1) {
      __stcg(part + row.z + c.w, acc);
      __threadfence();
      if (atomicAdd(done + c.x, 1) < row.w - 1) return;
      __threadfence();
      acc = 0.0;
      for (int k = 0; k < row.w; ++k) acc += __ldcg(part + row.z + k);
    }
    const double p = v[row.y];
    out[~xdst[row.x]] = row.x < nbot ? (y[row.x] - acc) / p : xs[row.x] - acc / p;
  }
}

// The bottom groups' lists with positions among the group's own entries (gpos, in order of first use)
// where those fit shared memory, else unchanged.
struct BottomLists {
  std::vector<int> gptr, gpos;
  std::vector<XdPos2> div;
  std::vector<XdPos4> dst, pairs;
  size_t most = 0;
};

BottomLists bottom_lists(const XdTreePlan &p) {
  BottomLists b;
  b.gptr.assign(1, 0);
  b.div = p.div;
  b.dst = p.dst;
  b.pairs = p.pairs;
  std::vector<int> local((size_t)p.nv, -1);
  for (int g = 0; g < p.ngroups; ++g) {
    const int l0 = p.glev[g], l1 = p.glev[g + 1];
    std::vector<int> used;
    auto at = [&](int &pos, bool set) {
      if (!set && local[pos] < 0) {
        local[pos] = (int)used.size();
        used.push_back(pos);
      }
      if (set) pos = local[pos];
    };
    auto walk = [&](bool set) {
      for (int d = p.ldst[l0]; d < p.ldst[l1]; ++d) {
        XdPos4 &ds = b.dst[d];
        at(ds.x, set);
        if (ds.w >= 0) {
          at(ds.y, set);
          at(ds.z, set);
          at(ds.w, set);
        } else {
          for (int k = ds.y; k < ds.y + ds.z; ++k) {
            at(b.pairs[k].x, set);
            at(b.pairs[k].y, set);
            at(b.pairs[k].z, set);
          }
        }
      }
      for (int d = p.ldiv[l0]; d < p.ldiv[l1]; ++d) {
        at(b.div[d].x, set);
        at(b.div[d].y, set);
      }
    };
    walk(false);
    if (used.size() <= (size_t)kBottomEntries) {
      walk(true);
      b.gpos.insert(b.gpos.end(), used.begin(), used.end());
      b.most = std::max(b.most, used.size());
    }
    b.gptr.push_back((int)b.gpos.size());
    for (int pos : used) local[pos] = -1;
  }
  return b;
}

template <class D, class T>
cudaError_t upload(D **d, const std::vector<T> &h) {
  static_assert(sizeof(D) == sizeof(T), "device and host records match");
  cudaError_t e = cudaMalloc(d, std::max<size_t>(1, h.size()) * sizeof(T));
  if (e != cudaSuccess || h.empty()) return e;
  return cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
}

}  // namespace

int xd_tree_upload(XdTree *t, const XdTreePlan &p, const int *perm_p, const int *perm_q) {
  t->n = p.n;
  t->F = p.F;
  t->ntop = p.ntop;
  t->ngroups = p.ngroups;
  t->nchains = p.nchains;
  t->nsd = (int)p.sdst.size();
  t->ntdiv = (int)p.tdiv.size();
  t->p0 = p.p0;
  t->nv = p.nv;
  t->nbot = p.nbot;
  t->ntail = (int)p.tail.size();
  t->l0 = p.l0;
  t->u0 = p.u0;
  t->t0 = p.t0;
  t->d0 = p.d0;
  std::vector<int> bsrc(p.n), xdst(p.n), joined(std::max(1, p.nchains), 0);
  for (int x = 0; x < p.n; ++x) {
    bsrc[x] = perm_p[p.order[x]];
    xdst[x] = perm_q[p.order[x]];
  }
  const BottomLists bottom = bottom_lists(p);
  t->bottom_smem = sizeof(double) * bottom.most;
  std::vector<int> grow(1, 0);
  size_t most = 0;
  for (int g = 0; g < p.ngroups; ++g) {
    grow.push_back(p.lrow[p.glev[g + 1]]);
    const size_t rows = grow[g + 1] - grow[g];
    if (rows <= (size_t)kPassRows) most = std::max(most, rows);
  }
  t->pass_smem = sizeof(double) * most;
  std::vector<XdPos4> tail, chunk;
  for (int r = 0; r < t->ntail; ++r) {
    const int x = p.tail[r], first = (int)chunk.size();
    xdst[x] = ~xdst[x];
    for (int e = p.tptr[r]; e < p.tptr[r + 1]; e += kTailChunk)
      chunk.push_back({r, e, std::min(e + kTailChunk, p.tptr[r + 1]), (int)chunk.size() - first});
    tail.push_back({x, p.diag[p.order[x]], first, (int)chunk.size() - first});
  }
  t->nchunk = (int)chunk.size();
  for (size_t k = 0; k + 1 < p.sptr.size(); ++k) t->schur_long = t->schur_long || p.sptr[k + 1] - p.sptr[k] > kSchurLong;
  for (size_t k = 0; k + 1 < p.lptr.size(); ++k) t->row_long = t->row_long || p.lptr[k + 1] - p.lptr[k] > kTopRowLong;
  for (int u = 0; u < 2; ++u)
    for (const XdPos4 &q : (u ? p.bwd : p.fwd).pass) t->pass_long[u] = t->pass_long[u] || (q.y >> 16 & 0xff) > 5;
  auto pass_attribute = [](auto *kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(double) * kPassRows);
  };
  for (int c : p.jchild) joined[c] = 1;
  cudaError_t e;
  auto upload_passes = [](XdTree::Passes &d, const XdPasses &h) {
    cudaError_t e = upload(&d.gptr, h.gptr);
    if (e == cudaSuccess) e = upload(&d.pass, h.pass);
    if (e == cudaSuccess) e = upload(&d.rows, h.rows);
    if (e == cudaSuccess) e = upload(&d.col, h.col);
    return e;
  };
  if ((e = upload_passes(t->d_fwd, p.fwd)) != cudaSuccess || (e = upload_passes(t->d_bwd, p.bwd)) != cudaSuccess ||
      (e = upload(&t->d_lptr, p.lptr)) != cudaSuccess || (e = upload(&t->d_lcol, p.lcol)) != cudaSuccess ||
      (e = upload(&t->d_tcol, p.tcol)) != cudaSuccess || (e = upload(&t->d_chunk, chunk)) != cudaSuccess ||
      (e = upload(&t->d_tail, tail)) != cudaSuccess || (e = upload(&t->d_bsrc, bsrc)) != cudaSuccess ||
      (e = upload(&t->d_xdst, xdst)) != cudaSuccess || (e = upload(&t->d_joined, joined)) != cudaSuccess ||
      (e = upload(&t->d_border, p.border)) != cudaSuccess || (e = upload(&t->d_grow, grow)) != cudaSuccess ||
      (e = pass_attribute(tree_pass_kernel<false, false>)) != cudaSuccess ||
      (e = pass_attribute(tree_pass_kernel<true, false>)) != cudaSuccess ||
      (e = pass_attribute(tree_pass_kernel<false, true>)) != cudaSuccess ||
      (e = pass_attribute(tree_pass_kernel<true, true>)) != cudaSuccess ||
      (e = cudaMalloc(&t->d_y, sizeof(double) * std::max(1, p.n))) != cudaSuccess ||
      (e = cudaMalloc(&t->d_x, sizeof(double) * std::max(1, p.n))) != cudaSuccess ||
      (e = cudaMalloc(&t->d_wbuf, sizeof(double) * std::max<size_t>(1, (size_t)p.nchains * p.F))) != cudaSuccess ||
      (e = cudaMalloc(&t->d_part, sizeof(double) * std::max(1, t->nchunk))) != cudaSuccess ||
      (e = cudaMalloc(&t->d_sctl, sizeof(int) * (2 + 2 * p.nchains + t->ntail))) != cudaSuccess ||
      (e = cudaMalloc(&t->d_v, sizeof(double) * std::max<long long>(1, p.nv))) != cudaSuccess ||
      (e = upload(&t->d_diag, p.diag)) != cudaSuccess || (e = upload(&t->d_glev, p.glev)) != cudaSuccess ||
      (e = upload(&t->d_ldiv, p.ldiv)) != cudaSuccess || (e = upload(&t->d_ldst, p.ldst)) != cudaSuccess ||
      (e = upload(&t->d_div, bottom.div)) != cudaSuccess || (e = upload(&t->d_dst, bottom.dst)) != cudaSuccess ||
      (e = upload(&t->d_gptr, bottom.gptr)) != cudaSuccess || (e = upload(&t->d_gpos, bottom.gpos)) != cudaSuccess ||
      (p.any_long && (e = upload(&t->d_llong, p.llong)) != cudaSuccess) ||
      (e = cudaFuncSetAttribute(tree_bottom_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(double) * kBottomEntries)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(tree_bottom_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(double) * kBottomEntries)) != cudaSuccess ||
      (e = upload(&t->d_pairs, bottom.pairs)) != cudaSuccess || (e = upload(&t->d_sdst, p.sdst)) != cudaSuccess ||
      (e = upload(&t->d_sptr, p.sptr)) != cudaSuccess || (e = upload(&t->d_spairs, p.spairs)) != cudaSuccess ||
      (e = upload(&t->d_tdiv, p.tdiv)) != cudaSuccess || (e = upload(&t->d_cptr, p.cptr)) != cudaSuccess ||
      (e = upload(&t->d_bptr, p.bptr)) != cudaSuccess || (e = upload(&t->d_blocks, p.blocks)) != cudaSuccess ||
      (e = upload(&t->d_jchild, p.jchild)) != cudaSuccess || (e = upload(&t->d_jmap, p.jmap)) != cudaSuccess ||
      (e = cudaMalloc(&t->d_jbuf, sizeof(double) * std::max<size_t>(1, (size_t)p.nchains * p.F * p.F))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(tree_top_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)Frame::bytes(kMaxFrame))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(tree_top_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)Frame::bytes(kMaxFrame))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(tree_forward_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)SolveSmem::bytes(kMaxFrame))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(tree_backward_chain_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)SolveSmem::bytes(kMaxFrame))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(tree_backward_chain_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)SolveSmem::bytes(kMaxFrame))) != cudaSuccess ||
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
                  (void *)t->d_jchild, (void *)t->d_jmap, (void *)t->d_jbuf, (void *)t->d_ctl, (void *)t->d_fwd.gptr,
                  (void *)t->d_fwd.pass, (void *)t->d_fwd.rows, (void *)t->d_fwd.col, (void *)t->d_bwd.gptr,
                  (void *)t->d_bwd.pass, (void *)t->d_bwd.rows, (void *)t->d_bwd.col, (void *)t->d_lptr,
                  (void *)t->d_lcol, (void *)t->d_tcol, (void *)t->d_chunk, (void *)t->d_tail, (void *)t->d_bsrc,
                  (void *)t->d_xdst, (void *)t->d_joined, (void *)t->d_border, (void *)t->d_y, (void *)t->d_x,
                  (void *)t->d_wbuf, (void *)t->d_part, (void *)t->d_sctl, (void *)t->d_grow, (void *)t->d_gptr,
                  (void *)t->d_gpos, (void *)t->d_llong})
    cudaFree(p);
  *t = XdTree();
}

int xd_tree_factor(XdTree *t, cudaStream_t st) {
  if (t->ngroups > 0)
    (t->d_llong ? tree_bottom_kernel<true> : tree_bottom_kernel<false>)<<<t->ngroups, kBottomThreads, t->bottom_smem, st>>>(
        t->d_glev, t->d_ldiv, t->d_ldst, t->d_llong, t->d_div, t->d_dst, t->d_pairs, t->d_gptr, t->d_gpos, t->d_v);
  if (t->nsd > 0) {
    const long long threads = (long long)t->nsd * kSchurLanes;
    (t->schur_long ? tree_schur_kernel<true> : tree_schur_kernel<false>)<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(t->nsd, t->d_sdst, t->d_sptr, t->d_spairs,
                                                                         t->d_v);
  }
  if (t->nchains > 0) {
    (t->divide ? tree_top_kernel<true> : tree_top_kernel<false>)<<<t->nchains, kTopThreads, Frame::bytes(t->F), st>>>(
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

int xd_tree_solve(XdTree *t, double *d_x, cudaStream_t st) {
  cudaError_t e;
  const int n = t->n, nc = t->nchains;
  const double *v = t->d_v;
  if (nc + t->ntail > 0 &&
      (e = cudaMemsetAsync(t->d_sctl, 0, sizeof(int) * (2 + 2 * nc + t->ntail), st)) != cudaSuccess)
    return xd_internal_fail(-3, std::string("triangular solve: ") + cudaGetErrorString(e));
  tree_rhs_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, t->d_bsrc, d_x, t->d_y);
  if (t->ngroups > 0)
    (t->pass_long[0] ? tree_pass_kernel<false, true> : tree_pass_kernel<false, false>)<<<t->ngroups, kPassThreads, t->pass_smem, st>>>(t->d_fwd.gptr, t->d_fwd.pass, t->d_fwd.rows,
                                                                 t->d_fwd.col, 0, v, nullptr, t->d_y, t->d_y, nullptr,
                                                                 nullptr, t->d_grow);
  if (nc > 0) {
    const int threads = (t->F + 31) / 32 * 32 + 32;
    (t->row_long ? tree_top_rows_kernel<true> : tree_top_rows_kernel<false>)<<<(t->ntop + 7) / 8, 256, 0, st>>>(t->nbot, n, t->d_lptr, t->d_lcol, v + t->l0, t->d_y);
    tree_forward_chain_kernel<<<nc, threads, SolveSmem::bytes(t->F), st>>>(
        t->F, t->d_cptr, t->d_bptr, t->d_blocks, t->d_jchild, t->d_jmap, t->d_wbuf, v + t->p0, t->d_y + t->nbot,
        t->d_sctl, t->d_sctl + 2);
    (t->divide ? tree_backward_chain_kernel<true> : tree_backward_chain_kernel<false>)<<<nc, threads, SolveSmem::bytes(t->F), st>>>(
        nc, t->F, t->d_cptr, t->d_bptr, t->d_blocks, t->d_jchild, t->d_border, v + t->p0, t->d_y, t->nbot, t->d_x,
        t->d_xdst, d_x, t->d_sctl + 1, t->d_sctl + 2 + nc, t->d_joined);
  }
  if (t->ngroups > 0)
    (t->pass_long[1] ? tree_pass_kernel<true, true> : tree_pass_kernel<true, false>)<<<t->ngroups, kPassThreads, t->pass_smem, st>>>(t->d_bwd.gptr, t->d_bwd.pass, t->d_bwd.rows,
                                                                t->d_bwd.col, t->u0, v, v + t->d0, t->d_y, t->d_x,
                                                                t->d_xdst, d_x, t->d_grow);
  if (t->nchunk > 0)
    tree_tail_kernel<<<t->nchunk, 256, 0, st>>>(t->d_chunk, t->d_tail, t->nbot, t->d_tcol, v + t->t0, v, t->d_y, t->d_x,
                                                t->d_xdst, t->d_part, t->d_sctl + 2 + 2 * nc, d_x);
  if ((e = cudaGetLastError()) != cudaSuccess)
    return xd_internal_fail(-3, std::string("triangular solve launch: ") + cudaGetErrorString(e));
  return 0;
}
