// Tensor-core kernels of the learned surrogate (include/xyce_surrogate.h): a BF16 GEMM on the
// 5th-generation tensor cores (tcgen05.mma, FP32 accumulator in tensor memory) with the fused
// epilogues the surrogate's forward and backward passes need, and the small kernels around it
// (loss gradient, bias gradient, split-K reduction, Adam).
//
// GEMM: C[M x N] = A[M x K] * B[N x K]^T, A and B row-major BF16 with K contiguous (K-major
// operands), M a multiple of 128, N = 16 or 128 per tile, K a multiple of 16. One CTA of 128
// threads computes one 128 x N tile over a K range (the whole K, or one split-K slice):
//   * warp 0 allocates N tensor-memory columns (lane m <-> row m of the tile);
//   * per K chunk of 64, all threads copy the A and B sub-tiles from global memory into shared
//     memory in the tensor core's no-swizzle K-major layout (8-row x 16-byte core matrices;
//     consecutive K core matrices 128 B apart, consecutive 8-row groups 1024 B apart);
//   * after a proxy fence and a barrier, one thread issues 4 tcgen05.mma (K = 16 each) and a
//     tcgen05.commit to an mbarrier; every thread waits on it (bounded) before the next chunk
//     overwrites shared memory;
//   * the epilogue reads the accumulator with tcgen05.ld (warp w reads lanes 32w..32w+31, so
//     thread t owns row 32w + t), applies the fused operation and writes global memory.
// Every wait on the mbarrier has an iteration limit; on expiry the kernel records an error code
// in a device flag, stops issuing work, waits (again bounded) for its own in-flight MMA, frees
// its tensor memory and returns, so the context stays usable and the host reports the failure.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/xyce_surrogate.h"

int xd_internal_fail(int code, const std::string &msg);

namespace {

constexpr int kThreads = 128;
constexpr int kTileM = 128;
constexpr int kChunkK = 64;
constexpr long long kSpinLimit = 20000000;  // mbarrier polls before a wait is declared failed

// ---- tcgen05 / mbarrier primitives (inline PTX) ------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Returns true once the barrier's phase `parity` has completed, false after kSpinLimit polls.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  const uint32_t a = smem_u32(bar);
  for (long long i = 0; i < kSpinLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Shared-memory matrix descriptor: no swizzle, K-major canonical layout. Fields (bit ranges):
// start address >> 4 [0,14), leading-dimension byte offset >> 4 [16,30) (distance between core
// matrices adjacent in K), stride-dimension byte offset >> 4 [32,46) (distance between 8-row
// groups), descriptor version 1 [46,48), base offset 0, layout type 0 (no swizzle) [61,64).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor, kind::f16: D format F32 [4,6) = 1, A format BF16 [7,10) = 1, B format
// BF16 [10,13) = 1, both K-major (bits 15, 16 = 0), N >> 3 at [17,23), M >> 4 at [24,29).
__host__ __device__ constexpr uint32_t instr_desc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      :
      : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp receives lane (base lane + t).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- epilogues -------------------------------------------------------------------------------

// SiLU and its derivative with the fast exponential and approximate division: the surrogate is
// not held to bit parity with a CPU (its outputs only seed Newton iterations).
__device__ __forceinline__ float silu(float z) { return __fdividef(z, 1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = __fdividef(1.0f, 1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// Byte offset of element (row r, column k) of a rows x kChunkK bf16 tile in the no-swizzle
// K-major layout: 8 x 8 core matrices of 128 B, K-adjacent ones 128 B apart, row groups 1024 B.
__device__ __forceinline__ uint32_t tile_off(int r, int kc) {
  return (uint32_t)((r >> 3) * 1024 + kc * 128 + (r & 7) * 16);
}

template <int TN>
__global__ void __launch_bounds__(kThreads) gemm_bf16_tc_kernel(xd_gemm_args g, int k_per_split) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // Layout: [A tile 128 x 64 bf16 = 16 KB][B tile TN x 64 bf16][mbarrier][tmem address]
  unsigned char *sA = smem_raw;
  unsigned char *sB = smem_raw + kTileM * kChunkK * 2;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sB + TN * kChunkK * 2);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar + 1);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int m0 = blockIdx.x * kTileM;
  const int n0 = blockIdx.y * TN;
  const int split = blockIdx.z;
  const int k_begin = split * k_per_split;
  int k_end = k_begin + k_per_split;
  if (k_end > g.K) k_end = g.K;
  constexpr uint32_t kCols = TN < 32 ? 32 : TN;  // allocation granularity is 32 columns

  if (warp == 0) tmem_alloc(tmem_slot, kCols);
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t idesc = instr_desc_bf16(kTileM, TN);
  const __nv_bfloat16 *A = static_cast<const __nv_bfloat16 *>(g.A);
  const __nv_bfloat16 *B = static_cast<const __nv_bfloat16 *>(g.B);
  __nv_bfloat16 *Zo = static_cast<__nv_bfloat16 *>(g.Z);
  __nv_bfloat16 *Ho = static_cast<__nv_bfloat16 *>(g.H);
  __nv_bfloat16 *HTo = static_cast<__nv_bfloat16 *>(g.HT);
  const __nv_bfloat16 *Zi = static_cast<const __nv_bfloat16 *>(g.Zin);

  uint32_t phase = 0;
  bool ok = true;
  int issued = 0;
  for (int k0 = k_begin; k0 < k_end && ok; k0 += kChunkK) {
    const int kc_n = min(kChunkK, k_end - k0) / 8;  // 8-element K chunks in this step (2, 4, 6 or 8)
    // Copy A (128 rows) and B (TN rows) sub-tiles: one 16-byte core-matrix row per copy.
    for (int i = tid; i < kTileM * kc_n; i += kThreads) {
      const int r = i / kc_n, kc = i % kc_n;
      const int gr = m0 + r;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (gr < g.M) v = *reinterpret_cast<const uint4 *>(A + (size_t)gr * g.lda + k0 + kc * 8);
      *reinterpret_cast<uint4 *>(sA + tile_off(r, kc)) = v;
    }
    for (int i = tid; i < TN * kc_n; i += kThreads) {
      const int r = i / kc_n, kc = i % kc_n;
      const int gr = n0 + r;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (gr < g.N) v = *reinterpret_cast<const uint4 *>(B + (size_t)gr * g.ldb + k0 + kc * 8);
      *reinterpret_cast<uint4 *>(sB + tile_off(r, kc)) = v;
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0) {
      const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
      for (int s = 0; s < kc_n / 2; ++s) {
        const uint64_t ad = smem_desc(a0 + s * 256, 128, 1024);
        const uint64_t bd = smem_desc(b0 + s * 256, 128, 1024);
        mma_bf16(tmem, ad, bd, idesc, (issued > 0 || s > 0) ? 1u : 0u);
      }
      mma_commit(bar);
    }
    ++issued;
    ok = __syncthreads_and(mbar_wait(bar, phase)) != 0;  // uniform across the CTA
    phase ^= 1u;
    tc_fence_after();
  }
  if (!ok) {
    // A wait expired: record it and drain (bounded) before releasing tensor memory.
    if (tid == 0) atomicExch(g.err, 1);
    mbar_wait(bar, phase ^ 1u);
  }
  // Epilogue: thread t of warp w owns tile row 32w + t (tensor-memory lane 32w + t).
  const int row = m0 + warp * 32 + (tid & 31);
  const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
  if (ok && issued > 0) {
#pragma unroll
    for (int c0 = 0; c0 < TN; c0 += (TN >= 32 ? 32 : 16)) {
      float v[32];
      if constexpr (TN >= 32) {
        tmem_ld32(lane_base + c0, v);
      } else {
        float w16[16];
        tmem_ld16(lane_base + c0, w16);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = w16[i];
      }
      constexpr int W = TN >= 32 ? 32 : 16;
      if (row < g.M) {
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const int n = n0 + c0 + i;
          if (n >= g.N) continue;
          float acc = v[i];
          switch (g.epilogue) {
            case XD_EPI_F32: {
              g.C32[(size_t)split * g.M * g.ldc + (size_t)row * g.ldc + n] = acc;
              break;
            }
            case XD_EPI_BIAS_F32: {
              g.C32[(size_t)row * g.ldc + n] = acc + g.bias[n];
              break;
            }
            case XD_EPI_BIAS_SILU: {
              const float z = acc + g.bias[n];
              const float h = silu(z);
              Zo[(size_t)row * g.ldc + n] = __float2bfloat16(z);
              Ho[(size_t)row * g.ldc + n] = __float2bfloat16(h);
              if (HTo) HTo[(size_t)n * g.ldt + row] = __float2bfloat16(h);
              break;
            }
            case XD_EPI_SILU_BACK: {
              const float z = __bfloat162float(Zi[(size_t)row * g.ldc + n]);
              const float d = acc * silu_grad(z);
              Ho[(size_t)row * g.ldc + n] = __float2bfloat16(d);
              if (HTo) HTo[(size_t)n * g.ldt + row] = __float2bfloat16(d);
              break;
            }
            default:
              break;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_free(tmem, kCols);
}

// ---- small kernels ---------------------------------------------------------------------------

// Mean-squared-error gradient of the network output (fp32 [M x ld]) against targets, written as
// BF16 in both layouts for the backward GEMMs, and the per-sample squared error.
__global__ void mse_grad_kernel(int M, int n_out, int ld, const float *__restrict__ y, const float *__restrict__ t,
                                float scale, __nv_bfloat16 *__restrict__ dz, __nv_bfloat16 *__restrict__ dzt,
                                int ldt, float *__restrict__ sq) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= M) return;
  float s = 0.0f;
  for (int n = 0; n < ld; ++n) {
    float d = 0.0f;
    if (n < n_out) {
      const float e = y[(size_t)row * ld + n] - t[(size_t)row * n_out + n];
      s += e * e;
      d = scale * e;
    }
    dz[(size_t)row * ld + n] = __float2bfloat16(d);
    dzt[(size_t)n * ldt + row] = __float2bfloat16(d);
  }
  if (sq) sq[row] = s;
}

// out[n] = sum over `count` rows of in[r * ld + n], one block per column, fixed reduction tree.
__global__ void column_sum_kernel(int rows, int cols, const float *__restrict__ in, int ld, float *__restrict__ out) {
  __shared__ float red[256];
  const int n = blockIdx.x;
  float acc = 0.0f;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) acc += in[(size_t)r * ld + n];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0 && n < cols) out[n] = red[0];
}

// Bias gradient: sum over the batch of the transposed BF16 gradient rows dzt[n][0..M).
__global__ void bias_grad_kernel(int M, int N, const __nv_bfloat16 *__restrict__ dzt, int ldt,
                                 float *__restrict__ db) {
  __shared__ float red[256];
  const int n = blockIdx.x;
  float acc = 0.0f;
  for (int r = threadIdx.x; r < M; r += blockDim.x) acc += __bfloat162float(dzt[(size_t)n * ldt + r]);
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0 && n < N) db[n] = red[0];
}

// Sums split-K partials part[s][i] for s = 0..splits-1 in order.
__global__ void splitk_sum_kernel(int n, int splits, const float *__restrict__ part, float *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float acc = 0.0f;
  for (int s = 0; s < splits; ++s) acc += part[(size_t)s * n + i];
  out[i] = acc;
}

// Adam on FP32 master parameters; refreshes the BF16 copies (row-major and, for matrices, the
// transpose used by the backward GEMM).
__global__ void adam_kernel(int rows, int cols, float *__restrict__ p, const float *__restrict__ grad,
                            float *__restrict__ m, float *__restrict__ v, float lr, float b1, float b2, float eps,
                            float c1, float c2, __nv_bfloat16 *__restrict__ p16, __nv_bfloat16 *__restrict__ p16t,
                            int ld16, int ld16t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * cols) return;
  const int r = i / cols, c = i % cols;
  const float gr = grad[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gr;
  const float vi = b2 * v[i] + (1.0f - b2) * gr * gr;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  if (p16) p16[(size_t)r * ld16 + c] = __float2bfloat16(pi);
  if (p16t) p16t[(size_t)c * ld16t + r] = __float2bfloat16(pi);
}

// First layer in FP32 on the CUDA cores: the network inputs (biases in volts, log-geometry) keep
// full precision, which BF16 (8-bit mantissa, ~4 mV at 1 V) would not give them. One thread per
// (sample, hidden unit): z = W1[u] . x + b1[u]; writes Z, H = silu(z) (BF16) and H transposed.
__global__ void input_layer_kernel(int M, int n_in, int n_hid, const float *__restrict__ x, int ldx,
                                   const float *__restrict__ w1, int ldw, const float *__restrict__ b1,
                                   __nv_bfloat16 *__restrict__ Z, __nv_bfloat16 *__restrict__ H,
                                   __nv_bfloat16 *__restrict__ HT, int ldt) {
  const int u = threadIdx.x;  // hidden unit
  const int row = blockIdx.x;
  if (u >= n_hid || row >= M) return;
  float z = b1[u];
  for (int i = 0; i < n_in; ++i) z += w1[u * ldw + i] * x[(size_t)row * ldx + i];
  const float h = silu(z);
  Z[(size_t)row * n_hid + u] = __float2bfloat16(z);
  H[(size_t)row * n_hid + u] = __float2bfloat16(h);
  if (HT) HT[(size_t)u * ldt + row] = __float2bfloat16(h);
}

// First-layer weight gradient in FP32: gw[u][i] = sum_r dzt[u][r] * x[r][i] for i < n_in, one
// block per hidden unit, fixed reduction tree.
__global__ void input_grad_kernel(int M, int n_in, const __nv_bfloat16 *__restrict__ dzt, int ldt,
                                  const float *__restrict__ x, int ldx, float *__restrict__ gw, int ldw) {
  __shared__ float red[8][256];
  const int u = blockIdx.x;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
  for (int r = threadIdx.x; r < M; r += blockDim.x) {
    const float d = __bfloat162float(dzt[(size_t)u * ldt + r]);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n_in) acc[i] += d * x[(size_t)r * ldx + i];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[i][threadIdx.x] = acc[i];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
#pragma unroll
      for (int i = 0; i < 8; ++i) red[i][threadIdx.x] += red[i][threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x < n_in) gw[u * ldw + threadIdx.x] = red[threadIdx.x][0];
}

// Surrogate inputs for circuit instances idx[k]: terminal voltages from the solution (ground ->
// 0), differences to the source, scaled by 1 / vmax, then the instance's scaled log W and log L.
__global__ void surrogate_features_kernel(int n, const int *__restrict__ idx, const int *__restrict__ nodes4,
                                          const double *__restrict__ sol, const float *__restrict__ geom2,
                                          float inv_vmax, float *__restrict__ x, int ldx) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int i = idx[k];
  double v[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int nd = nodes4[4 * i + t];
    v[t] = nd >= 0 ? sol[nd] : 0.0;
  }
  x[(size_t)k * ldx + 0] = (float)((v[1] - v[2]) * inv_vmax);  // Vgs
  x[(size_t)k * ldx + 1] = (float)((v[0] - v[2]) * inv_vmax);  // Vds
  x[(size_t)k * ldx + 2] = (float)((v[3] - v[2]) * inv_vmax);  // Vbs
  x[(size_t)k * ldx + 3] = geom2[2 * i];
  x[(size_t)k * ldx + 4] = geom2[2 * i + 1];
}

// Decodes the surrogate's outputs y = asinh(value / scale) for instances idx[k] and stages the
// terminal currents and charges in the exact load's slot layout (slot-major, 16 x n_inst):
// F = (Id, 0, -Id, 0) at (D, G, S, B), Q = (Qd, Qg, -(Qg + Qd + Qb), Qb), limiter slots zero.
__global__ void surrogate_stage_kernel(int n, const int *__restrict__ idx, const float *__restrict__ y, int ldy,
                                       const float *__restrict__ out_scale, int n_inst, double *__restrict__ stage) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int i = idx[k];
  const float *yr = y + (size_t)k * ldy;
  const double id = sinh((double)yr[0]) * out_scale[0];
  const double qg = sinh((double)yr[1]) * out_scale[1];
  const double qd = sinh((double)yr[2]) * out_scale[2];
  const double qb = sinh((double)yr[3]) * out_scale[3];
  const size_t N = (size_t)n_inst;
  stage[0 * N + i] = id;
  stage[1 * N + i] = 0.0;
  stage[2 * N + i] = -id;
  stage[3 * N + i] = 0.0;
  stage[4 * N + i] = qd;
  stage[5 * N + i] = qg;
  stage[6 * N + i] = -(qg + qd + qb);
  stage[7 * N + i] = qb;
#pragma unroll
  for (int s = 8; s < 16; ++s) stage[s * N + i] = 0.0;
}

// ---- fused inference: the whole 5 -> 128 -> 128 -> 128 -> 128 -> 16 network in one kernel -----

constexpr int kFusedThreads = 256;  // 8 warps: two per tensor-memory lane quarter
constexpr int kHid = 128;
constexpr int kOutPad = 16;
// Shared-memory layout of a 128-row x 128-K BF16 operand: 8 x 8 core matrices, K-adjacent ones
// 128 B apart, 8-row groups 2048 B apart.
__device__ __forceinline__ uint32_t off128(int r, int kc) {
  return (uint32_t)((r >> 3) * 2048 + kc * 128 + (r & 7) * 16);
}

// A block works on kFwdGroups tiles at a time, a group of kFusedThreads threads each with its own
// activation tile, tensor-memory columns and barriers over the shared weights: one group's tensor-core
// products and waits run under the other's epilogues, whose exponentials and reciprocals (two of the
// 16-a-clock special-function operations per activation, 55 us for 250k samples on 148 SMs) are
// the bound. 250k samples take 120 us, 1M 398 us (two groups: 131 and 459; one group, without the
// next tile's inputs and the weights' copies in flight: 297 us and 1.85 ms).
constexpr int kFwdGroups = 3;
struct FusedSmem {
  unsigned char w[3][kHid * kHid * 2];   // hidden layers 2..4, [out][in] K-major
  unsigned char w5[kOutPad * kHid * 2];  // output layer, 16 x 128
  unsigned char act[kFwdGroups][kHid * kHid * 2];  // activation tiles (A operands), 128 x 128
  float w1[kHid * 8];                    // first layer, FP32, 128 x n_in (n_in <= 8)
  float b[4 * kHid + kOutPad];           // biases of layers 1..5
  uint64_t bar[kFwdGroups];
  uint32_t tmem;
};
static_assert(sizeof(FusedSmem) <= 227 * 1024, "one block's shared memory");

// First layer of eight hidden units from u on, on the CUDA cores (FP32, inputs added in order).
template <int NIN>
__device__ __forceinline__ void first_layer8(const float *w1, const float *b, const float (&xi)[8], int n_in, bool on,
                                             __nv_bfloat16 (&h8)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float z = b[j];
    float w[8];
    *reinterpret_cast<float4 *>(w) = *reinterpret_cast<const float4 *>(w1 + j * 8);
    *reinterpret_cast<float4 *>(w + 4) = *reinterpret_cast<const float4 *>(w1 + j * 8 + 4);
    if constexpr (NIN > 0) {
#pragma unroll
      for (int i = 0; i < NIN; ++i) z += w[i] * xi[i];
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < n_in) z += w[i] * xi[i];
    }
    h8[j] = __float2bfloat16(on ? silu(z) : 0.0f);
  }
}

template <int NIN>
__global__ void __launch_bounds__(kFwdGroups *kFusedThreads, 1) mlp_forward_fused_kernel(xd_mlp_net net, int n,
                                                                                        const float *x, int ldx,
                                                                                        float *y, int ldy, int *err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  FusedSmem &S = *reinterpret_cast<FusedSmem *>(smem_raw);
  constexpr int kAll = kFwdGroups * kFusedThreads;
  const int group = threadIdx.x / kFusedThreads, tid = threadIdx.x % kFusedThreads, warp = tid >> 5, lane = tid & 31;
  // Stage the weights once per CTA, under the first tiles' first layer.
  auto stage = [&](unsigned char *dst, const void *src, int rows) {
    const __nv_bfloat16 *W = static_cast<const __nv_bfloat16 *>(src);
    for (int i = threadIdx.x; i < rows * 16; i += kAll) {
      const int r = i >> 4, kc = i & 15;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + off128(r, kc))),
                   "l"(W + (size_t)r * kHid + kc * 8)
                   : "memory");
    }
  };
  for (int l = 0; l < 3; ++l) stage(S.w[l], net.w[l], kHid);
  stage(S.w5, net.w5, kOutPad);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int i = threadIdx.x; i < kHid * 8; i += kAll)
    S.w1[i] = i % 8 < net.n_in ? net.w1[(i / 8) * net.ldw1 + i % 8] : 0.0f;
  for (int i = threadIdx.x; i < 4 * kHid + kOutPad; i += kAll) {
    const int l = i / kHid, u = i % kHid;
    S.b[i] = (l < 4) ? net.b[l][u] : net.b[4][i - 4 * kHid];
  }
  if (threadIdx.x < 32) tmem_alloc(&S.tmem, 512);
  if (threadIdx.x < kFwdGroups) {
    mbar_init(&S.bar[threadIdx.x], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem + group * kHid;
  const uint32_t idesc_h = instr_desc_bf16(kTileM, kHid);
  const uint32_t idesc_o = instr_desc_bf16(kTileM, kOutPad);
  unsigned char *act = S.act[group];
  uint64_t *bar = &S.bar[group];
  const int quarter = warp & 3;           // tensor-memory lanes 32q .. 32q + 31
  const int half = warp >> 2;             // columns [64 half, 64 half + 64)
  const int row = quarter * 32 + lane;    // the tile row this thread owns in the epilogues
  const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
  uint32_t phase = 0;
  // The group's barrier, which also tells every thread whether all waits so far were in time: the
  // threads of a group leave their loop together, or one would be left at a barrier of its own.
  bool ok = true, mine = true;
  auto group_sync = [&]() {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((uint32_t)mine), "r"(1 + group), "n"(kFusedThreads)
        : "memory");
    return all != 0;
  };
  const int tiles = (n + kTileM - 1) / kTileM, stride = gridDim.x * kFwdGroups;
  bool staged = false;
  float xi[8];
  auto load_x = [&](int tile) {
    const int g = tile * kTileM + row;
#pragma unroll
    for (int i = 0; i < 8; ++i) xi[i] = (i < net.n_in && g < n) ? x[(size_t)g * ldx + i] : 0.0f;
  };
  int tile = group * gridDim.x + blockIdx.x;
  load_x(tile);
  for (; tile < tiles && ok; tile += stride) {
    const int g = tile * kTileM + row;
    for (int c8 = 0; c8 < 8; ++c8) {
      const int u = half * 64 + c8 * 8;
      __align__(16) __nv_bfloat16 h8[8];
      first_layer8<NIN>(S.w1 + u * 8, S.b + u, xi, net.n_in, g < n, h8);
      *reinterpret_cast<uint4 *>(act + off128(row, half * 8 + c8)) = *reinterpret_cast<uint4 *>(h8);
    }
    load_x(tile + stride);  // the next tile's inputs, under this one's layers
    if (!staged) {
      // All groups' copies; a group without a tile meets the others below.
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_proxy_async_smem();
      asm volatile("bar.sync 0;" ::: "memory");
      staged = true;
    }
    // Layers 2..5 on the tensor cores.
    for (int l = 0; l < 4; ++l) {
      fence_proxy_async_smem();
      tc_fence_before();
      ok = group_sync();
      tc_fence_after();
      if (!ok) break;
      const bool last = (l == 3);
      if (tid == 0) {
        const uint32_t wb = last ? smem_u32(S.w5) : smem_u32(S.w[l]), ab = smem_u32(act);
        for (int s = 0; s < 8; ++s)
          mma_bf16(tmem, smem_desc(ab + s * 256, 128, 2048), smem_desc(wb + s * 256, 128, 2048),
                   last ? idesc_o : idesc_h, s > 0 ? 1u : 0u);
        mma_commit(bar);
      }
      mine = mbar_wait(bar, phase) && mine;
      phase ^= 1u;
      tc_fence_after();
      if (!last) {
        // Epilogue: bias + SiLU, written back as the next layer's operand.
#pragma unroll
        for (int c0 = 0; c0 < 64; c0 += 32) {
          float v[32];
          __syncwarp();
          tmem_ld32(lane_base + half * 64 + c0, v);
#pragma unroll
          for (int c8 = 0; c8 < 4; ++c8) {
            const float *b = S.b + (l + 1) * kHid + half * 64 + c0 + c8 * 8;
            __align__(16) __nv_bfloat16 h8[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) h8[j] = __float2bfloat16(silu(v[c8 * 8 + j] + b[j]));
            *reinterpret_cast<uint4 *>(act + off128(row, (half * 64 + c0) / 8 + c8)) = *reinterpret_cast<uint4 *>(h8);
          }
        }
      } else if (half == 0) {
        float v[16];
        __syncwarp();
        tmem_ld16(lane_base, v);
        if (g < n) {
#pragma unroll
          for (int j = 0; j < kOutPad; ++j) y[(size_t)g * ldy + j] = v[j] + S.b[4 * kHid + j];
        }
      }
    }
  }
  if (!staged) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_proxy_async_smem();
    asm volatile("bar.sync 0;" ::: "memory");
  }
  if (!group_sync()) {  // an expired wait: record it and drain (bounded) before tensor memory goes
    if (tid == 0) atomicExch(err, 1);
    mbar_wait(bar, phase ^ 1u);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32) tmem_free(S.tmem, 512);
}

// ---- fused training step ------------------------------------------------------------------------
// One 128-sample tile at a time through the whole network and back in one kernel: the activations
// of the four hidden layers stay in shared memory (a layer's is overwritten by its gradient once
// the next layer's weight gradient has read it), the weights pass through two buffers, and the
// weight gradients of the three 128 x 128 layers accumulate in tensor memory over the block's tiles.
// Every product runs from the same row-major tiles: a weight gradient dZ^T H and a backward product
// dZ W read them as MN-major operands, so nothing is transposed. Pre-activations go through global
// memory (BF16, as the layer-by-layer path rounds them). A second kernel sums the blocks' partial
// gradients in block order and applies Adam. The layer-by-layer path is ~60 launches and writes and
// reads every activation and its transpose: a step on 16,384 samples takes 929 us that way, 98 us
// fused (with the copies of the batch; 5 GFLOP, so either is bound by latencies: a tile's eight
// layer steps follow one another).

constexpr int kTileBytes = kHid * kHid * 2;
constexpr int kPartW5 = 3 * kHid * kHid;                 // partials: W2..W4, W5 (transposed), W1, biases
constexpr int kPartW1 = kPartW5 + kHid * kOutPad;
constexpr int kPartB = kPartW1 + kHid * 8;
constexpr int kPartSize = kPartB + 4 * kHid + kOutPad;

struct TrainSmem {
  unsigned char h[4][kTileBytes];        // activations, then gradients, of the hidden layers
  unsigned char w[2][kTileBytes];        // W2 / W4, W3
  unsigned char w5[kOutPad * kHid * 2];
  unsigned char dy[kTileM * kOutPad * 2];  // output gradient, 8 x 8 core matrices, row groups 256 B apart
  float w1[kHid * 8];
  float b[4 * kHid + kOutPad];
  float x[kTileM * 8];
  uint64_t bar;
  uint32_t tmem;
};
static_assert(sizeof(TrainSmem) <= 227 * 1024, "one block's shared memory");

// MN-major operand flags of the instruction descriptor (A: bit 15, B: bit 16).
constexpr uint32_t kMnA = 1u << 15, kMnB = 1u << 16;

__device__ __forceinline__ void stage_weights(unsigned char *dst, const void *src, int tid) {
  const __nv_bfloat16 *W = static_cast<const __nv_bfloat16 *>(src);
  for (int i = tid; i < kHid * 16; i += kFusedThreads) {
    const int r = i >> 4, kc = i & 15;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + off128(r, kc))),
                 "l"(W + (size_t)r * kHid + kc * 8)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Sums over the tile's rows of a gradient tile's columns, each row times its weight: warp w takes
// rows 16 w .. 16 w + 15, lane i & 7 one row of each group of eight; per 8-column group the eight lanes' sums
// are exchanged so that each lane keeps one column. acc[k]: column (4 k + lane / 8) * 8 + col(lane).
__device__ __forceinline__ void column_sums(const unsigned char *tile, float w0, float w1, int warp, int lane,
                                            float (&acc)[4]) {
  const int i = lane & 7, q = lane >> 3;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int kc = 4 * k + q;
    float s[8];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const uint4 v = *reinterpret_cast<const uint4 *>(tile + (2 * warp + c) * 2048 + kc * 128 + i * 16);
      const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
      const float w = c ? w1 : w0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        s[2 * j] = c ? s[2 * j] + w * f.x : w * f.x;
        s[2 * j + 1] = c ? s[2 * j + 1] + w * f.y : w * f.y;
      }
    }
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {
      const bool up = i & h;
#pragma unroll
      for (int j = 0; j < h; ++j) {
        const float keep = up ? s[j + h] : s[j], give = up ? s[j] : s[j + h];
        s[j] = keep + __shfl_xor_sync(0xffffffffu, give, h);
      }
    }
    acc[k] += s[0];
  }
}
__device__ __forceinline__ int column_of(int k, int lane) { return (4 * k + (lane >> 3)) * 8 + (lane & 7); }

__global__ void __launch_bounds__(kFusedThreads, 1) mlp_train_kernel(xd_mlp_train_args a, int tiles) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  TrainSmem &S = *reinterpret_cast<TrainSmem *>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  stage_weights(S.w[0], a.w16[1], tid);
  stage_weights(S.w[1], a.w16[2], tid);
  {
    const __nv_bfloat16 *W = static_cast<const __nv_bfloat16 *>(a.w16[4]);
    for (int i = tid; i < kOutPad * 16; i += kFusedThreads) {
      const int r = i >> 4, kc = i & 15;
      *reinterpret_cast<uint4 *>(S.w5 + off128(r, kc)) = *reinterpret_cast<const uint4 *>(W + (size_t)r * kHid + kc * 8);
    }
  }
  for (int i = tid; i < kHid * 8; i += kFusedThreads) S.w1[i] = i % 8 < a.n_in ? a.w[0][(i / 8) * a.ldw1 + i % 8] : 0.0f;
  for (int i = tid; i < 4 * kHid + kOutPad; i += kFusedThreads) {
    const int l = i / kHid, u = i % kHid;
    S.b[i] = l < 4 ? a.b[l][u] : a.b[4][i - 4 * kHid];
  }
  if (warp == 0) tmem_alloc(&S.tmem, 512);
  if (tid == 0) {
    mbar_init(&S.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem;
  const int quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane;
  const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
  uint32_t phase = 0;
  bool ok = true;
  float gb[4][4] = {}, gw1[5][4] = {}, gb5 = 0.0f, g5[8] = {};  // sums over the block's tiles
  float gwx[3][4] = {};                                         // first-layer inputs 6 to 8
  // Everything written to shared memory is visible to the tensor core and the last reads of tensor
  // memory are done; one thread issues, all wait.
  auto begin = [&]() {
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  };
  auto finish = [&]() {
    ok = __syncthreads_and(mbar_wait(&S.bar, phase)) != 0;
    phase ^= 1u;
    tc_fence_after();
  };
  // D[128 x N] (+)= A B over `steps` K steps of 16; an operand advances sa / sb bytes per step.
  auto product = [&](uint32_t d, uint32_t A, uint32_t la, uint32_t ssa, uint32_t sa, uint32_t B, uint32_t lb, uint32_t ssb,
                     uint32_t sb, uint32_t idesc, int steps, bool add) {
    for (int s = 0; s < steps; ++s)
      mma_bf16(tmem + d, smem_desc(A + s * sa, la, ssa), smem_desc(B + s * sb, lb, ssb), idesc, add || s > 0 ? 1u : 0u);
  };
  const uint32_t kFwd = instr_desc_bf16(kTileM, kHid), kOut = instr_desc_bf16(kTileM, kOutPad);
  bool first = true;
  for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, first = false) {
    const int g = tile * kTileM + row;
    for (int i = tid; i < kTileM * 8; i += kFusedThreads) {
      const int r = tile * kTileM + i / 8;
      S.x[i] = i % 8 < a.n_in && r < a.n ? a.x[(size_t)r * a.ldx + i % 8] : 0.0f;
    }
    __syncthreads();
    // Layer 1 on the CUDA cores (FP32).
    {
      float xi[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) xi[i] = S.x[row * 8 + i];
      __nv_bfloat16 *Z = static_cast<__nv_bfloat16 *>(a.z[0]) + (size_t)g * kHid;
      for (int c8 = 0; c8 < 8; ++c8) {
        __align__(16) __nv_bfloat16 z8[8], h8[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int u = half * 64 + c8 * 8 + j;
          float z = S.b[u];
          for (int i = 0; i < a.n_in; ++i) z += S.w1[u * 8 + i] * xi[i];
          z8[j] = __float2bfloat16(z);
          h8[j] = __float2bfloat16(silu(z));
        }
        *reinterpret_cast<uint4 *>(S.h[0] + off128(row, half * 8 + c8)) = *reinterpret_cast<uint4 *>(h8);
        *reinterpret_cast<uint4 *>(Z + half * 64 + c8 * 8) = *reinterpret_cast<uint4 *>(z8);
      }
    }
    // Layers 2..4: W2 in buffer 0, W3 in buffer 1, then W4 in buffer 0.
    for (int l = 1; l < 4 && ok; ++l) {
      if (l == 3) asm volatile("cp.async.wait_group 0;" ::: "memory");
      begin();
      if (tid == 0) {
        product(0, smem_u32(S.h[l - 1]), 128, 2048, 256, smem_u32(S.w[(l - 1) & 1]), 128, 2048, 256, kFwd, 8, false);
        mma_commit(&S.bar);
      }
      finish();
      if (!ok) break;
      if (l == 1) stage_weights(S.w[0], a.w16[3], tid);
      __nv_bfloat16 *Z = static_cast<__nv_bfloat16 *>(a.z[l]) + (size_t)g * kHid;
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 32) {
        float v[32];
        tmem_ld32(lane_base + half * 64 + c0, v);
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) {
          __align__(16) __nv_bfloat16 z8[8], h8[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float z = v[c8 * 8 + j] + S.b[l * kHid + half * 64 + c0 + c8 * 8 + j];
            z8[j] = __float2bfloat16(z);
            h8[j] = __float2bfloat16(silu(z));
          }
          const int kc = (half * 64 + c0) / 8 + c8;
          *reinterpret_cast<uint4 *>(S.h[l] + off128(row, kc)) = *reinterpret_cast<uint4 *>(h8);
          *reinterpret_cast<uint4 *>(Z + kc * 8) = *reinterpret_cast<uint4 *>(z8);
        }
      }
    }
    if (!ok) break;
    // Output layer, squared error and its gradient.
    begin();
    if (tid == 0) {
      product(0, smem_u32(S.h[3]), 128, 2048, 256, smem_u32(S.w5), 128, 2048, 256, kOut, 8, false);
      mma_commit(&S.bar);
    }
    finish();
    if (!ok) break;
    if (half == 0) {
      float v[16];
      tmem_ld16(lane_base, v);
      float sq = 0.0f, d[16];
      __align__(16) __nv_bfloat16 d8[16];
#pragma unroll
      for (int j = 0; j < kOutPad; ++j) {
        v[j] += S.b[4 * kHid + j];
        d[j] = 0.0f;
        if (j < a.n_out && g < a.n) {
          const float e = v[j] - a.t[(size_t)g * a.n_out + j];
          sq += e * e;
          d[j] = a.scale * e;
        }
        d8[j] = __float2bfloat16(d[j]);
        d[j] = __bfloat162float(d8[j]);
      }
      *reinterpret_cast<uint4 *>(S.dy + (row >> 3) * 256 + (row & 7) * 16) = *reinterpret_cast<uint4 *>(d8);
      *reinterpret_cast<uint4 *>(S.dy + (row >> 3) * 256 + 128 + (row & 7) * 16) = *reinterpret_cast<uint4 *>(d8 + 8);
      if (g < a.n) {
        a.sq[g] = sq;
#pragma unroll
        for (int j = 0; j < kOutPad; j += 4)
          *reinterpret_cast<float4 *>(a.y + (size_t)g * kOutPad + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
      // Sixteen sums over 32 lanes: lane keeps output (lane / 2 with its bits as exchanged).
#pragma unroll
      for (int h = 8; h > 0; h >>= 1) {
        const bool up = lane & (2 * h);
#pragma unroll
        for (int j = 0; j < h; ++j) {
          const float keep = up ? d[j + h] : d[j], give = up ? d[j] : d[j + h];
          d[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
      }
      gb5 += d[0] + __shfl_xor_sync(0xffffffffu, d[0], 1);
    }
    // W5's gradient, transposed: H4^T dY, 128 x 16, added up in registers.
    begin();
    if (tid == 0) {
      product(0, smem_u32(S.h[3]), 2048, 128, 4096, smem_u32(S.dy), 256, 128, 512, kOut | kMnA | kMnB, 8, false);
      mma_commit(&S.bar);
    }
    finish();
    if (!ok) break;
    {
      float v[16];
      tmem_ld16(lane_base, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) g5[j] += half ? v[j + 8] : v[j];
    }
    // Backward through layers 4..1: dH_l = dZ_{l+1} W_{l+1} (and layer l + 1's weight gradient beside it),
    // dZ_l = dH_l silu'(z_l) in the place of H_l.
    for (int l = 3; l >= 0 && ok; --l) {
      if (l == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
      begin();
      if (tid == 0) {
        if (l == 3) {
          product(0, smem_u32(S.dy), 128, 256, 256, smem_u32(S.w5), 2048, 128, 4096, kFwd | kMnB, 1, false);
        } else {
          product(0, smem_u32(S.h[l + 1]), 128, 2048, 256, smem_u32(S.w[l & 1]), 2048, 128, 4096, kFwd | kMnB, 8, false);
          product(128 + l * 128, smem_u32(S.h[l + 1]), 2048, 128, 4096, smem_u32(S.h[l]), 2048, 128, 4096,
                  kFwd | kMnA | kMnB, 8, !first);
        }
        mma_commit(&S.bar);
      }
      // Meanwhile: this thread's pre-activations, and the column sums of layer l + 1's gradient.
      uint4 zq[8];
      const uint4 *Z = reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(a.z[l]) + (size_t)g * kHid +
                                                       half * 64);
#pragma unroll
      for (int i = 0; i < 8; ++i) zq[i] = Z[i];
      if (l < 3) column_sums(S.h[l + 1], 1.0f, 1.0f, warp, lane, gb[l + 1]);
      finish();
      if (!ok) break;
      if (l == 2) stage_weights(S.w[0], a.w16[1], tid);  // W4 has been read: W2 for the last product and the next tile
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 32) {
        float v[32];
        tmem_ld32(lane_base + half * 64 + c0, v);
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) {
          const __nv_bfloat16 *z8 = reinterpret_cast<const __nv_bfloat16 *>(&zq[c0 / 8 + c8]);
          __align__(16) __nv_bfloat16 d8[8];
#pragma unroll
          for (int j = 0; j < 8; ++j)
            d8[j] = __float2bfloat16(v[c8 * 8 + j] * silu_grad(__bfloat162float(z8[j])));
          *reinterpret_cast<uint4 *>(S.h[l] + off128(row, (half * 64 + c0) / 8 + c8)) = *reinterpret_cast<uint4 *>(d8);
        }
      }
    }
    if (!ok) break;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    column_sums(S.h[0], 1.0f, 1.0f, warp, lane, gb[0]);
    const float *x0 = S.x + (16 * warp + (lane & 7)) * 8, *x1 = x0 + 64;
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (i < a.n_in) column_sums(S.h[0], x0[i], x1[i], warp, lane, gw1[i]);
#pragma unroll
    for (int i = 5; i < 8; ++i)
      if (i < a.n_in) column_sums(S.h[0], x0[i], x1[i], warp, lane, gwx[i - 5]);
    __syncthreads();
  }
  if (!ok) {
    if (tid == 0) atomicExch(a.err, 1);
    mbar_wait(&S.bar, phase ^ 1u);
  } else {
    // The block's partial gradients.
    float *P = a.part + (size_t)blockIdx.x * kPartSize;
    for (int l = 0; l < 3; ++l)
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 32) {
        float v[32];
        tmem_ld32(lane_base + 128 + l * 128 + half * 64 + c0, v);
        float4 *to = reinterpret_cast<float4 *>(P + l * kHid * kHid + row * kHid + half * 64 + c0);
#pragma unroll
        for (int j = 0; j < 8; ++j) to[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
#pragma unroll
    for (int j = 0; j < 8; ++j) P[kPartW5 + row * kOutPad + half * 8 + j] = g5[j];
    // Across the warps, in order, through shared memory (the activations' place).
    float *red = reinterpret_cast<float *>(S.h[0]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = column_of(k, lane);
#pragma unroll
      for (int l = 0; l < 4; ++l) red[(warp * 12 + l) * kHid + c] = gb[l][k];
#pragma unroll
      for (int i = 0; i < 5; ++i) red[(warp * 12 + 4 + i) * kHid + c] = gw1[i][k];
#pragma unroll
      for (int i = 0; i < 3; ++i) red[(warp * 12 + 9 + i) * kHid + c] = gwx[i][k];
    }
    float *red5 = red + 8 * 12 * kHid;
    if (half == 0 && (lane & 1) == 0) red5[warp * kOutPad + (lane >> 1)] = gb5;
    __syncthreads();
    for (int i = tid; i < 12 * kHid; i += kFusedThreads) {
      float s = 0.0f;
      for (int w = 0; w < 8; ++w) s += red[w * 12 * kHid + i];
      const int q = i / kHid, c = i % kHid;
      if (q < 4)
        P[kPartB + q * kHid + c] = s;
      else
        P[kPartW1 + c * 8 + q - 4] = s;
    }
    if (tid < kOutPad) {
      float s = 0.0f;
      for (int w = 0; w < 4; ++w) s += red5[w * kOutPad + tid];
      P[kPartB + 4 * kHid + tid] = s;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_free(tmem, 512);
}

// Adds the blocks' partial gradients in block order and applies Adam, one thread per parameter; the
// padding (inputs from n_in, outputs from n_out on) stays zero. What bounds it is the round trips of
// a thread's reads (27 MB in all from L2, one and a half blocks to an SM), so the sum is unrolled 32
// times: a step at batch 16,384 took 97 us unrolled 8 times, 93 us now.
__global__ void __launch_bounds__(256) mlp_apply_kernel(xd_mlp_train_args a, int blocks) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= kPartSize) return;
  float gr = 0.0f;
#pragma unroll 32
  for (int k = 0; k < blocks; ++k) gr += a.part[(size_t)k * kPartSize + i];
  int l, r, c = 0;
  bool bias = false, pad = false;
  if (i < kPartW5) {
    l = 1 + i / (kHid * kHid);
    r = i / kHid % kHid;
    c = i % kHid;
  } else if (i < kPartW1) {
    l = 4;
    r = (i - kPartW5) % kOutPad;
    c = (i - kPartW5) / kOutPad;
    pad = r >= a.n_out;
  } else if (i < kPartB) {
    l = 0;
    r = (i - kPartW1) / 8;
    c = (i - kPartW1) % 8;
    if (c >= a.n_in) return;
  } else {
    bias = true;
    l = min((i - kPartB) / kHid, 4);
    r = i - kPartB - l * kHid;
    pad = l == 4 && r >= a.n_out;
  }
  if (pad) gr = 0.0f;
  const int ld = l == 0 ? a.ldw1 : kHid, at = bias ? r : r * ld + c;
  float *p = bias ? a.b[l] : a.w[l], *m = bias ? a.mb[l] : a.mw[l], *v = bias ? a.vb[l] : a.vw[l];
  (bias ? a.gb[l] : a.gw[l])[at] = gr;
  const float mi = a.adam.beta1 * m[at] + (1.0f - a.adam.beta1) * gr;
  const float vi = a.adam.beta2 * v[at] + (1.0f - a.adam.beta2) * gr * gr;
  m[at] = mi;
  v[at] = vi;
  const float pi = pad ? 0.0f : p[at] - a.adam.lr * (mi / a.adam.bias_corr1) / (sqrtf(vi / a.adam.bias_corr2) + a.adam.eps);
  p[at] = pi;
  if (!bias) {
    static_cast<__nv_bfloat16 *>(a.w16[l])[at] = __float2bfloat16(pi);
    static_cast<__nv_bfloat16 *>(a.w16t[l])[(size_t)c * (l == 4 ? kOutPad : kHid) + r] = __float2bfloat16(pi);
  }
}

int cuda_err(cudaError_t e, const char *where) {
  return xd_internal_fail(-3, std::string("CUDA error in ") + where + ": " + cudaGetErrorString(e));
}

}  // namespace

extern "C" {

int xd_gemm_bf16(const xd_gemm_args *g, int splits, void *stream) {
  if (!g || !g->A || !g->B || !g->err) return xd_internal_fail(-1, "null GEMM argument");
  if (g->M <= 0 || g->N <= 0 || g->K <= 0 || (g->K % 16) != 0 || (g->lda % 8) != 0 || (g->ldb % 8) != 0)
    return xd_internal_fail(-1, "GEMM needs K and the leading dimensions to be multiples of 16 / 8");
  if ((reinterpret_cast<uintptr_t>(g->A) | reinterpret_cast<uintptr_t>(g->B)) & 15)
    return xd_internal_fail(-1, "GEMM operands must be 16-byte aligned");
  if (g->tile_n != 16 && g->tile_n != 128) return xd_internal_fail(-1, "GEMM tile_n must be 16 or 128");
  if (splits < 1) splits = 1;
  if (splits > 1 && g->epilogue != XD_EPI_F32) return xd_internal_fail(-1, "split-K needs the plain F32 epilogue");
  int k_per = (g->K + splits - 1) / splits;
  k_per = (k_per + kChunkK - 1) / kChunkK * kChunkK;
  const int used = (g->K + k_per - 1) / k_per;
  dim3 grid((g->M + kTileM - 1) / kTileM, (g->N + g->tile_n - 1) / g->tile_n, used);
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = (size_t)kTileM * kChunkK * 2 + (size_t)g->tile_n * kChunkK * 2 + 16;
  if (g->tile_n == 128) {
    cudaFuncSetAttribute(gemm_bf16_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gemm_bf16_tc_kernel<128><<<grid, kThreads, smem, st>>>(*g, k_per);
  } else {
    gemm_bf16_tc_kernel<16><<<grid, kThreads, smem, st>>>(*g, k_per);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_err(e, "gemm_bf16_tc_kernel launch");
  return used;
}

int xd_mlp_input_layer(int M, int n_in, int n_hid, const float *d_x, int ldx, const float *d_w1, int ldw,
                       const float *d_b1, void *d_z, void *d_h, void *d_ht, int ldt, void *stream) {
  if (M <= 0 || n_in <= 0 || n_in > 8 || n_hid <= 0 || n_hid > 1024 || !d_x || !d_w1 || !d_b1 || !d_z || !d_h)
    return xd_internal_fail(-1, "bad input-layer arguments");
  input_layer_kernel<<<M, n_hid, 0, (cudaStream_t)stream>>>(M, n_in, n_hid, d_x, ldx, d_w1, ldw, d_b1,
                                                            (__nv_bfloat16 *)d_z, (__nv_bfloat16 *)d_h,
                                                            (__nv_bfloat16 *)d_ht, ldt);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "input_layer_kernel");
}

int xd_mlp_input_grad(int M, int n_in, int n_hid, const void *d_dzt, int ldt, const float *d_x, int ldx,
                      float *d_gw, int ldw, void *stream) {
  if (M <= 0 || n_in <= 0 || n_in > 8 || n_hid <= 0 || !d_dzt || !d_x || !d_gw)
    return xd_internal_fail(-1, "bad input-grad arguments");
  input_grad_kernel<<<n_hid, 256, 0, (cudaStream_t)stream>>>(M, n_in, (const __nv_bfloat16 *)d_dzt, ldt, d_x, ldx,
                                                             d_gw, ldw);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "input_grad_kernel");
}

int xd_surrogate_features(int n, const int *d_idx, const int *d_nodes4, const double *d_sol, const float *d_geom2,
                          float vmax, float *d_x, int ldx, void *stream) {
  if (n < 0 || (n > 0 && (!d_idx || !d_nodes4 || !d_sol || !d_geom2 || !d_x)) || ldx < 5 || vmax <= 0.0f)
    return xd_internal_fail(-1, "bad surrogate-feature arguments");
  if (n == 0) return 0;
  surrogate_features_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(n, d_idx, d_nodes4, d_sol, d_geom2,
                                                                               1.0f / vmax, d_x, ldx);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "surrogate_features_kernel");
}

int xd_surrogate_stage(int n, const int *d_idx, const float *d_y, int ldy, const float *d_out_scale, int n_inst,
                       double *d_stage, void *stream) {
  if (n < 0 || (n > 0 && (!d_idx || !d_y || !d_out_scale || !d_stage)) || ldy < 4 || n_inst < n)
    return xd_internal_fail(-1, "bad surrogate-stage arguments");
  if (n == 0) return 0;
  surrogate_stage_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(n, d_idx, d_y, ldy, d_out_scale, n_inst,
                                                                            d_stage);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "surrogate_stage_kernel");
}

int xd_mlp_forward(const xd_mlp_net *net, int n, const float *d_x, int ldx, float *d_y, int ldy, int *d_err,
                   int max_ctas, void *stream) {
  if (!net || !net->w1 || !net->w5 || !d_x || !d_y || !d_err || n < 0 || net->n_in < 1 || net->n_in > 8 ||
      ldy < kOutPad)
    return xd_internal_fail(-1, "bad fused-forward arguments");
  for (int l = 0; l < 3; ++l)
    if (!net->w[l]) return xd_internal_fail(-1, "bad fused-forward weights");
  for (int l = 0; l < 5; ++l)
    if (!net->b[l]) return xd_internal_fail(-1, "bad fused-forward biases");
  if ((reinterpret_cast<uintptr_t>(net->w[0]) | reinterpret_cast<uintptr_t>(net->w[1]) |
       reinterpret_cast<uintptr_t>(net->w[2]) | reinterpret_cast<uintptr_t>(net->w5)) & 15)
    return xd_internal_fail(-1, "fused-forward weights must be 16-byte aligned");
  if (n == 0) return 0;
  const int tiles = (n + kTileM - 1) / kTileM;
  int sms = 148;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int grid = tiles < sms ? tiles : sms;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  const size_t smem = sizeof(FusedSmem);
  auto kernel = net->n_in == 5 ? mlp_forward_fused_kernel<5> : mlp_forward_fused_kernel<0>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_err(e, "cudaFuncSetAttribute(mlp_forward_fused_kernel)");
  kernel<<<grid, kFwdGroups * kFusedThreads, smem, (cudaStream_t)stream>>>(*net, n, d_x, ldx, d_y, ldy, d_err);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "mlp_forward_fused_kernel");
}

int xd_mse_grad(int M, int n_out, int ld, const float *d_y, const float *d_target, float scale, void *d_dz,
                void *d_dzt, int ldt, float *d_sq, void *stream) {
  if (M <= 0 || !d_y || !d_target || !d_dz || !d_dzt) return xd_internal_fail(-1, "bad mse arguments");
  mse_grad_kernel<<<(M + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
      M, n_out, ld, d_y, d_target, scale, (__nv_bfloat16 *)d_dz, (__nv_bfloat16 *)d_dzt, ldt, d_sq);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "mse_grad_kernel");
}

int xd_bias_grad(int M, int N, const void *d_dzt, int ldt, float *d_db, void *stream) {
  if (M <= 0 || N <= 0 || !d_dzt || !d_db) return xd_internal_fail(-1, "bad bias-grad arguments");
  bias_grad_kernel<<<N, 256, 0, (cudaStream_t)stream>>>(M, N, (const __nv_bfloat16 *)d_dzt, ldt, d_db);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "bias_grad_kernel");
}

int xd_splitk_sum(int n, int splits, const float *d_part, float *d_out, void *stream) {
  if (n <= 0 || splits <= 0 || !d_part || !d_out) return xd_internal_fail(-1, "bad split-K arguments");
  splitk_sum_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(n, splits, d_part, d_out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "splitk_sum_kernel");
}

int xd_column_sum(int rows, int cols, const float *d_in, int ld, float *d_out, void *stream) {
  if (rows <= 0 || cols <= 0 || !d_in || !d_out) return xd_internal_fail(-1, "bad column-sum arguments");
  column_sum_kernel<<<cols, 256, 0, (cudaStream_t)stream>>>(rows, cols, d_in, ld, d_out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "column_sum_kernel");
}

int xd_adam(int rows, int cols, float *d_p, const float *d_grad, float *d_m, float *d_v, const xd_adam_args *a,
            void *d_p16, void *d_p16t, int ld16, int ld16t, void *stream) {
  if (rows <= 0 || cols <= 0 || !d_p || !d_grad || !d_m || !d_v || !a) return xd_internal_fail(-1, "bad Adam args");
  const int n = rows * cols;
  adam_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
      rows, cols, d_p, d_grad, d_m, d_v, a->lr, a->beta1, a->beta2, a->eps, a->bias_corr1, a->bias_corr2,
      (__nv_bfloat16 *)d_p16, (__nv_bfloat16 *)d_p16t, ld16, ld16t);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "adam_kernel");
}

int xd_mlp_train_part_size(int n, int *blocks) {
  if (n <= 0 || !blocks) return xd_internal_fail(-1, "bad training-step arguments");
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (n + kTileM - 1) / kTileM;
  *blocks = tiles < sms ? tiles : sms;
  return kPartSize;
}

int xd_mlp_train_step(const xd_mlp_train_args *a, void *stream) {
  if (!a || a->n <= 0 || a->n_in < 1 || a->n_in > 8 || a->n_out < 1 || a->n_out > kOutPad || a->ldx < a->n_in ||
      a->ldw1 < a->n_in || !a->x || !a->t || !a->y || !a->sq || !a->part || !a->err)
    return xd_internal_fail(-1, "bad training-step arguments");
  uintptr_t align = reinterpret_cast<uintptr_t>(a->y) | reinterpret_cast<uintptr_t>(a->part);
  for (int l = 0; l < 5; ++l) {
    if (!a->w[l] || !a->b[l] || !a->gw[l] || !a->gb[l] || !a->mw[l] || !a->vw[l] || !a->mb[l] || !a->vb[l] ||
        !a->w16[l] || !a->w16t[l] || (l < 4 && !a->z[l]))
      return xd_internal_fail(-1, "null training-step buffer");
    align |= reinterpret_cast<uintptr_t>(a->w16[l]);
    if (l < 4) align |= reinterpret_cast<uintptr_t>(a->z[l]);
  }
  if (align & 15) return xd_internal_fail(-1, "training-step buffers must be 16-byte aligned");
  int blocks = 0;
  xd_mlp_train_part_size(a->n, &blocks);
  const size_t smem = sizeof(TrainSmem);
  cudaError_t e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_err(e, "cudaFuncSetAttribute(mlp_train_kernel)");
  cudaStream_t st = (cudaStream_t)stream;
  mlp_train_kernel<<<blocks, kFusedThreads, smem, st>>>(*a, (a->n + kTileM - 1) / kTileM);
  mlp_apply_kernel<<<(kPartSize + 255) / 256, 256, 0, st>>>(*a, blocks);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_err(e, "mlp_train_kernel");
}

}  // extern "C"
