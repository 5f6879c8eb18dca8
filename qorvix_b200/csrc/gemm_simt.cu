// C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores: plain float32 multiply-adds, no tensor
// cores, no reduced-precision mode.  This is the matrix product of the true 32-bit path and
// the fallback for shapes the tensor-core kernels refuse.  The reference's GEMV
// (cuda/src/cuda_backend.cu:291-312, out[r] = dot(W[r,:], x)) computes the same numbers one
// row at a time.
//
// Each output element is accumulated by one thread walking k = 0..K-1 in ascending order,
// so a value does not depend on M, on the tile it falls in, or on anything else in the batch.
//
// Rows of both operands are staged as they lie (k contiguous, a row padded by 16 bytes so that 16-byte reads of
// neighbouring rows miss one another's banks), STAGES - 1 tiles ahead by cp.async where the operands are float32 on 16 bytes, else (other
// types, odd strides) through registers, all of a thread's elements of the next tile in flight under the present one's multiply-adds; and
// a thread reads four k of a row at a time.  Two tile shapes: 16 x 32 (64 k, 2 x 2 outputs a thread) where 64 x 64 tiles would be few
// or mostly padding, else 64 x 64 (32 k, 4 x 4 a thread).  Few CTAs are bound by the chain of K dependent multiply-adds and the
// trips to memory ahead of it: with one tile of 16 k at a time and no copy in flight, 192 / 512 k took 20 / 51 us (3 rows), with three
// tiles of 64 k 3.6 / 8.4 us behind the kernel ahead.  So products of one wave of CTAs get a ring of eight tiles, and the weights' halves of the
// first ones are asked for ahead of the wait for the kernel ahead where the caller says that no launch may still write them (a model's
// weights): 2.5 / 5.0 us.
#include "common.cuh"
#include "per_device.h"

__device__ __forceinline__ void gs_cp16(float* dst, const float* src, bool live) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(live ? 16 : 0) : "memory");
}

// GLU: the rows of W come in groups of 32, 16 gate rows and the 16 up rows of the same features; a thread of a 16 x 32 tile holds both sums of a
// feature, and C[M, N / 2] = act(gate) * up, as the activation's own kernel has it (the same bits).  Bound as the plain product of its size; a
// launch and a trip of the sums through memory less: replies of a 32-bit model of three layers (d 192, f 512) 679 us with two launches,
// 662 with one, in turn on one GPU.
template <typename TA, typename TW, typename TC, int BM, int BN, int BK, int TM, int TN, int STAGES, bool ASYNC, bool GLU = false>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_simt_kernel(TC* __restrict__ C, const TA* __restrict__ A,
                                                                        const TW* __restrict__ W, int M, int N, int K,
                                                                        int lda, int ldw, int ldc, int accumulate, int settled, GluAct glu) {
  constexpr int THREADS = (BM / TM) * (BN / TN), LD = BK + 4, ROWS = BM + BN, PIECES = BK / 4;
  extern __shared__ __align__(16) float gs_ring[];
  float(*ring)[ROWS * LD] = (float(*)[ROWS * LD])gs_ring;            // [STAGES]
  const int tid = threadIdx.x;
  constexpr int TX = BN / TN, TY = BM / TM;        // a thread's outputs: rows ty + TY * i, columns tx + TX * j
  const int tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  const int tiles = (K + BK - 1) / BK;
  auto stage = [&](int t, int first, int last) {   // rows first .. last - 1 of tile t (A's, then W's) into its buffer; zeros beyond the matrices
    float* dst = ring[t % STAGES];
    const int k0 = t * BK;
#pragma unroll 4
    for (int e = first * PIECES + tid; e < last * PIECES; e += THREADS) {
      const int r = e / PIECES, k = k0 + (e % PIECES) * 4;
      const bool is_a = r < BM;
      const int g = is_a ? m0 + r : n0 + r - BM;
      const bool live = (is_a ? g < M : g < N) && k < K;
      const float* src = is_a ? (const float*)A + (size_t)g * lda + k : (const float*)W + (size_t)g * ldw + k;
      gs_cp16(dst + r * LD + (e % PIECES) * 4, live ? src : (const float*)W, live);
    }
  };
  if (ASYNC && settled)
    for (int t = 0; t < STAGES - 1 && t < tiles; ++t) stage(t, BM, ROWS);      // (with the first commit below)
  pdl_wait();
  pdl_launch_dependents();
  constexpr int PER_A = BM * BK / THREADS, PER_W = BN * BK / THREADS;
  static_assert(BM * BK % THREADS == 0 && BN * BK % THREADS == 0, "every thread stages as many elements");
  TA va[PER_A];
  TW vw[PER_W];
  auto fetch = [&](int t) {                        // tile t's elements, zeros beyond the matrices ...
#pragma unroll
    for (int i = 0; i < PER_A; ++i) {
      const int e = tid + i * THREADS, r = m0 + e / BK, k = t * BK + e % BK;
      va[i] = r < M && k < K ? A[(size_t)r * lda + k] : from_f<TA>(0.f);
    }
#pragma unroll
    for (int i = 0; i < PER_W; ++i) {
      const int e = tid + i * THREADS, r = n0 + e / BK, k = t * BK + e % BK;
      vw[i] = r < N && k < K ? W[(size_t)r * ldw + k] : from_f<TW>(0.f);
    }
  };
  auto put = [&](int t) {                          // ... into its buffer
    float* dst = ring[t % STAGES];
#pragma unroll
    for (int i = 0; i < PER_A; ++i) { const int e = tid + i * THREADS; dst[(e / BK) * LD + e % BK] = to_f(va[i]); }
#pragma unroll
    for (int i = 0; i < PER_W; ++i) { const int e = tid + i * THREADS; dst[(BM + e / BK) * LD + e % BK] = to_f(vw[i]); }
  };
  if (ASYNC) {
    for (int t = 0; t < STAGES - 1; ++t) {
      if (t < tiles) stage(t, 0, BM);
      if (t < tiles && !settled) stage(t, BM, ROWS);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  } else if (tiles > 0) {
    fetch(0);
    put(0);
  }
  for (int t = 0; t < tiles; ++t) {
    if (ASYNC) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                               // tile t has landed; the buffer filled next was read a tile ago
    if (ASYNC) {
      if (t + STAGES - 1 < tiles) stage(t + STAGES - 1, 0, ROWS);
      asm volatile("cp.async.commit_group;" ::: "memory");
    } else if (t + 1 < tiles) {
      fetch(t + 1);
    }
    const float* as = ring[t % STAGES] + ty * LD;
    const float* ws = ring[t % STAGES] + (BM + tx) * LD;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      float4 a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *(const float4*)(as + i * TY * LD + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *(const float4*)(ws + j * TX * LD + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
        }
    }
    if (!ASYNC && t + 1 < tiles) put(t + 1);
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty + TY * i;
    if (gm >= M) continue;
    if constexpr (GLU) {
      static_assert(BN == 32 && TN == 2, "a thread's two columns are a gate and its up value");
      if (n0 < N) C[(size_t)gm * ldc + n0 / 2 + tx] = from_f<TC>(glu_apply(acc[i][0], acc[i][1], glu));
      continue;
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx + TX * j;
      if (gn >= N) continue;
      TC* c = C + (size_t)gm * ldc + gn;
      float v = acc[i][j];
      if (accumulate) v += to_f(*c);
      *c = from_f<TC>(v);
    }
  }
}

#define GS_SETTLED 0x100
template <typename TA, typename TW, typename TC>
static int launch(void* C, const void* A, const void* W, int M, int N, int K, int lda, int ldw,
                  int ldc, int flags, cudaStream_t st) {
  const bool async = sizeof(TA) == 4 && sizeof(TW) == 4 && ((lda | ldw | K) & 3) == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  // 16 x 32 tiles where most rows of a 64-row tile would be padding, or where 64 x 64 tiles would leave SMs without one
  const long long big = (long long)((N + 63) / 64) * ((M + 63) / 64);
  const bool small = M <= 32 || big < 148;
  dim3 grid(small ? (N + 31) / 32 : (N + 63) / 64, small ? (M + 15) / 16 : (M + 63) / 64);
  if (grid.y > 65535) return QV_ERR_TOO_LARGE;
#define GS_LAUNCH(BM, BN, BK, TM, TN, ST, AS)                                                                                    \
  do {                                                                                                                           \
    constexpr size_t smem = (size_t)ST * (BM + BN) * (BK + 4) * 4;                                                               \
    static PerDevice allowed;                                                                                                    \
    if (smem > 48 * 1024) {                                                                                                      \
      const int rc = qv_allow_smem(gemm_simt_kernel<TA, TW, TC, BM, BN, BK, TM, TN, ST, AS>, smem, allowed);                     \
      if (rc) return rc;                                                                                                         \
    }                                                                                                                            \
    return qv_launch(gemm_simt_kernel<TA, TW, TC, BM, BN, BK, TM, TN, ST, AS>, grid, dim3((BM / TM) * (BN / TN)), smem, st, (TC*)C, \
                     (const TA*)A, (const TW*)W, M, N, K, lda, ldw, ldc, (flags & 0xff) != 0, flags & GS_SETTLED, GluAct{0, 0.f, 0.f}); \
  } while (0)
  if (small) {
    if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4) {
      if (async && (long long)grid.x * grid.y <= 148) GS_LAUNCH(16, 32, 64, 2, 2, 8, true);      // a CTA an SM
      if (async) GS_LAUNCH(16, 32, 64, 2, 2, 3, true);
    }
    GS_LAUNCH(16, 32, 64, 2, 2, 2, false);
  }
  if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4) {
    if (async) GS_LAUNCH(64, 64, 32, 4, 4, 2, true);
  }
  GS_LAUNCH(64, 64, 32, 4, 4, 2, false);
#undef GS_LAUNCH
}

// dtypes: a_dt/w_dt/c_dt in {f32, bf16}; flags: 1 adds to what C holds, GS_SETTLED: no launch that may still run writes W, which the
// kernel then reads ahead of its wait for the launch in front.
extern "C" int qv_gemm_simt(void* C, const void* A, const void* W, int M, int N, int K, int lda,
                            int ldw, int ldc, int a_dt, int w_dt, int c_dt, int flags,
                            void* stream) {
  if (M <= 0 || N <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const int key = a_dt * 4 + w_dt * 2 + c_dt;
  switch (key) {
    case 0: return launch<float, float, float>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
    case 1: return launch<float, float, bf16>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
    case 2: return launch<float, bf16, float>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
    case 3: return launch<float, bf16, bf16>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
    case 4: return launch<bf16, float, float>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
    case 5: return launch<bf16, float, bf16>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
    case 6: return launch<bf16, bf16, float>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
    case 7: return launch<bf16, bf16, bf16>(C, A, W, M, N, K, lda, ldw, ldc, flags, st);
  }
  return QV_ERR_UNSUPPORTED;
}

// C[M, N / 2] = act(gate) * up for W [N, K] with gate and up rows in groups of 16, float32 throughout; act as GluAct::kind.  Products of one wave of
// 16 x 32 tiles in whole 16-byte pieces only (QV_ERR_UNSUPPORTED else: the product and the activation are then two launches).  settled: as
// GS_SETTLED.
extern "C" int qv_gemm_simt_glu(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int act, float limit, float slope,
                                int settled, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (act < 0 || act > 2 || N % 32 || ((lda | ldw | K) & 3) || (((uintptr_t)A | (uintptr_t)W) & 15)) return QV_ERR_UNSUPPORTED;
  if (C < A + (size_t)(M - 1) * lda + K && A < C + (size_t)(M - 1) * ldc + N / 2) return QV_ERR_UNSUPPORTED;      // a result over its own rows: two launches
  const dim3 grid(N / 32, (M + 15) / 16);
  const bool small = M <= 32 || (long long)((N + 63) / 64) * ((M + 63) / 64) < 148;
  if (!small || (long long)grid.x * grid.y > 148) return QV_ERR_UNSUPPORTED;
  constexpr size_t smem = (size_t)8 * (16 + 32) * (64 + 4) * 4;
  auto kernel = gemm_simt_kernel<float, float, float, 16, 32, 64, 2, 2, 8, true, true>;
  static PerDevice allowed;
  const int rc = qv_allow_smem(kernel, smem, allowed);
  if (rc) return rc;
  return qv_launch(kernel, grid, dim3(128), smem, (cudaStream_t)stream, C, A, W, M, N, K, lda, ldw, ldc, 0, settled,
                   GluAct{act, limit, slope});
}
