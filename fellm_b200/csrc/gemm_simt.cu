// C[M,N] = A[M,K] * W[N,K]^T on CUDA cores with float32 FMA: the true 32-bit matrix product
// (no TF32, no reduced-precision staging), and the product for any mix of bfloat16/float32
// operands that the tensor-core kernels do not take.
//
// FeLLM counterpart: bf16_matmul_rows / f32_matmul_rows, one thread per output
// (plugins/cuda_kernels/src/oxide_kernels.rs:3165-3225).  Like them, every output element is one
// chain acc = fma(a[m,k], w[n,k], acc) for k = 0..K-1, so its value does not depend on M, on the
// tile it falls in, or on what else is in the batch.
#include "common.cuh"

#define BM 64
#define BN 64
#define BK 16

// EPI 0: C = acc (+bias);  EPI 2: C = max(acc (+bias), 0)^2;  EPI 1: C(float) = C + acc (+bias)   (residual accumulate)
template <typename TA, typename TW, typename TO, int EPI>
__global__ void __launch_bounds__(256)
gemm_tn_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const float* __restrict__ bias,
                    TO* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc,
                    long long sa = 0, long long sw = 0, long long sc = 0) {
  FELLM_TRACE_SCOPE(TRACE_GEMM_SIMT);
  // a batch of products (blockIdx.z): member b reads A + b sa, W + b sw and writes C + b sc (elements)
  A += (size_t)blockIdx.z * sa; W += (size_t)blockIdx.z * sw; C += (size_t)blockIdx.z * sc;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  int tid = threadIdx.x;
  int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads, 4 x 4 outputs each
  int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 rows x 16 k = 1024 elements per operand, 4 per thread; k fastest for coalescing
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int e = tid + i * 256;
      int r = e >> 4, kk = e & 15;
      int gm = m0 + r, gn = n0 + r, gk = k0 + kk;
      As[kk][r] = (gm < M && gk < K) ? to_f(A[(size_t)gm * lda + gk]) : 0.f;
      Ws[kk][r] = (gn < N && gk < K) ? to_f(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      if (EPI == 2) { v = fmaxf(v, 0.f); v *= v; }
      size_t o = (size_t)gm * ldc + gn;
      if (EPI == 1) C[o] = from_f<TO>(to_f(C[o]) + v);
      else C[o] = from_f<TO>(v);
    }
  }
}

// All three float32, rows that start on 16 bytes and K a multiple of 4: the same chains, fed by cp.async through a ring of
// FP_STAGES stages of 32 k.  A thread keeps TM x TN outputs whose rows and columns are TBM / TM and TBN / TN apart, and reads
// four k of a row at a time (row stride 36 floats: the 8 rows of a quarter warp in different banks).  Bound by those reads
// where rows are many (4 x 4 outputs: 32 floats from shared memory for 64 multiply-adds) and by the warps' latency: 8 x 4
// outputs a thread halve the warps and take 49 and 63 us where 4 x 4 take 48 ([201, 2048, 1024]) and 44 ([201, 1024, 1024]); the
// kernel above, without loads in flight under its sums, takes 95 for either.  Tiles of 64 x 64 where they fill three
// quarters of the SMs, of 32 x 64 where those fill half, else 16 x 32 and 8 x 32 with few outputs a thread: a product of a
// decode step is a few chains of K dependent multiply-adds, and more warps walk them side by side.
#define FP_STAGES 4
#define FP_BK 32
#define FP_LD 36
__device__ __forceinline__ void fp_copy16(float* dst, const float* src, bool live) {
  const int n = live ? 16 : 0;                     // (0: the 16 bytes are zeros)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(n) : "memory");
}

template <int TBM, int TBN, int TM, int TN, int EPI>
__global__ void __launch_bounds__(TBM * TBN / (TN * TM))
gemm_tn_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                   float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
  FELLM_TRACE_SCOPE(TRACE_GEMM_SIMT);
  extern __shared__ __align__(16) float fp_smem[];
  constexpr int THREADS = TBM * TBN / (TN * TM), TX = TBN / TN, TY = TBM / TM, STAGE = (TBM + TBN) * FP_LD;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
  auto fetch = [&](int step) {
    float* st = fp_smem + (step % FP_STAGES) * STAGE;
    const int k0 = step * FP_BK;
    for (int x = tid; x < (TBM + TBN) * (FP_BK / 4); x += THREADS) {
      const int r = x / (FP_BK / 4), k = k0 + (x % (FP_BK / 4)) * 4;
      const bool is_a = r < TBM;
      const int row = is_a ? m0 + r : n0 + r - TBM;
      const bool live = k < K && row < (is_a ? M : N);
      fp_copy16(st + r * FP_LD + k - k0, live ? (is_a ? A + (size_t)row * lda + k : W + (size_t)row * ldw + k) : A, live);
    }
  };
  const int steps = (K + FP_BK - 1) / FP_BK;
#pragma unroll
  for (int s = 0; s < FP_STAGES - 1; ++s) {
    if (s < steps) fetch(s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(FP_STAGES - 2) : "memory");
    __syncthreads();                               // this stage is here; the one before it is free
    if (s + FP_STAGES - 1 < steps) fetch(s + FP_STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* As = fp_smem + (s % FP_STAGES) * STAGE + ty * FP_LD;
    const float* Ws = fp_smem + (s % FP_STAGES) * STAGE + (TBM + tx) * FP_LD;
#pragma unroll
    for (int k = 0; k < FP_BK; k += 4) {
      float4 a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *(const float4*)(As + TY * i * FP_LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *(const float4*)(Ws + TX * j * FP_LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {              // (each output's chain in the order of k)
          acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]); acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]); acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
        }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty + TY * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx + TX * j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      if (EPI == 2) { v = fmaxf(v, 0.f); v *= v; }
      const size_t o = (size_t)gm * ldc + gn;
      C[o] = EPI == 1 ? C[o] + v : v;
    }
  }
}

template <int TBM, int TBN, int TM, int TN>
static int launch_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, int epi,
                      cudaStream_t s) {
  auto kern = epi == 2 ? gemm_tn_f32_kernel<TBM, TBN, TM, TN, 2> : epi ? gemm_tn_f32_kernel<TBM, TBN, TM, TN, 1> : gemm_tn_f32_kernel<TBM, TBN, TM, TN, 0>;
  const int smem = FP_STAGES * (TBM + TBN) * FP_LD * (int)sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  kern<<<dim3(ceil_div(N, TBN), ceil_div(M, TBM)), TBM * TBN / (TN * TM), smem, s>>>(A, W, bias, C, M, N, K, lda, ldw, ldc);
  return launch_status();
}

template <typename TA, typename TW, typename TO>
static int launch_epi(const void* A, const void* W, const float* bias, void* C, int M, int N, int K,
                      int lda, int ldw, int ldc, int epi, cudaStream_t s) {
  dim3 grid(ceil_div(N, BN), ceil_div(M, BM));
  if (epi == 2)
    gemm_tn_simt_kernel<TA, TW, TO, 2><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, bias, (TO*)C, M, N, K, lda, ldw, ldc);
  else if (epi)
    gemm_tn_simt_kernel<TA, TW, TO, 1><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, bias, (TO*)C, M, N, K, lda, ldw, ldc);
  else
    gemm_tn_simt_kernel<TA, TW, TO, 0><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, bias, (TO*)C, M, N, K, lda, ldw, ldc);
  return launch_status();
}

// dtype codes: 0 = float32, 1 = bfloat16.  epi: 0 store, 1 add into C (float32), 2 store max(v, 0)^2.
FELLM_API int fellm_gemm_simt(const void* A, int a_dt, const void* W, int w_dt, const float* bias,
                              void* C, int c_dt, int M, int N, int K, int lda, int ldw, int ldc,
                              int epi, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  if (!A || !W || !C || K <= 0) return FELLM_ERR_ARG;
  if (epi < 0 || epi > 2 || (epi == 1 && c_dt != 0)) return FELLM_ERR_ARG;
  int key = a_dt * 4 + w_dt * 2 + c_dt;
  if (key == 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && !(((uintptr_t)A | (uintptr_t)W) & 15)) {
    const float *a = (const float*)A, *w = (const float*)W;
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 148;
    if (M > 32 && (long long)ceil_div(N, 64) * ceil_div(M, 64) >= sms * 3 / 4) return launch_f32<64, 64, 4, 4>(a, w, bias, (float*)C, M, N, K, lda, ldw, ldc, epi, s);
    if (M > 16 && (long long)ceil_div(N, 64) * ceil_div(M, 32) >= sms / 2) return launch_f32<32, 64, 4, 4>(a, w, bias, (float*)C, M, N, K, lda, ldw, ldc, epi, s);
    if (M > 8) return launch_f32<16, 32, 2, 2>(a, w, bias, (float*)C, M, N, K, lda, ldw, ldc, epi, s);
    return launch_f32<8, 32, 2, 1>(a, w, bias, (float*)C, M, N, K, lda, ldw, ldc, epi, s);
  }
  switch (key) {
    case 0: return launch_epi<float, float, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, epi, s);
    case 2: return launch_epi<float, bf16, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, epi, s);
    case 4: return launch_epi<bf16, float, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, epi, s);
    case 5: return launch_epi<bf16, float, bf16>(A, W, bias, C, M, N, K, lda, ldw, ldc, epi, s);
    case 6: return launch_epi<bf16, bf16, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, epi, s);
    case 7: return launch_epi<bf16, bf16, bf16>(A, W, bias, C, M, N, K, lda, ldw, ldc, epi, s);
    default: return FELLM_ERR_ARG;   // float32 activations never round down to a bfloat16 result
  }
}

// A batch of such products in one launch: member b computes C_b[M, N] = A_b[M, K] W_b[N, K]^T with A_b = A + b sa,
// W_b = W + b sw, C_b = C + b sc (strides in elements): the heads of a layer, each with a matrix of its own, on
// column blocks of the same rows.  Every output is the same k-ordered chain as in the single product.
FELLM_API int fellm_gemm_simt_batched(const void* A, int a_dt, const void* W, int w_dt, void* C, int c_dt, int batch,
                                      int M, int N, int K, int lda, int ldw, int ldc, long long sa, long long sw,
                                      long long sc, cudaStream_t s) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (!A || !W || !C || K <= 0) return FELLM_ERR_ARG;
  if (batch > 65535) return FELLM_ERR_SIZE;
  dim3 grid(ceil_div(N, BN), ceil_div(M, BM), batch);
#define BATCHED(TA_, TW_, TO_) gemm_tn_simt_kernel<TA_, TW_, TO_, 0><<<grid, 256, 0, s>>>((const TA_*)A, (const TW_*)W, nullptr, (TO_*)C, M, N, K, lda, ldw, ldc, sa, sw, sc)
  switch (a_dt * 4 + w_dt * 2 + c_dt) {
    case 0: BATCHED(float, float, float); break;
    case 2: BATCHED(float, bf16, float); break;
    case 4: BATCHED(bf16, float, float); break;
    case 5: BATCHED(bf16, float, bf16); break;
    case 6: BATCHED(bf16, bf16, float); break;
    case 7: BATCHED(bf16, bf16, bf16); break;
    default: return FELLM_ERR_ARG;
  }
#undef BATCHED
  return launch_status();
}
