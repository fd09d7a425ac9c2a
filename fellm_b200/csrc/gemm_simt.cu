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
// four k of a row at a time (row stride 36 floats: the 8 rows of a quarter warp in different banks), the next four's on their
// way under the sums.  A 16-byte load takes four wavefronts of shared memory, two where lanes one or two apart ask for the same: a
// warp's 4 x 8 threads have rows and columns in alternate bits of the lane's number, 16 wavefronts for the 16 cycles of its 4 x 4 x 4
// multiply-adds (24 before).  Bound by those and, with few warps, by their latency.  us at K = 1,024, loads numbered row after row and
// used as they came / now: [201, 2048] 47 / 33, [201, 1024] 39 / 20, [256, 9216] 146 / 114, [48, 1024] 25 / 10, [8, 1024] 18 / 10.
// The tile: 16 x 32 of 2 x 2 outputs a thread takes some 5.6 us a block and SM side by side, 64 x 64 of 4 x 4 29 and never less
// than 33: the latter where that is less and its rows are filled ([256, 9216] 114 / 163, [33, 6176] 34 / 23, [201, 2048] 35 / 33, [256, 1024],
// K = 4,608 151 / 94).  8 x 32 for up to 8 rows.
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
  // a warp is 4 x 8 threads of the tile, rows in bits 0 and 4 of the lane's number, columns in bits 1 to 3
  static_assert(TX % 8 == 0 && TY % 4 == 0, "a warp is 4 x 8 threads");
  const int tid = threadIdx.x, lane = tid & 31, wx = (tid >> 5) % (TX / 8), wy = (tid >> 5) / (TX / 8);
  const int tx = 8 * wx + ((lane >> 1) & 7), ty = 4 * wy + (lane & 1) + 2 * (lane >> 4);
  const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
  // a thread's copies: the same rows in every step, 16 bytes each
  constexpr int COPIES = ((TBM + TBN) * (FP_BK / 4) + THREADS - 1) / THREADS, APART = THREADS / (FP_BK / 4);
  constexpr bool WHOLE = COPIES * THREADS == (TBM + TBN) * (FP_BK / 4);           // every thread has as many
  const float* src[COPIES];
  bool in[COPIES];
  const int r0 = tid / (FP_BK / 4), kq = (tid % (FP_BK / 4)) * 4;
#pragma unroll
  for (int c = 0; c < COPIES; ++c) {
    const int r = r0 + c * APART, row = r < TBM ? m0 + r : n0 + r - TBM;
    in[c] = row < (r < TBM ? M : N);
    src[c] = !in[c] ? A : (r < TBM ? A + (size_t)row * lda : W + (size_t)row * ldw) + kq;
  }
  auto fetch = [&](int step) {
    float* st = fp_smem + (step % FP_STAGES) * STAGE + r0 * FP_LD + kq;
    const int k0 = step * FP_BK;
    const bool k_in = k0 + kq < K;
#pragma unroll
    for (int c = 0; c < COPIES; ++c)
      if (WHOLE || r0 + c * APART < TBM + TBN) fp_copy16(st + c * APART * FP_LD, in[c] && k_in ? src[c] + k0 : A, in[c] && k_in);
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
    // four k at a time, the next four's on their way under the sums
    float4 a[2][TM], w[2][TN];
    auto read = [&](int k, int to) {
#pragma unroll
      for (int i = 0; i < TM; ++i) a[to][i] = *(const float4*)(As + TY * i * FP_LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[to][j] = *(const float4*)(Ws + TX * j * FP_LD + k);
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < FP_BK; k += 4) {
      const int at = (k >> 2) & 1;
      if (k + 4 < FP_BK) read(k + 4, at ^ 1);
      // (each output's chain in the order of k)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[at][i].x, w[at][j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[at][i].y, w[at][j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[at][i].z, w[at][j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[at][i].w, w[at][j].w, acc[i][j]);
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
    const long long large = (long long)ceil_div(N, 64) * ceil_div(M, 64), small = (long long)ceil_div(N, 32) * ceil_div(M, 16);
    if (10 * small > 59ll * sms && 10 * small > 52 * large) return launch_f32<64, 64, 4, 4>(a, w, bias, (float*)C, M, N, K, lda, ldw, ldc, epi, s);
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
