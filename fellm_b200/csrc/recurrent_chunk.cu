// Recurrences whose decay depends on the token (recurrent.cu's delta rule, decay with a bonus, gated write) over prompt
// portions, in chunks of 32 tokens, float32 arithmetic on CUDA cores.
//
// All of them are, per head with a state S [dk, dv] and per token vectors A, B, G, K [dk], v [dv] and scalars beta, c,
//     u_t = beta_t (v_t - S_(t-1)^T A_t)   (delta rule)      or   u_t = v_t
//     o_t = S_(t-1)^T B_t + c_t u_t
//     S_t = diag(G_t) S_(t-1) + K_t u_t^T
// With P_t = G_1 .. G_t (element by element, t counted from the chunk's first token) and D_(t,s) = G_(s+1) .. G_t, a chunk
// that starts from the state S needs no walk over its tokens:
//     L_ts = sum_i A_ti D_(t-1,s),i K_si,   M_ts = sum_i B_ti D_(t-1,s),i K_si  (s < t),   M_tt = c_t
//     (I + diag(beta) L) U = diag(beta) (V - (P_(t-1) A_t)_t S)        (forward substitution, a column a thread)
//     O = (P_(t-1) B_t)_t S + M U,      S' = diag(P_last) S + (D_(last,s) K_s)_s^T U
// Every factor is a product of decays, formed by multiplication alone: no logarithm, no division, so a decay of zero or
// one that underflows is what it is in the token-by-token walk.
//
// Two kernels.  `prep` (a block a chunk and head, all side by side): the token vectors, L and M with one running product a
// column, the substitution for (P A) and V, the scaled B and K.  `walk` (a block a head and 16 value columns): chunk
// after chunk, the state in registers, three small products a chunk; the next chunk's operands arrive by cp.async meanwhile.
// Bound by: walk, its float32 multiply-adds (a chunk of 32 tokens at dk = 128: 0.16 M a block, 1,250 cycles at 128 a
// cycle) and the shared-memory reads and five barriers around them; the scan walks one token after another, a reduction
// over dk and ~500 cycles each.  16 columns a block: a prompt of 16 heads of 128 is 128 blocks for 148 SMs.
// 32 tokens a chunk: L and M cost 32 / 2 multiply-adds a token, channel and matrix, an eighth of the walk's.
//
// A later token's infinity or NaN stays out of an earlier token's sums, as in the walk token by token: masked pairs are
// skipped or selected away, never multiplied by zero.
//
// Sums run in another order than the scan's (equal up to float32 rounding), so the engine uses this form for portions of
// the bfloat16 engine; the 32-bit engine keeps the scan and with it the same bits for a prompt under every cut.
// A head's state lies column by column in its slot (element (i, j) at j * dk + i), as the scan keeps it.
#include "common.cuh"

#define RK_C 32            // tokens of a chunk
#define RK_NV 16           // value columns of a walk's block
#define RK_LP 36           // row stride of a chunk's 32 x 32 matrices
#define RK_THREADS 256

enum RkMode { RK_DELTA_HEAD = 0, RK_DELTA_CHANNEL = 1, RK_DECAY_BONUS = 2, RK_GATED_WRITE = 3 };

struct RkArgs {
  const void* q; const void* k; const void* v; int ld, v_off;      // rows of ld elements: q (or r; q raw), k (or f raw) behind their own pointers, v at v + v_off
  const float* small; int lds, b_off, a_off;                       // delta: beta's logit, the per-head decay's logit
  const float* A_log; const float* dt_bias;
  const float* gch;                                                // decay per channel [T, H dk]
  const float* bonus;                                              // [H, dk]
  const float* lower; const float* fbias;                          // gated write [H dk]
  const int* item_start; const int* item_slot;
  float* state; long long slot_stride;
  float* out;                                                      // [T, H dv]
  float* W; float* Q; float* K; float* U; float* M; float* P;      // per (chunk, head): [32][dk] x 3, [32][dv], [32][36], [dk]
  int H, G, dv, min_rows;
};

// Chunks of an item lie behind one another from here on: rows before it / 32 + its number is free of overlaps, and the
// chunks of a step are at most T / 32 + items.
__device__ __forceinline__ int rk_first_chunk(int row0, int item) { return row0 / RK_C + item; }

template <int E> __device__ __forceinline__ void rk_load(const float* p, float* o) {
  if (E == 4) { const float4 f = *(const float4*)p; o[0] = f.x; o[1] = f.y; o[E - 2] = f.z; o[E - 1] = f.w; }
  else { const float2 f = *(const float2*)p; o[0] = f.x; o[1] = f.y; }
}
template <int E> __device__ __forceinline__ void rk_load(const bf16* p, float* o) {
#pragma unroll
  for (int e = 0; e < E; e += 2) { const float2 f = __bfloat1622float2(*(const __nv_bfloat162*)(p + e)); o[e] = f.x; o[e + 1] = f.y; }
}
template <int E> __device__ __forceinline__ void rk_store(float* p, const float* o) {
  if (E == 4) *(float4*)p = make_float4(o[0], o[1], o[E - 2], o[E - 1]);
  else *(float2*)p = make_float2(o[0], o[1]);
}
__device__ __forceinline__ float rk_softplus(float v) { return v > 20.f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float rk_sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }

// ---------------------------------------------------------------- prep
template <int MODE, int DK, typename TA>
__global__ void __launch_bounds__(RK_THREADS)
rk_prep_kernel(const RkArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* A = sm;                                   // [32][DK]
  float* B = A + RK_C * DK;
  float* Gd = B + RK_C * DK;
  float* KK = Gd + RK_C * DK;
  float* Lt = KK + RK_C * DK;                      // [s][t]: beta_t L_ts
  float* Mm = Lt + RK_C * RK_LP;                   // [t][s]
  float* beta = Mm + RK_C * RK_LP;
  float* cc = beta + RK_C;
  constexpr bool DELTA = MODE <= RK_DELTA_CHANNEL;
  constexpr int E = DK / 32;
  const int item = blockIdx.z, h = blockIdx.y, c = blockIdx.x;
  const int r0 = a.item_start[item], n = a.item_start[item + 1] - r0;
  if (n < a.min_rows || c * RK_C >= n) return;
  const int len = min(RK_C, n - c * RK_C), row0 = r0 + c * RK_C;
  const size_t cell = (size_t)(rk_first_chunk(r0, item) + c) * a.H + h;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = h / (a.H / a.G);
  for (int x = tid; x < RK_C * RK_LP; x += RK_THREADS) Mm[x] = 0.f;

  // ---- the token vectors: a warp takes tokens warp, warp + 8, ..; a lane E consecutive elements
  {
    const TA* qp = (const TA*)a.q + (size_t)g * DK + lane * E;
    const TA* kp = (const TA*)a.k + (size_t)g * DK + lane * E;
    float q[4][E], k[4][E], w[4][E], lb[4], la[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = warp + 8 * u;
#pragma unroll
      for (int e = 0; e < E; ++e) { q[u][e] = k[u][e] = 0.f; w[u][e] = 1.f; }
      lb[u] = la[u] = 0.f;
      if (t < len) {
        const size_t row = (size_t)(row0 + t);
        rk_load<E>(qp + row * a.ld, q[u]);
        rk_load<E>(kp + row * a.ld, k[u]);
        if (MODE == RK_DELTA_CHANNEL || MODE == RK_DECAY_BONUS) rk_load<E>(a.gch + (row * a.H + h) * DK + lane * E, w[u]);
        if (DELTA) lb[u] = a.small[row * a.lds + a.b_off + h];
        if (MODE == RK_DELTA_HEAD) la[u] = a.small[row * a.lds + a.a_off + h];
      }
    }
    const float rate = MODE == RK_DELTA_HEAD ? expf(a.A_log[h]) : 0.f, bias = MODE == RK_DELTA_HEAD ? a.dt_bias[h] : 0.f;
    float x0[E], x1[E];
    if (MODE == RK_DECAY_BONUS) rk_load<E>(a.bonus + (size_t)h * DK + lane * E, x0);
    if (MODE == RK_GATED_WRITE) { rk_load<E>(a.lower + (size_t)h * DK + lane * E, x0); rk_load<E>(a.fbias + (size_t)h * DK + lane * E, x1); }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = warp + 8 * u;
      float av[E], bv[E], gv[E], kv[E], cv = 0.f, be = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) { av[e] = bv[e] = kv[e] = 0.f; gv[e] = 1.f; }
      if (t < len) {                                              // (the same for a whole warp)
        if (DELTA) {
          float sq = 0.f, sk = 0.f, kq = 0.f;
#pragma unroll
          for (int e = 0; e < E; ++e) { sq = fmaf(q[u][e], q[u][e], sq); sk = fmaf(k[u][e], k[u][e], sk); kq = fmaf(k[u][e], q[u][e], kq); }
          sq = warp_sum(sq); sk = warp_sum(sk); kq = warp_sum(kq);
          const float kn = 1.0f / sqrtf(sk + 1e-6f);
          const float qn = 1.0f / (sqrtf(sq + 1e-6f) * sqrtf((float)DK));
          const float gs = MODE == RK_DELTA_HEAD ? expf(-rate * rk_softplus(la[u] + bias)) : 0.f;
#pragma unroll
          for (int e = 0; e < E; ++e) {
            gv[e] = MODE == RK_DELTA_CHANNEL ? w[u][e] : gs;
            kv[e] = k[u][e] * kn;
            av[e] = gv[e] * kv[e];
            bv[e] = gv[e] * (q[u][e] * qn);
          }
          cv = kq * kn * qn; be = rk_sigmoid(lb[u]);
        } else if (MODE == RK_DECAY_BONUS) {
#pragma unroll
          for (int e = 0; e < E; ++e) { bv[e] = q[u][e]; kv[e] = k[u][e]; gv[e] = w[u][e]; cv = fmaf(q[u][e] * x0[e], k[u][e], cv); }
          cv = warp_sum(cv); be = 1.f;
        } else {
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const float qq = q[u][e] / (1.0f + expf(-q[u][e]));
            const float f = fmaf(1.0f - x0[e], rk_sigmoid(k[u][e] + x1[e]), x0[e]);
            gv[e] = f; kv[e] = 1.0f - f; bv[e] = f * qq;
            cv = fmaf(kv[e], qq, cv);
          }
          cv = warp_sum(cv); be = 1.f;
        }
      }
      const int o = t * DK + lane * E;
      if (DELTA) rk_store<E>(A + o, av);
      rk_store<E>(B + o, bv); rk_store<E>(Gd + o, gv); rk_store<E>(KK + o, kv);
      if (lane == 0) { beta[t] = be; cc[t] = cv; }
    }
  }
  __syncthreads();

  // ---- L and M: eight lanes a column s (four columns a warp), channels 4 ig + 32 m + e a lane; X = D_(t-1,s) K_s
  {
    constexpr int MB = DK / 32;
    const int ig = lane & 7, s = 4 * warp + (lane >> 3);
    unsigned long long X[2 * MB];
#pragma unroll
    for (int m = 0; m < 2 * MB; ++m) X[m] = 0ull;
    for (int t = 4 * warp; t < len; ++t) {
      const int o = t * DK + 4 * ig;
      if (t > 4 * warp) {
        unsigned long long l2 = 0ull, m2 = 0ull;
#pragma unroll
        for (int m = 0; m < MB; ++m) {
          const ulonglong2 b = *(const ulonglong2*)(B + o + 32 * m);
          m2 = fma_f2(b.x, X[2 * m], m2); m2 = fma_f2(b.y, X[2 * m + 1], m2);
          if (DELTA) {
            const ulonglong2 x = *(const ulonglong2*)(A + o + 32 * m);
            l2 = fma_f2(x.x, X[2 * m], l2); l2 = fma_f2(x.y, X[2 * m + 1], l2);
          }
        }
        float lo, hi;
        unpack_f2(m2, lo, hi);
        float ms = lo + hi, ls = 0.f;
        if (DELTA) { unpack_f2(l2, lo, hi); ls = lo + hi; }
#pragma unroll
        for (int x = 1; x < 8; x <<= 1) {
          ms += __shfl_xor_sync(0xffffffffu, ms, x);
          if (DELTA) ls += __shfl_xor_sync(0xffffffffu, ls, x);
        }
        if (ig == 0 && t > s) {
          Mm[t * RK_LP + s] = ms;
          if (DELTA) Lt[s * RK_LP + t] = beta[t] * ls;
        }
      }
      const bool own = t == s;
      if (own && ig == 0) Mm[t * RK_LP + t] = cc[t];
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        const ulonglong2 gd = *(const ulonglong2*)(Gd + o + 32 * m);
        const ulonglong2 kk = *(const ulonglong2*)(KK + o + 32 * m);
        // (before its own token a column is not zero times a decay but zero)
        X[2 * m] = own ? kk.x : t < s ? 0ull : mul_f2(X[2 * m], gd.x);
        X[2 * m + 1] = own ? kk.y : t < s ? 0ull : mul_f2(X[2 * m + 1], gd.y);
      }
    }
  }
  __syncthreads();

  // ---- running products of the decays: forward into A and B (up to the token before), backward into K (behind the token)
  if (tid < DK) {
    float p = 1.f;
#pragma unroll 8
    for (int t = 0; t < RK_C; ++t) {
      const int o = t * DK + tid;
      const float gd = Gd[o];
      if (DELTA) A[o] *= p;
      B[o] *= p;
      p *= gd;
    }
    a.P[cell * DK + tid] = p;
  } else if (tid < 2 * DK) {
    float p = 1.f;
#pragma unroll 8
    for (int t = RK_C - 1; t >= 0; --t) {
      const int o = t * DK + tid - DK;
      KK[o] *= p;
      p *= Gd[o];
    }
  }
  __syncthreads();
  float* Qg = a.Q + cell * (RK_C * DK); float* Kg = a.K + cell * (RK_C * DK); float* Mg = a.M + cell * (RK_C * RK_LP);
  for (int x = tid * 4; x < RK_C * DK; x += RK_THREADS * 4) {
    *(float4*)(Qg + x) = *(const float4*)(B + x);
    *(float4*)(Kg + x) = *(const float4*)(KK + x);
  }
  for (int x = tid * 4; x < RK_C * RK_LP; x += RK_THREADS * 4) *(float4*)(Mg + x) = *(const float4*)(Mm + x);

  // ---- (I + beta L) [W | U0] = beta [P A | V], a column a thread; without the delta rule U0 = V
  float* Ug = a.U + cell * ((size_t)RK_C * a.dv); float* Wg = a.W + cell * (RK_C * DK);
  const TA* vp = (const TA*)a.v + a.v_off + (size_t)h * a.dv;
  for (int col = tid; col < (DELTA ? DK : 0) + a.dv; col += RK_THREADS) {
    const bool is_w = DELTA && col < DK;
    const int j = DELTA ? col - DK : col;
    float x[RK_C];
#pragma unroll
    for (int t = 0; t < RK_C; ++t) {
      x[t] = 0.f;
      if (is_w) x[t] = A[t * DK + col];
      else if (t < len) x[t] = to_f(vp[(size_t)(row0 + t) * a.ld + j]);
    }
    if (DELTA) {
#pragma unroll
      for (int t = 0; t < RK_C; ++t) x[t] *= beta[t];
#pragma unroll
      for (int s = 0; s < RK_C - 1; ++s)
#pragma unroll
        for (int t0 = (s + 1) & ~3; t0 < RK_C; t0 += 4) {
          const float4 l = *(const float4*)(Lt + s * RK_LP + t0);
          if (t0 > s) x[t0] = t0 < len ? fmaf(-l.x, x[s], x[t0]) : 0.f;
          if (t0 + 1 > s) x[t0 + 1] = t0 + 1 < len ? fmaf(-l.y, x[s], x[t0 + 1]) : 0.f;
          if (t0 + 2 > s) x[t0 + 2] = t0 + 2 < len ? fmaf(-l.z, x[s], x[t0 + 2]) : 0.f;
          x[t0 + 3] = t0 + 3 < len ? fmaf(-l.w, x[s], x[t0 + 3]) : 0.f;
        }
    }
#pragma unroll
    for (int t = 0; t < RK_C; ++t) {
      if (is_w) Wg[t * DK + col] = x[t];
      else Ug[(size_t)t * a.dv + j] = x[t];
    }
  }
}

// ---------------------------------------------------------------- walk
__device__ __forceinline__ void rk_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <bool DELTA, int DK>
struct RkStage {
  static constexpr int NR = DELTA ? 2 * RK_C : RK_C;          // rows of the product with the state: W under Q, or Q alone
  static constexpr int AP = DK + 4;                           // their stride: eight rows' 16 bytes in different banks
  static constexpr int A = 0, K = A + NR * AP, M = K + RK_C * DK, U = M + RK_C * RK_LP, P = U + RK_C * RK_NV, FLOATS = P + DK;
};

template <bool DELTA, int DK>
__device__ __forceinline__ void rk_fetch(const RkArgs& a, float* buf, size_t cell, int j0, int tid) {
  using S = RkStage<DELTA, DK>;
  constexpr int V = DK / 4;
  const float* Qg = a.Q + cell * (RK_C * DK); const float* Kg = a.K + cell * (RK_C * DK); const float* Wg = a.W + cell * (RK_C * DK);
  for (int x = tid; x < RK_C * V; x += RK_THREADS) {
    const int t = x / V, i = (x - t * V) * 4;
    if (DELTA) rk_copy16(buf + S::A + t * S::AP + i, Wg + t * DK + i);
    rk_copy16(buf + S::A + (t + (DELTA ? RK_C : 0)) * S::AP + i, Qg + t * DK + i);
    rk_copy16(buf + S::K + t * DK + i, Kg + t * DK + i);
  }
  const float* Mg = a.M + cell * (RK_C * RK_LP);
  for (int x = tid; x < RK_C * RK_LP / 4; x += RK_THREADS) rk_copy16(buf + S::M + 4 * x, Mg + 4 * x);
  const float* Ug = a.U + cell * ((size_t)RK_C * a.dv) + j0;
  for (int x = tid; x < RK_C * RK_NV / 4; x += RK_THREADS) {
    const int t = x / (RK_NV / 4), j = (x - t * (RK_NV / 4)) * 4;
    rk_copy16(buf + S::U + t * RK_NV + j, Ug + (size_t)t * a.dv + j);
  }
  if (tid < DK / 4) rk_copy16(buf + S::P + 4 * tid, a.P + cell * DK + 4 * tid);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <bool DELTA, int DK>
__global__ void __launch_bounds__(RK_THREADS)
rk_walk_kernel(const RkArgs a) {
  extern __shared__ __align__(16) float sm[];
  using S = RkStage<DELTA, DK>;
  constexpr int KW = DK / 8;                       // key rows of the state a warp keeps
  constexpr int RPL = KW / 8;                      // of them a lane
  constexpr int PP = RK_NV + 4;                    // row stride of the partial sums
  float* part = sm + 2 * S::FLOATS;                // [8 warps][NR][PP]
  float* Us = part + 8 * S::NR * PP;               // [32][16]
  float* St = Us + RK_C * RK_NV;                   // [8 warps][16 columns][KW], 16-byte groups swizzled by column / 4
  const int item = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * RK_NV;
  const int r0 = a.item_start[item], n = a.item_start[item + 1] - r0;
  if (n < a.min_rows || n <= 0) return;
  const int chunks = (n + RK_C - 1) / RK_C;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rg = lane >> 2, cg = lane & 3;
  const size_t cell0 = (size_t)rk_first_chunk(r0, item) * a.H + h;
  rk_fetch<DELTA, DK>(a, sm, cell0, j0, tid);

  // this lane's part of the state: rows warp * KW + RPL * rg + r, columns j0 + 4 cg + x
  float* slot = a.state + (size_t)a.item_slot[item] * a.slot_stride + (size_t)h * DK * a.dv;
  const int i0 = warp * KW + RPL * rg;
  float s[RPL][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int r = 0; r < RPL; ++r) s[r][x] = slot[(size_t)(j0 + 4 * cg + x) * DK + i0 + r];
  float* Sw = St + warp * (RK_NV * KW);
  constexpr int GM = KW / 4 - 1;                   // 16-byte groups of a column, less one
  auto put_state = [&]() {
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const int i = RPL * rg + r, col = 4 * cg + x;
        Sw[col * KW + 4 * ((i >> 2) ^ (cg & GM)) + (i & 3)] = s[r][x];
      }
  };
  put_state();

  for (int c = 0; c < chunks; ++c) {
    const float* buf = sm + (c & 1) * S::FLOATS;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();                               // this chunk's operands are here; the other buffer, the sums and U are free
    if (c + 1 < chunks) rk_fetch<DELTA, DK>(a, sm + ((c + 1) & 1) * S::FLOATS, cell0 + (size_t)(c + 1) * a.H, j0, tid);

    // ---- [W; Q] S over this warp's key rows: a lane rows rg + 8 m, columns 4 cg + x; pairs of key rows an operation
    {
      constexpr int NM = S::NR / 8;
      unsigned long long acc[NM][4];
#pragma unroll
      for (int m = 0; m < NM; ++m)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[m][x] = 0ull;
      const float* Ab = buf + S::A + rg * S::AP + warp * KW;
#pragma unroll
      for (int kk = 0; kk < KW / 4; ++kk) {
        ulonglong2 sv[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) sv[x] = *(const ulonglong2*)(Sw + (4 * cg + x) * KW + 4 * (kk ^ (cg & GM)));
#pragma unroll
        for (int m = 0; m < NM; ++m) {
          const ulonglong2 av = *(const ulonglong2*)(Ab + 8 * m * S::AP + 4 * kk);
#pragma unroll
          for (int x = 0; x < 4; ++x) { acc[m][x] = fma_f2(av.x, sv[x].x, acc[m][x]); acc[m][x] = fma_f2(av.y, sv[x].y, acc[m][x]); }
        }
      }
      float* pw = part + (warp * S::NR + rg) * PP + 4 * cg;
#pragma unroll
      for (int m = 0; m < NM; ++m) {
        float o[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) { float lo, hi; unpack_f2(acc[m][x], lo, hi); o[x] = lo + hi; }
        *(float4*)(pw + 8 * m * PP) = make_float4(o[0], o[1], o[2], o[3]);
      }
    }
    __syncthreads();

    // ---- the eight warps' sums in warp order; a thread a row and four columns
    const int row = tid >> 2, jc = 4 * (tid & 3);
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < S::NR) {
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float4 p = *(const float4*)(part + (w * S::NR + row) * PP + jc);
        r.x += p.x; r.y += p.y; r.z += p.z; r.w += p.w;
      }
    }
    const float* U = buf + S::U;
    if (DELTA) {
      if (row < RK_C) {
        const float4 u0 = *(const float4*)(U + row * RK_NV + jc);
        *(float4*)(Us + row * RK_NV + jc) = make_float4(u0.x - r.x, u0.y - r.y, u0.z - r.z, u0.w - r.w);
      }
      __syncthreads();
      U = Us;
    }

    // ---- O = Q S + M U: the threads that hold Q's rows
    const int t = DELTA ? row - RK_C : row;
    if (t >= 0 && t < RK_C) {
      const int rows_here = min(RK_C, n - c * RK_C);
      const float* Mt = buf + S::M + t * RK_LP;
#pragma unroll 2
      for (int x = 0; x < RK_C; x += 4) {
        if (x > (t | 7)) break;                    // (a warp's eight rows end together)
        const float4 m = *(const float4*)(Mt + x);
        const float mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 u = *(const float4*)(U + (x + e) * RK_NV + jc);
          if (x + e <= t) { r.x = fmaf(mm[e], u.x, r.x); r.y = fmaf(mm[e], u.y, r.y); r.z = fmaf(mm[e], u.z, r.z); r.w = fmaf(mm[e], u.w, r.w); }
        }
      }
      if (t < rows_here) *(float4*)(a.out + (size_t)(r0 + c * RK_C + t) * ((size_t)a.H * a.dv) + (size_t)h * a.dv + j0 + jc) = r;
    }

    // ---- S = P S + K^T U
    {
      const float* Kb = buf + S::K + i0;
      const float* Pb = buf + S::P + i0;
      float k1[RPL];
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        const float p = Pb[q];
#pragma unroll
        for (int x = 0; x < 4; ++x) s[q][x] *= p;
      }
#pragma unroll 8
      for (int t2 = 0; t2 < RK_C; ++t2) {
        if (RPL == 2) { const float2 f = *(const float2*)(Kb + t2 * DK); k1[0] = f.x; k1[RPL - 1] = f.y; }
        else k1[0] = Kb[t2 * DK];
        const float4 u = *(const float4*)(U + t2 * RK_NV + 4 * cg);
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          s[q][0] = fmaf(k1[q], u.x, s[q][0]); s[q][1] = fmaf(k1[q], u.y, s[q][1]);
          s[q][2] = fmaf(k1[q], u.z, s[q][2]); s[q][3] = fmaf(k1[q], u.w, s[q][3]);
        }
      }
    }
    __syncwarp();
    put_state();
    __syncwarp();
  }
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int r = 0; r < RPL; ++r) slot[(size_t)(j0 + 4 * cg + x) * DK + i0 + r] = s[r][x];
}

// ---------------------------------------------------------------- launches
template <int MODE, int DK, typename TA>
static int rk_launch(const RkArgs& a, int n_items, int max_rows, cudaStream_t stream) {
  constexpr bool DELTA = MODE <= RK_DELTA_CHANNEL;
  const size_t sm_prep = (size_t)(4 * RK_C * DK + 2 * RK_C * RK_LP + 2 * RK_C) * sizeof(float);
  using S = RkStage<DELTA, DK>;
  const size_t sm_walk = (size_t)(2 * S::FLOATS + 8 * S::NR * (RK_NV + 4) + RK_C * RK_NV + RK_NV * DK) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(rk_prep_kernel<MODE, DK, TA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_prep);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(rk_walk_kernel<DELTA, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_walk);
  if (e != cudaSuccess) return (int)e;
  rk_prep_kernel<MODE, DK, TA><<<dim3((max_rows + RK_C - 1) / RK_C, a.H, n_items), RK_THREADS, sm_prep, stream>>>(a);
  rk_walk_kernel<DELTA, DK><<<dim3(a.dv / RK_NV, a.H, n_items), RK_THREADS, sm_walk, stream>>>(a);
  return launch_status();
}

// Floats of scratch for a step of T rows.
FELLM_API long long fellm_recurrent_chunk_scratch(int T, int n_items, int H, int dk, int dv) {
  const long long chunks = T / RK_C + n_items;
  return chunks * H * ((long long)RK_C * (3 * dk + dv + RK_LP) + dk);
}

// mode 0 / 1: the delta rule with a decay per head / channel (q, k [T, G dk] and v [T, H dv] in rows of ld elements, as
// fellm_delta_scan takes them); 2: decay and bonus (r, k, v [T, H dk]); 3: gated write (q raw, f raw, v).  Items of fewer
// than min_rows rows are left alone.  16-byte rows: see the checks.
FELLM_API int fellm_recurrent_chunk(int mode, const void* q, const void* k, const void* v, int is_bf16, int ld, int v_off,
                                    const float* small, int lds, int b_off, int a_off, const float* A_log, const float* dt_bias,
                                    const float* gch, const float* bonus, const float* lower, const float* fbias, float* state,
                                    long long slot_stride, const int* item_start, const int* item_slot, float* out, float* scratch,
                                    int T, int n_items, int max_rows, int min_rows, int H, int G, int dk, int dv, cudaStream_t stream) {
  if (n_items <= 0 || T <= 0) return 0;
  if ((dk != 64 && dk != 128) || dv < RK_NV || dv % RK_NV || H < 1 || G < 1 || H % G || max_rows < 1 || min_rows < 1 || mode < 0 || mode > 3 ||
      n_items > 65535 || H > 65535) return FELLM_ERR_SIZE;
  if (!q || !k || !v || !state || !item_start || !item_slot || !out || !scratch) return FELLM_ERR_ARG;
  if ((mode <= 1 && !small) || (mode == 0 && (!A_log || !dt_bias)) || ((mode == 1 || mode == 2) && !gch) || (mode == 2 && !bonus) ||
      (mode == 3 && (!lower || !fbias)) || (mode == 3 && is_bf16)) return FELLM_ERR_ARG;
  // vector loads: a lane's 2 or 4 elements; the scratch and the outputs in 16 bytes
  const uintptr_t mask = (uintptr_t)(dk / 32) * (is_bf16 ? 2 : 4) - 1, rows = (uintptr_t)ld * (is_bf16 ? 2 : 4);
  const uintptr_t fm = (uintptr_t)(dk / 32) * 4 - 1;
  if ((((uintptr_t)q | (uintptr_t)k | rows) & mask) || (((uintptr_t)gch | (uintptr_t)bonus | (uintptr_t)lower | (uintptr_t)fbias) & fm) ||
      (((uintptr_t)scratch | (uintptr_t)out) & 15)) return FELLM_ERR_SIZE;
  RkArgs a = {};
  a.q = q; a.k = k; a.v = v; a.ld = ld; a.v_off = v_off; a.small = small; a.lds = lds; a.b_off = b_off; a.a_off = a_off;
  a.A_log = A_log; a.dt_bias = dt_bias; a.gch = gch; a.bonus = bonus; a.lower = lower; a.fbias = fbias;
  a.item_start = item_start; a.item_slot = item_slot; a.state = state; a.slot_stride = slot_stride; a.out = out;
  a.H = H; a.G = G; a.dv = dv; a.min_rows = min_rows;
  const size_t cells = (size_t)(T / RK_C + n_items) * H;
  a.W = scratch; a.Q = a.W + cells * (RK_C * dk); a.K = a.Q + cells * (RK_C * dk); a.U = a.K + cells * (RK_C * dk);
  a.M = a.U + cells * ((size_t)RK_C * dv); a.P = a.M + cells * (RK_C * RK_LP);
#define RK_GO(MODE_, TA_) (dk == 128 ? rk_launch<MODE_, 128, TA_>(a, n_items, max_rows, stream) : rk_launch<MODE_, 64, TA_>(a, n_items, max_rows, stream))
  if (mode == 0) return is_bf16 ? RK_GO(0, bf16) : RK_GO(0, float);
  if (mode == 1) return is_bf16 ? RK_GO(1, bf16) : RK_GO(1, float);
  if (mode == 2) return is_bf16 ? RK_GO(2, bf16) : RK_GO(2, float);
  return RK_GO(3, float);
#undef RK_GO
}
