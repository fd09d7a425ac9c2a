// Recurrences whose decay depends on the token (recurrent.cu's delta rule, decay with a bonus, gated write) over prompt
// portions, in chunks of 32 tokens, on CUDA cores: float32, the sums that every later one hangs on in 64 bits.
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
// `prep` (a block a chunk and head, all side by side): the token vectors, L and M with one running product a column, the
// substitution for (P A) and V, the scaled B and K.  Then, in one `walk` (a block a head and 16 value columns), states and outputs
// chunk after chunk; or, for long portions, what hangs together in a chain first and the outputs of all chunks side by
// side behind it (`out`): with the delta rule the `chain` W S, K^T U (the state in front of every chunk goes to memory), without
// it the `states` S' = P S + K^T V, element by element.  Each sum in the walk's order: a portion's bits do not depend on which of the two runs.
// Bound by: the reads of shared memory.  A load of 16 bytes a lane takes four wavefronts, or two where lanes one or two apart ask for the
// same (of 8 bytes: two or one), whatever else they share; so a tile's row and column groups lie in alternate bits of the
// lane's number (walk 188 -> 158 us, prep 85 -> 74 of the first size below, with the same bits).  A lane's tile of 4 x 4 (or 2 x 4) results then takes a wavefront for
// about every FMA instruction of a warp.  16 columns a block: a prompt of 16 heads of 128 is 128 blocks for 148 SMs.
// 2,048 tokens of 16 heads of 128 x 128, delta rule: scan 791 us, prep 85 + walk 188 as it was, here prep 74 + chain 105 + out 44 (one walk:
// 158), graph of the three 269 -> 215; decay per channel 284 -> 226; three prompts of 1,537 tokens, 8 heads, gated write: scan 274, 100 -> 64;
// 1,100 tokens in two prompts, 16 heads of 64, decay and bonus 69 -> 44.
// 32 tokens a chunk: L and M cost 32 / 2 multiply-adds a token, channel and matrix, an eighth of the walk's.
//
// A later token's infinity or NaN stays out of an earlier token's sums, as in the walk token by token: masked pairs are
// skipped or selected away, never multiplied by zero.
//
// Rounding: with float32 throughout, the substitution's 31 steps and the sums of 128 products behind L, M and c made the delta
// rule's results less exact than the walk token by token.  So in prep the lanes' partial sums of those products are joined
// in 64 bits, the substitution runs in them (a finished row is rounded once, to what walk works with), and the running
// products of the decays are sums of two floats.  Relative error against float64, scan / here, mean over five sizes and
// three seeds: delta rule outputs 1.34e-7 / 1.22e-7, states 9.0e-8 / 8.6e-8, with keys nearly alike and beta 0.99 1.45e-7 /
// 1.35e-7, 8.7e-8 / 8.4e-8; decay per channel 1.22e-7 / 1.08e-7, 7.8e-8 / 7.3e-8; decay and bonus 8.3e-8 / 6.8e-8, 3.15e-8 /
// 3.09e-8; gated write 6.2e-8 / 5.9e-8, 1.09e-7 / 1.07e-7.  It costs 6 us of the 263 of the first size above (21 of 264 with a
// decay per channel, 4 of 68 with a bonus; the gated write gains 5 of 106 through its smaller blocks).
// Sums run in another order than the scan's, so the engine uses this form for portions of the bfloat16 engine; the 32-bit
// engine keeps the scan and with it the same bits for a prompt under every cut.
// A head's state lies column by column in its slot (element (i, j) at j * dk + i), as the scan keeps it.
#include "common.cuh"

#define RK_C 32            // tokens of a chunk
#define RK_NV 16           // value columns of a walk's block
#define RK_LP 36           // row stride of a chunk's 32 x 32 matrices in the image
#define RK_LM 34           // and, in 64 bits, in prep's shared memory
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
  float* image; float* U; float* S;                                // per (chunk, head): an RkImage; [dv / 16][32][16]; the state in front of it [dv][dk] (or null: outputs in the walk)
  int H, G, dv, min_rows, n_items, cells;                          // cells: places for the step's chunks
};

// Chunks of an item lie behind one another from here on: rows before it / 32 + its number is free of overlaps, and the
// chunks of a step are at most T / 32 + items.
__device__ __forceinline__ int rk_first_chunk(int row0, int item) { return row0 / RK_C + item; }

// Which item the step's chunk x belongs to: the last one whose chunks start at or before x (a place between two items' chunks belongs to
// nobody: its item's rows end before it).  The lanes of a warp look at 32 items at once.
__device__ __forceinline__ int rk_item_of(const int* item_start, int n_items, int x) {
  int item = 0;
  for (int i0 = 0; i0 < n_items; i0 += 32) {
    const int i = i0 + (threadIdx.x & 31);
    const unsigned before = __ballot_sync(0xffffffffu, i < n_items && rk_first_chunk(item_start[i], i) <= x);
    if (!before) break;
    item = i0 + 31 - __clz(before);
  }
  return item;
}

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

// warp_sum with one rounding at the end.
__device__ __forceinline__ float rk_sum(float v) {
  double d = v;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
  return (float)d;
}

// A running product of decays as an unrounded sum of two floats: its error stays below a rounding of the product, where a
// single float's grows with every factor.
struct RkProduct {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void by(float g) {
    const float p = hi * g, rest = fmaf(hi, g, -p);
    lo = fmaf(lo, g, rest); hi = p;
  }
  __device__ __forceinline__ float times(float v) const {
    const float r = v * hi;
    return fabsf(r) < INFINITY ? fmaf(v, hi, v * lo) : r;          // (an infinity times a rest of zero is not a number)
  }
};

// What prep leaves of a chunk and head, in the order its readers take it (their copies are then linear): the chain reads W, K and
// P, the states of the recurrences without the delta rule K and P, the outputs Q and M.
template <bool DELTA, int DK>
struct RkImage {
  static constexpr int AP = DK + 4;                           // row stride of W and Q: eight rows' 16 bytes in different banks
  static constexpr int W = 0, K = W + (DELTA ? RK_C * AP : 0), P = K + RK_C * DK, WALK = P + DK;
  static constexpr int Q = WALK, M = Q + RK_C * AP, FLOATS = M + RK_C * RK_LP, OUT = FLOATS - Q;
};

// ---------------------------------------------------------------- prep
template <int MODE, int DK, typename TA>
__global__ void __launch_bounds__(RK_THREADS, 3)
rk_prep_kernel(const RkArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* A = sm;                                   // [32][DK]
  float* B = A + RK_C * DK;
  float* Gd = B + RK_C * DK;
  float* KK = Gd + RK_C * DK;
  float* cc = KK + RK_C * DK;
  double* beta = (double*)(cc + RK_C);             // (delta)
  double* LM = beta + RK_C;                        // [32][RK_LM]: [s][t], t > s: beta_t L_ts; [t][s], s <= t: M_ts
  constexpr bool DELTA = MODE <= RK_DELTA_CHANNEL;
  constexpr int E = DK / 32;
  const int item = rk_item_of(a.item_start, a.n_items, blockIdx.x), h = blockIdx.y;
  const int r0 = a.item_start[item], n = a.item_start[item + 1] - r0, c = blockIdx.x - rk_first_chunk(r0, item);
  if (n < a.min_rows || c < 0 || c * RK_C >= n) return;           // (c < 0: rows in front of the first item)
  const int len = min(RK_C, n - c * RK_C), row0 = r0 + c * RK_C;
  const size_t cell = (size_t)blockIdx.x * a.H + h;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = h / (a.H / a.G);
  for (int x = tid; x < RK_C * RK_LM; x += RK_THREADS) LM[x] = 0.0;

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
          sq = rk_sum(sq); sk = rk_sum(sk); kq = rk_sum(kq);
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
          cv = rk_sum(cv);
        } else {
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const float qq = q[u][e] / (1.0f + expf(-q[u][e]));
            const float f = fmaf(1.0f - x0[e], rk_sigmoid(k[u][e] + x1[e]), x0[e]);
            gv[e] = f; kv[e] = 1.0f - f; bv[e] = f * qq;
            cv = fmaf(kv[e], qq, cv);
          }
          cv = rk_sum(cv);
        }
      }
      const int o = t * DK + lane * E;
      if (DELTA) rk_store<E>(A + o, av);
      rk_store<E>(B + o, bv); rk_store<E>(Gd + o, gv); rk_store<E>(KK + o, kv);
      if (lane == 0) { cc[t] = cv; if (DELTA) beta[t] = be; }
    }
  }
  __syncthreads();

  // ---- L and M: eight lanes a column s (four columns a warp), channels 4 ig + 32 m + e a lane; X = D_(t-1,s) K_s.
  // Four tokens a round: their (up to) eight sums go through the eight lanes together, seven shuffles for all of them.
  {
    constexpr int MB = DK / 32;
    const int ig = (lane >> 1) & 7, s = 4 * warp + (lane & 1) + 2 * (lane >> 4);        // (neighbouring lanes read the same)
    unsigned long long X[2 * MB];
#pragma unroll
    for (int m = 0; m < 2 * MB; ++m) X[m] = 0ull;
#pragma unroll 1
    for (int t0 = 4 * warp; t0 < len; t0 += 4) {
      const bool first = t0 == 4 * warp;                       // the columns' own tokens
      float sum[8];                                            // M of four tokens, L of four tokens
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = t0 + j, o = t * DK + 4 * ig;
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
        sum[j] = lo + hi;
        unpack_f2(l2, lo, hi);
        sum[4 + j] = lo + hi;
        if (first) {
          const bool own = t == s;
#pragma unroll
          for (int m = 0; m < MB; ++m) {
            const ulonglong2 gd = *(const ulonglong2*)(Gd + o + 32 * m);
            const ulonglong2 kk = *(const ulonglong2*)(KK + o + 32 * m);
            // (before its own token a column is not zero times a decay but zero)
            X[2 * m] = own ? kk.x : t < s ? 0ull : mul_f2(X[2 * m], gd.x);
            X[2 * m + 1] = own ? kk.y : t < s ? 0ull : mul_f2(X[2 * m + 1], gd.y);
          }
        } else {
#pragma unroll
          for (int m = 0; m < MB; ++m) {
            const ulonglong2 gd = *(const ulonglong2*)(Gd + o + 32 * m);
            X[2 * m] = mul_f2(X[2 * m], gd.x); X[2 * m + 1] = mul_f2(X[2 * m + 1], gd.y);
          }
        }
      }
      // lane ig ends with the whole of sum[4 (ig & 1) + 2 ((ig >> 1) & 1) + (ig >> 2)]
      const bool b0 = ig & 1, b1 = ig & 2, b2 = ig & 4;
      double q4[4], q2[2], v;                      // (the lanes' sums are joined in 64 bits, for half of the products' error)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float give = DELTA && !b0 ? sum[4 + j] : sum[j], keep = DELTA && b0 ? sum[4 + j] : sum[j];
        q4[j] = (double)keep + (double)__shfl_xor_sync(0xffffffffu, give, 2);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const double give = b1 ? q4[j] : q4[2 + j], keep = b1 ? q4[2 + j] : q4[j];
        q2[j] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
      }
      {
        const double give = b2 ? q2[0] : q2[1], keep = b2 ? q2[1] : q2[0];
        v = keep + __shfl_xor_sync(0xffffffffu, give, 8);
      }
      const int t = t0 + (b1 ? 2 : 0) + (b2 ? 1 : 0);
      if (t > s) {
        if (DELTA && b0) LM[s * RK_LM + t] = beta[t] * v;
        else if (!b0) LM[t * RK_LM + s] = v;
      } else if (t == s && !b0) LM[t * RK_LM + t] = (double)cc[t];
    }
  }
  __syncthreads();

  using I = RkImage<DELTA, DK>;
  float* img = a.image + cell * I::FLOATS;
  // ---- running products of the decays: forward into A and B (up to the token before), backward into K (behind the token)
  if (tid < DK) {
    RkProduct p;
#pragma unroll 8
    for (int t = 0; t < RK_C; ++t) {
      const int o = t * DK + tid;
      const float gd = Gd[o];
      if (DELTA) A[o] = p.times(A[o]);
      B[o] = p.times(B[o]);
      p.by(gd);
    }
    img[I::P + tid] = p.hi + p.lo;
  } else if (tid < 2 * DK) {
    RkProduct p;
#pragma unroll 8
    for (int t = RK_C - 1; t >= 0; --t) {
      const int o = t * DK + tid - DK;
      KK[o] = p.times(KK[o]);
      p.by(Gd[o]);
    }
  }
  __syncthreads();
  for (int x = tid * 4; x < RK_C * DK; x += RK_THREADS * 4) {
    const int t = x / DK, i = x - t * DK;
    *(float4*)(img + I::Q + t * I::AP + i) = *(const float4*)(B + x);
    *(float4*)(img + I::K + x) = *(const float4*)(KK + x);
  }
  for (int x = tid; x < RK_C * RK_C; x += RK_THREADS) {
    const int t = x / RK_C, s = x % RK_C;
    img[I::M + t * RK_LP + s] = s <= t ? (float)LM[t * RK_LM + s] : 0.f;
  }

  // ---- (I + beta L) [W | U0] = beta [P A | V], a column a thread; without the delta rule U0 = V
  float* Ug = a.U + cell * ((size_t)RK_C * a.dv);
  const TA* vp = (const TA*)a.v + a.v_off + (size_t)h * a.dv;
  for (int col = tid; col < (DELTA ? DK : 0) + a.dv; col += RK_THREADS) {
    const bool is_w = DELTA && col < DK;
    const int j = DELTA ? col - DK : col;
    auto put = [&](int t, float x) {
      if (is_w) img[I::W + t * I::AP + col] = x;
      else Ug[((size_t)(j / RK_NV) * RK_C + t) * RK_NV + j % RK_NV] = x;
    };
    if (DELTA) {
      // products and sums in 64 bits, half of the tokens at a time (their registers); a finished value is the float that the
      // walk over the chunks works with
      constexpr int HC = RK_C / 2;
      float done[HC];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float in[HC];
        double x[HC];
#pragma unroll
        for (int i = 0; i < HC; ++i) {
          const int t = half * HC + i;
          in[i] = 0.f;
          if (is_w) in[i] = A[t * DK + col];
          else if (t < len) in[i] = to_f(vp[(size_t)(row0 + t) * a.ld + j]);
        }
        asm volatile("" ::: "memory");             // (all on their way before the first is waited for)
#pragma unroll
        for (int i = 0; i < HC; ++i) x[i] = (double)in[i] * beta[half * HC + i];
        if (half) {
#pragma unroll
          for (int s = 0; s < HC; ++s) {
            const double xs = (double)done[s];
#pragma unroll
            for (int i = 0; i < HC; i += 2) {
              const double2 l = *(const double2*)(LM + s * RK_LM + HC + i);
              x[i] = fma(-l.x, xs, x[i]); x[i + 1] = fma(-l.y, xs, x[i + 1]);
            }
          }
        }
#pragma unroll
        for (int s = 0; s < HC; ++s) {
          const float f = (float)x[s];
          const double xs = (double)f;
          done[s] = f;
          put(half * HC + s, f);
#pragma unroll
          for (int i = (s + 1) & ~1; i < HC; i += 2) {
            const double2 l = *(const double2*)(LM + (half * HC + s) * RK_LM + half * HC + i);
            if (i > s) x[i] = fma(-l.x, xs, x[i]);
            x[i + 1] = fma(-l.y, xs, x[i + 1]);
          }
        }
      }
    } else {
      float x[RK_C];                               // (all on their way before the first is stored)
#pragma unroll
      for (int t = 0; t < RK_C; ++t) x[t] = t < len ? to_f(vp[(size_t)(row0 + t) * a.ld + j]) : 0.f;
#pragma unroll
      for (int t = 0; t < RK_C; ++t) put(t, x[t]);
    }
  }
}

// ---------------------------------------------------------------- walk
__device__ __forceinline__ void rk_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// The delta rule's chain: W S, U = U0 - W S, S = P S + K^T U.  What the outputs need of it, the state in front of every chunk
// and U, goes to memory.
#define RK_PP RK_NV         // row stride of the partial sums (a warp writes eight whole rows, reads four)

template <int DK>
__device__ __forceinline__ void rk_fetch(const RkArgs& a, float* buf, size_t cell, int tile, int tid) {
  using I = RkImage<true, DK>;
  const float* img = a.image + cell * I::FLOATS;
#pragma unroll
  for (int x = 4 * tid; x < I::WALK; x += 4 * RK_THREADS) rk_copy16(buf + x, img + x);
  const float* Ug = a.U + cell * ((size_t)RK_C * a.dv) + (size_t)tile * (RK_C * RK_NV);
  if (tid < RK_C * RK_NV / 4) rk_copy16(buf + I::WALK + 4 * tid, Ug + 4 * tid);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// 32 rows (at A, stride AP) times the state, over a warp's KW key rows: a lane rows rg + 8 m, columns 4 cg + x; pairs of
// key rows an operation.  The sums go to part [32][RK_PP].
template <int KW, int AP>
__device__ __forceinline__ void rk_rows_by_state(const float* A, const float* Sw, float* part, int rg, int cg) {
  constexpr int GM = KW / 4 - 1;
  unsigned long long acc[4][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[m][x] = 0ull;
  A += rg * AP;
#pragma unroll
  for (int kk = 0; kk < KW / 4; ++kk) {
    ulonglong2 sv[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) sv[x] = *(const ulonglong2*)(Sw + (4 * cg + x) * KW + 4 * (kk ^ (cg & GM)));
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const ulonglong2 av = *(const ulonglong2*)(A + 8 * m * AP + 4 * kk);
#pragma unroll
      for (int x = 0; x < 4; ++x) { acc[m][x] = fma_f2(av.x, sv[x].x, acc[m][x]); acc[m][x] = fma_f2(av.y, sv[x].y, acc[m][x]); }
    }
  }
  part += rg * RK_PP + 4 * cg;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    float o[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) { float lo, hi; unpack_f2(acc[m][x], lo, hi); o[x] = lo + hi; }
    *(float4*)(part + 8 * m * RK_PP) = make_float4(o[0], o[1], o[2], o[3]);
  }
}

// the eight warps' sums of a row and two columns, in warp order
__device__ __forceinline__ float2 rk_gather(const float* part, int row, int col) {
  float2 r = make_float2(0.f, 0.f);
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const float2 p = *(const float2*)(part + (w * RK_C + row) * RK_PP + col);
    r.x += p.x; r.y += p.y;
  }
  return r;
}

template <int DK>
__global__ void __launch_bounds__(RK_THREADS)
rk_chain_kernel(const RkArgs a) {
  extern __shared__ __align__(16) float sm[];
  using I = RkImage<true, DK>;
  constexpr int STAGE = I::WALK + RK_C * RK_NV;
  constexpr int KW = DK / 8;                       // key rows of the state a warp keeps
  constexpr int RPL = KW / 8;                      // of them a lane
  constexpr int GM = KW / 4 - 1;                   // 16-byte groups of a column, less one
  float* partW = sm + 2 * STAGE;                   // [8 warps][32][RK_PP]
  float* St = partW + 8 * RK_C * RK_PP;            // [8 warps][16 columns][KW], 16-byte groups swizzled by column / 4
  float* Us = St + RK_NV * DK;                     // [32][16]
  const int item = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * RK_NV;
  const int r0 = a.item_start[item], n = a.item_start[item + 1] - r0;
  if (n < a.min_rows || n <= 0) return;
  const int chunks = (n + RK_C - 1) / RK_C;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rg = (lane & 1) + 2 * (lane >> 3), cg = (lane >> 1) & 3;       // (each shared by lanes one or two apart: see above)
  const size_t cell0 = (size_t)rk_first_chunk(r0, item) * a.H + h;
  rk_fetch<DK>(a, sm, cell0, blockIdx.x, tid);

  // a lane's part of the state: rows warp * KW + RPL * rg + r, columns j0 + 4 cg + x
  float* slot = a.state + (size_t)a.item_slot[item] * a.slot_stride + (size_t)h * DK * a.dv;
  const int i0 = warp * KW + RPL * rg;
  float s[RPL][4];
  float* Sw = St + warp * (RK_NV * KW);            // (a warp's key rows: written and read by the warp alone)
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int r = 0; r < RPL; ++r) s[r][x] = slot[(size_t)(j0 + 4 * cg + x) * DK + i0 + r];
  const int row = tid >> 3, jc = 2 * (tid & 7);                // gathering: a thread a row and two columns

  for (int c = 0; c < chunks; ++c) {
    const float* buf = sm + (c & 1) * STAGE;
    const size_t cell = cell0 + (size_t)c * a.H;
    float* Sg = a.S + cell * ((size_t)a.dv * DK) + (size_t)j0 * DK + i0;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int i = RPL * rg, col = 4 * cg + x;
      float* at = Sw + col * KW + 4 * ((i >> 2) ^ (cg & GM)) + (i & 3);
      if (RPL == 2) *(float2*)at = make_float2(s[0][x], s[RPL - 1][x]);
      else *at = s[0][x];
      if (RPL == 2) *(float2*)(Sg + (4 * cg + x) * DK) = make_float2(s[0][x], s[RPL - 1][x]);
      else Sg[(4 * cg + x) * DK] = s[0][x];
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();          // this chunk's operands are here; the other buffer, the sums and U are free
    if (c + 1 < chunks) rk_fetch<DK>(a, sm + ((c + 1) & 1) * STAGE, cell + a.H, blockIdx.x, tid);
    rk_rows_by_state<KW, I::AP>(buf + I::W + warp * KW, Sw, partW + warp * (RK_C * RK_PP), rg, cg);
    __syncthreads();
    {
      const float2 r = rk_gather(partW, row, jc), u0 = *(const float2*)(buf + I::WALK + row * RK_NV + jc);
      const float2 u = make_float2(u0.x - r.x, u0.y - r.y);
      *(float2*)(Us + row * RK_NV + jc) = u;
      *(float2*)(a.U + cell * ((size_t)RK_C * a.dv) + (size_t)blockIdx.x * (RK_C * RK_NV) + row * RK_NV + jc) = u;
    }
    const float* Kb = buf + I::K + i0;
    const float* Pb = buf + I::P + i0;
    float k1[RPL];
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      const float p = Pb[q];
#pragma unroll
      for (int x = 0; x < 4; ++x) s[q][x] *= p;
    }
    __syncthreads();
#pragma unroll 16
    for (int t2 = 0; t2 < RK_C; ++t2) {
      if (RPL == 2) { const float2 f = *(const float2*)(Kb + t2 * DK); k1[0] = f.x; k1[RPL - 1] = f.y; }
      else k1[0] = Kb[t2 * DK];
      const float4 u = *(const float4*)(Us + t2 * RK_NV + 4 * cg);
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        s[q][0] = fmaf(k1[q], u.x, s[q][0]); s[q][1] = fmaf(k1[q], u.y, s[q][1]);
        s[q][2] = fmaf(k1[q], u.z, s[q][2]); s[q][3] = fmaf(k1[q], u.w, s[q][3]);
      }
    }
  }
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int r = 0; r < RPL; ++r) slot[(size_t)(j0 + 4 * cg + x) * DK + i0 + r] = s[r][x];
}

// ---------------------------------------------------------------- walk, outputs and all
// Short portions wait for launches more than for work: states and outputs in one walk over the chunks, a launch less.
// Two groups of eight warps.  The first walks the state: W S, U = U0 - W S, S = P S + K^T U; the second makes the
// outputs, Q S + M U, from the state in front of the chunk as it lies in shared memory and the first group's U: what the
// outputs cost runs beside the chain and not in it, and sixteen warps hide each other's waits.
#define RK_WALK_THREADS 512
__device__ __forceinline__ void rk_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void rk_bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

template <bool DELTA, int DK>
__device__ __forceinline__ void rk_fetch_all(const RkArgs& a, float* buf, size_t cell, int tile, int tid) {
  using I = RkImage<DELTA, DK>;
  const float* img = a.image + cell * I::FLOATS;
#pragma unroll
  for (int x = 4 * tid; x < I::FLOATS; x += 4 * RK_WALK_THREADS) rk_copy16(buf + x, img + x);
  const float* Ug = a.U + cell * ((size_t)RK_C * a.dv) + (size_t)tile * (RK_C * RK_NV);
  if (tid < RK_C * RK_NV / 4) rk_copy16(buf + I::FLOATS + 4 * tid, Ug + 4 * tid);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <bool DELTA, int DK>
__global__ void __launch_bounds__(RK_WALK_THREADS)
rk_walk_kernel(const RkArgs a) {
  extern __shared__ __align__(16) float sm[];
  using I = RkImage<DELTA, DK>;
  constexpr int STAGE = I::FLOATS + RK_C * RK_NV;
  constexpr int KW = DK / 8;                       // key rows of the state a warp keeps
  constexpr int RPL = KW / 8;                      // of them a lane
  constexpr int GM = KW / 4 - 1;                   // 16-byte groups of a column, less one
  float* partQ = sm + 2 * STAGE;                   // [8 warps][32][RK_PP]
  float* St = partQ + 8 * RK_C * RK_PP;            // two of [8 warps][16 columns][KW], 16-byte groups swizzled by column / 4
  float* partW = St + 2 * RK_NV * DK;              // (delta) as partQ
  float* Us = partW + 8 * RK_C * RK_PP;            // (delta) [32][16]
  const int item = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * RK_NV;
  const int r0 = a.item_start[item], n = a.item_start[item + 1] - r0;
  if (n < a.min_rows || n <= 0) return;
  const int chunks = (n + RK_C - 1) / RK_C;
  const int tid = threadIdx.x, gtid = tid & 255, warp = (tid >> 5) & 7, lane = tid & 31;
  const bool walker = tid < 256;
  const int rg = (lane & 1) + 2 * (lane >> 3), cg = (lane >> 1) & 3;
  const size_t cell0 = (size_t)rk_first_chunk(r0, item) * a.H + h;
  rk_fetch_all<DELTA, DK>(a, sm, cell0, blockIdx.x, tid);

  // a walker's part of the state: rows warp * KW + RPL * rg + r, columns j0 + 4 cg + x
  float* slot = a.state + (size_t)a.item_slot[item] * a.slot_stride + (size_t)h * DK * a.dv;
  const int i0 = warp * KW + RPL * rg;
  float s[RPL][4];
  auto put_state = [&](int c) {
    float* Sw = St + (c & 1) * (RK_NV * DK) + warp * (RK_NV * KW);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int i = RPL * rg, col = 4 * cg + x;
      float* at = Sw + col * KW + 4 * ((i >> 2) ^ (cg & GM)) + (i & 3);
      if (RPL == 2) *(float2*)at = make_float2(s[0][x], s[RPL - 1][x]);
      else *at = s[0][x];
    }
  };
  if (walker) {
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int r = 0; r < RPL; ++r) s[r][x] = slot[(size_t)(j0 + 4 * cg + x) * DK + i0 + r];
    put_state(0);
  }
  const int row = gtid >> 3, jc = 2 * (gtid & 7);                // gathering: a thread a row and two columns

  for (int c = 0; c < chunks; ++c) {
    const float* buf = sm + (c & 1) * STAGE;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();          // this chunk's operands and state are here; the other buffers, the sums and U are free
    if (c + 1 < chunks) rk_fetch_all<DELTA, DK>(a, sm + ((c + 1) & 1) * STAGE, cell0 + (size_t)(c + 1) * a.H, blockIdx.x, tid);
    const float* U = DELTA ? Us : buf + I::FLOATS;
    const float* Sw = St + (c & 1) * (RK_NV * DK) + warp * (RK_NV * KW);
    if (walker) {
      if (DELTA) {
        rk_rows_by_state<KW, I::AP>(buf + I::W + warp * KW, Sw, partW + warp * (RK_C * RK_PP), rg, cg);
        rk_bar_sync(1, 256);
        const float2 r = rk_gather(partW, row, jc), u0 = *(const float2*)(buf + I::FLOATS + row * RK_NV + jc);
        *(float2*)(Us + row * RK_NV + jc) = make_float2(u0.x - r.x, u0.y - r.y);
        rk_bar_sync(1, 256);
        rk_bar_arrive(2, 512);                     // U is there for the other group
      }
      const float* Kb = buf + I::K + i0;
      const float* Pb = buf + I::P + i0;
      float k1[RPL];
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        const float p = Pb[q];
#pragma unroll
        for (int x = 0; x < 4; ++x) s[q][x] *= p;
      }
#pragma unroll 16
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
      put_state(c + 1);
    } else {
      rk_rows_by_state<KW, I::AP>(buf + I::Q + warp * KW, Sw, partQ + warp * (RK_C * RK_PP), rg, cg);
      rk_bar_sync(3, 256);
      float2 r = rk_gather(partQ, row, jc);
      if (DELTA) rk_bar_sync(2, 512);
      const float* Mt = buf + I::M + row * RK_LP;
#pragma unroll 2
      for (int x = 0; x <= (row | 3); x += 4) {    // (a warp's four rows end together)
        const float4 m = *(const float4*)(Mt + x);
        const float mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 u = *(const float2*)(U + (x + e) * RK_NV + jc);
          if (x + e <= row) { r.x = fmaf(mm[e], u.x, r.x); r.y = fmaf(mm[e], u.y, r.y); }
        }
      }
      if (c * RK_C + row < n) *(float2*)(a.out + (size_t)(r0 + c * RK_C + row) * ((size_t)a.H * a.dv) + (size_t)h * a.dv + j0 + jc) = r;
    }
  }
  if (walker) {
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int r = 0; r < RPL; ++r) slot[(size_t)(j0 + 4 * cg + x) * DK + i0 + r] = s[r][x];
  }
}

// Without the delta rule the states are S' = P S + K^T V, element by element: the walk's multiply-adds in the walk's order and so with its
// bits, without the outputs.  A block of two warps a head, RK_SR key rows and 16 value columns, a thread four key rows of two columns, so
// that a portion of 8 heads of 128 gives every SM quarter a warp; RK_AHEAD chunks' operands on their way under the sums.  (Blocks of all
// key rows, four columns a thread, reach 64 SMs there: prep, states and outputs of 2,048 tokens 134 us for 90.  K^T V summed in prep, chunks
// side by side, takes 85, but rounds in another order and makes a state's error larger, 3.09e-8 -> 3.4e-8 with decay and bonus.)
#define RK_AHEAD 4
#define RK_SR 32           // key rows a block
#define RK_STATES_THREADS 64
template <int DK>
__global__ void __launch_bounds__(RK_STATES_THREADS)
rk_states_kernel(const RkArgs a) {
  using I = RkImage<false, DK>;
  constexpr int P = RK_C * RK_SR, V = P + RK_SR, STAGE = V + RK_C * RK_NV;
  __shared__ __align__(16) float sm[(RK_AHEAD + 1) * STAGE];           // [32][RK_SR] of K, P, [32][16] of V
  const int item = blockIdx.z, h = blockIdx.y, tile = blockIdx.x / (DK / RK_SR), i0 = RK_SR * (blockIdx.x % (DK / RK_SR));
  const int r0 = a.item_start[item], n = a.item_start[item + 1] - r0;
  if (n < a.min_rows || n <= 0) return;
  const int chunks = (n + RK_C - 1) / RK_C;
  const int tid = threadIdx.x, lane = tid & 31;
  // a thread's key rows i .. i + 3, columns j and j + 1 (each shared by lanes one or two apart)
  const int i = 4 * ((lane & 1) + 2 * (lane >> 3)), j = 8 * (tid >> 5) + 2 * ((lane >> 1) & 3);
  const size_t cell0 = (size_t)rk_first_chunk(r0, item) * a.H + h;
  auto fetch = [&](int c, int at) {
    if (c < chunks) {
      const size_t cell = cell0 + (size_t)c * a.H;
      float* to = sm + at * STAGE;
      const float* img = a.image + cell * I::FLOATS + i0;
#pragma unroll
      for (int x = tid; x < P / 4; x += RK_STATES_THREADS) rk_copy16(to + 4 * x, img + I::K + (x / (RK_SR / 4)) * DK + 4 * (x % (RK_SR / 4)));
      if (tid < RK_SR / 4) rk_copy16(to + P + 4 * tid, img + I::P + 4 * tid);
      const float* Vg = a.U + cell * ((size_t)RK_C * a.dv) + (size_t)tile * (RK_C * RK_NV);
#pragma unroll
      for (int x = tid; x < RK_C * RK_NV / 4; x += RK_STATES_THREADS) rk_copy16(to + V + 4 * x, Vg + 4 * x);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < RK_AHEAD; ++c) fetch(c, c);

  const size_t at0 = (size_t)(tile * RK_NV + j) * DK + i0 + i;
  float* slot = a.state + (size_t)a.item_slot[item] * a.slot_stride + (size_t)h * DK * a.dv + at0;
  float* Sg = a.S + cell0 * ((size_t)a.dv * DK) + at0;
  const size_t s_step = (size_t)a.H * a.dv * DK;
  float s[2][4];
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int r = 0; r < 4; ++r) s[x][r] = slot[x * DK + r];
  int now = 0, free = RK_AHEAD;
  for (int c = 0; c < chunks; ++c, Sg += s_step) {
#pragma unroll
    for (int x = 0; x < 2; ++x) *(float4*)(Sg + x * DK) = make_float4(s[x][0], s[x][1], s[x][2], s[x][3]);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(RK_AHEAD - 1) : "memory");
    __syncthreads();          // this chunk's operands are here, everyone is done with the chunk before
    fetch(c + RK_AHEAD, free);
    const float* K = sm + now * STAGE;
    const float4 p = *(const float4*)(K + P + i);
#pragma unroll
    for (int x = 0; x < 2; ++x) { s[x][0] *= p.x; s[x][1] *= p.y; s[x][2] *= p.z; s[x][3] *= p.w; }
#pragma unroll 16
    for (int t = 0; t < RK_C; ++t) {
      const float4 k = *(const float4*)(K + t * RK_SR + i);
      const float2 v = *(const float2*)(K + V + t * RK_NV + j);
      s[0][0] = fmaf(k.x, v.x, s[0][0]); s[0][1] = fmaf(k.y, v.x, s[0][1]); s[0][2] = fmaf(k.z, v.x, s[0][2]); s[0][3] = fmaf(k.w, v.x, s[0][3]);
      s[1][0] = fmaf(k.x, v.y, s[1][0]); s[1][1] = fmaf(k.y, v.y, s[1][1]); s[1][2] = fmaf(k.z, v.y, s[1][2]); s[1][3] = fmaf(k.w, v.y, s[1][3]);
    }
    free = now;
    now = now == RK_AHEAD ? 0 : now + 1;
  }
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int r = 0; r < 4; ++r) slot[x * DK + r] = s[x][r];
}

// ---------------------------------------------------------------- outputs
// O = Q S + M U of every chunk, side by side: a block a chunk, head and 64 columns; a warp 16 rows x 32 columns, a lane rows
// rg + 4 m and four neighbouring columns.  The 32 floats of a key row pair a lane takes from shared memory feed 32 multiply-adds: bound by those.
// Sums as the eight warps of one chain would make them: DK / 8 key rows at a time, pairs of rows an operation, then the parts in order.
#define RK_OUT_THREADS 128
#define RK_OUT_COLS 64
template <bool DELTA, int DK>
__global__ void __launch_bounds__(RK_OUT_THREADS)
rk_out_kernel(const RkArgs a) {
  extern __shared__ __align__(16) float sm[];
  using I = RkImage<DELTA, DK>;
  constexpr int KW = DK / 8, SP = DK + 4, UP = RK_OUT_COLS + 4;
  float* Q = sm;                                   // [32][AP], and M [32][RK_LP] behind it
  float* M = Q + RK_C * I::AP;
  float* S = Q + I::OUT;                 // [64 columns][SP]: column j of 32 at row 8 (j % 4) + j / 4, so that a lane's four are 8 rows apart
  float* U = S + RK_OUT_COLS * SP;                 // [32][UP]
  const int item = rk_item_of(a.item_start, a.n_items, blockIdx.x), h = blockIdx.y, j0 = blockIdx.z * RK_OUT_COLS;
  const int r0 = a.item_start[item], n = a.item_start[item + 1] - r0, c = blockIdx.x - rk_first_chunk(r0, item);
  if (n < a.min_rows || c < 0 || c * RK_C >= n) return;           // (c < 0: rows in front of the first item)
  const int cols = min(RK_OUT_COLS, a.dv - j0);    // (a multiple of 16)
  const size_t cell = (size_t)blockIdx.x * a.H + h;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* img = a.image + cell * I::FLOATS + I::Q;
  const float* Sg = a.S + cell * ((size_t)a.dv * DK) + (size_t)j0 * DK;
  const float* Ug = a.U + cell * ((size_t)RK_C * a.dv) + (size_t)(j0 / RK_NV) * (RK_C * RK_NV);
  // four groups of copies, a quarter of the key rows each: the products start behind the first
  constexpr int KQ = DK / 4;
#pragma unroll
  for (int part = 0; part < 4; ++part) {
    if (part == 0) for (int x = 4 * tid; x < I::OUT; x += 4 * RK_OUT_THREADS) rk_copy16(Q + x, img + x);
    for (int x = 4 * tid; x < cols * KQ; x += 4 * RK_OUT_THREADS) {
      const int j = x / KQ, k = part * KQ + x % KQ;
      rk_copy16(S + ((j & ~31) + 8 * (j & 3) + ((j & 31) >> 2)) * SP + k, Sg + (size_t)j * DK + k);
    }
    if (part == 3)
      for (int x = 4 * tid; x < cols * RK_C; x += 4 * RK_OUT_THREADS) {
        const int tile = x / (RK_C * RK_NV), y = x % (RK_C * RK_NV);
        rk_copy16(U + (y / RK_NV) * UP + tile * RK_NV + y % RK_NV, Ug + x);
      }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  const int rg = (lane & 1) + 2 * (lane >> 4), cg = (lane >> 1) & 7, row0 = 16 * (warp & 1) + rg, col0 = 32 * (warp >> 1);
  float r[4][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int x = 0; x < 4; ++x) r[m][x] = 0.f;
  const float* Qr = Q + row0 * I::AP;
  const float* Sc = S + (col0 + cg) * SP;
#pragma unroll 1
  for (int w = 0; w < 8; ++w) {
    if (w == 0) asm volatile("cp.async.wait_group 3;\n" ::: "memory");
    else if (w == 2) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
    else if (w == 4) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    else if (w == 6) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (!(w & 1)) __syncthreads();
    unsigned long long acc[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[m][x] = 0ull;
#pragma unroll
    for (int kk = 0; kk < KW / 4; ++kk) {
      const int k = w * KW + 4 * kk;
      ulonglong2 sv[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) sv[x] = *(const ulonglong2*)(Sc + 8 * x * SP + k);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const ulonglong2 qv = *(const ulonglong2*)(Qr + 4 * m * I::AP + k);
#pragma unroll
        for (int x = 0; x < 4; ++x) { acc[m][x] = fma_f2(qv.x, sv[x].x, acc[m][x]); acc[m][x] = fma_f2(qv.y, sv[x].y, acc[m][x]); }
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int x = 0; x < 4; ++x) { float lo, hi; unpack_f2(acc[m][x], lo, hi); r[m][x] += lo + hi; }
  }
  const float* Uc = U + col0 + 4 * cg;
#pragma unroll 1
  for (int t = 0; t < 16 * (warp & 1) + 16; t += 4) {
    float4 mv[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) mv[m] = *(const float4*)(M + (row0 + 4 * m) * RK_LP + t);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 u = *(const float4*)(Uc + (t + e) * UP);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float f = e == 0 ? mv[m].x : e == 1 ? mv[m].y : e == 2 ? mv[m].z : mv[m].w;
        if (t + e <= row0 + 4 * m) {               // (a later token's values stay out, whatever they are)
          r[m][0] = fmaf(f, u.x, r[m][0]); r[m][1] = fmaf(f, u.y, r[m][1]);
          r[m][2] = fmaf(f, u.z, r[m][2]); r[m][3] = fmaf(f, u.w, r[m][3]);
        }
      }
    }
  }
  if (col0 + 4 * cg >= cols) return;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int t = c * RK_C + row0 + 4 * m;
    if (t < n) *(float4*)(a.out + (size_t)(r0 + t) * ((size_t)a.H * a.dv) + (size_t)h * a.dv + j0 + col0 + 4 * cg) = make_float4(r[m][0], r[m][1], r[m][2], r[m][3]);
  }
}

// ---------------------------------------------------------------- launches
template <int MODE, int DK, typename TA>
static int rk_launch(const RkArgs& a, cudaStream_t stream) {
  constexpr bool DELTA = MODE <= RK_DELTA_CHANNEL;
  using I = RkImage<DELTA, DK>;
  const size_t sm_prep = (size_t)(4 * RK_C * DK + RK_C) * sizeof(float) + (RK_C * RK_LM + RK_C) * sizeof(double);
  // (more than half of an SM's shared memory: two blocks on one SM and none on another made one portion among single tokens, whose blocks
  // have nothing to do, a third longer)
  size_t sm_chain = (size_t)(2 * (RkImage<true, DK>::WALK + RK_C * RK_NV) + 8 * RK_C * RK_PP + RK_NV * DK + RK_C * RK_NV) * sizeof(float);
  if (sm_chain < 116 * 1024) sm_chain = 116 * 1024;
  const size_t sm_out = (size_t)(I::OUT + RK_OUT_COLS * (DK + 4) + RK_C * (RK_OUT_COLS + 4)) * sizeof(float);
  const size_t sm_walk = (size_t)(2 * (I::FLOATS + RK_C * RK_NV) + 8 * RK_C * RK_PP + 2 * RK_NV * DK + (DELTA ? 8 * RK_C * RK_PP + RK_C * RK_NV : 0)) * sizeof(float);
  const int tiles = (a.dv + RK_OUT_COLS - 1) / RK_OUT_COLS;
  if (tiles > 65535) return FELLM_ERR_SIZE;
  cudaError_t e = cudaFuncSetAttribute(rk_prep_kernel<MODE, DK, TA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_prep);
  if (e == cudaSuccess && !a.S) e = cudaFuncSetAttribute(rk_walk_kernel<DELTA, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_walk);
  if (e == cudaSuccess && a.S && DELTA) e = cudaFuncSetAttribute(rk_chain_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_chain);
  if (e == cudaSuccess && a.S) e = cudaFuncSetAttribute(rk_out_kernel<DELTA, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_out);
  if (e != cudaSuccess) return (int)e;
  // (ordinary launches: as programmatic dependents the next kernel's blocks take the SMs' shared memory while they wait; 2,048 tokens of
  // the delta rule 214 -> 291 us)
  rk_prep_kernel<MODE, DK, TA><<<dim3(a.cells, a.H), RK_THREADS, sm_prep, stream>>>(a);
  if (!a.S) {
    rk_walk_kernel<DELTA, DK><<<dim3(a.dv / RK_NV, a.H, a.n_items), RK_WALK_THREADS, sm_walk, stream>>>(a);
    return launch_status();
  }
  if (DELTA) rk_chain_kernel<DK><<<dim3(a.dv / RK_NV, a.H, a.n_items), RK_THREADS, sm_chain, stream>>>(a);
  else rk_states_kernel<DK><<<dim3(a.dv / RK_NV * (DK / RK_SR), a.H, a.n_items), RK_STATES_THREADS, 0, stream>>>(a);
  rk_out_kernel<DELTA, DK><<<dim3(a.cells, a.H, tiles), RK_OUT_THREADS, sm_out, stream>>>(a);
  return launch_status();
}

static long long rk_image_floats(int mode, int dk) {
  if (dk == 128) return mode <= RK_DELTA_CHANNEL ? RkImage<true, 128>::FLOATS : RkImage<false, 128>::FLOATS;
  return mode <= RK_DELTA_CHANNEL ? RkImage<true, 64>::FLOATS : RkImage<false, 64>::FLOATS;
}

// Floats of scratch for a step of T rows.
FELLM_API long long fellm_recurrent_chunk_scratch(int mode, int T, int n_items, int H, int dk, int dv, int apart) {
  return (T / RK_C + (long long)n_items) * H * (rk_image_floats(mode, dk) + (long long)(RK_C + (apart ? dk : 0)) * dv);
}

// mode 0 / 1: the delta rule with a decay per head / channel (q, k [T, G dk] and v [T, H dv] in rows of ld elements, as
// fellm_delta_scan takes them); 2: decay and bonus (r, k, v [T, H dk]); 3: gated write (q raw, f raw, v).  Items of fewer
// than min_rows rows are left alone.  apart: the outputs beside one another behind the states (scratch for that), else in one walk with them.  16-byte rows: see the checks.
FELLM_API int fellm_recurrent_chunk(int mode, const void* q, const void* k, const void* v, int is_bf16, int ld, int v_off,
                                    const float* small, int lds, int b_off, int a_off, const float* A_log, const float* dt_bias,
                                    const float* gch, const float* bonus, const float* lower, const float* fbias, float* state,
                                    long long slot_stride, const int* item_start, const int* item_slot, float* out, float* scratch,
                                    int T, int n_items, int min_rows, int H, int G, int dk, int dv, int apart, cudaStream_t stream) {
  if (n_items <= 0 || T <= 0) return 0;
  if ((dk != 64 && dk != 128) || dv < RK_NV || dv % RK_NV || H < 1 || G < 1 || H % G || min_rows < 1 || mode < 0 || mode > 3 ||
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
  a.H = H; a.G = G; a.dv = dv; a.min_rows = min_rows; a.n_items = n_items; a.cells = T / RK_C + n_items;
  const size_t cells = (size_t)(T / RK_C + n_items) * H;
  a.image = scratch; a.U = scratch + cells * (size_t)rk_image_floats(mode, dk); a.S = apart ? a.U + cells * ((size_t)RK_C * dv) : nullptr;
#define RK_GO(MODE_, TA_) (dk == 128 ? rk_launch<MODE_, 128, TA_>(a, stream) : rk_launch<MODE_, 64, TA_>(a, stream))
  if (mode == 0) return is_bf16 ? RK_GO(0, bf16) : RK_GO(0, float);
  if (mode == 1) return is_bf16 ? RK_GO(1, bf16) : RK_GO(1, float);
  if (mode == 2) return is_bf16 ? RK_GO(2, bf16) : RK_GO(2, float);
  return RK_GO(3, float);
#undef RK_GO
}
