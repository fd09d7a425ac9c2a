// Causal GQA attention over the paged float32 cache, heads of 64, 1, 2 or 4 of them a kv head: the 32-bit engine's attention
// of the LFM2 shapes, float32 arithmetic on CUDA cores.  What paged_attention_simt_kernel (attention_simt.cu) computes; there a
// block is a (row, head), so every row and head reads its keys and values again, a lane a key (104 us for 201 rows of 16
// heads behind 250 tokens each; 39 here).
//
// Here a block of four warps takes a kv head and RB neighbouring rows: a tile of 32 keys is read once for its RB x R queries,
// 8 lanes a key and 32 bytes a lane.  The partial dot products of a lane's eight keys go through the eight lanes by a
// transposing butterfly (lane j ends with the whole score of key j), the softmax runs on a key a lane, the probabilities
// come back by shuffles.  Warp w takes tiles w, w + 4, .. of a row's keys, counted from the first position the row sees, and
// the warps' parts are added in their order: the order of every sum depends on the row's position alone, not on the cut of
// the prompt, on RB, on the batch or on the pages.  Rows of several requests in a block are taken request by request.
// Bound by: the instructions, 16 multiply-adds for each loaded element of a key and its value at eight queries.
#include "common.cuh"

#define AF_WARPS 4
#define AF_HD 64

struct AfArgs {
  const float* q; const float* pool; const int* block_table; const int* positions; const int* row_slot; float* out;
  int max_pages, T, H, G, page_tokens, layer, layers_in_group, window, ldq;
  float scale;
};

__device__ __forceinline__ void af_load8(const float* p, float* f) {
  *(float4*)f = *(const float4*)p;
  *(float4*)(f + 4) = *(const float4*)(p + 4);
}

template <int R, int RB>
__global__ void __launch_bounds__(AF_WARPS * 32)
attention_f32_kernel(const AfArgs a) {
  constexpr int Q = R * RB;                        // queries of the block: row r, head x at r * R + x
  __shared__ __align__(16) float part[AF_WARPS][Q][AF_HD + 4];
  const int g = blockIdx.y, first = blockIdx.x * RB, n_rows = min(RB, a.T - first);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 3, sub = lane & 7;
  const size_t record = (size_t)a.G * a.page_tokens * 2 * AF_HD;

  for (int run = 0; run < n_rows;) {
    const int slot = a.row_slot[first + run];
    int end = run + 1;
    while (end < n_rows && a.row_slot[first + end] == slot) ++end;
    const int* bt = a.block_table + (size_t)slot * a.max_pages;
    int pos[RB], last = -1;
    float q[Q][8], acc[Q][8], m[Q], l[Q];
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const bool in = r >= run && r < end;
      pos[r] = in ? a.positions[first + r] : -1;
      last = max(last, pos[r]);
#pragma unroll
      for (int x = 0; x < R; ++x) {
        const int i = r * R + x;
#pragma unroll
        for (int e = 0; e < 8; ++e) { q[i][e] = 0.f; acc[i][e] = 0.f; }
        if (in) af_load8(a.q + (size_t)(first + r) * a.ldq + (size_t)(g * R + x) * AF_HD + 8 * sub, q[i]);
        m[i] = -INFINITY; l[i] = 0.f;
      }
    }
    // (RB > 1 goes without a window: all rows' tiles are counted from position 0)
    const int k_begin = (a.window > 0 && last - a.window + 1 > 0) ? last - a.window + 1 : 0;
    for (int k0 = k_begin + 32 * warp; k0 <= last; k0 += 32 * AF_WARPS) {
      const float* rows[8];                        // this lane's 32 bytes of its eight keys: k0 + 4 i + grp
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int kj = min(k0 + 4 * i + grp, last);                  // (beyond: the last key once more, masked below)
        const int page = max(bt[kj / a.page_tokens], 0);             // an unmapped entry (-1) must never become an address
        rows[i] = a.pool + ((size_t)page * a.layers_in_group + a.layer) * record + ((size_t)g * a.page_tokens + kj % a.page_tokens) * AF_HD + 8 * sub;
      }
      // lane `sub` ends with the whole scores of key k0 + 4 sub + grp: pairs (i, i + 4), then (i, i + 2), then (0, 1)
      float p[Q];
      {
        float v2[2][Q];
#pragma unroll
        for (int i2 = 0; i2 < 2; ++i2) {
          float v1[2][Q];
#pragma unroll
          for (int i1 = 0; i1 < 2; ++i1) {
            const int i = i2 + 2 * i1;
            float k_lo[8], k_hi[8];
            af_load8(rows[i], k_lo); af_load8(rows[i + 4], k_hi);
#pragma unroll
            for (int t = 0; t < Q; ++t) {
              float x = 0.f, y = 0.f;
#pragma unroll
              for (int e = 0; e < 8; ++e) { x = fmaf(q[t][e], k_lo[e], x); y = fmaf(q[t][e], k_hi[e], y); }
              const bool up = sub & 4;
              v1[i1][t] = (up ? y : x) + __shfl_xor_sync(0xffffffffu, up ? x : y, 4);
            }
          }
#pragma unroll
          for (int t = 0; t < Q; ++t) {
            const bool up = sub & 2;
            v2[i2][t] = (up ? v1[1][t] : v1[0][t]) + __shfl_xor_sync(0xffffffffu, up ? v1[0][t] : v1[1][t], 2);
          }
        }
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const bool up = sub & 1;
          p[t] = (up ? v2[1][t] : v2[0][t]) + __shfl_xor_sync(0xffffffffu, up ? v2[0][t] : v2[1][t], 1);
        }
      }
      const int kj = k0 + 4 * sub + grp;
#pragma unroll
      for (int t = 0; t < Q; ++t) {
        const int at = pos[t / R];
        if (k0 > at) { p[t] = 0.f; continue; }     // (the same for the whole warp) the row sees none of these keys
        const bool seen = kj <= at;
        const float x = seen ? p[t] * a.scale : -INFINITY;
        const float mn = fmaxf(m[t], warp_max(x)), corr = expf(m[t] - mn);
        p[t] = seen ? expf(x - mn) : 0.f;
        m[t] = mn;
        l[t] = fmaf(l[t], corr, p[t]);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[t][e] *= corr;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float v[8];
        af_load8(rows[i] + (size_t)a.G * a.page_tokens * AF_HD, v);
        const int key = k0 + 4 * i + grp;
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const float pr = __shfl_sync(0xffffffffu, p[t], i, 8);
          if (key <= pos[t / R]) {                 // (a masked key's value is not touched: 0 * NaN)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[t][e] = fmaf(pr, v[e], acc[t][e]);
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < Q; ++t) {
      l[t] = warp_sum(l[t]);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        acc[t][e] += __shfl_xor_sync(0xffffffffu, acc[t][e], 8);
        acc[t][e] += __shfl_xor_sync(0xffffffffu, acc[t][e], 16);
      }
      if (grp == 0) {
        *(float4*)&part[warp][t][8 * sub] = make_float4(acc[t][0], acc[t][1], acc[t][2], acc[t][3]);
        *(float4*)&part[warp][t][8 * sub + 4] = make_float4(acc[t][4], acc[t][5], acc[t][6], acc[t][7]);
      }
      if (lane == 0) { part[warp][t][AF_HD] = m[t]; part[warp][t][AF_HD + 1] = l[t]; }
    }
    __syncthreads();
    for (int x = run * R * AF_HD + threadIdx.x; x < end * R * AF_HD; x += AF_WARPS * 32) {
      const int t = x / AF_HD, e = x - t * AF_HD;
      float M = -INFINITY, o = 0.f, L = 0.f;
#pragma unroll
      for (int w = 0; w < AF_WARPS; ++w) M = fmaxf(M, part[w][t][AF_HD]);
#pragma unroll
      for (int w = 0; w < AF_WARPS; ++w) {
        // a warp without a key (m = -inf, l = 0) counts nothing; one whose scores were no numbers keeps them
        const float mw = part[w][t][AF_HD], lw = part[w][t][AF_HD + 1];
        const float f = (mw == -INFINITY && lw == 0.f) ? 0.f : expf(mw - M);
        o = fmaf(part[w][t][e], f, o); L = fmaf(lw, f, L);
      }
      a.out[((size_t)(first + t / R) * a.H + g * R + t % R) * AF_HD + e] = o * (1.0f / L);
    }
    __syncthreads();
    run = end;
  }
}

// q [T, ldq] float32 (heads at column 0, normed and rotated), out [T, H * 64]; pool [pages, layers_in_group, record], a record
// the keys [G][page_tokens][64] and then the values; window 0: none.
FELLM_API int fellm_attention_f32(const float* q, int ldq, const float* pool, const int* block_table, int max_pages, const int* positions,
                                  const int* row_slot, float* out, int T, int H, int G, int hd, int page_tokens, int layer,
                                  int layers_in_group, float scale, int window, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!q || !pool || !block_table || !positions || !row_slot || !out) return FELLM_ERR_ARG;
  if (hd != AF_HD || G < 1 || G > 65535 || H % G || page_tokens < 1 || (ldq & 3) || (((uintptr_t)q | (uintptr_t)pool) & 15)) return FELLM_ERR_SIZE;
  const AfArgs a = {q, pool, block_table, positions, row_slot, out, max_pages, T, H, G, page_tokens, layer, layers_in_group, window, ldq, scale};
  // Neighbouring rows share a tile's reading where there are rows enough and no window: eight queries a block where their blocks go three
  // times (two heads a kv head) or one and a half times (one, four) into the SMs, else four: more blocks, each with half the registers.
  // us, eight / four queries a block, 8 kv heads; two heads: 201 rows behind 300 40.7 / 36.0, 64 behind 500 29.5 / 18.1, 32 behind 100 12.9 /
  // 7.6, 256 behind 500 64.6 / 71.6, 1,024 194 / 212; one head: 200 rows 35.1 / 17.3, 256 behind 500 34.7 / 38.2; four heads: 32 behind 100
  // 13.5 / 8.9, 64 behind 500 29.9 / 36.5.
  const bool many = window <= 0 && T >= 32;
  const int R = H / G;
  const bool eight = R <= 4 && 2ll * ceil_div(T, 8 / (R < 1 ? 1 : R)) * G >= (R == 2 ? 6ll : 3ll) * fellm_sm_count();
#define AF_GO(R_, RB_) attention_f32_kernel<R_, RB_><<<dim3(ceil_div(T, RB_), G), AF_WARPS * 32, 0, stream>>>(a)
  switch (R) {
    case 1: if (many && eight) AF_GO(1, 8); else if (many) AF_GO(1, 4); else AF_GO(1, 1); break;
    case 2: if (many && eight) AF_GO(2, 4); else if (many) AF_GO(2, 2); else AF_GO(2, 1); break;
    case 4: if (many && eight) AF_GO(4, 2); else AF_GO(4, 1); break;
    default: return FELLM_ERR_SIZE;
  }
#undef AF_GO
  return launch_status();
}
