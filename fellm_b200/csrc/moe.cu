// Routed experts (a mixture of small gated feed-forwards): everything between the router's logits and the sum
// that goes into the residual stream, without a word to the host.
//
//   moe_route     softmax over the experts in float32, the `top` largest per token (ties: the lower expert), their
//                 scores as they are (or renormalised to sum 1)
//   moe_plan      (three kernels) the (token, choice) pairs sorted by expert: a count per tile of pairs and expert,
//                 an exclusive scan in the order (expert, tile), each pair's place; and the table of row tiles
//                 (expert, first row, rows) that the grouped products walk
//   moe_gemm      grouped product over the table: C[r, :] = A[row(r), :] W[e]^T, with the input rows gathered by
//                 token (first product, SiLU(gate) * up in the epilogue) or taken in sorted order (second product)
//   moe_combine   x[t, :] += sum_c score[t, c] * y[place(t, c), :], c in order (an identity expert: score[t, c] * h[t, :])
//
// A row's arithmetic depends on the row alone: a pair's place among its expert's rows moves it inside a tile, never
// into another sum; every sum over K runs in the order of K; the sum over a token's experts runs in the order of the
// choices.  So a token's result does not depend on the batch, and no atomics touch data.
#include "common.cuh"

#define MOE_MAX_TOP 16
#define PLAN_TILE 1024
#define MOE_FEW_TOKENS 128      // below: launched as dependents of the kernel in front

__device__ __forceinline__ void unpack8(const uint4& raw, float* f) {
  const __nv_bfloat162* h = (const __nv_bfloat162*)&raw;
#pragma unroll
  for (int e = 0; e < 4; ++e) { float2 v = __bfloat1622float2(h[e]); f[2 * e] = v.x; f[2 * e + 1] = v.y; }
}

// ---------------------------------------------------------------- routing
// One warp: softmax over z[0..E) in float32, the `top` largest (ties: the lower expert) into idx / w.
__device__ __forceinline__ void route_warp(const float* z, int E, int top, int renorm, int* idx, float* w, int lane) {
  float m = -INFINITY;
  for (int e = lane; e < E; e += 32) m = fmaxf(m, z[e]);
  m = warp_max(m);
  float sum = 0.f;
  for (int e = lane; e < E; e += 32) sum += expf(z[e] - m);
  sum = warp_sum(sum);
  int taken[MOE_MAX_TOP];
  float tw[MOE_MAX_TOP];
  float chosen = 0.f;
#pragma unroll
  for (int c = 0; c < MOE_MAX_TOP; ++c) {
    if (c >= top) break;
    float best = -INFINITY; int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      bool free_ = true;
#pragma unroll
      for (int p = 0; p < MOE_MAX_TOP; ++p) if (p < c && taken[p] == e) free_ = false;
      const float v = z[e];
      if (free_ && (v > best || (v == best && e < bi))) { best = v; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    taken[c] = bi;
    tw[c] = expf(best - m) / sum;
    chosen += tw[c];
  }
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < MOE_MAX_TOP; ++c) {
      if (c >= top) break;
      idx[c] = taken[c];
      w[c] = renorm ? tw[c] / chosen : tw[c];
    }
  }
}

// One warp, the choice form: scores s_e = sigmoid(z_e) or, soft, softmax(z)_e over all E; the choice looks at s_e + corr_e
// (corr may be null, and either may be negative) and only inside the `keep` groups (of n_groups equal groups of neighbouring experts) whose `gtop` largest choice scores sum
// highest (ties: the lower group); the `top` largest choice scores among those (ties: the lower expert); weights = the
// chosen experts' plain scores, over their sum + 1e-20 when renorm.  work: shared memory of E + n_groups floats.
__device__ __forceinline__ void route_choice_warp(int soft, const float* z, const float* corr, int E, int top, int renorm,
                                                   int n_groups, int keep, int gtop, float* work, int* idx, float* w, int lane) {
  float* choice = work;                 // [E]
  float* gscore = work + E;             // [n_groups]; -inf once a group is taken, then +inf marks the kept ones
  float zmax = 0.f, zsum = 1.f;
  if (soft) {
    zmax = -INFINITY; zsum = 0.f;
    for (int e = lane; e < E; e += 32) zmax = fmaxf(zmax, z[e]);
    zmax = warp_max(zmax);
    for (int e = lane; e < E; e += 32) zsum += expf(z[e] - zmax);
    zsum = warp_sum(zsum);
  }
  auto score = [&](int e) { return soft ? expf(z[e] - zmax) / zsum : 1.0f / (1.0f + expf(-z[e])); };
  for (int e = lane; e < E; e += 32) choice[e] = score(e) + (corr ? corr[e] : 0.f);
  __syncwarp();
  if (n_groups > 1 && keep < n_groups) {
    const int per = E / n_groups;
    for (int g = lane; g < n_groups; g += 32) {
      // the sum of the group's gtop largest choice scores: gtop passes over the group, each taking the next largest
      float sum = 0.f;
      int last_i = -1; float last_v = INFINITY;
      for (int c = 0; c < gtop && c < per; ++c) {
        float best = -INFINITY; int bi = -1;
        for (int i = 0; i < per; ++i) {
          const float v = choice[g * per + i];
          const bool after = v < last_v || (v == last_v && i > last_i);      // not yet taken, in (value desc, index asc) order
          if (after && (bi < 0 || v > best)) { best = v; bi = i; }
        }
        sum += best; last_v = best; last_i = bi;
      }
      gscore[g] = sum;
    }
    __syncwarp();
    for (int c = 0; c < keep; ++c) {
      float best = -INFINITY; int bi = 0x7fffffff;
      for (int g = lane; g < n_groups; g += 32) {
        const float v = gscore[g];
        if (v != INFINITY && (bi == 0x7fffffff || v > best || (v == best && g < bi))) { best = v; bi = g; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > best || (ov == best && oi < bi))) { best = ov; bi = oi; }
      }
      if (lane == 0 && bi != 0x7fffffff) gscore[bi] = INFINITY;
      __syncwarp();
    }
    for (int e = lane; e < E; e += 32) if (gscore[e / per] != INFINITY) choice[e] = -INFINITY;
    __syncwarp();
  }
  int taken[MOE_MAX_TOP];
  float tw[MOE_MAX_TOP];
  float chosen = 0.f;
#pragma unroll
  for (int c = 0; c < MOE_MAX_TOP; ++c) {
    if (c >= top) break;
    float best = -INFINITY; int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      bool free_ = true;
#pragma unroll
      for (int p = 0; p < MOE_MAX_TOP; ++p) if (p < c && taken[p] == e) free_ = false;
      const float v = choice[e];
      if (free_ && (bi == 0x7fffffff || v > best || (v == best && e < bi))) { best = v; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > best || (ov == best && oi < bi))) { best = ov; bi = oi; }
    }
    taken[c] = bi;
    tw[c] = score(bi);
    chosen += tw[c];
  }
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < MOE_MAX_TOP; ++c) {
      if (c >= top) break;
      idx[c] = taken[c];
      w[c] = renorm ? tw[c] / (chosen + 1e-20f) : tw[c];
    }
  }
}

// One warp per token.  logits float32 [T, ld]; idx [T, top] int32; w [T, top] float32.
__global__ void __launch_bounds__(128)
moe_route_kernel(const float* __restrict__ logits, int ld, int T, int E, int top, int renorm,
                 int* __restrict__ idx, float* __restrict__ w) {
  const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (warp >= T) return;
  route_warp(logits + (size_t)warp * ld, E, top, renorm, idx + (size_t)warp * top, w + (size_t)warp * top, lane);
}

FELLM_API int fellm_moe_route(const float* logits, int ld, int T, int E, int top, int renorm, int* idx, float* w,
                              cudaStream_t stream) {
  if (T <= 0) return 0;
  if (E < 1 || top < 1 || top > E || top > MOE_MAX_TOP) return FELLM_ERR_SIZE;
  if (!logits || !idx || !w) return FELLM_ERR_ARG;
  moe_route_kernel<<<(T + 3) / 4, 128, 0, stream>>>(logits, ld, T, E, top, renorm, idx, w);
  return launch_status();
}

// The router's product and the routing in one kernel: a block per token, its warps take the experts by turns
// (z_e = sum_k h[k] Wr[e, k] in float32: a lane sums its share of k in order, the lanes are added by a butterfly: the
// order depends on K alone), then the first warp routes.  h [T, ldh] and Wr [E, K] bfloat16 or float32.  VEC (both
// bfloat16, K a multiple of 8, rows on 16-byte boundaries): a lane takes eight k at a time.
// Bound by its latencies: the matrix comes from memory, so the blocks ask the L2 for it, a share each, while they wait for the
// kernel in front, and up to 16 experts have a warp each at once.
// The five launches of a layer as dependents, this and the plan's scan by a warp: 8 tokens, two of twelve choices, width 1,024, experts of
// 3,328: two layers 83.2 -> 75.3 us; 1 token 62.0 -> 55.8; 48 tokens of width 2,048 1,010 -> 1,007.
#define ROUTER_WARPS 8
#define ROUTER_WARPS_ROW 16
template <typename TA, typename TW, bool VEC>
__global__ void __launch_bounds__(ROUTER_WARPS_ROW * 32)
moe_router_kernel(const TA* h, int ldh, const TW* __restrict__ Wr, int K, int E, int top, int renorm,
                  int* idx, float* w, int form, const float* __restrict__ corr,
                  int n_groups, int keep, int gtop, const float* __restrict__ bias) {
  extern __shared__ float zs[];                 // [E]; the choice forms: + [E + n_groups]
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const size_t bytes = (size_t)E * K * sizeof(TW), step = (size_t)gridDim.x * blockDim.x * 128;
  for (size_t i = ((size_t)t * blockDim.x + threadIdx.x) * 128; i < bytes; i += step)
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)Wr + i));
  pdl_wait();
  pdl_launch_dependents();
  const TA* hr = h + (size_t)t * ldh;
  for (int e = warp; e < E; e += warps) {
    const TW* wr = Wr + (size_t)e * K;
    float s = 0.f;
    if constexpr (VEC) {
#pragma unroll 4
      for (int k = lane * 8; k < K; k += 256) {
        float a[8], b[8];
        unpack8(*(const uint4*)(hr + k), a); unpack8(*(const uint4*)(wr + k), b);
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(a[j], b[j], s);
      }
    } else {
      for (int k = lane; k < K; k += 32) s = fmaf(to_f(hr[k]), to_f(wr[k]), s);
    }
    s = warp_sum(s);
    if (lane == 0) zs[e] = bias ? s + bias[e] : s;
  }
  __syncthreads();
  if (warp == 0) {
    if (form) route_choice_warp(form == 2, zs, corr, E, top, renorm, n_groups, keep, gtop, zs + E, idx + (size_t)t * top, w + (size_t)t * top, lane);
    else route_warp(zs, E, top, renorm, idx + (size_t)t * top, w + (size_t)t * top, lane);
  }
}

// The same sums for many tokens (bfloat16, as VEC above): a warp a token, its experts four at a time against one reading
// of h, so that no warp waits while another routes.
__global__ void __launch_bounds__(ROUTER_WARPS * 32)
moe_router_many_kernel(const bf16* __restrict__ h, int ldh, const bf16* __restrict__ Wr, int T, int K, int E, int top, int renorm,
                       int* __restrict__ idx, float* __restrict__ w, int form, const float* __restrict__ corr,
                       int n_groups, int keep, int gtop, const float* __restrict__ bias, int per_warp) {
  extern __shared__ float zs_all[];             // per_warp floats a warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.x * ROUTER_WARPS + warp;
  if (t >= T) return;
  float* zs = zs_all + (size_t)warp * per_warp;
  const bf16* hr = h + (size_t)t * ldh;
  for (int e0 = 0; e0 < E; e0 += 4) {
    const bf16* wr[4];
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i) wr[i] = Wr + (size_t)min(e0 + i, E - 1) * K;
#pragma unroll 2
    for (int k = lane * 8; k < K; k += 256) {
      float a[8];
      unpack8(*(const uint4*)(hr + k), a);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float b[8];
        unpack8(*(const uint4*)(wr[i] + k), b);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[i] = fmaf(a[j], b[j], s[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i] = warp_sum(s[i]);
      if (lane == 0 && e0 + i < E) zs[e0 + i] = bias ? s[i] + bias[e0 + i] : s[i];
    }
  }
  __syncwarp();
  if (form) route_choice_warp(form == 2, zs, corr, E, top, renorm, n_groups, keep, gtop, zs + E, idx + (size_t)t * top, w + (size_t)t * top, lane);
  else route_warp(zs, E, top, renorm, idx + (size_t)t * top, w + (size_t)t * top, lane);
}

FELLM_API int fellm_moe_router(const void* h, int h_bf16, int ldh, const void* Wr, int w_bf16, int T, int K, int E, int top,
                               int renorm, int* idx, float* w, int form, const float* corr, int n_groups, int keep,
                               int gtop, const float* bias, cudaStream_t stream) {
  // bias (float32 [E] or null) is added to the logits before anything looks at them.
  // form = 0: softmax scores over all experts, the largest chosen.  form = 1: sigmoid scores, form = 2: softmax scores over
  // all experts, both with a correction added for the choice (corr float32 [E] or null) and the choice limited to `keep` of
  // n_groups groups ranked by their gtop best choice scores.
  if (T <= 0) return 0;
  if (n_groups < 1) n_groups = 1;
  if (E < 1 || top < 1 || top > E || top > MOE_MAX_TOP || (size_t)(2 * E + n_groups) * sizeof(float) > 48 * 1024) return FELLM_ERR_SIZE;
  if (form < 0 || form > 2 || (form && (E % n_groups || keep < 1 || keep > n_groups || gtop < 1 || top > (E / n_groups) * keep))) return FELLM_ERR_SIZE;
  if (!h || !Wr || !idx || !w) return FELLM_ERR_ARG;
  const size_t sh = (size_t)(form ? 2 * E + n_groups : E) * sizeof(float);
  // (few tokens: a dependent of the kernel in front; its blocks are there, and their matrix, when that one ends)
  const int warps = E < 4 ? 4 : E < ROUTER_WARPS_ROW ? E : ROUTER_WARPS_ROW;
  int rc = 0;
#define ROUTER(TA_, TW_, V_) rc = launch_k_class(T < MOE_FEW_TOKENS ? 1 : 0, moe_router_kernel<TA_, TW_, V_>, dim3(T), dim3(warps * 32), sh, stream, 1, \
        (const TA_*)h, ldh, (const TW_*)Wr, K, E, top, renorm, idx, w, form, corr, n_groups, keep, gtop, bias)
  const bool vec = h_bf16 && w_bf16 && K % 8 == 0 && ldh % 8 == 0 && (((uintptr_t)h | (uintptr_t)Wr) & 15) == 0;
  if (vec && T >= 256 && sh * ROUTER_WARPS <= 48 * 1024) {
    moe_router_many_kernel<<<(T + ROUTER_WARPS - 1) / ROUTER_WARPS, ROUTER_WARPS * 32, sh * ROUTER_WARPS, stream>>>(
        (const bf16*)h, ldh, (const bf16*)Wr, T, K, E, top, renorm, idx, w, form, corr, n_groups, keep, gtop, bias, (int)(sh / sizeof(float)));
    return launch_status();
  }
  if (vec) ROUTER(bf16, bf16, true);
  else if (h_bf16) { if (w_bf16) ROUTER(bf16, bf16, false); else ROUTER(bf16, float, false); }
  else { if (w_bf16) ROUTER(float, bf16, false); else ROUTER(float, float, false); }
#undef ROUTER
  return rc;
}

// ---------------------------------------------------------------- the plan
// Pairs p = t * top + c, P of them.  A choice beyond the E experts (an identity expert: the token's input handed on, no
// product) is no row of the plan: its place is -1.  n_tiles[0]: row tiles, n_tiles[1]: sorted rows.  Tile i of PLAN_TILE
// pairs: counts[i][e] and each pair's rank among the pairs of its tile that chose the same expert before it.
__global__ void __launch_bounds__(PLAN_TILE)
moe_count_kernel(const int* __restrict__ idx, int P, int E, int* __restrict__ counts, int* __restrict__ rank, int per_warp) {
  extern __shared__ int sh[];
  const int p = blockIdx.x * PLAN_TILE + threadIdx.x;
  const int e = p < P && idx[p] < E ? idx[p] : -1;
  if (per_warp) {
    // [32 warps][E]: a warp's pairs of each expert; then, down the warps, those in front of it
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < 32 * E; i += PLAN_TILE) sh[i] = 0;
    __syncthreads();
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int before = __popc(same & ((1u << lane) - 1));
    if (e >= 0 && before == 0) sh[warp * E + e] = __popc(same);
    __syncthreads();
    for (int i = threadIdx.x; i < E; i += PLAN_TILE) {
      int n = 0;
      for (int w = 0; w < 32; ++w) { const int c = sh[w * E + i]; sh[w * E + i] = n; n += c; }
      counts[(size_t)blockIdx.x * E + i] = n;
    }
    __syncthreads();
    if (e >= 0) rank[p] = sh[warp * E + e] + before;
    return;
  }
  int* ex = sh;                          // [PLAN_TILE]
  ex[threadIdx.x] = e;
  for (int i = threadIdx.x; i < E; i += PLAN_TILE) counts[(size_t)blockIdx.x * E + i] = 0;
  __syncthreads();
  if (e < 0) return;
  int r = 0;
  for (int j = 0; j < (int)threadIdx.x; ++j) r += ex[j] == e;
  rank[p] = r;
  // the last pair of its expert in the tile knows the count
  bool last = true;
  for (int j = threadIdx.x + 1; j < PLAN_TILE && last; ++j) last = ex[j] != e;
  if (last) counts[(size_t)blockIdx.x * E + e] = r + 1;
}

// One block.  base[i][e] = first sorted row of tile i's pairs of expert e (experts in order, tiles in order inside an
// expert); row tiles of BM rows: table[n] = (expert, first row, rows), n_tiles.
__global__ void __launch_bounds__(1024)
moe_scan_kernel(const int* __restrict__ counts, int n_plan_tiles, int E, int BM, int* __restrict__ base,
                int* __restrict__ table, int* __restrict__ n_tiles) {
  extern __shared__ int sh[];            // [E] rows of an expert, then [E] its first row, then [E] its first row tile
  int* rows = sh; int* first = sh + E; int* first_tile = sh + 2 * E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int n = 0;
    for (int i = 0; i < n_plan_tiles; ++i) n += counts[(size_t)i * E + e];
    rows[e] = n;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0, tiles = 0;
    for (int e = 0; e < E; ++e) { first[e] = at; first_tile[e] = tiles; at += rows[e]; tiles += (rows[e] + BM - 1) / BM; }
    n_tiles[0] = tiles; n_tiles[1] = at;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int at = first[e];
    for (int i = 0; i < n_plan_tiles; ++i) { base[(size_t)i * E + e] = at; at += counts[(size_t)i * E + e]; }
    int n = first_tile[e];
    for (int r = 0; r < rows[e]; r += BM, ++n) {
      table[3 * n] = e; table[3 * n + 1] = first[e] + r; table[3 * n + 2] = min(BM, rows[e] - r);
    }
  }
}

// sorted[place] = pair, place_of[pair] = place (-1: an identity expert's)
__global__ void moe_place_kernel(const int* __restrict__ idx, const int* __restrict__ rank, const int* __restrict__ base,
                                 int P, int E, int* __restrict__ sorted, int* __restrict__ place_of) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  if (idx[p] >= E) { place_of[p] = -1; return; }
  const int place = base[(size_t)(p / PLAN_TILE) * E + idx[p]] + rank[p];
  sorted[place] = p;
  place_of[p] = place;
}

// Up to PLAN_TILE pairs (a decode step): count, scan and places in one block of a thread a pair; the first warp scans, an expert a lane.
__global__ void __launch_bounds__(PLAN_TILE)
moe_plan_small_kernel(const int* idx, int P, int E, int BM, int* sorted, int* place_of, int* table, int* n_tiles) {
  __shared__ int ex[PLAN_TILE];
  extern __shared__ int sh[];            // [E] rows of an expert, then [E] its first row
  int* rows = sh; int* first = sh + E;
  const int p = threadIdx.x;
  for (int i = p; i < E; i += blockDim.x) rows[i] = 0;
  pdl_wait();
  pdl_launch_dependents();
  const int e = p < P && idx[p] < E ? idx[p] : -1;
  ex[p] = e;
  __syncthreads();
  int r = 0;
  if (e >= 0) {
    for (int j = 0; j < p; ++j) r += ex[j] == e;
    bool last = true;
    for (int j = p + 1; j < P && last; ++j) last = ex[j] != e;
    if (last) rows[e] = r + 1;
  }
  __syncthreads();
  if (p < 32) {
    int at = 0, tiles = 0;               // rows and row tiles of the experts before these 32
    for (int i0 = 0; i0 < E; i0 += 32) {
      const int i = i0 + p, n = i < E ? rows[i] : 0, nt = (n + BM - 1) / BM;
      int sum = n, sum_t = nt;
#pragma unroll
      for (int o = 1; o < 32; o *= 2) {
        const int a = __shfl_up_sync(0xffffffffu, sum, o), b = __shfl_up_sync(0xffffffffu, sum_t, o);
        if (p >= o) { sum += a; sum_t += b; }
      }
      const int f = at + sum - n;
      if (i < E) first[i] = f;
      for (int q = 0, k = tiles + sum_t - nt; q < n; q += BM, ++k) {
        table[3 * k] = i; table[3 * k + 1] = f + q; table[3 * k + 2] = min(BM, n - q);
      }
      at += __shfl_sync(0xffffffffu, sum, 31);
      tiles += __shfl_sync(0xffffffffu, sum_t, 31);
    }
    if (p == 0) { n_tiles[0] = tiles; n_tiles[1] = at; }
  }
  __syncthreads();
  if (p < P && e < 0) place_of[p] = -1;
  if (e >= 0) {
    const int place = first[e] + r;
    sorted[place] = p;
    place_of[p] = place;
  }
}

// scratch (int32): counts [tiles][E] | base [tiles][E] | rank [P]
FELLM_API int fellm_moe_plan(const int* idx, int P, int E, int BM, int* scratch, int* sorted, int* place_of, int* table,
                             int* n_tiles, cudaStream_t stream) {
  if (P <= 0) return 0;
  if (E < 1 || BM < 1) return FELLM_ERR_SIZE;
  if (!idx || !scratch || !sorted || !place_of || !table || !n_tiles) return FELLM_ERR_ARG;
  if (P <= PLAN_TILE && (size_t)2 * E * sizeof(int) <= 40 * 1024) {
    return launch_k_class(P < MOE_FEW_TOKENS ? 1 : 0, moe_plan_small_kernel, dim3(1), dim3((P + 31) / 32 * 32), (size_t)2 * E * sizeof(int), stream, 1,
                          idx, P, E, BM, sorted, place_of, table, n_tiles);
  }
  const int tiles = (P + PLAN_TILE - 1) / PLAN_TILE;
  int* counts = scratch; int* base = counts + (size_t)tiles * E; int* rank = base + (size_t)tiles * E;
  const bool per_warp = E <= 320;        // 40 KB of counts; more experts: every pair looks at the tile's others
  moe_count_kernel<<<tiles, PLAN_TILE, (per_warp ? (size_t)32 * E : PLAN_TILE) * sizeof(int), stream>>>(idx, P, E, counts, rank, per_warp);
  const size_t sh = (size_t)3 * E * sizeof(int);
  if (sh > 48 * 1024) return FELLM_ERR_SIZE;
  moe_scan_kernel<<<1, 1024, sh, stream>>>(counts, tiles, E, BM, base, table, n_tiles);
  moe_place_kernel<<<(P + 255) / 256, 256, 0, stream>>>(idx, rank, base, P, E, sorted, place_of);
  return launch_status();
}

// ---------------------------------------------------------------- grouped products, float32 FMA
// Every output is ONE chain of fused multiply-adds over k = 0..K-1: the 32-bit engine's product, and the bfloat16
// engine's where the tensor-core kernel below does not take a size.
// GATED: W[e] is [2N, K]; the epilogue stores SiLU(gate) * up.  inter = 0: the N gate rows first, then the N up
// rows; inter = 1: blocks of 8 gate rows and 8 up rows by turns (the layout the tcgen05 product's epilogue reads).
// Rows of A: gather[row] / top when gather is given (a pair's token), else the sorted row itself.
__device__ __forceinline__ int gate_row(int n, int inter) { return inter ? ((n >> 3) << 4) + (n & 7) : n; }
__device__ __forceinline__ int up_row(int n, int N, int inter) { return inter ? ((n >> 3) << 4) + 8 + (n & 7) : N + n; }
#define FB 64
#define FK 16
template <typename TA, typename TW, typename TO, bool GATED>
__global__ void __launch_bounds__(256)
moe_gemm_fma_kernel(const TA* __restrict__ A, int lda, const int* __restrict__ gather, int top,
                    const TW* __restrict__ W, TO* __restrict__ C, int ldc, int N, int K,
                    const int* __restrict__ table, const int* __restrict__ n_tiles, int inter, float act_limit, float act_alpha) {
  if ((int)blockIdx.x >= *n_tiles) return;
  __shared__ float As[FK][FB + 1];
  __shared__ float Ws[GATED ? 2 : 1][FK][FB + 1];
  __shared__ int arow[FB];
  const int e = table[3 * blockIdx.x], row0 = table[3 * blockIdx.x + 1], rows = table[3 * blockIdx.x + 2];
  const int n0 = blockIdx.y * FB;
  const TW* We = W + (size_t)e * (GATED ? 2 : 1) * N * K;
  for (int r = threadIdx.x; r < FB; r += 256)
    arow[r] = r < rows ? (gather ? gather[row0 + r] / top : row0 + r) : -1;
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;       // 4 columns x 4 rows a thread
  float acc[4][4], acc2[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = acc2[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += FK) {
    for (int i = threadIdx.x; i < FB * FK; i += 256) {
      const int r = i / FK, k = i - r * FK;
      const int ar = arow[r];
      As[k][r] = (ar >= 0 && k0 + k < K) ? to_f(A[(size_t)ar * lda + k0 + k]) : 0.f;
      const int n = n0 + r;
      const bool ok = n < N && k0 + k < K;
      Ws[0][k][r] = ok ? to_f(We[(size_t)(GATED ? gate_row(n, inter) : n) * K + k0 + k]) : 0.f;
      if (GATED) Ws[1][k][r] = ok ? to_f(We[(size_t)up_row(n, N, inter) * K + k0 + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < FK; ++k) {
      float a[4], b[4], b2[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) { b[j] = Ws[0][k][tx * 4 + j]; if (GATED) b2[j] = Ws[1][k][tx * 4 + j]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
          if (GATED) acc2[i][j] = fmaf(a[i], b2[j], acc2[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (GATED) {
        // in the bfloat16 engine gate and up are activations like those of the dense feed-forward: rounded first
        float g = to_f(from_f<TA>(v)), u = to_f(from_f<TA>(acc2[i][j]));
        v = glu_act(g, u, act_limit, act_alpha);
      }
      C[(size_t)(row0 + r) * ldc + n] = from_f<TO>(v);
    }
  }
}

// ---------------------------------------------------------------- grouped products, bfloat16 tensor cores
// 64 rows x 64 columns a CTA (x 2 column sets when GATED), K in steps of 32 through shared memory (rows padded to 40
// elements: the fragment loads of a warp fall on different banks), four warps of 16 rows each, mma.m16n8k16 with
// float32 accumulators.  A token's sum over K is the same chain of MMAs wherever the row lies in its tile.
#define TB 64
#define TK 32
#define TLD 40
__device__ __forceinline__ void mma16816(float* d, const unsigned* a, const unsigned* b) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <typename TO, bool GATED>
__global__ void __launch_bounds__(128)
moe_gemm_mma_kernel(const bf16* __restrict__ A, int lda, const int* __restrict__ gather, int top,
                    const bf16* __restrict__ W, TO* __restrict__ C, int ldc, int N, int K,
                    const int* __restrict__ table, const int* __restrict__ n_tiles, int inter, float act_limit, float act_alpha) {
  if ((int)blockIdx.x >= *n_tiles) return;
  __shared__ __align__(16) bf16 As[2][TB * TLD];
  __shared__ __align__(16) bf16 Ws[2][(GATED ? 2 : 1) * TB * TLD];
  __shared__ int arow[TB];
  const int e = table[3 * blockIdx.x], row0 = table[3 * blockIdx.x + 1], rows = table[3 * blockIdx.x + 2];
  const int n0 = blockIdx.y * TB;
  const bf16* We = W + (size_t)e * (GATED ? 2 : 1) * N * K;
  for (int r = threadIdx.x; r < TB; r += 128)
    arow[r] = r < rows ? (gather ? gather[row0 + r] / top : row0 + r) : -1;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  constexpr int NB = GATED ? 16 : 8;                   // blocks of 8 columns a warp: 64 columns (and 64 of the up set)
  float acc[NB][4];
#pragma unroll
  for (int j = 0; j < NB; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  // a thread copies 16 bytes at a time: 64 rows x 4 vectors of A, and of each column set of W
  auto stage = [&](int buf, int k0) {
    for (int i = threadIdx.x; i < TB * 4; i += 128) {
      const int r = i >> 2, kv = (i & 3) * 8;
      uint4 va = make_uint4(0, 0, 0, 0), vw = make_uint4(0, 0, 0, 0), vw2 = make_uint4(0, 0, 0, 0);
      const int ar = arow[r];
      if (ar >= 0 && k0 + kv < K) va = *(const uint4*)(A + (size_t)ar * lda + k0 + kv);
      const int n = n0 + r;
      if (n < N && k0 + kv < K) {
        vw = *(const uint4*)(We + (size_t)(GATED ? gate_row(n, inter) : n) * K + k0 + kv);
        if (GATED) vw2 = *(const uint4*)(We + (size_t)up_row(n, N, inter) * K + k0 + kv);
      }
      *(uint4*)(&As[buf][r * TLD + kv]) = va;
      *(uint4*)(&Ws[buf][r * TLD + kv]) = vw;
      if (GATED) *(uint4*)(&Ws[buf][(TB + r) * TLD + kv]) = vw2;
    }
  };
  const int n_k = (K + TK - 1) / TK;
  stage(0, 0);
  __syncthreads();
  for (int kb = 0; kb < n_k; ++kb) {
    const int buf = kb & 1;
    if (kb + 1 < n_k) stage(buf ^ 1, (kb + 1) * TK);
    const bf16* as = As[buf] + (warp * 16) * TLD;
#pragma unroll
    for (int kk = 0; kk < TK; kk += 16) {
      unsigned a[4];
      a[0] = *(const unsigned*)(as + gid * TLD + kk + tig * 2);
      a[1] = *(const unsigned*)(as + (gid + 8) * TLD + kk + tig * 2);
      a[2] = *(const unsigned*)(as + gid * TLD + kk + 8 + tig * 2);
      a[3] = *(const unsigned*)(as + (gid + 8) * TLD + kk + 8 + tig * 2);
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const bf16* ws = Ws[buf] + (j * 8 + gid) * TLD + kk + tig * 2;
        unsigned b[2];
        b[0] = *(const unsigned*)ws;
        b[1] = *(const unsigned*)(ws + 8);
        mma16816(acc[j], a, b);
      }
    }
    __syncthreads();
  }
  // c0, c1: row gid, columns 2 tig, 2 tig + 1; c2, c3: row gid + 8
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int r = warp * 16 + gid + half * 8;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int n = n0 + j * 8 + tig * 2 + c;
        if (n >= N) continue;
        float v = acc[j][half * 2 + c];
        if (GATED) {
          const float g = to_f(from_f<bf16>(v)), u = to_f(from_f<bf16>(acc[8 + j][half * 2 + c]));
          v = glu_act(g, u, act_limit, act_alpha);
        }
        C[(size_t)(row0 + r) * ldc + n] = from_f<TO>(v);
      }
    }
  }
}

// Few rows (a decode step): the product is bound by reading each chosen expert's matrix once.  A warp takes a slab of 16 weight
// rows (GATED: eight gate rows and their eight up rows) as the rows of mma.m16n8k16 and a slice of K; its columns are up to
// eight rows of A (more rows: again, the weights then come from L2).  A lane loads 8 consecutive k of rows g and g + 8 and
// feeds them, and the same k of A's row g, as the k slots {2c, 2c + 1, 2c + 8, 2c + 9} of two MMAs: 16-byte loads of both
// operands without shared memory, and VU chunks of 32 k (VU KB of weights a warp) on their way at once.  The slices of K of a slab
// are warps of one block, added in their order.  bfloat16 only; K a multiple of 8.  Every MMA starts from zero and the chunks' are
// added in pairs, in float32: an MMA that adds into its accumulator truncates.  Relative error of float32 results of 3,328 (6,144)
// products against float64: one chain of MMAs 3.8e-7 (7.4e-7), here 0.84e-7 (0.88e-7), float32 multiply-adds 0.90e-7 (1.09e-7); both
// products of 8 tokens 28.8 us either way.
// A warp a column and float32 FMA, four rows at once, spent its time on the conversions and multiply-adds of the weights it
// streamed: 8 tokens, two of twelve choices each, width 1,024, experts of 3,328: 27.3 us (up) and 20.6 us (down) there, 15.4
// and 9.7 here (82 and 41 MB of matrices met); 30 tokens 67 and 64 us there, 26 and 16 here.
#define VW 8            // warps a block
#define VU 8            // chunks of 32 k on their way
__device__ __forceinline__ void slab_mma(float (&s)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(s[0]), "+f"(s[1]), "+f"(s[2]), "+f"(s[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <typename TO, bool GATED, int KS>
__global__ void __launch_bounds__(VW * 32)
moe_slabs_kernel(const bf16* A, int lda, const int* gather, int top, const bf16* __restrict__ W, TO* C, int ldc, int N, int K,
                const int* table, const int* n_tiles, int inter, float act_limit, float act_alpha) {
  __shared__ float4 part[VW][32];
  pdl_wait();
  pdl_launch_dependents();
  if ((int)blockIdx.x >= *n_tiles) return;
  const int e = table[3 * blockIdx.x], row0 = table[3 * blockIdx.x + 1], rows = table[3 * blockIdx.x + 2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int slab = blockIdx.y * (VW / KS) + warp / KS, ks = warp % KS;
  const int n0 = slab * (GATED ? 8 : 16), na = n0 + g, nb = GATED ? na : na + 8;         // this lane's columns of the result
  const bf16* We = W + (size_t)e * (GATED ? 2 : 1) * N * K;
  const bf16* wa = We + (size_t)(GATED ? gate_row(min(na, N - 1), inter) : min(na, N - 1)) * K;
  const bf16* wb = We + (size_t)(GATED ? up_row(min(nb, N - 1), N, inter) : min(nb, N - 1)) * K;
  const int chunks = (K + 31) / 32, per = (chunks + KS - 1) / KS, first = ks * per, last = n0 < N ? min(chunks, first + per) : 0;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (int r0 = 0; r0 < rows; r0 += 8) {
    const int r = row0 + r0 + g;
    const bool live = r0 + g < rows;
    const bf16* ar = nullptr;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c0 = first; c0 < last; c0 += VU) {
      uint4 a[VU], b[VU], x[VU];
#pragma unroll
      for (int u = 0; u < VU; ++u) {
        const int k = (c0 + u) * 32 + 8 * c;
        const bool in = c0 + u < last && k < K;
        a[u] = in ? *(const uint4*)(wa + k) : zero;
        b[u] = in ? *(const uint4*)(wb + k) : zero;
      }
      if (!ar && live) ar = A + (size_t)(gather ? gather[r] / top : r) * lda;           // (behind the first weights)
#pragma unroll
      for (int u = 0; u < VU; ++u) {
        const int k = (c0 + u) * 32 + 8 * c;
        x[u] = (live && c0 + u < last && k < K) ? *(const uint4*)(ar + k) : zero;
      }
      float t[VU][4];                              // a chunk's two MMAs, then sums of neighbours
#pragma unroll
      for (int u = 0; u < VU; ++u) {
        float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
        slab_mma(lo, a[u].x, b[u].x, a[u].y, b[u].y, x[u].x, x[u].y);
        slab_mma(hi, a[u].z, b[u].z, a[u].w, b[u].w, x[u].z, x[u].w);
#pragma unroll
        for (int i = 0; i < 4; ++i) t[u][i] = lo[i] + hi[i];
      }
#pragma unroll
      for (int d = 1; d < VU; d *= 2)
#pragma unroll
        for (int u = 0; u < VU; u += 2 * d)
#pragma unroll
          for (int i = 0; i < 4; ++i) t[u][i] += t[u + d][i];
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] += t[0][i];
    }
    if (KS > 1) {
      __syncthreads();                             // (the parts before these have been added)
      part[warp][lane] = make_float4(s[0], s[1], s[2], s[3]);
      __syncthreads();
      if (ks == 0) {
#pragma unroll
        for (int w = 1; w < KS; ++w) {
          const float4 p = part[warp + w][lane];
          s[0] += p.x; s[1] += p.y; s[2] += p.z; s[3] += p.w;
        }
      }
    }
    if (ks == 0) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {                // result rows 2 c and 2 c + 1
        const int rr = r0 + 2 * c + j;
        if (rr >= rows) continue;
        TO* to = C + (size_t)(row0 + rr) * ldc;
        if (GATED) {
          if (na < N) to[na] = from_f<TO>(glu_act(to_f(from_f<bf16>(s[j])), to_f(from_f<bf16>(s[2 + j])), act_limit, act_alpha));
        } else {
          if (na < N) to[na] = from_f<TO>(s[j]);
          if (nb < N) to[nb] = from_f<TO>(s[2 + j]);
        }
      }
    }
  }
}

template <typename TO, bool GATED>
static int moe_slabs_launch(const void* A, int lda, const int* gather, int top, const void* W, void* C, int ldc, int N, int K, const int* table,
                            const int* n_tiles, int max_tiles, int inter, float act_limit, float act_alpha, cudaStream_t stream) {
  // slices of K of a slab: VU chunks each where there are eight of them or fewer
  const int chunks = (K + 31) / 32, slabs = ceil_div(N, GATED ? 8 : 16);
  int rc = 0;
#define MOE_SLABS(KS_) rc = launch_k_class(1, moe_slabs_kernel<TO, GATED, KS_>, dim3(max_tiles, ceil_div(slabs, VW / KS_)), dim3(VW * 32), 0, stream, 1, \
        (const bf16*)A, lda, gather, top, (const bf16*)W, (TO*)C, ldc, N, K, table, n_tiles, inter, act_limit, act_alpha)
  if (chunks > 4 * VU) MOE_SLABS(8); else if (chunks > 2 * VU) MOE_SLABS(4); else if (chunks > VU) MOE_SLABS(2); else MOE_SLABS(1);
#undef MOE_SLABS
  return rc;
}

// A [*, lda] (bfloat16 or float32), W [E][(gated ? 2 : 1) * N][K] of the same kind; C [P, ldc]: bfloat16 or float32
// when gated (the activation), float32 otherwise.  max_tiles: the table's capacity = the launch's first extent.
FELLM_API int fellm_moe_gemm(const void* A, int a_bf16, int lda, const int* gather, int top, const void* W, int w_bf16,
                             void* C, int c_bf16, int ldc, int N, int K, int gated, const int* table, const int* n_tiles,
                             int max_tiles, int use_mma, int inter, int few_rows, float act_limit, float act_alpha, cudaStream_t stream) {
  if (max_tiles <= 0) return 0;
  if (N < 1 || K < 1 || top < 1) return FELLM_ERR_SIZE;
  if (!A || !W || !C || !table || !n_tiles) return FELLM_ERR_ARG;
  if (a_bf16 != w_bf16 || (!gated && c_bf16) || (gated && c_bf16 != a_bf16)) return FELLM_ERR_ARG;
  const bool mma = use_mma && a_bf16 && K % 8 == 0 && lda % 8 == 0 && ((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0;
  if (mma && few_rows) {
    return gated ? moe_slabs_launch<bf16, true>(A, lda, gather, top, W, C, ldc, N, K, table, n_tiles, max_tiles, inter, act_limit, act_alpha, stream)
                 : moe_slabs_launch<float, false>(A, lda, gather, top, W, C, ldc, N, K, table, n_tiles, max_tiles, inter, act_limit, act_alpha, stream);
  }
  if (mma) {
    dim3 grid(max_tiles, (N + TB - 1) / TB);
    if (gated)
      moe_gemm_mma_kernel<bf16, true><<<grid, 128, 0, stream>>>((const bf16*)A, lda, gather, top, (const bf16*)W, (bf16*)C, ldc, N, K, table, n_tiles, inter, act_limit, act_alpha);
    else
      moe_gemm_mma_kernel<float, false><<<grid, 128, 0, stream>>>((const bf16*)A, lda, gather, top, (const bf16*)W, (float*)C, ldc, N, K, table, n_tiles, inter, act_limit, act_alpha);
    return launch_status();
  }
  dim3 grid(max_tiles, (N + FB - 1) / FB);
  if (a_bf16) {
    if (gated)
      moe_gemm_fma_kernel<bf16, bf16, bf16, true><<<grid, 256, 0, stream>>>((const bf16*)A, lda, gather, top, (const bf16*)W, (bf16*)C, ldc, N, K, table, n_tiles, inter, act_limit, act_alpha);
    else
      moe_gemm_fma_kernel<bf16, bf16, float, false><<<grid, 256, 0, stream>>>((const bf16*)A, lda, gather, top, (const bf16*)W, (float*)C, ldc, N, K, table, n_tiles, inter, act_limit, act_alpha);
  } else {
    if (gated)
      moe_gemm_fma_kernel<float, float, float, true><<<grid, 256, 0, stream>>>((const float*)A, lda, gather, top, (const float*)W, (float*)C, ldc, N, K, table, n_tiles, inter, act_limit, act_alpha);
    else
      moe_gemm_fma_kernel<float, float, float, false><<<grid, 256, 0, stream>>>((const float*)A, lda, gather, top, (const float*)W, (float*)C, ldc, N, K, table, n_tiles, inter, act_limit, act_alpha);
  }
  return launch_status();
}

// ---------------------------------------------------------------- rows in sorted order
// out[r, :] = a[sorted[r] / top, :]   (bfloat16, K a multiple of 8: 16 bytes a thread): the input of the tcgen05
// grouped product, whose TMA boxes want an expert's rows side by side.
__global__ void moe_gather_kernel(const bf16* __restrict__ a, int lda, const int* __restrict__ sorted, int top,
                                  bf16* __restrict__ out, int K, const int* __restrict__ n_tiles) {
  const int r = blockIdx.x;
  if (r >= n_tiles[1]) return;
  const bf16* src = a + (size_t)(sorted[r] / top) * lda;
  bf16* dst = out + (size_t)r * K;
  for (int k = threadIdx.x * 8; k < K; k += blockDim.x * 8) *(uint4*)(dst + k) = *(const uint4*)(src + k);
}

FELLM_API int fellm_moe_gather(const void* a, int lda, const int* sorted, int top, void* out, int P, int K, const int* n_tiles,
                               cudaStream_t stream) {
  if (P <= 0) return 0;
  if (!a || !sorted || !out || !n_tiles) return FELLM_ERR_ARG;
  if (K % 8 || lda % 8 || ((uintptr_t)a % 16) || ((uintptr_t)out % 16)) return FELLM_ERR_SIZE;
  moe_gather_kernel<<<P, 128, 0, stream>>>((const bf16*)a, lda, sorted, top, (bf16*)out, K, n_tiles);
  return launch_status();
}

// ---------------------------------------------------------------- the weighted sum into the residual stream
// x[t, :] += sum_c w[t, c] * r_c, c = 0 .. top-1 in order, float32 (store: x[t, :] = the sum); r_c = y[place_of[t * top +
// c], :], or, place -1 (an identity expert), the token's input h[t, :].
template <typename TH>
__global__ void moe_combine_kernel(float* __restrict__ x, const float* __restrict__ y, const int* __restrict__ place_of,
                                   const float* __restrict__ w, const TH* __restrict__ h, int ldh, int top, int d, int store) {
  const int t = blockIdx.x;
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    float s = 0.f;
    for (int c = 0; c < top; ++c) {
      const int place = place_of[(size_t)t * top + c];
      s = fmaf(w[(size_t)t * top + c], place < 0 ? to_f(h[(size_t)t * ldh + i]) : y[(size_t)place * d + i], s);
    }
    x[(size_t)t * d + i] = store ? s : x[(size_t)t * d + i] + s;
  }
}

// The same, d a multiple of 4 and everything on 16-byte boundaries (h on 8): four elements a thread.
__device__ __forceinline__ float4 load4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 raw = *(const uint2*)p;
  const __nv_bfloat162* h2 = (const __nv_bfloat162*)&raw;
  const float2 a = __bfloat1622float2(h2[0]), b = __bfloat1622float2(h2[1]);
  return make_float4(a.x, a.y, b.x, b.y);
}
template <typename TH>
__global__ void moe_combine_vec_kernel(float* x, const float* y, const int* place_of, const float* w, const TH* h, int ldh, int T, int top,
                                       int d4, int store) {
  pdl_wait();
  pdl_launch_dependents();
  const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= (long long)T * d4) return;
  const int t = (int)(u / d4), i = 4 * (int)(u - (long long)t * d4), d = 4 * d4;
  float4* dst = (float4*)(x + (size_t)t * d + i);
  const float4 old = store ? make_float4(0.f, 0.f, 0.f, 0.f) : *dst;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int c = 0; c < top; ++c) {
    const int place = place_of[(size_t)t * top + c];
    const float f = w[(size_t)t * top + c];
    const float4 v = place < 0 ? load4(h + (size_t)t * ldh + i) : load4(y + (size_t)place * d + i);
    s.x = fmaf(f, v.x, s.x); s.y = fmaf(f, v.y, s.y); s.z = fmaf(f, v.z, s.z); s.w = fmaf(f, v.w, s.w);
  }
  *dst = store ? s : make_float4(old.x + s.x, old.y + s.y, old.z + s.z, old.w + s.w);
}

// h [T, ldh] (bfloat16 or float32): needed where a plan has identity experts, else null.
FELLM_API int fellm_moe_combine(float* x, const float* y, const int* place_of, const float* w, const void* h, int h_bf16, int ldh,
                                int T, int top, int d, int store, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!x || !y || !place_of || !w) return FELLM_ERR_ARG;
  if (d % 4 == 0 && (((uintptr_t)x | (uintptr_t)y | (uintptr_t)h) & 15) == 0 && ldh % 4 == 0) {
    const int d4 = d / 4;
    const unsigned blocks = (unsigned)(((long long)T * d4 + 127) / 128);
    const int cls = T < MOE_FEW_TOKENS ? 1 : 0;
    if (h_bf16) return launch_k_class(cls, moe_combine_vec_kernel<bf16>, dim3(blocks), dim3(128), 0, stream, 1, x, y, place_of, w, (const bf16*)h, ldh, T, top, d4, store);
    return launch_k_class(cls, moe_combine_vec_kernel<float>, dim3(blocks), dim3(128), 0, stream, 1, x, y, place_of, w, (const float*)h, ldh, T, top, d4, store);
  }
  const int threads = d >= 256 ? 256 : 128;
  if (h_bf16) moe_combine_kernel<bf16><<<T, threads, 0, stream>>>(x, y, place_of, w, (const bf16*)h, ldh, top, d, store);
  else moe_combine_kernel<float><<<T, threads, 0, stream>>>(x, y, place_of, w, (const float*)h, ldh, top, d, store);
  return launch_status();
}
