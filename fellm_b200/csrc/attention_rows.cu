// Attention of single rows (decode steps) over the paged bfloat16 cache with float32 scores, probabilities and sums on CUDA
// cores, for the forms the tensor-core decode kernels do not take (biases by distance, query temperatures, chunks, values
// that are the keys) and wherever probabilities are to stay 32-bit: what paged_attention_simt_kernel (attention_simt.cu)
// computes for such a row, for key sizes of 64 and 128 and 1, 2 or 4 heads a kv head.
//
// That kernel has a block a (row, head) and a lane a key: every head of a group reads the group's keys again, a lane's
// loads are a key's 128 bytes one after another, and the values are read row by row behind them (48 us for 12 rows of 16
// heads over 1,024 keys; 13 MB of cache).  Here a warp takes 32 keys for ALL heads of the group: LPK lanes a key, 16 bytes a
// lane, the 32 keys' K and V all in flight at once; the partial dot products of 32 keys go through the lanes by a
// transposing butterfly that leaves lane j with the whole scores of key j; the softmax runs on a key a lane; then every lane
// adds its 8 elements of its keys' values, the probabilities by shuffles.  A row and kv head's keys are dealt out in tiles of
// 32 over the warps of up to eight parts of four warps (a.parts, by the window or chunk alone: ~1 tile a warp for a window of
// 1,024), whose sums lie in shared memory until all are there and are then added in one fixed order.  A cluster has as many
// blocks as fill the device; a block of a smaller one takes several neighbouring parts one after another.  So a row's bits
// do not depend on how many rows decode beside it (the same 12 rows: 9.5 us; 48 rows 20.9, 128 rows 63; with the shares by the
// batch, in whose order rows were added before, 8.9, 19.3 and 62.5).  Bound by: latency, one round trip to memory for the page
// numbers, one for keys and values, one to the other blocks' sums.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

#define AR_WARPS 4
#define AR_PARTS 8            // most parts of a row's keys

struct ArArgs {
  const bf16* q; const bf16* pool; const int* block_table; const int* positions; const int* row_slot;
  bf16* out; int* status;
  const float* gate; const float* slopes; const bf16* og;
  int parts, ldq, max_pages, H, G, page_shift, layer, layers_in_group, window, chunk, ldg, ldog, qt_every, new_k_off, new_v_off;
  float scale, softcap, qt_coef;
};

__device__ __forceinline__ void ar_unpack(const uint4& raw, float* f) {
  const __nv_bfloat162* h = (const __nv_bfloat162*)&raw;
#pragma unroll
  for (int e = 0; e < 4; ++e) { const float2 v = __bfloat1622float2(h[e]); f[2 * e] = v.x; f[2 * e + 1] = v.y; }
}

template <int HD, int R, bool VK>
__global__ void __launch_bounds__(AR_WARPS * 32, HD != 64 || VK ? 1 : R == 2 ? 4 : R == 4 ? 3 : 1)       // (blocks an SM: see ar_launch)
attention_rows_kernel(const ArArgs a) {
  constexpr int LPK = HD / 8, KPI = 32 / LPK, NI = 32 / KPI;        // lanes a key, keys a load, loads a tile (= LPK)
  typedef float Sums[AR_WARPS][R][HD + 4];                           // a part's: per warp and head the elements, then m, l
  extern __shared__ __align__(16) float ar_smem[];
  Sums* sums = (Sums*)ar_smem;                                       // the block's parts'
  __shared__ float factor[R][AR_PARTS * AR_WARPS], total[R];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = gridDim.x, rank = blockIdx.x, g = blockIdx.y, row = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane / LPK, sub = lane % LPK;
  // Launched as a programmatic dependent of the kernel that makes q (and this token's key and value): who is where is read ahead of
  // the wait, a warp's first page number with it (copies from the host write them, no kernel of a step).
  const int pos = a.positions[row];
  const int* bt = a.block_table + (size_t)a.row_slot[row] * a.max_pages;
  int k_begin = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
  if (a.chunk > 0) k_begin = max(k_begin, pos / a.chunk * a.chunk);
  const int pt = 1 << a.page_shift;
  const size_t record = (size_t)a.G * pt * (VK ? HD : 2 * HD);
  const bf16* qrow = a.q + (size_t)row * a.ldq;
  const bool fused = a.new_k_off >= 0;

  const int n_parts = a.parts / cs, e0 = 8 * sub + (HD == 64 ? 4 * (grp & 1) + 2 * (grp >> 1) : 4 * grp);
  const int first = k_begin + 32 * (rank * n_parts * AR_WARPS + warp);
  int page = first <= pos ? bt[min(first + lane, pos) >> a.page_shift] : 0;
  pdl_wait();

  float q[R][8];
  const float qt = a.qt_every > 0 ? 1.0f + a.qt_coef * logf((float)((pos + 1) / a.qt_every + 1)) : 1.0f;
  float slope[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    ar_unpack(*(const uint4*)(qrow + (size_t)(g * R + r) * HD + 8 * sub), q[r]);
#pragma unroll
    for (int e = 0; e < 8; ++e) q[r][e] *= qt;
    slope[r] = a.slopes ? a.slopes[g * R + r] : 0.f;
  }

  for (int i = 0; i < n_parts; ++i) {
    const int p = rank * n_parts + i;
    float m[R], l[R];
    float acc[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[r][e] = 0.f;
    }

    for (int k0 = k_begin + 32 * (p * AR_WARPS + warp); k0 <= pos; k0 += 32 * AR_WARPS * a.parts) {
      if (k0 != first) page = bt[min(k0 + lane, pos) >> a.page_shift];
      page = max(page, 0);                                          // an unmapped entry (-1) must never become an address
      uint4 kr[NI], vr[VK ? 1 : NI];
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int j = i * KPI + grp, kj = min(k0 + j, pos);            // (beyond the row: the row's own key once more, masked below)
        const int pg = __shfl_sync(0xffffffffu, page, j);
        const bf16* krow = a.pool + ((size_t)pg * a.layers_in_group + a.layer) * record + ((size_t)g * pt + (kj & (pt - 1))) * HD;
        const bf16* vrow = krow + (size_t)a.G * pt * HD;
        if (fused && kj == pos) {
          krow = qrow + a.new_k_off + (size_t)g * HD;
          vrow = qrow + a.new_v_off + (size_t)g * HD;
        }
        kr[i] = *(const uint4*)(krow + 8 * sub);
        if (!VK) vr[i] = *(const uint4*)(vrow + 8 * sub);
      }
      float s[R][NI];
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        float kf[8];
        ar_unpack(kr[i], kf);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float d = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) d = fmaf(q[r][e], kf[e], d);
          s[r][i] = d;
        }
      }
      // a key's LPK partial sums, for NI = LPK keys of this lane group: lane `sub` ends with the whole of key sub * KPI + grp
      float pr[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int w = LPK / 2; w > 0; w >>= 1) {
          const bool up = sub & w;
#pragma unroll
          for (int i = 0; i < w; ++i) {
            const float give = up ? s[r][i] : s[r][i + w], keep = up ? s[r][i + w] : s[r][i];
            s[r][i] = keep + __shfl_xor_sync(0xffffffffu, give, w);
          }
        }
      }
      const int kj = k0 + sub * KPI + grp;
      const bool seen = kj <= pos;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float x = s[r][0] * a.scale;
        if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
        x -= slope[r] * (float)(pos - kj);
        x = seen ? x : -INFINITY;
        const float mn = fmaxf(m[r], warp_max(x));                     // (a tile holds a key that the row sees)
        pr[r] = seen ? expf(x - mn) : 0.f;
        const float corr = expf(m[r] - mn);
        m[r] = mn;
        l[r] = fmaf(l[r], corr, pr[r]);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[r][e] *= corr;
      }
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const bool live = k0 + i * KPI + grp <= pos;                   // (a masked key's value is not touched: 0 * NaN)
        float vf[8];
        ar_unpack(VK ? kr[i] : vr[VK ? 0 : i], vf);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float pi = __shfl_sync(0xffffffffu, pr[r], i, LPK);
          if (live) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[r][e] = fmaf(pi, vf[e], acc[r][e]);
          }
        }
      }
    }

    // the lane groups' sums: a lane ends with HD / 32 of the elements, from e0 on
#pragma unroll
    for (int r = 0; r < R; ++r) {
      l[r] = warp_sum(l[r]);
#pragma unroll
      for (int w = LPK, n = 4; w < 32; w <<= 1, n >>= 1) {
        const bool up = lane & w;
#pragma unroll
        for (int e = 0; e < n; ++e) {
          const float give = up ? acc[r][e] : acc[r][e + n], keep = up ? acc[r][e + n] : acc[r][e];
          acc[r][e] = keep + __shfl_xor_sync(0xffffffffu, give, w);
        }
      }
      float* to = sums[i][warp][r];
      if (HD == 64) *(float2*)(to + e0) = make_float2(acc[r][0], acc[r][1]);
      else *(float4*)(to + e0) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
      if (lane == 0) *(float2*)(to + HD) = make_float2(m[r], l[r]);
    }
  }

  pdl_launch_dependents();                         // (the next product's weights beside the merge, not beside the keys)
  // the step's own key and value into their page: nobody in this launch reads them from there
  if (fused && rank == 0 && warp == 0) {
    const int page = bt[pos >> a.page_shift];
    if (page < 0) {
      if (lane == 0 && a.status) atomicExch(a.status, 2);
    } else if (lane < LPK) {
      bf16* krow = const_cast<bf16*>(a.pool) + ((size_t)page * a.layers_in_group + a.layer) * record + ((size_t)g * pt + (pos & (pt - 1))) * HD;
      *(uint4*)(krow + 8 * lane) = *(const uint4*)(qrow + a.new_k_off + (size_t)g * HD + 8 * lane);
      if (!VK) *(uint4*)(krow + (size_t)a.G * pt * HD + 8 * lane) = *(const uint4*)(qrow + a.new_v_off + (size_t)g * HD + 8 * lane);
    }
  }

  if (cs > 1) cluster.sync(); else __syncthreads();
  const int shift = __ffs(n_parts) - 1;                              // (a power of two)
  auto sums_of = [&](int p, int w, int r) {
    float* to = sums[p & (n_parts - 1)][w][r];
    return cs > 1 ? cluster.map_shared_rank(to, p >> shift) : to;
  };
  // what a warp's sums count, a lane a (part, warp): -1 for one without keys
  if (warp < R) {
    const int p = lane / AR_WARPS;
    const float2 ml = p < a.parts ? *(const float2*)(sums_of(p, lane % AR_WARPS, warp) + HD) : make_float2(-INFINITY, 0.f);
    const bool none = ml.x == -INFINITY && ml.y == 0.f;
    const float M = warp_max(ml.x), f = none ? 0.f : expf(ml.x - M), L = warp_sum(ml.y * f);
    factor[warp][lane] = none ? -1.f : f;
    if (lane == 0) total[warp] = L;
  }
  __syncthreads();
  // every block finishes its share of the elements: four lanes an aligned four of them, a warp's sums each, then an element each
  const int share = R * HD / cs, w = lane & 3;
  for (int x0 = 0; x0 < share; x0 += AR_WARPS * 32) {
    const bool live = x0 + (int)threadIdx.x < share;
    const int x = rank * share + (live ? x0 + (int)threadIdx.x : w);
    const int r = x / HD, e = x - r * HD, h = g * R + r;
    float4 from[AR_PARTS];
    float f[AR_PARTS], o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int p = 0; p < AR_PARTS; ++p) {
      f[p] = factor[r][p * AR_WARPS + w];
      from[p] = !(f[p] < 0.f) ? *(const float4*)(sums_of(p, w, r) + (e & ~3)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int p = 0; p < AR_PARTS; ++p) {
      if (f[p] < 0.f) continue;
      o4[0] = fmaf(from[p].x, f[p], o4[0]); o4[1] = fmaf(from[p].y, f[p], o4[1]);
      o4[2] = fmaf(from[p].z, f[p], o4[2]); o4[3] = fmaf(from[p].w, f[p], o4[3]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float give = (w & 2) ? o4[i] : o4[i + 2], keep = (w & 2) ? o4[i + 2] : o4[i];
      o4[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    const float give = (w & 1) ? o4[0] : o4[1], keep = (w & 1) ? o4[1] : o4[0];
    float o = keep + __shfl_xor_sync(0xffffffffu, give, 1);
    if (!live) continue;
    float inv = 1.0f / total[r];
    if (a.gate) inv *= 1.0f / (1.0f + expf(-a.gate[(size_t)row * a.ldg + h]));
    o *= inv;
    if (a.og) o *= 1.0f / (1.0f + expf(-__bfloat162float(a.og[(size_t)row * a.ldog + (size_t)h * HD + e])));
    a.out[((size_t)row * a.H + h) * HD + e] = __float2bfloat16_rn(o);
  }
  if (cs > 1) cluster.sync();                                        // nobody leaves while its sums are being read
}

// How many clusters of cs blocks the device holds at once (asked once per device and size of the cluster, the shared memory of a block
// following it; 0: not known).
template <int HD, int R, bool VK>
static int ar_resident_clusters(int cs, size_t smem) {
  static int cached[64][AR_PARTS + 1][AR_PARTS + 1];
  const int per = (int)(smem / (AR_WARPS * R * (HD + 4) * sizeof(float)));          // parts a block, 1..8
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || per > AR_PARTS) return 0;
  int& n = cached[dev][cs][per];
  if (!n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs); cfg.blockDim = dim3(AR_WARPS * 32); cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int got = 0;
    if (cudaOccupancyMaxActiveClusters(&got, attention_rows_kernel<HD, R, VK>, &cfg) != cudaSuccess) { cudaGetLastError(); got = 0; }
    n = got + 1;
  }
  return n - 1;
}

template <int HD, int R, bool VK>
static int ar_launch(const ArArgs& a, int T, int cs, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs, a.G, T); cfg.blockDim = dim3(AR_WARPS * 32); cfg.stream = stream;
  cfg.dynamicSmemBytes = (size_t)(a.parts / cs) * AR_WARPS * R * (HD + 4) * sizeof(float);
  if (cfg.dynamicSmemBytes > 40 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(attention_rows_kernel<HD, R, VK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
    if (e != cudaSuccess) return (int)e;
  }
  // A programmatic dependent (four layers with their products, us before / so: two heads a kv head, 1 token 68.8 / 56.6, 24 tokens 148.6 /
  // 128.0; four heads, 1 token 73.6 / 63.3, 12 tokens 94.1 / 91.0), except where its clusters just fill a device that holds two blocks an SM: beside the
  // blocks of the kernel in front not all of them find room, and a second round costs more (values that are keys, 4 tokens, 32 heads, 8
  // kv heads, clusters of 8: 70 / 81 us for four layers).  Blocks an SM matter as much: 12 tokens of four heads a kv head (384 blocks)
  // 86 us with three, 108 with two and more registers; of two heads, 8 tokens, 275 with four and 290 with three.
  const long long clusters = (long long)a.G * T;
  const int fit = ar_resident_clusters<HD, R, VK>(cs, cfg.dynamicSmemBytes);
  const bool full = fit * cs <= 2 * fellm_sm_count() && clusters <= fit && 10 * clusters > 9ll * fit;
  return launch_k_class(full ? 0 : 1, attention_rows_kernel<HD, R, VK>, cfg.gridDim, cfg.blockDim, cfg.dynamicSmemBytes, stream, cs, a);
}

// Rows of q [T, ldq] (heads at column 0, H x hd bfloat16), each at its own position of its own slot; the other arguments as
// fellm_paged_attention_general's, vd 0 (values that are the keys) or hd; og [T, ldog] bfloat16 (null: none): the result times
// its sigmoid, element by element; parts: 1, 2, 4 or 8 shares of a row's keys (the order of its sums), cluster: as many blocks a
// (row, kv head) or fewer.
FELLM_API int fellm_attention_rows(const void* q, const void* pool, const int* block_table, int max_pages, const int* positions,
                                   const int* row_slot, void* out, int T, int H, int G, int hd, int vd, int page_tokens, int layer,
                                   int layers_in_group, float scale, int window, int ldq, float softcap, int chunk, const float* gate,
                                   int ldg, const float* slopes, float qt_coef, int qt_every, int new_k_off, int new_v_off, int* status,
                                   const void* og, int ldog, int parts, int cluster, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!q || !pool || !block_table || !positions || !row_slot || !out) return FELLM_ERR_ARG;
  if (G < 1 || H % G || (hd != 64 && hd != 128) || (vd && vd != hd) || T > 65535 || G > 65535) return FELLM_ERR_SIZE;
  const int R = H / G;
  if ((R != 1 && R != 2 && R != 4) || page_tokens < 1 || (page_tokens & (page_tokens - 1))) return FELLM_ERR_SIZE;
  if ((parts != 1 && parts != 2 && parts != 4 && parts != AR_PARTS) || cluster < 1 || cluster > parts || parts % cluster) return FELLM_ERR_ARG;
  if ((((uintptr_t)q | (uintptr_t)pool) & 15) || (ldq & 7) || (new_k_off >= 0 && ((new_k_off & 7) || (vd && (new_v_off & 7))))) return FELLM_ERR_SIZE;
  ArArgs a;
  a.q = (const bf16*)q; a.pool = (const bf16*)pool; a.block_table = block_table; a.positions = positions; a.row_slot = row_slot;
  a.out = (bf16*)out; a.status = status; a.gate = gate; a.slopes = slopes; a.og = (const bf16*)og;
  a.parts = parts; a.ldq = ldq; a.max_pages = max_pages; a.H = H; a.G = G; a.layer = layer; a.layers_in_group = layers_in_group;
  a.window = window; a.chunk = chunk; a.ldg = ldg; a.ldog = ldog; a.qt_every = qt_every; a.new_k_off = new_k_off; a.new_v_off = new_v_off;
  a.scale = scale; a.softcap = softcap; a.qt_coef = qt_coef;
  a.page_shift = 0;
  while ((1 << a.page_shift) < page_tokens) ++a.page_shift;
#define AR_R(HD_, VK_) (R == 1 ? ar_launch<HD_, 1, VK_>(a, T, cluster, stream) : R == 2 ? ar_launch<HD_, 2, VK_>(a, T, cluster, stream) \
                      : ar_launch<HD_, 4, VK_>(a, T, cluster, stream))
  if (hd == 64) return vd ? AR_R(64, false) : AR_R(64, true);
  return vd ? AR_R(128, false) : AR_R(128, true);
#undef AR_R
}
