// Latent attention over the paged cache on tensor cores (mma.sync.m16n8k16, ldmatrix, cp.async): bfloat16 queries and
// cache rows, float32 scores, softmax and sums.  Compiled for one pair of sizes: -DLAT_RK (the latent, a multiple of
// 32 up to 512) and -DLAT_DR (the rotated key part; LAT_RK + LAT_DR a multiple of 16).
//
// A token's cache row is [c (RK) | rotated key part (DR)], one for all heads; a query row is [W_uk,h^T qn (RK) |
// rotated qr (DR)] per (token, head).  score = scale (query . row); the value of a key is the first RK elements of
// its row.  So all H heads of a token are rows of ONE product against the same keys.  Two kernels:
//
// Portions of prompts (latent_attention_kernel): a CTA takes MQ = 16 NG consecutive (token, head) rows of one item, walks
// the keys its rows can see in tiles of KT = 16 NC through a two-stage cp.async ring, and its NG x NC warps split a tile two
// ways: warp (i, j) computes the scores of row group i against keys [16 j, 16 j + 16) of the tile and leaves them in shared
// memory; after a barrier it reads its group's scores for the whole tile, does the online softmax for them (the NC warps of
// a group do the same arithmetic and hold the same m and l), and adds P V for the value elements [j RK / NC,
// (j + 1) RK / NC), which it alone accumulates: a row's read-out of RK float32 sums lies across NC warps' registers.  NG = 4,
// NC = 2: 64 rows, key tiles of 32.
//
// Single tokens (latent_tokens_kernel): 16 rows (the heads of a token) and a share of their keys, whole tiles, a CTA of eight warps;
// tiles of 64 keys, of 32 where the latent is no multiple of 64.  A warp makes the scores of eight keys, a thread the probabilities of
// four (16 threads a row), a warp the sums of an eighth of the value elements.  Few shares are a cluster, whose sums stay in shared memory and are
// put together through distributed shared memory, every CTA its part of the elements.  More shares (long contexts of few requests), or
// clusters that the device does not hold at once, leave (m, l, sums) in a scratch buffer that latent_merge_kernel puts
// together (a block a row: 8 x the parallelism of a merge by the CTA that finishes last, which was tried and cost 40 us a
// layer).  Which of the two runs is not in the bits: the shares, and every sum's order, are the same.  Index arrays and cache rows are read
// ahead of the wait for the kernel in front: see the kernel.
// Bound by: latency, of the index arrays, of the keys, of the chains of a tile (tiles by four warps that each did the softmax of all
// rows took 6,700 instructions a warp).  8 tokens of 8 heads over 1,024 keys of 1,152 bytes with the product in front: four warps and a merge
// 18.7 us, here 12.8 (1 token over 100 keys 15.1 -> 9.9, 48 tokens over 1,024 32.3 -> 27.3).  Shares in portions of 16 keys, and scores as the
// sum of two chains of MMAs, take 12.1 and 8.0 us; they round otherwise, and a row's bits then depend on how the shares are put together.
//
// A key counts for the row of a token at position p iff p - window < key <= p (window 0: every key up to p).  A
// sink per head joins the denominator once: exp(sink_h), not scaled, no value.  Rows of an item have consecutive
// positions; key tiles start at multiples of KT, so a tile lies in one page (page_tokens % KT == 0).
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

#ifndef LAT_RK
#define LAT_RK 512
#endif
#ifndef LAT_DR
#define LAT_DR 64
#endif

constexpr int RK = LAT_RK, DR = LAT_DR, D = RK + DR;
static_assert(RK % 32 == 0 && RK >= 32 && RK <= 512 && DR >= 0 && D % 16 == 0, "latent sizes the tensor-core kernel takes");
constexpr int CPR = D / 8;                          // 16-byte chunks per row
constexpr bool SWZ = (CPR % 8 == 0);                // rows of whole 128-byte lines: XOR swizzle
constexpr int ROWB = D * 2 + (SWZ ? 0 : 16);        // else 16 bytes of padding spread the banks
constexpr int KS = D / 16;                          // k16 steps over a row
constexpr float LOG2E = 1.4426950408889634f;
constexpr int MAX_SPLITS = 32;                     // ranges a single token's key walk is split into, at most

__device__ __forceinline__ int tile_off(int row, int chunk) {
  return row * ROWB + ((SWZ ? (chunk ^ (row & 7)) : chunk) << 4);
}
__device__ __forceinline__ void cp_async16(unsigned smem_addr, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr), "l"(gmem));
}
__device__ __forceinline__ void st_shared_zero16(unsigned smem_addr) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};\n" ::"r"(smem_addr), "r"(0u));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }
__device__ __forceinline__ void ldsm_x4(unsigned* r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(unsigned* r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float* d, const unsigned* a, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *(unsigned*)&v;
}

struct LatArgs {
  const bf16* q;            // [rows of all items][H][D]; with qsrc: [rows][H][RK], the rotated part comes from qsrc
  const bf16* qsrc;         // or null: [rows][ldq], head h's rotated part (DR elements, not yet rotated) at column h q_head + q_rot_off
  int ldq, q_head, q_rot_off, n_rot;
  const float* freq; float mag;      // pairs (2i, 2i + 1), i < n_rot / 2: angle = float(position) freq[i], cos and sin times mag
  const bf16* pool;         // [pages][layers_in_group][page_tokens][D]
  const int* block_table; int max_pages;
  const int* positions; const int* row_slot; const int* item_start;
  bf16* out;                // [rows][H][RK]
  float* scratch;           // n_splits > 1 and no cluster: [rows * H][n_splits][RK + 2]
  const float* sinks;       // [H] or null
  int H, page_tokens, layer, layers_in_group, window, n_splits, cluster, single;       // single: every item is one token
  int ready;                // the index arrays and the cache are complete before the kernel in front ends: see latent_tokens_kernel
  float scale_log2;
};

template <int NG, int NC>
__global__ void __launch_bounds__(NG * NC * 32, 1) latent_attention_kernel(LatArgs a) {
  constexpr int KT = 16 * NC, MQ = 16 * NG, NTH = NG * NC * 32, DVW = RK / NC, NT = DVW / 8, SLD = KT + 8, KK = KT / 16;
  static_assert(DVW % 16 == 0, "a warp's share of the value elements is a multiple of 16");
  extern __shared__ __align__(128) unsigned char smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wi = warp / NC, wj = warp % NC, g = lane >> 2, c = lane & 3;
  const int item = blockIdx.y, H = a.H;
  const int r_begin = a.item_start[item];
  const int n_rows = (a.item_start[item + 1] - r_begin) * H;
  // (an item's last rows see the most keys: their CTAs start first, the short walks of its first rows fill the tail)
  const int R0 = (int)(gridDim.x - 1 - blockIdx.x) * MQ;
  if (R0 >= n_rows) return;
  const int rows_here = min(MQ, n_rows - R0);
  const int pos0 = a.positions[r_begin];
  const int* bt = a.block_table + (size_t)a.row_slot[r_begin] * a.max_pages;
  const int pos_lo = pos0 + R0 / H, pos_hi = pos0 + (R0 + rows_here - 1) / H;
  int key_begin = a.window > 0 ? max(0, pos_lo - a.window + 1) : 0;
  key_begin &= ~(KT - 1);
  const int n_tiles = (pos_hi + 1 - key_begin + KT - 1) / KT;

  const unsigned q_s = (unsigned)__cvta_generic_to_shared(smem), k_s = q_s + MQ * ROWB;
  float* S_s = (float*)(smem + (MQ + 2 * KT) * ROWB);

  // the CTA's query rows (rows beyond the item's end are zeros)
  {
    const int q_ld = a.qsrc ? RK : D;
    const bf16* qg = a.q + ((size_t)r_begin * H + R0) * q_ld;
    for (int ch = tid; ch < MQ * CPR; ch += NTH) {
      const int r = ch / CPR, cc = ch - r * CPR;
      if (r >= rows_here) st_shared_zero16(q_s + tile_off(r, cc));
      else if (cc < RK / 8 || !a.qsrc) cp_async16(q_s + tile_off(r, cc), qg + (size_t)r * q_ld + cc * 8);
      else {
        // eight elements of the head's rotated part, rotated by the row's position on their way in
        const int R = R0 + r, t = R / H, h = R - t * H, e0 = (cc - RK / 8) * 8;
        uint4 raw = *(const uint4*)(a.qsrc + (size_t)(r_begin + t) * a.ldq + (size_t)h * a.q_head + a.q_rot_off + e0);
        __nv_bfloat162* pr = (__nv_bfloat162*)&raw;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (e0 + 2 * i < a.n_rot) {
            float2 uv = __bfloat1622float2(pr[i]);
            float sn, cs;
            sincosf((float)(pos0 + t) * a.freq[(e0 >> 1) + i], &sn, &cs);
            sn *= a.mag; cs *= a.mag;
            pr[i] = __floats2bfloat162_rn(uv.x * cs - uv.y * sn, uv.y * cs + uv.x * sn);
          }
        }
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(q_s + tile_off(r, cc)), "r"(raw.x), "r"(raw.y), "r"(raw.z), "r"(raw.w));
      }
    }
  }
  // keys beyond the last visible one are zeros: they are masked, but a value of a freed page's bits must not
  // reach a product (0 * NaN)
  auto load_tile = [&](int t, int buf) {
    const int k0 = key_begin + t * KT;
    const int page = max(bt[k0 / a.page_tokens], 0);
    const bf16* src = a.pool + (((size_t)page * a.layers_in_group + a.layer) * a.page_tokens + (k0 % a.page_tokens)) * D;
    const unsigned dst = k_s + buf * KT * ROWB;
    const int n_keys = min(KT, pos_hi + 1 - k0);
    for (int ch = tid; ch < KT * CPR; ch += NTH) {
      const int r = ch / CPR, cc = ch - r * CPR;
      if (r < n_keys) cp_async16(dst + tile_off(r, cc), src + (size_t)r * D + cc * 8);
      else st_shared_zero16(dst + tile_off(r, cc));
    }
  };

  // rows g and g + 8 of the warp's group
  const int Rg0 = R0 + wi * 16 + g, Rg1 = Rg0 + 8;
  const int hi0 = pos0 + min(Rg0, n_rows - 1) / H, hi1 = pos0 + min(Rg1, n_rows - 1) / H;
  const int lo0 = a.window > 0 ? hi0 - a.window + 1 : 0, lo1 = a.window > 0 ? hi1 - a.window + 1 : 0;
  const int grp_lo = pos0 + min(R0 + wi * 16, n_rows - 1) / H, grp_hi = pos0 + min(R0 + wi * 16 + 15, n_rows - 1) / H;
  const int grp_first = a.window > 0 ? grp_lo - a.window + 1 : 0;

  float o[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;

  load_tile(0, 0);
  cp_async_commit();
  for (int t = 0; t < n_tiles; ++t) {
    const int buf = t & 1;
    cp_async_wait_all();
    __syncthreads();                   // tile t has landed; everyone is done with the other buffer and with S_s
    if (t + 1 < n_tiles) load_tile(t + 1, buf ^ 1);
    cp_async_commit();
    const int k0 = key_begin + t * KT;
    const bool live = k0 <= grp_hi && k0 + KT - 1 >= grp_first;        // some row of the group sees some key of the tile
    const unsigned kb = k_s + buf * KT * ROWB;
    if (live) {
      float s[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll 6
      for (int ks = 0; ks < KS; ++ks) {
        unsigned af[4], bq[4];
        ldsm_x4(af, q_s + tile_off(wi * 16 + (lane & 15), 2 * ks + (lane >> 4)));
        ldsm_x4(bq, kb + tile_off(wj * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * ks + ((lane >> 3) & 1)));
        mma16816(s[0], af, bq[0], bq[1]);
        mma16816(s[1], af, bq[2], bq[3]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float* d0 = S_s + (wi * 16 + g) * SLD + wj * 16 + 8 * i + 2 * c;
        *(float2*)d0 = make_float2(s[i][0], s[i][1]);
        *(float2*)(d0 + 8 * SLD) = make_float2(s[i][2], s[i][3]);
      }
    }
    __syncthreads();
    if (!live) continue;
    // the group's scores for the whole tile, in the layout of the P V product's first operand
    float p0[KK][4], p1[KK][4];
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) {
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int col = 16 * kk + 8 * hf + 2 * c;
        const float2 v0 = *(const float2*)(S_s + (wi * 16 + g) * SLD + col);
        const float2 v1 = *(const float2*)(S_s + (wi * 16 + g + 8) * SLD + col);
        const int kj = k0 + col;
        p0[kk][2 * hf] = (kj <= hi0 && kj >= lo0) ? v0.x * a.scale_log2 : -INFINITY;
        p0[kk][2 * hf + 1] = (kj + 1 <= hi0 && kj + 1 >= lo0) ? v0.y * a.scale_log2 : -INFINITY;
        p1[kk][2 * hf] = (kj <= hi1 && kj >= lo1) ? v1.x * a.scale_log2 : -INFINITY;
        p1[kk][2 * hf + 1] = (kj + 1 <= hi1 && kj + 1 >= lo1) ? v1.y * a.scale_log2 : -INFINITY;
        mx0 = fmaxf(mx0, fmaxf(p0[kk][2 * hf], p0[kk][2 * hf + 1]));
        mx1 = fmaxf(mx1, fmaxf(p1[kk][2 * hf], p1[kk][2 * hf + 1]));
      }
    }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
    const float mu0 = mn0 == -INFINITY ? 0.f : mn0, mu1 = mn1 == -INFINITY ? 0.f : mn1;      // a row that has seen nothing yet
    const float corr0 = exp2f(m0 - mu0), corr1 = exp2f(m1 - mu1);
    m0 = mn0; m1 = mn1;
    float sum0 = 0.f, sum1 = 0.f;
    unsigned pa[KK][4];
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        p0[kk][e] = exp2f(p0[kk][e] - mu0); sum0 += p0[kk][e];
        p1[kk][e] = exp2f(p1[kk][e] - mu1); sum1 += p1[kk][e];
      }
      pa[kk][0] = pack_bf16(p0[kk][0], p0[kk][1]); pa[kk][1] = pack_bf16(p1[kk][0], p1[kk][1]);
      pa[kk][2] = pack_bf16(p0[kk][2], p0[kk][3]); pa[kk][3] = pack_bf16(p1[kk][2], p1[kk][3]);
    }
    l0 = l0 * corr0 + sum0; l1 = l1 * corr1 + sum1;
#pragma unroll
    for (int n = 0; n < NT; ++n) { o[n][0] *= corr0; o[n][1] *= corr0; o[n][2] *= corr1; o[n][3] *= corr1; }
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) {
#pragma unroll
      for (int n2 = 0; n2 < NT / 2; ++n2) {
        unsigned vb[4];
        ldsm_x4_trans(vb, kb + tile_off(16 * kk + (lane & 7) + (((lane >> 3) & 1) << 3), wj * (DVW / 8) + 2 * n2 + (lane >> 4)));
        mma16816(o[2 * n2], pa[kk], vb[0], vb[1]);
        mma16816(o[2 * n2 + 1], pa[kk], vb[2], vb[3]);
      }
    }
  }
  cp_async_wait_all();

  l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const size_t row_g0 = (size_t)r_begin * H + Rg0;         // the (token, head) row among all rows of the step
  if (a.sinks) {
    l0 += exp2f(a.sinks[Rg0 % H] * LOG2E - m0);
    l1 += exp2f(a.sinks[Rg1 % H] * LOG2E - m1);
  }
  const float inv0 = 1.0f / l0, inv1 = 1.0f / l1;
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int col = wj * DVW + 8 * n + 2 * c;
    if (Rg0 < n_rows) *(__nv_bfloat162*)(a.out + row_g0 * RK + col) = __floats2bfloat162_rn(o[n][0] * inv0, o[n][1] * inv0);
    if (Rg1 < n_rows) *(__nv_bfloat162*)(a.out + (row_g0 + 8) * RK + col) = __floats2bfloat162_rn(o[n][2] * inv1, o[n][3] * inv1);
  }
}

// ---------------------------------------------------------------- single tokens
constexpr int LT_WARPS = 8, LT_KT = RK % 64 == 0 ? 64 : 32, LT_ROWS = 16, LT_MAX_CLUSTER = 16;
constexpr int LT_SLD = LT_KT + 4, LT_PLD = LT_KT + 8;        // row strides of the scores (float32) and the probabilities (bfloat16)
constexpr int LT_OLD = RK + 4;                               // and of the sums that a cluster puts together
constexpr int LT_GROUPS = (RK / 16 + LT_WARPS - 1) / LT_WARPS;                // 16 value elements each, a warp's: warp, warp + 8, ..
constexpr size_t LT_KEYS = (size_t)2 * LT_KT * ROWB;
constexpr size_t LT_SUMS = (size_t)LT_ROWS * LT_OLD * sizeof(float);
constexpr size_t LT_SMEM = LT_ROWS * ROWB + (LT_KEYS > LT_SUMS ? LT_KEYS : LT_SUMS);

__global__ void __launch_bounds__(LT_WARPS * 32, 1) latent_tokens_kernel(LatArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(16) float S_s[LT_ROWS * LT_SLD];
  __shared__ __align__(16) bf16 P_s[LT_ROWS * LT_PLD];
  __shared__ float corr_s[LT_ROWS];
  __shared__ float2 ml_s[LT_ROWS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3, H = a.H;
  const int rank = blockIdx.x, item = blockIdx.y, R0 = blockIdx.z * LT_ROWS;
  pdl_launch_dependents();
  // With `ready` launched as a programmatic dependent, and what the caller vouches for is read ahead of the wait: a kernel launched the
  // ordinary way (the product that makes q) lies between this one and whatever wrote the index arrays and the cache with this
  // step's own rows, and it started when those had ended.  Only q is waited for.
  if (!a.ready) pdl_wait();
  const int r_begin = a.single ? item : a.item_start[item], n_rows = a.single ? H : (a.item_start[item + 1] - r_begin) * H;
  if (R0 >= n_rows) { pdl_wait(); return; }        // (the same for a whole cluster)
  const int rows_here = min(LT_ROWS, n_rows - R0), pos0 = a.positions[r_begin];
  const int* bt = a.block_table + (size_t)a.row_slot[r_begin] * a.max_pages;
  auto token_of = [&](int R) { return a.single ? 0 : R / H; };                  // which of the item's tokens a row belongs to
  const int pos_lo = pos0 + token_of(R0), pos_hi = pos0 + token_of(R0 + rows_here - 1);
  // this CTA's share of the keys, whole tiles
  int key_begin = (a.window > 0 ? max(0, pos_lo - a.window + 1) : 0) & ~(LT_KT - 1);
  const int all = (pos_hi + 1 - key_begin + LT_KT - 1) / LT_KT, per = (all + a.n_splits - 1) / a.n_splits;
  const int n_tiles = max(0, min(per, all - rank * per));
  key_begin += LT_KT * rank * per;
  const int key_end = min(pos_hi + 1, key_begin + LT_KT * n_tiles);

  const unsigned q_s = (unsigned)__cvta_generic_to_shared(smem), k_s = q_s + LT_ROWS * ROWB;
  // A tile's portions with a key, two warps each, eight rows a warp: 16 keys lie in one page, so a warp looks one page up and its
  // rows lie behind one another.  Keys beyond the last visible one are zeros: they are masked, but a value of a freed page's
  // bits must not reach a product (0 * NaN).
  auto rows_of = [&](int t) {                      // this warp's eight rows of a tile (an address without keys is not read)
    const int k0 = min(key_begin + t * LT_KT + 16 * (warp >> 1), max(key_end - 1, 0)) & ~15;
    const int page = max(bt[k0 / a.page_tokens], 0);             // an unmapped entry (-1) must never become an address
    return a.pool + (((size_t)page * a.layers_in_group + a.layer) * a.page_tokens + (k0 % a.page_tokens + 8 * (warp & 1))) * D;
  };
  auto load_tile = [&](int t, const bf16* src) {
    const int at = 16 * (warp >> 1) + 8 * (warp & 1), n_keys = key_end - (key_begin + t * LT_KT) - at;
    if (at < LT_KT && n_keys + 8 * (warp & 1) > 0) {             // (the portion has a key)
      const unsigned dst = k_s + (t & 1) * LT_KT * ROWB;
#pragma unroll
      for (int i = 0; i < (8 * CPR + 31) / 32; ++i) {
        const int ch = lane + 32 * i, r = ch / CPR;
        if (8 * CPR % 32 && r >= 8) break;
        if (r < n_keys) cp_async16(dst + tile_off(at + r, ch - r * CPR), src + ch * 8);
        else st_shared_zero16(dst + tile_off(at + r, ch - r * CPR));
      }
    }
    cp_async_commit();
  };
  if (n_tiles > 0) {
    const bf16 *first = rows_of(0), *second = rows_of(1);
    load_tile(0, first);
    if (n_tiles > 1) load_tile(1, second);
  }
  // the rotated part's pairs (a thread's PAIRS): their angles do not wait either
  constexpr int PAIRS = (LT_ROWS * DR / 2 + LT_WARPS * 32 - 1) / (LT_WARPS * 32), HALF = DR / 2 > 0 ? DR / 2 : 1;
  float sn[PAIRS > 0 ? PAIRS : 1], cs[PAIRS > 0 ? PAIRS : 1];
  if (a.qsrc) {
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
      const int x = tid + LT_WARPS * 32 * i, r = x / HALF, p = x % HALF;
      sn[i] = 0.f; cs[i] = 1.f;
      if (r < rows_here && 2 * p < a.n_rot) {
        sincosf((float)(pos0 + token_of(R0 + r)) * a.freq[p], &sn[i], &cs[i]);
        sn[i] *= a.mag; cs[i] *= a.mag;
      }
    }
  }
  pdl_wait();
  // the query rows (rows beyond the item's end are zeros)
  {
    const int q_ld = a.qsrc ? RK : D, chunks = q_ld / 8;
    const bf16* qg = a.q + ((size_t)r_begin * H + R0) * q_ld;
    for (int r = warp; r < LT_ROWS; r += LT_WARPS)
      for (int cc = lane; cc < chunks; cc += 32) {
        if (r < rows_here) cp_async16(q_s + tile_off(r, cc), qg + (size_t)r * q_ld + cc * 8);
        else st_shared_zero16(q_s + tile_off(r, cc));
      }
    if (a.qsrc) {
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) {
        const int x = tid + LT_WARPS * 32 * i, r = x / HALF, p = x % HALF;
        if (r >= LT_ROWS) break;
        __nv_bfloat162 v = __floats2bfloat162_rn(0.f, 0.f);
        if (r < rows_here) {
          const int t = token_of(R0 + r), h = R0 + r - t * H;
          v = *(const __nv_bfloat162*)(a.qsrc + (size_t)(r_begin + t) * a.ldq + (size_t)h * a.q_head + a.q_rot_off + 2 * p);
          if (2 * p < a.n_rot) {
            const float2 uv = __bfloat1622float2(v);
            v = __floats2bfloat162_rn(uv.x * cs[i] - uv.y * sn[i], uv.y * cs[i] + uv.x * sn[i]);
          }
        }
        asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(q_s + tile_off(r, RK / 8 + p / 4) + 4 * (p % 4)), "r"(*(const unsigned*)&v));
      }
    }
    cp_async_commit();
  }
  // a thread's row and four keys of the softmax: 16 threads a row, keys 16 sp + sk and sk + 8 and the ones behind them, as a lane of an
  // MMA's first operand holds them
  const int sr = tid >> 4, sp = (tid >> 2) & 3, sk = 16 * sp + 2 * (tid & 3);
  const bool has_keys = sp < LT_KT / 16;
  const int hi = pos0 + token_of(min(R0 + sr, n_rows - 1)), lo = a.window > 0 ? hi - a.window + 1 : 0;
  float m = -INFINITY, l = 0.f;
  float o[LT_GROUPS][2][4];
#pragma unroll
  for (int i = 0; i < LT_GROUPS; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) o[i][j][0] = o[i][j][1] = o[i][j][2] = o[i][j][3] = 0.f;

  for (int t = 0; t < n_tiles; ++t) {
    if (t > 0 && t + 1 < n_tiles) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    else cp_async_wait_all();
    __syncthreads();                   // the tile and q are here
    const int k0 = key_begin + t * LT_KT, n16 = min(LT_KT / 16, (key_end - k0 + 15) / 16);
    const unsigned kb = k_s + (t & 1) * LT_KT * ROWB;
    if (warp < 2 * n16) {
      // scores of keys 8 warp .. + 8, one chain of MMAs: two steps of 16 elements a load of theirs
      float s[4] = {};
      const unsigned krow = 8 * warp + (lane & 7);
#pragma unroll 6
      for (int ks = 0; ks < KS / 2; ++ks) {
        unsigned a0[4], a1[4], b[4];
        ldsm_x4(a0, q_s + tile_off(lane & 15, 4 * ks + (lane >> 4)));
        ldsm_x4(a1, q_s + tile_off(lane & 15, 4 * ks + 2 + (lane >> 4)));
        ldsm_x4(b, kb + tile_off(krow, 4 * ks + (lane >> 3)));
        mma16816(s, a0, b[0], b[1]);
        mma16816(s, a1, b[2], b[3]);
      }
      if (KS & 1) {
        unsigned a0[4], b[4];
        ldsm_x4(a0, q_s + tile_off(lane & 15, 2 * (KS - 1) + (lane >> 4)));
        ldsm_x4(b, kb + tile_off(krow, 2 * (KS - 1) + ((lane >> 3) & 1)));        // (the last two matrices: the first two once more)
        mma16816(s, a0, b[0], b[1]);
      }
      float* to = S_s + g * LT_SLD + 8 * warp + 2 * c;
      *(float2*)to = make_float2(s[0], s[1]);
      *(float2*)(to + 8 * LT_SLD) = make_float2(s[2], s[3]);
    }
    __syncthreads();
    {
      float x[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (has_keys) {
        const float2 lo2 = *(const float2*)(S_s + sr * LT_SLD + sk), hi2 = *(const float2*)(S_s + sr * LT_SLD + sk + 8);
        const float raw[4] = {lo2.x, lo2.y, hi2.x, hi2.y};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int kj = k0 + sk + (e & 1) + 8 * (e >> 1);
          if (kj <= hi && kj >= lo) x[e] = raw[e] * a.scale_log2;
        }
      }
      float mx = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
      const float mn = fmaxf(m, mx), mu = mn == -INFINITY ? 0.f : mn;              // (a row that has seen nothing yet)
      const float corr = exp2f(m - mu);
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = exp2f(x[e] - mu);
      // a tile's sum, portion after portion of four threads' keys: the last portion's threads have it
      float sum = 0.f;
#pragma unroll
      for (int p = 0; p < LT_KT / 16; ++p) {
        const float before = p ? __shfl_sync(0xffffffffu, sum, (lane & 16) | (4 * (p - 1)) | (lane & 3)) : 0.f;
        if (sp == p) sum = (((before + x[0]) + x[1]) + x[2]) + x[3];
      }
      l = l * corr + sum;
      m = mn;
      if (has_keys) {
        *(unsigned*)(P_s + sr * LT_PLD + sk) = pack_bf16(x[0], x[1]);
        *(unsigned*)(P_s + sr * LT_PLD + sk + 8) = pack_bf16(x[2], x[3]);
      }
      if ((tid & 15) == 0) corr_s[sr] = corr;
    }
    __syncthreads();
    const float corr0 = corr_s[g], corr1 = corr_s[g + 8];
#pragma unroll
    for (int i = 0; i < LT_GROUPS; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) { o[i][j][0] *= corr0; o[i][j][1] *= corr0; o[i][j][2] *= corr1; o[i][j][3] *= corr1; }
#pragma unroll
    for (int kk = 0; kk < LT_KT / 16; ++kk) {
      if (kk >= n16) break;
      unsigned pa[4];
      ldsm_x4(pa, (unsigned)__cvta_generic_to_shared(P_s + (lane & 15) * LT_PLD + 16 * kk + 8 * (lane >> 4)));
#pragma unroll
      for (int i = 0; i < LT_GROUPS; ++i) {
        const int grp = warp + LT_WARPS * i;
        if ((RK / 16) % LT_WARPS && grp >= RK / 16) break;
        unsigned vb[4];
        ldsm_x4_trans(vb, kb + tile_off(16 * kk + (lane & 15), 2 * grp + (lane >> 4)));
        mma16816(o[i][0], pa, vb[0], vb[1]);
        mma16816(o[i][1], pa, vb[2], vb[3]);
      }
    }
    if (t + 2 < n_tiles) {
      const bf16* src = rows_of(t + 2);
      __syncthreads();                 // everyone is done with the tile
      load_tile(t + 2, src);
    }
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1); l += __shfl_xor_sync(0xffffffffu, l, 2);
  cp_async_wait_all();
  __syncthreads();                     // (the keys' place is free; P_s and corr_s are read)
  const size_t row_g = (size_t)r_begin * H + R0;
  const bool apart = a.n_splits > 1 && !a.cluster;
  // the rows' sums, in shared memory for the cluster (in the keys' place) or in the scratch buffer
  float* const os = (float*)(smem + LT_ROWS * ROWB);
#pragma unroll
  for (int i = 0; i < LT_GROUPS; ++i) {
    const int grp = warp + LT_WARPS * i;
    if ((RK / 16) % LT_WARPS && grp >= RK / 16) break;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int col = 16 * grp + 8 * j + 2 * c;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = g + 8 * e;
        const float2 v = make_float2(o[i][j][2 * e], o[i][j][2 * e + 1]);
        if (!apart) *(float2*)(os + r * LT_OLD + col) = v;
        else if (r < rows_here) *(float2*)(a.scratch + ((row_g + r) * a.n_splits + rank) * (RK + 2) + col) = v;
      }
    }
  }
  if ((tid & 15) == 4 * (LT_KT / 16 - 1)) {
    if (!apart) ml_s[sr] = make_float2(m, l);
    else if (sr < rows_here) *(float2*)(a.scratch + ((row_g + sr) * a.n_splits + rank) * (RK + 2) + RK) = make_float2(m, l);
  }
  if (apart) return;
  cg::cluster_group cluster = cg::this_cluster();
  const int n = a.n_splits;
  if (n > 1) cluster.sync(); else __syncthreads();
  // every CTA a share of the elements, four a thread
  const int total = rows_here * (RK / 4), share = (total + n - 1) / n, end = min(total, (rank + 1) * share);
  for (int x = rank * share + tid; x < end; x += LT_WARPS * 32) {
    const int r = x / (RK / 4), col = 4 * (x - r * (RK / 4));
    float2 ml[LT_MAX_CLUSTER];
    float4 v[8];
    auto sums_of = [&](int q) { return *(const float4*)(cluster.map_shared_rank(os, q) + r * LT_OLD + col); };
#pragma unroll
    for (int q = 0; q < LT_MAX_CLUSTER; ++q) if (q < n) ml[q] = *(const float2*)(cluster.map_shared_rank(ml_s, q) + r);
#pragma unroll
    for (int q = 0; q < 8; ++q) if (q < n) v[q] = sums_of(q);
    float M = -INFINITY, L = 0.f;
#pragma unroll
    for (int q = 0; q < LT_MAX_CLUSTER; ++q) if (q < n) M = fmaxf(M, ml[q].x);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < LT_MAX_CLUSTER; ++q)
      if (q < n) {
        // as latent_merge_kernel (a share without a visible key counts nothing; the only share counts as it is)
        const bool counts = n == 1 || ml[q].x > -INFINITY;
        const float w = n == 1 ? 1.f : counts ? exp2f(ml[q].x - M) : 0.f;
        if (counts) L = __fadd_rn(L, __fmul_rn(ml[q].y, w));
        const float4 o = q < 8 ? v[q & 7] : sums_of(q);
        acc.x = fmaf(o.x, w, acc.x); acc.y = fmaf(o.y, w, acc.y); acc.z = fmaf(o.z, w, acc.z); acc.w = fmaf(o.w, w, acc.w);
      }
    if (a.sinks) L += exp2f(a.sinks[(R0 + r) % H] * LOG2E - M);
    const float inv = 1.0f / L;
    *(uint2*)(a.out + (row_g + r) * RK + col) = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
  }
  if (n > 1) cluster.sync();                       // nobody leaves while its sums are being read
}

// The ranges of a split key walk put together, in the order of the ranges: out = sum_s O_s 2^(m_s - m) / (sum_s l_s
// 2^(m_s - m) + 2^(sink - m)), m = max_s m_s.  A block per (token, head) row.
__global__ void __launch_bounds__(256) latent_merge_kernel(const float* scratch, bf16* __restrict__ out,
                                                           const float* __restrict__ sinks, int H, int n_splits) {
  __shared__ float sm_m[MAX_SPLITS], sm_w[MAX_SPLITS];
  pdl_launch_dependents();
  pdl_wait();
  const size_t row = blockIdx.x;
  const float* base = scratch + row * n_splits * (RK + 2);
  if (threadIdx.x < n_splits) {                    // every range's (m, l) at once
    sm_m[threadIdx.x] = base[(size_t)threadIdx.x * (RK + 2) + RK];
    sm_w[threadIdx.x] = base[(size_t)threadIdx.x * (RK + 2) + RK + 1];
  }
  __syncthreads();
  float m = -INFINITY;
  for (int s = 0; s < n_splits; ++s) m = fmaxf(m, sm_m[s]);
  float L = 0.f;
  for (int s = 0; s < n_splits; ++s) if (sm_m[s] > -INFINITY) L = __fadd_rn(L, __fmul_rn(sm_w[s], exp2f(sm_m[s] - m)));      // (as a cluster adds them)
  if (sinks) L += exp2f(sinks[row % H] * LOG2E - m);
  const float inv = 1.0f / L;
  __syncthreads();
  if (threadIdx.x < n_splits) sm_w[threadIdx.x] = sm_m[threadIdx.x] > -INFINITY ? exp2f(sm_m[threadIdx.x] - m) : 0.f;
  __syncthreads();
  const int e = 2 * threadIdx.x;                   // RK / 2 threads: two neighbouring elements each, all ranges asked for at once
  if (e < RK) {
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 16
    for (int s = 0; s < n_splits; ++s) {
      const float2 v = *(const float2*)(base + (size_t)s * (RK + 2) + e);
      acc.x = fmaf(v.x, sm_w[s], acc.x); acc.y = fmaf(v.y, sm_w[s], acc.y);
    }
    *(__nv_bfloat162*)(out + row * RK + e) = __floats2bfloat162_rn(acc.x * inv, acc.y * inv);
  }
}

template <int NG, int NC>
static int launch_latent(const LatArgs& a, int n_items, int max_item_rows, int rows_total, cudaStream_t stream) {
  constexpr int KT = 16 * NC, MQ = 16 * NG;
  if (a.page_tokens % KT) return FELLM_ERR_SIZE;
  const size_t smem = (size_t)(MQ + 2 * KT) * ROWB + (size_t)MQ * (KT + 8) * sizeof(float);
  auto kern = latent_attention_kernel<NG, NC>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  dim3 grid(ceil_div(max_item_rows * a.H, MQ), n_items, 1);
  return launch_k_class(launch_class_for_rows(rows_total, 0), kern, grid, dim3(NG * NC * 32), smem, stream, 1, a);
}

static int launch_tokens(const LatArgs& a, int n_items, int max_item_rows, int rows_total, cudaStream_t stream) {
  if (a.page_tokens % LT_KT) return FELLM_ERR_SIZE;
  cudaError_t e = cudaFuncSetAttribute(latent_tokens_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LT_SMEM);
  if (e == cudaSuccess && a.cluster && a.n_splits > 8) e = cudaFuncSetAttribute(latent_tokens_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return (int)e;
  dim3 grid(a.n_splits, n_items, ceil_div(max_item_rows * a.H, LT_ROWS));
  int rc = launch_k_class(a.ready ? 1 : launch_class_for_rows(rows_total, 0), latent_tokens_kernel, grid, dim3(LT_WARPS * 32), LT_SMEM, stream, a.cluster ? a.n_splits : 1, a);
  if (rc || a.n_splits == 1 || a.cluster) return rc;
  return launch_k_class(launch_class_for_rows(rows_total, 0), latent_merge_kernel, dim3(rows_total * a.H), dim3(RK / 2 < 32 ? 32 : RK / 2), 0, stream, 1,
                        (const float*)a.scratch, a.out, a.sinks, a.H, a.n_splits);
}

// How many clusters of `size` CTAs of the single tokens' kernel the device holds at once (asked once per device and size; 0: none).
FELLM_API int fellm_latent_token_clusters(int size) {
  static int cached[64][LT_MAX_CLUSTER + 1];
  int dev = 0;
  if (size < 1 || size > LT_MAX_CLUSTER || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!cached[dev][size]) {
    int n = 0;
    if (cudaFuncSetAttribute(latent_tokens_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LT_SMEM) != cudaSuccess) return 0;
    if (size > 8 && cudaFuncSetAttribute(latent_tokens_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) { cudaGetLastError(); return 0; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size); cfg.blockDim = dim3(LT_WARPS * 32); cfg.dynamicSmemBytes = LT_SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = size; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, latent_tokens_kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
    cached[dev][size] = n > 0 ? n + 1 : 1;
  }
  return cached[dev][size] - 1;
}

FELLM_API int fellm_latent_attention_rk() { return RK; }
FELLM_API int fellm_latent_attention_dr() { return DR; }

// variant 0: 64 rows a CTA (portions of prompts), n_splits must be 1; variant 1: 16 rows a CTA (single tokens),
// qsrc (or null): the queries' rotated parts are read from there and rotated in the kernel, and q holds the RK
// elements of a (token, head) row alone.  n_splits >= 1 shares of the keys: as a cluster (up to 16), or (up to 32) with scratch of rows * H * n_splits * (RK + 2) floats when above 1.
// ready (variant 1): see latent_tokens_kernel.
FELLM_API int fellm_latent_attention_mma(const void* q, const void* pool, const int* block_table, int max_pages,
                                         const int* positions, const int* row_slot, const int* item_start, int n_items,
                                         int max_item_rows, int rows_total, void* out, float* scratch, int n_splits, int H,
                                         int page_tokens, int layer, int layers_in_group, float scale, int window,
                                         const float* sinks, int variant, const void* qsrc, int ldq, int q_head, int q_rot_off,
                                         const float* freq, int n_rot, float mag, int cluster, int ready, cudaStream_t stream) {
  if (n_items <= 0 || rows_total <= 0 || max_item_rows <= 0) return 0;
  if (!q || !pool || !block_table || !positions || !row_slot || !item_start || !out) return FELLM_ERR_ARG;
  if (H < 1 || page_tokens < 1 || n_splits < 1 || n_splits > MAX_SPLITS || (n_splits > 1 && variant != 1) || (cluster && n_splits > LT_MAX_CLUSTER) ||
      (n_splits > 1 && !cluster && !scratch)) return FELLM_ERR_ARG;
  if (qsrc && ((ldq | q_head | q_rot_off) % 8 || ((size_t)qsrc & 15) || n_rot < 0 || n_rot > DR || (n_rot & 1) || (n_rot && !freq))) return FELLM_ERR_SIZE;
  LatArgs a;
  a.qsrc = DR ? (const bf16*)qsrc : nullptr; a.ldq = ldq; a.q_head = q_head; a.q_rot_off = q_rot_off; a.n_rot = n_rot; a.freq = freq; a.mag = mag;
  a.q = (const bf16*)q; a.pool = (const bf16*)pool; a.block_table = block_table; a.max_pages = max_pages;
  a.positions = positions; a.row_slot = row_slot; a.item_start = item_start; a.out = (bf16*)out; a.scratch = scratch;
  a.sinks = sinks; a.H = H; a.page_tokens = page_tokens; a.layer = layer; a.layers_in_group = layers_in_group;
  a.window = window > 0 ? window : 0; a.n_splits = n_splits; a.cluster = cluster && n_splits > 1; a.ready = ready; a.single = max_item_rows == 1 && n_items == rows_total; a.scale_log2 = scale * LOG2E;
  if (variant == 0) return launch_latent<4, 2>(a, n_items, max_item_rows, rows_total, stream);
  return launch_tokens(a, n_items, max_item_rows, rows_total, stream);
}
