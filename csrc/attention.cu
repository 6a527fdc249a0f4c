// Paged GQA attention for decode (single query, split-KV) and ragged causal prefill
// with a cached KV prefix. Cache layout: K, V = [num_blocks, Hkv, page_size, D] bf16.
//
// Both kernels stream 64-token K/V tiles of one KV head into swizzled shared memory
// with cp.async (double buffered; the per-token block-table lookup makes any page size
// work) and run QK^T / PV on the warp-level tensor path with fp32 online softmax.
// All q heads of a KV-head group share the tile: in decode they are the rows of one
// 16-row MMA tile and the four warps split the tile's tokens; in prefill the CTA's 64
// rows are (token, group-head) pairs.
//
// Behavioural counterparts in the reference: the single-query kernel with sliding
// window and attention sinks and its split-KV variant
// (src/parallax_extensions/kernels/paged_attention/paged_attention.metal:794-1347),
// and the prefix-aware prefill (src/parallax/utils/prefix_cache_utils.py:11-144).
#include <cuda_fp8.h>

#include <atomic>
#include <type_traits>

#include "attention_score.cuh"
#include "common.cuh"
#include "pxl_api.h"
#include "pxl_noalloc.h"

namespace {
using namespace pxl;

constexpr int TILE = 64;  // KV tokens per shared-memory tile
constexpr float kLog2e = 1.4426950408889634f;

struct KVTileArgs {
  const void* k_cache;   // bf16 elements, or e4m3 bytes for the FP8 kernels
  const void* v_cache;
  const int* block_table;  // row of this sequence
  int max_blocks;
  int64_t num_blocks;
  int Hkv;
  int kvh;
  int page_size;
};

// byte offset of 16-byte chunk `chunk` of row `row` inside a [TILE][D] bf16 tile
template <int D>
__device__ __forceinline__ uint32_t tile_off(int row, int chunk) {
  return static_cast<uint32_t>(row * (D * 2) + ((chunk ^ (row & 7)) << 4));
}
// Same for a tile that TMA wrote with the 128-byte swizzle: two halves of [TILE][64] elements
// (128-byte rows); inside a half the 16-byte chunk c of row r sits at position c ^ (r % 8).
__device__ __forceinline__ uint32_t tile_off_sw128(int row, int chunk) {
  return static_cast<uint32_t>((chunk >> 3) * (64 * 128) + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
}

// Eight e4m3 bytes -> eight bf16 (exact: every e4m3 value is a bf16 value), as one 16-byte vector.
__device__ __forceinline__ uint4 e4m3x8_to_bf16x8(uint2 raw) {
  uint4 out;
  uint32_t* o = &out.x;
  const uint32_t w[2] = {raw.x, raw.y};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_fp8x2_storage_t pair = static_cast<__nv_fp8x2_storage_t>((w[i >> 1] >> ((i & 1) * 16)) & 0xffffu);
    const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(pair, __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
    o[i] = pack_bf16x2(f.x, f.y);
  }
  return out;
}

// Issue the loads of K and V rows for tokens [tok0, tok0+TILE) ∩ [0, hi): cp.async for a bf16 cache;
// for an e4m3 cache (FP8) each thread reads 8 bytes, widens them to bf16 and stores the 16-byte
// chunk itself, so that the MMA code behind it is the same. The scales of an e4m3 cache are applied
// by the caller (K: folded into the score scale, V: into the output normalisation).
template <int D, bool FP8 = false>
__device__ __forceinline__ void load_kv_tile(const KVTileArgs& a, int tok0, int hi, uint32_t k_smem,
                                             uint32_t v_smem, int* status) {
  constexpr int CPR = D / 8;  // 8-element chunks per row
  constexpr int ITERS = TILE * CPR / 128;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    const int c = i * 128 + threadIdx.x;
    const int row = c / CPR;
    const int chunk = c % CPR;
    const int tok = tok0 + row;
    bool pred = tok < hi;
    int64_t base = 0;
    if (pred) {
      const int bi = tok / a.page_size;
      const int blk = (bi < a.max_blocks) ? a.block_table[bi] : -1;
      if (blk < 0 || blk >= a.num_blocks) {
        pred = false;
        if (status) atomicCAS(status, 0, PXL_DEV_BAD_BLOCK_PREFILL);
      } else {
        base = ((static_cast<int64_t>(blk) * a.Hkv + a.kvh) * a.page_size + (tok % a.page_size)) *
                   D +
               chunk * 8;
      }
    }
    const uint32_t off = tile_off<D>(row, chunk);
    if constexpr (FP8) {
      uint2 kr = make_uint2(0u, 0u), vr = make_uint2(0u, 0u);
      if (pred) {
        kr = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint8_t*>(a.k_cache) + base));
        vr = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint8_t*>(a.v_cache) + base));
      }
      const uint4 kb = e4m3x8_to_bf16x8(kr), vb = e4m3x8_to_bf16x8(vr);
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(k_smem + off), "r"(kb.x), "r"(kb.y),
                   "r"(kb.z), "r"(kb.w) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(v_smem + off), "r"(vb.x), "r"(vb.y),
                   "r"(vb.z), "r"(vb.w) : "memory");
    } else {
      cp_async_16(k_smem + off, static_cast<const bf16*>(a.k_cache) + base, pred);
      cp_async_16(v_smem + off, static_cast<const bf16*>(a.v_cache) + base, pred);
    }
  }
}

// S[16 x 16] += Q[16 x D] * K[tokens r0..r0+15]^T ; s[j] is the n-tile of tokens r0+8j..
template <int D, bool SW128 = false>
__device__ __forceinline__ void qk_16x16(const uint32_t (&qf)[D / 16][4], uint32_t k_smem, int r0,
                                         float (&s0)[4], float (&s1)[4]) {
  const int lane = threadIdx.x & 31;
  const int mi = lane >> 3;
  const int row = r0 + (mi >> 1) * 8 + (lane & 7);
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    uint32_t r[4];
    ldmatrix_x4(r, k_smem + (SW128 ? tile_off_sw128(row, ks * 2 + (mi & 1)) : tile_off<D>(row, ks * 2 + (mi & 1))));
    const uint32_t b0[2] = {r[0], r[1]};
    const uint32_t b1[2] = {r[2], r[3]};
    mma_m16n8k16_bf16(s0, qf[ks], b0);
    mma_m16n8k16_bf16(s1, qf[ks], b1);
  }
}

// O[16 x D] += P[16 x 16] * V[tokens r0..r0+15]
template <int D, bool SW128 = false>
__device__ __forceinline__ void pv_16x16(const uint32_t (&pf)[4], uint32_t v_smem, int r0,
                                         float (&o)[D / 8][4]) {
  const int lane = threadIdx.x & 31;
  const int mi = lane >> 3;
  const int row = r0 + (mi & 1) * 8 + (lane & 7);
#pragma unroll
  for (int np = 0; np < D / 16; ++np) {
    uint32_t r[4];
    ldmatrix_x4_trans(r, v_smem + (SW128 ? tile_off_sw128(row, np * 2 + (mi >> 1)) : tile_off<D>(row, np * 2 + (mi >> 1))));
    const uint32_t b0[2] = {r[0], r[1]};
    const uint32_t b1[2] = {r[2], r[3]};
    mma_m16n8k16_bf16(o[2 * np], pf, b0);
    mma_m16n8k16_bf16(o[2 * np + 1], pf, b1);
  }
}

// Tiles of the keys [0, keep) and [lo, hi), first to last: those of the kept keys that lie before the window's first tile,
// then the window's (keep <= 0: none kept).
struct KeyTiles {
  int front, first, total;
  __device__ KeyTiles(int lo, int hi, int keep) {
    first = lo / TILE;
    const int kept = keep > 0 ? ceil_div(keep, TILE) : 0;
    front = kept < first ? kept : first;
    total = hi > lo ? front + ceil_div(hi, TILE) - first : 0;
  }
  __device__ int operator[](int i) const { return i < front ? i : first + i - front; }
};

__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
  return v;
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}

// =============================================================================== decode
template <int D, bool FP8 = false, int SM = kPlain>
__global__ void __launch_bounds__(128)
attn_decode_kernel(const bf16* __restrict__ q, int64_t q_stride, const void* __restrict__ k_cache,
                   const void* __restrict__ v_cache, const int* __restrict__ block_tables,
                   const int* __restrict__ ctx_lens, bf16* __restrict__ out,
                   float* __restrict__ workspace, const float* __restrict__ sinks, int Hq, int Hkv,
                   int page_size, int max_blocks, int64_t num_blocks, float scale_log2, int window,
                   int keep, int num_splits, float v_scale, const ScoreArgs sa, int* status) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int TILE_BYTES = TILE * D * 2;
  const uint32_t k_smem0 = smem_u32(smem);
  const uint32_t v_smem0 = k_smem0 + 2 * TILE_BYTES;

  const int kvh = blockIdx.x, b = blockIdx.y, split = blockIdx.z;
  const int G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ctx = ctx_lens[b];
  const int hi = ctx;
  const int lo = (window > 0 && ctx > window) ? ctx - window : 0;
  const KeyTiles tiles(lo, hi, keep);
  const int per_split = ceil_div(tiles.total, num_splits);
  const int t_begin = split * per_split;
  const int t_end = min(tiles.total, t_begin + per_split);

  KVTileArgs ka{k_cache, v_cache, block_tables + static_cast<size_t>(b) * max_blocks, max_blocks,
                num_blocks, Hkv, kvh, page_size};

  // Q fragments: row r of the MMA tile is q head kvh*G + r (rows >= G are zero)
  uint32_t qf[D / 16][4];
  {
    const int r_lo = lane >> 2, r_hi = r_lo + 8;
    const bf16* q_lo = q + static_cast<size_t>(b) * q_stride + (kvh * G + r_lo) * D;
    const bf16* q_hi = q + static_cast<size_t>(b) * q_stride + (kvh * G + r_hi) * D;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      const int c = ks * 16 + 2 * (lane & 3);
      qf[ks][0] = r_lo < G ? *reinterpret_cast<const uint32_t*>(q_lo + c) : 0u;
      qf[ks][1] = r_hi < G ? *reinterpret_cast<const uint32_t*>(q_hi + c) : 0u;
      qf[ks][2] = r_lo < G ? *reinterpret_cast<const uint32_t*>(q_lo + c + 8) : 0u;
      qf[ks][3] = r_hi < G ? *reinterpret_cast<const uint32_t*>(q_hi + c + 8) : 0u;
    }
  }

  float bias2[2] = {0.f, 0.f};  // of this thread's two rows
  if constexpr (SM == kSigmoid) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = (lane >> 2) + h * 8;
      if (r < G) bias2[h] = sa.bias[kvh * G + r] * kLog2e;
    }
  }
  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY};
  float l_run[2] = {0.f, 0.f};

  int buf = 0;
  if (t_begin < t_end) load_kv_tile<D, FP8>(ka, tiles[t_begin] * TILE, hi, k_smem0, v_smem0, status);
  cp_async_commit();
  for (int t = t_begin; t < t_end; ++t) {
    cp_async_wait<0>();
    __syncthreads();
    if (t + 1 < t_end)
      load_kv_tile<D, FP8>(ka, tiles[t + 1] * TILE, hi, k_smem0 + (buf ^ 1) * TILE_BYTES,
                      v_smem0 + (buf ^ 1) * TILE_BYTES, status);
    cp_async_commit();

    const int r0 = warp * 16;
    const int tok_base = tiles[t] * TILE + r0;
    if (tok_base < hi && (tok_base + 16 > lo || tok_base < keep)) {  // warp-uniform
      float s[2][4];
#pragma unroll
      for (int j = 0; j < 2; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
      qk_16x16<D>(qf, k_smem0 + buf * TILE_BYTES, r0, s[0], s[1]);
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int tok = tok_base + j * 8 + 2 * (lane & 3) + (e & 1);
          const bool valid = tok < hi && (tok >= lo || tok < keep);
          if constexpr (SM == kSigmoid) {
            s[j][e] = valid ? sigmoid_weight(s[j][e], scale_log2, bias2[e >> 1]) : 0.f;
          } else {
            s[j][e] = valid ? score_log2<SM>(s[j][e], scale_log2, sa) : -INFINITY;
            mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
          }
        }
      }
      if constexpr (SM != kSigmoid) {
        float corr[2], m_use[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          mx[h] = quad_max(mx[h]);
          const float m_new = fmaxf(m_run[h], mx[h]);
          m_use[h] = (m_new == -INFINITY) ? 0.f : m_new;
          corr[h] = exp2f(m_run[h] - m_use[h]);
          m_run[h] = m_new;
        }
        float ps[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[j][e] = exp2f(s[j][e] - m_use[e >> 1]);
            ps[e >> 1] += s[j][e];
          }
        l_run[0] = l_run[0] * corr[0] + ps[0];
        l_run[1] = l_run[1] * corr[1] + ps[1];
#pragma unroll
        for (int i = 0; i < D / 8; ++i) {
          o[i][0] *= corr[0];
          o[i][1] *= corr[0];
          o[i][2] *= corr[1];
          o[i][3] *= corr[1];
        }
      }
      uint32_t pf[4];
      pf[0] = pack_bf16x2(s[0][0], s[0][1]);
      pf[1] = pack_bf16x2(s[0][2], s[0][3]);
      pf[2] = pack_bf16x2(s[1][0], s[1][1]);
      pf[3] = pack_bf16x2(s[1][2], s[1][3]);
      pv_16x16<D>(pf, v_smem0 + buf * TILE_BYTES, r0, o);
    }
    buf ^= 1;
  }
  cp_async_wait<0>();
  __syncthreads();

  // ---- merge the four warps' partial softmax states through shared memory
  float* o_sm = reinterpret_cast<float*>(smem);          // [4][16][D]
  float* m_sm = o_sm + 4 * 16 * D;                       // [4][16]
  float* l_sm = m_sm + 4 * 16;                           // [4][16]
  l_run[0] = quad_sum(l_run[0]);
  l_run[1] = quad_sum(l_run[1]);
  {
    const int r_lo = lane >> 2, r_hi = r_lo + 8;
    float* ow = o_sm + warp * 16 * D;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const int c = i * 8 + 2 * (lane & 3);
      ow[r_lo * D + c] = o[i][0];
      ow[r_lo * D + c + 1] = o[i][1];
      ow[r_hi * D + c] = o[i][2];
      ow[r_hi * D + c + 1] = o[i][3];
    }
    if ((lane & 3) == 0) {
      m_sm[warp * 16 + r_lo] = m_run[0];
      m_sm[warp * 16 + r_hi] = m_run[1];
      l_sm[warp * 16 + r_lo] = l_run[0];
      l_sm[warp * 16 + r_hi] = l_run[1];
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += 128) {
    const int r = idx / D, d = idx % D;
    const int head = kvh * G + r;
    if constexpr (SM == kSigmoid) {  // weights as they are: sums of the warps, of the splits
      float acc = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) acc += o_sm[(w * 16 + r) * D + d];
      if (num_splits == 1) out[(static_cast<size_t>(b) * Hq + head) * D + d] = __float2bfloat16(acc);
      else workspace[((static_cast<size_t>(b) * Hq + head) * num_splits + split) * D + d] = acc;
      continue;
    }
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, m_sm[w * 16 + r]);
    const float sink = (sinks && num_splits == 1) ? sinks[head] * kLog2e : -INFINITY;
    const float Mx = fmaxf(M, sink);
    const float Mu = (Mx == -INFINITY) ? 0.f : Mx;
    float L = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = exp2f(m_sm[w * 16 + r] - Mu);
      L += l_sm[w * 16 + r] * f;
      acc += o_sm[(w * 16 + r) * D + d] * f;
    }
    if (num_splits == 1) {
      const float denom = L + exp2f(sink - Mu);
      out[(static_cast<size_t>(b) * Hq + head) * D + d] =
          __float2bfloat16(denom > 0.f ? acc / denom * v_scale : 0.f);
    } else {
      // partial: normalised output + log2-sum-exp
      float* po = workspace;
      float* plse = workspace + static_cast<size_t>(gridDim.y) * Hq * num_splits * D;
      const size_t row = (static_cast<size_t>(b) * Hq + head) * num_splits + split;
      po[row * D + d] = L > 0.f ? acc / L * v_scale : 0.f;
      if (d == 0) plse[row] = L > 0.f ? Mu + log2f(L) : -INFINITY;
    }
  }
}

// ---- decode, TMA-fed variant (D = 128; page_size 16, 32 or 64) ------------------------------------
// A (block, kv head) page of the cache is one contiguous [page, 128] matrix, so a KV tile of 64
// tokens is 64 / page box loads per operand half: one thread issues them through the TMA engine
// (128-byte swizzle, completion on an mbarrier) up to three tiles ahead of the four consumer warps.
// This removes the per-thread address arithmetic and the 2048 cp.async instructions per tile of the
// kernel above, which was issue-bound at half of the DRAM bandwidth. The issuing lane sits in a warp
// of its own (warp 4) and the stages are handed back through "empty" mbarriers (one arrival per
// consumer warp), so the consumer warps never meet at a CTA-wide barrier inside the loop: with the
// producer inside warp 0 and a __syncthreads per tile the top stall was that barrier.
// ---- split-KV results met inside a thread-block cluster (2 to 8 splits of few sequences: splits_together): the CTAs of a
// (sequence, key head) write their partial outputs, maxima and sums into each other's shared memory, a share of the columns to each,
// and each adds up what it got. Saves the workspace's round trip and a kernel whose launch is most of its 4 to 5 us, once per layer of
// a chat. Written rather than read: one barrier instead of two and no remote load's latency (1 x 777 keys in 7 splits: 6.5 us, 5.5 now).
constexpr int kMaxClusterSplits = 8;

struct SplitParts {  // in shared memory that nothing else uses: the other CTAs write to it while this one is still at its keys
  float* base;       // [splits][share], then maxima and sums [kMaxClusterSplits][16]
  int splits, rank, share;
  static constexpr int kOut = 16 * 128 + kMaxClusterSplits, kFloats = kOut + 2 * kMaxClusterSplits * 16;

  __device__ __forceinline__ SplitParts(void* at, int splits, int rank, int G)
      : base(static_cast<float*>(at)), splits(splits), rank(rank), share(ceil_div(G * 128, splits)) {}
  __device__ __forceinline__ void put(int at, int to, float v) const { st_shared_cluster_f32(cluster_map_shared(smem_u32(base + at), to), v); }
  // element d of row r of this CTA's partial output, relative to the row's maximum M, and its sum L (both scaled by 2^shift)
  __device__ __forceinline__ void give(int r, int d, float acc, float M, float L) const {
    const int idx = r * 128 + d, to = idx / share;
    put(rank * share + idx - to * share, to, acc);
    if (d < splits) {
      put(kOut + rank * 16 + r, d, M);
      put(kOut + (kMaxClusterSplits + rank) * 16 + r, d, L);
    }
  }
  // Every thread of every CTA of the cluster calls this, also after a failed wait.
  template <int SM>
  __device__ __forceinline__ void add(int G, int head0, const float* sinks, float shift, float v_scale, bf16* out, bool failed) const {
    constexpr int D = 128;
    __syncwarp();
    cluster_sync_all();
    if (failed || threadIdx.x >= 128) return;
    const int end = min(share, G * D - rank * share);
    for (int j = threadIdx.x; j < end; j += 128) {
      const int idx = rank * share + j, r = idx / D, head = head0 + r;
      float acc = 0.f;
      if constexpr (SM == kSigmoid) {
        for (int s = 0; s < splits; ++s) acc += base[s * share + j];
        out[static_cast<size_t>(head) * D + idx % D] = __float2bfloat16(acc);
      } else {
        const float sink = sinks ? sinks[head] * kLog2e : -INFINITY;
        float m[kMaxClusterSplits], M = sink;
#pragma unroll
        for (int s = 0; s < kMaxClusterSplits; ++s) {
          m[s] = s < splits ? base[kOut + s * 16 + r] : -INFINITY;
          M = fmaxf(M, m[s]);
        }
        const float Mu = (M == -INFINITY) ? 0.f : M;
        float denom = exp2f(sink - Mu + shift);
#pragma unroll
        for (int s = 0; s < kMaxClusterSplits; ++s) {
          if (s >= splits) break;
          const float f = exp2f(m[s] - Mu);
          denom += base[kOut + (kMaxClusterSplits + s) * 16 + r] * f;
          acc += base[s * share + j] * f;
        }
        out[static_cast<size_t>(head) * D + idx % D] = __float2bfloat16(denom > 0.f ? acc / denom * v_scale : 0.f);
      }
    }
  }
};

// Producer warp: the blocks of the pages of 32 / (pages per tile) tiles at a time, one per lane, the next ones read while these are
// used. Read tile by tile, the latency of a table read was the time of a tile: 1.2 us (e4m3 0.7) with one CTA per SM, whatever the
// consumers did.
struct TileBlocks {
  const int* bt;
  KeyTiles tiles;
  int t_begin, n_tiles, page_size, shift, hi, max_blocks;  // shift: log2(pages per tile)
  int64_t num_blocks;
  int* status;
  int now = 0, ahead = 0;

  __device__ __forceinline__ int look(int it) const {
    const int lane = threadIdx.x & 31;
    it += lane >> shift;
    if (it >= n_tiles) return 0;
    int bi = (tiles[t_begin + it] << shift) + (lane & ((1 << shift) - 1));
    if (bi * page_size >= hi) bi = (hi - 1) / page_size;  // beyond the context: re-read the last page (masked)
    return bi < max_blocks ? bt[bi] : -1;
  }
  __device__ __forceinline__ void begin() { ahead = look(0); }
  // block of page lane % ppt of tile `it`; called by the whole warp, tile after tile
  __device__ __forceinline__ int operator()(int it) {
    const int per = 32 >> shift, i = it & (per - 1);
    if (i == 0) {
      now = ahead;
      ahead = look(it + per);  // not looked at before it is needed
      if (now < 0 || now >= num_blocks) {
        if (status) atomicCAS(status, 0, PXL_DEV_BAD_BLOCK_DECODE);
        now = 0;
      }
    }
    return __shfl_sync(0xffffffffu, now, (i << shift) + (threadIdx.x & ((1 << shift) - 1)));
  }
};

// The 16 rows of a warp's products (rows >= G of a key head's query heads are zero; rows 8 to 15 are left out of the softmax where
// HIGH is false): queries, running softmax and output of the keys that it has seen.
template <int SM, bool HIGH>
struct RowsBf16 {
  static constexpr int D = 128, kRows = HIGH ? 2 : 1, kKeys = 16;  // kRows: of this thread, lane / 4 and lane / 4 + 8; keys per step
  uint32_t qf[D / 16][4];
  float bias2[2], o[D / 8][4], m_run[2], l_run[2];

  // q: first query head of the key head
  __device__ __forceinline__ void begin(const bf16* q, int G, int head0, float, const ScoreArgs& sa) {
    const int lane = threadIdx.x & 31, r_lo = lane >> 2, r_hi = r_lo + 8;
    const bf16 *q_lo = q + r_lo * D, *q_hi = q + r_hi * D;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      const int c = ks * 16 + 2 * (lane & 3);
      qf[ks][0] = r_lo < G ? *reinterpret_cast<const uint32_t*>(q_lo + c) : 0u;
      qf[ks][1] = HIGH && r_hi < G ? *reinterpret_cast<const uint32_t*>(q_hi + c) : 0u;
      qf[ks][2] = r_lo < G ? *reinterpret_cast<const uint32_t*>(q_lo + c + 8) : 0u;
      qf[ks][3] = HIGH && r_hi < G ? *reinterpret_cast<const uint32_t*>(q_hi + c + 8) : 0u;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      bias2[h] = 0.f;
      if constexpr (SM == kSigmoid)
        if (r_lo + h * 8 < G) bias2[h] = sa.bias[head0 + r_lo + h * 8] * kLog2e;
      m_run[h] = -INFINITY;
      l_run[h] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  }

  // Keys r0 .. r0 + 15 of a tile; the first is token tok_base.
  __device__ __forceinline__ void step(uint32_t k_smem, uint32_t v_smem, int r0, int tok_base, int lo, int hi, int keep, float scale_log2,
                                       const ScoreArgs& sa) {
    if (!(tok_base < hi && (tok_base + kKeys > lo || tok_base < keep))) return;  // warp-uniform
    const int lane = threadIdx.x & 31;
    float s[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
    qk_16x16<D, true>(qf, k_smem, r0, s[0], s[1]);
    const bool whole = tok_base + kKeys <= hi && (tok_base >= lo || tok_base + kKeys <= keep);  // every token is seen
    float corr[2] = {1.f, 1.f};
#pragma unroll
    for (int h = 0; h < kRows; ++h) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 2 * h; e < 2 * h + 2; ++e) {
          if constexpr (SM == kSigmoid) s[j][e] = sigmoid_weight(s[j][e], scale_log2, bias2[h]);
          else s[j][e] = score_log2<SM>(s[j][e], scale_log2, sa);
          if (!whole) {
            const int tok = tok_base + j * 8 + 2 * (lane & 3) + (e & 1);
            if (!(tok < hi && (tok >= lo || tok < keep))) s[j][e] = SM == kSigmoid ? 0.f : -INFINITY;
          }
          if constexpr (SM != kSigmoid) mx = fmaxf(mx, s[j][e]);
        }
      if constexpr (SM != kSigmoid) {
        const float m_new = fmaxf(m_run[h], quad_max(mx));
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        corr[h] = exp2f(m_run[h] - m_use);
        m_run[h] = m_new;
        float ps = 0.f;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 2 * h; e < 2 * h + 2; ++e) {
            s[j][e] = exp2f(s[j][e] - m_use);
            ps += s[j][e];
          }
        l_run[h] = l_run[h] * corr[h] + ps;
      }
    }
    if (SM != kSigmoid && __any_sync(0xffffffffu, corr[0] != 1.f || (HIGH && corr[1] != 1.f))) {
#pragma unroll
      for (int i = 0; i < D / 8; ++i)
#pragma unroll
        for (int e = 0; e < 2 * kRows; ++e) o[i][e] *= corr[e >> 1];
    }
    uint32_t pf[4];
    pf[0] = pack_bf16x2(s[0][0], s[0][1]);
    pf[1] = HIGH ? pack_bf16x2(s[0][2], s[0][3]) : 0u;
    pf[2] = pack_bf16x2(s[1][0], s[1][1]);
    pf[3] = HIGH ? pack_bf16x2(s[1][2], s[1][3]) : 0u;
    pv_16x16<D, true>(pf, v_smem, r0, o);
  }

  // columns of the accumulator registers o[i][0], o[i][1], o[i + 1][0], o[i + 1][1] (i even): two pairs, 8 apart
  template <typename F>
  static __device__ __forceinline__ void columns(const float (&o)[D / 8][4], int i, int row, F put) {
    const int c = i * 8 + 2 * (threadIdx.x & 3);
    put(c, o[i][2 * row], o[i][2 * row + 1]);
    put(c + 8, o[i + 1][2 * row], o[i + 1][2 * row + 1]);
  }
};

constexpr int kDecStages = 3;
constexpr int kDecThreads = 160;  // 4 consumer warps + 1 producer warp

// CLUSTER: the splits of a (sequence, key head) are a cluster and add their results (SplitParts); else through the workspace
template <int SM, bool CLUSTER, bool HIGH>
__global__ void __launch_bounds__(kDecThreads, 2)
attn_decode_tma_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const bf16* __restrict__ q, int64_t q_stride, const int* __restrict__ block_tables,
                       const int* __restrict__ ctx_lens, bf16* __restrict__ out, float* __restrict__ workspace,
                       const float* __restrict__ sinks, int Hq, int Hkv, int page_size, int max_blocks,
                       int64_t num_blocks, float scale_log2, int window, int keep, int num_splits, const ScoreArgs sa,
                       int* status) {
  constexpr int D = 128;
  constexpr int TILE_BYTES = TILE * D * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t stage0 = smem_u32(smem);  // stage s: K tile at s * 2 * TILE_BYTES, V tile behind it
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kDecStages * 2 * TILE_BYTES);  // full[S], empty[S]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * kDecStages);
  const uint32_t full0 = smem_u32(bars);
  const uint32_t empty0 = smem_u32(bars + kDecStages);
  const int kvh = blockIdx.x, b = blockIdx.y, split = blockIdx.z;
  const int G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ctx = ctx_lens[b];
  const int hi = ctx;
  const int lo = (window > 0 && ctx > window) ? ctx - window : 0;
  const KeyTiles tiles(lo, hi, keep);
  const int per_split = ceil_div(tiles.total, num_splits);
  const int t_begin = split * per_split;
  const int t_end = min(tiles.total, t_begin + per_split);
  const int n_tiles = t_end > t_begin ? t_end - t_begin : 0;
  const int* bt = block_tables + static_cast<size_t>(b) * max_blocks;
  const int shift = page_size == 16 ? 2 : page_size == 32 ? 1 : 0, ppt = 1 << shift;  // pages per tile

  if constexpr (CLUSTER) cluster_arrive_all();  // its shared memory may be written to from here on
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kDecStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 4);  // one arrival per consumer warp
    }
    mbar_fence_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  // the tables and the lengths of a step are there before its first kernel, the queries and the new keys after the wait
  TileBlocks blocks{bt, tiles, t_begin, n_tiles, page_size, shift, hi, max_blocks, num_blocks, status};
  if (warp == 4) blocks.begin();
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();

  int failed = 0;
  if (warp == 4) {
    // ---- producer warp, up to kDecStages tiles ahead of the consumers. Lane p issues the four box loads of page p of the tile.
    for (int it = 0; it < n_tiles; ++it) {
      const int stage = it % kDecStages;
      const int blk = blocks(it);
      int okf = 1;
      if (it >= kDecStages && lane == 0)
        okf = mbar_wait_bounded(empty0 + 8 * stage, ((it / kDecStages) - 1) & 1, abort_flag, status,
                                PXL_DEV_TIMEOUT_EMPTY) ? 1 : 0;
      okf = __shfl_sync(0xffffffffu, okf, 0);
      if (!okf) {
        failed = 1;
        break;
      }
      const uint32_t bar = full0 + 8 * stage;
      const uint32_t k_dst = stage0 + stage * 2 * TILE_BYTES, v_dst = k_dst + TILE_BYTES;
      if (lane == 0) mbar_arrive_expect_tx(bar, 2 * TILE_BYTES);
      __syncwarp();
      if (lane < ppt) {
        const int row0 = (blk * Hkv + kvh) * page_size;
        const uint32_t off = lane * page_size * 128;
        tma_load_2d(k_dst + off, &tm_k, bar, 0, row0);
        tma_load_2d(k_dst + TILE * 128 + off, &tm_k, bar, 64, row0);
        tma_load_2d(v_dst + off, &tm_v, bar, 0, row0);
        tma_load_2d(v_dst + TILE * 128 + off, &tm_v, bar, 64, row0);
      }
    }
  }

  RowsBf16<SM, HIGH> rows;
  rows.begin(q + static_cast<size_t>(b) * q_stride + kvh * G * D, G, kvh * G, scale_log2, sa);
  float (&o)[D / 8][4] = rows.o;
  float (&m_run)[2] = rows.m_run, (&l_run)[2] = rows.l_run;

  for (int it = 0; warp < 4 && it < n_tiles; ++it) {
    const int stage = it % kDecStages;
    if (!mbar_wait_bounded(full0 + 8 * stage, (it / kDecStages) & 1, abort_flag, status, PXL_DEV_TIMEOUT_FULL)) {
      failed = 1;
      break;  // reported to the whole CTA at the barrier behind the loop
    }
    const uint32_t k_smem = stage0 + stage * 2 * TILE_BYTES;
    rows.step(k_smem, k_smem + TILE_BYTES, warp * 16, tiles[t_begin + it] * TILE + warp * 16, lo, hi, keep, scale_log2, sa);
    __syncwarp();
    if (lane == 0) mbar_arrive(empty0 + 8 * stage);  // this warp is done with the stage
  }
  const SplitParts parts(bars + 16, num_splits, split, G);
  if (__syncthreads_or(failed)) {
    // loads that are still in flight must land before the CTA's shared memory is released
    __nanosleep(200000);
    if constexpr (CLUSTER) {  // the other CTAs of the cluster wait for this one
      cluster_wait_all();
      parts.add<SM>(G, kvh * G, sinks, 0.f, 1.f, out, true);
    }
    return;
  }

  // ---- merge the four warps' partial softmax states through shared memory
  float* o_sm = reinterpret_cast<float*>(smem);          // [4][16][D]
  float* m_sm = o_sm + 4 * 16 * D;                       // [4][16]
  float* l_sm = m_sm + 4 * 16;                           // [4][16]
  l_run[0] = quad_sum(l_run[0]);
  l_run[1] = quad_sum(l_run[1]);
  if (warp < 4) {
    const int r_lo = lane >> 2, r_hi = r_lo + 8;
    float* ow = o_sm + warp * 16 * D;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const int c = i * 8 + 2 * (lane & 3);
      *reinterpret_cast<float2*>(ow + r_lo * D + c) = make_float2(o[i][0], o[i][1]);
      if constexpr (HIGH) *reinterpret_cast<float2*>(ow + r_hi * D + c) = make_float2(o[i][2], o[i][3]);
    }
    if ((lane & 3) == 0) {
      m_sm[warp * 16 + r_lo] = m_run[0];
      m_sm[warp * 16 + r_hi] = m_run[1];
      l_sm[warp * 16 + r_lo] = l_run[0];
      l_sm[warp * 16 + r_hi] = l_run[1];
    }
  }
  __syncwarp();
  if constexpr (CLUSTER) cluster_wait_all();
  __syncthreads();
  for (int idx = threadIdx.x; warp < 4 && idx < G * D; idx += 128) {
    const int r = idx / D, d = idx % D;
    const int head = kvh * G + r;
    if constexpr (SM == kSigmoid) {  // weights as they are: sums of the warps, of the splits
      float acc = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) acc += o_sm[(w * 16 + r) * D + d];
      if constexpr (CLUSTER) {
        parts.give(r, d, acc, 0.f, 0.f);
        continue;
      }
      if (num_splits == 1) out[(static_cast<size_t>(b) * Hq + head) * D + d] = __float2bfloat16(acc);
      else workspace[((static_cast<size_t>(b) * Hq + head) * num_splits + split) * D + d] = acc;
      continue;
    }
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, m_sm[w * 16 + r]);
    const float sink = (!CLUSTER && sinks && num_splits == 1) ? sinks[head] * kLog2e : -INFINITY;
    const float Mx = fmaxf(M, sink);
    const float Mu = (Mx == -INFINITY) ? 0.f : Mx;
    float L = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = exp2f(m_sm[w * 16 + r] - Mu);
      L += l_sm[w * 16 + r] * f;
      acc += o_sm[(w * 16 + r) * D + d] * f;
    }
    if constexpr (CLUSTER) {
      parts.give(r, d, acc, M, L);
    } else if (num_splits == 1) {
      const float denom = L + exp2f(sink - Mu);
      out[(static_cast<size_t>(b) * Hq + head) * D + d] = __float2bfloat16(denom > 0.f ? acc / denom : 0.f);
    } else {
      float* po = workspace;
      float* plse = workspace + static_cast<size_t>(gridDim.y) * Hq * num_splits * D;
      const size_t row = (static_cast<size_t>(b) * Hq + head) * num_splits + split;
      po[row * D + d] = L > 0.f ? acc / L : 0.f;
      if (d == 0) plse[row] = L > 0.f ? Mu + log2f(L) : -INFINITY;
    }
  }
  if constexpr (CLUSTER) parts.add<SM>(G, kvh * G, sinks, 0.f, 1.f, out + static_cast<size_t>(b) * Hq * D, false);
}

// ---- decode over e4m3 pages, TMA-fed (D = 128; page_size 16, 32 or 64) -------------------------------------
// The pages stay bytes up to the fragments: a tile of 64 tokens is 8 KB of K and 8 KB of V (one 128-byte swizzled row per
// token), so the same shared memory holds twice the tiles of the kernel above, and an operand is converted once, by the thread
// that multiplies it. Widening 8 bytes at a time into shared memory on the way in (the kernel without TMA) took 1170 us for 128
// rows x 3600 keys x 8 heads, 0.8 TB/s, bound by issue. One full wave (37 rows x 4096 keys x 8 heads) takes 52 us, 6.0 TB/s; 64 us
// when the block table was read tile by tile (TileBlocks) and each warp took 16 tokens of every tile, two chains of dependent
// products, one softmax and twice the shuffles, instead of 32 of every other one. Rows 8 to 15 of the products are nobody's with up
// to 8 query heads per key head: HIGH = false leaves their softmax out.
//
// e4m3 becomes f16 with one instruction per two values, exactly, and the products are f16 ones. What the other operands lose in
// range against bf16 they make up for in mantissa: a row of q is scaled by a power of two that puts its largest value at 2^13
// (undone in the score's scale), so that a bf16 value is kept exactly down to 2^-30 of it; probabilities carry a factor of 2^15,
// the largest that f16 holds, and are rounded to 2^-11 (bf16: 2^-8) down to 2^-29, below which a term is under the rounding of
// the fp32 sums. Error against 64 bits, outputs rounded to bf16 (1.60e-3 by itself), in this order before and now: equal scores
// 2.11e-3 and 1.67e-3, scores of deviation 1 2.22 and 1.67, of 8 1.607 and 1.598, one value of q of 1e6 2.18 and 1.67.
//   K: which columns a k-step of the MMA takes is free as long as q takes the same. Lane t of a quad takes columns 32 t .. 32 t
//      + 31 of its token as two 16-byte loads, four per k-step.
//   V: ldmatrix.trans moves pairs of columns; a byte permutation puts the two tokens of a column side by side, so that one
//      n-tile holds the even columns of 16 and the next the odd ones.
constexpr int kE4Stages = 6;
constexpr int kE4Tile = TILE * 128;  // bytes of K (or V) of a tile
constexpr float kPShift = 15.f;      // log2 of the factor on the probabilities

__device__ __forceinline__ uint32_t e4m3x2_to_f16x2(uint32_t two) {
  uint32_t r;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(static_cast<unsigned short>(two)));
  return r;
}
__device__ __forceinline__ void mma_m16n8k16_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_f16x2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <bool HIGH>
struct RowsE4m3 {
  static constexpr int D = 128, kRows = HIGH ? 2 : 1, kKeys = 32;
  uint32_t qf[D / 16][4];
  float row_scale[2], o[D / 8][4], m_run[2], l_run[2];

  // q: first query head of the key head; each row is scaled by a power of two
  __device__ __forceinline__ void begin(const bf16* q, int G, int, float scale_log2, const ScoreArgs&) {
    const int lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = g8 + h * 8;
      float mx = 0.f;
      if ((HIGH || h == 0) && r < G) {
        const bf16* row = q + r * D + t4 * 32;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          qf[ks][h] = *reinterpret_cast<const uint32_t*>(row + ks * 4);
          qf[ks][2 + h] = *reinterpret_cast<const uint32_t*>(row + ks * 4 + 2);
          const float2 x = unpack_bf16x2(qf[ks][h]), y = unpack_bf16x2(qf[ks][2 + h]);
          mx = fmaxf(fmaxf(fmaxf(mx, fabsf(x.x)), fabsf(x.y)), fmaxf(fabsf(y.x), fabsf(y.y)));
        }
      } else {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) qf[ks][h] = qf[ks][2 + h] = 0u;
      }
      if (!HIGH && h == 1) break;
      mx = quad_max(mx);
      int up = 267 - static_cast<int>(__float_as_uint(mx) >> 23);  // exponent bits of the factor: the largest value to [2^13, 2^14)
      up = up < 1 ? 1 : up > 253 ? 253 : up;
      const float f = __uint_as_float(static_cast<uint32_t>(up) << 23);
      row_scale[h] = __uint_as_float(static_cast<uint32_t>(254 - up) << 23) * scale_log2;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const float2 x = unpack_bf16x2(qf[ks][2 * p + h]);
          qf[ks][2 * p + h] = pack_f16x2(x.x * f, x.y * f);
        }
    }
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    m_run[0] = m_run[1] = -INFINITY;
    l_run[0] = l_run[1] = 0.f;
  }

  // Keys r0 .. r0 + 31 of a tile; the first is token tok_base.
  __device__ __forceinline__ void step(uint32_t k_smem, uint32_t v_smem, int r0, int tok_base, int lo, int hi, int keep, float,
                                       const ScoreArgs&) {
    if (!(tok_base < hi && (tok_base + kKeys > lo || tok_base < keep))) return;  // warp-uniform
    const int lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
    float s[kKeys / 8][4];  // 8 tokens each
#pragma unroll
    for (int j = 0; j < kKeys / 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t w[kKeys / 8][4];
#pragma unroll
      for (int j = 0; j < kKeys / 8; ++j) {
        const int row = r0 + j * 8 + g8;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w[j][0]), "=r"(w[j][1]), "=r"(w[j][2]), "=r"(w[j][3])
                     : "r"(k_smem + row * 128 + (((t4 * 2 + c) ^ (row & 7)) << 4)));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < kKeys / 8; ++j)
          mma_m16n8k16_f16(s[j], qf[c * 4 + i], e4m3x2_to_f16x2(w[j][i] & 0xffffu), e4m3x2_to_f16x2(w[j][i] >> 16));
    }
    const bool whole = tok_base + kKeys <= hi && (tok_base >= lo || tok_base + kKeys <= keep);  // every token is seen
    float corr[2] = {1.f, 1.f}, ps[2] = {0.f, 0.f};
#pragma unroll
    for (int h = 0; h < kRows; ++h) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < kKeys / 8; ++j)
#pragma unroll
        for (int e = 2 * h; e < 2 * h + 2; ++e) {
          s[j][e] *= row_scale[h];
          if (!whole) {
            const int tok = tok_base + j * 8 + 2 * t4 + (e & 1);
            if (!(tok < hi && (tok >= lo || tok < keep))) s[j][e] = -INFINITY;
          }
          mx = fmaxf(mx, s[j][e]);
        }
      const float m_new = fmaxf(m_run[h], quad_max(mx));
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
      corr[h] = exp2f(m_run[h] - m_use);
      m_run[h] = m_new;
#pragma unroll
      for (int j = 0; j < kKeys / 8; ++j)
#pragma unroll
        for (int e = 2 * h; e < 2 * h + 2; ++e) {
          s[j][e] = exp2f(s[j][e] - m_use + kPShift);
          ps[h] += s[j][e];
        }
      l_run[h] = l_run[h] * corr[h] + ps[h];
    }
    if (__any_sync(0xffffffffu, corr[0] != 1.f || (HIGH && corr[1] != 1.f))) {
#pragma unroll
      for (int i = 0; i < D / 8; ++i)
#pragma unroll
        for (int e = 0; e < 2 * kRows; ++e) o[i][e] *= corr[e >> 1];
    }
    if (!whole) {
      // The pages come whole. A probability of 0 times a NaN byte of a token that is not seen (what the page's last owner left
      // behind the context) would be NaN: this warp's rows of such tokens become zeros, in the first and last tiles only.
      for (int i = lane; i < kKeys * 8; i += 32) {
        const int tok = tok_base + (i >> 3);
        if (!(tok < hi && (tok >= lo || tok < keep))) st_shared_zero16(v_smem + (r0 + (i >> 3)) * 128 + (i & 7) * 16);
      }
      fence_proxy_async_smem();  // the stage is loaded again
      __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < kKeys / 16; ++k) {
      uint32_t pf[4];
      pf[0] = pack_f16x2(s[2 * k][0], s[2 * k][1]);
      pf[1] = HIGH ? pack_f16x2(s[2 * k][2], s[2 * k][3]) : 0u;
      pf[2] = pack_f16x2(s[2 * k + 1][0], s[2 * k + 1][1]);
      pf[3] = HIGH ? pack_f16x2(s[2 * k + 1][2], s[2 * k + 1][3]) : 0u;
      const int mi = lane >> 3, row = r0 + k * 16 + (mi & 1) * 8 + (lane & 7);
#pragma unroll
      for (int c = 0; c < 8; c += 2) {  // 16 columns per 16-byte chunk
        uint32_t r[4];  // chunk c: tokens 0-7, 8-15; chunk c + 1: the same
        ldmatrix_x4_trans(r, v_smem + row * 128 + (((c + (mi >> 1)) ^ (row & 7)) << 4));
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = __byte_perm(r[i], 0u, 0x3120);  // even column of both tokens | odd column
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          mma_m16n8k16_f16(o[(c + h) * 2], pf, e4m3x2_to_f16x2(r[2 * h] & 0xffffu), e4m3x2_to_f16x2(r[2 * h + 1] & 0xffffu));
          mma_m16n8k16_f16(o[(c + h) * 2 + 1], pf, e4m3x2_to_f16x2(r[2 * h] >> 16), e4m3x2_to_f16x2(r[2 * h + 1] >> 16));
        }
      }
    }
  }

  // columns of the accumulator registers o[i][0], o[i + 1][0], o[i][1], o[i + 1][1] (i even): four in a row
  template <typename F>
  static __device__ __forceinline__ void columns(const float (&o)[D / 8][4], int i, int row, F put) {
    const int c = i * 8 + 4 * (threadIdx.x & 3);
    put(c, o[i][2 * row], o[i + 1][2 * row]);
    put(c + 2, o[i][2 * row + 1], o[i + 1][2 * row + 1]);
  }
};

template <bool CLUSTER, bool HIGH>
__global__ void __launch_bounds__(kDecThreads, 2)
attn_decode_e4m3_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                        const bf16* __restrict__ q, int64_t q_stride, const int* __restrict__ block_tables,
                        const int* __restrict__ ctx_lens, bf16* __restrict__ out, float* __restrict__ workspace,
                        const float* __restrict__ sinks, int Hq, int Hkv, int page_size, int max_blocks,
                        int64_t num_blocks, float scale_log2, int window, int keep, int num_splits, float v_scale, int* status) {
  constexpr int D = 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t stage0 = smem_u32(smem);  // stage s: K at s * 2 * kE4Tile, V behind it
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kE4Stages * 2 * kE4Tile);  // full[S], empty[S]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * kE4Stages);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kE4Stages);
  const int kvh = blockIdx.x, b = blockIdx.y, split = blockIdx.z;
  const int G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hi = ctx_lens[b];
  const int lo = (window > 0 && hi > window) ? hi - window : 0;
  const KeyTiles tiles(lo, hi, keep);
  const int per_split = ceil_div(tiles.total, num_splits);
  const int t_begin = split * per_split;
  const int t_end = min(tiles.total, t_begin + per_split);
  const int n_tiles = t_end > t_begin ? t_end - t_begin : 0;
  const int* bt = block_tables + static_cast<size_t>(b) * max_blocks;
  const int shift = page_size == 16 ? 2 : page_size == 32 ? 1 : 0, ppt = 1 << shift;  // pages per tile

  if constexpr (CLUSTER) cluster_arrive_all();  // its shared memory may be written to from here on
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kE4Stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 2);  // one arrival per consumer warp
    }
    mbar_fence_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  // the tables and the lengths of a step are there before its first kernel, the queries and the new keys after the wait
  TileBlocks blocks{bt, tiles, t_begin, n_tiles, page_size, shift, hi, max_blocks, num_blocks, status};
  if (warp == 4) blocks.begin();
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();

  int failed = 0;
  if (warp == 4) {  // producer: lane p issues the two boxes of page p of the tile
    for (int it = 0; it < n_tiles; ++it) {
      const int stage = it % kE4Stages;
      const int blk = blocks(it);
      int okf = 1;
      if (it >= kE4Stages && lane == 0)
        okf = mbar_wait_bounded(empty0 + 8 * stage, ((it / kE4Stages) - 1) & 1, abort_flag, status, PXL_DEV_TIMEOUT_EMPTY) ? 1 : 0;
      okf = __shfl_sync(0xffffffffu, okf, 0);
      if (!okf) {
        failed = 1;
        break;
      }
      const uint32_t bar = full0 + 8 * stage, dst = stage0 + stage * 2 * kE4Tile + lane * page_size * 128;
      if (lane == 0) mbar_arrive_expect_tx(bar, 2 * kE4Tile);
      __syncwarp();
      if (lane < ppt) {
        const int row0 = (blk * Hkv + kvh) * page_size;
        tma_load_2d(dst, &tm_k, bar, 0, row0);
        tma_load_2d(dst + kE4Tile, &tm_v, bar, 0, row0);
      }
    }
  }

  const int g8 = lane >> 2, t4 = lane & 3;
  RowsE4m3<HIGH> rows;
  rows.begin(q + static_cast<size_t>(b) * q_stride + kvh * G * D, G, kvh * G, scale_log2, ScoreArgs{});
  float (&o)[D / 8][4] = rows.o;
  float (&m_run)[2] = rows.m_run, (&l_run)[2] = rows.l_run;

  // Warps 0 and 1 take the even tiles, 2 and 3 the odd ones, 32 tokens each. A stage has to belong to one pair (an even number of
  // them): another pair that is a use ahead would take the parity of the use before last for its own.
  static_assert(kE4Stages % 2 == 0);
  for (int it = warp >> 1; warp < 4 && it < n_tiles; it += 2) {
    const int stage = it % kE4Stages;
    if (!mbar_wait_bounded(full0 + 8 * stage, (it / kE4Stages) & 1, abort_flag, status, PXL_DEV_TIMEOUT_FULL)) {
      failed = 1;
      break;  // reported to the whole CTA at the barrier behind the loop
    }
    const uint32_t k_smem = stage0 + stage * 2 * kE4Tile;
    const int r0 = (warp & 1) * 32;
    rows.step(k_smem, k_smem + kE4Tile, r0, tiles[t_begin + it] * TILE + r0, lo, hi, keep, scale_log2, ScoreArgs{});
    __syncwarp();
    if (lane == 0) mbar_arrive(empty0 + 8 * stage);  // this warp is done with the stage
  }
  const SplitParts parts(bars + 16, num_splits, split, G);
  if (__syncthreads_or(failed)) {
    // loads that are still in flight must land before the CTA's shared memory is released
    __nanosleep(200000);
    if constexpr (CLUSTER) {  // the other CTAs of the cluster wait for this one
      cluster_wait_all();
      parts.add<kPlain>(G, kvh * G, sinks, 0.f, 1.f, out, true);
    }
    return;
  }

  // ---- merge the four warps' partial softmax states through shared memory
  float* o_sm = reinterpret_cast<float*>(smem);          // [4][16][D]
  float* m_sm = o_sm + 4 * 16 * D;                       // [4][16]
  float* l_sm = m_sm + 4 * 16;                           // [4][16]
  l_run[0] = quad_sum(l_run[0]);
  l_run[1] = quad_sum(l_run[1]);
  if (warp < 4) {
    float* ow = o_sm + warp * 16 * D;
#pragma unroll
    for (int i = 0; i < D / 8; i += 2) {  // accumulator columns 2 t, 2 t + 1 of an even and an odd tile: columns 4 t .. 4 t + 3
      const int c = i * 8 + t4 * 4;
      *reinterpret_cast<float4*>(ow + g8 * D + c) = make_float4(o[i][0], o[i + 1][0], o[i][1], o[i + 1][1]);
      if constexpr (HIGH) *reinterpret_cast<float4*>(ow + (g8 + 8) * D + c) = make_float4(o[i][2], o[i + 1][2], o[i][3], o[i + 1][3]);
    }
    if (t4 == 0) {
      m_sm[warp * 16 + g8] = m_run[0];
      m_sm[warp * 16 + g8 + 8] = m_run[1];
      l_sm[warp * 16 + g8] = l_run[0];
      l_sm[warp * 16 + g8 + 8] = l_run[1];
    }
  }
  __syncwarp();
  if constexpr (CLUSTER) cluster_wait_all();
  __syncthreads();
  for (int idx = threadIdx.x; warp < 4 && idx < G * D; idx += 128) {
    const int r = idx / D, d = idx % D;
    const int head = kvh * G + r;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, m_sm[w * 16 + r]);
    const float sink = (!CLUSTER && sinks && num_splits == 1) ? sinks[head] * kLog2e : -INFINITY;
    const float Mx = fmaxf(M, sink);
    const float Mu = (Mx == -INFINITY) ? 0.f : Mx;
    float L = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = exp2f(m_sm[w * 16 + r] - Mu);
      L += l_sm[w * 16 + r] * f;
      acc += o_sm[(w * 16 + r) * D + d] * f;
    }
    if constexpr (CLUSTER) {
      parts.give(r, d, acc, M, L);
    } else if (num_splits == 1) {
      const float denom = L + exp2f(sink - Mu + kPShift);
      out[(static_cast<size_t>(b) * Hq + head) * D + d] = __float2bfloat16(denom > 0.f ? acc / denom * v_scale : 0.f);
    } else {
      float* po = workspace;
      float* plse = workspace + static_cast<size_t>(gridDim.y) * Hq * num_splits * D;
      const size_t row = (static_cast<size_t>(b) * Hq + head) * num_splits + split;
      po[row * D + d] = L > 0.f ? acc / L * v_scale : 0.f;
      if (d == 0) plse[row] = L > 0.f ? Mu + log2f(L) - kPShift : -INFINITY;
    }
  }
  if constexpr (CLUSTER) parts.add<kPlain>(G, kvh * G, sinks, kPShift, v_scale, out + static_cast<size_t>(b) * Hq * D, false);
}

// ---- decode of many rows: every CTA the same number of tiles ------------------------------------------------------
// The tiles of all (sequence, key head) pairs stand in a row, and CTA c of n takes the c-th n-th of it: rows of any lengths end
// together, where a grid of pairs has a last wave (1024 pairs on 296 places are 3.46 waves) and waits for its longest row. The loads
// run on from one pair into the next: the ring of stages is filled with the next pair's keys, and its table read, while the results of
// the one before are put together, which by CTA per pair is 2 to 4 us in which a CTA loads nothing. A pair that lies in several CTAs is
// added up from the workspace by a second kernel: each CTA leaves at most the end of one pair (place 0) and the start of another (1).
// Against a grid of pairs (8 key heads, us): e4m3 128 x 4096 keys 169 and 154 (0.94 of the bandwidth), 40 x 4000 81 and 56; bf16 40 x
// 4000 121 and 95, 296 x 512 104 and 93, 512 x 100 78 and 47. Bounds: memory; over e4m3 pages and short rows the consumers, two warps
// per scheduler that convert and multiply one behind the other.
struct DecodeWork {
  const int* ctx_lens;
  int B, Hkv, window, keep;

  __device__ __forceinline__ KeyTiles tiles(int b, int& lo, int& hi) const {
    hi = __ldg(ctx_lens + b);
    lo = (window > 0 && hi > window) ? hi - window : 0;
    return KeyTiles(lo, hi, keep);
  }
  __device__ __forceinline__ int weight(int b) const {  // a pair without keys has a result too
    int lo, hi;
    const int n = tiles(b, lo, hi).total;
    return n > 0 ? n : 1;
  }
  __device__ __forceinline__ int64_t total() const {  // whole warp
    int sum = 0;
    for (int b = threadIdx.x & 31; b < B; b += 32) sum += weight(b);
    return static_cast<int64_t>(__reduce_add_sync(0xffffffffu, sum)) * Hkv;
  }
  // The pair that tile `pos` of the row belongs to, and which of its tiles it is; whole warp.
  __device__ __forceinline__ void find(int64_t pos, int& b, int& kvh, int& t) const {
    const int lane = threadIdx.x & 31;
    int64_t before = 0;  // of the chunk of 32 sequences
    for (int b0 = 0; b0 < B; b0 += 32) {
      const int w = b0 + lane < B ? weight(b0 + lane) : 0;
      int incl = w;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
      }
      const uint32_t past = __ballot_sync(0xffffffffu, before + static_cast<int64_t>(incl) * Hkv > pos);
      if (past) {
        const int at = __ffs(past) - 1;
        const int rest = static_cast<int>(pos - before - static_cast<int64_t>(__shfl_sync(0xffffffffu, incl - w, at)) * Hkv);
        const int wa = __shfl_sync(0xffffffffu, w, at);
        b = b0 + at;
        kvh = rest / wa;
        t = rest % wa;
        return;
      }
      before += static_cast<int64_t>(__shfl_sync(0xffffffffu, incl, 31)) * Hkv;
    }
    b = B, kvh = 0, t = 0;
  }
};

// Where the CTAs' shares begin: the first total % ctas of them are one tile longer.
struct DecodeShares {
  int64_t each;
  int longer;
  __device__ __forceinline__ DecodeShares(int64_t total, int ctas) : each(total / ctas), longer(static_cast<int>(total % ctas)) {}
  __device__ __forceinline__ int64_t operator[](int cta) const { return each * cta + min(cta, longer); }
};

// One CTA's way along the row, a pair (or the part of one that is its share) at a time.
struct DecodeWalk {
  DecodeWork work;
  int left, b, kvh, t, weight, take, lo, hi;  // tiles left; of the pair, tiles t .. t + take of `weight`
  KeyTiles tiles;

  __device__ __forceinline__ DecodeWalk(const DecodeWork& w, int cta, int ctas) : work(w), tiles(0, 0, 0) {
    const DecodeShares at(work.total(), ctas);
    left = static_cast<int>(at[cta + 1] - at[cta]);
    b = kvh = t = weight = take = lo = hi = 0;
    if (left > 0) {
      work.find(at[cta], b, kvh, t);
      enter();
    }
  }
  __device__ __forceinline__ void enter() {
    tiles = work.tiles(b, lo, hi);
    weight = tiles.total > 0 ? tiles.total : 1;
    take = min(left, weight - t);
  }
  __device__ __forceinline__ int count() const { return tiles.total > 0 ? take : 0; }
  __device__ __forceinline__ bool whole() const { return take == weight; }
  __device__ __forceinline__ void next() {
    left -= take;
    t += take;
    if (t == weight) {
      t = 0;
      if (++kvh == work.Hkv) kvh = 0, ++b;
    }
    if (left > 0) enter();
  }
};

template <bool F8, int SM>
using DecodeRows = std::conditional_t<F8, RowsE4m3<false>, RowsBf16<SM, false>>;
template <bool F8>
constexpr int kEvenSmem = 1024 + (F8 ? kE4Stages * 2 * kE4Tile : kDecStages * 4 * TILE * 128) + 3 * 4096 + 3 * 2 * 32 * 4 + 128;

template <bool F8, int SM>
__global__ void __launch_bounds__(kDecThreads, 2)
attn_decode_even_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const bf16* __restrict__ q,
                        int64_t q_stride, const int* __restrict__ block_tables, const int* __restrict__ ctx_lens,
                        bf16* __restrict__ out, float* __restrict__ workspace, const float* __restrict__ sinks, int B, int Hq, int Hkv,
                        int page_size, int max_blocks, int64_t num_blocks, float scale_log2, int window, int keep, float v_scale,
                        const ScoreArgs sa, int* status) {
  constexpr int D = 128, STAGES = F8 ? kE4Stages : kDecStages, TILE_BYTES = TILE * D * (F8 ? 1 : 2);
  using Rows = DecodeRows<F8, SM>;
  constexpr float kShift = F8 ? kPShift : 0.f;  // log2 of the factor on the probabilities
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t stage0 = smem_u32(smem);                                     // stage s: K at s * 2 * TILE_BYTES, V behind it
  float4* parts = reinterpret_cast<float4*>(smem + STAGES * 2 * TILE_BYTES);  // [3][8][32]: outputs of a warp, lane by lane
  float* part_m = reinterpret_cast<float*>(parts + 3 * 8 * 32);               // [3][32]
  float* part_l = part_m + 3 * 32;
  uint64_t* bars = reinterpret_cast<uint64_t*>(part_l + 3 * 32);  // full[S], empty[S]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * STAGES);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
  const int G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int shift = page_size == 16 ? 2 : page_size == 32 ? 1 : 0, ppt = 1 << shift;  // pages per tile

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, F8 ? 2 : 4);  // one arrival per warp that reads the stage
    }
    mbar_fence_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  // the lengths and the tables of a step are there before its first kernel, the queries and the new keys after the wait
  const DecodeWork work{ctx_lens, B, Hkv, window, keep};
  DecodeWalk walk(work, blockIdx.x, gridDim.x);
  auto blocks_of = [&](const DecodeWalk& w) {
    return TileBlocks{block_tables + static_cast<size_t>(w.left > 0 ? w.b : 0) * max_blocks, w.tiles, w.t, w.left > 0 ? w.count() : 0,
                      page_size, shift, w.hi, max_blocks, num_blocks, status};
  };
  TileBlocks blocks = blocks_of(walk);
  if (warp == 4) blocks.begin();
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();

  int failed = 0;
  int g = 0;  // tiles so far: tile g is in stage g % STAGES
  if (warp == 4) {  // producer: lane p issues the boxes of page p of the tile
    while (walk.left > 0 && !failed) {
      const int n = walk.count(), kvh = walk.kvh;
      walk.next();
      TileBlocks ahead = blocks_of(walk);
      ahead.begin();  // in flight during this pair
      for (int it = 0; it < n; ++it, ++g) {
        const int stage = g % STAGES;
        const int blk = blocks(it);
        int okf = 1;
        if (g >= STAGES && lane == 0)
          okf = mbar_wait_bounded(empty0 + 8 * stage, ((g / STAGES) - 1) & 1, abort_flag, status, PXL_DEV_TIMEOUT_EMPTY) ? 1 : 0;
        okf = __shfl_sync(0xffffffffu, okf, 0);
        if (!okf) {
          failed = 1;
          break;
        }
        const uint32_t bar = full0 + 8 * stage;
        const uint32_t dst = stage0 + stage * 2 * TILE_BYTES + lane * page_size * 128;
        if (lane == 0) mbar_arrive_expect_tx(bar, 2 * TILE_BYTES);
        __syncwarp();
        if (lane < ppt) {
          const int row0 = (blk * Hkv + kvh) * page_size;
          tma_load_2d(dst, &tm_k, bar, 0, row0);
          if constexpr (!F8) tma_load_2d(dst + TILE * 128, &tm_k, bar, 64, row0);
          tma_load_2d(dst + TILE_BYTES, &tm_v, bar, 0, row0);
          if constexpr (!F8) tma_load_2d(dst + TILE_BYTES + TILE * 128, &tm_v, bar, 64, row0);
        }
      }
      blocks = ahead;
    }
  } else {
    Rows rows;
    const int r0 = (F8 ? warp & 1 : warp) * Rows::kKeys;
    // after a failed wait the warp goes on to the end without loads or products: the others meet it at the barriers
    for (; walk.left > 0; walk.next()) {
      const int n = walk.count(), head0 = walk.kvh * G;
      rows.begin(q + static_cast<size_t>(walk.b) * q_stride + head0 * D, G, head0, scale_log2, sa);
      if (lane < 2 * G && walk.left > walk.take) {  // the next pair's queries, to be near when they are wanted
        const int kvh = walk.kvh + 1 < Hkv ? walk.kvh + 1 : 0, b = walk.b + (kvh == 0 ? 1 : 0);
        asm volatile("prefetch.global.L1 [%0];" ::"l"(q + static_cast<size_t>(b) * q_stride + kvh * G * D + lane * 64));
      }
      for (int it = 0; it < n; ++it, ++g) {
        if (F8 && (g & 1) != (warp >> 1)) continue;  // warps 0 and 1 take the even stages, 2 and 3 the odd ones (attn_decode_e4m3_kernel)
        const int stage = g % STAGES;
        if (!failed)
          failed = __any_sync(0xffffffffu, !mbar_wait_bounded(full0 + 8 * stage, (g / STAGES) & 1, abort_flag, status, PXL_DEV_TIMEOUT_FULL));
        if (failed) continue;
        const uint32_t k_smem = stage0 + stage * 2 * TILE_BYTES;
        rows.step(k_smem, k_smem + TILE_BYTES, r0, walk.tiles[walk.t + it] * TILE + r0, walk.lo, walk.hi, keep, scale_log2, sa);
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * stage);
      }

      // warps 2 and 3 hand their results to 0 and 1, 1 to 0; a register goes to the same lane
      auto give = [&](int p) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          parts[(p * 8 + i) * 32 + lane] = make_float4(rows.o[2 * i][0], rows.o[2 * i][1], rows.o[2 * i + 1][0], rows.o[2 * i + 1][1]);
        part_m[p * 32 + lane] = rows.m_run[0];
        part_l[p * 32 + lane] = rows.l_run[0];
      };
      auto add = [&](int p) {
        float fa = 1.f, fb = 1.f;
        if constexpr (SM != kSigmoid) {
          const float m = part_m[p * 32 + lane], M = fmaxf(rows.m_run[0], m), Mu = M == -INFINITY ? 0.f : M;
          fa = exp2f(rows.m_run[0] - Mu);
          fb = exp2f(m - Mu);
          rows.m_run[0] = M;
          rows.l_run[0] = rows.l_run[0] * fa + part_l[p * 32 + lane] * fb;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 x = parts[(p * 8 + i) * 32 + lane];
          rows.o[2 * i][0] = rows.o[2 * i][0] * fa + x.x * fb;
          rows.o[2 * i][1] = rows.o[2 * i][1] * fa + x.y * fb;
          rows.o[2 * i + 1][0] = rows.o[2 * i + 1][0] * fa + x.z * fb;
          rows.o[2 * i + 1][1] = rows.o[2 * i + 1][1] * fa + x.w * fb;
        }
      };
      if (warp >= 2) give(warp - 2);
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (warp < 2) add(warp);
      if (warp == 1) give(2);
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (warp == 0) {
        add(2);
        const int r = lane >> 2;
        const float M = rows.m_run[0], L = quad_sum(rows.l_run[0]);
        if (r < G && !failed) {
          if (walk.whole()) {
            float f = 1.f;
            if constexpr (SM != kSigmoid) {
              const float sink = sinks ? sinks[head0 + r] * kLog2e : -INFINITY;
              const float Mx = fmaxf(M, sink), Mu = Mx == -INFINITY ? 0.f : Mx;
              const float e = exp2f(M - Mu), denom = L * e + exp2f(sink - Mu + kShift);
              f = denom > 0.f ? e / denom * v_scale : 0.f;
            }
            bf16* dst = out + (static_cast<size_t>(walk.b) * Hq + head0 + r) * D;
#pragma unroll
            for (int i = 0; i < D / 8; i += 2)
              Rows::columns(rows.o, i, 0, [&](int c, float x, float y) { *reinterpret_cast<uint32_t*>(dst + c) = pack_bf16x2(x * f, y * f); });
          } else {
            const size_t place = static_cast<size_t>(blockIdx.x) * 2 + (walk.t == 0 ? 1 : 0);
            float* po = workspace + place * G * (D + 2);
#pragma unroll
            for (int i = 0; i < D / 8; i += 2)
              Rows::columns(rows.o, i, 0, [&](int c, float x, float y) { *reinterpret_cast<float2*>(po + r * D + c) = make_float2(x, y); });
            if ((lane & 3) == 0) po[G * D + r] = M, po[G * D + G + r] = L;
          }
        }
      }
    }
  }
  if (__syncthreads_or(failed)) __nanosleep(200000);  // loads that are still in flight must land before the shared memory is released
}

// Adds up the pairs that lie in several CTAs of attn_decode_even_kernel. Block x: the pair that the border between CTAs x and x + 1 cuts,
// if no border before it does. Four query heads at a time, so that their loads are in flight together.
template <int SM>
__global__ void __launch_bounds__(128)
attn_decode_even_reduce_kernel(const float* __restrict__ workspace, const float* __restrict__ sinks, const int* __restrict__ ctx_lens,
                               bf16* __restrict__ out, int B, int Hq, int Hkv, int window, int keep, float shift, float v_scale) {
  constexpr int D = 128, R = 4;
  const DecodeWork work{ctx_lens, B, Hkv, window, keep};
  const int ctas = gridDim.x + 1, cut = blockIdx.x + 1, d = threadIdx.x, G = Hq / Hkv;
  const DecodeShares at(work.total(), ctas);
  const int64_t pos = at[cut];
  int b, kvh, t;
  work.find(pos, b, kvh, t);
  const int64_t begin = pos - t;
  const bool mine = t > 0 && b < B && at[cut - 1] <= begin;
  int last = cut;  // CTA that ends the pair; all of them up to it have tiles of it
  if (mine)
    for (const int64_t end = begin + work.weight(b); at[last + 1] < end;) ++last;
  pdl_wait();
  pdl_launch_dependents();
  if (!mine) return;
  const size_t place = static_cast<size_t>(G) * (D + 2);
  auto part = [&](int x) { return workspace + (static_cast<size_t>(x) * 2 + (x < cut ? 1 : 0)) * place; };
  for (int r0 = 0; r0 < G; r0 += R) {
    float acc[R], denom[R], M[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      acc[i] = 0.f;
      M[i] = sinks && r0 + i < G ? sinks[kvh * G + r0 + i] * kLog2e : -INFINITY;
      denom[i] = M[i] == -INFINITY ? 0.f : exp2f(shift);  // the sink's share, relative to M
    }
    for (int x = cut - 1; x <= last; ++x) {
      const float* p = part(x) + r0 * D + d;
      const float *pm = part(x) + G * D + r0, *pl = pm + G;
      float o[R], m[R], l[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const bool in = r0 + i < G;
        o[i] = in ? p[i * D] : 0.f;
        if constexpr (SM != kSigmoid) {
          m[i] = in ? pm[i] : -INFINITY;
          l[i] = in ? pl[i] : 0.f;
        }
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if constexpr (SM == kSigmoid) {
          acc[i] += o[i];
        } else {
          const float Mn = fmaxf(M[i], m[i]), Mu = Mn == -INFINITY ? 0.f : Mn;
          const float f = exp2f(M[i] - Mu), g = exp2f(m[i] - Mu);
          acc[i] = acc[i] * f + o[i] * g;
          denom[i] = denom[i] * f + l[i] * g;
          M[i] = Mn;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (r0 + i >= G) break;
      float res = acc[i];
      if constexpr (SM != kSigmoid) res = denom[i] > 0.f ? res / denom[i] * v_scale : 0.f;
      out[(static_cast<size_t>(b) * Hq + kvh * G + r0 + i) * D + d] = __float2bfloat16(res);
    }
  }
}

template <int D, int SM = kPlain>
__global__ void __launch_bounds__(D)
attn_decode_reduce_kernel(const float* __restrict__ workspace, const float* __restrict__ sinks,
                          bf16* __restrict__ out, int Hq, int num_splits) {
  pdl_wait();
  pdl_launch_dependents();
  const int head = blockIdx.x, b = blockIdx.y, d = threadIdx.x;
  const float* po = workspace;
  const float* plse = workspace + static_cast<size_t>(gridDim.y) * Hq * num_splits * D;
  const size_t row0 = (static_cast<size_t>(b) * Hq + head) * num_splits;
  if constexpr (SM == kSigmoid) {
    float sum = 0.f;
    for (int s = 0; s < num_splits; ++s) sum += po[(row0 + s) * D + d];
    out[(static_cast<size_t>(b) * Hq + head) * D + d] = __float2bfloat16(sum);
    return;
  }
  const float sink = sinks ? sinks[head] * kLog2e : -INFINITY;
  float M = sink;
  for (int s = 0; s < num_splits; ++s) M = fmaxf(M, plse[row0 + s]);
  const float Mu = (M == -INFINITY) ? 0.f : M;
  float denom = exp2f(sink - Mu), acc = 0.f;
  for (int s = 0; s < num_splits; ++s) {
    const float w = exp2f(plse[row0 + s] - Mu);
    denom += w;
    acc += w * po[(row0 + s) * D + d];
  }
  out[(static_cast<size_t>(b) * Hq + head) * D + d] =
      __float2bfloat16(denom > 0.f ? acc / denom : 0.f);
}

// ============================================================================== prefill
template <int D, bool FP8 = false, int SM = kPlain>
__global__ void __launch_bounds__(128)
attn_prefill_kernel(const bf16* __restrict__ q, int64_t q_stride, const void* __restrict__ k_cache,
                    const void* __restrict__ v_cache, const int* __restrict__ block_tables,
                    const int* __restrict__ cu_q, const int* __restrict__ ctx_lens,
                    bf16* __restrict__ out, int64_t out_stride, const float* __restrict__ sinks,
                    int Hq, int Hkv, int page_size, int max_blocks, int64_t num_blocks,
                    float scale_log2, int window, int keep, float v_scale, const ScoreArgs sa, int* status) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int TILE_BYTES = TILE * D * 2;
  const uint32_t k_smem0 = smem_u32(smem);
  const uint32_t v_smem0 = k_smem0 + 2 * TILE_BYTES;

  const int qt = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int G = Hq / Hkv;
  const int TQ = 64 / G;  // query tokens per CTA (rows = TQ * G <= 64)
  const int q0 = cu_q[b];
  const int q_len = cu_q[b + 1] - q0;
  if (qt * TQ >= q_len) return;
  const int ctx = ctx_lens[b];
  const int prefix = ctx - q_len;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // rows owned by this thread: r_lo = warp*16 + lane/4, r_hi = r_lo + 8
  int rtok[2], rhead[2];
  bool rvalid[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = warp * 16 + (lane >> 2) + h * 8;
    const int tq = qt * TQ + r / G;
    rvalid[h] = (r < TQ * G) && (tq < q_len);
    rtok[h] = tq;
    rhead[h] = kvh * G + r % G;
  }
  uint32_t qf[D / 16][4];
  {
    const bf16* q_lo = q + static_cast<size_t>(q0 + rtok[0]) * q_stride + rhead[0] * D;
    const bf16* q_hi = q + static_cast<size_t>(q0 + rtok[1]) * q_stride + rhead[1] * D;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      const int c = ks * 16 + 2 * (lane & 3);
      qf[ks][0] = rvalid[0] ? *reinterpret_cast<const uint32_t*>(q_lo + c) : 0u;
      qf[ks][1] = rvalid[1] ? *reinterpret_cast<const uint32_t*>(q_hi + c) : 0u;
      qf[ks][2] = rvalid[0] ? *reinterpret_cast<const uint32_t*>(q_lo + c + 8) : 0u;
      qf[ks][3] = rvalid[1] ? *reinterpret_cast<const uint32_t*>(q_hi + c + 8) : 0u;
    }
  }
  // visible key range per row: [rlo, rpos]
  int rpos[2], rlo[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    rpos[h] = rvalid[h] ? prefix + rtok[h] : -1;
    rlo[h] = (window > 0 && rpos[h] >= window) ? rpos[h] - window + 1 : 0;
  }
  // warp-level bounds (rows of one warp span consecutive tokens)
  const int w_tok_first = qt * TQ + (warp * 16) / G;
  const int w_tok_last = min(q_len - 1, qt * TQ + (warp * 16 + 15) / G);
  const bool warp_active = (warp * 16 < TQ * G) && (w_tok_first < q_len);
  const int w_hi = prefix + w_tok_last;  // last visible key for this warp
  const int w_lo = (window > 0 && prefix + w_tok_first >= window) ? prefix + w_tok_first - window + 1 : 0;

  // CTA-level key range
  const int c_tok_last = min(q_len - 1, qt * TQ + TQ - 1);
  const int c_hi = prefix + c_tok_last + 1;  // exclusive
  const int c_lo = (window > 0 && prefix + qt * TQ >= window) ? prefix + qt * TQ - window + 1 : 0;
  const KeyTiles tiles(c_lo, c_hi, keep);

  KVTileArgs ka{k_cache, v_cache, block_tables + static_cast<size_t>(b) * max_blocks, max_blocks,
                num_blocks, Hkv, kvh, page_size};

  float bias2[2] = {0.f, 0.f};
  if constexpr (SM == kSigmoid) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (rvalid[h]) bias2[h] = sa.bias[rhead[h]] * kLog2e;
  }
  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY};
  float l_run[2] = {0.f, 0.f};

  int buf = 0;
  load_kv_tile<D, FP8>(ka, tiles[0] * TILE, c_hi, k_smem0, v_smem0, status);
  cp_async_commit();
  for (int t = 0; t < tiles.total; ++t) {
    cp_async_wait<0>();
    __syncthreads();
    if (t + 1 < tiles.total)
      load_kv_tile<D, FP8>(ka, tiles[t + 1] * TILE, c_hi, k_smem0 + (buf ^ 1) * TILE_BYTES,
                      v_smem0 + (buf ^ 1) * TILE_BYTES, status);
    cp_async_commit();

    const int tok0 = tiles[t] * TILE;
    if (warp_active && tok0 <= w_hi && (tok0 + TILE > w_lo || tok0 < keep)) {
      const uint32_t ks_addr = k_smem0 + buf * TILE_BYTES;
      const uint32_t vs_addr = v_smem0 + buf * TILE_BYTES;
      float s[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
      for (int g = 0; g < 4; ++g) qk_16x16<D>(qf, ks_addr, g * 16, s[2 * g], s[2 * g + 1]);

      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int h = e >> 1;
          const int tok = tok0 + j * 8 + 2 * (lane & 3) + (e & 1);
          const bool valid = tok <= rpos[h] && (tok >= rlo[h] || tok < keep);
          if constexpr (SM == kSigmoid) {
            s[j][e] = valid ? sigmoid_weight(s[j][e], scale_log2, bias2[h]) : 0.f;
          } else {
            s[j][e] = valid ? score_log2<SM>(s[j][e], scale_log2, sa) : -INFINITY;
            mx[h] = fmaxf(mx[h], s[j][e]);
          }
        }
      if constexpr (SM != kSigmoid) {
        float corr[2], m_use[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          mx[h] = quad_max(mx[h]);
          const float m_new = fmaxf(m_run[h], mx[h]);
          m_use[h] = (m_new == -INFINITY) ? 0.f : m_new;
          corr[h] = exp2f(m_run[h] - m_use[h]);
          m_run[h] = m_new;
        }
        float ps[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[j][e] = exp2f(s[j][e] - m_use[e >> 1]);
            ps[e >> 1] += s[j][e];
          }
        l_run[0] = l_run[0] * corr[0] + ps[0];
        l_run[1] = l_run[1] * corr[1] + ps[1];
#pragma unroll
        for (int i = 0; i < D / 8; ++i) {
          o[i][0] *= corr[0];
          o[i][1] *= corr[0];
          o[i][2] *= corr[1];
          o[i][3] *= corr[1];
        }
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint32_t pf[4];
        pf[0] = pack_bf16x2(s[2 * g][0], s[2 * g][1]);
        pf[1] = pack_bf16x2(s[2 * g][2], s[2 * g][3]);
        pf[2] = pack_bf16x2(s[2 * g + 1][0], s[2 * g + 1][1]);
        pf[3] = pack_bf16x2(s[2 * g + 1][2], s[2 * g + 1][3]);
        pv_16x16<D>(pf, vs_addr, g * 16, o);
      }
    }
    buf ^= 1;
  }
  cp_async_wait<0>();

#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!rvalid[h]) continue;
    float L = quad_sum(l_run[h]);
    float M = m_run[h];
    const float sink = sinks ? sinks[rhead[h]] * kLog2e : -INFINITY;
    const float Mx = fmaxf(M, sink);
    const float Mu = (Mx == -INFINITY) ? 0.f : Mx;
    const float f = exp2f(M - Mu);
    const float denom = L * f + exp2f(sink - Mu);
    const float inv = SM == kSigmoid ? 1.f : denom > 0.f ? f / denom * v_scale : 0.f;
    bf16* dst = out + static_cast<size_t>(q0 + rtok[h]) * out_stride + rhead[h] * D;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const int c = i * 8 + 2 * (lane & 3);
      *reinterpret_cast<uint32_t*>(dst + c) =
          pack_bf16x2(o[i][2 * h] * inv, o[i][2 * h + 1] * inv);
    }
  }
}

inline int check_launch() { return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA; }

template <typename K>
int set_smem(K kern, int bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
                 cudaSuccess
             ? PXL_OK
             : PXL_ERR_CUDA;
}

}  // namespace

// Splits of a decode step: the count with the lowest estimate, us = (tiles of a mean row's split + start) x waves of CTAs + adding + what
// the longest row's split takes beyond a mean one's. A last wave of few CTAs costs nearly as much as a full one, which
// ceil(2 SMs / CTAs), the rule before, did not see; where rows differ in length it is filled by the rows behind (`behind`: the part
// of that cost that stays).
//
// Pages the TMA unit reads (head dim 128): 2 CTAs per SM; `part` us per tile of 64 keys while the memory is not full (less behind a
// full wave, whose rows do not end together), `full` beside a full chip of others, `alone` where the others are done. Adding is
// cheaper inside a cluster than through the workspace, whose bytes grow with the query heads per key head. Tiles dealt out evenly
// (attn_decode_even_kernel, asked for by splits that give two places per CTA) take `full` for each and a start, a sum and a share per
// pair (more where short pairs stand beside long ones: even_short per pair, for CTAs that have many, and even_each per tile), and the
// reduction a time per four query heads and CTA that the longest row lies in. The kernel for other pages and head dim 64: 5 CTAs per
// SM (3 at 128), 1.2 us per tile (1.5 at 128, 2 of e4m3 bytes), always through the workspace.
//
// Fitted to the times of every count, in a chain of launches, for 2410 batches (TMA, pages of 64 and of 16; 750 of the other kernel)
// of 1 to 512 rows, 16 to 100000 keys, 1 to 8 key heads and 1 to 16 query heads for each: rows alike, within a quarter, one of up to
// 60 times the others, spread evenly or over their logarithm. Time over the fastest measured, mean and worst, with the rule before,
// with every row taken for as long as the longest, and now:
//   bf16, pages of 64  1.27 4.8   1.20 6.4   1.01 1.2     e4m3, pages of 64  1.34 7.4   1.14 7.9   1.01 1.4
//   bf16, pages of 16  1.38 12.7  1.30 13.9  1.01 1.2     e4m3, pages of 16  1.43 13.5  1.16 13.5  1.01 1.3
//   bf16, head dim 64  1.59 8.5   1.09 3.3   1.02 1.2     e4m3, head dim 64  1.77 7.7   1.13 3.7   1.02 1.2
//   bf16, other pages  1.54 6.5   1.17 5.8   1.03 1.3     e4m3, other pages  1.75 7.5   1.27 6.9   1.03 1.4
// 8 key heads, splits or even (us, with the rule before and now):
//   rows x keys        bf16                       e4m3
//   1 x 777            4:  8.1      7:    6.7     4:  7.5     7:     6.4
//   16 x 1280          3: 24.6      2:   17.8     3: 18.6     2:    12.9
//   40 x 4000          1: 121       even: 95      1: 81       even: 56
//   512 x 100          1: 78        even: 47      1: 71       even: 57
//   1 x 32768 and
//     31 x 1000        2: 183       even: 62      2: 167      even: 48   (every row for as long as the longest: bf16 1: 284)
//
// total_ctx: keys of all rows together, 0 where it is not known: rows as long as the longest.
PXL_EXPORT int pxl_attn_decode_splits_of(int B, int Hq, int Hkv, int D, int page_size, int cache_fp8, int max_ctx, int64_t total_ctx) {
  struct Line {
    float start, part, part_behind, full, cluster, add, add_split, add_wave;
    float even, even_pair, even_short, even_each, even_part, even_margin, alone;
  };
  static constexpr Line kLines[2][2] = {{{1.9f, 0.9f, 0.65f, 1.4f, 1.45f, 2.5f, 0.14f, 0.23f, 8.9f, 0.85f, 0.f, 0.35f, 0.5f, 0.95f, 0.65f},
                                         {1.9f, 1.04f, 1.f, 1.4f, 1.6f, 2.1f, 0.12f, 0.3f, 8.9f, 0.46f, 0.f, 0.52f, 0.37f, 0.96f, 0.88f}},
                                        {{2.3f, 0.61f, 0.7f, 0.68f, 2.4f, 1.4f, 0.23f, 0.49f, 9.f, 0.3f, 7.f, 0.16f, 0.4f, 0.98f, 0.55f},
                                         {3.f, 0.61f, 0.64f, 0.72f, 2.05f, 1.7f, 0.12f, 0.27f, 8.f, 0.f, 4.3f, 0.02f, 0.4f, 0.99f, 0.46f}}};
  const Line& c = kLines[cache_fp8 ? 1 : 0][page_size < 64 ? 1 : 0];  // (a tile of four pages is four times the boxes)
  const bool tma = D == 128 && (page_size == 16 || page_size == 32 || page_size == 64);
  const int64_t pairs = static_cast<int64_t>(B) * Hkv;
  const int chip = 2 * pxl_host::num_sms(), slots = tma ? chip : (D == 64 ? 5 : 3) * pxl_host::num_sms();
  const float tile = cache_fp8 ? 2.f : D == 64 ? 1.2f : 1.5f;  // of the other kernel
  if (max_ctx < 1) max_ctx = 1;
  const int tiles = pxl::ceil_div(max_ctx, TILE);
  // a mean row, as a part of the longest (its last tile is half full)
  float mean = 1.f;
  if (total_ctx > 0 && total_ctx < static_cast<int64_t>(B) * max_ctx)
    mean = fminf(1.f, (static_cast<float>(total_ctx) / (static_cast<float>(B) * TILE) + 0.5f) / static_cast<float>(tiles));
  const float behind = fmaxf(0.f, 1.f - 4.f * (1.f - mean));
  const int group = Hkv > 0 ? Hq / Hkv : 0;
  const bool even = tma && group > 0 && group <= 8 && pairs > 0 && pairs * 64 >= 2 * chip;
  int best = 1, last = 0;
  float best_us = 0.f;
  for (int s = 1; s <= 64 && s <= tiles; ++s) {
    const int per = pxl::ceil_div(tiles, s);
    if (per == last) continue;  // no fewer tiles for the longest split
    last = per;
    const int64_t ctas = pairs * s, full = ctas / slots, rest = ctas % slots;
    if (even && s > 1 && ctas >= 2 * chip) break;  // asks for the even kernel
    const float waves = static_cast<float>(ctas) / static_cast<float>(chip), wave = static_cast<float>(rest) / slots;
    const float mine = static_cast<float>(per) * mean, longer = static_cast<float>(per) - mine;
    auto last_wave = [&](float us, float share) { return rest == 0 ? 0.f : full ? us * behind + share * (1.f - behind) : us; };
    float us;
    if (tma) {
      const float share = c.full * wave;
      us = (mine + c.start) * (c.full * static_cast<float>(full) + last_wave(fmaxf(full ? c.part_behind : c.part, share), share));
      us += longer * c.alone;
      if (s > 1) us += s <= kMaxClusterSplits && waves <= 0.9375f ? c.cluster : c.add + c.add_split * s + c.add_wave * group * waves;
    } else {
      us = (mine * (static_cast<float>(full) + last_wave(1.f, wave)) + longer) * tile;
      if (s > 1) us += 2.f + 0.08f * s + 0.8f * waves;
    }
    if (s == 1 || us < best_us) best = s, best_us = us;
  }
  if (even) {
    const float waves = static_cast<float>(pairs) / static_cast<float>(chip), each = waves * mean * static_cast<float>(tiles);  // tiles per CTA
    const float parts = fmaxf(0.f, static_cast<float>(tiles) / fmaxf(each, 1.f) - 1.f);
    const float us = c.full * each + c.even + c.even_pair * waves + c.even_part * pxl::ceil_div(group, 4) * parts +
                     (1.f - mean) * (c.even_short * waves + c.even_each * each);
    if (us < c.even_margin * best_us) best = pairs >= chip ? 2 : static_cast<int>((2 * chip + pairs - 1) / pairs);
  }
  return best;
}

PXL_EXPORT int pxl_attn_decode_splits(int B, int Hq, int Hkv, int D, int page_size, int cache_fp8, int max_ctx) {
  return pxl_attn_decode_splits_of(B, Hq, Hkv, D, page_size, cache_fp8, max_ctx, 0);
}

namespace {
constexpr int kDecSmem = 1024 + kDecStages * 2 * TILE * 128 * 2 + 128 + SplitParts::kFloats * 4,
              kE4Smem = 1024 + kE4Stages * 2 * kE4Tile + 128 + SplitParts::kFloats * 4;

// Clusters of `splits` CTAs of a kernel that are on the chip at once; asked for once per device and size.
template <auto Kernel>
int resident_clusters(int splits, int smem) {
  static std::atomic<int> known[64][kMaxClusterSplits + 1];  // count + 1
  std::atomic<int>& entry = known[pxl_host::current_device_slot()][splits];
  if (const int n = entry.load(std::memory_order_relaxed)) return n - 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1, 1, splits);
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(splits);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (set_smem(Kernel, smem) || cudaOccupancyMaxActiveClusters(&n, Kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  entry.store(n + 1, std::memory_order_relaxed);
  return n;
}

// Whether the splits of `pairs` (sequence, key head) pairs add their results inside clusters: where all of them are on the chip at
// once. Then the reduction's launch is saved (8 rows x 8 key heads x 777 keys in 4 splits: 10.9 us for the two kernels, 9.9 for the
// one). A cluster that has to wait waits for as many places at once, which costs more than that: 8 rows x 8 key heads x 2100 keys
// in 5 splits 20.8 and 24.5 us, 48 x 4 in 2 splits 48.0 and 49.7.
template <auto Together>
bool splits_together(int64_t pairs, int splits, int smem) {
  return splits > 1 && splits <= kMaxClusterSplits && pairs <= resident_clusters<Together>(splits, smem);
}

// Whether a step's tiles are dealt out evenly (attn_decode_even_kernel): the workspace of `splits` holds two results per CTA.
bool decode_even(int64_t pairs, int splits, int group, const float* workspace) {
  return splits > 1 && group <= 8 && pairs * splits >= 4ll * pxl_host::num_sms() && (reinterpret_cast<uintptr_t>(workspace) & 7) == 0;
}

template <bool F8, int SM>
int launch_decode_even(const CUtensorMap& tk, const CUtensorMap& tv, const bf16* q, int64_t q_stride, const int* block_tables,
                       const int* ctx_lens, bf16* out, float* workspace, const float* sinks, int B, int Hq, int Hkv, int page_size,
                       int max_blocks, int64_t num_blocks, float scale_log2, int window, int keep, float v_scale, const ScoreArgs& sa,
                       int* status, cudaStream_t stream) {
  static bool done[64] = {false};  // function attributes are per device
  const int dev = pxl_host::current_device_slot();
  if (!done[dev]) {
    if (set_smem(attn_decode_even_kernel<F8, SM>, kEvenSmem<F8>)) return PXL_ERR_CUDA;
    done[dev] = true;
  }
  const int ctas = 2 * pxl_host::num_sms();
  pxl_host::launch(attn_decode_even_kernel<F8, SM>, dim3(ctas), kDecThreads, kEvenSmem<F8>, stream, tk, tv, q, q_stride, block_tables,
                   ctx_lens, out, workspace, sinks, B, Hq, Hkv, page_size, max_blocks, num_blocks, scale_log2, window, keep, v_scale, sa,
                   status);
  pxl_host::launch(attn_decode_even_reduce_kernel<SM>, dim3(ctas - 1), 128, 0, stream, workspace, sinks, ctx_lens, out, B, Hq,
                   Hkv, window, keep, F8 ? kPShift : 0.f, v_scale);
  return check_launch();
}

// One kernel of the splits (grid.z): alone, as clusters that add their results, or with the reduction behind it.
template <auto Alone, auto Together, auto Reduce, typename... Args>
int launch_decode_splits(dim3 grid, int smem, int B, int Hq, const float* workspace, const float* sinks, void* out, cudaStream_t stream,
                         Args... args) {
  const int splits = static_cast<int>(grid.z);
  static bool done[64] = {false};  // function attributes are per device
  const int dev = pxl_host::current_device_slot();
  if (!done[dev]) {
    if (set_smem(Alone, smem) || set_smem(Together, smem)) return PXL_ERR_CUDA;
    done[dev] = true;
  }
  if (!splits_together<Together>(static_cast<int64_t>(grid.x) * grid.y, splits, smem)) {
    pxl_host::launch(Alone, grid, kDecThreads, smem, stream, args...);
    if (splits > 1) pxl_host::launch(Reduce, dim3(Hq, B), 128, 0, stream, workspace, sinks, static_cast<bf16*>(out), Hq, splits);
    return check_launch();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(splits);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pxl_host::chained() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, Together, args...) == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

int attn_decode_impl(const void* q, int64_t q_stride, const void* k_cache, const void* v_cache,
                     const int* block_tables, const int* ctx_lens, void* out, float* workspace,
                     const float* sinks, int B, int Hq, int Hkv, int D, int page_size, int max_blocks,
                     int64_t num_blocks, float scale, int window, int keep_first, int num_splits, int max_ctx,
                     bool cache_fp8, float k_scale, float v_scale, float softcap, const float* sig_bias, int* status,
                     pxl_stream_t stream) {
  if (B <= 0) return PXL_OK;
  const int mode = score_mode(softcap, sig_bias);
  const ScoreArgs sa = score_args(scale, softcap, sig_bias);
  if (cache_fp8 && mode != kPlain) return PXL_ERR_INVALID_ARG;
  if (Hkv <= 0 || Hq % Hkv || Hq / Hkv > 16 || page_size <= 0) return PXL_ERR_INVALID_ARG;
  if (num_splits <= 0) num_splits = pxl_attn_decode_splits(B, Hq, Hkv, D, page_size, cache_fp8, max_ctx);
  if (num_splits > 1 && workspace == nullptr) return PXL_ERR_INVALID_ARG;
  const float scale_log2 = scale * kLog2e;
  dim3 grid(Hkv, B, num_splits);
  if (!cache_fp8 && D == 128 && (page_size == 16 || page_size == 32 || page_size == 64) &&
      num_blocks * Hkv * page_size < (1ll << 31)) {
    // TMA-fed kernel: the cache is a 2-D matrix [blocks * Hkv * page, 128], one box = one page half
    CUtensorMap tk, tv;
    const uint64_t rows = static_cast<uint64_t>(num_blocks) * Hkv * page_size;
    if (!pxl_host::make_tmap_2d(&tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, k_cache, rows, 128, 128, page_size, 64) ||
        !pxl_host::make_tmap_2d(&tv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, v_cache, rows, 128, 128, page_size, 64))
      return PXL_ERR_TENSORMAP;
    auto run = [&](auto sm, auto high) {
      constexpr int M = decltype(sm)::value;
      constexpr bool H = decltype(high)::value;
      if (decode_even(static_cast<int64_t>(B) * Hkv, num_splits, Hq / Hkv, workspace))
        return launch_decode_even<false, M>(tk, tv, static_cast<const bf16*>(q), q_stride, block_tables, ctx_lens,
                                            static_cast<bf16*>(out), workspace, sinks, B, Hq, Hkv, page_size, max_blocks, num_blocks,
                                            scale_log2, window, keep_first, 1.f, sa, status, stream);
      return launch_decode_splits<attn_decode_tma_kernel<M, false, H>, attn_decode_tma_kernel<M, true, H>, attn_decode_reduce_kernel<128, M>>(
          grid, kDecSmem, B, Hq, workspace, sinks, out, stream, tk, tv, static_cast<const bf16*>(q), q_stride, block_tables, ctx_lens,
          static_cast<bf16*>(out), workspace, sinks, Hq, Hkv, page_size, max_blocks, num_blocks, scale_log2, window, keep_first,
          num_splits, sa, status);
    };
    auto go = [&](auto sm) { return Hq / Hkv > 8 ? run(sm, std::true_type{}) : run(sm, std::false_type{}); };
    if (mode == kSigmoid) return go(std::integral_constant<int, kSigmoid>{});
    if (mode == kCapped) return go(std::integral_constant<int, kCapped>{});
    return go(std::integral_constant<int, kPlain>{});
  }
  if (cache_fp8 && D == 128 && (page_size == 16 || page_size == 32 || page_size == 64) &&
      num_blocks * Hkv * page_size < (1ll << 31) &&
      ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) == 0) {
    CUtensorMap tk, tv;
    const uint64_t rows = static_cast<uint64_t>(num_blocks) * Hkv * page_size;
    if (!pxl_host::make_tmap_2d(&tk, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, k_cache, rows, 128, 128, page_size, 128) ||
        !pxl_host::make_tmap_2d(&tv, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, v_cache, rows, 128, 128, page_size, 128))
      return PXL_ERR_TENSORMAP;
    if (decode_even(static_cast<int64_t>(B) * Hkv, num_splits, Hq / Hkv, workspace))
      return launch_decode_even<true, kPlain>(tk, tv, static_cast<const bf16*>(q), q_stride, block_tables, ctx_lens,
                                              static_cast<bf16*>(out), workspace, sinks, B, Hq, Hkv, page_size, max_blocks, num_blocks,
                                              scale_log2 * k_scale, window, keep_first, v_scale, sa, status, stream);
    auto go = [&](auto high) {
      constexpr bool H = decltype(high)::value;
      return launch_decode_splits<attn_decode_e4m3_kernel<false, H>, attn_decode_e4m3_kernel<true, H>,
                                  attn_decode_reduce_kernel<128, kPlain>>(
        grid, kE4Smem, B, Hq, workspace, sinks, out, stream, tk, tv, static_cast<const bf16*>(q), q_stride, block_tables, ctx_lens,
        static_cast<bf16*>(out), workspace, sinks, Hq, Hkv, page_size, max_blocks, num_blocks, scale_log2 * k_scale, window, keep_first,
        num_splits, v_scale, status);
    };
    return Hq / Hkv > 8 ? go(std::true_type{}) : go(std::false_type{});
  }
#define PXL_DEC(DD, F8, M)                                                                       \
  {                                                                                              \
    constexpr int SMEM = 4 * TILE * DD * 2 > (4 * 16 * DD + 128) * 4 ? 4 * TILE * DD * 2         \
                                                                     : (4 * 16 * DD + 128) * 4;  \
    static bool done[64] = {false};                                                              \
    const int dev = pxl_host::current_device_slot();                                                       \
    if (!done[dev]) {                                                                            \
      if (set_smem(attn_decode_kernel<DD, F8, M>, SMEM)) return PXL_ERR_CUDA;                       \
      done[dev] = true;                                                                          \
    }                                                                                            \
    attn_decode_kernel<DD, F8, M><<<grid, 128, SMEM, stream>>>(                                  \
        static_cast<const bf16*>(q), q_stride, k_cache, v_cache, block_tables, ctx_lens,         \
        static_cast<bf16*>(out), workspace, sinks, Hq, Hkv, page_size, max_blocks, num_blocks,   \
        scale_log2 * k_scale, window, keep_first, num_splits, v_scale, sa, status);              \
    if (num_splits > 1)                                                                          \
      pxl_host::launch(attn_decode_reduce_kernel<DD, M>, dim3(Hq, B), DD, 0, stream, workspace,  \
                       sinks, static_cast<bf16*>(out), Hq, num_splits);                          \
  }
  if (D != 64 && D != 128) return PXL_ERR_INVALID_ARG;
  if (cache_fp8) {
    if (D == 128) PXL_DEC(128, true, kPlain)
    else PXL_DEC(64, true, kPlain)
  } else if (mode == kSigmoid) {
    if (D == 128) PXL_DEC(128, false, kSigmoid)
    else PXL_DEC(64, false, kSigmoid)
  } else if (mode == kCapped) {
    if (D == 128) PXL_DEC(128, false, kCapped)
    else PXL_DEC(64, false, kCapped)
  } else {
    if (D == 128) PXL_DEC(128, false, kPlain)
    else PXL_DEC(64, false, kPlain)
  }
#undef PXL_DEC
  return check_launch();
}
}  // namespace

PXL_EXPORT int pxl_attn_decode_launches(int B, int Hkv, int D, int page_size, int num_splits, int cache_fp8, float softcap,
                                        int sigmoid) {
  if (num_splits <= 1) return 1;
  if (D != 128 || (page_size != 16 && page_size != 32 && page_size != 64)) return 2;
  const int64_t pairs = static_cast<int64_t>(B) * Hkv;
  const bool one = cache_fp8       ? splits_together<attn_decode_e4m3_kernel<true, true>>(pairs, num_splits, kE4Smem)
                   : sigmoid       ? splits_together<attn_decode_tma_kernel<kSigmoid, true, true>>(pairs, num_splits, kDecSmem)
                   : softcap > 0.f ? splits_together<attn_decode_tma_kernel<kCapped, true, true>>(pairs, num_splits, kDecSmem)
                                   : splits_together<attn_decode_tma_kernel<kPlain, true, true>>(pairs, num_splits, kDecSmem);
  return one ? 1 : 2;
}

PXL_EXPORT int pxl_attn_decode(const void* q, int64_t q_stride, const void* k_cache,
                               const void* v_cache,
                               const int* block_tables, const int* ctx_lens, void* out,
                               float* workspace, const float* sinks, int B, int Hq, int Hkv, int D,
                               int page_size, int max_blocks, int64_t num_blocks, float scale,
                               int window, int keep_first, int num_splits, int max_ctx, float softcap,
                               const float* sig_bias, int* status, pxl_stream_t stream) {
  return attn_decode_impl(q, q_stride, k_cache, v_cache, block_tables, ctx_lens, out, workspace, sinks,
                          B, Hq, Hkv, D, page_size, max_blocks, num_blocks, scale, window, keep_first, num_splits,
                          max_ctx, false, 1.f, 1.f, softcap, sig_bias, status, stream);
}

// Decode attention over e4m3 caches written by pxl_qk_norm_rope_cache_fp8 / pxl_reshape_and_cache_fp8
// with the same scales, which are folded into the score scale (K) and the output normalisation (V). Head dim 128 and pages of 16, 32 or
// 64: bytes up to the fragments, f16 products (attn_decode_e4m3_kernel); other sizes widen the bytes to bf16 on their way into
// shared memory.
PXL_EXPORT int pxl_attn_decode_fp8(const void* q, int64_t q_stride, const void* k_cache,
                                   const void* v_cache, const int* block_tables,
                                   const int* ctx_lens, void* out, float* workspace,
                                   const float* sinks, int B, int Hq, int Hkv, int D, int page_size,
                                   int max_blocks, int64_t num_blocks, float scale, int window,
                                   int num_splits, int max_ctx, float k_scale, float v_scale,
                                   int* status, pxl_stream_t stream) {
  if (!(k_scale > 0.f) || !(v_scale > 0.f)) return PXL_ERR_INVALID_ARG;
  return attn_decode_impl(q, q_stride, k_cache, v_cache, block_tables, ctx_lens, out, workspace, sinks,
                          B, Hq, Hkv, D, page_size, max_blocks, num_blocks, scale, window, 0, num_splits,
                          max_ctx, true, k_scale, v_scale, 0.f, nullptr, status, stream);
}

namespace {
int attn_prefill_impl(const void* q, int64_t q_stride, const void* k_cache, const void* v_cache,
                      const int* block_tables, const int* cu_q, const int* ctx_lens, void* out,
                      int64_t out_stride, const float* sinks, int B, int max_q_len, int Hq, int Hkv,
                      int D, int page_size, int max_blocks, int64_t num_blocks, float scale,
                      int window, int keep_first, bool cache_fp8, float k_scale, float v_scale, float softcap,
                      const float* sig_bias, int* status, pxl_stream_t stream) {
  if (B <= 0 || max_q_len <= 0) return PXL_OK;
  const int mode = score_mode(softcap, sig_bias);
  const ScoreArgs sa = score_args(scale, softcap, sig_bias);
  if (cache_fp8 && mode != kPlain) return PXL_ERR_INVALID_ARG;
  if (Hkv <= 0 || Hq % Hkv || Hq / Hkv > 64 || page_size <= 0) return PXL_ERR_INVALID_ARG;
  const int G = Hq / Hkv;
  const int TQ = 64 / G;
  const float scale_log2 = scale * kLog2e;
  dim3 grid(pxl::ceil_div(max_q_len, TQ), Hkv, B);
#define PXL_PRE(DD, F8, M)                                                                       \
  {                                                                                              \
    constexpr int SMEM = 4 * TILE * DD * 2;                                                      \
    static bool done[64] = {false};                                                              \
    const int dev = pxl_host::current_device_slot();                                             \
    if (!done[dev]) {                                                                            \
      if (set_smem(attn_prefill_kernel<DD, F8, M>, SMEM)) return PXL_ERR_CUDA;                      \
      done[dev] = true;                                                                          \
    }                                                                                            \
    attn_prefill_kernel<DD, F8, M><<<grid, 128, SMEM, stream>>>(                                 \
        static_cast<const bf16*>(q), q_stride, k_cache, v_cache, block_tables, cu_q, ctx_lens,   \
        static_cast<bf16*>(out), out_stride, sinks, Hq, Hkv, page_size, max_blocks, num_blocks,  \
        scale_log2 * k_scale, window, keep_first, v_scale, sa, status);                          \
  }
  if (D != 64 && D != 128) return PXL_ERR_INVALID_ARG;
  if (cache_fp8) {
    if (D == 128) PXL_PRE(128, true, kPlain)
    else PXL_PRE(64, true, kPlain)
  } else if (mode == kSigmoid) {
    if (D == 128) PXL_PRE(128, false, kSigmoid)
    else PXL_PRE(64, false, kSigmoid)
  } else if (mode == kCapped) {
    if (D == 128) PXL_PRE(128, false, kCapped)
    else PXL_PRE(64, false, kCapped)
  } else {
    if (D == 128) PXL_PRE(128, false, kPlain)
    else PXL_PRE(64, false, kPlain)
  }
#undef PXL_PRE
  return check_launch();
}
}  // namespace

PXL_EXPORT int pxl_attn_prefill(const void* q, int64_t q_stride, const void* k_cache,
                                const void* v_cache, const int* block_tables, const int* cu_q,
                                const int* ctx_lens, void* out, int64_t out_stride,
                                const float* sinks, int B, int max_q_len, int Hq, int Hkv, int D,
                                int page_size, int max_blocks, int64_t num_blocks, float scale,
                                int window, int keep_first, float softcap, const float* sig_bias, int* status,
                                pxl_stream_t stream) {
  return attn_prefill_impl(q, q_stride, k_cache, v_cache, block_tables, cu_q, ctx_lens, out, out_stride,
                           sinks, B, max_q_len, Hq, Hkv, D, page_size, max_blocks, num_blocks, scale,
                           window, keep_first, false, 1.f, 1.f, softcap, sig_bias, status, stream);
}

// Prefix-aware prefill over e4m3 caches (see pxl_attn_decode_fp8).
PXL_EXPORT int pxl_attn_prefill_fp8(const void* q, int64_t q_stride, const void* k_cache,
                                    const void* v_cache, const int* block_tables, const int* cu_q,
                                    const int* ctx_lens, void* out, int64_t out_stride,
                                    const float* sinks, int B, int max_q_len, int Hq, int Hkv, int D,
                                    int page_size, int max_blocks, int64_t num_blocks, float scale,
                                    int window, float k_scale, float v_scale, int* status,
                                    pxl_stream_t stream) {
  if (!(k_scale > 0.f) || !(v_scale > 0.f)) return PXL_ERR_INVALID_ARG;
  return attn_prefill_impl(q, q_stride, k_cache, v_cache, block_tables, cu_q, ctx_lens, out, out_stride,
                           sinks, B, max_q_len, Hq, Hkv, D, page_size, max_blocks, num_blocks, scale,
                           window, 0, true, k_scale, v_scale, 0.f, nullptr, status, stream);
}

// ----------------------------------------------------------------------------------------
// Allocation-free decode attention (see pxl_noalloc.h). The scratch for the split-KV partial
// results is this file-scope device array. In host code `g_decode_static_scratch` is only a
// stand-in for the symbol, not a device address, so the launcher asks the runtime for the
// real address once per device and hands that pointer to the kernels.
static __device__ __align__(256) float g_decode_static_scratch[PXL_DECODE_STATIC_SCRATCH_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
// Written by whichever host thread asks first; two threads racing on the first call store the
// same value, and the atomic makes that store and the later loads well defined.
std::atomic<float*> g_static_scratch_addr[kMaxDevices];

// Device address of the scratch array on the current device, or nullptr on error.
float* static_scratch_ptr() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  float* known = g_static_scratch_addr[dev].load(std::memory_order_acquire);
  if (known == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_decode_static_scratch) != cudaSuccess || p == nullptr) {
      cudaGetLastError();  // leave no sticky error behind for the caller
      return nullptr;
    }
    known = static_cast<float*>(p);
    g_static_scratch_addr[dev].store(known, std::memory_order_release);
  }
  return known;
}
}  // namespace

PXL_EXPORT int pxl_attn_decode_static_scratch(const void* q, int64_t q_stride, const void* k_cache,
                                              const void* v_cache, const int* block_tables,
                                              const int* ctx_lens, void* out, const float* sinks,
                                              int B, int Hq, int Hkv, int D, int page_size,
                                              int max_blocks, int64_t num_blocks, float scale,
                                              int window, int num_splits, int* status,
                                              pxl_stream_t stream) {
  if (B <= 0) return PXL_OK;
  if (num_splits < 1 || Hq <= 0 || D <= 0) return PXL_ERR_INVALID_ARG;
  float* scratch = nullptr;
  if (num_splits > 1) {
    const int64_t need = static_cast<int64_t>(B) * Hq * num_splits * (D + 2);
    if (need > static_cast<int64_t>(PXL_DECODE_STATIC_SCRATCH_FLOATS)) return PXL_ERR_TOO_LARGE;
    scratch = static_scratch_ptr();
    if (scratch == nullptr) return PXL_ERR_CUDA;
  }
  // Every (sequence, head, split) partial that the reduction reads is written by the main
  // kernel of this same call, so the array needs no clearing between calls.
  return pxl_attn_decode(q, q_stride, k_cache, v_cache, block_tables, ctx_lens, out, scratch, sinks,
                         B, Hq, Hkv, D, page_size, max_blocks, num_blocks, scale, window, 0, num_splits,
                         0, 0.f, nullptr, status, stream);
}
