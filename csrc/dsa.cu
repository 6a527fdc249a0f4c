// DeepSeek sparse attention (V3.2 "lightning indexer"): key scoring, top-k selection, key store.
//
//   score[t, j] = sum_h relu(q_idx[t, h, :] . k_idx[j, :]) * w[t, h]      for j <= position(t)
//
// The reference scores one context token per threadgroup (dsa_indexer.metal:34-116, launch in
// dsa_indexer.cpp:153-196) and selects the top-k with a framework argpartition
// (parallax_extensions/ops.py:361-367). Here one CTA scores 128 keys for all index
// heads of a group of tokens with tensor-core MMAs, and a radix select picks the k best positions per query row
// without sorting.
#include "common.cuh"
#include "pxl_api.h"
#include "tc_issue.cuh"

namespace {
using namespace pxl;

constexpr int kDi = 128;          // index head dim
constexpr int kHiMax = 64;        // index heads handled per CTA (one pass)
constexpr int kKeyTile = 64;      // rows of the score matrix are padded to this
constexpr int kPitch = kDi + 8;   // smem row pitch (elements)

__device__ __forceinline__ int find_seq(const int* cu_q, int B, int t) {
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_q[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Row of the index cache that holds key kp of a sequence. An entry outside the cache or behind the table is reported and read as block 0.
__device__ __forceinline__ int64_t key_row(const int* bt, int kp, int page, int max_blocks, int64_t num_blocks, int* status) {
  const int bi = kp / page;
  int blk = bi < max_blocks ? bt[bi] : -1;
  if (blk < 0 || blk >= num_blocks) {
    if (status) atomicCAS(status, 0, PXL_DEV_BAD_INDEX);
    blk = 0;
  }
  return static_cast<int64_t>(blk) * page + kp % page;
}

// One CTA scores 128 keys for a group of consecutive tokens. Keys are the rows of the products and index heads the columns: a
// warp keeps the fragments of its 32 keys in registers for as long as the tokens are of one sequence (a token costs its queries,
// 16 KB of shared memory, and no key is read again), and the weighted sum over the heads stays inside a thread up to two
// shuffles. (Decoded tokens, other numbers of heads; prompts of 32 or 64 heads: dsa_scores_tc_kernel.) With a CTA per token and 64 keys, queries and keys were loaded anew for each 64 x 64 product and the sum over the
// heads went through shuffles of every accumulator and shared-memory atomics: 640 us for 1000 tokens x 5500 keys beside 16 x 8000,
// 324 us this way.
constexpr int kScoreKeys = 128, kScoreThreads = 128;

struct ScoreSmem {
  bf16 k[kScoreKeys * kPitch];
  bf16 q[2][kHiMax * kPitch];
};

// grid (key tiles, groups of `group` tokens); columns [0, width) of a row of scores are written
__global__ void __launch_bounds__(kScoreThreads) dsa_scores_kernel(const bf16* __restrict__ q, const float* __restrict__ w,
                                                                   const bf16* __restrict__ cache,
                                                                   const int* __restrict__ block_tables,
                                                                   const int* __restrict__ cu_q,
                                                                   const int* __restrict__ positions,
                                                                   float* __restrict__ scores, int64_t ld_scores, int width, int T,
                                                                   int B, int Hi, int max_blocks, int page, int group,
                                                                   int64_t num_blocks, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t raw[];
  ScoreSmem& sm = *reinterpret_cast<ScoreSmem*>(raw);
  const int j0 = blockIdx.x * kScoreKeys;
  const int first = blockIdx.y * group, last = first + group < T ? first + group : T;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, qd = lane & 3, mi = lane >> 3;
  auto load_q = [&](int t, int buf) {
    if (t < last) {
      for (int c = tid; c < kHiMax * (kDi / 8); c += kScoreThreads) {
        const int r = c / (kDi / 8), ch = c % (kDi / 8);
        cp_async_16(smem_u32(&sm.q[buf][r * kPitch + ch * 8]), q + (static_cast<size_t>(t) * Hi + (r < Hi ? r : 0)) * kDi + ch * 8,
                    r < Hi);
      }
    }
    cp_async_commit();
  };
  int seq = -1, seq_end = first;  // tokens of the sequence in registers: up to seq_end
  uint32_t kf[2][kDi / 16][4];
  load_q(first, 0);
  for (int t = first; t < last; ++t) {
    const int buf = (t - first) & 1, pos = positions[t];
    __syncthreads();  // the other buffer's queries were read
    load_q(t + 1, buf ^ 1);
    float* out = scores + static_cast<size_t>(t) * ld_scores;
    const bool seen = j0 <= pos;
    if (seen && t >= seq_end) {
      seq = cu_q ? find_seq(cu_q, B, t) : t;
      seq_end = cu_q ? cu_q[seq + 1] : t + 1;
      if (seq_end > T) seq_end = T;
      int limit = pos;  // what the group's tokens of the sequence see, in whatever order they are
      for (int i = t + 1; i < seq_end && i < last; ++i) limit = max(limit, positions[i]);
      const int* bt = block_tables + static_cast<size_t>(seq) * max_blocks;
      constexpr int kStep = kScoreThreads / 16;  // keys per step, two of a warp; lane l looks up one of them for step l / 2
      const int mine = j0 + (lane >> 1) * kStep + warp * 2 + (lane & 1);
      const int64_t at = mine <= limit ? key_row(bt, mine, page, max_blocks, num_blocks, status) : 0;
#pragma unroll 4
      for (int i = 0; i < kScoreKeys / kStep; ++i) {
        const int r = i * kStep + warp * 2 + (lane >> 4), ch = lane & 15;
        const int64_t key = __shfl_sync(0xffffffffu, at, 2 * i + (lane >> 4));
        cp_async_16(smem_u32(&sm.k[r * kPitch + ch * 8]), cache + key * kDi + ch * 8, j0 + r <= limit);
      }
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int ks = 0; ks < kDi / 16; ++ks)
          ldmatrix_x4(kf[m][ks], smem_u32(&sm.k[(warp * 32 + m * 16 + (lane & 15)) * kPitch + ks * 16 + (lane >> 4) * 8]));
    } else {
      cp_async_wait<1>();
      __syncthreads();
    }
    float part[2][2] = {};
    if (seen) {
      const float* wt = w + static_cast<size_t>(t) * Hi;
#pragma unroll 1
      for (int np = 0; np < kHiMax / 16; ++np) {  // 16 heads
        float s[2][2][4] = {};
#pragma unroll
        for (int ks = 0; ks < kDi / 16; ++ks) {
          uint32_t qb[4];
          ldmatrix_x4(qb, smem_u32(&sm.q[buf][(np * 16 + (mi >> 1) * 8 + (lane & 7)) * kPitch + ks * 16 + (mi & 1) * 8]));
          const uint32_t b0[2] = {qb[0], qb[1]}, b1[2] = {qb[2], qb[3]};
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            mma_m16n8k16_bf16(s[m][0], kf[m][ks], b0);
            mma_m16n8k16_bf16(s[m][1], kf[m][ks], b1);
          }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const int h = np * 16 + n * 8 + qd * 2;
          const float w0 = h < Hi ? wt[h] : 0.f, w1 = h + 1 < Hi ? wt[h + 1] : 0.f;
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              part[m][e] += fmaxf(s[m][n][2 * e], 0.f) * w0 + fmaxf(s[m][n][2 * e + 1], 0.f) * w1;
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float v = part[m][e];
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        const int j = j0 + warp * 32 + m * 16 + e * 8 + g;
        if (qd == 0 && j < width) out[j] = j <= pos ? v : -INFINITY;
      }
  }
  cp_async_wait<0>();
}

// ---- the same on the 5th-generation tensor cores: prompts, 32 or 64 index heads -----------------------------------
// 256 keys, two accumulators of 128 rows, stay in shared memory; the queries of 128 / HI tokens are the 128 columns of a product and
// stream past them, 32 KB per 1024 clocks of products (a single accumulator of keys would take 64 bytes a clock, all that an SM gets
// from L2). A thread of the sixteen warps behind the products has one key and half of the tokens: 64 columns of its row, clipped, times the heads'
// weights, no exchange. Two pairs of accumulators, so that sums and products overlap: 256 columns x 2 of tensor memory. Warp 0 loads queries,
// warp 1 issues products; the keys come through the other warps, whose waits for the last product also free them. Bound by the
// products, 54 us for the 90 GFLOP of 1000 tokens x 5500 keys at the rate of plain ones, and by the 2.5 instructions per score of the
// other warps, which take as long: 287 us with mma.sync, 115 with eight such warps, 99 now (0.91 PFLOP/s); 4096 x 14336 2909 and 992;
// 32 heads 284 and 60.
constexpr int kTcTokens = 16;  // fewest tokens of a step's prompts
constexpr int kTcKeys = 256, kTcCols = 128, kTcStages = 3, kTcWarps = 16, kTcThreads = 64 + 32 * kTcWarps;
struct TcScoreSmem {
  uint8_t k[2][2][128 * 128];             // [accumulator][half of the columns]: 128-byte swizzled rows
  uint8_t q[kTcStages][2][kTcCols * 128];
  uint64_t qfull[kTcStages], qempty[kTcStages], afull[2], aempty[2], keys;
  uint32_t tmem;
  int abort_flag;
};

// The tokens [first, last) of a CTA: runs of one sequence, and of those, tiles of TOK tokens that see some key of the CTA.
template <int TOK, typename Run, typename Tile>
__device__ __forceinline__ void score_tiles(const int* positions, const int* cu_q, int B, int first, int last, int j0, Run run, Tile tile) {
  for (int t = first; t < last;) {
    const int seq = find_seq(cu_q, B, t), end = min(max(cu_q[seq + 1], t + 1), last);
    if (!run(seq, t, end)) return;
    for (int i = t; i < end; i += TOK) {
      bool seen = false;
#pragma unroll
      for (int e = 0; e < TOK; ++e) seen |= i + e < end && __ldg(positions + i + e) >= j0;
      if (!tile(i, min(TOK, end - i), seen)) return;
    }
    t = end;
  }
}

template <int HI>
__global__ void __launch_bounds__(kTcThreads, 1)
dsa_scores_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const float* __restrict__ w, const bf16* __restrict__ cache,
                     const int* __restrict__ block_tables, const int* __restrict__ cu_q, const int* __restrict__ positions,
                     float* __restrict__ scores, int64_t ld_scores, int width, int T, int B, int max_blocks, int page, int group,
                     int64_t num_blocks, int* status) {
  constexpr int TOK = kTcCols / HI;
  extern __shared__ uint8_t raw[];
  TcScoreSmem& sm = *reinterpret_cast<TcScoreSmem*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j0 = blockIdx.x * kTcKeys;
  const int first = (gridDim.y - 1 - blockIdx.y) * group, last = min(T, first + group);  // late tokens, which see the most, begin
  volatile int* abort_flag = &sm.abort_flag;
  if (threadIdx.x == 0) {
    sm.abort_flag = 0;
    for (int i = 0; i < kTcStages; ++i) mbar_init(smem_u32(&sm.qfull[i]), 1), mbar_init(smem_u32(&sm.qempty[i]), 1);
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&sm.afull[i]), 1), mbar_init(smem_u32(&sm.aempty[i]), kTcWarps);
    mbar_init(smem_u32(&sm.keys), kTcWarps);
    mbar_fence_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_q);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&sm.tmem), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sm.tmem;
  pdl_wait();
  pdl_launch_dependents();

  bool ok = true;
  if (warp == 0) {
    const uint32_t leader = elect_leader();
    int stage = 0;
    uint32_t phase = 1;
    score_tiles<TOK>(positions, cu_q, B, first, last, j0, [&](int, int, int) { return true; }, [&](int t, int, bool seen) {
      if (!seen) return true;
      const uint32_t full = smem_u32(&sm.qfull[stage]);
      ok = wait_warp(smem_u32(&sm.qempty[stage]), phase, abort_flag, status, PXL_DEV_TIMEOUT_EMPTY);
      if (!ok) return false;
      expect_tx(full, 2 * kTcCols * 128, leader);
      tma_box(smem_u32(sm.q[stage][0]), &tm_q, full, 0, t * HI, leader);
      tma_box(smem_u32(sm.q[stage][1]), &tm_q, full, 64, t * HI, leader);
      if (++stage == kTcStages) stage = 0, phase ^= 1;
      return true;
    });
  } else if (warp == 1) {
    const uint32_t leader = elect_leader();
    constexpr uint32_t idesc = umma_idesc(128, kTcCols, 1, 1);
    const uint64_t dk = umma_desc_k_sw128(smem_u32(sm.k)), dq = umma_desc_k_sw128(smem_u32(sm.q));
    int stage = 0, buf = 0;
    uint32_t phase = 0, aphase = 1, kphase = 0;
    bool fresh = true;
    score_tiles<TOK>(positions, cu_q, B, first, last, j0,
                     [&](int, int, int) {
                       fresh = true;
                       return true;
                     },
                     [&](int, int, bool seen) {
                       if (!seen) return true;
                       if (fresh) {
                         ok = wait_warp(smem_u32(&sm.keys), kphase, abort_flag, status, PXL_DEV_TIMEOUT_FULL);
                         kphase ^= 1;
                         fresh = false;
                       }
                       ok = ok && wait_warp(smem_u32(&sm.aempty[buf]), aphase, abort_flag, status, PXL_DEV_TIMEOUT_TMEM_EMPTY);
                       ok = ok && wait_warp(smem_u32(&sm.qfull[stage]), phase, abort_flag, status, PXL_DEV_TIMEOUT_FULL);
                       if (!ok) return false;
                       tc_fence_after_sync();
                       const uint64_t b = dq + stage * (2 * kTcCols * 128 >> 4);
#pragma unroll
                       for (int m = 0; m < 2; ++m)
#pragma unroll
                         for (int k = 0; k < 8; ++k)
                           mma_ss(tmem + (buf * 2 + m) * kTcCols, dk + ((m * 2 + k / 4) * 128 * 128 >> 4) + (k & 3) * 2,
                                  b + ((k / 4) * kTcCols * 128 >> 4) + (k & 3) * 2, idesc, k > 0 ? 1u : 0u, leader);
                       commit(smem_u32(&sm.qempty[stage]), leader);
                       commit(smem_u32(&sm.afull[buf]), leader);
                       if (++stage == kTcStages) stage = 0, phase ^= 1;
                       buf ^= 1;
                       if (buf == 0) aphase ^= 1;
                       return true;
                     });
  } else {
    const int m = (warp - 2) >> 2 & 1, e0 = (warp - 2) / 8 * (TOK / 2), row = m * 128 + (warp & 3) * 32 + lane, j = j0 + row;  // warp % 4: the lanes of tensor memory
    int buf = 0;
    uint32_t aphase = 0;
    score_tiles<TOK>(
        positions, cu_q, B, first, last, j0,
        [&](int seq, int t, int end) {  // the keys of a sequence, as far as these tokens see; all products with the last ones are done
          int limit = -1;
          for (int i = t + lane; i < end; i += 32) limit = max(limit, positions[i]);
          limit = __reduce_max_sync(0xffffffffu, limit);
          if (limit < j0) return true;
          const int* bt = block_tables + static_cast<size_t>(seq) * max_blocks;
          constexpr int kStep = 2 * kTcWarps;  // keys per step, two of a warp; lane l looks up one of them for step l / 2
          const int first_key = (warp - 2) * 2, mine = j0 + (lane >> 1) * kStep + first_key + (lane & 1);
          const int64_t at = lane < 2 * kTcKeys / kStep && mine <= limit ? key_row(bt, mine, page, max_blocks, num_blocks, status) : 0;
#pragma unroll 4
          for (int i = 0; i < kTcKeys / kStep; ++i) {
            const int r = i * kStep + first_key + (lane >> 4), ch = lane & 15;
            const int64_t key = __shfl_sync(0xffffffffu, at, 2 * i + (lane >> 4));
            cp_async_16(smem_u32(sm.k[r >> 7][ch >> 3]) + (r & 127) * 128 + (((ch & 7) ^ (r & 7)) << 4), cache + key * kDi + ch * 8,
                        j0 + r <= limit);
          }
          cp_async_commit();
          cp_async_wait<0>();
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sm.keys));
          return true;
        },
        [&](int t, int n, bool seen) {
          float* out = scores + static_cast<size_t>(t) * ld_scores + j;
          if (!seen) {
            for (int e = e0; e < e0 + TOK / 2; ++e)
              if (e < n && j < width) out[e * ld_scores] = -INFINITY;
            return true;
          }
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sm.afull[buf]), aphase, abort_flag, status, PXL_DEV_TIMEOUT_TMEM_FULL)) != 0;
          if (!ok) return false;
          tc_fence_after_sync();
          const uint32_t acc = tmem + (buf * 2 + m) * kTcCols + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll
          for (int i = 0; i < TOK / 2; ++i) {
            const int e = e0 + i, te = min(t + e, T - 1);
            const float4* wt = reinterpret_cast<const float4*>(w + static_cast<size_t>(te) * HI);
            float sum[4] = {};
#pragma unroll
            for (int c = 0; c < HI; c += 32) {
              uint32_t r[32];
              tmem_ld_32x32b_x32(acc + e * HI + c, r);
              tmem_ld_wait();
#pragma unroll
              for (int v = 0; v < 8; ++v) {
                const float4 f = __ldg(wt + c / 4 + v);
                sum[0] = fmaf(fmaxf(__uint_as_float(r[4 * v]), 0.f), f.x, sum[0]);
                sum[1] = fmaf(fmaxf(__uint_as_float(r[4 * v + 1]), 0.f), f.y, sum[1]);
                sum[2] = fmaf(fmaxf(__uint_as_float(r[4 * v + 2]), 0.f), f.z, sum[2]);
                sum[3] = fmaf(fmaxf(__uint_as_float(r[4 * v + 3]), 0.f), f.w, sum[3]);
              }
            }
            if (i == TOK / 2 - 1) {  // the accumulator is read
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&sm.aempty[buf]));
            }
            if (e < n && j < width) out[e * ld_scores] = j <= __ldg(positions + te) ? (sum[0] + sum[1]) + (sum[2] + sum[3]) : -INFINITY;
          }
          buf ^= 1;
          if (buf == 0) aphase ^= 1;
          return true;
        });
  }
  __syncwarp();
  if (!ok || *abort_flag) __nanosleep(200000);  // loads that are still in flight must land before the shared memory is released
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

__device__ __forceinline__ uint32_t order_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// One CTA per query row: radix select of the k largest scores among positions [0, pos], eight bits a pass. Rows of up to 8192 scores
// are read once and stay in registers (HELD). What it takes is chains, not bytes (24 KB a row): lanes that fall into one bin add once
// (the first bits of scores are few different ones), a warp finds the bin of the k-th score with one scan, and places in the list are
// given out a warp at a time. One thread per score and per bin, 1000 rows of 5500 scores and k = 2048 took 62 us, 16 of 8000 35 us;
// 40 and 17 us now (64 rows of 60000, which do not fit the registers: 125 and 97).
constexpr int kTopkThreads = 512, kTopkHeld = 16;
template <bool HELD>
__global__ void __launch_bounds__(kTopkThreads) topk_select_kernel(const float* __restrict__ scores, int64_t ld,
                                                                   const int* __restrict__ positions, int k, int* __restrict__ out,
                                                                   int64_t ld_out) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ int hist[256];
  __shared__ uint32_t s_prefix;
  __shared__ int s_remaining, s_gt, s_eq;
  const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const int n = positions[t] + 1;
  const float* s = scores + static_cast<size_t>(t) * ld;
  int* o = out + static_cast<size_t>(t) * ld_out;
  if (n <= k) {  // nothing to select: the attention kernel reads "row starts with -1" as dense
    for (int i = tid; i < k; i += kTopkThreads) o[i] = -1;
    return;
  }
  const bool held = HELD && n <= kTopkThreads * kTopkHeld;
  uint32_t keys[HELD ? kTopkHeld : 1];
  if constexpr (HELD) {
#pragma unroll
    for (int c = 0; c < kTopkHeld; ++c) {
      const int i = c * kTopkThreads + tid;
      keys[c] = held && i < n ? order_key(s[i]) : 0u;
    }
  }
  auto each = [&](auto f) {  // f(position, whether it is one, key), whole warps
    if constexpr (HELD) {
      if (held) {
#pragma unroll
        for (int c = 0; c < kTopkHeld; ++c)
          if (c * kTopkThreads < n) f(c * kTopkThreads + tid, c * kTopkThreads + tid < n, keys[c]);
        return;
      }
    }
    for (int c = 0; c < n; c += 4 * kTopkThreads) {
      uint32_t u[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = c + e * kTopkThreads + tid;
        u[e] = i < n ? order_key(s[i]) : 0u;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + e * kTopkThreads < n) f(c + e * kTopkThreads + tid, c + e * kTopkThreads + tid < n, u[e]);
    }
  };
  uint32_t prefix = 0, mask = 0;
  int remaining = k;
  for (int shift = 24; shift >= 0; shift -= 8) {
    if (tid < 256) hist[tid] = 0;
    if (tid == 0) s_gt = s_eq = 0;
    __syncthreads();
    each([&](int, bool is, uint32_t u) {
      const bool in = is && (u & mask) == prefix;
      const uint32_t bin = (u >> shift) & 255;
      if (shift < 24) {  // (many bins: matching costs more than it saves)
        if (in) atomicAdd(&hist[bin], 1);
        return;
      }
      const uint32_t lanes = __ballot_sync(0xffffffffu, in);
      if (in) {
        const uint32_t same = __match_any_sync(lanes, bin);
        if (lane == __ffs(same) - 1) atomicAdd(&hist[bin], __popc(same));
      }
    });
    __syncthreads();
    if (tid < 32) {  // lane l: bins 255 - 8 l downwards; the first at which the count from above reaches `remaining`
      int mine[8], sum = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += mine[i] = hist[255 - 8 * lane - i];
      int upto = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += up;
      }
      const uint32_t reach = __ballot_sync(0xffffffffu, upto >= remaining);
      if (lane == (reach ? __ffs(reach) - 1 : 31)) {
        int above = upto - sum, bin = 255 - 8 * lane;
#pragma unroll
        for (int i = 0; i < 7; ++i) {
          if (above + mine[i] >= remaining) break;
          above += mine[i];
          --bin;
        }
        s_prefix = prefix | (static_cast<uint32_t>(bin) << shift);
        s_remaining = remaining - above;
      }
    }
    __syncthreads();
    prefix = s_prefix;
    remaining = s_remaining;
    mask |= 0xffu << shift;
  }
  const int n_gt = k - remaining;  // `remaining` of the keys equal to the threshold still fit
  each([&](int i, bool is, uint32_t u) {
    const uint32_t gt = __ballot_sync(0xffffffffu, is && u > prefix), eq = __ballot_sync(0xffffffffu, is && u == prefix);
    const uint32_t below = (1u << lane) - 1;
    int at_gt = 0, at_eq = 0;
    if (lane == 0) {
      if (gt) at_gt = atomicAdd(&s_gt, __popc(gt));
      if (eq) at_eq = atomicAdd(&s_eq, __popc(eq));
    }
    at_gt = __shfl_sync(0xffffffffu, at_gt, 0) + __popc(gt & below);
    at_eq = __shfl_sync(0xffffffffu, at_eq, 0) + __popc(eq & below);
    if (is && u > prefix) {
      if (at_gt < n_gt) o[at_gt] = i;
    } else if (is && u == prefix) {
      if (at_eq < remaining) o[n_gt + at_eq] = i;
    }
  });
}

__global__ void store_rows_kernel(const bf16* __restrict__ src, int64_t ld, const int64_t* __restrict__ slots,
                                  bf16* __restrict__ cache, int D, int64_t num_slots, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const int64_t slot = slots[t];
  if (slot < 0) return;
  if (slot >= num_slots) {
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, PXL_DEV_BAD_INDEX);
    return;
  }
  for (int i = threadIdx.x; i < D / 8; i += blockDim.x)
    st_bf16x8(cache + slot * D + i * 8, ld_bf16x8(src + t * ld + i * 8));
}

// Indexer pre-processing of one step, one block (128 threads) per token:
//   q_idx[t, h, :R]  <- interleaved RoPE at position(t), in place (every index head)
//   cache[slot(t)]   <- RoPE(LayerNorm(kv[t, k_off : k_off + Di]) * w + b) on the first R dims
//   w_out[t, h]      <- kv[t, w_off + h] * w_scale                              (fp32)
// The model code did this with five framework calls per layer (layer norm, two rotations, two concatenations)
// and a separate store; semantics follow the reference's indexer (deepseek_v32.py:84-238).
__global__ void __launch_bounds__(128)
dsa_index_prep_kernel(bf16* __restrict__ q_idx, int64_t ldq, const bf16* __restrict__ kv, int64_t ldkv, int k_off,
                      int w_off, const bf16* __restrict__ ln_w, const bf16* __restrict__ ln_b, float ln_eps,
                      const float* __restrict__ cos_sin, const int* __restrict__ positions, int max_pos,
                      const int64_t* __restrict__ slots, bf16* __restrict__ cache, int64_t num_slots,
                      float* __restrict__ w_out, float w_scale, int Hi, int R, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float red[32];
  __shared__ float y_s[kDi];
  const int t = blockIdx.x, d = threadIdx.x;
  const int pos = positions[t];
  const bool pos_ok = pos >= 0 && (max_pos <= 0 || pos < max_pos);
  if (!pos_ok && d == 0 && status) atomicCAS(status, 0, PXL_DEV_BAD_POSITION);
  const float* cs = cos_sin + static_cast<size_t>(pos_ok ? pos : 0) * R;
  const int half = R >> 1;
  // ---- head weights
  if (d < Hi) w_out[static_cast<size_t>(t) * Hi + d] = __bfloat162float(kv[t * ldkv + w_off + d]) * w_scale;
  // ---- queries: one thread per (head, pair)
  if (pos_ok) {
    for (int idx = d; idx < Hi * half; idx += blockDim.x) {
      const int h = idx / half, i = idx % half;
      bf16* p = q_idx + t * ldq + static_cast<int64_t>(h) * kDi + 2 * i;
      const float x0 = __bfloat162float(p[0]), x1 = __bfloat162float(p[1]);
      const float c = cs[i], sn = cs[half + i];
      p[0] = __float2bfloat16(x0 * c - x1 * sn);
      p[1] = __float2bfloat16(x0 * sn + x1 * c);
    }
  }
  // ---- key: layer norm over the Di dims (two passes in fp32), rotation, store
  const float x = __bfloat162float(kv[t * ldkv + k_off + d]);
  const float mean = block_reduce_sum(x, red) * (1.f / kDi);
  const float dx = x - mean;
  const float var = block_reduce_sum(dx * dx, red) * (1.f / kDi);
  const float y = dx * rsqrtf(var + ln_eps) * __bfloat162float(ln_w[d]) + (ln_b ? __bfloat162float(ln_b[d]) : 0.f);
  y_s[d] = y;
  __syncthreads();
  float out = y;
  if (pos_ok && d < R) {
    const int i = d >> 1;
    const float c = cs[i], sn = cs[half + i];
    out = (d & 1) ? y_s[d - 1] * sn + y * c : y * c - y_s[d + 1] * sn;
  }
  const int64_t slot = slots[t];
  if (slot < 0) return;
  if (slot >= num_slots) {
    if (d == 0 && status) atomicCAS(status, 0, PXL_DEV_BAD_INDEX);
    return;
  }
  cache[slot * kDi + d] = __float2bfloat16(out);
}

}  // namespace

PXL_EXPORT int pxl_dsa_index_prep(void* q_idx, int64_t ldq, const void* kv, int64_t ldkv, int k_off, int w_off,
                                  const void* ln_w, const void* ln_b, float ln_eps, const float* cos_sin,
                                  const int* positions, int max_pos, const int64_t* slots, void* cache,
                                  int64_t num_slots, float* w_out, float w_scale, int T, int Hi, int Di, int R,
                                  int* status, cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (Di != kDi || Hi <= 0 || Hi > 128 || R <= 0 || R > Di || (R & 1)) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(dsa_index_prep_kernel, T, 128, 0, stream, static_cast<pxl::bf16*>(q_idx), ldq, static_cast<const pxl::bf16*>(kv),
                                               ldkv, k_off, w_off, static_cast<const pxl::bf16*>(ln_w),
                                               static_cast<const pxl::bf16*>(ln_b), ln_eps, cos_sin, positions,
                                               max_pos, slots, static_cast<pxl::bf16*>(cache), num_slots, w_out,
                                               w_scale, Hi, R, status);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

namespace {
int launch_scores(const void* q, const float* w, const void* index_cache, const int* block_tables, const int* cu_q, const int* positions,
                  float* scores, int64_t ld_scores, int T, int B, int Hi, int Di, int max_blocks, int page, int max_ctx,
                  int64_t num_blocks, int* status, cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (Di != kDi || Hi <= 0 || Hi > kHiMax || max_ctx <= 0) return PXL_ERR_INVALID_ARG;
  const int width = pxl::ceil_div(max_ctx, kKeyTile) * kKeyTile;  // (the last tile of 128 keys may reach past it)
  if (width > ld_scores) return PXL_ERR_INVALID_ARG;
  static bool done[64] = {false};
  const int dev = pxl_host::current_device_slot();
  if (!done[dev]) {
    if (cudaFuncSetAttribute(dsa_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(ScoreSmem)) != cudaSuccess)
      return PXL_ERR_CUDA;
    done[dev] = true;
  }
  const int tiles = pxl::ceil_div(max_ctx, kScoreKeys);
  // prompts: as many tokens per CTA as still leave every SM three of them, and no more than bring anything; decoded tokens have
  // a sequence each
  int group = cu_q ? static_cast<int>(static_cast<int64_t>(T) * tiles / (3 * pxl_host::num_sms())) : 1;
  group = group < 1 ? 1 : group > 16 ? 16 : group;
  while (pxl::ceil_div(T, group) > 65535) group *= 2;
  pxl_host::launch(dsa_scores_kernel, dim3(tiles, pxl::ceil_div(T, group)), kScoreThreads, sizeof(ScoreSmem), stream,
                   static_cast<const pxl::bf16*>(q), w, static_cast<const pxl::bf16*>(index_cache), block_tables, cu_q, positions, scores,
                   ld_scores, width, T, B, Hi, max_blocks, page, group, num_blocks, status);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

template <int HI>
int launch_scores_tc(const void* q, const float* w, const void* cache, const int* block_tables, const int* cu_q, const int* positions,
                     float* scores, int64_t ld_scores, int width, int T, int B, int max_blocks, int page, int max_ctx,
                     int64_t num_blocks, int* status, cudaStream_t stream) {
  constexpr int smem = 1024 + sizeof(TcScoreSmem);
  static bool done[64] = {false};
  const int dev = pxl_host::current_device_slot();
  if (!done[dev]) {
    if (cudaFuncSetAttribute(dsa_scores_tc_kernel<HI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return PXL_ERR_CUDA;
    done[dev] = true;
  }
  CUtensorMap tq;
  if (!pxl_host::make_tmap_2d(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q, static_cast<uint64_t>(T) * HI, kDi, kDi, kTcCols, 64))
    return PXL_ERR_TENSORMAP;
  // A prompt without a cached part leaves half of the tiles empty: eight waves where a CTA still has 48 tokens for its keys, two
  // otherwise, and the late tokens' begin (4096 tokens of 4096: 329 us in two waves, 238 in eight).
  const int tiles = pxl::ceil_div(max_ctx, kTcKeys), tok = kTcCols / HI;
  int groups = 8 * pxl_host::num_sms() / tiles;
  if (groups < 1 || T / groups < 48) groups = 2 * pxl_host::num_sms() / tiles;
  groups = groups < 1 ? 1 : groups;
  const int group = pxl::ceil_div(pxl::ceil_div(T, groups), tok) * tok;
  pxl_host::launch(dsa_scores_tc_kernel<HI>, dim3(tiles, pxl::ceil_div(T, group)), kTcThreads, smem, stream, tq, w,
                   static_cast<const pxl::bf16*>(cache), block_tables, cu_q, positions, scores, ld_scores, width, T, B, max_blocks, page,
                   group, num_blocks, status);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}
}  // namespace

PXL_EXPORT int pxl_dsa_index_scores(const void* q, const float* w, const void* index_cache, const int* block_tables, const int* cu_q,
                                    const int* positions, float* scores, int64_t ld_scores, int T, int B, int Hi, int Di,
                                    int max_blocks, int page, int max_ctx, cudaStream_t stream) {
  return launch_scores(q, w, index_cache, block_tables, cu_q, positions, scores, ld_scores, T, B, Hi, Di, max_blocks, page, max_ctx,
                       INT64_MAX, nullptr, stream);  // (the size of the cache is not known)
}

// pxl_dsa_index_scores with a status word: prompts of 32 or 64 index heads go to the tensor cores' kernel from 16 tokens on
// (16 tokens x 6000 keys 16.6 and 14.6 us, 64 x 2000 18.9 and 14.6; below, both are as long as their launch), if there is a tile of
// tokens, 128 / heads, for each: a prompt of fewer loads its 256 keys for a product that is mostly padding. us, other kernel and this one:
//   prompts x tokens x keys   16 x 1 x 2000   16 x 1 x 6000   32 x 1 x 6000   16 x 2 x 6000   32 x 2 x 6000   16 x 4 x 6000
//   64 heads                   8.4 12.3        16.2 22.6       36.5 40.8       28.7 22.8       47.7 32.8       39.7 25.5
//   32 heads                  12.2 31.6        24.3 34.3       36.4 41.7       31.1 34.1       46.7 41.7       40.0 27.2
PXL_EXPORT int pxl_dsa_index_scores_status(const void* q, const float* w, const void* index_cache, const int* block_tables, const int* cu_q,
                                           const int* positions, float* scores, int64_t ld_scores, int T, int B, int Hi, int Di,
                                           int max_blocks, int page, int max_ctx, int64_t num_blocks, int* status, cudaStream_t stream) {
  const int width = max_ctx > 0 ? pxl::ceil_div(max_ctx, kKeyTile) * kKeyTile : 0;
  if (cu_q != nullptr && T >= kTcTokens && Di == kDi && (Hi == 32 || Hi == 64) && T >= static_cast<int64_t>(kTcCols / Hi) * B && width > 0 && width <= ld_scores && page > 0 &&
      ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(index_cache)) & 15) == 0 &&
      static_cast<int64_t>(T) * Hi < (1ll << 31)) {
    if (Hi == 64)
      return launch_scores_tc<64>(q, w, index_cache, block_tables, cu_q, positions, scores, ld_scores, width, T, B, max_blocks, page,
                                  max_ctx, num_blocks, status, stream);
    return launch_scores_tc<32>(q, w, index_cache, block_tables, cu_q, positions, scores, ld_scores, width, T, B, max_blocks, page, max_ctx,
                                num_blocks, status, stream);
  }
  return launch_scores(q, w, index_cache, block_tables, cu_q, positions, scores, ld_scores, T, B, Hi, Di, max_blocks, page, max_ctx,
                       num_blocks, status, stream);
}

PXL_EXPORT int pxl_topk_select(const float* scores, int64_t ld, const int* positions, int T, int k, int* out,
                               int64_t ld_out, cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (k <= 0 || ld_out < k) return PXL_ERR_INVALID_ARG;
  if (ld <= kTopkThreads * kTopkHeld) pxl_host::launch(topk_select_kernel<true>, T, kTopkThreads, 0, stream, scores, ld, positions, k, out, ld_out);
  else pxl_host::launch(topk_select_kernel<false>, T, kTopkThreads, 0, stream, scores, ld, positions, k, out, ld_out);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

PXL_EXPORT int pxl_store_rows(const void* src, int64_t ld, const int64_t* slots, void* cache, int T, int D,
                              int64_t num_slots, int* status, cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (D % 8 || ld % 8) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(store_rows_kernel, T, 64, 0, stream, static_cast<const pxl::bf16*>(src), ld, slots,
                                          static_cast<pxl::bf16*>(cache), D, num_slots, status);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}
