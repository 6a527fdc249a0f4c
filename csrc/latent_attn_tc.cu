// Latent attention on the 5th-generation tensor cores, prompts and decoding alike (bf16; see latent_attn.cu for
// the op). One kernel serves every size with L + R <= 576.
//
// A query row is a (token, head) pair: q [T, H, L + R] is a matrix of T * H rows that all read the same cached
// rows, so a CTA takes 128 consecutive rows of one sequence - 128 / H tokens (one token and a block of 128 heads
// when H > 128) - and walks the keys that its first and last token may see in tiles of 64.
//
//   warp 4    : TMA producer. The query tile once (chunks of 64 columns, 128-byte swizzle), then tiles of cache
//               rows (page boxes), chunk by chunk. A cache row is key AND value and is loaded once: the chunks this
//               CTA accumulates as values go to whole-tile V buffers, all others - needed for the scores only - to a
//               ring of chunk slots that are free again as soon as the scores have read them.
//               With key lists (attention over an indexer's best keys) a CTA takes one token, whose listed rows are
//               gathered four at a time (tile::gather4); tokens without a list take the page boxes.
//   warp 6    : the same for the value buffers. A full query tile leaves room for few of them (64 keys x 256 columns), so the loads
//               of a tile's values wait for the product of a tile before; in a warp of their own they don't hold back the loads
//               for the scores of the next tiles.
//   warps 7-9 : with key lists, half of the listed rows by copies of a warp (see there): four rows of a chunk cost the TMA unit
//               32 to 40 clocks, 144 of them per tile set the pace. 1000 tokens x 2048 listed keys, 128 heads: 1632 us with all
//               rows gathered by TMA, 1180 with the values copied by two warps, 1107 with two of the five other chunks, too.
//   warp 5    : MMA issuer. S = Q K^T over L + R (both operands K-major) into one of two TMEM score buffers, chunk
//               by chunk as the loads land, so the scores of tile i + 1 are computed while the softmax warps work
//               on tile i; then O += P V, P from tensor memory, V taken MN-major from the V buffer, all of its
//               columns by one instruction per 16 keys (narrow instructions cost almost as much as wide ones).
//   warps 0-3 : softmax, one row per thread (its TMEM lane): mask (causal, window), running reference maximum
//               that only moves when a row grew by more than 2^8 (then the TMEM rows of O are rescaled), P
//               back to tensor memory as bf16 (two buffers), row sums in fp32; at the end the sink and the
//               division.
//
// The wide case (L = 512 and up to 64 columns more; 9 chunks) has loops of its own for the producers and the MMA warp, with
// constant counts. What bounded it was not the tensor cores (1950 of 4040 clocks a tile) and not the loads, but one warp's
// instructions: the addresses, descriptors and branches between two products, and instructions that were not in the cache (53
// misses a tile; 14 with the slow paths of the waits out of line). 64 sequences of 4096 keys, 128 heads, pages of 16: 153 -> 106 us
// (pages of 64: 151 -> 100); 16 heads x 1024 keys: 45 -> 28; two prompt slices of 300 behind 1700: 617 -> 417.
//
// O takes 64 TMEM columns per 64 latent columns and scores need room beside it, so a CTA accumulates at most 256
// latent columns; wider latents run as several CTAs per query tile that repeat the scores (L = 512: two). The host
// sizes the ring and the number of V buffers to what the query tile leaves of shared memory.
// Every wait is bounded; on expiry the kernel records a status code, all roles unwind, TMEM is freed.
#include "attention_rows.cuh"
#include "common.cuh"
#include "pxl_api.h"
#include "tc_issue.cuh"

namespace {
using namespace pxl;

constexpr int kRows = 128;
constexpr int kQChunk = kRows * 128;   // bytes of 64 columns of a full query tile
constexpr int kMaxV = 4;               // 64-column latent chunks a CTA accumulates
constexpr int NK = 64;                 // keys per tile
constexpr int kKvChunk = NK * 128;     // bytes of 64 columns of a key tile
constexpr int kMaxSlots = 16, kMaxVBufs = 3;
constexpr int kProducerWarp = 4, kMmaWarp = 5, kValueWarp = 6, kRowWarp = 7, kKeyRowWarp = 8;
constexpr int threads_of(bool lists) { return lists ? 320 : 224; }
constexpr int kBarBytes = 512;
constexpr int kMaxSmem = 227 * 1024;
constexpr float kLog2eF = 1.4426950408889634f;

struct TcArgs {
  const int* block_tables;
  const int* cu_q;      // null: token i is the only query of sequence i
  const int* ctx_lens;
  bf16* out;            // [T, H, L]
  const float* sinks;
  const int* topk;      // [T, topk_stride] key positions of every token (first one negative: all keys), or null
  int topk_k, topk_stride;
  int H, L, D, page, max_blocks, window, vsplit, head_blocks;
  int k_slots, v_bufs;  // ring slots for score-only chunks, buffers for value chunks
  int q_rows;           // rows of the query tile kept in shared memory (decoding: the heads of one token)
  int q_tmem;           // first column chunks of a full query tile that are kept in tensor memory instead
  const bf16 *q, *cache;
  int64_t num_blocks;
  float scale_log2;
  int* status;
};

// B stored as 64-column chunks of [key rows, 64]: MN-major, 8-row groups 1024 B apart, chunks kKvChunk apart
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
  return (umma_desc_k_sw128(addr) & ~(0x3fffull << 16)) | (static_cast<uint64_t>(kKvChunk >> 4) << 16);
}
// Zeros over the rows of a value buffer (`chunks` of NK rows x 128 bytes) whose bits are set, by 128 threads. A function of its own
// and not inlined: each CTA calls it once ahead of its tiles with no bit set, while the first loads are on their way, so that its
// instructions are at hand in the last tile (inlined and cold it cost 2.5 us of 141 for 64 sequences of 4096 keys; 0 this way).
__device__ __noinline__ void clear_rows(uint32_t v, int chunks, uint32_t rows, uint32_t rows2) {
#pragma unroll 1
  for (int k = threadIdx.x >> 3; k < NK; k += 16) {
    if (!((k < 32 ? rows : rows2) >> (k & 31) & 1u)) continue;
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) st_shared_zero16(v + c * kKvChunk + k * 128 + (threadIdx.x & 7) * 16);
  }
  fence_proxy_async_smem();
}

// WIDE: nine column chunks, eight of them values (L = 512 and up to 64 columns more), in two CTAs of four value chunks.
constexpr int kWideKeys = 5, kWideFirst = 3, kWideVBufs = 3;  // score-only chunks, those of the first group, value buffers
constexpr int kWideSlots = 2 * kWideFirst;

template <bool LISTS, bool WIDE>
__global__ void __launch_bounds__(threads_of(LISTS), 1)
latent_attn_tc_kernel(const __grid_constant__ CUtensorMap tm_q_map, const __grid_constant__ CUtensorMap tm_kv,
                      const __grid_constant__ CUtensorMap tm_row, const TcArgs a) {
  constexpr uint32_t kIdescS = umma_idesc(kRows, NK, 1, 1);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int nck = WIDE ? 9 : ceil_div(a.D, 64);
  // The MMA always reads 128 rows. With fewer in shared memory the rest are whatever follows (other chunks, the
  // key ring): those rows' scores are masked and their outputs never stored.
  const uint32_t q_chunk = a.q_rows * 128;
  const uint32_t sm_q = smem_u32(smem);
  const int q_tmem = WIDE ? kMaxV : a.q_tmem, v_bufs = WIDE ? kWideVBufs : a.v_bufs, k_slots = WIDE ? kWideSlots : a.k_slots;
  const int nqs = nck - q_tmem;  // query chunks in shared memory
  // latent chunks of this CTA
  const int vs = blockIdx.x % a.vsplit, tile = blockIdx.x / a.vsplit;
  const int ncv = WIDE ? 8 : ceil_div(a.L, 64), per = WIDE ? kMaxV : ceil_div(ncv, a.vsplit);
  const int v0 = vs * per;
  const int nv = WIDE ? kMaxV : ncv - v0 < per ? ncv - v0 : per;
  const int nkc = nck - nv;                                   // chunks that only the scores read
  auto k_chunk = [&](int j) { return j < v0 ? j : j + nv; };  // their column chunks
  const uint32_t sm_v = sm_q + nqs * q_chunk;
  const uint32_t sm_k = sm_v + v_bufs * per * kKvChunk;
  // query chunk i in shared memory: with WIDE those of the score-only chunks, in their order, and tensor memory has the others
  auto q_col = [&](int i) { return WIDE ? k_chunk(i) : q_tmem + i; };
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + nqs * q_chunk + (v_bufs * per + k_slots) * kKvChunk);
  // q_full | v_full, v_empty [kMaxVBufs] | k_full, k_empty [kMaxSlots] | s_full, p_ready, o_full [2]
  const uint32_t q_full = smem_u32(bars), v_full = q_full + 8, v_empty = v_full + 8 * kMaxVBufs,
                 k_full = v_empty + 8 * kMaxVBufs, k_empty = k_full + 8 * kMaxSlots, s_full = k_empty + 8 * kMaxSlots,
                 p_ready = s_full + 16, o_full = p_ready + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1 + 2 * kMaxVBufs + 2 * kMaxSlots + 6);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  pdl_wait();

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int b = blockIdx.z, hb = blockIdx.y;
  const int t0 = a.cu_q ? a.cu_q[b] : b;
  const int len = a.cu_q ? a.cu_q[b + 1] - t0 : 1;
  const int ctx = a.ctx_lens[b];
  const int h0 = hb * kRows;
  const int heads = a.H - h0 < kRows ? a.H - h0 : kRows;  // heads per token of this tile
  const int tpt = !LISTS && a.H <= kRows ? kRows / a.H : 1;  // tokens per tile
  const int tok0 = tile * tpt;
  if (tok0 >= len) return;  // uniform for the CTA, before any barrier or allocation
  const int ntok = len - tok0 < tpt ? len - tok0 : tpt;
  const int rows = ntok * heads;
  const int64_t row0 = static_cast<int64_t>(t0 + tok0) * a.H + h0;  // row of q / out
  const int pos0 = ctx - len + tok0;
  const int hi = pos0 + ntok;  // keys [lo, hi) are visible to some row
  const int lo = (a.window > 0 && pos0 - a.window + 1 > 0) ? pos0 - a.window + 1 : 0;
  const int* list = nullptr;  // of this CTA's token
  if constexpr (LISTS) {
    list = a.topk + static_cast<int64_t>(t0 + tok0) * a.topk_stride;
    if (list[0] < 0) list = nullptr;
  }
  const bool listed = LISTS && list != nullptr;
  const int t_begin = listed ? 0 : lo / NK;
  const int n_tiles = __shfl_sync(0xffffffffu, ceil_div(listed ? a.topk_k : hi, NK) - t_begin, 0);

  // the CTAs of a query tile start half of a list apart, so that they don't ask L2 for the same rows at the same time
  auto list_tile = [&](int it) { const int t = it + (vs & 1) * (n_tiles >> 1); return t >= n_tiles ? t - n_tiles : t; };

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(q_full, q_tmem > 0 ? 5 : 1);  // the TMA producer, and the warps that write the chunks in tensor memory
    for (int s = 0; s < v_bufs; ++s) {
      mbar_init(v_full + 8 * s, WIDE && listed ? 2 : 1);
      mbar_init(v_empty + 8 * s, 1);
    }
    for (int s = 0; s < k_slots; ++s) {
      mbar_init(k_full + 8 * s, WIDE && listed && s == 1 ? 2 : 1);
      mbar_init(k_empty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full + 8 * s, 1);
      mbar_init(p_ready + 8 * s, 4);  // one arrival per softmax warp
      mbar_init(o_full + 8 * s, 1);
    }
    mbar_fence_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_q_map);
    tma_prefetch_desc(&tm_kv);
  }
  const uint32_t tmem_cols = !WIDE && 64 * per + 3 * NK + 32 * q_tmem <= 256 ? 256 : 512;  // O | two score | two probability buffers | q
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_launch_dependents();
  const uint32_t tm_o = *tmem_slot;             // O: 64 columns per latent chunk
  const uint32_t tm_s = tm_o + 64 * per;        // two score buffers of NK columns
  // two probability buffers of NK / 2 columns (WIDE: in place of the tile's scores); 32 columns per query chunk
  const uint32_t tm_p = WIDE ? tm_s : tm_s + 2 * NK, p_step = WIDE ? NK : NK / 2;
  const uint32_t tm_q = WIDE ? tm_s + 2 * NK : tm_p + NK;

  if (warp >= kRowWarp && !(WIDE && listed)) {
    // (listed rows only)
  } else if (warp == kProducerWarp || warp >= kValueWarp) {
    // ------------------------------------------------------------------ TMA producers
    // Lane p looks up the block of piece p of the tile; one lane issues all boxes.
    const uint32_t leader = elect_leader();
    const bool keys = warp == kProducerWarp, values = warp == kValueWarp;
    if (keys) {
      if (leader) mbar_arrive_expect_tx(q_full, nqs * q_chunk);
      __syncwarp();
      for (int c = 0; c < nqs; ++c) tma_box(sm_q + c * q_chunk, &tm_q_map, q_full, q_col(c) * 64, static_cast<int>(row0), leader);
    }
    const int* bt = a.block_tables + static_cast<int64_t>(b) * a.max_blocks;
    const int box = a.page < NK ? a.page : NK;
    const int pieces = NK / box;
    bool ok = true;
    // wait for the buffer behind `bar_empty` to be free again (its `use`-th use), announce `bytes`
    auto acquire = [&](uint32_t bar_empty, uint32_t bar_full, int use, uint32_t bytes) {
      bool free = true;
      if (use > 0) free = wait_warp(bar_empty, (use - 1) & 1, abort_flag, a.status, PXL_DEV_TIMEOUT_EMPTY);
      if (free && leader) mbar_arrive_expect_tx(bar_full, bytes);
      __syncwarp();
      return free;
    };
    auto tile_row = [&](int it) {  // cache row of this lane's piece of tile `it`
      int row = 0;
      if (lane < pieces && it < n_tiles) {
        int key = (t_begin + it) * NK + lane * box;
        if (key >= ctx) key = (ctx - 1) / box * box;  // beyond the context: re-read its last piece (masked)
        const int bi = key / a.page;
        int64_t blk = bi < a.max_blocks ? bt[bi] : -1;
        if (blk < 0 || blk >= a.num_blocks) {
          if (a.status) atomicCAS(a.status, 0, PXL_DEV_BAD_BLOCK_PREFILL);
          blk = 0;
        }
        row = static_cast<int>(blk * a.page + key % a.page);
      }
      return row;
    };
    auto listed_row = [&](int j) {  // cache row of entry j of the list; entries that name no visible key are masked
      int kp = j < a.topk_k ? list[j] : 0;
      if (kp < 0 || kp > pos0) kp = 0;
      const int bi = kp / a.page;
      int64_t blk = bi < a.max_blocks ? bt[bi] : -1;
      if (blk < 0 || blk >= a.num_blocks) {
        if (a.status) atomicCAS(a.status, 0, PXL_DEV_BAD_BLOCK_PREFILL);
        blk = 0;
      }
      return static_cast<int>(blk * a.page + kp % a.page);
    };
    // chunk of 64 columns from column x of the tile's 64 listed rows
    int rows64[LISTS ? NK : 1];
    auto spread = [&](int row, int row2) {  // two rows in every lane -> all rows in every lane, once for all chunks of a tile
      if constexpr (LISTS) {
#pragma unroll
        for (int i = 0; i < NK; ++i) rows64[i] = __shfl_sync(0xffffffffu, i < 32 ? row : row2, i & 31);
      }
    };
    auto gather = [&](uint32_t dst, uint32_t bar, int x) {
      if constexpr (LISTS) {
#pragma unroll
        for (int g = 0; g < NK / 4; ++g)
          tma_gather4(dst + g * 512, &tm_row, bar, x, rows64[4 * g], rows64[4 * g + 1], rows64[4 * g + 2], rows64[4 * g + 3], leader);
      }
    };
    int slot = 0, slot_use = 0, vb = 0, vb_use = 0;
    if (WIDE && listed && warp >= kKeyRowWarp) {
      // The second group of score-only chunks of listed rows, half of the rows each, by copies of the warp: two rows at a time.
      const int half = (warp - kKeyRowWarp) * 32, second = lane >> 4, j = kWideFirst + ((lane >> 3) & 1);
      const int col = k_chunk(j) * 64 + (lane & 7) * 8;
      const bool in = col < a.D;  // (columns past the row are zeros)
      const bf16* cols = a.cache + (in ? col : 0);
      const uint32_t at = sm_k + j * kKvChunk + half * 128;
      int row = listed_row(list_tile(0) * NK + half + lane);
      for (int it = 0; ok && it < n_tiles; ++it) {
        const int next = listed_row(list_tile(it + 1) * NK + half + lane);
        if (it > 0) ok = wait_warp(k_empty + 8, (it - 1) & 1, abort_flag, a.status, PXL_DEV_TIMEOUT_EMPTY);
        if (!ok) break;
#pragma unroll 8
        for (int i = 0; i < 16; ++i)
          cp_async_16(at + (2 * i + second) * 128 + (((lane & 7) ^ ((2 * i + second) & 7)) << 4),
                      cols + static_cast<int64_t>(__shfl_sync(0xffffffffu, row, 2 * i + second)) * a.D, in);
        row = next;
        cp_async_commit();
        cp_async_wait<0>();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(k_full + 8);
      }
      cp_async_wait<0>();
      ok = false;  // done
    } else if (WIDE && listed && !keys) {
      // The values of listed rows, half of a tile's rows each: 256 columns of a row are 512 neighbouring bytes, one copy of the
      // whole warp, and take nothing of the TMA unit, which spends 32 to 40 clocks on four rows of a chunk and would set the pace
      // with the values, too. A tile is handed on when the copies of the next one are on their way.
      const int half = (warp == kRowWarp) * 32;
      const bf16* cols = a.cache + v0 * 64 + lane * 8;
      const uint32_t at = sm_v + (lane >> 3) * kKvChunk + half * 128;
      int row = listed_row(list_tile(0) * NK + half + lane);
      for (int it = 0; ok && it <= n_tiles; ++it) {
        if (it < n_tiles) {
          const int next = listed_row(list_tile(it + 1) * NK + half + lane);
          if (vb_use > 0) ok = wait_warp(v_empty + 8 * vb, (vb_use - 1) & 1, abort_flag, a.status, PXL_DEV_TIMEOUT_EMPTY);
          if (!ok) break;
#pragma unroll 8
          for (int i = 0; i < 32; ++i)
            cp_async_16(at + vb * (kMaxV * kKvChunk) + i * 128 + (((lane & 7) ^ (i & 7)) << 4),
                        cols + static_cast<int64_t>(__shfl_sync(0xffffffffu, row, i)) * a.D, true);
          row = next;
        }
        cp_async_commit();
        if (it > 0) {
          cp_async_wait<1>();
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(v_full + 8 * (vb == 0 ? kWideVBufs - 1 : vb - 1));
        }
        if (++vb == kWideVBufs) {
          vb = 0;
          ++vb_use;
        }
      }
      cp_async_wait<0>();
      ok = false;  // done
    }
    int row = listed ? listed_row(list_tile(0) * NK + lane) : tile_row(0), row2 = listed ? listed_row(list_tile(0) * NK + 32 + lane) : 0;
    for (int it = 0; ok && it < n_tiles; ++it) {
      // its table reads are in flight while this tile is issued
      const int next_row = listed ? listed_row(list_tile(it + 1) * NK + lane) : tile_row(it + 1);
      const int next_row2 = listed ? listed_row(list_tile(it + 1) * NK + 32 + lane) : 0;
      if (listed) spread(row, row2);
      if constexpr (WIDE) {  // two groups of chunks, a barrier each
        if (keys) {
          ok = acquire(k_empty, k_full, it, kWideFirst * kKvChunk);
          if (!ok) break;
          if (listed) {
#pragma unroll 1
            for (int j = 0; j < kWideFirst; ++j) gather(sm_k + j * kKvChunk, k_full, k_chunk(j) * 64);
          } else {
#pragma unroll 1
            for (int p = 0; p < pieces; ++p) {
              const int r = __shfl_sync(0xffffffffu, row, p);
#pragma unroll
              for (int j = 0; j < kWideFirst; ++j) tma_box(sm_k + j * kKvChunk + p * box * 128, &tm_kv, k_full, k_chunk(j) * 64, r, leader);
            }
          }
          if (!listed) {
            ok = acquire(k_empty + 8, k_full + 8, it, (kWideKeys - kWideFirst) * kKvChunk);
            if (!ok) break;
#pragma unroll 1
            for (int p = 0; p < pieces; ++p) {
              const int r = __shfl_sync(0xffffffffu, row, p);
#pragma unroll
              for (int j = kWideFirst; j < kWideKeys; ++j)
                tma_box(sm_k + j * kKvChunk + p * box * 128, &tm_kv, k_full + 8, k_chunk(j) * 64, r, leader);
            }
          }
        }
      } else {
        auto key_chunk = [&](int j, uint32_t dst, uint32_t bar) {
          if (listed) gather(dst, bar, k_chunk(j) * 64);
          else
            for (int p = 0; p < pieces; ++p)
              tma_box(dst + p * box * 128, &tm_kv, bar, k_chunk(j) * 64, __shfl_sync(0xffffffffu, row, p), leader);
        };
        for (int j = 0; ok && keys && j < nkc; ++j) {
          ok = acquire(k_empty + 8 * slot, k_full + 8 * slot, slot_use, kKvChunk);
          if (ok) key_chunk(j, sm_k + slot * kKvChunk, k_full + 8 * slot);
          if (++slot == k_slots) {
            slot = 0;
            ++slot_use;
          }
        }
      }
      if (ok && values) ok = acquire(v_empty + 8 * vb, v_full + 8 * vb, vb_use, nv * kKvChunk);
      if (!WIDE && ok && values && listed)  // (WIDE: copies, above)
        for (int c = 0; c < nv; ++c) gather(sm_v + (vb * per + c) * kKvChunk, v_full + 8 * vb, (v0 + c) * 64);
      else if (ok && values)
        for (int p = 0; p < pieces; ++p) {
          const int r = __shfl_sync(0xffffffffu, row, p);
#pragma unroll
          for (int c = 0; c < nv; ++c)
            tma_box(sm_v + (vb * per + c) * kKvChunk + p * box * 128, &tm_kv, v_full + 8 * vb, (v0 + c) * 64, r, leader);
        }
      if (++vb == v_bufs) {
        vb = 0;
        ++vb_use;
      }
      row = next_row;
      row2 = next_row2;
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------------ MMA issuer
    if constexpr (WIDE) {
      // The scores of tile it, then the product of tile it - 1 under the softmax of tile it. All counts are constants and the code
      // has no branches but the waits: one warp issues these instructions one after the other, so that every address it computes
      // and every branch it takes between two products is time in which the tensor cores have nothing to do.
      const uint32_t leader = elect_leader();
      constexpr uint32_t kIdescPV = umma_idesc(kRows, 64 * kMaxV, 1, 1) | (1u << 16);  // B (V) is MN-major
      constexpr uint32_t kChunkD = kKvChunk >> 4;
      const uint64_t dq = umma_desc_k_sw128(sm_q), dk = umma_desc_k_sw128(sm_k);
      const uint32_t q_step = q_chunk >> 4;
      auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        const bool there = wait_warp(bar, parity, abort_flag, a.status, code);
        tc_fence_after_sync();
        return there;
      };
      auto product = [&](int it, uint32_t v) {  // O += P V
        if (!wait(p_ready + 8 * (it & 1), (it >> 1) & 1, PXL_DEV_TIMEOUT_TMEM_EMPTY)) return false;
        const uint64_t dv = desc_mn_sw128(v);
        const uint32_t p = tm_s + (it & 1) * NK;
#pragma unroll
        for (int ks = 0; ks < NK / 16; ++ks) mma_ts(tm_o, p + ks * 8, dv + 128 * ks, kIdescPV, (it > 0 || ks > 0) ? 1u : 0u, leader);
        commit(o_full + 8 * (it & 1), leader);
        return true;
      };
      bool ok = wait(q_full, 0, PXL_DEV_TIMEOUT_FULL);
      int vb = 0, vb_phase = 0, pv = kWideVBufs - 1;  // value buffers of this tile and of the one before
      for (int it = 0; ok && it <= n_tiles; ++it) {
        if (it < n_tiles) {
          const uint32_t d = tm_s + (it & 1) * NK;
          ok = wait(k_full, it & 1, PXL_DEV_TIMEOUT_FULL);
          if (!ok) break;
#pragma unroll
          for (int j = 0; j < kWideFirst; ++j)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              mma_ss(d, dq + j * q_step + 2 * ks, dk + j * kChunkD + 2 * ks, kIdescS, j == 0 && ks == 0 ? 0u : 1u, leader);
          commit(k_empty, leader);
          ok = wait(k_full + 8, it & 1, PXL_DEV_TIMEOUT_FULL);
          if (!ok) break;
#pragma unroll
          for (int j = kWideFirst; j < kWideKeys; ++j)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ss(d, dq + j * q_step + 2 * ks, dk + j * kChunkD + 2 * ks, kIdescS, 1u, leader);
          commit(k_empty + 8, leader);
          ok = wait(v_full + 8 * vb, vb_phase, PXL_DEV_TIMEOUT_FULL);
          if (!ok) break;
          const uint64_t dkv = umma_desc_k_sw128(sm_v + vb * (kMaxV * kKvChunk));
#pragma unroll
          for (int j = 0; j < kMaxV; ++j)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ts(d, tm_q + j * 32 + ks * 8, dkv + j * kChunkD + 2 * ks, kIdescS, 1u, leader);
          commit(s_full + 8 * (it & 1), leader);
        }
        if (it > 0) {
          ok = product(it - 1, sm_v + pv * (kMaxV * kKvChunk));
          if (ok) commit(v_empty + 8 * pv, leader);
        }
        pv = vb;
        if (++vb == kWideVBufs) {
          vb = 0;
          vb_phase ^= 1;
        }
      }
    } else {
      const uint32_t leader = elect_leader();
      const uint32_t idesc_pv = umma_idesc(kRows, 64 * nv, 1, 1) | (1u << 16);  // B (V) is MN-major
      const uint64_t dq0 = umma_desc_k_sw128(sm_q);
      // descriptors advance by 16-byte units: 2 per k-step inside a chunk (columns past D are zeros on both sides)
      auto ready = [](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test(bar, parity)) != 0; };
      auto s_chunk = [&](int it, int col_chunk, uint32_t rows_addr, bool first) {  // S[it % 2] (+)= Q[:, chunk] K[:, chunk]^T
        const uint64_t dk = umma_desc_k_sw128(rows_addr);
        const uint32_t d = tm_s + (it & 1) * NK;
        if (col_chunk < q_tmem) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            mma_ts(d, tm_q + col_chunk * 32 + ks * 8, dk + 2 * ks, kIdescS, first && ks == 0 ? 0u : 1u, leader);
        } else {
          const uint64_t dq = dq0 + static_cast<uint64_t>(col_chunk - q_tmem) * (q_chunk >> 4);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) mma_ss(d, dq + 2 * ks, dk + 2 * ks, kIdescS, first && ks == 0 ? 0u : 1u, leader);
        }
      };
      // Whichever is ready goes next: the product of a tile whose probabilities are written, or the next chunk of the
      // scores (at most one tile ahead of the products: two score buffers). A load in flight never holds back a
      // product, which is what frees the buffers for the loads after it.
      bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(q_full, 0, abort_flag, a.status, PXL_DEV_TIMEOUT_FULL));
      int next_s = 0, next_pv = 0;   // tiles whose scores / products come next
      int j = 0, slot = 0, slot_phase = 0;  // score-only chunk of tile next_s and its ring slot
      int s_vb = 0, s_vb_phase = 0, pv_vb = 0;
      uint64_t since = 0;
      uint32_t spins = 0;
      while (ok && next_pv < n_tiles) {
        bool moved = false;
        if (next_s < n_tiles && next_s <= next_pv + 1) {
          while (j < nkc && ready(k_full + 8 * slot, slot_phase)) {
            tc_fence_after_sync();
            s_chunk(next_s, k_chunk(j), sm_k + slot * kKvChunk, j == 0);
            commit(k_empty + 8 * slot, leader);  // free again once these have read it
            ++j;
            if (++slot == k_slots) {
              slot = 0;
              slot_phase ^= 1;
            }
            moved = true;
          }
          if (j == nkc && ready(v_full + 8 * s_vb, s_vb_phase)) {
            tc_fence_after_sync();
            const uint32_t v = sm_v + s_vb * per * kKvChunk;
            for (int c = 0; c < nv; ++c) s_chunk(next_s, v0 + c, v + c * kKvChunk, nkc == 0 && c == 0);
            commit(s_full + 8 * (next_s & 1), leader);
            ++next_s;
            j = 0;
            if (++s_vb == v_bufs) {
              s_vb = 0;
              s_vb_phase ^= 1;
            }
            moved = true;
          }
        }
        if (next_pv < next_s && ready(p_ready + 8 * (next_pv & 1), (next_pv >> 1) & 1)) {  // O += P V
          tc_fence_after_sync();
          const uint64_t dv = desc_mn_sw128(sm_v + pv_vb * per * kKvChunk);
          const uint32_t p = tm_p + (next_pv & 1) * (NK / 2);
#pragma unroll
          for (int ks = 0; ks < NK / 16; ++ks)
            mma_ts(tm_o, p + ks * 8, dv + 128 * ks, idesc_pv, (next_pv > 0 || ks > 0) ? 1u : 0u, leader);
          commit(o_full + 8 * (next_pv & 1), leader);
          commit(v_empty + 8 * pv_vb, leader);
          ++next_pv;
          if (++pv_vb == v_bufs) pv_vb = 0;
          moved = true;
        }
        if (moved) {
          spins = 0;
          since = 0;
        } else if ((++spins & 0x3ffu) == 0) {
          const uint64_t now = global_timer_ns();
          if (since == 0) since = now;
          const bool late = now - since > kWaitLimitNs;
          if (late && leader) {
            *abort_flag = 1;
            if (a.status) atomicCAS(a.status, 0, PXL_DEV_TIMEOUT_TMEM_EMPTY);
          }
          ok = __all_sync(0xffffffffu, !late && !*abort_flag);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax warps
    const int r = warp * 32 + lane;  // query row = TMEM lane
    const int pos = pos0 + r / heads, head = h0 + r % heads;
    const bool row_valid = r < rows;
    const int key_lo = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    const int key_hi = row_valid ? pos + 1 : 0;
    const uint32_t lane_sel = static_cast<uint32_t>(warp * 32) << 16;
    float m_run = -INFINITY, l_run = 0.f;
    int failed = 0;
    if (q_tmem > 0) {  // this row's part of the query chunks in tensor memory, two columns per word; two chunks in flight
      const bf16* src = a.q + (row0 + r) * a.D + (WIDE ? v0 * 64 : 0);
      for (int c = 0; c < q_tmem; c += 2) {
        uint32_t v[2][32] = {};
        if (row_valid) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const bf16x8 x = ld_bf16x8(src + c * 64 + j * 8);
#pragma unroll
            for (int k = 0; k < 4; ++k) v[j >> 3][(j & 7) * 4 + k] = x.u[k];
          }
        }
        tmem_st_32x32b_x32(tm_q + c * 32 + lane_sel, v[0]);
        tmem_st_32x32b_x32(tm_q + c * 32 + 32 + lane_sel, v[1]);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    // of the listed keys of a tile, those that are visible (a bit each)
    uint32_t seen[2] = {0u, 0u};
    auto entry = [&](int j) { return listed && j < a.topk_k ? list[j] : -1; };
    auto visible = [&](int kp, int kp2) {
      seen[0] = __ballot_sync(0xffffffffu, kp >= 0 && kp <= pos0);
      seen[1] = __ballot_sync(0xffffffffu, kp2 >= 0 && kp2 <= pos0);
    };
    if (listed) visible(entry(list_tile(0) * NK + lane), entry(list_tile(0) * NK + 32 + lane));
    clear_rows(sm_v, nv, 0u, 0u);
    for (int it = 0; it < n_tiles; ++it) {
      const int par = it & 1;
      const int next = entry(list_tile(it + 1) * NK + lane), next2 = entry(list_tile(it + 1) * NK + 32 + lane);
      failed = !wait_warp(s_full + 8 * par, (it >> 1) & 1, abort_flag, a.status, PXL_DEV_TIMEOUT_TMEM_FULL);  // (warp-uniform: the TMEM accesses are)
      if (failed) break;
      tc_fence_after_sync();
      uint32_t sc[NK];
#pragma unroll
      for (int c = 0; c < NK; c += 32)
        tmem_ld_32x32b_x32(tm_s + par * NK + c + lane_sel, *reinterpret_cast<uint32_t(*)[32]>(&sc[c]));
      tmem_ld_wait();
      const int key0 = (t_begin + it) * NK;
      int ma = key_lo - key0, me = key_hi - key0;  // this row sees columns [ma, me)
      if (listed) {
        ma = 0, me = NK;
        if (__builtin_expect((seen[0] & seen[1]) != 0xffffffffu, 0)) {
#pragma unroll
          for (int j = 0; j < NK; ++j)
            if (!(seen[j >> 5] >> (j & 31) & 1u)) sc[j] = 0xff800000u;  // -inf
        }
      }
      if (__builtin_expect(!__all_sync(0xffffffffu, ma <= 0 && me >= NK), 0)) {
#pragma unroll
        for (int j = 0; j < NK; ++j)
          if (j < ma || j >= me) sc[j] = 0xff800000u;  // -inf
      }
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < NK; j += 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) m4[k] = fmaxf(m4[k], __uint_as_float(sc[j + k]));
      }
      const float m_new = fmaxf(m_run, fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale_log2);  // scale > 0
      if (it == 0) {
        m_run = m_new;
      } else if (__builtin_expect(__any_sync(0xffffffffu, m_new > m_run + 8.f), 0)) {
        // O accumulates relative to m_run: move the reference and rescale, once O of the tile before is complete
        failed = !wait_warp(o_full + 8 * (par ^ 1), ((it - 1) >> 1) & 1, abort_flag, a.status, PXL_DEV_TIMEOUT_TMEM_FULL);
        if (failed) break;
        const float corr = fast_exp2(m_run - (m_new == -INFINITY ? 0.f : m_new));
        m_run = m_new;
        l_run *= corr;
        tc_fence_after_sync();
        for (int c = 0; c < nv * 64; c += 32) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tm_o + lane_sel + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
          tmem_st_32x32b_x32(tm_o + lane_sel + c, v);
        }
        tmem_st_wait();
      }
      const float m_use = (m_run == -INFINITY) ? 0.f : m_run;
      // the P buffer was last read by the product of tile it - 2 (WIDE: which the scores of this tile, in the same place, followed)
      if (!WIDE && it >= 2) {
        failed = !wait_warp(o_full + 8 * par, ((it - 2) >> 1) & 1, abort_flag, a.status, PXL_DEV_TIMEOUT_TMEM_FULL);
        if (failed) break;
        tc_fence_after_sync();
      }
      // The denominator sums what the product sums, the rounded probabilities: m_run is not always the maximum, so a key that
      // carries the softmax alone has a rounded one, and only the same rounding below the line cancels it (sharp scores over 2000
      // keys, error against 64 bits: 2.07e-3 with the unrounded sum, below 1.95e-3 this way; 0.3 % of a decoding pass).
      uint64_t sum2[2] = {0ull, 0ull};
      uint32_t pk[NK / 2];
#pragma unroll
      for (int j = 0; j < NK; j += 2) {
        const float p0 = fast_exp2(fmaf(__uint_as_float(sc[j]), a.scale_log2, -m_use));
        const float p1 = fast_exp2(fmaf(__uint_as_float(sc[j + 1]), a.scale_log2, -m_use));
        pk[j >> 1] = pack_bf16x2(p0, p1);
        const float2 r = unpack_bf16x2(pk[j >> 1]);
        sum2[(j >> 1) & 1] = add2(sum2[(j >> 1) & 1], pair2(r.x, r.y));
      }
      const float2 both = unpair2(add2(sum2[0], sum2[1]));
      l_run += both.x + both.y;
#pragma unroll
      for (int c = 0; c < NK / 2; c += 16)
        tmem_st_32x32b_x16(tm_p + par * p_step + c + lane_sel, *reinterpret_cast<uint32_t(*)[16]>(&pk[c]));
      tmem_st_wait();
      if (__builtin_expect(listed ? (seen[0] & seen[1]) != 0xffffffffu : key0 < lo || key0 + NK > hi, 0)) {
        // Rows that no query of the tile sees (behind the context, ahead of the window, stand-ins of a list's empty entries): a
        // probability of 0 times what is no number there would be NaN. The scores have read these buffers, the product has not.
        if (!listed) {
          auto below = [](int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; };
          const int from = lo - key0, to = hi - key0;
          seen[0] = below(to) & ~below(from), seen[1] = below(to - 32) & ~below(from - 32);
        }
        clear_rows(sm_v + it % v_bufs * per * kKvChunk, nv, ~seen[0], ~seen[1]);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready + 8 * par);
      if (listed) visible(next, next2);
    }
    if (!failed)
      failed = !wait_warp(o_full + 8 * ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1, abort_flag, a.status, PXL_DEV_TIMEOUT_TMEM_FULL);
    if (!failed) {
      float denom = l_run, f = 1.f;
      if (a.sinks && row_valid) {
        const float sink = a.sinks[head] * kLog2eF;
        const float M = fmaxf(m_run, sink);
        f = exp2f(m_run - M);
        denom = denom * f + exp2f(sink - M);
      }
      const float inv = denom > 0.f ? f / denom : 0.f;
      bf16* dst = a.out + (row0 + r) * a.L + v0 * 64;
      const int ncol = a.L - v0 * 64 < nv * 64 ? a.L - v0 * 64 : nv * 64;
      tc_fence_after_sync();
      for (int c = 0; c < nv * 64; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(tm_o + lane_sel + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int c8 = 0; c8 < 32; c8 += 8) {
          bf16x8 ov;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            ov.u[j] = pack_bf16x2(__uint_as_float(v[c8 + 2 * j]) * inv, __uint_as_float(v[c8 + 2 * j + 1]) * inv);
          if (row_valid && c + c8 < ncol) st_bf16x8(dst + c + c8, ov);
        }
      }
      tc_fence_before_sync();
    }
  }

  // ---------------------------------------------------------------------- teardown
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);  // loads that are still in flight must land before smem is released
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == kMmaWarp) tmem_dealloc(tm_o, tmem_cols);
}

struct TilePlan {
  int k_slots, v_bufs, q_tmem, smem;
};

// Ring slots and V buffers beside a query tile of q_rows rows, q_tmem chunks of which are in tensor memory; false when the sizes
// do not fit.
bool plan_tiles(int L, int D, int q_rows, int page, int q_tmem, TilePlan* p) {
  if (page % 8 != 0 || (page % NK != 0 && NK % page != 0)) return false;
  const int nck = ceil_div(D, 64), ncv = ceil_div(L, 64);
  const int vsplit = ceil_div(ncv, kMaxV), per = ceil_div(ncv, vsplit);
  const int nkc = nck - (ncv - (vsplit - 1) * per);  // score-only chunks of the CTA that has most of them
  const int q_bytes = (nck - q_tmem) * q_rows * 128;
  const int slots = (kMaxSmem - 1024 - kBarBytes - q_bytes) / kKvChunk;
  p->k_slots = 0;
  p->q_tmem = q_tmem;
  for (int vb = kMaxVBufs; vb >= 1; --vb) {
    const int ks = slots - vb * per;
    if (ks >= (vb > 1 ? nkc + 1 : (nkc > 0 ? 1 : 0))) {
      p->v_bufs = vb;
      p->k_slots = ks < kMaxSlots ? ks : kMaxSlots;
      if (p->k_slots < 1) p->k_slots = 1;
      const int tiles = q_bytes + (vb * per + p->k_slots) * kKvChunk;
      const int reach = (nck - q_tmem - 1) * q_rows * 128 + kQChunk;  // what the MMA reads of the query tile
      p->smem = 1024 + (tiles > reach ? tiles : reach) + kBarBytes;
      return p->smem <= kMaxSmem;
    }
  }
  return false;
}

// A full query tile may leave room for one V buffer: the loads of a tile's values then wait for the product of the tile before it, a
// load latency per tile. O, scores and probabilities leave 64 columns of tensor memory, which hold two of the query chunks: room for
// a second buffer (576 columns, 64 sequences behind 4096 tokens: 196 -> 182 us; these have the wide form now, with four chunks there).
bool plan_tiles(int L, int D, int q_rows, int page, TilePlan* p) {
  const bool fits = plan_tiles(L, D, q_rows, page, 0, p);
  TilePlan other;
  if (fits && p->v_bufs == 1 && q_rows == kRows && D >= 192 && plan_tiles(L, D, q_rows, page, 2, &other) && other.v_bufs > 1) *p = other;
  return fits;
}
}  // namespace

PXL_EXPORT int pxl_latent_attn_tc_supported(int L, int R, int page, float scale) {
  TilePlan plan;
  return L > 0 && R >= 0 && L % 8 == 0 && R % 8 == 0 && page > 0 && page % 8 == 0 && scale > 0.f &&
         plan_tiles(L, L + R, kRows, page, &plan);
}

PXL_EXPORT int pxl_latent_attn_tc(const void* q, const void* cache, const int* block_tables, const int* cu_q,
                                  const int* ctx_lens, void* out, const float* sinks, const int* topk, int topk_k, int topk_stride,
                                  int B, int max_q, int total_q, int H, int L, int R, int page, int max_blocks, int64_t num_blocks,
                                  float scale, int window, int* status, cudaStream_t stream) {
  if (B <= 0 || max_q <= 0 || total_q <= 0) return PXL_OK;
  if (H <= 0 || B > 65535 || !pxl_latent_attn_tc_supported(L, R, page, scale)) return PXL_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15)
    return PXL_ERR_INVALID_ARG;
  if (num_blocks * page >= (1ll << 31) || static_cast<int64_t>(total_q) * H >= (1ll << 31)) return PXL_ERR_TOO_LARGE;
  TcArgs a{};
  TilePlan plan;
  // short queries (decoding) leave most of the tile's rows empty: keep only the others, and more keys in flight
  if (topk && (topk_k <= 0 || window > 0)) return PXL_ERR_INVALID_ARG;
  const int rows = (topk ? 1 : max_q) * (H < kRows ? H : kRows);
  a.q_rows = rows >= kRows ? kRows : pxl::ceil_div(rows, 8) * 8;
  if (!plan_tiles(L, L + R, a.q_rows, page, &plan)) return PXL_ERR_INVALID_ARG;
  a.k_slots = plan.k_slots;
  a.v_bufs = plan.v_bufs;
  a.q_tmem = plan.q_tmem;
  a.q = static_cast<const pxl::bf16*>(q);
  a.cache = static_cast<const pxl::bf16*>(cache);
  a.block_tables = block_tables;
  a.cu_q = cu_q;
  a.ctx_lens = ctx_lens;
  a.out = static_cast<pxl::bf16*>(out);
  a.sinks = sinks;
  a.topk = topk, a.topk_k = topk_k, a.topk_stride = topk_stride;
  a.H = H, a.L = L, a.D = L + R, a.page = page, a.max_blocks = max_blocks, a.window = window, a.num_blocks = num_blocks;
  a.vsplit = pxl::ceil_div(pxl::ceil_div(L, 64), kMaxV);
  a.head_blocks = pxl::ceil_div(H, kRows);
  a.scale_log2 = scale * kLog2eF;
  a.status = status;
  CUtensorMap tq, tkv, trow;
  if (!pxl_host::make_tmap_2d(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q, static_cast<uint64_t>(total_q) * H, a.D, a.D,
                              a.q_rows, 64) ||
      !pxl_host::make_tmap_2d(&tkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, cache, static_cast<uint64_t>(num_blocks) * page, a.D,
                              a.D, page < NK ? page : NK, 64) ||
      !pxl_host::make_tmap_2d(&trow, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, cache, static_cast<uint64_t>(num_blocks) * page, a.D,
                              a.D, 1, 64))
    return PXL_ERR_TENSORMAP;
  const int tpt = !topk && H <= kRows ? kRows / H : 1;
  const dim3 grid(pxl::ceil_div(max_q, tpt) * a.vsplit, a.head_blocks, B);
  // WIDE at its own shared memory: five query chunks, three value buffers, six slots
  const bool wide = pxl::ceil_div(a.D, 64) == 9 && pxl::ceil_div(L, 64) == 8;
  const int tiles = (9 - kMaxV) * a.q_rows * 128 + (kWideVBufs * kMaxV + kWideSlots) * kKvChunk;
  const int reach = (9 - kMaxV - 1) * a.q_rows * 128 + kQChunk;
  const int smem = wide ? 1024 + (tiles > reach ? tiles : reach) + kBarBytes : plan.smem;
  static_assert(1024 + (9 - kMaxV) * kQChunk + (kWideVBufs * kMaxV + kWideSlots) * kKvChunk + kBarBytes <= kMaxSmem, "shared memory of a CTA");
  const auto kern = topk ? (wide ? latent_attn_tc_kernel<true, true> : latent_attn_tc_kernel<true, false>)
                         : (wide ? latent_attn_tc_kernel<false, true> : latent_attn_tc_kernel<false, false>);
  static bool configured[64] = {false};
  const int dev = pxl_host::current_device_slot();
  if (!configured[dev]) {
    for (const auto k : {latent_attn_tc_kernel<false, false>, latent_attn_tc_kernel<false, true>, latent_attn_tc_kernel<true, false>,
                         latent_attn_tc_kernel<true, true>})
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess) return PXL_ERR_CUDA;
    configured[dev] = true;
  }
  pxl_host::launch(kern, grid, dim3(threads_of(topk != nullptr)), smem, stream, tq, tkv, trow, a);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}
