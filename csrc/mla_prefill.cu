// Latent attention of prompts with keys and values expanded per head (DeepSeek-V3 family: 128 + 64 key columns, 128 values).
//
// A prompt that starts at its first token finds no keys but its own. For those the up-projection can be done once per token -
// [k | v] of every head = latent x W_kvb^T, one plain product - and attention runs on 192 key and 128 value columns per head: 320
// multiply-adds per (query, key) pair where the absorbed form, which scores and sums 576 and 512 latent columns, takes 1088.
// (Decoding and key lists stay absorbed: there the expansion would be paid per cached token for a row or two. Slices behind a cached
// prefix stay absorbed, too, though only because nothing expands the prefix: 1024 rows would pay for it.)
//
// One CTA = two blocks of 128 queries of one head, which share the tiles of 128 keys and take turns on the tensor pipe as the two
// heads of attn_prefill_pair_kernel do: P_u V, then S_u of the next tile, u = 0, 1, while the other block's softmax runs; P
// replaces S in tensor memory. The first block ends a tile earlier than the second. Shared memory holds both query tiles, two
// key tiles and one value tile (224 KB); rotated key columns are the same for all heads and are read from the latent rows.
// Bound: 2 x 128 x 128 x 320 multiply-adds (4096 a clock) against 2 x 128 x 128 exponentials (16 a clock) per tile of keys, 2560 and
// 2048 clocks.
// 2 prompts of 2048 tokens, 128 heads: 371 us (0.93 PFLOP/s) beside 25 us for the rotation and the rows and 75 us for the
// expansion; the absorbed form's kernel takes 2770 us.
#include "attention_rows.cuh"
#include "common.cuh"
#include "pxl_api.h"

namespace {
using namespace pxl;

constexpr int kQ = 128, kT = 128, kNope = 128, kRot = 64, kV = 128, kLat = 512;
constexpr int kQk = kNope + kRot, kQkChunks = kQk / 64;
constexpr int kHalf = 128 * 128;  // bytes of 64 columns of 128 rows
constexpr int kQBytes = kQkChunks * kHalf, kKBytes = kQkChunks * kHalf, kVBytes = 2 * kHalf, kKBufs = 2;
constexpr int kOffK = 2 * kQBytes, kOffV = kOffK + kKBufs * kKBytes, kOffBars = kOffV + kVBytes;
constexpr int kSmem = 1024 + kOffBars + 256;
constexpr int kSoftmaxWarps = 8, kProducerWarp = 8, kMmaWarp = 9, kThreads = 384;
constexpr float kLog2eF = 1.4426950408889634f;
constexpr uint32_t kIdescS = umma_idesc(kQ, kT, 1, 1), kIdescPV = umma_idesc(kQ, kV, 1, 1) | (1u << 16);  // B (V) is MN-major

__global__ void __launch_bounds__(kThreads, 1)
mla_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv,
                   const __grid_constant__ CUtensorMap tm_rows, const int* __restrict__ cu_q, bf16* __restrict__ out, int H,
                   float scale_log2, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t sm0 = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffBars);
  // q_full | k_full, k_empty [2] | v_full, v_empty | s_full, o_full [2 blocks] | p_ready [2 blocks][2 halves]
  const uint32_t q_full = smem_u32(bars), k_full = q_full + 8, k_empty = k_full + 16, v_full = k_empty + 16, v_empty = v_full + 8,
                 s_full = v_empty + 8, o_full = s_full + 16, p_ready = o_full + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  pdl_wait();
  const int b = blockIdx.z, head = blockIdx.y;
  const int t0 = cu_q[b], L = cu_q[b + 1] - t0;
  // heavy blocks (late queries see the most keys) are scheduled first
  const int q0 = (static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x)) * 2 * kQ;
  if (q0 >= L) return;  // uniform for the CTA, before any barrier or allocation
  auto rows_of = [&](int u) { const int left = L - q0 - u * kQ; return left < 0 ? 0 : left < kQ ? left : kQ; };
  auto tiles_of = [&](int u) { return rows_of(u) > 0 ? q0 / kT + u + 1 : 0; };
  const int n0 = __shfl_sync(0xffffffffu, tiles_of(0), 0), n1 = __shfl_sync(0xffffffffu, tiles_of(1), 0), n_all = n1 > n0 ? n1 : n0;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(q_full, 1);
    for (int s = 0; s < kKBufs; ++s) {
      mbar_init(k_full + 8 * s, 1);
      mbar_init(k_empty + 8 * s, 1);
    }
    mbar_init(v_full, 1);
    mbar_init(v_empty, 1);
    for (int u = 0; u < 2; ++u) {
      mbar_init(s_full + 8 * u, 1);
      mbar_init(o_full + 8 * u, 1);
      for (int h = 0; h < 2; ++h) mbar_init(p_ready + 16 * u + 8 * h, 4);  // one arrival per softmax warp of the block
    }
    mbar_fence_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_kv);
    tma_prefetch_desc(&tm_rows);
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), 512);  // S_0 | S_1 | O_0 | O_1
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_launch_dependents();
  const uint32_t tm_s = *tmem_slot, tm_o = tm_s + 2 * kT;

  // a softmax thread holds 128 scores: 384 threads x 168 registers at launch cover 256 x 208 + 128 x 80
  if (warp >= kSoftmaxWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    if (warp == kProducerWarp) {
      // ------------------------------------------------------------------ TMA producer
      const uint32_t leader = elect_leader();
      if (leader) mbar_arrive_expect_tx(q_full, 2 * kQBytes);
      __syncwarp();
      for (int u = 0; u < 2; ++u)  // (rows past the sequence: the next one's, or zeros past the last)
        for (int c = 0; c < kQkChunks; ++c)
          tma_box(sm0 + u * kQBytes + c * kHalf, &tm_q, q_full, head * kQk + c * 64, t0 + q0 + u * kQ, leader);
      auto free = [&](uint32_t bar, int use) {
        return use == 0 ||
               __all_sync(0xffffffffu, mbar_wait_bounded(bar, (use - 1) & 1, abort_flag, status, PXL_DEV_TIMEOUT_EMPTY));
      };
      for (int it = 0; it < n_all; ++it) {
        const int row = t0 + it * kT, s = it % kKBufs;
        if (!free(k_empty + 8 * s, it / kKBufs)) break;
        const uint32_t k = sm0 + kOffK + s * kKBytes;
        if (leader) mbar_arrive_expect_tx(k_full + 8 * s, kKBytes);
        __syncwarp();
        for (int c = 0; c < 2; ++c) tma_box(k + c * kHalf, &tm_kv, k_full + 8 * s, head * (kNope + kV) + c * 64, row, leader);
        tma_box(k + 2 * kHalf, &tm_rows, k_full + 8 * s, kLat, row, leader);
        if (!free(v_empty, it)) break;
        if (leader) mbar_arrive_expect_tx(v_full, kVBytes);
        __syncwarp();
        for (int c = 0; c < 2; ++c) tma_box(sm0 + kOffV + c * kHalf, &tm_kv, v_full, head * (kNope + kV) + kNope + c * 64, row, leader);
      }
    } else if (warp == kMmaWarp) {
      // ------------------------------------------------------------------ MMA issuer
      const uint32_t leader = elect_leader();
      auto wait = [&](uint32_t bar, int parity, int code) {
        const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, abort_flag, status, code));
        tc_fence_after_sync();
        return ok;
      };
      auto k_ready = [&](int it) { return wait(k_full + 8 * (it % kKBufs), (it / kKBufs) & 1, PXL_DEV_TIMEOUT_FULL); };
      auto issue_s = [&](int u, int it) {
        const uint32_t q = sm0 + u * kQBytes, k = sm0 + kOffK + it % kKBufs * kKBytes;
#pragma unroll
        for (int ks = 0; ks < kQk / 16; ++ks) {
          const uint32_t off = (ks >> 2) * kHalf + (ks & 3) * 32;
          mma_ss(tm_s + u * kT, umma_desc_k_sw128(q + off), umma_desc_k_sw128(k + off), kIdescS, ks > 0 ? 1u : 0u, leader);
        }
        commit(s_full + 8 * u, leader);
      };
      auto tiles = [&](int u) { return u ? n1 : n0; };
      bool ok = wait(q_full, 0, PXL_DEV_TIMEOUT_FULL) && k_ready(0);
      if (ok) {
        issue_s(0, 0);
        if (n1 > 0) issue_s(1, 0);
        commit(k_empty, leader);
      }
      // V tile as B operand of all 128 columns: two 64-column chunks kHalf apart
      const uint64_t dv = (umma_desc_k_sw128(sm0 + kOffV) & ~(0x3fffull << 16)) | (static_cast<uint64_t>(kHalf >> 4) << 16);
      for (int it = 0; ok && it < n_all; ++it) {
        ok = wait(v_full, it & 1, PXL_DEV_TIMEOUT_FULL);
        if (ok && it + 1 < n_all) ok = k_ready(it + 1);
        if (const int seen = L - it * kT; ok && seen < kT) {
          // The last tile ends in the next prompt of the batch: a probability of 0 times what is no number there would be NaN
          for (int i = lane; i < (kT - seen) * 16; i += 32)
            st_shared_zero16(sm0 + kOffV + ((i >> 3) & 1) * kHalf + (seen + (i >> 4)) * 128 + (i & 7) * 16);
          fence_proxy_async_smem();
          __syncwarp();
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (!ok || it >= tiles(u)) continue;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            ok = ok && wait(p_ready + 16 * u + 8 * h, it & 1, PXL_DEV_TIMEOUT_TMEM_EMPTY);
            if (!ok) break;
#pragma unroll
            for (int ks = 4 * h; ks < 4 * h + 4; ++ks)  // 16 keys: 8 columns of P, 16 rows of V
              mma_ts(tm_o + u * kV, tm_s + u * kT + ks * 8, dv + 128 * ks, kIdescPV, (it > 0 || ks > 0) ? 1u : 0u, leader);
          }
          if (!ok) break;
          if (it + 1 == tiles(u)) commit(o_full + 8 * u, leader);
          if (u == 1 || n1 <= it) commit(v_empty, leader);  // the last block that reads this tile
          if (it + 1 < tiles(u)) issue_s(u, it + 1);
        }
        if (ok && it + 1 < n_all) commit(k_empty + 8 * ((it + 1) % kKBufs), leader);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    const int u = warp >> 2, q4 = warp & 3, r = q4 * 32 + lane;  // query row = TMEM lane
    const int rows = rows_of(u), n_tiles = u ? n1 : n0, first_q = q0 + u * kQ, q_pos = first_q + r;
    const bool row_valid = r < rows;
    const uint32_t lane_sel = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t my_s = tm_s + u * kT + lane_sel, my_o = tm_o + u * kV + lane_sel;
    const ScoreArgs sa{};
    float m_run = -INFINITY;
    uint64_t l2[2] = {0ull, 0ull};
    int failed = 0;
    for (int it = 0; it < n_tiles; ++it) {
      failed = mbar_wait_bounded(s_full + 8 * u, it & 1, abort_flag, status, PXL_DEV_TIMEOUT_TMEM_FULL) ? 0 : 1;
      failed = __any_sync(0xffffffffu, failed);  // warp-uniform: the TMEM accesses below are warp-wide
      if (failed) break;
      tc_fence_after_sync();
      const int key0 = it * kT, e = (row_valid ? q_pos + 1 : 0) - key0;
      softmax_tile<kPlain>(my_s, my_o, it == 0, key0 + kT - 1 <= first_q, [&](int j) { return j >= e; }, scale_log2, sa, 0.f, m_run, l2,
                           p_ready + 16 * u);
    }
    if (n_tiles > 0) {
      if (!failed) failed = mbar_wait_bounded(o_full + 8 * u, 0, abort_flag, status, PXL_DEV_TIMEOUT_TMEM_FULL) ? 0 : 1;
      failed = __any_sync(0xffffffffu, failed);
      if (!failed) {
        const float2 la = unpair2(add2(l2[0], l2[1]));
        const float denom = la.x + la.y;
        tc_fence_after_sync();
        store_row(my_o, denom > 0.f ? 1.f / denom : 0.f, out + (static_cast<int64_t>(t0 + q_pos) * H + head) * kV, row_valid);
        tc_fence_before_sync();
      }
    }
  }

  // ---------------------------------------------------------------------- teardown
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);  // loads that are still in flight must land before smem is released
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == kMmaWarp) tmem_dealloc(tm_s, 512);
}

// interleaved rotation of the last 64 of every head's 192 columns, in place
__global__ void __launch_bounds__(256) mla_rotate_kernel(bf16* __restrict__ q, int64_t ld, const float* __restrict__ cos_sin,
                                                         const int* __restrict__ positions, int max_pos, int H, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, p = positions[t];
  if (p < 0 || p >= max_pos) {
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, PXL_DEV_BAD_POSITION);
    return;
  }
  const float* cs = cos_sin + static_cast<int64_t>(p) * kRot;
  for (int i = threadIdx.x; i < H * (kRot / 8); i += 256) {
    const int c = i % (kRot / 8) * 8;
    bf16* x = q + t * ld + i / (kRot / 8) * kQk + kNope + c;
    const bf16x8 v = ld_bf16x8(x);
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(v.u[j]);
      const float co = cs[c / 2 + j], si = cs[kRot / 2 + c / 2 + j];
      o.u[j] = pack_bf16x2(f.x * co - f.y * si, f.x * si + f.y * co);
    }
    st_bf16x8(x, o);
  }
}
}  // namespace

PXL_EXPORT int pxl_mla_rotate(void* q, int64_t ld, const float* cos_sin, const int* positions, int max_pos, int T, int H, int nope,
                              int rot, int* status, cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (nope != kNope || rot != kRot || H <= 0 || (ld % 8) || (reinterpret_cast<uintptr_t>(q) & 15)) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(mla_rotate_kernel, T, 256, 0, stream, static_cast<pxl::bf16*>(q), ld, cos_sin, positions, max_pos, H, status);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

PXL_EXPORT int pxl_mla_prefill(const void* q, const void* kv, const void* rows, const int* cu_q, void* out, int B, int max_q, int T,
                               int H, int nope, int rot, int vdim, int latent, float scale, int* status, cudaStream_t stream) {
  if (B <= 0 || max_q <= 0 || T <= 0) return PXL_OK;
  if (nope != kNope || rot != kRot || vdim != kV || latent != kLat || H <= 0 || H > 65535 || B > 65535 || !(scale > 0.f))
    return PXL_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kv) | reinterpret_cast<uintptr_t>(rows) |
       reinterpret_cast<uintptr_t>(out)) & 15)
    return PXL_ERR_INVALID_ARG;
  CUtensorMap tq, tkv, trows;
  const uint64_t qw = static_cast<uint64_t>(H) * kQk, kw = static_cast<uint64_t>(H) * (kNope + kV);
  if (!pxl_host::make_tmap_2d(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q, T, qw, qw, kQ, 64) ||
      !pxl_host::make_tmap_2d(&tkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, kv, T, kw, kw, kT, 64) ||
      !pxl_host::make_tmap_2d(&trows, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, T, kLat + kRot, kLat + kRot, kT, 64))
    return PXL_ERR_TENSORMAP;
  static bool configured[64] = {false};
  const int dev = pxl_host::current_device_slot();
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(mla_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return PXL_ERR_CUDA;
    configured[dev] = true;
  }
  pxl_host::launch(mla_prefill_kernel, dim3(pxl::ceil_div(max_q, 2 * kQ), H, B), kThreads, kSmem, stream, 
      tq, tkv, trows, cu_q, static_cast<pxl::bf16*>(out), H, scale * kLog2eF, status);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}
