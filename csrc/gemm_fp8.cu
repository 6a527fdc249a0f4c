// Block-scaled fp8 (e4m3) GEMM on the 5th-generation tensor cores:
//
//   C[m, n] = sum_kb  a_s[m, kb] * w_s[n / 64, kb] * sum_{k in block kb} A[m, k] * W[n, k]
//
// A: activations quantised in 1 x 128 groups (a_s [M, K/128] fp32), W: weights quantised in
// 128 x 128 blocks; the weight scales are passed at 64-row granularity (w_s [N/64, K/128]) so
// that gate/up matrices interleaved in groups of 64 rows keep their own scales. This is the
// DeepSeek-V3 checkpoint format, which the reference hands to its GPU backends as
// `quantization="fp8"` (src/parallax/sglang/model_runner.py:358-366).
//
// One CTA per 128 x 128 output tile, two CTAs per SM. Per 128-wide K block the MMA warp issues
// four tcgen05.mma (kind::f8f6f4, K = 32) into one of two TMEM partial accumulators; the four
// epilogue warps drain each finished partial with tcgen05.ld and add it, multiplied by the
// block's scales, to fp32 accumulators held in registers. Draining partial kb overlaps the
// MMAs of block kb + 1. Few output tiles (decoding) split K over the CTAs of a cluster, which add their partial sums through
// distributed shared memory. Dense and grouped (per-expert m-tile lists) modes; epilogues: plain,
// +residual, SiLU-mul. Every wait is time-bounded.
#include <cuda_fp8.h>

#include "common.cuh"
#include "pxl_api.h"
#include "tc_issue.cuh"

namespace {
using namespace pxl;

constexpr int FM = 128, FN = 128, FK = 128;  // tile; FK bytes = one 128-byte swizzle row of fp8
constexpr int F_STAGES = 3;
constexpr int F_STAGE_BYTES = (FM + FN) * FK;  // 32 KB
constexpr int F_SMEM = 1024 + F_STAGES * F_STAGE_BYTES + 256;
// Scales of four K blocks, fetched one group of four ahead by the thread that uses them (no barrier): a scale per row of A and
// two per 64 rows of W. Read where they are needed, they were most of the kernel: a load of every thread's own line per K block
// between "the product is there" and its promotion (44 % of the warps' cycles waiting for L1, 24 % hits). The four products of a
// dense layer of 4000 tokens (7168 wide, 18432 inside): 4.38 -> 2.88 ms, and 2.65 (1.7 PFLOP/s) with the sums promoted in pairs.
// A thread without a row fetches none: copies of one address by many lanes go out one by one, and with 64 of 128 rows they took
// longer than the product (36864 x 7168, 64 rows: 97 -> 48 us; one row, whose three idle warps no longer promote either: 155 -> 45).
constexpr int F_GROUP = 4;
constexpr int F_THREADS = 192;

struct Fp8Args {
  const float* a_s;   // [M, kb_total]
  const float* w_s;   // [w_rows / 64, kb_total]
  bf16* C;
  const bf16* residual;
  int ldc, M, N, K, epi;
  // grouped mode
  const int* mt_expert;
  const int* mt_row0;
  const int* mt_row_end;
  const int* num_mt;
  int w_rows_per_expert;
  // SPLIT: CTAs of a cluster, one per K range; K blocks per range (a multiple of F_GROUP)
  int splits, kb_per;
  int stage_bytes;  // of a stage that are loaded
  int early;        // launched in a chain: the weights of the first stages go out ahead of the wait
};

constexpr int kPartPitch = FN + 4;  // floats of a row of partial sums: 16-byte stores of a quarter warp hit distinct banks

template <bool SPLIT>
__global__ void __launch_bounds__(F_THREADS, 2)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                const Fp8Args g, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + F_STAGES * F_STAGE_BYTES);
  __shared__ __align__(16) float scales[2][4][32][F_GROUP];  // [buffer][epilogue warp][lane]: of the thread's row
  __shared__ __align__(16) float w_scales[2][4][2][F_GROUP];
  // bars: [0,S) full, [S,2S) empty, [2S,2S+2) part_full, [2S+2,2S+4) part_empty
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * F_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + F_STAGES);
  const uint32_t pfull0 = smem_u32(bars + 2 * F_STAGES), pempty0 = smem_u32(bars + 2 * F_STAGES + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (g.num_mt != nullptr) pdl_wait();  // the list of tiles comes from the kernels before
  // ---- tile coordinates
  const int num_n = ceil_div(g.N, FN);
  int a_row, b_row, row_end, n_blk;
  {
    const int tile = SPLIT ? blockIdx.x / g.splits : blockIdx.x;
    if (g.num_mt != nullptr) {
      const int mt = tile / num_n;
      if (mt >= *g.num_mt) return;
      n_blk = tile % num_n;
      a_row = g.mt_row0[mt];
      row_end = g.mt_row_end[mt];
      b_row = g.mt_expert[mt] * g.w_rows_per_expert + n_blk * FN;
    } else {
      const int num_m = ceil_div(g.M, FM);
      n_blk = tile / num_m;
      a_row = (tile % num_m) * FM;
      row_end = g.M;
      b_row = n_blk * FN;
    }
  }
  const int kb_total = g.K / FK;
  const int kb_base = SPLIT ? static_cast<int>(cluster_cta_rank()) * g.kb_per : 0;  // this CTA's K blocks
  const int num_kb = SPLIT ? (kb_total - kb_base < g.kb_per ? kb_total - kb_base : g.kb_per) : kb_total;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < F_STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(pfull0 + 8 * a, 1);
      mbar_init(pempty0 + 8 * a, 4);
    }
    mbar_fence_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 2 * FN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // weights of the first stages, under the tail of the kernel before (no kernel of a launch chain writes weights)
  if (warp == 0 && lane == 0 && g.early) {
    for (int kb = 0; kb < F_STAGES && kb < num_kb; ++kb) {
      mbar_arrive_expect_tx(full0 + 8 * kb, g.stage_bytes);
      tma_load_2d(smem_u32(smem + kb * F_STAGE_BYTES + FM * FK), &tmap_b, full0 + 8 * kb, (kb_base + kb) * FK, b_row);
    }
  }
  pdl_wait();
  pdl_launch_dependents();

  // (the issuing loops run with all lanes, so that their addresses and descriptors are uniform; see tc_issue.cuh)
  if (warp == 0) {
    const uint32_t leader = elect_leader(), s0 = smem_u32(smem);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < num_kb; ++kb) {
      const uint32_t fb = full0 + 8 * stage, at = s0 + stage * F_STAGE_BYTES;
      if (kb >= F_STAGES || !g.early) {
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(empty0 + 8 * stage, phase ^ 1, abort_flag, status, PXL_DEV_TIMEOUT_EMPTY))) break;
        expect_tx(fb, g.stage_bytes, leader);
        tma_box(at + FM * FK, &tmap_b, fb, (kb_base + kb) * FK, b_row, leader);
      }
      tma_box(at, &tmap_a, fb, (kb_base + kb) * FK, a_row, leader);
      if (++stage == F_STAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc(FM, FN, 0, 0);  // e4m3 x e4m3 -> fp32
    const uint32_t leader = elect_leader();
    const uint64_t da0 = umma_desc_k_sw128(smem_u32(smem)), db0 = umma_desc_k_sw128(smem_u32(smem) + FM * FK);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < num_kb; ++kb) {
      const int part = kb & 1;
      const uint32_t pphase = (kb >> 1) & 1;
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(pempty0 + 8 * part, pphase ^ 1, abort_flag, status, PXL_DEV_TIMEOUT_TMEM_EMPTY))) break;
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(full0 + 8 * stage, phase, abort_flag, status, PXL_DEV_TIMEOUT_FULL))) break;
      tc_fence_after_sync();
      const uint64_t da = da0 + stage * (F_STAGE_BYTES >> 4), db = db0 + stage * (F_STAGE_BYTES >> 4);
#pragma unroll
      for (int k = 0; k < FK / 32; ++k) mma_f8_ss(tmem_base + part * FN, da + 2 * k, db + 2 * k, idesc, k > 0 ? 1u : 0u, leader);
      commit(empty0 + 8 * stage, leader);
      commit(pfull0 + 8 * part, leader);
      if (++stage == F_STAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
  } else if (a_row + (warp & 3) * 32 >= row_end) {
    // ---- an epilogue warp whose rows are all behind the tile's last one hands the partial sums back as they come
    bool ok = true;
    for (int kb = 0; ok && kb < num_kb; ++kb) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(pfull0 + 8 * (kb & 1), (kb >> 1) & 1, abort_flag, status, PXL_DEV_TIMEOUT_TMEM_FULL)) != 0;
      if (ok && lane == 0) mbar_arrive(pempty0 + 8 * (kb & 1));
    }
  } else {
    // ---- epilogue warps: thread = one accumulator row
    const int q = warp & 3;
    const int row = a_row + q * 32 + lane;
    const bool row_ok = row < row_end;
    const float* as_row = g.a_s + static_cast<size_t>(row_ok ? row : a_row) * kb_total + kb_base;
    const float* ws0 = g.w_s + static_cast<size_t>(b_row / 64) * kb_total + kb_base;
    const bool whole = kb_total % F_GROUP == 0 && ((reinterpret_cast<uintptr_t>(g.a_s) | reinterpret_cast<uintptr_t>(g.w_s)) & 15) == 0;
    auto fetch = [&](int kb) {  // scales of K blocks kb .. kb + 3
      const int buf = (kb / F_GROUP) & 1;
      auto copy = [&](float* dst, const float* src) {
        if (whole) {
          cp_async_16(smem_u32(dst), src + kb, true);
        } else {
          for (int i = 0; i < F_GROUP && kb + i < num_kb; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst + i)), "l"(src + kb + i) : "memory");
        }
      };
      if (kb < num_kb) {
        if (row_ok) copy(scales[buf][q][lane], as_row);
        if (lane < 2) copy(w_scales[buf][q][lane], ws0 + lane * kb_total);
      }
      cp_async_commit();
    };
    fetch(0);
    float acc[FN];
#pragma unroll
    for (int i = 0; i < FN; ++i) acc[i] = 0.f;
    bool ok = true;
    for (int kb = 0; kb < num_kb; ++kb) {
      const int part = kb & 1, buf = (kb / F_GROUP) & 1;
      const uint32_t pphase = (kb >> 1) & 1;
      if (kb % F_GROUP == 0) {
        __syncwarp();  // the other buffer's weight scales were read by every lane
        fetch(kb + F_GROUP);
        cp_async_wait<1>();
        __syncwarp();
      }
      const float sa = scales[buf][q][lane][kb % F_GROUP];
      const float s0 = sa * w_scales[buf][q][0][kb % F_GROUP], s1 = sa * w_scales[buf][q][1][kb % F_GROUP];
      ok = mbar_wait_bounded(pfull0 + 8 * part, pphase, abort_flag, status, PXL_DEV_TIMEOUT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + part * FN + (static_cast<uint32_t>(q * 32) << 16);
      // 16 columns are on their way while the 16 before them are added, two per instruction (32 columns at a time without the
      // overlap: a tenth slower than the sums one by one; in pairs this way: 7168 x 18432, 4000 tokens 666 -> 614 us).
      // The sums stay single numbers that are put into pairs here: held as pairs and taken apart behind the loop they cost registers and a
      // microsecond at its end (100 tokens x 1024 x 512 9.5 us, 7.5 this way; 7.6 one by one).
      uint32_t r[2][16];
      tmem_ld_32x32b_x16(t_row, r[0]);
#pragma unroll
      for (int c = 0; c < FN; c += 16) {
        tmem_ld_wait();
        if (c + 16 < FN) tmem_ld_32x32b_x16(t_row + c + 16, r[((c >> 4) + 1) & 1]);
        const uint32_t sc = __float_as_uint(c < 64 ? s0 : s1);
        const uint64_t sc2 = (static_cast<uint64_t>(sc) << 32) | sc;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          uint64_t x;
          asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(r[(c >> 4) & 1][j]), "r"(r[(c >> 4) & 1][j + 1]));
          uint64_t y;
          asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(acc[c + j]), "f"(acc[c + j + 1]));
          y = fma2(x, sc2, y);
          asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[c + j]), "=f"(acc[c + j + 1]) : "l"(y));
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(pempty0 + 8 * part);
    }
    cp_async_wait<0>();
    if constexpr (SPLIT) {
      // every load and product of this CTA is done: its stages take the partial sums
      if (ok) {
        float* part = reinterpret_cast<float*>(smem) + (q * 32 + lane) * kPartPitch;
#pragma unroll
        for (int c = 0; c < FN; c += 4) *reinterpret_cast<float4*>(part + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
      }
    } else if (ok && row_ok) {
      if (g.epi == PXL_EPI_SILU_MUL) {
        // columns [0,64) gate, [64,128) up of the same 64 outputs
        bf16* dst = g.C + static_cast<size_t>(row) * g.ldc + n_blk * (FN / 2);
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          bf16x8 o;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float g0 = acc[v * 8 + 2 * j], g1 = acc[v * 8 + 2 * j + 1];
            g0 = g0 / (1.f + __expf(-g0));
            g1 = g1 / (1.f + __expf(-g1));
            o.u[j] = pack_bf16x2(g0 * acc[64 + v * 8 + 2 * j], g1 * acc[64 + v * 8 + 2 * j + 1]);
          }
          if (n_blk * (FN / 2) + v * 8 < g.N / 2) st_bf16x8(dst + v * 8, o);
        }
      } else {
        const size_t off = static_cast<size_t>(row) * g.ldc + n_blk * FN;
#pragma unroll
        for (int v = 0; v < 16; ++v) {
          if (n_blk * FN + v * 8 >= g.N) continue;
          float f[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = acc[v * 8 + j];
          if (g.epi == PXL_EPI_RESIDUAL) {
            const bf16x8 rr = ld_bf16x8(g.residual + off + v * 8);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 t2 = unpack_bf16x2(rr.u[j]);
              f[2 * j] += t2.x;
              f[2 * j + 1] += t2.y;
            }
          }
          bf16x8 o;
#pragma unroll
          for (int j = 0; j < 4; ++j) o.u[j] = pack_bf16x2(f[2 * j], f[2 * j + 1]);
          st_bf16x8(g.C + off + v * 8, o);
        }
      }
    }
  }

  if constexpr (SPLIT) {
    // Every thread of every CTA passes both barriers, also after a failed wait (all other waits are bounded). Between them CTA r
    // adds its share of the tile's rows over the cluster, in K order, and writes it.
    __syncwarp();
    cluster_sync_all();
    if (warp >= 2) {
      const int rows = row_end - a_row < FM ? row_end - a_row : FM, share = ceil_div(rows, g.splits);
      const int r0 = static_cast<int>(cluster_cta_rank()) * share, r1 = r0 + share < rows ? r0 + share : rows;
      const bool glu = g.epi == PXL_EPI_SILU_MUL;
      const int chunks = glu ? FN / 16 : FN / 8;  // of 8 outputs
      for (int i = static_cast<int>(threadIdx.x) - 64; i < (r1 - r0) * chunks; i += 128) {
        const int r = r0 + i / chunks, c = i % chunks * 8;
        float f[16] = {};
        for (int s = 0; s < g.splits; ++s) {
          const uint32_t src = cluster_map_shared(smem_u32(smem) + (r * kPartPitch + c) * 4, s);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (v >= 2 && !glu) break;
            const float4 x = ld_shared_cluster_f32x4(src + (v & 1) * 16 + (v >> 1) * 256);  // (the up columns: 64 further)
            f[4 * v] += x.x, f[4 * v + 1] += x.y, f[4 * v + 2] += x.z, f[4 * v + 3] += x.w;
          }
        }
        const size_t off = static_cast<size_t>(a_row + r) * g.ldc + (glu ? n_blk * (FN / 2) : n_blk * FN) + c;
        if (glu) {
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = f[j] / (1.f + __expf(-f[j])) * f[8 + j];
        } else if (g.epi == PXL_EPI_RESIDUAL) {
          const bf16x8 rr = ld_bf16x8(g.residual + off);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 t2 = unpack_bf16x2(rr.u[j]);
            f[2 * j] += t2.x;
            f[2 * j + 1] += t2.y;
          }
        }
        bf16x8 o;
#pragma unroll
        for (int j = 0; j < 4; ++j) o.u[j] = pack_bf16x2(f[2 * j], f[2 * j + 1]);
        st_bf16x8(g.C + off, o);
      }
    }
    __syncwarp();
    cluster_sync_all();  // nobody leaves while its sums are being read
  }
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, 2 * FN);
}

// half a warp per group of 128 columns, 8 columns per lane: amax -> e4m3 + scale. Every group is on its own, so that a few
// rows (decoding) fill the chip like many do: one warp walking a row took 22 us for 64 rows; 2.3 us this way.
__global__ void __launch_bounds__(256) quant_fp8_rows_kernel(const bf16* __restrict__ x, int64_t ld,
                                                             uint8_t* __restrict__ q, float* __restrict__ s, int64_t total,
                                                             int groups) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 16 + (threadIdx.x >> 4);
  const int l = threadIdx.x & 15;
  const bool in = i < total;  // (whole half warps; the other half takes part in the shuffles)
  const int64_t row = in ? i / groups : 0;
  const int g = in ? static_cast<int>(i - row * groups) : 0;
  const bf16* src = x + row * ld + g * 128 + l * 8;
  float v[8];
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const bf16x8 w = ld_bf16x8(src);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(w.u[j]);
      v[2 * j] = f.x, v[2 * j + 1] = f.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __bfloat162float(src[j]);
  }
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = fmaxf(amax, 1e-12f) / 448.f;
  const float inv = 1.f / scale;
  uint32_t packed[2] = {0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const __nv_fp8_storage_t b = __nv_cvt_float_to_fp8(v[j] * inv, __NV_SATFINITE, __NV_E4M3);
    packed[j >> 2] |= static_cast<uint32_t>(b) << (8 * (j & 3));
  }
  if (!in) return;
  uint8_t* dst = q + i * 128 + l * 8;
  if ((reinterpret_cast<uintptr_t>(q) & 7) == 0) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
  } else {  // (q starts on 4 bytes)
    reinterpret_cast<uint32_t*>(dst)[0] = packed[0];
    reinterpret_cast<uint32_t*>(dst)[1] = packed[1];
  }
  if (l == 0) s[i] = scale;
}

int launch_fp8(const void* A, const void* W, Fp8Args g, uint64_t a_rows, uint64_t w_rows, int lda, int ldw,
               int tiles, int* status, cudaStream_t stream) {
  CUtensorMap ta, tb;
  const int box = a_rows < FM ? pxl::ceil_div(static_cast<int>(a_rows), 8) * 8 : FM;
  g.stage_bytes = (box + FN) * FK;
  if (!pxl_host::make_tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, A, a_rows, g.K, lda, box, FK)) return PXL_ERR_TENSORMAP;
  if (!pxl_host::make_tmap_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, W, w_rows, g.K, ldw, FN, FK)) return PXL_ERR_TENSORMAP;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(gemm_fp8_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_fp8_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM) != cudaSuccess)
      return PXL_ERR_CUDA;
    configured[dev] = true;
  }
  if (g.splits > 1) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * g.splits));
    cfg.blockDim = dim3(F_THREADS);
    cfg.dynamicSmemBytes = F_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(g.splits);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    g.early = pxl_host::chained();
    cfg.numAttrs = g.early ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_fp8_kernel<true>, ta, tb, g, status) == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
  }
  g.early = pxl_host::launch_chain() == pxl_host::kInChain;
  pxl_host::launch(gemm_fp8_kernel<false>, tiles, F_THREADS, F_SMEM, stream, ta, tb, g, status);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

// CTAs per output tile (a power of two): two CTAs fit an SM, and a K range has at least eight blocks. The output and down
// projections of 64 rows (56 tiles, K of 16384 and 18432) took 85 us each on 56 SMs and take 38 us on 224 CTAs.
int fp8_splits(int tiles, int kb_total) {
  int s = 1;
  while (s < 8 && tiles * s * 2 <= 2 * pxl_host::num_sms() && kb_total / (s * 2) >= 8) s *= 2;
  return s;
}

}  // namespace

PXL_EXPORT int pxl_gemm_fp8_block(const void* A, const float* a_s, const void* W, const float* w_s, void* C,
                                  const void* residual, int M, int N, int K, int lda, int ldw, int ldc, int epi,
                                  int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return PXL_ERR_INVALID_ARG;
  if ((K % FK) || (N % FN) || (lda % 16) || (ldw % 16) || (ldc % 8)) return PXL_ERR_INVALID_ARG;
  if (epi != PXL_EPI_NONE && epi != PXL_EPI_RESIDUAL && epi != PXL_EPI_SILU_MUL) return PXL_ERR_INVALID_ARG;
  if (epi == PXL_EPI_RESIDUAL && residual == nullptr) return PXL_ERR_INVALID_ARG;
  if (epi == PXL_EPI_SILU_MUL && (N % FN)) return PXL_ERR_INVALID_ARG;
  Fp8Args g{};
  g.a_s = a_s; g.w_s = w_s; g.C = static_cast<pxl::bf16*>(C); g.residual = static_cast<const pxl::bf16*>(residual);
  g.ldc = ldc; g.M = M; g.N = N; g.K = K; g.epi = epi;
  const int tiles = pxl::ceil_div(M, FM) * pxl::ceil_div(N, FN), kb_total = K / FK;
  g.splits = fp8_splits(tiles, kb_total);
  g.kb_per = pxl::ceil_div(pxl::ceil_div(kb_total, g.splits), F_GROUP) * F_GROUP;
  // no empty range: its accumulators would be added as they are (a power of two of CTAs stays one)
  while (g.splits > 1 && (g.splits - 1) * g.kb_per >= kb_total) {
    g.splits /= 2;
    g.kb_per = pxl::ceil_div(pxl::ceil_div(kb_total, g.splits), F_GROUP) * F_GROUP;
  }
  return launch_fp8(A, W, g, M, N, lda, ldw, tiles, status, stream);
}

PXL_EXPORT int pxl_gemm_fp8_block_grouped(const void* A, const float* a_s, const void* W, const float* w_s, void* C,
                                          int P, int E, int N, int K, int lda, int ldw, int ldc,
                                          const int* mt_expert, const int* mt_row0, const int* mt_row_end,
                                          const int* num_mt, int max_m_tiles, int epi, int* status,
                                          cudaStream_t stream) {
  if (P <= 0 || E <= 0 || N <= 0 || K <= 0 || max_m_tiles <= 0) return PXL_ERR_INVALID_ARG;
  if ((K % FK) || (N % FN) || (lda % 16) || (ldw % 16) || (ldc % 8)) return PXL_ERR_INVALID_ARG;
  if (epi != PXL_EPI_NONE && epi != PXL_EPI_SILU_MUL) return PXL_ERR_INVALID_ARG;
  Fp8Args g{};
  g.a_s = a_s; g.w_s = w_s; g.C = static_cast<pxl::bf16*>(C);
  g.ldc = ldc; g.M = P; g.N = N; g.K = K; g.epi = epi;
  g.mt_expert = mt_expert; g.mt_row0 = mt_row0; g.mt_row_end = mt_row_end; g.num_mt = num_mt;
  g.w_rows_per_expert = N;
  const int tiles = max_m_tiles * (N / FN);
  return launch_fp8(A, W, g, P, static_cast<uint64_t>(E) * N, lda, ldw, tiles, status, stream);
}

PXL_EXPORT int pxl_quant_fp8_rows(const void* x, int64_t ld, void* q, float* scales, int T, int K,
                                  cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (K % 128) return PXL_ERR_INVALID_ARG;
  const int64_t total = static_cast<int64_t>(T) * (K / 128);
  pxl_host::launch(quant_fp8_rows_kernel, static_cast<unsigned>((total + 15) / 16), 256, 0, stream, static_cast<const pxl::bf16*>(x), ld, static_cast<uint8_t*>(q), scales, total, K / 128);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}
