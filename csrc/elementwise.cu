// Memory-bound elementwise / normalisation kernels: RMSNorm(+residual), fused per-head
// q/k-norm + RoPE + paged-cache scatter, activation-and-multiply, row gather.
//
// These replace what the reference reaches through third-party GPU layers
// (RMSNorm / RoPE / SiLU-mul, src/parallax/server/executor/sglang_executor.py:419-452)
// and its own Metal cache-scatter kernel
// (src/parallax_extensions/kernels/reshape_and_cache/reshape_and_cache.metal:32-96).
#include <cuda_fp8.h>

#include <type_traits>

#include "common.cuh"
#include "pxl_api.h"

namespace {
using namespace pxl;

// ----------------------------------------------------------------------------- RMSNorm
// Rows of any length: read twice (the second time from L1 / L2).
template <bool HAS_RES>
__global__ void __launch_bounds__(256)
rmsnorm_long_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ out,
               bf16* __restrict__ residual, int H, float eps, float w_offset) {
  __shared__ float red[32];
  pdl_wait();
  pdl_launch_dependents();
  const size_t row = blockIdx.x;
  const bf16* xr = x + row * H;
  bf16* rr = HAS_RES ? residual + row * H : nullptr;
  bf16* outr = out + row * H;
  const int nvec = H >> 3;
  float ss = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    bf16x8 a = ld_bf16x8(xr + v * 8);
    if constexpr (HAS_RES) {
      const bf16x8 b = ld_bf16x8(rr + v * 8);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 fa = unpack_bf16x2(a.u[j]);
        const float2 fb = unpack_bf16x2(b.u[j]);
        a.u[j] = pack_bf16x2(fa.x + fb.x, fa.y + fb.y);
      }
      st_bf16x8(rr + v * 8, a);  // the sum (rounded to bf16) is the new residual stream
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(a.u[j]);
      ss += f.x * f.x + f.y * f.y;
    }
  }
  ss = block_reduce_sum(ss, red);
  const float inv = rsqrtf(ss / static_cast<float>(H) + eps);
  const bf16* src = HAS_RES ? rr : xr;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const bf16x8 a = ld_bf16x8(src + v * 8);
    const bf16x8 ww = ld_bf16x8(w + v * 8);
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(a.u[j]);
      const float2 g = unpack_bf16x2(ww.u[j]);
      o.u[j] = pack_bf16x2(f.x * inv * (g.x + w_offset), f.y * inv * (g.y + w_offset));
    }
    st_bf16x8(outr + v * 8, o);
  }
}

// One block per row, the row and the weights held in registers: one read and one write of every element, one block-wide
// sum. NV = 16-byte vectors per thread. Bound by latency up to a few hundred rows (load, reduction, store), by memory beyond:
// the weights are on their way before the row's sum is known, and a row is spread over as many threads as a block of NV vectors
// per thread takes, so that all SMs have rows already at a batch of about a hundred. (One warp per row, eight rows per block,
// left 8 of 148 SMs at work for 64 rows: 64 x 7168 took 10.8 us and takes 2.3, 128 x 4096 6.5 and 2.1, 4096 x 7168 40.2 and 22.4,
// 5.2 TB/s.)
template <bool HAS_RES, int NV>
__global__ void __launch_bounds__(1024)
rmsnorm_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ out, bf16* __restrict__ residual,
               int H, float eps, float w_offset) {
  __shared__ float red[32];
  const size_t row = blockIdx.x;
  const bf16* xr = x + row * H;
  bf16* rr = HAS_RES ? residual + row * H : nullptr;
  bf16* outr = out + row * H;
  const int nvec = H >> 3;
  bf16x8 a[NV], g[NV];
  pdl_wait();
  pdl_launch_dependents();
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) a[i] = ld_bf16x8(xr + v * 8);
  }
  if constexpr (HAS_RES) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        const bf16x8 b = ld_bf16x8(rr + v * 8);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 fa = unpack_bf16x2(a[i].u[j]);
          const float2 fb = unpack_bf16x2(b.u[j]);
          a[i].u[j] = pack_bf16x2(fa.x + fb.x, fa.y + fb.y);
        }
        st_bf16x8(rr + v * 8, a[i]);  // the sum (rounded to bf16) is the new residual stream
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) g[i] = ld_bf16x8(w + v * 8);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (threadIdx.x + i * blockDim.x < nvec) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(a[i].u[j]);
        ss += f.x * f.x + f.y * f.y;
      }
    }
  }
  ss = warp_reduce_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = warp_reduce_sum((threadIdx.x & 31) < (blockDim.x >> 5) ? red[threadIdx.x & 31] : 0.f);
  const float inv = rsqrtf(ss / static_cast<float>(H) + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      bf16x8 o;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(a[i].u[j]);
        const float2 gg = unpack_bf16x2(g[i].u[j]);
        o.u[j] = pack_bf16x2(f.x * inv * (gg.x + w_offset), f.y * inv * (gg.y + w_offset));
      }
      st_bf16x8(outr + v * 8, o);
    }
  }
}

// One warp per row, the row held in registers between the sum of squares and the scaling: one read
// and one write of every element, no block-wide barrier, eight rows per block. NV = 16-byte vectors per lane (H <= NV * 256).
template <bool HAS_RES, int NV>
__global__ void __launch_bounds__(256)
rmsnorm_warp_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ out,
                    bf16* __restrict__ residual, int T, int H, float eps, float w_offset) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= T) return;
  const bf16* xr = x + static_cast<size_t>(row) * H;
  bf16* rr = HAS_RES ? residual + static_cast<size_t>(row) * H : nullptr;
  bf16* outr = out + static_cast<size_t>(row) * H;
  const int nvec = H >> 3;
  bf16x8 a[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) a[i] = ld_bf16x8(xr + v * 8);
  }
  if constexpr (HAS_RES) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        const bf16x8 b = ld_bf16x8(rr + v * 8);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 fa = unpack_bf16x2(a[i].u[j]);
          const float2 fb = unpack_bf16x2(b.u[j]);
          a[i].u[j] = pack_bf16x2(fa.x + fb.x, fa.y + fb.y);
        }
        st_bf16x8(rr + v * 8, a[i]);  // the sum (rounded to bf16) is the new residual stream
      }
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (lane + 32 * i < nvec) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(a[i].u[j]);
        ss += f.x * f.x + f.y * f.y;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float inv = rsqrtf(ss / static_cast<float>(H) + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) {
      const bf16x8 ww = ld_bf16x8(w + v * 8);
      bf16x8 o;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(a[i].u[j]);
        const float2 g = unpack_bf16x2(ww.u[j]);
        o.u[j] = pack_bf16x2(f.x * inv * (g.x + w_offset), f.y * inv * (g.y + w_offset));
      }
      st_bf16x8(outr + v * 8, o);
    }
  }
}

// Row-strided variant (rows of a column slice of a wider matrix; in place when out == x).
__global__ void __launch_bounds__(256)
rmsnorm_strided_kernel(const bf16* __restrict__ x, int64_t ldx, const bf16* __restrict__ w, bf16* __restrict__ out,
                       int64_t ldo, int H, float eps, float w_offset) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float red[32];
  const size_t row = blockIdx.x;
  const bf16* xr = x + row * ldx;
  bf16* outr = out + row * ldo;
  const int nvec = H >> 3;
  float ss = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const bf16x8 a = ld_bf16x8(xr + v * 8);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(a.u[j]);
      ss += f.x * f.x + f.y * f.y;
    }
  }
  ss = block_reduce_sum(ss, red);
  const float inv = rsqrtf(ss / static_cast<float>(H) + eps);
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const bf16x8 a = ld_bf16x8(xr + v * 8);
    const bf16x8 ww = ld_bf16x8(w + v * 8);
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(a.u[j]);
      const float2 g = unpack_bf16x2(ww.u[j]);
      o.u[j] = pack_bf16x2(f.x * inv * (g.x + w_offset), f.y * inv * (g.y + w_offset));
    }
    st_bf16x8(outr + v * 8, o);
  }
}

// ------------------------------------------------- q/k norm + RoPE + cache scatter
// One warp per (token, head slot). Head slots: [0,Hq) q heads, [Hq,Hq+Hkv) k heads,
// [Hq+Hkv, Hq+2Hkv) v heads. D <= 256, D % 32 == 0... each lane owns D/32 contiguous dims.
// FP8: the caches hold e4m3 bytes; a value is stored as value * inv_scale (saturating), the
// attention kernels multiply by the scale again when they read it (the reference's optional
// fp8 cache: src/parallax_extensions/kernels/reshape_and_cache/reshape_and_cache.metal:32-96).
__device__ __forceinline__ uint8_t to_e4m3(float x) {
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3));
}

template <int D, bool FP8 = false>
__global__ void __launch_bounds__(256)
qk_norm_rope_cache_kernel(bf16* __restrict__ qkv, const bf16* __restrict__ q_norm_w,
                          const bf16* __restrict__ k_norm_w, const float* __restrict__ cos_sin,
                          const int* __restrict__ positions,
                          const int64_t* __restrict__ slot_mapping, void* __restrict__ k_cache,
                          void* __restrict__ v_cache, int T, int Hq, int Hkv, int rot_dim,
                          int page_size, int64_t num_slots, float eps, float w_offset,
                          float k_inv_scale, float v_inv_scale, int max_pos, int* status) {
  constexpr int EPL = D / 32;  // elements per lane
  __shared__ float sh[8][D];
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int heads = Hq + 2 * Hkv;
  const int64_t gw = static_cast<int64_t>(blockIdx.x) * 8 + warp;
  if (gw >= static_cast<int64_t>(T) * heads) return;
  const int t = static_cast<int>(gw / heads);
  const int hs = static_cast<int>(gw % heads);
  bf16* src = qkv + static_cast<size_t>(t) * heads * D + static_cast<size_t>(hs) * D;

  const bool is_q = hs < Hq;
  const bool is_k = !is_q && hs < Hq + Hkv;
  const int64_t slot = slot_mapping ? slot_mapping[t] : -1;

  float v[EPL];
#pragma unroll
  for (int j = 0; j < EPL; ++j) v[j] = __bfloat162float(src[lane * EPL + j]);

  if (is_q || is_k) {
    const bf16* nw = is_q ? q_norm_w : k_norm_w;
    if (nw) {
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < EPL; ++j) ss += v[j] * v[j];
      ss = warp_reduce_sum(ss);
      const float inv = rsqrtf(ss / static_cast<float>(D) + eps);
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        // match a bf16 module: normalised value is rounded before RoPE
        v[j] = __bfloat162float(
            __float2bfloat16(v[j] * inv * (__bfloat162float(nw[lane * EPL + j]) + w_offset)));
      }
    }
    const int p = rot_dim > 0 ? positions[t] : 0;
    const bool p_ok = p >= 0 && (max_pos <= 0 || p < max_pos);
    if (rot_dim > 0 && !p_ok && status && lane == 0) atomicCAS(status, 0, PXL_DEV_BAD_POSITION);
    if (rot_dim > 0 && p_ok) {   // a position outside the table is reported, its row is left unrotated
#pragma unroll
      for (int j = 0; j < EPL; ++j) sh[warp][lane * EPL + j] = v[j];
      __syncwarp();
      const int half = rot_dim >> 1;
      const float* cs = cos_sin + static_cast<size_t>(p) * rot_dim;
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int e = lane * EPL + j;
        if (e < rot_dim) {
          const int i = e < half ? e : e - half;
          const float c = cs[i], s = cs[half + i];
          const float partner = e < half ? -sh[warp][e + half] : sh[warp][e - half];
          v[j] = v[j] * c + partner * s;
        }
      }
    }
  }

  if (is_q) {
#pragma unroll
    for (int j = 0; j < EPL; ++j) src[lane * EPL + j] = __float2bfloat16(v[j]);
    return;
  }
  if (slot < 0) return;
  if (slot >= num_slots) {
    if (status && lane == 0) atomicCAS(status, 0, PXL_DEV_BAD_SLOT);
    return;
  }
  const int kvh = is_k ? hs - Hq : hs - Hq - Hkv;
  const int64_t blk = slot / page_size;
  const int off = static_cast<int>(slot % page_size);
  const int64_t at = ((blk * Hkv + kvh) * page_size + off) * static_cast<int64_t>(D);
  if constexpr (FP8) {
    uint8_t* dst = static_cast<uint8_t*>(is_k ? k_cache : v_cache) + at;
    const float inv = is_k ? k_inv_scale : v_inv_scale;
#pragma unroll
    for (int j = 0; j < EPL; ++j) dst[lane * EPL + j] = to_e4m3(v[j] * inv);
  } else {
    bf16* dst = static_cast<bf16*>(is_k ? k_cache : v_cache) + at;
#pragma unroll
    for (int j = 0; j < EPL; ++j) dst[lane * EPL + j] = __float2bfloat16(v[j]);
  }
}

// The same by 16-byte vectors: 8 elements per lane, D / 8 lanes per head, a block per token (SPLIT: gridDim.y blocks) whose lane
// groups take its heads in turn with the token's cosines and sines in registers. A rotation pairs lane l with l +- rot_dim / 16, so nothing goes through
// shared memory. 5903 rows x 48 heads: 50 us, 2.9 TB/s read and written (86 us with a warp per head and four 2-byte accesses a lane).
template <int D, bool FP8, bool SPLIT>
__global__ void __launch_bounds__(256)
qk_norm_rope_rows_kernel(bf16* __restrict__ qkv, const bf16* __restrict__ q_norm_w, const bf16* __restrict__ k_norm_w,
                         const float* __restrict__ cos_sin, const int* __restrict__ positions,
                         const int64_t* __restrict__ slot_mapping, void* __restrict__ k_cache, void* __restrict__ v_cache, int Hq,
                         int Hkv, int rot_dim, int page_size, int64_t num_slots, float eps, float w_offset, float k_inv_scale,
                         float v_inv_scale, int max_pos, int* status) {
  constexpr int LPH = D / 8, kGroups = 256 / LPH;
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, group = threadIdx.x / LPH, l = threadIdx.x % LPH, e0 = l * 8;
  const int heads = Hq + 2 * Hkv, half = rot_dim >> 1;
  bf16* row = qkv + static_cast<size_t>(t) * heads * D;
  const int64_t slot = slot_mapping ? slot_mapping[t] : -1;
  if (slot >= num_slots && status && threadIdx.x == 0) atomicCAS(status, 0, PXL_DEV_BAD_SLOT);
  const int p = rot_dim > 0 ? positions[t] : 0;
  const bool p_ok = p >= 0 && (max_pos <= 0 || p < max_pos);
  if (rot_dim > 0 && !p_ok && status && threadIdx.x == 0) atomicCAS(status, 0, PXL_DEV_BAD_POSITION);
  const bool turned = rot_dim > 0 && p_ok;  // a position outside the table is reported, its row is left unrotated
  const bool mine = turned && e0 < rot_dim, low = e0 < half;
  float cs[8], sn[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) cs[j] = sn[j] = 0.f;
  if (mine) {
    const float* c = cos_sin + static_cast<size_t>(p) * rot_dim + (low ? e0 : e0 - half);
#pragma unroll
    for (int j = 0; j < 8; ++j) cs[j] = c[j], sn[j] = c[half + j];
  }
  const int lane = threadIdx.x & 31, partner = mine ? (low ? lane + half / 8 : lane - half / 8) : lane;
  int64_t cache_row = -1;  // of head 0
  if (slot >= 0 && slot < num_slots) cache_row = (slot / page_size * Hkv) * page_size + slot % page_size;
  for (int h0 = SPLIT ? blockIdx.y * kGroups : 0; h0 < heads; h0 += SPLIT ? gridDim.y * kGroups : kGroups) {  // (every lane of a warp stays in for the shuffles)
    const int hs = h0 + group;
    const bool in = hs < heads, is_q = hs < Hq, is_k = !is_q && hs < Hq + Hkv;
    const bf16x8 zero8 = {{0u, 0u, 0u, 0u}};
    const bf16x8 x = in ? ld_bf16x8(row + hs * D + e0) : zero8;
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(x.u[j]);
      v[2 * j] = f.x, v[2 * j + 1] = f.y;
    }
    const bf16* nw = is_q ? q_norm_w : is_k ? k_norm_w : nullptr;
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
#pragma unroll
    for (int o = 1; o < LPH; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (nw) {
      const float inv = rsqrtf(ss / static_cast<float>(D) + eps);
      const bf16x8 w = ld_bf16x8(nw + e0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // match a bf16 module: the normalised value is rounded before RoPE
        const float2 f = unpack_bf16x2(w.u[j]);
        v[2 * j] = __bfloat162float(__float2bfloat16(v[2 * j] * inv * (f.x + w_offset)));
        v[2 * j + 1] = __bfloat162float(__float2bfloat16(v[2 * j + 1] * inv * (f.y + w_offset)));
      }
    }
    if (turned) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float other = __shfl_sync(0xffffffffu, v[j], partner);
        if (mine && (is_q || is_k)) v[j] = v[j] * cs[j] + (low ? -other : other) * sn[j];
      }
    }
    if (!in) continue;
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) o.u[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
    if (is_q) {
      st_bf16x8(row + hs * D + e0, o);
      continue;
    }
    if (cache_row < 0) continue;
    const int64_t at = (cache_row + static_cast<int64_t>(is_k ? hs - Hq : hs - Hq - Hkv) * page_size) * D + e0;
    if constexpr (FP8) {
      const float inv = is_k ? k_inv_scale : v_inv_scale;
      uint32_t b[2] = {0u, 0u};
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j >> 2] |= static_cast<uint32_t>(to_e4m3(v[j] * inv)) << (8 * (j & 3));
      *reinterpret_cast<uint2*>(static_cast<uint8_t*>(is_k ? k_cache : v_cache) + at) = make_uint2(b[0], b[1]);
    } else {
      st_bf16x8(static_cast<bf16*>(is_k ? k_cache : v_cache) + at, o);
    }
  }
}

// ------------------------------------------------------------ plain cache scatter
template <bool FP8>
__global__ void __launch_bounds__(256)
reshape_and_cache_kernel(const bf16* __restrict__ k, const bf16* __restrict__ v, int64_t k_stride,
                         int64_t v_stride, const int64_t* __restrict__ slot_mapping,
                         void* __restrict__ k_cache_v, void* __restrict__ v_cache_v, int Hkv, int Dk,
                         int Dv, int page_size, int64_t num_slots, float k_inv_scale,
                         float v_inv_scale, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  using CT = typename std::conditional<FP8, uint8_t, bf16>::type;
  CT* k_cache = static_cast<CT*>(k_cache_v);
  CT* v_cache = static_cast<CT*>(v_cache_v);
  auto conv = [](bf16 x, float inv) -> CT {
    if constexpr (FP8) return to_e4m3(__bfloat162float(x) * inv);
    else return x;
  };
  const int t = blockIdx.x;
  const int64_t slot = slot_mapping[t];
  if (slot < 0) return;
  if (slot >= num_slots) {
    if (status && threadIdx.x == 0) atomicCAS(status, 0, PXL_DEV_BAD_SLOT);
    return;
  }
  const int64_t blk = slot / page_size;
  const int off = static_cast<int>(slot % page_size);
  if (k_cache) {
    for (int i = threadIdx.x; i < Hkv * Dk; i += blockDim.x) {
      const int h = i / Dk, d = i % Dk;
      k_cache[((blk * Hkv + h) * page_size + off) * static_cast<int64_t>(Dk) + d] =
          conv(k[t * k_stride + i], k_inv_scale);
    }
  }
  if (v_cache) {
    for (int i = threadIdx.x; i < Hkv * Dv; i += blockDim.x) {
      const int h = i / Dv, d = i % Dv;
      v_cache[((blk * Hkv + h) * page_size + off) * static_cast<int64_t>(Dv) + d] =
          conv(v[t * v_stride + i], v_inv_scale);
    }
  }
}

// --------------------------------------------------------------- act(gate) * up
__device__ __forceinline__ float act_mul(float g, float u, int mode, float limit) {
  if (mode == 0) return g / (1.f + __expf(-g)) * u;
  if (mode == 1) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.f + __expf(-1.702f * g)) * (u + 1.f);
  }
  const float c = 0.7978845608028654f;
  const float t = tanhf(c * (g + 0.044715f * g * g * g));
  return 0.5f * g * (1.f + t) * u;
}

__global__ void __launch_bounds__(256)
act_mul_kernel(const bf16* __restrict__ x, bf16* __restrict__ out, int I, int mode, float limit) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t row = blockIdx.x;
  const bf16* g = x + row * 2 * I;
  const bf16* u = g + I;
  bf16* o = out + row * I;
  for (int v = threadIdx.x; v < (I >> 3); v += blockDim.x) {
    const bf16x8 a = ld_bf16x8(g + v * 8);
    const bf16x8 b = ld_bf16x8(u + v * 8);
    bf16x8 r;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 fa = unpack_bf16x2(a.u[j]);
      const float2 fb = unpack_bf16x2(b.u[j]);
      r.u[j] = pack_bf16x2(act_mul(fa.x, fb.x, mode, limit), act_mul(fa.y, fb.y, mode, limit));
    }
    st_bf16x8(o + v * 8, r);
  }
}

// --------------------------------------------------------------------- row gather
template <typename IdT>
__global__ void __launch_bounds__(128)
gather_rows_kernel(const bf16* __restrict__ table, const IdT* __restrict__ ids,
                   bf16* __restrict__ out, int H, int64_t num_rows, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t t = blockIdx.x;
  int64_t id = static_cast<int64_t>(ids[t]);
  if (id < 0 || id >= num_rows) {
    if (status && threadIdx.x == 0) atomicCAS(status, 0, PXL_DEV_BAD_ROW_ID);
    id = 0;
  }
  const bf16* src = table + id * H;
  bf16* dst = out + t * H;
  for (int v = threadIdx.x; v < (H >> 3); v += blockDim.x)
    st_bf16x8(dst + v * 8, ld_bf16x8(src + v * 8));
}

__global__ void __launch_bounds__(256) add_inplace_kernel(bf16* y, const bf16* x, int64_t nvec) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nvec) return;
  bf16x8 a = ld_bf16x8(y + i * 8);
  const bf16x8 b = ld_bf16x8(x + i * 8);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 fa = unpack_bf16x2(a.u[j]);
    const float2 fb = unpack_bf16x2(b.u[j]);
    a.u[j] = pack_bf16x2(fa.x + fb.x, fa.y + fb.y);
  }
  st_bf16x8(y + i * 8, a);
}

inline int check_launch() { return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA; }

}  // namespace

PXL_EXPORT int pxl_rmsnorm(const void* x, const void* weight, void* out, void* residual, int T,
                           int H, float eps, float w_offset, pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (H % 8) return PXL_ERR_INVALID_ARG;
  const bf16* xp = static_cast<const bf16*>(x);
  const bf16* wp = static_cast<const bf16*>(weight);
  bf16* op = static_cast<bf16*>(out);
  bf16* rp = static_cast<bf16*>(residual);
  if (H <= 2048 && T >= (H <= 512 ? 1536 : 2048)) {
    // short rows by the thousand: blocks of eight rows, a block for each would be bound by their number (8192 x 1024: 7.2 us
    // against 9.6; 4096 x 1536: 5.9 against 6.1; 1024 rows are better off with a block each, 2.5 against 3.2, and up to 512 columns
    // 1536 rows are as fast either way, 2047 x 256 2.6 and 3.1)
    const unsigned grid = static_cast<unsigned>((T + 7) / 8);
    if (residual)
      pxl_host::launch(rmsnorm_warp_kernel<true, 8>, grid, 256, 0, stream, xp, wp, op, rp, T, H, eps, w_offset);
    else
      pxl_host::launch(rmsnorm_warp_kernel<false, 8>, grid, 256, 0, stream, xp, wp, op, rp, T, H, eps, w_offset);
    return check_launch();
  }
  const int nvec = H >> 3;
  if (H <= 16384 && !(residual && H > 8192 && T >= 1024)) {
    // vectors per thread: two for the shortest chain while the SMs are not full, four once throughput counts (128 x 4096: 2.1 us
    // with two, 2.3 with four; 1016 x 7168: 8.6 and 6.9; 8192 x 4096: 28.7 and 23.2). With a residual a thread has two rows' loads
    // in flight anyway, and a store ahead of the sum: one (16 x 1024: 2.0 us, 2.5 with two; 4096 x 4096: 22.4, and 26.2 with four), up
    // to the width at which that is a block of 1024 threads and many rows want several blocks per SM: 4096 x 12288 71 us, rows read
    // twice 66.
    int nv = residual ? 1 : T < 512 ? 2 : 4;
    while (nvec > nv * 1024) nv *= 2;
    const int threads = pxl::ceil_div(pxl::ceil_div(nvec, nv), 32) * 32;
    auto go = [&](auto kern) { pxl_host::launch(kern, T, threads, 0, stream, xp, wp, op, rp, H, eps, w_offset); };
    if (residual) nv == 1 ? go(rmsnorm_kernel<true, 1>) : go(rmsnorm_kernel<true, 2>);
    else nv == 2 ? go(rmsnorm_kernel<false, 2>) : go(rmsnorm_kernel<false, 4>);
    return check_launch();
  }
  if (residual)
    pxl_host::launch(rmsnorm_long_kernel<true>, T, 256, 0, stream, xp, wp, op, rp, H, eps, w_offset);
  else
    pxl_host::launch(rmsnorm_long_kernel<false>, T, 256, 0, stream, xp, wp, op, static_cast<bf16*>(nullptr), H, eps, w_offset);
  return check_launch();
}

PXL_EXPORT int pxl_rmsnorm_strided(const void* x, int64_t ldx, const void* weight, void* out, int64_t ldo, int T,
                                   int H, float eps, float w_offset, pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if ((H % 8) || (ldx % 8) || (ldo % 8)) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(rmsnorm_strided_kernel, T, 256, 0, stream, static_cast<const bf16*>(x), ldx, static_cast<const bf16*>(weight),
                                                static_cast<bf16*>(out), ldo, H, eps, w_offset);
  return check_launch();
}

namespace {
int qk_norm_rope_cache_impl(void* qkv, const void* q_norm_w, const void* k_norm_w,
                            const float* cos_sin, const int* positions,
                            const int64_t* slot_mapping, void* k_cache, void* v_cache, int T, int Hq,
                            int Hkv, int D, int rot_dim, int page_size, int64_t num_slots, float eps,
                            float norm_w_offset, bool cache_fp8, float k_inv_scale,
                            float v_inv_scale, int max_pos, int* status, pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (rot_dim > D || (rot_dim & 1)) return PXL_ERR_INVALID_ARG;
  // vectors of 16 bytes: whole lanes on either side of a rotation, rows, weights and pages aligned
  const auto off16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  if ((D == 64 || D == 128 || D == 256) && rot_dim % 16 == 0 && !off16(qkv) && !off16(q_norm_w) && !off16(k_norm_w) &&
      !off16(k_cache) && !off16(v_cache)) {
    // A block that walks all heads of its token is a chain of rounds, which few tokens cannot hide: their heads go over as many
    // blocks as keep the chip busy, four of 256 threads per SM. 40 heads, a block per token and this way: 1 token 3.58 and
    // 2.61 us, 48 tokens 3.71 and 2.89, 256 tokens 4.20 and 3.92 (a warp per head: 2.69, 3.15 and 5.74).
    const int rounds = ceil_div(Hq + 2 * Hkv, 256 * 8 / D), room = 4 * pxl_host::num_sms() / T;
    const dim3 grid(T, room < 1 ? 1 : room < rounds ? room : rounds);
    auto go = [&](auto whole, auto split) {
      pxl_host::launch(grid.y > 1 ? split : whole, grid, 256, 0, stream, static_cast<bf16*>(qkv), static_cast<const bf16*>(q_norm_w),
                       static_cast<const bf16*>(k_norm_w), cos_sin, positions, slot_mapping, k_cache, v_cache, Hq, Hkv, rot_dim, page_size,
                       num_slots, eps, norm_w_offset, k_inv_scale, v_inv_scale, max_pos, status);
    };
    if (cache_fp8) {
      if (D == 64) go(qk_norm_rope_rows_kernel<64, true, false>, qk_norm_rope_rows_kernel<64, true, true>);
      else if (D == 128) go(qk_norm_rope_rows_kernel<128, true, false>, qk_norm_rope_rows_kernel<128, true, true>);
      else go(qk_norm_rope_rows_kernel<256, true, false>, qk_norm_rope_rows_kernel<256, true, true>);
    } else {
      if (D == 64) go(qk_norm_rope_rows_kernel<64, false, false>, qk_norm_rope_rows_kernel<64, false, true>);
      else if (D == 128) go(qk_norm_rope_rows_kernel<128, false, false>, qk_norm_rope_rows_kernel<128, false, true>);
      else go(qk_norm_rope_rows_kernel<256, false, false>, qk_norm_rope_rows_kernel<256, false, true>);
    }
    return check_launch();
  }
  const int64_t warps = static_cast<int64_t>(T) * (Hq + 2 * Hkv);
  const unsigned grid = static_cast<unsigned>((warps + 7) / 8);
#define PXL_QKROPE(DD)                                                                        \
  if (cache_fp8)                                                                              \
    pxl_host::launch(qk_norm_rope_cache_kernel<DD, true>, grid, 256, 0, stream,                \
        static_cast<bf16*>(qkv), static_cast<const bf16*>(q_norm_w),                          \
        static_cast<const bf16*>(k_norm_w), cos_sin, positions, slot_mapping, k_cache,        \
        v_cache, T, Hq, Hkv, rot_dim, page_size, num_slots, eps, norm_w_offset, k_inv_scale,  \
        v_inv_scale, max_pos, status);                                                        \
  else                                                                                        \
    pxl_host::launch(qk_norm_rope_cache_kernel<DD, false>, grid, 256, 0, stream,               \
        static_cast<bf16*>(qkv), static_cast<const bf16*>(q_norm_w),                          \
        static_cast<const bf16*>(k_norm_w), cos_sin, positions, slot_mapping, k_cache,        \
        v_cache, T, Hq, Hkv, rot_dim, page_size, num_slots, eps, norm_w_offset, 1.f, 1.f,     \
        max_pos, status)
  switch (D) {
    case 64: PXL_QKROPE(64); break;
    case 96: PXL_QKROPE(96); break;
    case 128: PXL_QKROPE(128); break;
    case 256: PXL_QKROPE(256); break;
    default: return PXL_ERR_INVALID_ARG;
  }
#undef PXL_QKROPE
  return check_launch();
}
}  // namespace

PXL_EXPORT int pxl_qk_norm_rope_cache(void* qkv, const void* q_norm_w, const void* k_norm_w,
                                      const float* cos_sin, const int* positions,
                                      const int64_t* slot_mapping, void* k_cache, void* v_cache,
                                      int T, int Hq, int Hkv, int D, int rot_dim, int page_size,
                                      int64_t num_slots, float eps, float norm_w_offset,
                                      int max_pos, int* status, pxl_stream_t stream) {
  return qk_norm_rope_cache_impl(qkv, q_norm_w, k_norm_w, cos_sin, positions, slot_mapping, k_cache,
                                 v_cache, T, Hq, Hkv, D, rot_dim, page_size, num_slots, eps,
                                 norm_w_offset, false, 1.f, 1.f, max_pos, status, stream);
}

// Same with e4m3 caches: K is stored as k / k_scale, V as v / v_scale (scales > 0).
PXL_EXPORT int pxl_qk_norm_rope_cache_fp8(void* qkv, const void* q_norm_w, const void* k_norm_w,
                                          const float* cos_sin, const int* positions,
                                          const int64_t* slot_mapping, void* k_cache, void* v_cache,
                                          int T, int Hq, int Hkv, int D, int rot_dim, int page_size,
                                          int64_t num_slots, float eps, float norm_w_offset,
                                          float k_scale, float v_scale, int max_pos, int* status,
                                          pxl_stream_t stream) {
  if (!(k_scale > 0.f) || !(v_scale > 0.f)) return PXL_ERR_INVALID_ARG;
  return qk_norm_rope_cache_impl(qkv, q_norm_w, k_norm_w, cos_sin, positions, slot_mapping, k_cache,
                                 v_cache, T, Hq, Hkv, D, rot_dim, page_size, num_slots, eps,
                                 norm_w_offset, true, 1.f / k_scale, 1.f / v_scale, max_pos, status, stream);
}

// dst[dst_idx[i]] = src[src_idx[i]]: the decode rows of a step take their input ids from the token
// tensor that the previous step sampled on the device (the host has not read those tokens yet).
__global__ void patch_i32_kernel(int* __restrict__ dst, const int* __restrict__ dst_idx, const int* __restrict__ src,
                                 const int* __restrict__ src_idx, int n, int dst_len, int src_len, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int d = dst_idx[i], s = src_idx[i];
  if (d < 0 || d >= dst_len || s < 0 || s >= src_len) {
    if (status) atomicCAS(status, 0, PXL_DEV_BAD_ROW_ID);
    return;
  }
  dst[d] = src[s];
}

// Self-test of the bounded peer wait: one thread waits for `flag` to reach `epoch` the way the fused
// kernels wait for a peer. With a flag that nothing sets the wait runs out after its limit (about 1.5 s),
// the kernel records PXL_DEV_TIMEOUT_PEER in *status and returns; *result is 1 if the flag arrived, 0 if
// the wait gave up. The context stays usable either way.
__global__ void bounded_wait_selftest_kernel(const uint32_t* flag, uint32_t epoch, int* result, int* status) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *result = flag_wait_bounded<false>(flag, epoch, nullptr, status) ? 1 : 0;
}

PXL_EXPORT int pxl_selftest_bounded_wait(const uint32_t* flag, uint32_t epoch, int* result, int* status,
                                         pxl_stream_t stream) {
  bounded_wait_selftest_kernel<<<1, 32, 0, stream>>>(flag, epoch, result, status);
  return check_launch();
}

PXL_EXPORT int pxl_patch_i32(int* dst, const int* dst_idx, const int* src, const int* src_idx, int n, int dst_len,
                             int src_len, int* status, pxl_stream_t stream) {
  if (n <= 0) return PXL_OK;
  pxl_host::launch(patch_i32_kernel, (n + 255) / 256, 256, 0, stream, dst, dst_idx, src, src_idx, n, dst_len, src_len, status);
  return check_launch();
}

PXL_EXPORT int pxl_reshape_and_cache(const void* k, const void* v, int64_t k_stride,
                                     int64_t v_stride, const int64_t* slot_mapping, void* k_cache,
                                     void* v_cache, int T, int Hkv, int Dk, int Dv, int page_size,
                                     int64_t num_slots, int* status, pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  pxl_host::launch(reshape_and_cache_kernel<false>, T, 256, 0, stream, static_cast<const bf16*>(k), static_cast<const bf16*>(v), k_stride, v_stride, slot_mapping,
      k_cache, v_cache, Hkv, Dk, Dv, page_size, num_slots, 1.f, 1.f, status);
  return check_launch();
}

PXL_EXPORT int pxl_reshape_and_cache_fp8(const void* k, const void* v, int64_t k_stride,
                                         int64_t v_stride, const int64_t* slot_mapping,
                                         void* k_cache, void* v_cache, int T, int Hkv, int Dk, int Dv,
                                         int page_size, int64_t num_slots, float k_scale,
                                         float v_scale, int* status, pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (!(k_scale > 0.f) || !(v_scale > 0.f)) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(reshape_and_cache_kernel<true>, T, 256, 0, stream, static_cast<const bf16*>(k), static_cast<const bf16*>(v), k_stride, v_stride, slot_mapping,
      k_cache, v_cache, Hkv, Dk, Dv, page_size, num_slots, 1.f / k_scale, 1.f / v_scale, status);
  return check_launch();
}

PXL_EXPORT int pxl_act_mul(const void* x, void* out, int T, int I, int mode, float limit,
                           pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (I % 8) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(act_mul_kernel, T, 256, 0, stream, static_cast<const bf16*>(x), static_cast<bf16*>(out), I,
                                        mode, limit);
  return check_launch();
}

PXL_EXPORT int pxl_gather_rows(const void* table, const void* ids, void* out, int T, int H,
                               int64_t num_rows, int ids_are_i64, int* status,
                               pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (H % 8) return PXL_ERR_INVALID_ARG;
  if (ids_are_i64)
    pxl_host::launch(gather_rows_kernel<int64_t>, T, 128, 0, stream, static_cast<const bf16*>(table),
                                                       static_cast<const int64_t*>(ids),
                                                       static_cast<bf16*>(out), H, num_rows,
                                                       status);
  else
    pxl_host::launch(gather_rows_kernel<int>, T, 128, 0, stream, static_cast<const bf16*>(table),
                                                   static_cast<const int*>(ids),
                                                   static_cast<bf16*>(out), H, num_rows, status);
  return check_launch();
}

PXL_EXPORT int pxl_add_inplace(void* y, const void* x, int64_t n, pxl_stream_t stream) {
  if (n <= 0) return PXL_OK;
  if (n % 8) return PXL_ERR_INVALID_ARG;
  const int64_t nvec = n / 8;
  pxl_host::launch(add_inplace_kernel, static_cast<unsigned>((nvec + 255) / 256), 256, 0, stream, static_cast<bf16*>(y), static_cast<const bf16*>(x), nvec);
  return check_launch();
}
