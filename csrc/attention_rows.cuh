// Softmax of the prefill attention kernels in which a thread owns a query row: 128 scores of a tile from tensor memory, P back to
// their place as bf16 (the A operand of the second product), O of 128 columns rescaled there when a maximum makes it necessary.
#pragma once

#include "attention_score.cuh"
#include "tc_issue.cuh"

namespace pxl {

__device__ __forceinline__ uint64_t pair2(float a, float b) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ float2 unpair2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// One tile. `masked(j)`: column j is not visible (asked unless `interior`). m_run: reference maximum, in log2 units; l2: row sums
// in two pairs. p_ready: barriers of the two halves of P, one arrival per warp. Warp-collective.
template <int SM, typename Masked>
__device__ __forceinline__ void softmax_tile(uint32_t my_s, uint32_t my_o, bool first, bool interior, Masked masked, float scale_log2,
                                             const ScoreArgs& sa, float bias2, float& m_run, uint64_t (&l2)[2], uint32_t p_ready) {
  constexpr int kT = 128, kD = 128;
  uint32_t sc[kT];
#pragma unroll
  for (int c = 0; c < kT; c += 32) tmem_ld_32x32b_x32(my_s + c, *reinterpret_cast<uint32_t(*)[32]>(&sc[c]));
  tmem_ld_wait();
  if constexpr (SM == kCapped) {
#pragma unroll
    for (int j = 0; j < kT; ++j) sc[j] = __float_as_uint(score_log2<SM>(__uint_as_float(sc[j]), 0.f, sa));
  }
  if (!interior) {
#pragma unroll
    for (int j = 0; j < kT; ++j)
      if (masked(j)) sc[j] = 0xff800000u;  // -inf
  }
  if constexpr (SM != kSigmoid) {
    float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < kT; j += 8) {
#pragma unroll
      for (int k = 0; k < 4; ++k) m4[k] = fmaxf(fmaxf(m4[k], __uint_as_float(sc[j + k])), __uint_as_float(sc[j + 4 + k]));
    }
    const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * (SM == kCapped ? 1.f : scale_log2);  // scale > 0
    const float m_new = fmaxf(m_run, mx);
    // O accumulates relative to m_run, which only moves when a row of the warp grew by more than 2^8: until then the stale
    // reference keeps every probability below 256, which bf16 and the fp32 sums hold without trouble
    if (first) {
      m_run = m_new;
    } else if (__any_sync(0xffffffffu, m_new > m_run + 8.f)) {
      const float corr = fast_exp2(m_run - (m_new == -INFINITY ? 0.f : m_new));
      m_run = m_new;
      const uint64_t c2 = pair2(corr, corr);
      l2[0] = fma2(l2[0], c2, 0ull), l2[1] = fma2(l2[1], c2, 0ull);
#pragma unroll
      for (int c = 0; c < kD; c += 16) {
        uint32_t v[16];
        tmem_ld_32x32b_x16(my_o + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
        tmem_st_32x32b_x16(my_o + c, v);
      }
    }
  }
  const float m_use = (m_run == -INFINITY) ? 0.f : m_run;
  const uint64_t scale2 = pair2(scale_log2, scale_log2), neg_m2 = pair2(-m_use, -m_use);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int c = h * 64; c < h * 64 + 64; c += 32) {
      uint32_t pk[16];
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float s0 = __uint_as_float(sc[c + j]), s1 = __uint_as_float(sc[c + j + 1]);
        float p0, p1;
        if constexpr (SM == kSigmoid) {
          p0 = sigmoid_weight(s0, scale_log2, bias2);  // (a masked score, -inf, gives 0)
          p1 = sigmoid_weight(s1, scale_log2, bias2);
        } else if constexpr (SM == kCapped) {
          p0 = fast_exp2(s0 - m_use);
          p1 = fast_exp2(s1 - m_use);
        } else {
          const float2 x = unpair2(fma2(pair2(s0, s1), scale2, neg_m2));
          p0 = fast_exp2(x.x);
          p1 = fast_exp2(x.y);
        }
        l2[(j >> 1) & 1] = add2(l2[(j >> 1) & 1], pair2(p0, p1));
        pk[j >> 1] = pack_bf16x2(p0, p1);
      }
      tmem_st_32x32b_x16(my_s + c / 2, pk);
    }
    tmem_st_wait();
    tc_fence_before_sync();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(p_ready + 8 * h);
  }
}

// 128 columns of this thread's row of O times `inv` to dst. Warp-collective.
__device__ __forceinline__ void store_row(uint32_t my_o, float inv, bf16* dst, bool valid) {
#pragma unroll
  for (int c = 0; c < 128; c += 32) {
    uint32_t v[32];
    tmem_ld_32x32b_x32(my_o + c, v);
    tmem_ld_wait();
#pragma unroll
    for (int c8 = 0; c8 < 32; c8 += 8) {
      bf16x8 ov;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        ov.u[j] = pack_bf16x2(__uint_as_float(v[c8 + 2 * j]) * inv, __uint_as_float(v[c8 + 2 * j + 1]) * inv);
      if (valid) st_bf16x8(dst + c + c8, ov);
    }
  }
}

}  // namespace pxl
