// Gated delta rule of the hybrid families, with one decay per head and token (Qwen3-Next / Qwen3.5):
//
//   S <- e^(g_t) S    d = b_t (v_t - S k_t)    S <- S + d k_t^T    o_t = S q_t
//   g_t = -exp(A_log) softplus(a_t + dt_bias)    b_t = sigmoid(b_t)    q, k unit vectors, q times dk^-1/2
//   out = rmsnorm(o_t) * norm_w * silu(z_t)
//
// The state [slots, Hv, Dv, 128] fp32 lives in per-request slots; a sequence whose first token of this step sits at position 0
// starts from zero. Counterpart of mlx-lm's gated_delta_update, through which the reference runs these layers
// (src/parallax/models/qwen3_next.py:149-230). Two forms:
//
//  * steps (decoding, unaligned rows): a CTA per (head, sequence) keeps the whole state in registers, 8 lanes per row of 128,
//    so that a warp's loads are whole 128-byte lines; S k and S q come out of one pass (o = e^g S q + (k . q) d). One pass
//    over the state: bound by memory. 96 rows x 32 heads of 128 x 128: 75 us, 5.3 TB/s of state read and written (134 us
//    with one thread per row of the state).
//  * chunks of 64 tokens (prompts), three kernels. With G_t the sum of g over the chunk up to t,
//        A_tj = b_t k_t.k_j e^(G_t - G_j)  (j < t)     P_tj = q_t.k_j e^(G_t - G_j)  (j <= t)     X = (1 + A)^-1 diag(b)
//        u = X (v - e^G K S_0)     o = e^G Q S_0 + P u     S_end = e^(G_n) S_0 + K^T (e^(G_n - G) u)
//    The first makes X and P of every chunk and head in parallel, the second walks the chunks of a (sequence, head, 32 columns
//    of v) with S in registers, the third norms and gates the heads. Because the decay is one number per token it stays out of
//    the products with q, k and v, which enter the tensor cores as the bf16 numbers they are; what is fp32 (S, X, P, u)
//    enters as the sum of three bf16 numbers, with every partial product above 2^-24, the triangular system is solved in fp32,
//    and o stays fp32 up to the norm. No exponent is positive. The kept state's error against 64 bits after 16 slices of 257
//    tokens is 0.8e-7 to 3.0e-7 for decays of 0.0025 to 7 per token (sums of two bf16 numbers: 3.4e-6 to 6.6e-6, and 314 us for the
//    walk). The walk is a chain of chunks, bound by the latency of its four products and three barriers; everything it reads is
//    one chunk ahead. Two prompts of 2950 tokens, 32 heads: 107 + 474 + 47 us for the three kernels (8.0 ms token by token);
//    their working space is at most 256 MB, longer prompts go through it in runs.
//
// This file is compiled without fast math: what enters the recurrence uses the accurate functions.
#include "common.cuh"
#include "pxl_api.h"

namespace {
using namespace pxl;

constexpr int DK = 128;      // key columns
constexpr int kChunk = 64;   // tokens of a chunk
constexpr int kBlock = 16;
constexpr int kSlice = 32;   // columns of v per CTA of the walk
constexpr float kUnitEps = 1e-6f;

struct GdArgs {
  const bf16* qkv;  // [T, ld]: q | k | v heads, behind the convolution
  int64_t ld;
  const bf16 *a, *b;  // [T, ld_ab]
  int64_t ld_ab;
  const float *A_log, *dt_bias;
  const bf16* z;
  int64_t ld_z;
  const bf16* norm_w;
  float* state;
  const int *seq_cu, *seq_slots, *positions;
  bf16* out;
  int64_t ldo;
  int Hk, Hv, Dv;
  float eps;
};

__device__ __forceinline__ float log_decay(const GdArgs& a, int t, int h) {
  const float z = __bfloat162float(a.a[t * a.ld_ab + h]) + a.dt_bias[h];
  return -expf(a.A_log[h]) * (fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))));
}
__device__ __forceinline__ float rate(const GdArgs& a, int t, int h) {
  return 1.f / (1.f + expf(-__bfloat162float(a.b[t * a.ld_ab + h])));
}
__device__ __forceinline__ float silu(float v) { return v / (1.f + expf(-v)); }

template <bool VEC>
__device__ __forceinline__ void load4(const bf16* p, float* v) {
  if constexpr (VEC) {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    const float2 x = unpack_bf16x2(w.x), y = unpack_bf16x2(w.y);
    v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __bfloat162float(p[j]);
  }
}

// ---- steps -------------------------------------------------------------------------------------------------
// 256 threads: 8 lanes x 32 rows, 4 rows per thread. Columns 4 l + 32 j (j = 0..3) of a row belong to lane l.
// VEC: rows of q and k start on 8 bytes.
template <bool VEC>
__global__ void __launch_bounds__(256, 2) delta_step_kernel(const GdArgs a, int seq0) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float red[2][8];
  const int hv = blockIdx.x, seq = seq0 + blockIdx.y, hk = hv / (a.Hv / a.Hk);
  const int l = threadIdx.x & 7, r0 = threadIdx.x >> 3, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = a.seq_cu[seq], t1 = a.seq_cu[seq + 1];
  if (t1 <= t0) return;
  const bool fresh = a.positions[t0] == 0;
  float* Sg = a.state + (static_cast<int64_t>(a.seq_slots[seq]) * a.Hv + hv) * a.Dv * DK + l * 4;
  float S[4][16];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!fresh && r0 + 32 * i < a.Dv) v = *reinterpret_cast<const float4*>(Sg + (r0 + 32 * i) * DK + j * 32);
      S[i][4 * j] = v.x, S[i][4 * j + 1] = v.y, S[i][4 * j + 2] = v.z, S[i][4 * j + 3] = v.w;
    }
  for (int t = t0; t < t1; ++t) {
    const bf16* row = a.qkv + t * a.ld;
    float q[16], k[16], qq = 0.f, kk = 0.f, qk = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      load4<VEC>(row + hk * DK + l * 4 + j * 32, q + 4 * j);
      load4<VEC>(row + (a.Hk + hk) * DK + l * 4 + j * 32, k + 4 * j);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      qq = fmaf(q[j], q[j], qq);
      kk = fmaf(k[j], k[j], kk);
      qk = fmaf(q[j], k[j], qk);
    }
    // What a long memory loses per token is a small difference from one: S + (e^g - 1) S does without the rounding of e^g, which
    // adds up over hundreds of tokens (16 x 257 tokens, decays of 0.0025: state error 7.2e-6, 6.7e-7 this way, in the same time; a
    // branch between two loops instead of the select takes 96 us for the 80 of 96 rows).
    const float g = log_decay(a, t, hv), beta = rate(a, t, hv);
    const bool slow = g > -0.5f;
    const float decay = slow ? expm1f(g) : expf(g);
    auto decayed = [&](float x) { return slow ? fmaf(decay, x, x) : decay * x; };
    float sk[4], sq[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sk[i] = sq[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        sk[i] = fmaf(S[i][j], k[j], sk[i]);
        sq[i] = fmaf(S[i][j], q[j], sq[i]);
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      qq += __shfl_xor_sync(0xffffffffu, qq, o);
      kk += __shfl_xor_sync(0xffffffffu, kk, o);
      qk += __shfl_xor_sync(0xffffffffu, qk, o);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sk[i] += __shfl_xor_sync(0xffffffffu, sk[i], o);
        sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
      }
    }
    const float ik = 1.f / sqrtf(kk + kUnitEps), iq = 1.f / sqrtf((qq + kUnitEps) * DK);
    float o[4], o2 = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + 32 * i;
      const float v = r < a.Dv ? __bfloat162float(row[2 * a.Hk * DK + hv * a.Dv + r]) : 0.f;
      const float d = (v - decayed(sk[i]) * ik) * beta;
      o[i] = decayed(sq[i]) * iq + qk * iq * ik * d;
      o2 = fmaf(o[i], o[i], o2);
      const float dk = d * ik;
#pragma unroll
      for (int j = 0; j < 16; ++j) S[i][j] = fmaf(dk, k[j], fmaf(decay, S[i][j], slow ? S[i][j] : 0.f));
    }
    // norm over the head: a row's 8 lanes hold the same number
    o2 += __shfl_xor_sync(0xffffffffu, o2, 8);
    o2 += __shfl_xor_sync(0xffffffffu, o2, 16);
    float* part = red[t & 1];  // two sets: a slow warp may still read the last token's
    if (lane == 0) part[warp] = o2;
    __syncthreads();
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) sum += part[w];
    const float inv = 1.f / sqrtf(sum / a.Dv + a.eps);
    const float mine = l == 0 ? o[0] : l == 1 ? o[1] : l == 2 ? o[2] : o[3];
    const int r = r0 + 32 * l;
    if (l < 4 && r < a.Dv)
      a.out[t * a.ldo + hv * a.Dv + r] = __float2bfloat16(mine * inv * __bfloat162float(a.norm_w[r]) *
                                                          silu(__bfloat162float(a.z[t * a.ld_z + hv * a.Dv + r])));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (r0 + 32 * i < a.Dv)
        *reinterpret_cast<float4*>(Sg + (r0 + 32 * i) * DK + j * 32) =
            make_float4(S[i][4 * j], S[i][4 * j + 1], S[i][4 * j + 2], S[i][4 * j + 3]);
}

// ---- chunks ------------------------------------------------------------------------------------------------
// What the kernels hand on, per (chunk, head), in bytes: X and P [64][64] fp32, factors of the rows, o
struct Record {
  static constexpr int X = 0, P = X + kChunk * kChunk * 4;
  static constexpr int F = P + kChunk * kChunk * 4;  // fp32: e^G ik | e^G iq | e^(G_n - G) ik | e^(G_n), padded to 256
  static constexpr int kFactors = 4 * kChunk;
  static constexpr int O = F + kFactors * 4;  // [64][Dv] fp32
  __host__ __device__ static int64_t bytes(int Dv) { return O + static_cast<int64_t>(kChunk) * Dv * 4; }
};

// Two fp32 numbers as sums of three bf16 numbers each (rounding 2^-27: none that fp32 does not have).
struct Parts {
  uint32_t v[3];
};
__device__ __forceinline__ Parts split3(float a, float b) {
  Parts p;
  p.v[0] = pack_bf16x2(a, b);
  float2 f = unpack_bf16x2(p.v[0]);
  a -= f.x, b -= f.y;
  p.v[1] = pack_bf16x2(a, b);
  f = unpack_bf16x2(p.v[1]);
  p.v[2] = pack_bf16x2(a - f.x, b - f.y);
  return p;
}

// chunk number `id` of the prompt slices: sequence and number within it; false past the last one. Warp-collective.
__device__ __forceinline__ bool find_chunk(const int* seq_cu, int seqs, int id, int& seq, int& index) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int s0 = 0; s0 < seqs; s0 += 32) {
    const int s = s0 + lane, n = s < seqs ? (seq_cu[s + 1] - seq_cu[s] + kChunk - 1) / kChunk : 0;
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    const unsigned past = __ballot_sync(0xffffffffu, base + sum > id);
    if (past) {
      const int w = __ffs(past) - 1;
      seq = s0 + w;
      index = id - base - __shfl_sync(0xffffffffu, sum - n, w);
      return true;
    }
    base += __shfl_sync(0xffffffffu, sum, 31);
  }
  return false;
}
// chunks of the sequences before `seq`. Warp-collective.
__device__ __forceinline__ int chunks_before(const int* seq_cu, int seq) {
  int n = 0;
  for (int s = threadIdx.x & 31; s < seq; s += 32) n += (seq_cu[s + 1] - seq_cu[s] + kChunk - 1) / kChunk;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}

constexpr int kPitch = DK + 8, kPitchF = kChunk + 4;

struct MakeSmem {
  bf16 q[kChunk][kPitch], k[kChunk][kPitch];
  float A[kChunk][kPitchF];  // below the diagonal
  float X[kChunk][kPitchF];  // (1 + A)^-1, blocks up to the diagonal
  float tmp[3][kBlock][kBlock + 4];
  float iq[kChunk], ik[kChunk], b[kChunk], gh[kChunk], gl[kChunk];  // G as the sum of two fp32 numbers
};

constexpr int kMakeThreads = 256;

// grid (chunks, heads). Warps 0 to 3: 16 rows of A each, warps 4 to 7: of P.
__global__ void __launch_bounds__(kMakeThreads) delta_make_kernel(const GdArgs a, int seqs, int chunk0, uint8_t* __restrict__ work) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t raw[];
  MakeSmem& s = *reinterpret_cast<MakeSmem*>(raw);
  const int h = blockIdx.y, hk = h / (a.Hv / a.Hk), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int seq, index;
  if (!find_chunk(a.seq_cu, seqs, chunk0 + blockIdx.x, seq, index)) return;
  const int t0 = a.seq_cu[seq] + index * kChunk, left = a.seq_cu[seq + 1] - t0, n = left < kChunk ? left : kChunk;
  uint8_t* rec = work + (static_cast<int64_t>(blockIdx.x) * a.Hv + h) * Record::bytes(a.Dv);
  const bf16* x = a.qkv + static_cast<int64_t>(t0) * a.ld;

  for (int i = tid; i < kChunk * (DK / 8); i += kMakeThreads) {
    const int r = i / (DK / 8), c = i % (DK / 8) * 8;
    const bf16* row = x + static_cast<int64_t>(r < n ? r : 0) * a.ld;
    cp_async_16(smem_u32(&s.q[r][c]), row + hk * DK + c, r < n);
    cp_async_16(smem_u32(&s.k[r][c]), row + (a.Hk + hk) * DK + c, r < n);
  }
  cp_async_commit();
  if (warp == 0) {  // sums of the log decays, two tokens per lane
    const int t = lane * 2;
    const double g0 = t < n ? log_decay(a, t0 + t, h) : 0.f, g1 = t + 1 < n ? log_decay(a, t0 + t + 1, h) : 0.f;
    double sum = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    const double first = sum - g1;
    s.gh[t] = static_cast<float>(first), s.gl[t] = static_cast<float>(first - static_cast<float>(first));
    s.gh[t + 1] = static_cast<float>(sum), s.gl[t + 1] = static_cast<float>(sum - static_cast<float>(sum));
  } else if (warp < 3) {
    const int t = (warp - 1) * 32 + lane;
    s.b[t] = t < n ? rate(a, t0 + t, h) : 0.f;
  }
  cp_async_wait<0>();
  __syncthreads();
  {  // the factors that make q and k unit vectors
    const int r = tid >> 2, part = tid & 3;
    float qq = 0.f, kk = 0.f;
#pragma unroll
    for (int i = 0; i < DK / 32; ++i) {
      const bf16x8 q = ld_bf16x8(&s.q[r][(i * 4 + part) * 8]), k = ld_bf16x8(&s.k[r][(i * 4 + part) * 8]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 qf = unpack_bf16x2(q.u[j]), kf = unpack_bf16x2(k.u[j]);
        qq += qf.x * qf.x + qf.y * qf.y;
        kk += kf.x * kf.x + kf.y * kf.y;
      }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      qq += __shfl_xor_sync(0xffffffffu, qq, o);
      kk += __shfl_xor_sync(0xffffffffu, kk, o);
    }
    if (part == 0) {
      s.iq[r] = 1.f / sqrtf((qq + kUnitEps) * DK);
      s.ik[r] = 1.f / sqrtf(kk + kUnitEps);
    }
  }
  __syncthreads();

  // ---- K K^T and Q K^T, blocks up to the diagonal
  const int g8 = lane >> 2, t2 = (lane & 3) * 2, mi = lane >> 3, r8 = lane & 7;
  {
    const bool score = warp >= 4;
    const int rb = warp & 3, row = rb * kBlock;
    const bf16(*rows)[kPitch] = score ? s.q : s.k;
    float d[4][2][4] = {};
    const uint32_t a_base = smem_u32(&rows[row + (lane & 15)][(lane >> 4) * 8]);
    const uint32_t b_base = smem_u32(&s.k[(mi >> 1) * 8 + r8][(mi & 1) * 8]);
#pragma unroll
    for (int kk = 0; kk < DK / 16; ++kk) {
      uint32_t af[4];
      ldmatrix_x4(af, a_base + kk * 32);
#pragma unroll
      for (int cb = 0; cb < 4; ++cb) {
        if (cb > rb) continue;
        uint32_t bfr[4];
        ldmatrix_x4(bfr, b_base + cb * kBlock * kPitch * 2 + kk * 32);
        const uint32_t b0[2] = {bfr[0], bfr[1]}, b1[2] = {bfr[2], bfr[3]};
        mma_m16n8k16_bf16(d[cb][0], af, b0);
        mma_m16n8k16_bf16(d[cb][1], af, b1);
      }
    }
#pragma unroll
    for (int cb = 0; cb < 4; ++cb) {
      if (cb > rb) continue;
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int t = row + g8 + e * 8, j = cb * kBlock + u * 8 + t2;
          float w[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const bool in = score ? j + c <= t : j + c < t;
            const float decay = in ? expf((s.gh[t] - s.gh[j + c]) + (s.gl[t] - s.gl[j + c])) : 0.f;
            w[c] = d[cb][u][2 * e + c] * decay * s.ik[j + c] * (score ? s.iq[t] : s.b[t] * s.ik[t]);
          }
          *reinterpret_cast<float2*>(score ? reinterpret_cast<float*>(rec + Record::P) + t * kChunk + j : &s.A[t][j]) =
              make_float2(w[0], w[1]);
        }
    }
  }
  if (tid < kChunk) {
    float* f = reinterpret_cast<float*>(rec + Record::F);
    const float e = expf(s.gh[tid]);
    f[tid] = e * s.ik[tid];
    f[kChunk + tid] = e * s.iq[tid];
    f[2 * kChunk + tid] = expf((s.gh[kChunk - 1] - s.gh[tid]) + (s.gl[kChunk - 1] - s.gl[tid])) * s.ik[tid];
    f[3 * kChunk + tid] = expf(s.gh[kChunk - 1]);
  }
  __syncthreads();

  // ---- X: the blocks on the diagonal, a column per thread, then the blocks below, one diagonal after the other
  if (tid < kChunk) {
    const int base = tid / kBlock * kBlock, c = tid % kBlock;
    float y[kBlock];
#pragma unroll
    for (int t = 0; t < kBlock; ++t) {
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < t; ++j) sum = fmaf(s.A[base + t][base + j], y[j], sum);
      y[t] = t == c ? 1.f : t < c ? 0.f : -sum;
      s.X[base + t][base + c] = y[t];
    }
  }
  __syncthreads();
  const int blk = tid >> 6, er = (tid & 63) >> 2, ec = (tid & 3) * 4;  // a block; a row and 4 columns of it
#pragma unroll
  for (int d = 1; d < kChunk / kBlock; ++d) {
    const int i0 = (blk + d) * kBlock, j0 = blk * kBlock;
    const bool mine = blk + d < kChunk / kBlock;
    if (mine) {
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int m = j0; m < i0; ++m) {
        const float w = s.A[i0 + er][m];
        const float4 v = *reinterpret_cast<const float4*>(&s.X[m][j0 + ec]);
        sum.x = fmaf(w, v.x, sum.x), sum.y = fmaf(w, v.y, sum.y), sum.z = fmaf(w, v.z, sum.z), sum.w = fmaf(w, v.w, sum.w);
      }
      *reinterpret_cast<float4*>(&s.tmp[blk][er][ec]) = sum;
    }
    __syncthreads();
    if (mine) {
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int m = 0; m < kBlock; ++m) {
        const float w = -s.X[i0 + er][i0 + m];
        const float4 v = *reinterpret_cast<const float4*>(&s.tmp[blk][m][ec]);
        sum.x = fmaf(w, v.x, sum.x), sum.y = fmaf(w, v.y, sum.y), sum.z = fmaf(w, v.z, sum.z), sum.w = fmaf(w, v.w, sum.w);
      }
      *reinterpret_cast<float4*>(&s.X[i0 + er][j0 + ec]) = sum;
    }
    __syncthreads();
  }
  for (int i = tid; i < kChunk * kChunk / 4; i += kMakeThreads) {
    const int t = i / (kChunk / 4), j = i % (kChunk / 4) * 4;
    if (j / kBlock > t / kBlock) continue;  // (the walk does not use the blocks above the diagonal)
    const float4 v = *reinterpret_cast<const float4*>(&s.X[t][j]);
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(rec + Record::X) + t * kChunk + j) =
        make_float4(v.x * s.b[j], v.y * s.b[j + 1], v.z * s.b[j + 2], v.w * s.b[j + 3]);
  }
}

constexpr int kPitchM = kChunk + 8;  // pairs of a quarter warp's rows hit distinct banks

struct WalkStage {
  bf16 q[kChunk][kPitch], k[kChunk][kPitch];
  float x[kChunk][kPitchM], p[kChunk][kPitchM];
  bf16 v[kChunk][kSlice + 8];
  float f[Record::kFactors];
};
struct WalkSmem {  // [3]: the parts of fp32 numbers
  WalkStage st[2];
  bf16 s[3][DK][kSlice + 8];
  bf16 r[3][kChunk][kSlice + 8];  // v - e^G K S
  bf16 u[3][kChunk][kSlice + 8];
  bf16 d[3][kChunk][kSlice + 8];  // e^(G_n - G) ik u
};
static_assert(sizeof(WalkSmem) <= 227 * 1024, "shared memory of a CTA");

template <int ROWS>
__device__ __forceinline__ void put_parts(bf16 (&dst)[3][ROWS][kSlice + 8], int r, int c, float a, float b) {
  const Parts p = split3(a, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(&dst[i][r][c]) = p.v[i];
}

// acc[0] + acc[1] + acc[2] += M B for 16 rows of an fp32 matrix and 16 rows x 16 columns of an operand in parts: the six products
// that are not below fp32's rounding, those of a size in an accumulator of their own.
template <int ROWS>
__device__ __forceinline__ void mul_parts(float (&acc)[3][2][4], const float (&m)[kChunk][kPitchM], int row, int col,
                                          const bf16 (&b)[3][ROWS][kSlice + 8], int k0, int c0) {
  const int lane = threadIdx.x & 31, mi = lane >> 3, r8 = lane & 7, g8 = lane >> 2, t2 = (lane & 3) * 2;
  uint32_t a[3][4], bp[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = *reinterpret_cast<const float2*>(&m[row + g8 + (i & 1) * 8][col + t2 + (i >> 1) * 8]);
    const Parts p = split3(v.x, v.y);
    a[0][i] = p.v[0], a[1][i] = p.v[1], a[2][i] = p.v[2];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) ldmatrix_x4_trans(bp[i], smem_u32(&b[i][k0 + (mi & 1) * 8 + r8][c0 + (mi >> 1) * 8]));
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; i + j < 3; ++j)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const uint32_t b2[2] = {bp[j][2 * n], bp[j][2 * n + 1]};
        mma_m16n8k16_bf16(acc[i + j][n], a[i], b2);
      }
}

// Warps 0 to 7 make u and keep the state, warps 8 to 15 make the outputs.
constexpr int kHalf = 8, kWalkThreads = 2 * kHalf * 32;

// grid (slices of v, heads, sequences): the chunks [chunk0, chunk0 + chunks) of one sequence, in order
__global__ void __launch_bounds__(kWalkThreads, 1) delta_walk_kernel(const GdArgs a, int chunk0, int chunks, uint8_t* __restrict__ work) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t raw[];
  WalkSmem& s = *reinterpret_cast<WalkSmem*>(raw);
  const int h = blockIdx.y, hk = h / (a.Hv / a.Hk), seq = blockIdx.z, v0 = blockIdx.x * kSlice;
  const int t0 = a.seq_cu[seq], n_all = a.seq_cu[seq + 1] - t0;
  const int mine = (n_all + kChunk - 1) / kChunk, base = chunks_before(a.seq_cu, seq);
  const int first = chunk0 > base ? chunk0 - base : 0, last = chunk0 + chunks - base < mine ? chunk0 + chunks - base : mine;
  if (first >= last) return;  // chunks of this sequence in the range: [first, last)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mi = lane >> 3, r8 = lane & 7, g8 = lane >> 2, t2 = (lane & 3) * 2;
  float* Sg = a.state + ((static_cast<int64_t>(a.seq_slots[seq]) * a.Hv + h) * a.Dv + v0) * DK;
  const bool fresh = first == 0 && a.positions[t0] == 0;
  auto record = [&](int i) { return work + (static_cast<int64_t>(base + i - chunk0) * a.Hv + h) * Record::bytes(a.Dv); };

  auto load = [&](int i) {
    WalkStage& st = s.st[i & 1];
    const uint8_t* rec = record(i);
    const int c0 = i * kChunk, n = n_all - c0 < kChunk ? n_all - c0 : kChunk;
    const bf16* x = a.qkv + static_cast<int64_t>(t0 + c0) * a.ld;
    for (int j = tid; j < kChunk * (DK / 8); j += kWalkThreads) {
      const int r = j / (DK / 8), c = j % (DK / 8) * 8;
      const bf16* row = x + static_cast<int64_t>(r < n ? r : 0) * a.ld;
      cp_async_16(smem_u32(&st.q[r][c]), row + hk * DK + c, r < n);
      cp_async_16(smem_u32(&st.k[r][c]), row + (a.Hk + hk) * DK + c, r < n);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {  // pieces of 16 bytes, 1024 in each of the two matrices
      const int r = tid / (kChunk / 4) + j * (kChunk / 2), c = tid % (kChunk / 4) * 4;
      if (c / kBlock > r / kBlock) continue;
      cp_async_16(smem_u32(&st.x[r][c]), rec + Record::X + (r * kChunk + c) * 4, true);
      cp_async_16(smem_u32(&st.p[r][c]), rec + Record::P + (r * kChunk + c) * 4, true);
    }
    if (tid < kChunk * (kSlice / 8)) {
      const int r = tid / (kSlice / 8), c = tid % (kSlice / 8) * 8;
      cp_async_16(smem_u32(&st.v[r][c]), x + static_cast<int64_t>(r < n ? r : 0) * a.ld + 2 * a.Hk * DK + h * a.Dv + v0 + c, r < n);
    } else if (tid < kChunk * (kSlice / 8) + Record::kFactors / 4) {
      const int c = (tid - kChunk * (kSlice / 8)) * 4;
      cp_async_16(smem_u32(&st.f[c]), rec + Record::F + c * 4, true);
    }
  };
  static_assert(kChunk * kChunk / 4 == 2 * kWalkThreads, "two pieces of X and P per thread");
  load(first);
  cp_async_commit();
  if (first + 1 < last) load(first + 1);
  cp_async_commit();

  // the keepers: rows 16 w of the state (key columns), all 32 columns of v, in the layout of the accumulators
  const bool keeper = warp < kHalf;
  const int w8 = warp % kHalf, rg = w8 & 3, ch = w8 >> 2;  // 16 tokens; half of the slice's columns
  float S[4][4];
  auto publish = [&]() {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) put_parts(s.s, w8 * 16 + g8 + e * 8, j * 8 + t2, S[j][2 * e], S[j][2 * e + 1]);
  };
  if (keeper) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        S[j][e] = fresh ? 0.f : Sg[static_cast<int64_t>(j * 8 + t2 + (e & 1)) * DK + w8 * 16 + g8 + (e >> 1) * 8];
    publish();
  }

  for (int i = first; i < last; ++i) {
    const WalkStage& st = s.st[i & 1];
    cp_async_wait<1>();
    __syncthreads();
    // ---- K S and Q S: 16 tokens x 16 columns per warp
    float o[2][4], part[3][2][4] = {};
    {
      const uint32_t rows = smem_u32(keeper ? &st.k[rg * 16 + (lane & 15)][(lane >> 4) * 8] : &st.q[rg * 16 + (lane & 15)][(lane >> 4) * 8]);
#pragma unroll
      for (int kk = 0; kk < DK / 16; ++kk) {
        uint32_t x[4], sp[4];
        ldmatrix_x4(x, rows + kk * 32);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          ldmatrix_x4_trans(sp, smem_u32(&s.s[i][kk * 16 + (mi & 1) * 8 + r8][ch * 16 + (mi >> 1) * 8]));
          const uint32_t b0[2] = {sp[0], sp[1]}, b1[2] = {sp[2], sp[3]};
          mma_m16n8k16_bf16(part[i][0], x, b0);
          mma_m16n8k16_bf16(part[i][1], x, b1);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        o[j][e] = (part[0][j][e] + (part[1][j][e] + part[2][j][e])) * st.f[(keeper ? 0 : kChunk) + rg * 16 + g8 + (e >> 1) * 8];
    if (keeper) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = rg * 16 + g8 + e * 8, c = ch * 16 + j * 8 + t2;
          const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(&st.v[r][c]));
          put_parts(s.r, r, c, v.x - o[j][2 * e], v.y - o[j][2 * e + 1]);
        }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // the keepers
      // ---- u = X (v - e^G K S)
      float u[3][2][4] = {};
      for (int kk = 0; kk <= rg; ++kk) mul_parts(u, st.x, rg * 16, kk * 16, s.r, kk * 16, ch * 16);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = rg * 16 + g8 + e * 8, c = ch * 16 + j * 8 + t2;
          const float w = st.f[2 * kChunk + r];
          const float x = u[0][j][2 * e] + (u[1][j][2 * e] + u[2][j][2 * e]);
          const float y = u[0][j][2 * e + 1] + (u[1][j][2 * e + 1] + u[2][j][2 * e + 1]);
          put_parts(s.u, r, c, x, y);
          put_parts(s.d, r, c, x * w, y * w);
        }
    }
    __syncthreads();
    if (!keeper) {
      // ---- o += P u (blocks up to this one)
      float pu[3][2][4] = {};
      for (int kk = 0; kk <= rg; ++kk) mul_parts(pu, st.p, rg * 16, kk * 16, s.u, kk * 16, ch * 16);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] += pu[0][j][e] + (pu[1][j][e] + pu[2][j][e]);
      float* og = reinterpret_cast<float*>(record(i) + Record::O) + v0;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<float2*>(og + static_cast<int64_t>(rg * 16 + g8 + e * 8) * a.Dv + ch * 16 + j * 8 + t2) =
              make_float2(o[j][2 * e], o[j][2 * e + 1]);
    } else {
      // ---- S = e^(G_n) S + K^T (e^(G_n - G) ik u)
      const float gn = st.f[3 * kChunk];
      float add[3][4][4] = {};
#pragma unroll
      for (int kk = 0; kk < kChunk / 16; ++kk) {
        uint32_t k[4];
        ldmatrix_x4_trans(k, smem_u32(&st.k[kk * 16 + (mi >> 1) * 8 + r8][w8 * 16 + (mi & 1) * 8]));
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            uint32_t dp[4];
            ldmatrix_x4_trans(dp, smem_u32(&s.d[i][kk * 16 + (mi & 1) * 8 + r8][c * 16 + (mi >> 1) * 8]));
            const uint32_t b0[2] = {dp[0], dp[1]}, b1[2] = {dp[2], dp[3]};
            mma_m16n8k16_bf16(add[i][2 * c], k, b0);
            mma_m16n8k16_bf16(add[i][2 * c + 1], k, b1);
          }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j][e] = fmaf(gn, S[j][e], add[0][j][e] + (add[1][j][e] + add[2][j][e]));
      publish();  // every read of the old state happened before the last barrier
    }
    __syncthreads();
    if (i + 2 < last) load(i + 2);  // into the stage that was just used
    cp_async_commit();
  }
  if (keeper) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        Sg[static_cast<int64_t>(j * 8 + t2 + (e & 1)) * DK + w8 * 16 + g8 + (e >> 1) * 8] = S[j][e];
  }
}

// grid (chunks, heads), a warp per token: out = rmsnorm(o) * norm_w * silu(z)
__global__ void __launch_bounds__(256) delta_norm_kernel(const GdArgs a, int seqs, int chunk0, const uint8_t* __restrict__ work) {
  pdl_wait();
  pdl_launch_dependents();
  const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int seq, index;
  if (!find_chunk(a.seq_cu, seqs, chunk0 + blockIdx.x, seq, index)) return;
  const int t0 = a.seq_cu[seq] + index * kChunk, left = a.seq_cu[seq + 1] - t0, n = left < kChunk ? left : kChunk;
  const float* o = reinterpret_cast<const float*>(work + (static_cast<int64_t>(blockIdx.x) * a.Hv + h) * Record::bytes(a.Dv) + Record::O);
  const int c = lane * 4;
  const bool live = c < a.Dv;
  float w[4] = {};
  if (live) {
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = __bfloat162float(a.norm_w[c + j]);
  }
  for (int r = warp; r < n; r += 8) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    uint2 zr = make_uint2(0u, 0u);
    const int64_t t = t0 + r;
    if (live) {
      v = *reinterpret_cast<const float4*>(o + static_cast<int64_t>(r) * a.Dv + c);
      zr = *reinterpret_cast<const uint2*>(a.z + t * a.ld_z + h * a.Dv + c);
    }
    const float inv = 1.f / sqrtf(warp_reduce_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) / a.Dv + a.eps);
    const float2 z0 = unpack_bf16x2(zr.x), z1 = unpack_bf16x2(zr.y);
    if (live)
      *reinterpret_cast<uint2*>(a.out + t * a.ldo + h * a.Dv + c) =
          make_uint2(pack_bf16x2(v.x * inv * w[0] * silu(z0.x), v.y * inv * w[1] * silu(z0.y)),
                     pack_bf16x2(v.z * inv * w[2] * silu(z1.x), v.w * inv * w[3] * silu(z1.y)));
  }
}

// The chunks are worked off in runs whose records fit the workspace.
int launch_chunked(const GdArgs& a, int seqs, int tokens, uint8_t* work, int64_t work_bytes, cudaStream_t stream) {
  static bool done[64] = {false};
  const int dev = pxl_host::current_device_slot();
  if (!done[dev]) {
    if (cudaFuncSetAttribute(delta_make_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(MakeSmem)) != cudaSuccess ||
        cudaFuncSetAttribute(delta_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(WalkSmem)) != cudaSuccess)
      return PXL_ERR_CUDA;
    done[dev] = true;
  }
  const int bound = tokens / kChunk + seqs;  // at most this many chunks
  const int64_t fit = work_bytes / (Record::bytes(a.Dv) * a.Hv);
  if (fit < 1 || seqs > 65535 || a.Hv > 65535) return PXL_ERR_TOO_LARGE;
  const int run = fit < bound ? static_cast<int>(fit) : bound;
  for (int c0 = 0; c0 < bound; c0 += run) {
    const int n = bound - c0 < run ? bound - c0 : run;
    pxl_host::launch(delta_make_kernel, dim3(n, a.Hv), kMakeThreads, sizeof(MakeSmem), stream, a, seqs, c0, work);
    pxl_host::launch(delta_walk_kernel, dim3(a.Dv / kSlice, a.Hv, seqs), kWalkThreads, sizeof(WalkSmem), stream, a, c0, n, work);
    pxl_host::launch(delta_norm_kernel, dim3(n, a.Hv), 256, 0, stream, a, seqs, c0, work);
  }
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

inline bool aligned(const void* p, int bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

// rows of 16 bytes (q, k, v), gates and outputs of 8: what the copies and stores of the chunked kernels take
inline bool chunkable(const GdArgs& a) {
  return a.Dv % kSlice == 0 && a.ld % 8 == 0 && aligned(a.qkv, 16) && a.ld_z % 4 == 0 && aligned(a.z, 8) && a.ldo % 4 == 0 &&
         aligned(a.out, 8);
}
}  // namespace

PXL_EXPORT int64_t pxl_gated_delta_workspace(int Hv, int Dv, int prefill_seqs, int prefill_tokens) {
  if (prefill_seqs <= 0 || Dv % kSlice) return 0;
  const int64_t one = Record::bytes(Dv) * Hv, all = one * (prefill_tokens / kChunk + prefill_seqs), cap = 256ll << 20;
  return all < cap ? all : one > cap ? one : cap / one * one;
}

PXL_EXPORT int pxl_gated_delta_rule(const void* qkv, int64_t ld_qkv, const void* a_in, const void* b_in, int64_t ld_ab,
                                    const float* A_log, const float* dt_bias, const void* z, int64_t ld_z,
                                    const void* norm_w, float* rec_state, const int* seq_cu, const int* seq_slots,
                                    const int* positions, void* out, int64_t ld_out, int B, int Hk, int Hv, int Dk,
                                    int Dv, float eps, int prefill_seqs, int prefill_tokens, void* work, int64_t work_bytes,
                                    cudaStream_t stream) {
  if (B <= 0) return PXL_OK;
  if (Dk != DK || Dv > 128 || Dv <= 0 || Hk <= 0 || Hv % Hk) return PXL_ERR_INVALID_ARG;
  const GdArgs a{static_cast<const pxl::bf16*>(qkv), ld_qkv, static_cast<const pxl::bf16*>(a_in), static_cast<const pxl::bf16*>(b_in),
                 ld_ab, A_log, dt_bias, static_cast<const pxl::bf16*>(z), ld_z, static_cast<const pxl::bf16*>(norm_w), rec_state,
                 seq_cu, seq_slots, positions, static_cast<pxl::bf16*>(out), ld_out, Hk, Hv, Dv, eps};
  int done = 0;
  if (prefill_seqs > 0 && work != nullptr && chunkable(a)) {
    const int code = launch_chunked(a, prefill_seqs, prefill_tokens, static_cast<uint8_t*>(work), work_bytes, stream);
    if (code != PXL_OK) return code;
    done = prefill_seqs;
  }
  const bool vec = ld_qkv % 4 == 0 && aligned(qkv, 8);
  for (; done < B; done += 65535) {
    const dim3 grid(Hv, B - done < 65535 ? B - done : 65535);
    if (vec) pxl_host::launch(delta_step_kernel<true>, grid, 256, 0, stream, a, done);
    else pxl_host::launch(delta_step_kernel<false>, grid, 256, 0, stream, a, done);
  }
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}
