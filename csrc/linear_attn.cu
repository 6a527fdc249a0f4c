// Gated DeltaNet linear-attention layers (Qwen3-Next / Qwen3.5 hybrids): short causal convolution with a carried window, and
// the gates around the mixers (the recurrence itself is in gated_delta.cu).
//
//   conv:   y[t, c] = silu( sum_j w[c, j] * u[t - (K-1) + j, c] ),  u = [carried window | x]
// The window lives in per-request slots [slots, C, K-1] bf16; a sequence whose first token of this step sits at position 0
// starts from zeros. The reference runs these layers through mlx-lm (src/parallax/models/qwen3_next.py:149-230) and keeps the
// states in a LinearCache (src/parallax/server/cache/linear_cache.py).
#include "common.cuh"
#include "pxl_api.h"

namespace {
using namespace pxl;

constexpr int kMaxConvK = 8;

// Decoded tokens (and sizes the kernel below does not take): grid (channel blocks, sequences); thread = one channel, walks the
// sequence's tokens in order
__global__ void __launch_bounds__(128) conv1d_silu_kernel(const bf16* __restrict__ x, int64_t ldx,
                                                          const bf16* __restrict__ w, const bf16* __restrict__ bias,
                                                          bf16* __restrict__ conv_state, const int* __restrict__ seq_cu,
                                                          const int* __restrict__ seq_slots,
                                                          const int* __restrict__ positions, bf16* __restrict__ out,
                                                          int64_t ldo, int C, int K) {
  pdl_wait();
  pdl_launch_dependents();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (c >= C) return;
  const int t0 = seq_cu[b], t1 = seq_cu[b + 1];
  if (t1 <= t0) return;
  const int slot = seq_slots[b];
  const bool fresh = positions[t0] == 0;
  float win[kMaxConvK];  // win[0..K-2] = previous inputs, oldest first
  float wk[kMaxConvK];
  bf16* st = conv_state + (static_cast<size_t>(slot) * C + c) * (K - 1);
  for (int j = 0; j < K - 1; ++j) win[j] = fresh ? 0.f : __bfloat162float(st[j]);
  for (int j = 0; j < K; ++j) wk[j] = __bfloat162float(w[c * K + j]);
  const float bs = bias ? __bfloat162float(bias[c]) : 0.f;
  for (int t = t0; t < t1; ++t) {
    const float xin = __bfloat162float(x[t * ldx + c]);
    float acc = bs + wk[K - 1] * xin;
    for (int j = 0; j < K - 1; ++j) acc += wk[j] * win[j];
    for (int j = 0; j + 1 < K - 1; ++j) win[j] = win[j + 1];
    win[K - 2] = xin;
    out[t * ldo + c] = __float2bfloat16(acc / (1.f + __expf(-acc)));
  }
  for (int j = 0; j < K - 1; ++j) st[j] = __float2bfloat16(win[j]);
}

// The same for windows of three (K = 4) and a pair of channels per thread: 12 bytes of window, 16 of weights and 4 of input are
// three independent vector loads, and the loops are known, so that nothing is kept in local memory. One token of 96 sequences x
// 8192 channels: 12.1 -> 5.5 us.
__global__ void __launch_bounds__(128) conv1d_silu_pair_kernel(const bf16* __restrict__ x, int64_t ldx, const bf16* __restrict__ w,
                                                               const bf16* __restrict__ bias, bf16* __restrict__ conv_state,
                                                               const int* __restrict__ seq_cu, const int* __restrict__ seq_slots,
                                                               const int* __restrict__ positions, bf16* __restrict__ out, int64_t ldo,
                                                               int C) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 2, b = blockIdx.y;
  pdl_wait();
  pdl_launch_dependents();
  if (c >= C) return;
  const int t0 = seq_cu[b], t1 = seq_cu[b + 1];
  if (t1 <= t0) return;
  const bool fresh = positions[t0] == 0;
  uint32_t* st = reinterpret_cast<uint32_t*>(conv_state + (static_cast<size_t>(seq_slots[b]) * C + c) * 3);
  const uint4 wr = *reinterpret_cast<const uint4*>(w + static_cast<size_t>(c) * 4);
  const uint32_t br = bias ? *reinterpret_cast<const uint32_t*>(bias + c) : 0u;
  uint32_t sr[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) sr[j] = fresh ? 0u : st[j];
  const float2 w0 = unpack_bf16x2(wr.x), w1 = unpack_bf16x2(wr.y), w2 = unpack_bf16x2(wr.z), w3 = unpack_bf16x2(wr.w);
  const float wk[2][4] = {{w0.x, w0.y, w1.x, w1.y}, {w2.x, w2.y, w3.x, w3.y}};
  const float2 bs = unpack_bf16x2(br), s0 = unpack_bf16x2(sr[0]), s1 = unpack_bf16x2(sr[1]), s2 = unpack_bf16x2(sr[2]);
  float win[2][3] = {{s0.x, s0.y, s1.x}, {s1.y, s2.x, s2.y}};  // oldest first
  for (int t = t0; t < t1; ++t) {
    const float2 in = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(x + t * ldx + c));
    float y[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float xin = e ? in.y : in.x;
      float acc = (e ? bs.y : bs.x) + wk[e][3] * xin;
#pragma unroll
      for (int j = 0; j < 3; ++j) acc += wk[e][j] * win[e][j];
      win[e][0] = win[e][1], win[e][1] = win[e][2], win[e][2] = xin;
      y[e] = acc / (1.f + __expf(-acc));
    }
    *reinterpret_cast<uint32_t*>(out + t * ldo + c) = pack_bf16x2(y[0], y[1]);
  }
  st[0] = pack_bf16x2(win[0][0], win[0][1]);
  st[1] = pack_bf16x2(win[0][2], win[1][0]);
  st[2] = pack_bf16x2(win[1][1], win[1][2]);
}

// Prompts: a thread walks a run of tokens of 8 channels, weights and last inputs in registers, inputs four tokens ahead. The
// walk of a whole sequence by one thread (above) is a chain of as many loads as it has tokens (2.0 ms for 5900 tokens x 8192
// channels); runs make it a streaming pass (57 us, 3.4 TB/s read and written). The slots are rewritten by a launch of its own, because the first tokens of a
// slice read what its last ones replace.
template <int K>
__global__ void __launch_bounds__(128) conv_run_kernel(const bf16* __restrict__ x, int64_t ldx, const bf16* __restrict__ w,
                                                       const bf16* __restrict__ bias, const bf16* __restrict__ conv_state,
                                                       const int* __restrict__ seq_cu, const int* __restrict__ seq_slots,
                                                       const int* __restrict__ positions, bf16* __restrict__ out, int64_t ldo,
                                                       int C, int seqs, int tokens, int run) {
  pdl_wait();
  pdl_launch_dependents();
  const int c = (blockIdx.x * 128 + threadIdx.x) * 8;
  if (c >= C) return;
  const int first = blockIdx.y * run, last = first + run < tokens ? first + run : tokens;
  int seq = 0;
  for (int hi = seqs - 1; seq < hi;) {  // the last sequence that starts at or before the run
    const int mid = (seq + hi + 1) >> 1;
    if (seq_cu[mid] <= first) seq = mid; else hi = mid - 1;
  }
  int end = seq_cu[seq + 1], start = seq_cu[seq];
  float wk[8][K], b0[8], hist[K - 1][8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
#pragma unroll
    for (int j = 0; j < K; ++j) wk[e][j] = __bfloat162float(w[(c + e) * K + j]);
    b0[e] = bias ? __bfloat162float(bias[c + e]) : 0.f;
  }
  auto unpack = [](const bf16x8& v, float (&f)[8]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 p = unpack_bf16x2(v.u[j]);
      f[2 * j] = p.x, f[2 * j + 1] = p.y;
    }
  };
  constexpr int kAhead = 4;
  const bf16x8 zero8 = {{0u, 0u, 0u, 0u}};
  const bf16* cur = x + first * ldx + c;
  bf16x8 ahead[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) ahead[i] = first + i < last ? ld_bf16x8(cur + i * ldx) : zero8;
  for (int t4 = first; t4 < last; t4 += kAhead) {
#pragma unroll
    for (int i4 = 0; i4 < kAhead; ++i4, cur += ldx) {
      const int t = t4 + i4;
      if (t >= last) break;
      while (end <= t) ++seq, start = end, end = seq_cu[seq + 1];
      if (t == first || t == start) {  // the inputs before this run, or of this sequence's earlier steps
        const int li = t - start;
        const bool fresh = li < K - 1 && positions[start] == 0;
#pragma unroll
        for (int j = 0; j < K - 1; ++j) {
          const int back = K - 1 - j;  // hist[j] is the input `back` tokens ago
          if (back <= li) {
            unpack(ld_bf16x8(cur - back * ldx), hist[j]);
          } else {
            const bf16* st = conv_state + (static_cast<size_t>(seq_slots[seq]) * C + c) * (K - 1) + li + j;
#pragma unroll
            for (int e = 0; e < 8; ++e) hist[j][e] = fresh ? 0.f : __bfloat162float(st[e * (K - 1)]);
          }
        }
      }
      float here[8];
      unpack(ahead[i4], here);
      if (t + kAhead < last) ahead[i4] = ld_bf16x8(cur + kAhead * ldx);
      bf16x8 o;
      float y[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        y[e] = b0[e] + wk[e][K - 1] * here[e];
#pragma unroll
        for (int j = 0; j < K - 1; ++j) y[e] += wk[e][j] * hist[j][e];
#pragma unroll
        for (int j = 0; j + 1 < K - 1; ++j) hist[j][e] = hist[j + 1][e];
        hist[K - 2][e] = here[e];
        y[e] = y[e] / (1.f + __expf(-y[e]));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) o.u[j] = pack_bf16x2(y[2 * j], y[2 * j + 1]);
      st_bf16x8(out + t * ldo + c, o);
    }
  }
}

// the slots of the prompt slices: the last K - 1 inputs (of older steps where the slice is shorter)
__global__ void __launch_bounds__(128) conv_window_kernel(const bf16* __restrict__ x, int64_t ldx, bf16* __restrict__ conv_state,
                                                          const int* __restrict__ seq_cu, const int* __restrict__ seq_slots,
                                                          const int* __restrict__ positions, int C, int K) {
  pdl_wait();
  pdl_launch_dependents();
  const int c = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
  if (c >= C) return;
  const int t0 = seq_cu[b], n = seq_cu[b + 1] - t0;
  if (n <= 0) return;
  const bool fresh = positions[t0] == 0;
  bf16* st = conv_state + (static_cast<size_t>(seq_slots[b]) * C + c) * (K - 1);
  for (int j = 0; j < K - 1; ++j) {
    const int li = n - (K - 1) + j;
    st[j] = li >= 0 ? x[(t0 + li) * ldx + c] : fresh ? __float2bfloat16(0.f) : st[j + n];
  }
}

// false: sizes or alignments that the kernel above does not take
bool launch_conv_run(const bf16* x, int64_t ldx, const bf16* w, const bf16* bias, bf16* conv_state, const int* seq_cu,
                     const int* seq_slots, const int* positions, bf16* out, int64_t ldo, int C, int K, int seqs, int tokens,
                     cudaStream_t stream) {
  if (C % 8 || ldx % 8 || ldo % 8 || K > 4 || seqs > 65535 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15))
    return false;
  const int blocks = ceil_div(C, 1024);
  // enough threads for every SM, runs long enough that a run's first loads do not count
  int run = ceil_div(tokens * blocks, 8 * pxl_host::num_sms());
  run = run < 4 ? 4 : run > 64 ? 64 : run;
  while (ceil_div(tokens, run) > 65535) run *= 2;
  const dim3 grid(blocks, ceil_div(tokens, run));
  const auto kern = K == 2 ? conv_run_kernel<2> : K == 3 ? conv_run_kernel<3> : conv_run_kernel<4>;
  pxl_host::launch(kern, grid, 128, 0, stream, x, ldx, w, bias, conv_state, seq_cu, seq_slots, positions, out, ldo, C, seqs, tokens, run);
  pxl_host::launch(conv_window_kernel, dim3(ceil_div(C, 128), seqs), 128, 0, stream, x, ldx, conv_state, seq_cu, seq_slots, positions, C, K);
  return true;
}

__global__ void sigmoid_gate_mul_kernel(const bf16* __restrict__ x, int64_t ldx, const bf16* __restrict__ gate,
                                        int64_t ldg, bf16* __restrict__ out, int64_t ldo, int n8) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  for (int v = threadIdx.x; v < n8; v += blockDim.x) {
    const bf16x8 a = ld_bf16x8(x + t * ldx + v * 8), g = ld_bf16x8(gate + t * ldg + v * 8);
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 av = unpack_bf16x2(a.u[j]), gv = unpack_bf16x2(g.u[j]);
      o.u[j] = pack_bf16x2(av.x / (1.f + __expf(-gv.x)), av.y / (1.f + __expf(-gv.y)));
    }
    st_bf16x8(out + t * ldo + v * 8, o);
  }
}

// out = (res +) x * sigmoid(gate[:, col / group]): one gate value per `group` consecutive columns (a head of the
// attention output, or a whole row for the shared expert's scalar gate); group is a multiple of 8
__global__ void gate_mul_grouped_kernel(const bf16* __restrict__ x, int64_t ldx, const bf16* __restrict__ gate,
                                        int64_t ldg, const bf16* __restrict__ res, int64_t ldr,
                                        bf16* __restrict__ out, int64_t ldo, int n8, int group8) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  for (int v = threadIdx.x; v < n8; v += blockDim.x) {
    const float g = __bfloat162float(gate[t * ldg + v / group8]);
    const float s = 1.f / (1.f + __expf(-g));
    const bf16x8 a = ld_bf16x8(x + t * ldx + v * 8);
    bf16x8 r;
    if (res != nullptr) r = ld_bf16x8(res + t * ldr + v * 8);
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 av = unpack_bf16x2(a.u[j]);
      float2 ov = make_float2(av.x * s, av.y * s);
      if (res != nullptr) {
        const float2 rv = unpack_bf16x2(r.u[j]);
        ov.x += rv.x;
        ov.y += rv.y;
      }
      o.u[j] = pack_bf16x2(ov.x, ov.y);
    }
    st_bf16x8(out + t * ldo + v * 8, o);
  }
}

// out[t] = x[t, :] . w  (one warp per row; the one-column projection of a scalar gate is too thin for a GEMM tile)
__global__ void row_dot_kernel(const bf16* __restrict__ x, int64_t ldx, const bf16* __restrict__ w,
                               bf16* __restrict__ out, int T, int k8) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (t >= T) return;
  const int lane = threadIdx.x % 32;
  float acc = 0.f;
  for (int v = lane; v < k8; v += 32) {
    const bf16x8 a = ld_bf16x8(x + t * ldx + v * 8), b = ld_bf16x8(w + v * 8);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 av = unpack_bf16x2(a.u[j]), bv = unpack_bf16x2(b.u[j]);
      acc += av.x * bv.x + av.y * bv.y;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) out[t] = __float2bfloat16(acc);
}

}  // namespace

PXL_EXPORT int pxl_causal_conv1d_silu(const void* x_, int64_t ldx, const void* w_, const void* bias_, void* conv_state_,
                                      const int* seq_cu, const int* seq_slots, const int* positions, void* out_,
                                      int64_t ldo, int B, int C, int K, int prefill_seqs, int prefill_tokens, cudaStream_t stream) {
  if (B <= 0) return PXL_OK;
  if (K < 2 || K > kMaxConvK) return PXL_ERR_INVALID_ARG;
  const auto *x = static_cast<const pxl::bf16*>(x_), *w = static_cast<const pxl::bf16*>(w_), *bias = static_cast<const pxl::bf16*>(bias_);
  auto *conv_state = static_cast<pxl::bf16*>(conv_state_), *out = static_cast<pxl::bf16*>(out_);
  int done = 0;
  if (prefill_seqs > 0 && prefill_tokens > 0 &&
      launch_conv_run(x, ldx, w, bias, conv_state, seq_cu, seq_slots, positions, out, ldo, C, K, prefill_seqs, prefill_tokens, stream))
    done = prefill_seqs;
  if (done < B) {
    // pairs of channels where rows and the tables start on the bytes that they take
    const bool pairs = K == 4 && C % 2 == 0 && ldx % 2 == 0 && ldo % 2 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
                       ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(conv_state) |
                         reinterpret_cast<uintptr_t>(out)) & 3) == 0;
    if (pairs)
      pxl_host::launch(conv1d_silu_pair_kernel, dim3(pxl::ceil_div(C, 256), B - done), 128, 0, stream, x, ldx, w, bias, conv_state,
                       seq_cu + done, seq_slots + done, positions, out, ldo, C);
    else
      pxl_host::launch(conv1d_silu_kernel, dim3(pxl::ceil_div(C, 128), B - done), 128, 0, stream, x, ldx, w, bias, conv_state,
                       seq_cu + done, seq_slots + done, positions, out, ldo, C, K);
  }
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

PXL_EXPORT int pxl_sigmoid_gate_mul(const void* x, int64_t ldx, const void* gate, int64_t ldg, void* out,
                                    int64_t ldo, int T, int N, cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (N % 8) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(sigmoid_gate_mul_kernel, T, 128, 0, stream, static_cast<const pxl::bf16*>(x), ldx,
                                                 static_cast<const pxl::bf16*>(gate), ldg,
                                                 static_cast<pxl::bf16*>(out), ldo, N / 8);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

PXL_EXPORT int pxl_gate_mul_grouped(const void* x, int64_t ldx, const void* gate, int64_t ldg, const void* res,
                                    int64_t ldr, void* out, int64_t ldo, int T, int N, int group,
                                    cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (N % 8 || group <= 0 || group % 8 || N % group) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(gate_mul_grouped_kernel, T, 128, 0, stream, static_cast<const pxl::bf16*>(x), ldx,
                                                 static_cast<const pxl::bf16*>(gate), ldg,
                                                 static_cast<const pxl::bf16*>(res), ldr,
                                                 static_cast<pxl::bf16*>(out), ldo, N / 8, group / 8);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}

PXL_EXPORT int pxl_row_dot(const void* x, int64_t ldx, const void* w, void* out, int T, int K, cudaStream_t stream) {
  if (T <= 0) return PXL_OK;
  if (K % 8) return PXL_ERR_INVALID_ARG;
  pxl_host::launch(row_dot_kernel, pxl::ceil_div(T, 4), 128, 0, stream, static_cast<const pxl::bf16*>(x), ldx,
                                                          static_cast<const pxl::bf16*>(w),
                                                          static_cast<pxl::bf16*>(out), T, K / 8);
  return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
}
