// Mixture-of-experts support kernels: top-k routing, token permutation (alignment to
// 128-row expert tiles), gather, and weighted combine. The expert FFNs themselves run on the
// grouped tcgen05 GEMM (gemm_tcgen05.cu).
//
// Routing semantics:
//   mode 0  softmax over all experts, top-k, optional renormalisation (Qwen3-MoE, GPT-OSS
//           style; the reference gets it from mlx-lm's switch layers, src/parallax/models/
//           qwen3_moe.py)
//           With a correction bias the choice is by score + bias, the weights stay the scores.
//   mode 1  sigmoid scores, selection on score + per-expert correction bias with optional
//           group-limited routing, weights = unbiased scores renormalised and scaled
//           (DeepSeek-V3 "noaux_tc"; MiniMax-M3 uses the ungrouped form,
//           src/parallax/models/minimax_m3.py:155-173)
// In either mode the choice can be limited to the topk_group best of n_group groups of neighbouring experts; a
// group counts as its best selection score (group_top 1) or the sum of its two best (group_top 2).
#include "common.cuh"
#include "pxl_api.h"

namespace {
using namespace pxl;

constexpr int kMaxEPL = 16;  // experts per lane: supports up to 512 experts

template <bool BF16>
__device__ __forceinline__ float load_score(const void* p, size_t i) {
  if constexpr (BF16) return __bfloat162float(static_cast<const bf16*>(p)[i]);
  else return static_cast<const float*>(p)[i];
}

// One warp per token; EPL: experts a lane holds (expert e belongs to lane e % 32).
template <bool BF16, int EPL>
__global__ void __launch_bounds__(128)
moe_route_kernel(const void* __restrict__ logits, int64_t ld, const float* __restrict__ e_bias, int T, int E,
                 int k, int mode, int renorm, int n_group, int topk_group, int group_top, float routed_scale,
                 int* __restrict__ out_ids, float* __restrict__ out_w) {
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + warp;
  if (t >= T) return;
  const int epl = (E + 31) / 32;
  float s[EPL];    // unbiased score (softmax prob or sigmoid)
  float sel[EPL];  // selection score
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    const int e = j * 32 + lane;
    s[j] = (j < epl && e < E) ? load_score<BF16>(logits, static_cast<size_t>(t) * ld + e) : -INFINITY;
    mx = fmaxf(mx, s[j]);
  }
  if (mode == 0) {
    mx = warp_reduce_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      s[j] = (s[j] == -INFINITY) ? 0.f : __expf(s[j] - mx);
      sum += s[j];
    }
    sum = warp_reduce_sum(sum);
    const float inv = 1.f / sum;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      const int e = j * 32 + lane;
      s[j] *= inv;
      sel[j] = (j < epl && e < E) ? s[j] + (e_bias ? e_bias[e] : 0.f) : -INFINITY;
    }
  } else {
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      const int e = j * 32 + lane;
      const bool ok = j < epl && e < E;
      s[j] = ok ? 1.f / (1.f + __expf(-s[j])) : 0.f;
      sel[j] = ok ? s[j] + (e_bias ? e_bias[e] : 0.f) : -INFINITY;
    }
  }
  if (n_group > 1 && topk_group < n_group) {
    // group score: its best selection score, or the sum of its two best
    const int gsize = E / n_group;
    float gscore_mine = -INFINITY;  // lane g (< n_group) holds the score of group g
    for (int g = 0; g < n_group; ++g) {
      float b1 = -INFINITY, b2 = -INFINITY;
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int e = j * 32 + lane;
        if (j < epl && e < E && e / gsize == g) {
          if (sel[j] > b1) { b2 = b1; b1 = sel[j]; }
          else if (sel[j] > b2) b2 = sel[j];
        }
      }
      // merge (b1, b2) pairs across lanes
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float o1 = __shfl_xor_sync(0xffffffffu, b1, o);
        const float o2 = __shfl_xor_sync(0xffffffffu, b2, o);
        const float n1 = fmaxf(b1, o1);
        const float n2 = fmaxf(fminf(b1, o1), fmaxf(b2, o2));
        b1 = n1; b2 = n2;
      }
      if (lane == g) gscore_mine = b1 + (group_top == 1 || b2 == -INFINITY ? 0.f : b2);
    }
    // pick topk_group groups; keep a bitmask of allowed groups (n_group <= 32)
    unsigned allowed = 0;
    float gs = lane < n_group ? gscore_mine : -INFINITY;
    for (int it = 0; it < topk_group; ++it) {
      float best = gs;
      int arg = lane;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
        if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
      }
      allowed |= 1u << arg;
      if (lane == arg) gs = -INFINITY;
    }
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      const int e = j * 32 + lane;
      if (j < epl && e < E && !((allowed >> (e / gsize)) & 1u)) sel[j] = -INFINITY;
    }
  }
  // iterative top-k over the warp
  float wsum = 0.f;
  float my_w = 0.f;
  int my_id = 0;
  for (int it = 0; it < k; ++it) {
    float best = -INFINITY;
    int arg = 0x7fffffff;
    float best_s = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      const int e = j * 32 + lane;
      if (j < epl && e < E && (sel[j] > best || (sel[j] == best && e < arg))) {
        best = sel[j]; arg = e; best_s = s[j];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
      const float os = __shfl_xor_sync(0xffffffffu, best_s, o);
      if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; best_s = os; }
    }
    if (arg != 0x7fffffff && (arg & 31) == lane) {
#pragma unroll
      for (int j = 0; j < EPL; ++j)
        if (j == (arg >> 5)) sel[j] = -INFINITY;  // static indices keep sel[] in registers
    }
    wsum += best_s;
    if (lane == it) { my_w = best_s; my_id = arg == 0x7fffffff ? 0 : arg; }
  }
  if (lane < k) {
    float w = my_w;
    if (renorm) w = w / fmaxf(wsum, 1e-20f);
    out_ids[static_cast<size_t>(t) * k + lane] = my_id;
    out_w[static_cast<size_t>(t) * k + lane] = w * routed_scale;
  }
}

// ------------------------------------------------------------------ alignment
// counts[e] = number of (token, slot) pairs routed to expert e (ids < 0 or >= E are skipped)
__global__ void moe_count_kernel(const int* __restrict__ ids, int n, int E, int e_lo, int e_hi,
                                 int* __restrict__ counts) {
  pdl_wait();
  pdl_launch_dependents();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int e = ids[i];
  if (e >= e_lo && e < e_hi && e < E) atomicAdd(&counts[e - e_lo], 1);
}

// Single block: exclusive scan of counts into 128-aligned... no padding is inserted: segments are
// contiguous; m-tiles are listed per expert. Writes offsets[E+1], the m-tile list and num_mt,
// and resets cursor[e] = offsets[e].
__global__ void __launch_bounds__(1024)
moe_scan_kernel(const int* __restrict__ counts, int E, int* __restrict__ offsets,
                int* __restrict__ cursor, int* __restrict__ mt_expert, int* __restrict__ mt_row0,
                int* __restrict__ mt_row_end, int* __restrict__ num_mt, int max_mt) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ int s_off[1025];
  __shared__ int s_mt[1025];
  const int tid = threadIdx.x;
  // serial scan by thread 0 is fine for E <= 1024 (a few microseconds)
  if (tid == 0) {
    int o = 0, m = 0;
    for (int e = 0; e < E; ++e) {
      s_off[e] = o;
      s_mt[e] = m;
      o += counts[e];
      m += (counts[e] + 127) / 128;
    }
    s_off[E] = o;
    s_mt[E] = m;
    *num_mt = m < max_mt ? m : max_mt;
  }
  __syncthreads();
  for (int e = tid; e <= E; e += blockDim.x) offsets[e] = s_off[e];
  for (int e = tid; e < E; e += blockDim.x) {
    cursor[e] = s_off[e];
    const int n_t = s_mt[e + 1] - s_mt[e];
    for (int i = 0; i < n_t; ++i) {
      const int mt = s_mt[e] + i;
      if (mt < max_mt) {
        mt_expert[mt] = e;
        mt_row0[mt] = s_off[e] + i * 128;
        mt_row_end[mt] = s_off[e + 1];
      }
    }
  }
}

// pos_of[i] = row of pair i in the permuted matrix (or -1), src_tok[row] = token of that row
__global__ void moe_place_kernel(const int* __restrict__ ids, int n, int k, int E, int e_lo,
                                 int e_hi, int* __restrict__ cursor, int* __restrict__ pos_of,
                                 int* __restrict__ src_tok) {
  pdl_wait();
  pdl_launch_dependents();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int e = ids[i];
  if (e >= e_lo && e < e_hi && e < E) {
    const int p = atomicAdd(&cursor[e - e_lo], 1);
    pos_of[i] = p;
    src_tok[p] = i / k;
  } else {
    pos_of[i] = -1;
  }
}

// All of it in one block, for as many pairs as one SM works off in less time than the other launches take: counts, scan and
// cursors stay in shared memory, and the counters need no zeros. 384 pairs: 2.7 us for 1.4 + 5.2 + 2.0 and a kernel that fills the
// counters; about 0.75 us more per 1024 pairs, so that 38400 take 31 us in place of 21: hence the bound.
constexpr int kAlignPairs = 1 << 13;
__global__ void __launch_bounds__(1024)
moe_align_kernel(const int* __restrict__ ids, int n, int k, int E, int e_lo, int e_hi, int* __restrict__ offsets,
                 int* __restrict__ mt_expert, int* __restrict__ mt_row0, int* __restrict__ mt_row_end, int* __restrict__ num_mt,
                 int max_mt, int* __restrict__ pos_of, int* __restrict__ src_tok) {
  __shared__ int cursor[1024];
  __shared__ int warp_rows[32], warp_tiles[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_local = e_hi - e_lo, e_end = e_hi < E ? e_hi : E;
  cursor[tid] = 0;
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();
#pragma unroll 4
  for (int i = tid; i < n; i += 1024) {
    const int e = ids[i];
    if (e >= e_lo && e < e_end) atomicAdd(&cursor[e - e_lo], 1);
  }
  __syncthreads();
  // thread = local expert: sums of the rows and the m-tiles before it
  const int rows = cursor[tid], tiles = (rows + 127) / 128;
  int r_sum = rows, t_sum = tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, r_sum, o), b = __shfl_up_sync(0xffffffffu, t_sum, o);
    if (lane >= o) r_sum += a, t_sum += b;
  }
  if (lane == 31) warp_rows[warp] = r_sum, warp_tiles[warp] = t_sum;
  __syncthreads();
  for (int w = 0; w < warp; ++w) r_sum += warp_rows[w], t_sum += warp_tiles[w];
  const int row0 = r_sum - rows, tile0 = t_sum - tiles;
  if (tid < n_local) {
    offsets[tid] = row0;
    for (int i = 0; i < tiles && tile0 + i < max_mt; ++i) {
      mt_expert[tile0 + i] = tid;
      mt_row0[tile0 + i] = row0 + i * 128;
      mt_row_end[tile0 + i] = r_sum;
    }
    if (tid == n_local - 1) {
      offsets[n_local] = r_sum;
      *num_mt = t_sum < max_mt ? t_sum : max_mt;
    }
  }
  cursor[tid] = row0;
  __syncthreads();
#pragma unroll 4
  for (int i = tid; i < n; i += 1024) {
    const int e = ids[i];
    int p = -1;
    if (e >= e_lo && e < e_end) {
      p = atomicAdd(&cursor[e - e_lo], 1);
      src_tok[p] = i / k;
    }
    pos_of[i] = p;
  }
}

// x_perm[p, :] = x[src_tok[p], :]   for p < *n_rows. A warp per U x 32 vectors of a row, all in flight: a block per row spends as long
// on starting blocks as on the copy (38400 rows x 2048: 42 us, now 31), a warp for the whole of a wide row is a chain of loads and stores.
// Few rows are bound by latency, many by their bytes (block per row, warp per row, now, us): 8 rows x 7168 2.8, 4.1, 2.1; 384 x 7168
// 3.4, 4.7, 2.9; 1024 x 2048 2.9, 2.6, 2.6; 8192 x 7168 24.4, 28.3, 23.2.
template <int U>
__global__ void __launch_bounds__(256)
moe_gather_kernel(const bf16* __restrict__ x, const int* __restrict__ src_tok,
                   const int* __restrict__ n_rows, bf16* __restrict__ x_perm, int H, int per_row) {
  pdl_wait();
  pdl_launch_dependents();
  const int part = blockIdx.x * 8 + (threadIdx.x >> 5), p = part / per_row;
  const int v0 = part % per_row * (32 * U) + (threadIdx.x & 31), nvec = H >> 3;
  if (p >= *n_rows) return;
  const bf16* src = x + static_cast<size_t>(src_tok[p]) * H;
  bf16* dst = x_perm + static_cast<size_t>(p) * H;
  bf16x8 w[U];
#pragma unroll
  for (int i = 0; i < U; ++i)
    if (v0 + 32 * i < nvec) w[i] = ld_bf16x8(src + (v0 + 32 * i) * 8);
#pragma unroll
  for (int i = 0; i < U; ++i)
    if (v0 + 32 * i < nvec) st_bf16x8(dst + (v0 + 32 * i) * 8, w[i]);
}

// x_perm[pos_of[t, j], :] = weights[t, j] * x[t, :]: rows in expert order whose routing weight is part of the input. One CTA
// per token reads its row once.
template <typename T, int VEC>
__global__ void __launch_bounds__(512) moe_scatter_rows_kernel(const T* __restrict__ x, int64_t ldx, const int* __restrict__ pos_of,
                                                               const float* __restrict__ w, T* __restrict__ x_perm, int k, int H) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ int rows[32];
  __shared__ float factors[32];
  const int64_t t = blockIdx.x;
  if (threadIdx.x < k) rows[threadIdx.x] = pos_of[t * k + threadIdx.x], factors[threadIdx.x] = w[t * k + threadIdx.x];
  __syncthreads();
  for (int c = threadIdx.x * VEC; c < H; c += blockDim.x * VEC) {
    float v[VEC];
    if constexpr (VEC == 8) {
      const bf16x8 b = ld_bf16x8(x + t * ldx + c);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(b.u[j]);
        v[2 * j] = f.x, v[2 * j + 1] = f.y;
      }
    } else {
      if constexpr (sizeof(T) == 4) v[0] = x[t * ldx + c];
      else v[0] = __bfloat162float(x[t * ldx + c]);
    }
    for (int s = 0; s < k; ++s) {
      const int p = rows[s];
      if (p < 0) continue;
      const float f = factors[s];
      T* dst = x_perm + static_cast<int64_t>(p) * H + c;
      if constexpr (VEC == 8) {
        bf16x8 o;
#pragma unroll
        for (int j = 0; j < 4; ++j) o.u[j] = pack_bf16x2(v[2 * j] * f, v[2 * j + 1] * f);
        st_bf16x8(dst, o);
      } else {
        if constexpr (sizeof(T) == 4) *dst = v[0] * f;
        else *dst = __float2bfloat16(v[0] * f);
      }
    }
  }
}

// out[t, :] = (base ? base[t, :] : 0) + sum_j w[t, j] * y_perm[pos_of[t*k + j], :]
// U rows at a time: their places first, then their vectors, then the sums in order. Four are fewer latencies one after the other, one
// leaves room for eight blocks per SM instead of five (one and four, us: 48 tokens x 2048, 8 experts each, 3.8 and 3.1; 512 x 7168, 8
// experts 24.8 and 18.2; 2000 of them 55.3 and 52.4; a single wave of eight blocks, 1024 of them, 30.3 and 32.5; two experts never gain,
// 1024 x 4096 8.4 and 11.1).
template <int U>
__global__ void __launch_bounds__(256)
moe_combine_kernel(const bf16* __restrict__ y_perm, const int* __restrict__ pos_of,
                   const float* __restrict__ w, const bf16* __restrict__ base,
                   bf16* __restrict__ out, int k, int H) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t t = blockIdx.x;
  for (int v = threadIdx.x; v < (H >> 3); v += blockDim.x) {
    float acc[8];
    if (base) {
      const bf16x8 b = ld_bf16x8(base + t * H + v * 8);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(b.u[j]);
        acc[2 * j] = f.x;
        acc[2 * j + 1] = f.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    }
    for (int s0 = 0; s0 < k; s0 += U) {
      int p[U];
      bf16x8 y[U];
#pragma unroll
      for (int i = 0; i < U; ++i) p[i] = s0 + i < k ? pos_of[t * k + s0 + i] : -1;
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (p[i] >= 0) y[i] = ld_bf16x8(y_perm + static_cast<size_t>(p[i]) * H + v * 8);
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (p[i] < 0) continue;
        const float ws = w[t * k + s0 + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(y[i].u[j]);
          acc[2 * j] += ws * f.x;
          acc[2 * j + 1] += ws * f.y;
        }
      }
    }
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) o.u[j] = pack_bf16x2(acc[2 * j], acc[2 * j + 1]);
    st_bf16x8(out + t * H + v * 8, o);
  }
}

inline int check_launch() { return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA; }

}  // namespace

PXL_EXPORT int pxl_moe_route(const void* logits, int64_t ld, int logits_bf16, const float* e_bias, int T, int E,
                             int k, int mode, int renorm, int n_group, int topk_group, int group_top,
                             float routed_scale, int* out_ids, float* out_w, pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (E <= 0 || E > 32 * kMaxEPL || k <= 0 || k > 32 || k > E) return PXL_ERR_INVALID_ARG;
  if (n_group > 32 || (n_group > 1 && E % n_group)) return PXL_ERR_INVALID_ARG;
  const unsigned grid = (T + 3) / 4;
  const int epl = (E + 31) / 32;
#define PXL_ROUTE(B16, EPL)                                                                                        \
  pxl_host::launch(moe_route_kernel<B16, EPL>, grid, 128, 0, stream, logits, ld, e_bias, T, E, k, mode, renorm, n_group, topk_group, \
                                                       group_top, routed_scale, out_ids, out_w)
#define PXL_ROUTE_EPL(B16)          \
  if (epl <= 1) PXL_ROUTE(B16, 1);  \
  else if (epl <= 2) PXL_ROUTE(B16, 2); \
  else if (epl <= 4) PXL_ROUTE(B16, 4); \
  else if (epl <= 8) PXL_ROUTE(B16, 8); \
  else PXL_ROUTE(B16, kMaxEPL)
  if (logits_bf16) {
    PXL_ROUTE_EPL(true);
  } else {
    PXL_ROUTE_EPL(false);
  }
#undef PXL_ROUTE_EPL
#undef PXL_ROUTE
  return check_launch();
}

// Whether pxl_moe_align takes one kernel for this many pairs.
PXL_EXPORT int pxl_moe_align_alone(int T, int k) { return static_cast<int64_t>(T) * k <= kAlignPairs; }

// Build the expert-sorted layout for experts [e_lo, e_hi) (all experts: 0, E).
// ids [T*k]; counts/cursor [n_local]; offsets [n_local+1]; m-tile arrays [max_mt]; pos_of [T*k];
// src_tok [T*k]. Unless pxl_moe_align_alone(T, k), `counts` must be zero on entry.
PXL_EXPORT int pxl_moe_align(const int* ids, int T, int k, int E, int e_lo, int e_hi, int* counts,
                             int* offsets, int* cursor, int* mt_expert, int* mt_row0,
                             int* mt_row_end, int* num_mt, int max_mt, int* pos_of, int* src_tok,
                             pxl_stream_t stream) {
  const int n = T * k;
  const int n_local = e_hi - e_lo;
  if (n <= 0 || n_local <= 0 || n_local > 1024) return PXL_ERR_INVALID_ARG;
  if (pxl_moe_align_alone(T, k)) {
    pxl_host::launch(moe_align_kernel, 1, 1024, 0, stream, ids, n, k, E, e_lo, e_hi, offsets, mt_expert, mt_row0, mt_row_end, num_mt,
                     max_mt, pos_of, src_tok);
    return check_launch();
  }
  const unsigned grid = (n + 255) / 256;
  pxl_host::launch(moe_count_kernel, grid, 256, 0, stream, ids, n, E, e_lo, e_hi, counts);
  pxl_host::launch(moe_scan_kernel, 1, 1024, 0, stream, counts, n_local, offsets, cursor, mt_expert, mt_row0,
                                          mt_row_end, num_mt, max_mt);
  pxl_host::launch(moe_place_kernel, grid, 256, 0, stream, ids, n, k, E, e_lo, e_hi, cursor, pos_of, src_tok);
  return check_launch();
}

PXL_EXPORT int pxl_moe_gather(const void* x, const int* src_tok, const int* n_rows, void* x_perm,
                              int max_rows, int H, pxl_stream_t stream) {
  if (max_rows <= 0) return PXL_OK;
  if (H % 8) return PXL_ERR_INVALID_ARG;
  const int nvec = H >> 3;
  auto go = [&](auto kern, int u) {
    const int per_row = pxl::ceil_div(nvec, 32 * u);
    pxl_host::launch(kern, pxl::ceil_div(max_rows * per_row, 8), 256, 0, stream, static_cast<const bf16*>(x), src_tok, n_rows,
                     static_cast<bf16*>(x_perm), H, per_row);
  };
  // four vectors per lane once they give the SMs a few warps each (2400 parts of four: 2.93 us with two, 3.07; 7168: 5.53 and 4.83)
  if (static_cast<int64_t>(max_rows) * pxl::ceil_div(nvec, 128) >= 4096) go(moe_gather_kernel<4>, 4);
  else go(moe_gather_kernel<2>, 2);
  return check_launch();
}

PXL_EXPORT int pxl_moe_scatter_rows(const void* x, int64_t ldx, const int* pos_of, const float* w, void* x_perm, int T, int k,
                                    int H, int is_f32, pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (k <= 0 || k > 32 || H <= 0) return PXL_ERR_INVALID_ARG;
  const int threads = H >= 4096 ? 512 : H >= 2048 ? 256 : 128;
  const bool vec = !is_f32 && !((ldx | H) & 7) && !((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(x_perm)) & 15);
  if (is_f32)
    pxl_host::launch(moe_scatter_rows_kernel<float, 1>, T, threads, 0, stream, static_cast<const float*>(x), ldx, pos_of, w,
                                                             static_cast<float*>(x_perm), k, H);
  else if (vec)
    pxl_host::launch(moe_scatter_rows_kernel<bf16, 8>, T, threads, 0, stream, static_cast<const bf16*>(x), ldx, pos_of, w,
                                                            static_cast<bf16*>(x_perm), k, H);
  else
    pxl_host::launch(moe_scatter_rows_kernel<bf16, 1>, T, threads, 0, stream, static_cast<const bf16*>(x), ldx, pos_of, w,
                                                            static_cast<bf16*>(x_perm), k, H);
  return check_launch();
}

PXL_EXPORT int pxl_moe_combine(const void* y_perm, const int* pos_of, const float* w,
                               const void* base, void* out, int T, int k, int H,
                               pxl_stream_t stream) {
  if (T <= 0) return PXL_OK;
  if (H % 8) return PXL_ERR_INVALID_ARG;
  auto go = [&](auto kern) {
    pxl_host::launch(kern, T, 256, 0, stream, static_cast<const bf16*>(y_perm), pos_of, w, static_cast<const bf16*>(base),
                     static_cast<bf16*>(out), k, H);
  };
  const int sms = pxl_host::num_sms();
  if (k <= 2 || (T > 5 * sms && T <= 8 * sms)) go(moe_combine_kernel<1>);  // (one wave of eight blocks per SM, more than one of five)
  else go(moe_combine_kernel<4>);
  return check_launch();
}
