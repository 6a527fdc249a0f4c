// C[m, n] = sum_k A[m, k] W[n, k] for a handful of rows (one to a few requests decoding), bf16 with fp32 sums.
//
// Every weight is read once and used M times: bound by memory, so nothing of a tensor-core product helps and its costs remain
// (tiles of 128 rows for M = 1, partial sums exchanged between the K ranges, TMA and TMEM set up per launch). Here a warp takes
// R rows of W over the whole of K, 16 bytes a lane and eight to twelve such loads in flight, and the sums of its lanes meet in one
// transposing shuffle reduction. The rows of A are shared by all warps and come from L1. Weights are not written by the kernel
// before, so the first loads go out ahead of the wait for it (programmatic dependent launch): in a chain of small layers they
// run under its tail.
#include "common.cuh"
#include "pxl_api.h"

namespace {
using namespace pxl;

constexpr int kWarps = 4, kHeadWarps = 8;
constexpr int kEpiHeads = 1000;  // a head's norm, rotation and place in the cache behind its product (HeadArgs)
constexpr int kHeadDim = 128, kHeadCtas = kHeadDim / 2 / kHeadWarps;

struct GemvArgs {
  const bf16 *A, *W, *residual, *bias;
  void* C;
  int M, N, K, lda, ldw, ldc;
  const bf16* norm_w;  // NORM: [K]; rows of A times norm_w + norm_offset over their root mean square, rounded to bf16
  float norm_eps, norm_offset;
};

// The query, key and value heads of a layer, all of 128 columns and rotated over the whole of them: the product's columns i and i + 64
// of a head are one warp's, so the rotation stays in it, and the eight CTAs of a head, a cluster, pass the warps' sums of squares round.
struct HeadArgs : GemvArgs {  // C: [M, N], the query heads' columns are written; keys and values go to the cache
  const bf16 *q_norm, *k_norm;  // [128] or null
  const float* cos_sin;         // [positions][128]
  const int* positions;
  const int64_t* slots;  // or null: no cache
  bf16 *k_cache, *v_cache;
  int Hq, Hkv, page_size, max_pos;
  int64_t num_slots;
  int* status;
};

__device__ __forceinline__ uint64_t widen(uint32_t two) {  // two bf16 -> two fp32 in a register pair
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(two << 16), "r"(two & 0xffff0000u));
  return v;
}

// MM rows of A (the last ones repeated where M is smaller), R rows of W per warp, U steps of 256 columns in flight.
// ONE: K fits one round of U steps, and the rows are held in registers.
// EPI: PXL_EPI_NONE, _RESIDUAL, _F32 or _SILU_MUL (R rows = R / 2 gate / up pairs, 64 rows apart in groups of 128)
template <int MM, int R, int U, int EPI, bool NORM, bool ONE, typename Args>
__device__ __forceinline__ void gemv_body(const Args& a) {
  constexpr bool kGlu = EPI == PXL_EPI_SILU_MUL, kHeads = EPI == kEpiHeads;
  const int lane = threadIdx.x & 31, wid = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int head = blockIdx.x / kHeadCtas, in_head = blockIdx.x % kHeadCtas * kHeadWarps + (threadIdx.x >> 5);  // kHeads
  const int n0 = kHeads ? head * kHeadDim + in_head : wid * R;  // first row of W; pairs: 2 x first output column
  if (n0 >= a.N) return;
  int row[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int c = n0 / 2 + r / 2;
    row[r] = kHeads ? n0 + r * (kHeadDim / 2) : kGlu ? c / 64 * 128 + c % 64 + (r & 1) * 64 : n0 + r;
  }
  uint4 w[U][R];
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * 256 + lane * 8;
#pragma unroll
      for (int r = 0; r < R; ++r)
        w[u][r] = k < a.K ? __ldcs(reinterpret_cast<const uint4*>(a.W + static_cast<int64_t>(row[r]) * a.ldw + k)) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  load(0);
  // What no kernel of the chain writes goes out ahead of the wait, what the kernel before wrote right behind it and all at once: in a
  // chain of small layers the products are a handful of load latencies one after the other. (The norm's weights only where K is
  // one round; for the first of several they would take registers from all.)
  constexpr bool kNormHeld = NORM && ONE;
  uint4 nw[kNormHeld ? U : 1];
  if constexpr (kNormHeld) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = u * 256 + lane * 8;
      nw[u] = k < a.K ? *reinterpret_cast<const uint4*>(a.norm_w + k) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  constexpr int V = MM * R, kSpan = 32 / V;  // number i of the results ends in lanes [i * kSpan, (i + 1) * kSpan)
  const int oi = lane / kSpan, om = oi / R, orow = oi % R;
  const bool stores = lane % kSpan == 0 && om < a.M && !(kGlu && (orow & 1));
  const int col = kHeads ? n0 + orow * (kHeadDim / 2) : kGlu ? (n0 + orow) / 2 : n0 + orow;
  const int64_t at = static_cast<int64_t>(om) * a.ldc + col;
  float add_bias = 0.f, add_res = 0.f;
  constexpr bool kEarly = V <= 8;  // (registers)
  if (kEarly && !kGlu && stores && a.bias) add_bias = __bfloat162float(a.bias[col]);
  [[maybe_unused]] float head_w = 0.f, cs = 1.f, sn = 0.f;
  [[maybe_unused]] int64_t slot = -1;
  [[maybe_unused]] bool head_normed = false, turned = false;
  if constexpr (kHeads) {
    const bf16* w = head < a.Hq ? a.q_norm : head < a.Hq + a.Hkv ? a.k_norm : nullptr;
    head_normed = w != nullptr;
    // the other CTAs' shared memory is written to later on: they have to have begun
    if (head_normed) cluster_arrive_all();
    if (head_normed) head_w = __bfloat162float(w[col - head * kHeadDim]) + a.norm_offset;
    const int m = om < a.M ? om : a.M - 1, p = a.positions[m];
    const bool p_ok = p >= 0 && (a.max_pos <= 0 || p < a.max_pos);
    slot = a.slots ? a.slots[m] : -1;
    turned = p_ok && head < a.Hq + a.Hkv;  // a position outside the table is reported, its row is left unrotated
    if (turned) {
      cs = a.cos_sin[static_cast<int64_t>(p) * kHeadDim + in_head];
      sn = a.cos_sin[static_cast<int64_t>(p) * kHeadDim + kHeadDim / 2 + in_head];
    }
    if (blockIdx.x == 0 && threadIdx.x < 32 && stores && orow == 0 && a.status) {
      if (slot >= a.num_slots) atomicCAS(a.status, 0, PXL_DEV_BAD_SLOT);
      if (!p_ok) atomicCAS(a.status, 0, PXL_DEV_BAD_POSITION);
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  const bf16* rows_a[MM];
#pragma unroll
  for (int m = 0; m < MM; ++m) rows_a[m] = a.A + static_cast<int64_t>(m < a.M ? m : a.M - 1) * a.lda;
  constexpr bool kHeld = ONE && MM == 1;  // (more rows would not fit the registers)
  uint4 held[kHeld ? U : 1];
  if constexpr (kHeld) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = u * 256 + lane * 8;
      held[u] = k < a.K ? *reinterpret_cast<const uint4*>(rows_a[0] + k) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if constexpr (EPI == PXL_EPI_RESIDUAL && kEarly) {
    if (stores) add_res = __bfloat162float(a.residual[at]);
  }
  float inv[MM];
  if constexpr (NORM) {
#pragma unroll
    for (int m = 0; m < MM; ++m) {
      float ss = 0.f;
      auto squares = [&](const uint4 v) {  // (by value: from a reference into memory four words come one by one, 7168 x 5120 19.7 us for 16.4)
        const uint32_t* p = &v.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(p[j]);
          ss += f.x * f.x + f.y * f.y;
        }
      };
      int k = lane * 8;
      if constexpr (kHeld) {
#pragma unroll
        for (int u = 0; u < U; ++u) squares(held[u]);
        k += U * 256;
      }
      for (; k < a.K; k += 256) squares(*reinterpret_cast<const uint4*>(rows_a[m] + k));
      inv[m] = rsqrtf(warp_reduce_sum(ss) / static_cast<float>(a.K) + a.norm_eps);
    }
  }
  uint64_t acc[MM][R] = {};
  for (int k0 = 0; k0 < a.K; k0 += U * 256) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * 256 + lane * 8;
      if (k >= a.K) break;
      uint64_t wv[R][4];
#pragma unroll
      for (int r = 0; r < R; ++r)
        wv[r][0] = widen(w[u][r].x), wv[r][1] = widen(w[u][r].y), wv[r][2] = widen(w[u][r].z), wv[r][3] = widen(w[u][r].w);
#pragma unroll
      for (int m = 0; m < MM; ++m) {
        uint4 xr = kHeld && k0 == 0 ? held[kHeld ? u : 0] : *reinterpret_cast<const uint4*>(rows_a[m] + k);
        if constexpr (NORM) {
          const uint4 nv = kNormHeld ? nw[kNormHeld ? u : 0] : *reinterpret_cast<const uint4*>(a.norm_w + k);
          const uint32_t* nx = &nv.x;
          uint32_t* xw = &xr.x;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(xw[j]), g = unpack_bf16x2(nx[j]);
            xw[j] = pack_bf16x2(f.x * inv[m] * (g.x + a.norm_offset), f.y * inv[m] * (g.y + a.norm_offset));
          }
        }
        const uint64_t x[4] = {widen(xr.x), widen(xr.y), widen(xr.z), widen(xr.w)};
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[m][r] = fma2(wv[r][j], x[j], acc[m][r]);
      }
    }
    if (ONE) break;
    if (k0 + U * 256 < a.K) load(k0 + U * 256);
  }
  // sums over the lanes: every exchange halves the numbers a lane holds, lanes V = MM * R apart end with the same one
  float v[V];
#pragma unroll
  for (int m = 0; m < MM; ++m)
#pragma unroll
    for (int r = 0; r < R; ++r) v[m * R + r] = __uint_as_float(static_cast<uint32_t>(acc[m][r])) + __uint_as_float(static_cast<uint32_t>(acc[m][r] >> 32));
  int o = 16;
#pragma unroll
  for (int n = V; n > 1; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float give = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  float sum = v[0];
  if constexpr (kGlu) {  // the up product sits kSpan lanes further
    const float up = __shfl_down_sync(0xffffffffu, sum, kSpan);
    sum = sum / (1.f + __expf(-sum)) * up;
  }
  if constexpr (kHeads) {
    __shared__ float squares[MM][kHeadDim / 2];  // of columns i and i + 64 of the head
    float x = __bfloat162float(__float2bfloat16(sum + __shfl_sync(0xffffffffu, add_bias, lane / kSpan * kSpan)));
    float other = __shfl_xor_sync(0xffffffffu, x, kSpan);
    if (head_normed) {  // the same in all CTAs of the cluster
      cluster_wait_all();
      if (orow == 0 && lane % kSpan < kHeadCtas)
        st_shared_cluster_f32(cluster_map_shared(smem_u32(&squares[om][in_head]), lane % kSpan), x * x + other * other);
      cluster_sync_all();
      float total = 0.f;
#pragma unroll
      for (int m = 0; m < MM; ++m) {
        const float t = warp_reduce_sum(squares[m][lane] + squares[m][lane + 32]);
        if (m == om) total = t;
      }
      const float inv_rms = rsqrtf(total / static_cast<float>(kHeadDim) + a.norm_eps);
      x = __bfloat162float(__float2bfloat16(x * inv_rms * head_w));  // rounded before the rotation, as a bf16 module does
      other = __shfl_xor_sync(0xffffffffu, x, kSpan);
    }
    // (a branch: cosine 1 and sine 0 would make NaN of what has an infinity or a NaN for its other half)
    const bf16 y = __float2bfloat16(turned ? x * cs + (orow == 0 ? -other : other) * sn : x);
    if (!stores) return;
    if (head < a.Hq) {
      static_cast<bf16*>(a.C)[at] = y;
    } else if (slot >= 0 && slot < a.num_slots) {
      const bool is_k = head < a.Hq + a.Hkv;
      const int kvh = head - a.Hq - (is_k ? 0 : a.Hkv);
      const int64_t line = (slot / a.page_size * a.Hkv + kvh) * a.page_size + slot % a.page_size;
      (is_k ? a.k_cache : a.v_cache)[line * kHeadDim + in_head + orow * (kHeadDim / 2)] = y;
    }
    return;
  }
  if (!stores) return;
  if constexpr (!kEarly) {
    if (!kGlu && a.bias) add_bias = __bfloat162float(a.bias[col]);
    if constexpr (EPI == PXL_EPI_RESIDUAL) add_res = __bfloat162float(a.residual[at]);
  }
  sum += add_bias;
  if constexpr (EPI == PXL_EPI_F32) {
    static_cast<float*>(a.C)[at] = sum;
  } else {
    if constexpr (EPI == PXL_EPI_RESIDUAL) sum += add_res;
    static_cast<bf16*>(a.C)[at] = __float2bfloat16(sum);
  }
}

template <int MM, int R, int U, int EPI, bool NORM, bool ONE>
__global__ void __launch_bounds__(kWarps * 32) gemv_kernel(const GemvArgs a) {
  gemv_body<MM, R, U, EPI, NORM, ONE>(a);
}
template <int MM, bool ONE>
__global__ void __cluster_dims__(kHeadCtas, 1, 1) __launch_bounds__(kHeadWarps * 32, 2) gemv_heads_kernel(const HeadArgs a) {
  gemv_body<MM, 2, 4, kEpiHeads, true, ONE>(a);
}

template <int MM, int R, int U, bool ONE>
int launch_one(const GemvArgs& a, int epi, cudaStream_t stream) {
  const dim3 grid(ceil_div(ceil_div(a.N, R), kWarps)), block(kWarps * 32);
  auto go = [&](auto kern) {
    pxl_host::launch(kern, grid, block, 0, stream, a);
    return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
  };
  if (a.norm_w) {
    if constexpr (MM <= PXL_GEMV_NORM_MAX_M) {
      if (epi == PXL_EPI_NONE) return go(gemv_kernel<MM, R, U, PXL_EPI_NONE, true, ONE>);
      if constexpr (R > 1)
        if (epi == PXL_EPI_SILU_MUL) return go(gemv_kernel<MM, R, U, PXL_EPI_SILU_MUL, true, ONE>);
    }
    return PXL_ERR_INVALID_ARG;
  }
  switch (epi) {
    case PXL_EPI_NONE: return go(gemv_kernel<MM, R, U, PXL_EPI_NONE, false, ONE>);
    case PXL_EPI_RESIDUAL: return go(gemv_kernel<MM, R, U, PXL_EPI_RESIDUAL, false, ONE>);
    case PXL_EPI_F32: return go(gemv_kernel<MM, R, U, PXL_EPI_F32, false, ONE>);
    case PXL_EPI_SILU_MUL:
      if constexpr (R > 1) return go(gemv_kernel<MM, R, U, PXL_EPI_SILU_MUL, false, ONE>);
    default: return PXL_ERR_INVALID_ARG;
  }
}

template <int MM, int R, int U>
int launch_epi(const GemvArgs& a, int epi, cudaStream_t stream) {
  return MM == 1 && a.K <= U * 256 ? launch_one<MM, R, U, MM == 1>(a, epi, stream) : launch_one<MM, R, U, false>(a, epi, stream);
}

template <int MM>
int launch_rows(const GemvArgs& a, int epi, cudaStream_t stream) {
  // rows of W per warp: as many as still give every SM a dozen warps
  const int want = 12 * pxl_host::num_sms();
  // (two rows with a norm, whose squares every warp adds up for itself: four rows of W from fewer warps on; 6144 x 4096 20.6 us with two, 15.9)
  if (a.N >= 4 * want || (MM == 2 && a.norm_w && a.N >= 3 * want)) return launch_epi<MM, 4, 2>(a, epi, stream);
  if (a.N >= 2 * want || epi == PXL_EPI_SILU_MUL) return launch_epi<MM, 2, 4>(a, epi, stream);
  // one row of W: the whole of it in flight up to K = 3072 (1024 x 2304 3.8 us in rounds of eight, 2.2 in one of twelve; 2048 x 3072 5.4 and
  // 4.1; longer rows take two rounds either way, 1024 x 3584 4.9 and 5.1, and sixteen steps beside the norm's weights spill)
  if (MM == 1 && a.K > 2048 && a.K <= 3072) return launch_epi<MM, 1, 12>(a, epi, stream);
  return launch_epi<MM, 1, 8>(a, epi, stream);
}

int run(const GemvArgs& a, int epi, cudaStream_t stream) {
  if (!pxl_gemv_bf16_takes(a.M, a.N, a.K, epi) || ((a.lda | a.ldw) & 7) ||
      ((reinterpret_cast<uintptr_t>(a.A) | reinterpret_cast<uintptr_t>(a.W) | reinterpret_cast<uintptr_t>(a.norm_w)) & 15))
    return PXL_ERR_INVALID_ARG;
  if (epi == PXL_EPI_RESIDUAL && a.residual == nullptr) return PXL_ERR_INVALID_ARG;
  if (a.M == 1) return launch_rows<1>(a, epi, stream);
  if (a.M == 2) return launch_rows<2>(a, epi, stream);
  return launch_rows<4>(a, epi, stream);
}
}  // namespace

// Where it beats the tensor cores: the rows of A cost it a load and an unpacking each per 16 bytes of W, so it is ahead for one
// row (4096 x 4096: 9.0 us against 10.7; 151936 x 1024: 46 against 55) and stays so up to four where K is short (4096 x 1024, four
// rows: 4.4 against 7.2) but not where the split along K of the other kernel pays (6144 x 4096, four rows: 17.3 against 12.3).
// Gated products have no such split: four rows at 24576 x 4096 take 39 us, six on the tensor cores 40.
PXL_EXPORT int pxl_gemv_bf16_takes(int M, int N, int K, int epi) {
  if (M <= 0 || M > PXL_GEMV_MAX_M || N % 8 || K % 8) return 0;
  if (epi == PXL_EPI_SILU_MUL) return N % 128 == 0;
  return (epi == PXL_EPI_NONE || epi == PXL_EPI_RESIDUAL || epi == PXL_EPI_F32) && M * K <= 14336;
}

// contract of pxl_gemm_bf16, for the sizes that pxl_gemv_bf16_takes() names
PXL_EXPORT int pxl_gemv_bf16(const void* A, const void* W, void* C, const void* residual, const void* bias, int M, int N, int K,
                             int lda, int ldw, int ldc, int epi, cudaStream_t stream) {
  return run(GemvArgs{static_cast<const pxl::bf16*>(A), static_cast<const pxl::bf16*>(W), static_cast<const pxl::bf16*>(residual),
                      static_cast<const pxl::bf16*>(bias), C, M, N, K, lda, ldw, ldc, nullptr, 0.f, 0.f},
             epi, stream);
}

PXL_EXPORT int pxl_gemv_bf16_norm(const void* A, const void* norm_w, float eps, float offset, const void* W, void* C, const void* bias,
                                  int M, int N, int K, int lda, int ldw, int ldc, int epi, cudaStream_t stream) {
  if (norm_w == nullptr || M > PXL_GEMV_NORM_MAX_M) return PXL_ERR_INVALID_ARG;
  return run(GemvArgs{static_cast<const pxl::bf16*>(A), static_cast<const pxl::bf16*>(W), nullptr, static_cast<const pxl::bf16*>(bias),
                      C, M, N, K, lda, ldw, ldc, static_cast<const pxl::bf16*>(norm_w), eps, offset},
             epi, stream);
}

// One launch for the norm, the product of the q, k and v heads and pxl_qk_norm_rope_cache behind it. The launches are what a layer of one
// row costs: six of them take the host 3.9 us each, longer than the chip needs; behind the product the rotation is 1 us of a cluster's
// barrier, where its own kernel takes 2.9.
PXL_EXPORT int pxl_gemv_bf16_qkv_takes(int M, int K, int Hq, int Hkv, int D, int rot_dim) {
  return M <= PXL_GEMV_NORM_MAX_M && D == kHeadDim && rot_dim == kHeadDim && Hq > 0 && Hkv > 0 &&
         pxl_gemv_bf16_takes(M, (Hq + 2 * Hkv) * D, K, PXL_EPI_NONE);
}

// Where that is faster than the product and the rotation apart: with a wave of clusters (of the 37 that two blocks per SM are, the GPCs
// take 32 to 36), and one row only if they are on every SM. Layers of one row, us, together and apart: 16 + 2 x 8 heads, 1024 wide 18.2
// and 18.5, 4096 wide 49.6 and 58.6; 32 + 2 x 8 heads, 4096 wide 98 and 96; 64 + 2 x 8, 5120 wide 198 and 181; 32 + 2 x 4, 2048 wide 34.0
// and 31.7; 8 + 2 x 2, 2048 wide 29.9 and 28.3 (two rows 35.1 and 36.4).
PXL_EXPORT int pxl_gemv_bf16_qkv_pays(int M, int Hq, int Hkv) {
  const int ctas = (Hq + 2 * Hkv) * kHeadCtas, sms = pxl_host::num_sms();
  return ctas * 8 <= 2 * sms * 7 && (M > 1 || ctas >= sms);
}

PXL_EXPORT int pxl_gemv_bf16_qkv(const void* A, const void* norm_w, float eps, float offset, const void* W, const void* bias, void* qkv,
                                 const void* q_norm_w, const void* k_norm_w, const float* cos_sin, const int* positions,
                                 const int64_t* slot_mapping, void* k_cache, void* v_cache, int M, int K, int Hq, int Hkv, int D,
                                 int rot_dim, int page_size, int64_t num_slots, int max_pos, int* status, cudaStream_t stream) {
  using pxl::bf16;
  if (!pxl_gemv_bf16_qkv_takes(M, K, Hq, Hkv, D, rot_dim) || norm_w == nullptr || page_size <= 0 ||
      ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(norm_w)) & 15))
    return PXL_ERR_INVALID_ARG;
  HeadArgs a{};
  a.A = static_cast<const bf16*>(A), a.W = static_cast<const bf16*>(W), a.bias = static_cast<const bf16*>(bias), a.C = qkv;
  a.M = M, a.N = (Hq + 2 * Hkv) * D, a.K = a.lda = a.ldw = K, a.ldc = a.N;
  a.norm_w = static_cast<const bf16*>(norm_w), a.norm_eps = eps, a.norm_offset = offset;
  a.q_norm = static_cast<const bf16*>(q_norm_w), a.k_norm = static_cast<const bf16*>(k_norm_w);
  a.cos_sin = cos_sin, a.positions = positions, a.slots = slot_mapping;
  a.k_cache = static_cast<bf16*>(k_cache), a.v_cache = static_cast<bf16*>(v_cache);
  a.Hq = Hq, a.Hkv = Hkv, a.page_size = page_size, a.max_pos = max_pos, a.num_slots = num_slots, a.status = status;
  const dim3 grid((Hq + 2 * Hkv) * kHeadCtas), block(kHeadWarps * 32);
  auto go = [&](auto kern) {
    pxl_host::launch(kern, grid, block, 0, stream, a);
    return cudaGetLastError() == cudaSuccess ? PXL_OK : PXL_ERR_CUDA;
  };
  if (M == 1) return K <= 1024 ? go(gemv_heads_kernel<1, true>) : go(gemv_heads_kernel<1, false>);
  return go(gemv_heads_kernel<2, false>);
}
