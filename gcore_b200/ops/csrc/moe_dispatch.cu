// Token movement around the grouped expert GEMMs of a mixture-of-experts layer on one GPU, forward and backward:
//   * moe_count / moe_place   from the chosen experts to every choice's row in the expert-sorted buffer, whose segments are
//                             padded to 128 rows; rows of one expert keep the order of the tokens (a counting sort: two
//                             launches instead of a radix sort and a dozen index operations);
//   * moe_gather              rows of the buffer, padding rows zeroed in the same pass (the weight gradient contracts over
//                             them);
//   * moe_combine             y[t] = sum_k w[t, k] rows[dest[t, k]]; without weights the gather's backward;
//   * moe_combine_bwd         d(rows) = w d(y), zero in padding rows, and d(w) = <d(y), rows>, one pass.
// Roundings to bf16 are where the layer has them as tensor operations, so that a training run keeps its numbers: of the
// weights and of every product, and of the gather's backward after every addition; sums of products run in 32 bits.
// All are bound by the bytes of the rows they move.  A layer of 128 experts, 2048 wide, top 8, with index operations -> with
// these kernels, us, forward / forward and backward: 600 tokens 909 / 4529 -> 654 / 2159, 4400 tokens 1704 / 6426 -> 901 /
// 2957, 8000 tokens 2406 / 8169 -> 1296 / 3877 (of the backward's gain 2.0 ms are the weight gradients' TMA reductions).
// And the logits of a decode step's router in 32 bits (router_logits).
#include "host_utils.h"
#include "row_ops.cuh"

namespace gkmp {
using namespace gk;

constexpr int CHUNK = 2048, THREADS = 256, WARPS = THREADS / 32, MAX_E = 512;

__global__ void __launch_bounds__(THREADS) moe_count_kernel(const long long* __restrict__ idx, int n, int E,
                                                            int* __restrict__ part) {
  __shared__ int hist[MAX_E];
  for (int e = threadIdx.x; e < E; e += THREADS) hist[e] = 0;
  __syncthreads();
  const int n0 = blockIdx.x * CHUNK, n1 = n0 + CHUNK < n ? n0 + CHUNK : n;
  for (int i = n0 + threadIdx.x; i < n1; i += THREADS) {
    const long long e = idx[i];
    if (e >= 0 && e < E) atomicAdd(&hist[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += THREADS) part[blockIdx.x * E + e] = hist[e];
}

// A CTA places the choices of its chunk, a warp 256 of them in order.  part: counts of every chunk (null: one chunk).
__global__ void __launch_bounds__(THREADS) moe_place_kernel(const long long* __restrict__ idx, int n, int E, int seg,
                                                            const int* __restrict__ part, int* __restrict__ dest,
                                                            int* __restrict__ src, int* __restrict__ offsets) {
  __shared__ int next[WARPS][MAX_E];   // rows of an expert that a warp's next choice of it comes behind
  __shared__ int total[MAX_E], off[MAX_E + 1], s_warp[WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < WARPS * MAX_E; i += THREADS) (&next[0][0])[i] = 0;
  __syncthreads();
  const int w0 = blockIdx.x * CHUNK + warp * (CHUNK / WARPS);
  int mine[CHUNK / THREADS];
#pragma unroll
  for (int j = 0; j < CHUNK / THREADS; ++j) {
    const int i = w0 + j * 32 + lane;
    const long long e = i < n ? idx[i] : -1;
    mine[j] = e >= 0 && e < E ? static_cast<int>(e) : -1;
    if (mine[j] >= 0) atomicAdd(&next[warp][mine[j]], 1);
  }
  __syncthreads();
  for (int e = tid; e < E; e += THREADS) {
    int before = 0, all = 0;
    if (part) {
      for (int c = 0; c < static_cast<int>(gridDim.x); ++c) {
        const int v = part[c * E + e];
        if (c < static_cast<int>(blockIdx.x)) before += v;
        all += v;
      }
    }
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const int v = next[w][e];
      next[w][e] = before;
      before += v;
    }
    total[e] = part ? all : before;
  }
  __syncthreads();
  // exclusive prefix sums of the padded counts: two experts per thread
  const int e0 = 2 * tid;
  const int a = e0 < E ? (total[e0] + seg - 1) / seg * seg : 0, b = e0 + 1 < E ? (total[e0 + 1] + seg - 1) / seg * seg : 0;
  int incl = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffff, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int before = incl - a - b;
  for (int w = 0; w < warp; ++w) before += s_warp[w];
  if (e0 == 0) off[0] = 0;
  if (e0 < E) off[e0 + 1] = before + a;
  if (e0 + 1 < E) off[e0 + 2] = before + a + b;
  __syncthreads();
  if (blockIdx.x == 0)
    for (int e = tid; e <= E; e += THREADS) offsets[e] = off[e];
#pragma unroll
  for (int j = 0; j < CHUNK / THREADS; ++j) {
    const int i = w0 + j * 32 + lane, e = mine[j];
    const unsigned same = __match_any_sync(0xffffffffu, e);
    if (e >= 0) {
      const int r = off[e] + next[warp][e] + __popc(same & ((1u << lane) - 1));
      dest[i] = r;
      src[r] = i;
    }
    __syncwarp();
    if (e >= 0 && (same >> lane) == 1u) next[warp][e] += __popc(same);   // the last lane of those with this expert
    __syncwarp();
  }
  for (int e = blockIdx.x; e < E; e += gridDim.x)
    for (int r = off[e] + total[e] + tid; r < off[e + 1]; r += THREADS) src[r] = -1;
}

// one warp per row
__global__ void __launch_bounds__(THREADS) moe_gather_kernel(const uint4* __restrict__ x, const int* __restrict__ src,
                                                             const int* __restrict__ n_rows, uint4* __restrict__ out, int K,
                                                             int vecs) {
  const int lane = threadIdx.x & 31, rows = *n_rows;
  for (int r = blockIdx.x * WARPS + (threadIdx.x >> 5); r < rows; r += gridDim.x * WARPS) {
    const int s = src[r];
    const uint4* from = x + static_cast<long long>(s < 0 ? 0 : s / K) * vecs;
    uint4* to = out + static_cast<long long>(r) * vecs;
#pragma unroll 4
    for (int c = lane; c < vecs; c += 32) to[c] = s < 0 ? make_uint4(0, 0, 0, 0) : from[c];
  }
}

struct alignas(16) bf16x8 { __nv_bfloat162 v[4]; };
__device__ __forceinline__ void unpack8(const uint4& r, float (&f)[8]) {
  const bf16x8& a = reinterpret_cast<const bf16x8&>(r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(a.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  bf16x8 a;
#pragma unroll
  for (int i = 0; i < 4; ++i) a.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return reinterpret_cast<const uint4&>(a);
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16(v)); }

// grid (column groups of blockDim.x 8-element units, tokens in turn)
template <bool WEIGHTS>
__global__ void __launch_bounds__(THREADS) moe_combine_kernel(const uint4* __restrict__ rows, const float* __restrict__ w,
                                                              const int* __restrict__ dest, uint4* __restrict__ y, int T,
                                                              int K, int vecs) {
  pdl_launch_dependents();
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= vecs) return;
  for (int t = blockIdx.y; t < T; t += gridDim.y) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      float f[8];
      unpack8(rows[static_cast<long long>(dest[t * K + k]) * vecs + c], f);
      const float wk = WEIGHTS ? round_bf16(w[t * K + k]) : 1.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = WEIGHTS ? acc[j] + round_bf16(wk * f[j]) : round_bf16(acc[j] + f[j]);
    }
    y[static_cast<long long>(t) * vecs + c] = pack8(acc);
  }
}

// one warp per row of the expert-sorted buffer
__global__ void __launch_bounds__(THREADS) moe_combine_bwd_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ rows,
                                                                  const float* __restrict__ w, const int* __restrict__ src,
                                                                  const int* __restrict__ n_rows, uint4* __restrict__ drows,
                                                                  float* __restrict__ dw, int K, int vecs) {
  const int lane = threadIdx.x & 31, total = *n_rows;
  for (int r = blockIdx.x * WARPS + (threadIdx.x >> 5); r < total; r += gridDim.x * WARPS) {
    const int s = src[r];
    uint4* to = drows + static_cast<long long>(r) * vecs;
    if (s < 0) {
      for (int c = lane; c < vecs; c += 32) to[c] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const uint4* g = dy + static_cast<long long>(s / K) * vecs;
    const uint4* v = rows + static_cast<long long>(r) * vecs;
    const float wk = round_bf16(w[s]);   // what the forward pass multiplied with
    float dot = 0.f;
#pragma unroll 4
    for (int c = lane; c < vecs; c += 32) {
      float a[8], b[8];
      unpack8(g[c], a);
      unpack8(v[c], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        dot += round_bf16(a[j] * b[j]);
        a[j] *= wk;
      }
      to[c] = pack8(a);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) dw[s] = round_bf16(dot);
  }
}

// logits[t, e] = h[t] . w[e] in 32 bits, a warp per expert and 16 tokens at a time (their rows wait in shared memory); also
// clears the experts' counters for the routing kernel that follows.  The library's 32-bit product took 10.5 us for 16 tokens,
// 2048 wide, 128 experts, beside a conversion of the tokens.
constexpr int RL_TOKENS = 16, RL_WARPS = 4;
__global__ void __launch_bounds__(RL_WARPS * 32) router_logits_kernel(const __nv_bfloat16* __restrict__ h,
                                                                      const float* __restrict__ w, float* __restrict__ logits,
                                                                      int* __restrict__ counts, int T, int E, int H) {
  extern __shared__ __align__(16) uint8_t rl_smem[];
  uint4* s_h = reinterpret_cast<uint4*>(rl_smem);   // [tokens][H]
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, e = blockIdx.x * RL_WARPS + (tid >> 5), vecs = H >> 3;
  const int t0 = blockIdx.y * RL_TOKENS, n = T - t0 < RL_TOKENS ? T - t0 : RL_TOKENS;
  if (counts && blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = tid; i < E; i += RL_WARPS * 32) counts[i] = 0;
  const uint4* from = reinterpret_cast<const uint4*>(h + static_cast<long long>(t0) * H);
#pragma unroll 4
  for (int i = tid; i < RL_TOKENS * vecs; i += RL_WARPS * 32) s_h[i] = i < n * vecs ? from[i] : make_uint4(0, 0, 0, 0);
  __syncthreads();
  if (e >= E) return;
  float acc[RL_TOKENS];
#pragma unroll
  for (int t = 0; t < RL_TOKENS; ++t) acc[t] = 0.f;
  const float4* wr = reinterpret_cast<const float4*>(w + static_cast<long long>(e) * H);
#pragma unroll 2
  for (int c = lane; c < vecs; c += 32) {
    const float4 a = __ldg(wr + 2 * c), b = __ldg(wr + 2 * c + 1);
#pragma unroll
    for (int t = 0; t < RL_TOKENS; ++t) {
      float f[8];
      unpack8(s_h[t * vecs + c], f);
      acc[t] = fmaf(a.x, f[0], fmaf(a.y, f[1], fmaf(a.z, f[2], fmaf(a.w, f[3], acc[t]))));
      acc[t] = fmaf(b.x, f[4], fmaf(b.y, f[5], fmaf(b.z, f[6], fmaf(b.w, f[7], acc[t]))));
    }
  }
#pragma unroll
  for (int t = 0; t < RL_TOKENS; ++t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
    if (lane == 0 && t < n) logits[static_cast<long long>(t0 + t) * E + e] = acc[t];
  }
}

static int row_blocks(long long rows) {
  const long long most = sm_count() * 16ll, want = (rows + WARPS - 1) / WARPS;
  return static_cast<int>(want < 1 ? 1 : want < most ? want : most);
}

}  // namespace gkmp

using namespace gkmp;

// Ints of scratch gk_moe_plan needs.
GK_EXPORT long long gk_moe_plan_scratch(int n, int E) {
  const long long chunks = (n + CHUNK - 1) / CHUNK;
  return chunks > 1 ? chunks * E : 0;
}

// idx [n] -> dest [n], src [rows the padded segments take] (-1 in padding rows), offsets [E + 1]; segments padded to `seg`.
GK_EXPORT int gk_moe_plan(const long long* idx, int n, int E, int seg, int* scratch, int* dest, int* src, int* offsets,
                          void* stream) {
  if (n < 1 || E < 1 || E > MAX_E || seg < 1) return -1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int chunks = (n + CHUNK - 1) / CHUNK;
  if (chunks > 1) {
    if (!scratch) return -2;
    moe_count_kernel<<<chunks, THREADS, 0, st>>>(idx, n, E, scratch);
  }
  moe_place_kernel<<<chunks, THREADS, 0, st>>>(idx, n, E, seg, chunks > 1 ? scratch : nullptr, dest, src, offsets);
  return launch_status();
}

// out [rows_bound, H] bf16: row r = x[src[r] / K], zero where src is -1, for the first *n_rows rows.
GK_EXPORT int gk_moe_gather(const void* x, const int* src, const int* n_rows, void* out, int rows_bound, int K, int H,
                            void* stream) {
  if (H % 8 || K < 1) return -1;
  moe_gather_kernel<<<row_blocks(rows_bound), THREADS, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), src, n_rows, static_cast<uint4*>(out), K, H / 8);
  return launch_status();
}

// w [T, K] or null (ones).
GK_EXPORT int gk_moe_combine(const void* rows, const float* w, const int* dest, void* y, int T, int K, int H, void* stream) {
  if (H % 8 || K < 1) return -1;
  if (T == 0) return 0;
  const int vecs = H / 8, threads = vecs >= THREADS ? THREADS : (vecs + 31) / 32 * 32;
  const int gx = (vecs + threads - 1) / threads;
  const int gy = T < sm_count() * 16 ? T : sm_count() * 16;
  launch_k(w ? moe_combine_kernel<true> : moe_combine_kernel<false>, dim3(gx, gy), dim3(threads), 0,
           reinterpret_cast<cudaStream_t>(stream), static_cast<const uint4*>(rows), w, dest, static_cast<uint4*>(y), T, K, vecs);
  return launch_status();
}

GK_EXPORT int gk_moe_combine_bwd(const void* dy, const void* rows, const float* w, const int* src, const int* n_rows,
                                 void* drows, float* dw, int rows_bound, int K, int H, void* stream) {
  if (H % 8 || K < 1) return -1;
  moe_combine_bwd_kernel<<<row_blocks(rows_bound), THREADS, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(dy), static_cast<const uint4*>(rows), w, src, n_rows, static_cast<uint4*>(drows), dw, K,
      H / 8);
  return launch_status();
}

// h [T, H] bf16, w [E, H] fp32 -> logits [T, E]; counts [E] (or null) cleared.  H a multiple of 8, at most 6144.
GK_EXPORT int gk_router_logits(const void* h, const float* w, float* logits, int* counts, int T, int E, int H, void* stream) {
  if (T < 1 || E < 1 || H % 8 || H < 8 || H > 6144) return -1;
  const int smem = RL_TOKENS * H * 2;
  static int configured = 0;
  if (smem > 48 * 1024 && !configured) {
    if (cudaFuncSetAttribute(router_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RL_TOKENS * 6144 * 2) != cudaSuccess)
      return -6;
    configured = 1;
  }
  launch_k(router_logits_kernel, dim3((E + RL_WARPS - 1) / RL_WARPS, (T + RL_TOKENS - 1) / RL_TOKENS), dim3(RL_WARPS * 32), smem,
           reinterpret_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(h), w, logits, counts, T, E, H);
  return launch_status();
}
