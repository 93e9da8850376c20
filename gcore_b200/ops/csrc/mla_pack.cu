// Latent attention around its projections (multi-head attention on a compressed latent and one rotated key for all heads):
//   * mla_expand        keys [T, heads, dn + dr] and values [T, heads, dv] out of the up-projected latent [T, heads, dn + dv]
//                       and the shared rotated key [T, dr], and the backward (the shared key's gradient is a sum over heads);
//   * latent_append     one decode token per request: norm of the latent, rotation of the shared key, both into the cache row.
// Bound by the bytes they move.  Keys and values of 3400 tokens, 128 heads of 128 + 64 / 128, as concatenations and copies ->
// here, us (floor 78): forward 481 -> 117, backward 525 -> 123.
#include "host_utils.h"
#include <cuda_bf16.h>

namespace gkml {
using namespace gk;

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

// Sizes in 16-byte units: n = dn / 8, r = dr / 8, v = dv / 8.
__global__ void __launch_bounds__(256) mla_expand_kernel(const uint4* __restrict__ kvu, const uint4* __restrict__ kr,
                                                         uint4* __restrict__ k, uint4* __restrict__ val, int T, int heads, int n,
                                                         int r, int v) {
  const unsigned per = n + r + v, units = heads * per;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    const uint4* src = kvu + static_cast<size_t>(t) * heads * (n + v);
    const uint4* key = kr + static_cast<size_t>(t) * r;
    uint4* kd = k + static_cast<size_t>(t) * heads * (n + r);
    uint4* vd = val + static_cast<size_t>(t) * heads * v;
#pragma unroll 4
    for (unsigned u = threadIdx.x; u < units; u += 256) {
      const int h = u / per, c = u - h * per;
      if (c < n) kd[h * (n + r) + c] = src[h * (n + v) + c];
      else if (c < n + r) kd[h * (n + r) + c] = key[c - n];
      else vd[h * v + c - n - r] = src[h * (n + v) + c - r];
    }
  }
}

// A CTA per token; r (a power of two, at most 32) threads side by side hold the columns of the shared key.
__global__ void __launch_bounds__(256) mla_expand_bwd_kernel(const uint4* __restrict__ dk, const uint4* __restrict__ dv,
                                                             uint4* __restrict__ dkvu, uint4* __restrict__ dkr, int T, int heads,
                                                             int n, int r, int v) {
  __shared__ float s_sum[256][9];
  const unsigned per = n + v, units = heads * per;
  const int col = threadIdx.x % r, group = threadIdx.x / r, groups = 256 / r;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    const uint4* kg = dk + static_cast<size_t>(t) * heads * (n + r);
    const uint4* vg = dv + static_cast<size_t>(t) * heads * v;
    uint4* out = dkvu + static_cast<size_t>(t) * units;
#pragma unroll 4
    for (unsigned u = threadIdx.x; u < units; u += 256) {
      const int h = u / per, c = u - h * per;
      out[u] = c < n ? kg[h * (n + r) + c] : vg[h * v + c - n];
    }
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int h = group; h < heads; h += groups) {
      float f[8];
      unpack8(kg[h * (n + r) + n + col], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += f[j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s_sum[threadIdx.x][j] = acc[j];
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < r) {
      for (int g = 1; g < groups; ++g) {
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += s_sum[g * r + threadIdx.x][j];
      }
      dkr[static_cast<size_t>(t) * r + threadIdx.x] = pack8(acc);
    }
    __syncthreads();
  }
}

// kv [B, ld]: latent (C values), then the shared key (dr values).  A CTA of 128 threads per request; C <= 1024.
__global__ void __launch_bounds__(128) latent_append_kernel(const __nv_bfloat16* __restrict__ kv, long long ld,
                                                            const __nv_bfloat16* __restrict__ gain, const int* __restrict__ pos,
                                                            const long long* __restrict__ slots, __nv_bfloat16* __restrict__ cache,
                                                            int C, int dr, float eps, float theta, int interleaved) {
  __shared__ float red[4];
  pdl_launch_dependents();
  const int tid = threadIdx.x, nv = C >> 3;
  uint4 gv = make_uint4(0, 0, 0, 0);
  if (tid < nv) gv = reinterpret_cast<const uint4*>(gain)[tid];
  pdl_wait();
  const int b = blockIdx.x;
  const __nv_bfloat16* row = kv + b * ld;
  __nv_bfloat16* out = cache + slots[b] * (C + dr);
  float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, ss = 0.f;
  if (tid < nv) unpack8(reinterpret_cast<const uint4*>(row)[tid], f);
#pragma unroll
  for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  const float rstd = rsqrtf(((red[0] + red[1]) + (red[2] + red[3])) / C + eps);
  if (tid < nv) {
    float g[8];
    unpack8(gv, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
    reinterpret_cast<uint4*>(out)[tid] = pack8(f);
  }
  const int half = dr >> 1;
  for (int i = tid; i < half; i += 128) {
    const float inv = __powf(theta, -2.f * i / dr);
    float s, c;
    sincosf(pos[b] * inv, &s, &c);
    const int i0 = interleaved ? 2 * i : i, i1 = interleaved ? 2 * i + 1 : i + half;
    const float a = __bfloat162float(row[C + i0]), d = __bfloat162float(row[C + i1]);
    out[C + i0] = __float2bfloat16(a * c - d * s);
    out[C + i1] = __float2bfloat16(d * c + a * s);
  }
}

static bool expand_ok(int heads, int dn, int dr, int dv) {
  return heads >= 1 && dn % 8 == 0 && dr % 8 == 0 && dv % 8 == 0 && dr >= 8 && dr <= 256 && 256 % (dr / 8) == 0;
}

}  // namespace gkml

using namespace gkml;

// kvu [T, heads, dn + dv], kr [T, dr] -> k [T, heads, dn + dr], v [T, heads, dv]; all bf16, contiguous, 16-byte aligned.
GK_EXPORT int gk_mla_expand(const void* kvu, const void* kr, void* k, void* v, int T, int heads, int dn, int dr, int dv,
                            void* stream) {
  if (!expand_ok(heads, dn, dr, dv)) return -1;
  if (T == 0) return 0;
  const int grid = T < sm_count() * 8 ? T : sm_count() * 8;
  mla_expand_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(kvu), static_cast<const uint4*>(kr), static_cast<uint4*>(k), static_cast<uint4*>(v), T, heads,
      dn / 8, dr / 8, dv / 8);
  return launch_status();
}

GK_EXPORT int gk_mla_expand_bwd(const void* dk, const void* dv_, void* dkvu, void* dkr, int T, int heads, int dn, int dr, int dv,
                                void* stream) {
  if (!expand_ok(heads, dn, dr, dv)) return -1;
  if (T == 0) return 0;
  const int grid = T < sm_count() * 8 ? T : sm_count() * 8;
  mla_expand_bwd_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(dk), static_cast<const uint4*>(dv_), static_cast<uint4*>(dkvu), static_cast<uint4*>(dkr), T,
      heads, dn / 8, dr / 8, dv / 8);
  return launch_status();
}

// slots [B]: cache row of every request (rows that rest share a row nobody reads).  C a multiple of 8, at most 1024.
GK_EXPORT int gk_latent_append(const void* kv, long long ld, const void* gain, const int* pos, const long long* slots, void* cache,
                               int B, int C, int dr, float eps, float theta, int interleaved, void* stream) {
  if (C % 8 || C < 8 || C > 1024 || dr % 8 || dr < 8 || ld % 8) return -1;
  if (B == 0) return 0;
  launch_k(latent_append_kernel, dim3(B), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream),
           static_cast<const __nv_bfloat16*>(kv), ld, static_cast<const __nv_bfloat16*>(gain), pos, slots,
           static_cast<__nv_bfloat16*>(cache), C, dr, eps, theta, interleaved);
  return launch_status();
}
