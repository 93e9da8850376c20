// Bandwidth-bound kernels of the transformer block and the optimizer: RMSNorm (+residual) fwd/bwd, RoPE
// fwd/bwd, SwiGLU fwd/bwd, fused Adam on the distributed-optimizer shard, squared-L2 norm, casts.
// All use 128-bit accesses; H, D and F must be multiples of 8.
//
// These stand in for the TransformerEngine / apex fused ops the reference reaches through Megatron-Core
// (gpatch_v4/training_backend/megatron_backend/mixin.py:311-348, optimizer.py:53-111).
#include "host_utils.h"
#include <cuda_bf16.h>

namespace gk {

struct alignas(16) bf16x8 { __nv_bfloat162 v[4]; };

__device__ __forceinline__ void unpack8(const bf16x8& a, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(a.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 a;
#pragma unroll
  for (int i = 0; i < 4; ++i) a.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return a;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffff, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffff, v, o));
  return v;
}
// Block-wide sum; `red` must hold 32 floats.  Every thread gets the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = lane < nw ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

// ------------------------------------------------------------------------------------------ RMSNorm
// y = (x [+ res]) * rstd * w ; optionally writes the summed residual stream to res_out.  Rows stay in registers between the
// sum of squares and the scaling, and the gains (weights of the model, which no kernel of a decode chain writes) are read
// before the wait for the kernel in front.  Every kernel adds the squares in the same order (thread, warp, block), so that a row
// gives the same bits in each.  us, forward with residual / backward, before -> now: 8000 x 3584 62 / 144 -> 53 / 102, 26000 x
// 4096 195 / 352 -> 154 / 192, 140000 heads of 128 217 / 633 -> 37 / 82 (calls of less than 80 us backward are host-bound).
//
// Rows of more than 256 values: a CTA per row, SLOTS 16-byte units per thread.
template <int SLOTS>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ res,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          __nv_bfloat16* __restrict__ y,
                                                          __nv_bfloat16* __restrict__ res_out,
                                                          float* __restrict__ rstd_out, int T, int H, float eps) {
  __shared__ float red[32];
  pdl_launch_dependents();
  const int nv = H >> 3;
  bf16x8 gain[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    const int i = threadIdx.x + s * 256;
    if (i < nv) gain[s] = reinterpret_cast<const bf16x8*>(w)[i];
  }
  pdl_wait();
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    const size_t at = static_cast<size_t>(row) * nv;
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x) + at;
    bf16x8 v[SLOTS], r[SLOTS];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int i = threadIdx.x + s * 256;
      if (i < nv) {
        v[s] = xr[i];
        if (res) r[s] = reinterpret_cast<const bf16x8*>(res)[at + i];
      }
    }
    float ss = 0.f;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int i = threadIdx.x + s * 256;
      if (i < nv) {
        float f[8];
        unpack8(v[s], f);
        if (res) {
          float g[8];
          unpack8(r[s], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] += g[j];
          v[s] = pack8(f);
          if (res_out) reinterpret_cast<bf16x8*>(res_out)[at + i] = v[s];
          unpack8(v[s], f);  // normalise what the residual stream actually stores
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
      }
    }
    ss = block_sum(ss, red);
    const float rstd = rsqrtf(ss / H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int i = threadIdx.x + s * 256;
      if (i < nv) {
        float f[8], g[8];
        unpack8(v[s], f);
        unpack8(gain[s], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
        reinterpret_cast<bf16x8*>(y)[at + i] = pack8(f);
      }
    }
  }
}

// Rows of at most 256 values (heads): LANES lanes of a warp per row, a CTA of eight warps for 256 / LANES rows.  With a CTA
// per row 16 of 256 threads had work.
template <int LANES>
__global__ void __launch_bounds__(256) rmsnorm_fwd_small_kernel(const __nv_bfloat16* __restrict__ x,
                                                                const __nv_bfloat16* __restrict__ res,
                                                                const __nv_bfloat16* __restrict__ w,
                                                                __nv_bfloat16* __restrict__ y,
                                                                __nv_bfloat16* __restrict__ res_out,
                                                                float* __restrict__ rstd_out, int T, int H, float eps) {
  pdl_launch_dependents();
  const int nv = H >> 3, i = threadIdx.x % LANES;
  float g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (i < nv) unpack8(reinterpret_cast<const bf16x8*>(w)[i], g);
  pdl_wait();
  constexpr int ROWS = 256 / LANES;
  for (long long r0 = static_cast<long long>(blockIdx.x) * ROWS; r0 < T; r0 += static_cast<long long>(gridDim.x) * ROWS) {
    const long long row = r0 + threadIdx.x / LANES;
    const bool mine = row < T && i < nv;
    const size_t at = static_cast<size_t>(row) * nv + i;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, ss = 0.f;
    if (mine) {
      unpack8(reinterpret_cast<const bf16x8*>(x)[at], f);
      if (res) {
        float a[8];
        unpack8(reinterpret_cast<const bf16x8*>(res)[at], a);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += a[j];
        const bf16x8 sum = pack8(f);
        if (res_out) reinterpret_cast<bf16x8*>(res_out)[at] = sum;
        unpack8(sum, f);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rstd = rsqrtf(ss / H + eps);
    if (mine) {
      if (i == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
      reinterpret_cast<bf16x8*>(y)[at] = pack8(f);
    }
  }
}

// dx = rstd * (g*w - x * rstd^2 * mean(g*w*x)) [+ dres] ; partial dw per CTA (reduced by a second kernel).  The gains and a
// row stay in registers; the next row's loads are under way while the CTA adds up this one's.
template <int SLOTS>
__global__ void __launch_bounds__(256) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ g,
                                                          const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          const float* __restrict__ rstd,
                                                          const __nv_bfloat16* __restrict__ dres,
                                                          __nv_bfloat16* __restrict__ dx,
                                                          float* __restrict__ dw_partial, int T, int H) {
  __shared__ float red[32];
  const int nv = H >> 3;
  float dw[SLOTS][8];
  bf16x8 wv[SLOTS], gv[SLOTS], xv[SLOTS], dv[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    const int i = threadIdx.x + s * 256;
    if (i < nv) wv[s] = reinterpret_cast<const bf16x8*>(w)[i];
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[s][j] = 0.f;
  }
  float rs = 0.f;
  auto load = [&](int row) {
    if (row >= T) return;
    const size_t at = static_cast<size_t>(row) * nv;
    rs = rstd[row];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int i = threadIdx.x + s * 256;
      if (i < nv) {
        gv[s] = reinterpret_cast<const bf16x8*>(g)[at + i];
        xv[s] = reinterpret_cast<const bf16x8*>(x)[at + i];
        if (dres) dv[s] = reinterpret_cast<const bf16x8*>(dres)[at + i];
      }
    }
  };
  load(blockIdx.x);
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    bf16x8 cg[SLOTS], cx[SLOTS], cd[SLOTS];
    const float crs = rs;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) { cg[s] = gv[s]; cx[s] = xv[s]; cd[s] = dv[s]; }
    load(row + gridDim.x);
    float dot = 0.f;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      if (threadIdx.x + s * 256 < nv) {
        float gf[8], xf[8], wf[8];
        unpack8(cg[s], gf);
        unpack8(cx[s], xf);
        unpack8(wv[s], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dot += gf[j] * wf[j] * xf[j];
          dw[s][j] += gf[j] * xf[j] * crs;
        }
      }
    }
    dot = block_sum(dot, red);
    const float c = dot * crs * crs / H;
    bf16x8* dxr = reinterpret_cast<bf16x8*>(dx) + static_cast<size_t>(row) * nv;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int i = threadIdx.x + s * 256;
      if (i < nv) {
        float gf[8], xf[8], wf[8], o[8];
        unpack8(cg[s], gf);
        unpack8(cx[s], xf);
        unpack8(wv[s], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = crs * (gf[j] * wf[j] - xf[j] * c);
        if (dres) {
          float d[8];
          unpack8(cd[s], d);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += d[j];
        }
        dxr[i] = pack8(o);
      }
    }
  }
  float* out = dw_partial + static_cast<size_t>(blockIdx.x) * H;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    const int i = threadIdx.x + s * 256;
    if (i < nv) {
#pragma unroll
      for (int j = 0; j < 8; ++j) out[i * 8 + j] = dw[s][j];
    }
  }
}

// Rows of at most 256 values: LANES lanes per row, two rows of a group under way.
template <int LANES>
__global__ void __launch_bounds__(256) rmsnorm_bwd_small_kernel(const __nv_bfloat16* __restrict__ g,
                                                                const __nv_bfloat16* __restrict__ x,
                                                                const __nv_bfloat16* __restrict__ w,
                                                                const float* __restrict__ rstd,
                                                                const __nv_bfloat16* __restrict__ dres,
                                                                __nv_bfloat16* __restrict__ dx,
                                                                float* __restrict__ dw_partial, int T, int H) {
  constexpr int ROWS = 256 / LANES, U = 2;
  __shared__ float s_dw[ROWS][LANES * 8];
  const int nv = H >> 3, i = threadIdx.x % LANES, group = threadIdx.x / LANES;
  float wf[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, dw[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (i < nv) unpack8(reinterpret_cast<const bf16x8*>(w)[i], wf);
  const long long step = static_cast<long long>(gridDim.x) * ROWS;
  for (long long r0 = static_cast<long long>(blockIdx.x) * ROWS; r0 < T; r0 += U * step) {
    bf16x8 gv[U], xv[U], dv[U];
    float rs[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long row = r0 + u * step + group;
      if (row < T && i < nv) {
        const size_t at = static_cast<size_t>(row) * nv + i;
        gv[u] = reinterpret_cast<const bf16x8*>(g)[at];
        xv[u] = reinterpret_cast<const bf16x8*>(x)[at];
        if (dres) dv[u] = reinterpret_cast<const bf16x8*>(dres)[at];
        rs[u] = rstd[row];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long row = r0 + u * step + group;
      const bool mine = row < T && i < nv;
      float gf[8], xf[8], dot = 0.f;
      if (mine) {
        unpack8(gv[u], gf);
        unpack8(xv[u], xf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dot += gf[j] * wf[j] * xf[j];
          dw[j] += gf[j] * xf[j] * rs[u];
        }
      }
#pragma unroll
      for (int o = LANES / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (mine) {
        const float c = dot * rs[u] * rs[u] / H;
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rs[u] * (gf[j] * wf[j] - xf[j] * c);
        if (dres) {
          float d[8];
          unpack8(dv[u], d);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += d[j];
        }
        reinterpret_cast<bf16x8*>(dx)[static_cast<size_t>(row) * nv + i] = pack8(o);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) s_dw[group][i * 8 + j] = dw[j];
  __syncthreads();
  if (static_cast<int>(threadIdx.x) < H) {
    float sum = 0.f;
    for (int k = 0; k < ROWS; ++k) sum += s_dw[k][threadIdx.x];
    dw_partial[static_cast<size_t>(blockIdx.x) * H + threadIdx.x] = sum;
  }
}

// Column sums of the CTAs' partials: 32 columns a CTA, eight threads share a column.
__global__ void __launch_bounds__(256) colsum_partial_kernel(const float* __restrict__ partial, float* __restrict__ out,
                                                             int nparts, int H, int accumulate) {
  __shared__ float s_sum[8][33];
  const int c = threadIdx.x & 31, k = threadIdx.x >> 5, i = blockIdx.x * 32 + c;
  float s = 0.f;
  if (i < H) {
#pragma unroll 8
    for (int p = k; p < nparts; p += 8) s += partial[static_cast<size_t>(p) * H + i];
  }
  s_sum[k][c] = s;
  __syncthreads();
  if (k == 0 && i < H) {
    for (int q = 1; q < 8; ++q) s += s_sum[q][c];
    out[i] = accumulate ? out[i] + s : s;
  }
}

constexpr int RMS_SMALL_H = 256, RMS_MAX_H = 256 * 8 * 4;

inline int rmsnorm_bwd_launch(const void* g, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                              float* dw_partial, float* dw, int dw_accumulate, int T, int H, int parts, cudaStream_t st) {
  const auto* gp = static_cast<const __nv_bfloat16*>(g);
  const auto* xp = static_cast<const __nv_bfloat16*>(x);
  const auto* wp = static_cast<const __nv_bfloat16*>(w);
  const auto* dp = static_cast<const __nv_bfloat16*>(dres);
  auto* op = static_cast<__nv_bfloat16*>(dx);
  const int rows = H <= 64 ? 32 : H <= 128 ? 16 : H <= RMS_SMALL_H ? 8 : 1;   // of a CTA at a time
  if (parts > (T + rows - 1) / rows) parts = T > 0 ? (T + rows - 1) / rows : 1;
  auto go = [&](auto kernel) { kernel<<<parts, 256, 0, st>>>(gp, xp, wp, rstd, dp, op, dw_partial, T, H); };
  if (H <= 64) go(rmsnorm_bwd_small_kernel<8>);
  else if (H <= 128) go(rmsnorm_bwd_small_kernel<16>);
  else if (H <= RMS_SMALL_H) go(rmsnorm_bwd_small_kernel<32>);
  else if (H <= 2048) go(rmsnorm_bwd_kernel<1>);
  else if (H <= 4096) go(rmsnorm_bwd_kernel<2>);
  else if (H <= 6144) go(rmsnorm_bwd_kernel<3>);
  else go(rmsnorm_bwd_kernel<4>);
  colsum_partial_kernel<<<(H + 31) / 32, 256, 0, st>>>(dw_partial, dw, parts, H, dw_accumulate);
  return launch_status();
}

// ------------------------------------------------------------------------------------------ RoPE
// In-place rotation of the first `rot` dims of every head (rotate-half / "neox" pairing: i <-> i + rot/2).
// x is [T, nheads, D] with token stride `stride_t` elements (so it can be a slice of a packed QKV buffer).
// sign = +1 forward, -1 backward (the transpose of a rotation is the rotation by the negated angle).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos, int T, int nheads, int D,
                            int rot, long long stride_t, float theta, float sign, int interleaved) {
  const int half = rot >> 1;
  const long long total = static_cast<long long>(T) * nheads * half;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(idx % half);
    const long long th = idx / half;
    const int h = static_cast<int>(th % nheads);
    const int t = static_cast<int>(th / nheads);
    const float inv = __powf(theta, -2.f * i / rot);
    float s, c;
    sincosf(pos[t] * inv, &s, &c);
    s *= sign;
    __nv_bfloat16* p = x + t * stride_t + static_cast<long long>(h) * D;
    const int i0 = interleaved ? 2 * i : i;
    const int i1 = interleaved ? 2 * i + 1 : i + half;
    const float a = __bfloat162float(p[i0]), b = __bfloat162float(p[i1]);
    p[i0] = __float2bfloat16(a * c - b * s);
    p[i1] = __float2bfloat16(b * c + a * s);
  }
}

// The same for aligned rows: 16-byte units, and one angle for all heads of a token.  A CTA takes `tokens` tokens of `heads`
// heads (grid: tokens, heads).  Rotates the values [off, off + rot) of every head; with y != x the other values are copied.
// 8000 tokens of 32 heads of 128: 35 us against 68 a pair at a time, 26000 tokens of 40 heads 139 against 309.
constexpr int ROPE_ANGLES = 1024, ROPE_MAX_ROT = 512;
__global__ void __launch_bounds__(256) rope_rows_kernel(const __nv_bfloat16* x, __nv_bfloat16* y, const int* __restrict__ pos,
                                                        int T, int nheads, int D, int off, int rot, long long ldx, long long ldy,
                                                        float theta, float sign, int interleaved, int tokens, int heads) {
  __shared__ float2 cs[ROPE_ANGLES];   // tokens * rot / 2
  const int half = rot >> 1, t0 = blockIdx.x * tokens, n = T - t0 < tokens ? T - t0 : tokens;
  const int h0 = blockIdx.y * heads, nh = nheads - h0 < heads ? nheads - h0 : heads;
  for (int k = threadIdx.x; k < n * half; k += 256) {
    const int tok = k / half, i = k - tok * half;
    const float inv = __powf(theta, -2.f * i / rot);
    float s, c;
    sincosf(pos[t0 + tok] * inv, &s, &c);
    cs[k] = make_float2(c, s * sign);
  }
  __syncthreads();
  const unsigned turned = interleaved ? rot >> 3 : rot >> 4;               // units of a head that rotate: one or two vectors
  const unsigned lead = off >> 3, kept = x == y ? 0 : (D - rot) >> 3;      // vectors that are copied, `lead` of them in front
  const unsigned per = turned + kept, units = n * nh * per;
  for (unsigned u = threadIdx.x; u < units; u += 256) {
    const unsigned th = u / per, k = u - th * per, tok = th / nh, h = h0 + th - tok * nh;
    const bf16x8* from = reinterpret_cast<const bf16x8*>(x + (t0 + tok) * ldx + static_cast<long long>(h) * D);
    bf16x8* to = reinterpret_cast<bf16x8*>(y + (t0 + tok) * ldy + static_cast<long long>(h) * D);
    if (k >= turned) {
      const unsigned c = k - turned < lead ? k - turned : k - turned + (rot >> 3);
      to[c] = from[c];
      continue;
    }
    const float2* ang = cs + tok * half;
    if (interleaved) {
      float f[8];
      unpack8(from[lead + k], f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float c = ang[4 * k + j].x, s = ang[4 * k + j].y, a = f[2 * j], b = f[2 * j + 1];
        f[2 * j] = a * c - b * s;
        f[2 * j + 1] = b * c + a * s;
      }
      to[lead + k] = pack8(f);
    } else {
      const unsigned other = lead + k + (half >> 3);
      float f[8], g[8];
      unpack8(from[lead + k], f);
      unpack8(from[other], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float c = ang[8 * k + j].x, s = ang[8 * k + j].y, a = f[j], b = g[j];
        f[j] = a * c - b * s;
        g[j] = b * c + a * s;
      }
      to[lead + k] = pack8(f);
      to[other] = pack8(g);
    }
  }
}

// A CTA for about 256 units of 16 bytes: several tokens of few heads where there are tokens enough to fill the GPU, a share of
// the heads where there are not.  128 heads of 128 + 64, the 64 rotated, us, four tokens a CTA -> here (split and rotated in two
// launches): 1 token 8.6 -> 2.3 (4.5), 32 tokens 28.8 -> 3.0 (6.1), 512 tokens 29.9 -> 14 (21.5), 3400 tokens 93 -> 83 (143).
static int rope_rows_launch(const void* x, void* y, const int* pos, int T, int nheads, int D, int off, int rot, long long ldx,
                            long long ldy, float theta, int backward, int interleaved, cudaStream_t st) {
  const int per = (interleaved ? rot >> 3 : rot >> 4) + (x == y ? 0 : (D - rot) >> 3), sms = sm_count();
  const long long units = static_cast<long long>(nheads) * per;   // of a token
  int tokens = 1, gy = 1;
  if (units < 256) {
    const int room = 2 * ROPE_ANGLES / rot, spare = T / (2 * sms);
    tokens = static_cast<int>(256 / units);
    if (tokens > room) tokens = room;
    if (tokens > spare) tokens = spare;
    if (tokens < 1) tokens = 1;
  } else {
    gy = (4 * sms + T - 1) / T;
    if (gy > (units + 255) / 256) gy = static_cast<int>((units + 255) / 256);
  }
  const int heads = (nheads + gy - 1) / gy;
  rope_rows_kernel<<<dim3((T + tokens - 1) / tokens, (nheads + heads - 1) / heads), 256, 0, st>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), pos, T, nheads, D, off, rot, ldx, ldy, theta,
      backward ? -1.f : 1.f, interleaved, tokens, heads);
  return launch_status();
}

// Same rotation with the angles given as tables cos / sin [T, rot / 2] (multi-axis rotary position ids of
// vision-language models: every frequency takes its angle from the temporal, height or width index of the token).
__global__ void rope_table_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ cs,
                                  const float* __restrict__ sn, int T, int nheads, int D, int rot, long long stride_t,
                                  float sign, int interleaved) {
  const int half = rot >> 1;
  const long long total = static_cast<long long>(T) * nheads * half;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(idx % half);
    const long long th = idx / half;
    const int h = static_cast<int>(th % nheads);
    const int t = static_cast<int>(th / nheads);
    const float c = cs[static_cast<long long>(t) * half + i];
    const float s = sn[static_cast<long long>(t) * half + i] * sign;
    __nv_bfloat16* p = x + t * stride_t + static_cast<long long>(h) * D;
    const int i0 = interleaved ? 2 * i : i;
    const int i1 = interleaved ? 2 * i + 1 : i + half;
    const float a = __bfloat162float(p[i0]), b = __bfloat162float(p[i1]);
    p[i0] = __float2bfloat16(a * c - b * s);
    p[i1] = __float2bfloat16(b * c + a * s);
  }
}

// ------------------------------------------------------------------------------------------ SwiGLU
// in [T, 2F] = [gate | up]; out [T, F] = silu(gate) * up
// A thread's (row, 8-wide column vector) pair advances by the grid stride without a division per element: one 64-bit
// division at entry, then carries (a division per element made the kernel issue-bound: 99 us for 9216 x 1536 outputs).
struct RowColIter {
  long long t;
  int i, di, nv;
  long long dt;
  __device__ RowColIter(int nv_) : nv(nv_) {
    const long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
    t = idx / nv;
    i = static_cast<int>(idx - t * nv);
    dt = step / nv;
    di = static_cast<int>(step - dt * nv);
  }
  __device__ void next() {
    t += dt;
    i += di;
    if (i >= nv) { i -= nv; ++t; }
  }
};

// n_rows (device, optional): rows at or beyond *n_rows are left untouched (expert-sorted buffers sized for the worst
// case carry a device-side count of the rows in use).
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out, long long T,
                                  int F, const int* __restrict__ n_rows) {
  pdl_launch_dependents();
  pdl_wait();
  const int nv = F >> 3;
  if (n_rows && *n_rows < T) T = *n_rows;
  for (RowColIter it(nv); it.t < T; it.next()) {
    const long long t = it.t;
    const int i = it.i;
    const bf16x8* row = reinterpret_cast<const bf16x8*>(in + t * 2 * F);
    float g[8], u[8];
    unpack8(row[i], g);
    unpack8(row[nv + i], u);
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    reinterpret_cast<bf16x8*>(out + t * F)[i] = pack8(g);
  }
}
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ in,
                                  __nv_bfloat16* __restrict__ din, long long T, int F) {
  const int nv = F >> 3;
  for (RowColIter it(nv); it.t < T; it.next()) {
    const long long t = it.t;
    const int i = it.i;
    const bf16x8* row = reinterpret_cast<const bf16x8*>(in + t * 2 * F);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(row[i], g);
    unpack8(row[nv + i], u);
    unpack8(reinterpret_cast<const bf16x8*>(dout + t * F)[i], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sg = 1.f / (1.f + __expf(-g[j]));
      const float silu = g[j] * sg;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * sg * (1.f + g[j] * (1.f - sg));
    }
    bf16x8* orow = reinterpret_cast<bf16x8*>(din + t * 2 * F);
    orow[i] = pack8(dg);
    orow[nv + i] = pack8(du);
  }
}

// ------------------------------------------------------------------------------------------ Adam
// One pass over the optimizer shard: unscale/clip the gradient, AdamW on the fp32 master, write the bf16
// parameter.  `scale_ptr` (device) holds the combined gradient multiplier (1/loss-scale * clip coefficient) so
// the clip coefficient never visits the host.
struct AdamArgs {
  float *master, *m, *v;
  const void* grad;
  __nv_bfloat16* param;   // or null
  long long n;
  float lr, b1, b2, eps, wd, bc1, bc2;
  const float* scale_ptr;
  float scale_val;
};
__device__ __forceinline__ float adam_one(const AdamArgs& a, float g, float& m, float& v, float p) {
  m = a.b1 * m + (1.f - a.b1) * g;
  v = a.b2 * v + (1.f - a.b2) * g * g;
  const float upd = (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps) + a.wd * p;
  return p - a.lr * upd;
}
// HBM-bound at 28 bytes moved per element (fp32 gradient).  VEC: a thread takes four neighbours at a time, so that it has
// 64 bytes in flight instead of 16 (700 M elements: 3.62 ms, 5.4 TB/s, against 4.69 ms; 45 M: 241 against 291 us).  One by one:
// unaligned shards, and the last elements in the same launch (63 elements: 2.3 us, 3.6 with a launch of their own).
template <bool GRAD32, bool VEC>
__global__ void __launch_bounds__(256) adam_kernel(const AdamArgs a) {
  const float scale = (a.scale_ptr ? *a.scale_ptr : 1.f) * a.scale_val;
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  if (VEC) {
    for (long long i = t * 4; i + 3 < a.n; i += step * 4) {
      float4 g;
      if (GRAD32) {
        g = __ldcs(reinterpret_cast<const float4*>(static_cast<const float*>(a.grad) + i));
      } else {
        const uint2 r = __ldcs(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(a.grad) + i));
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
        g = make_float4(x.x, x.y, y.x, y.y);
      }
      float4 m = __ldcs(reinterpret_cast<const float4*>(a.m + i)), v = __ldcs(reinterpret_cast<const float4*>(a.v + i));
      float4 p = __ldcs(reinterpret_cast<const float4*>(a.master + i));
      p.x = adam_one(a, g.x * scale, m.x, v.x, p.x);
      p.y = adam_one(a, g.y * scale, m.y, v.y, p.y);
      p.z = adam_one(a, g.z * scale, m.z, v.z, p.z);
      p.w = adam_one(a, g.w * scale, m.w, v.w, p.w);
      __stcs(reinterpret_cast<float4*>(a.m + i), m);
      __stcs(reinterpret_cast<float4*>(a.v + i), v);
      __stcs(reinterpret_cast<float4*>(a.master + i), p);
      if (a.param) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(p.x, p.y), hi = __floats2bfloat162_rn(p.z, p.w);
        uint2 r;
        r.x = *reinterpret_cast<const uint32_t*>(&lo);
        r.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(a.param + i) = r;
      }
    }
  }
  for (long long i = (VEC ? a.n / 4 * 4 : 0) + t; i < a.n; i += step) {
    const float g = (GRAD32 ? static_cast<const float*>(a.grad)[i]
                            : __bfloat162float(static_cast<const __nv_bfloat16*>(a.grad)[i])) * scale;
    float m = a.m[i], v = a.v[i];
    const float p = adam_one(a, g, m, v, a.master[i]);
    a.m[i] = m;
    a.v[i] = v;
    a.master[i] = p;
    if (a.param) a.param[i] = __float2bfloat16(p);
  }
}

// Every thread keeps four partial sums; VEC (16-byte aligned input): 16 bytes a load, four loads in flight (700 M fp32: 468 us,
// 6.0 TB/s, against 729 us; 45 M: 47 against 64 us).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) sumsq_kernel(const T* __restrict__ x, long long n, float* __restrict__ out) {
  __shared__ float red[32];
  constexpr int W = 16 / sizeof(T);
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  long long done = 0;
  if (VEC) {
    const long long nv = n / W;
    const uint4* xv = reinterpret_cast<const uint4*>(x);
    auto add = [](uint4 r, float& acc) {
      const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const float f = static_cast<float>(e[j]);
        acc += f * f;
      }
    };
    long long i = t;
    for (; i + 3 * step < nv; i += 4 * step) {
      uint4 r[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) r[u] = __ldg(xv + i + u * step);
#pragma unroll
      for (int u = 0; u < 4; ++u) add(r[u], s[u]);
    }
    for (; i < nv; i += step) add(__ldg(xv + i), s[0]);
    done = nv * W;
  }
  for (long long i = done + t; i < n; i += step) {
    const float f = static_cast<float>(x[i]);
    s[1] += f * f;
  }
  const float sum = block_sum((s[0] + s[1]) + (s[2] + s[3]), red);
  if (threadIdx.x == 0) atomicAdd(out, sum);
}

// dst(bf16 or fp32) (+)= scale * src
__global__ void axpy_cast_kernel(const void* __restrict__ src, int src_fp32, void* __restrict__ dst, int dst_fp32,
                                 long long n, float scale, int accumulate) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float f = (src_fp32 ? reinterpret_cast<const float*>(src)[i]
                        : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(src)[i])) * scale;
    if (dst_fp32) {
      float* d = reinterpret_cast<float*>(dst);
      d[i] = accumulate ? d[i] + f : f;
    } else {
      __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(dst);
      d[i] = __float2bfloat16(accumulate ? __bfloat162float(d[i]) + f : f);
    }
  }
}

inline int grid_for(long long work_items, int threads, int waves = 8) {
  long long b = (work_items + threads - 1) / threads;
  const long long cap = static_cast<long long>(sm_count()) * waves;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace gk

using namespace gk;

GK_EXPORT int gk_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out, float* rstd,
                             int T, int H, float eps, void* stream) {
  if (H % 8 || H > RMS_MAX_H) return -1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto go = [&](auto kernel, int grid, int threads) {
    launch_k(kernel, dim3(grid > 0 ? grid : 1), dim3(threads), 0, st, static_cast<const __nv_bfloat16*>(x),
             static_cast<const __nv_bfloat16*>(res), static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y),
             static_cast<__nv_bfloat16*>(res_out), rstd, T, H, eps);
    return launch_status();
  };
  const int nv = H / 8, sms = sm_count();
  if (H <= 64) return go(rmsnorm_fwd_small_kernel<8>, grid_for(T, 32), 256);
  if (H <= 128) return go(rmsnorm_fwd_small_kernel<16>, grid_for(T, 16), 256);
  if (H <= RMS_SMALL_H) return go(rmsnorm_fwd_small_kernel<32>, grid_for(T, 8), 256);
  const int grid = T < sms * 8 ? T : sms * 8;
  if (nv <= 256) return go(rmsnorm_fwd_kernel<1>, grid, 256);
  if (nv <= 512) return go(rmsnorm_fwd_kernel<2>, grid, 256);
  return go(rmsnorm_fwd_kernel<4>, grid, 256);
}

// Per-head RMSNorm of the query and key heads of packed [q | k | v] rows, in place (decode / prefill of models with
// q / k layer norms): one warp per (token, head), D <= 256.  Replaces two norm launches over reshaped copies and the
// copies back into the packed rows.
__global__ void qk_headnorm_kernel(__nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
                                   const __nv_bfloat16* __restrict__ wk, long long T, int Hq, int Hk, int D,
                                   long long stride_t, float eps) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long warp = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const long long nwarps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const int heads = Hq + Hk;
  const int nv = D >> 3;
  for (long long w = warp; w < T * heads; w += nwarps) {
    const long long t = w / heads;
    const int h = static_cast<int>(w - t * heads);
    bf16x8* row = reinterpret_cast<bf16x8*>(qkv + t * stride_t + static_cast<long long>(h) * D);
    const bf16x8* g = reinterpret_cast<const bf16x8*>(h < Hq ? wq : wk);
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float ss = 0.f;
    if (lane < nv) {
      unpack8(row[lane], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffff, ss, off);
    const float rstd = rsqrtf(ss / D + eps);
    if (lane < nv) {
      float gw[8];
      unpack8(g[lane], gw);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * gw[j];
      row[lane] = pack8(f);
    }
  }
}

GK_EXPORT int gk_qk_headnorm(void* qkv, const void* wq, const void* wk, long long T, int Hq, int Hk, int D,
                             long long stride_t, float eps, void* stream) {
  if (D % 8 || D > 256 || stride_t % 8) return -1;
  if (T == 0) return 0;
  launch_k(qk_headnorm_kernel, dim3(grid_for(T * (Hq + Hk) * 32, 256)), dim3(256), 0,
           reinterpret_cast<cudaStream_t>(stream), reinterpret_cast<__nv_bfloat16*>(qkv),
           reinterpret_cast<const __nv_bfloat16*>(wq), reinterpret_cast<const __nv_bfloat16*>(wk), T, Hq, Hk, D, stride_t,
           eps);
  return launch_status();
}

GK_EXPORT int gk_rmsnorm_bwd_parts(int T) {
  const int cap = sm_count() * 2;
  return T < cap ? (T > 0 ? T : 1) : cap;
}

// dw_partial must hold gk_rmsnorm_bwd_parts(T) * H floats.
GK_EXPORT int gk_rmsnorm_bwd(const void* g, const void* x, const void* w, const float* rstd, const void* dres,
                             void* dx, float* dw_partial, float* dw, int dw_accumulate, int T, int H, void* stream) {
  if (H % 8 || H > RMS_MAX_H) return -1;
  return rmsnorm_bwd_launch(g, x, w, rstd, dres, dx, dw_partial, dw, dw_accumulate, T, H, gk_rmsnorm_bwd_parts(T),
                            reinterpret_cast<cudaStream_t>(stream));
}

static bool rope_rows_ok(const void* x, const void* y, int D, int off, int rot, long long ldx, long long ldy, int interleaved) {
  return D % 8 == 0 && off % 8 == 0 && rot % (interleaved ? 8 : 16) == 0 && rot >= 8 && rot <= ROPE_MAX_ROT && off + rot <= D &&
         ldx % 8 == 0 && ldy % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
}

// y = x [T, nheads, D] (contiguous rows, 16-byte aligned, y != x) with the values [off, off + rot) of every head rotated.
GK_EXPORT int gk_rope_copy(const void* x, void* y, const int* pos, int T, int nheads, int D, int off, int rot, float theta,
                           int backward, int interleaved, void* stream) {
  if (T == 0 || nheads == 0) return 0;   // both null then
  const long long ld = static_cast<long long>(nheads) * D;
  if (x == y || !rope_rows_ok(x, y, D, off, rot, ld, ld, interleaved)) return -1;
  return rope_rows_launch(x, y, pos, T, nheads, D, off, rot, ld, ld, theta, backward, interleaved,
                          reinterpret_cast<cudaStream_t>(stream));
}

GK_EXPORT int gk_rope(void* x, const int* pos, int T, int nheads, int D, int rot, long long stride_t, float theta,
                      int backward, int interleaved, void* stream) {
  if (rot % 2 || rot > D) return -1;
  const long long total = static_cast<long long>(T) * nheads * (rot / 2);
  if (total == 0) return 0;
  // Below about 100k pairs a launch is all latency, and a thread per pair has the shorter chain (us, pairs -> rows: 32 heads of
  // 128, 16 tokens 1.9 -> 2.4, 64 tokens 2.5 -> 2.5, 512 tokens 6.7 -> 4.4; one head of 64, 1024 tokens 1.9 -> 2.2).
  if (total >= 98304 && rope_rows_ok(x, x, D, 0, rot, stride_t, stride_t, interleaved))
    return rope_rows_launch(x, x, pos, T, nheads, D, 0, rot, stride_t, stride_t, theta, backward, interleaved,
                            reinterpret_cast<cudaStream_t>(stream));
  rope_kernel<<<grid_for(total, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<__nv_bfloat16*>(x), pos, T, nheads, D, rot, stride_t, theta, backward ? -1.f : 1.f,
      interleaved);
  return launch_status();
}

GK_EXPORT int gk_rope_table(void* x, const float* cs, const float* sn, int T, int nheads, int D, int rot,
                            long long stride_t, int backward, int interleaved, void* stream) {
  if (rot % 2 || rot > D) return -1;
  const long long total = static_cast<long long>(T) * nheads * (rot / 2);
  if (total == 0) return 0;
  rope_table_kernel<<<grid_for(total, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<__nv_bfloat16*>(x), cs, sn, T, nheads, D, rot, stride_t, backward ? -1.f : 1.f, interleaved);
  return launch_status();
}

static int swiglu_fwd_launch(const void* in, void* out, long long T, int F, const int* n_rows, void* stream) {
  if (F % 8) return -1;
  if (T == 0) return 0;
  launch_k(swiglu_fwd_kernel, dim3(grid_for(T * (F / 8), 256)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
      reinterpret_cast<const __nv_bfloat16*>(in), reinterpret_cast<__nv_bfloat16*>(out), T, F, n_rows);
  return launch_status();
}

GK_EXPORT int gk_swiglu_fwd(const void* in, void* out, long long T, int F, void* stream) {
  return swiglu_fwd_launch(in, out, T, F, nullptr, stream);
}

// rows at or beyond *n_rows (device) are not computed
GK_EXPORT int gk_swiglu_fwd_rows(const void* in, void* out, long long T, int F, const int* n_rows, void* stream) {
  return swiglu_fwd_launch(in, out, T, F, n_rows, stream);
}

GK_EXPORT int gk_swiglu_bwd(const void* dout, const void* in, void* din, long long T, int F, void* stream) {
  if (F % 8) return -1;
  if (T == 0) return 0;
  swiglu_bwd_kernel<<<grid_for(T * (F / 8), 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(dout), reinterpret_cast<const __nv_bfloat16*>(in),
      reinterpret_cast<__nv_bfloat16*>(din), T, F);
  return launch_status();
}

GK_EXPORT int gk_adam(float* master, float* m, float* v, const void* grad, int grad_fp32, void* param, long long n,
                      float lr, float b1, float b2, float eps, float wd, int step, const float* scale_ptr,
                      float scale_val, void* stream) {
  if (n == 0) return 0;
  const float bc1 = 1.f - powf(b1, static_cast<float>(step));
  const float bc2 = 1.f - powf(b2, static_cast<float>(step));
  const AdamArgs a = {master, m, v, grad, reinterpret_cast<__nv_bfloat16*>(param), n, lr, b1, b2, eps, wd, bc1, bc2,
                      scale_ptr, scale_val};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto bits = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
  const bool vec = ((bits(master) | bits(m) | bits(v) | (grad_fp32 ? bits(grad) : 0)) & 15) == 0 &&
                   ((bits(param) | bits(grad)) & 7) == 0;
  auto go = [&](auto kernel, int grid) { kernel<<<grid, 256, 0, st>>>(a); };
  if (vec) {
    const int grid = grid_for(n / 4, 256);
    if (grad_fp32) go(adam_kernel<true, true>, grid);
    else go(adam_kernel<false, true>, grid);
  } else {
    const int grid = grid_for(n, 256);
    if (grad_fp32) go(adam_kernel<true, false>, grid);
    else go(adam_kernel<false, false>, grid);
  }
  return launch_status();
}

// out[0] += sum(x^2); the caller zeroes out[0].
GK_EXPORT int gk_sumsq(const void* x, int is_fp32, long long n, float* out, void* stream) {
  if (n == 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && n >= 2048;   // below, one element a thread is one load deep
  // 64 bytes a thread; short inputs one load a thread as far as there are SMs (10000 fp32: 2.6 -> 2.0 us)
  const int once = grid_for(n * (is_fp32 ? 4 : 2) / 16, 256, 1), four = grid_for(n * (is_fp32 ? 4 : 2) / 64, 256);
  const int grid = !vec ? grid_for(n, 256, 4) : once > four ? once : four;
  if (is_fp32) {
    const float* f = static_cast<const float*>(x);
    if (vec) sumsq_kernel<float, true><<<grid, 256, 0, st>>>(f, n, out);
    else sumsq_kernel<float, false><<<grid, 256, 0, st>>>(f, n, out);
  } else {
    const __nv_bfloat16* h = static_cast<const __nv_bfloat16*>(x);
    if (vec) sumsq_kernel<__nv_bfloat16, true><<<grid, 256, 0, st>>>(h, n, out);
    else sumsq_kernel<__nv_bfloat16, false><<<grid, 256, 0, st>>>(h, n, out);
  }
  return launch_status();
}

GK_EXPORT int gk_axpy_cast(const void* src, int src_fp32, void* dst, int dst_fp32, long long n, float scale,
                           int accumulate, void* stream) {
  if (n == 0) return 0;
  axpy_cast_kernel<<<grid_for(n, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(src, src_fp32, dst,
                                                                                        dst_fp32, n, scale,
                                                                                        accumulate);
  return launch_status();
}

// ---------------------------------------------------------------------------------------------------------------
// Allocation-free variant of gk_rmsnorm_bwd (declared and documented in no_alloc.h).
#include "no_alloc.h"

namespace gk {
// Scratch for the per-CTA weight-gradient partials.  In host code this name is only a handle for the symbol: the
// device address has to be looked up (once per device) before it can be given to a kernel.
static __device__ __align__(256) float g_noalloc_rms_scratch[GK_NOALLOC_RMSNORM_MAX_PARTS * GK_NOALLOC_RMSNORM_MAX_H];
constexpr int NOALLOC_MAX_DEVICES = 64;
static float* g_noalloc_rms_ptr[NOALLOC_MAX_DEVICES] = {nullptr};
}  // namespace gk

GK_EXPORT int gk_rmsnorm_bwd_noalloc(const void* g, const void* x, const void* w, const float* rstd, const void* dres,
                                     void* dx, float* dw, int dw_accumulate, int T, int H, void* stream) {
  if (H % 8) return -1;
  if (H > GK_NOALLOC_RMSNORM_MAX_H) {
    fprintf(stderr, "[gcore_b200] gk_rmsnorm_bwd_noalloc: H=%d exceeds the built-in scratch (max H %d)\n", H,
            GK_NOALLOC_RMSNORM_MAX_H);
    return -2;
  }
  if (T <= 0) return 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return -3;
  if (!g_noalloc_rms_ptr[dev]) {
    // first call on this device: resolve the device address of the file-scope array
    float* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_rms_scratch);
    if (e != cudaSuccess || !p) {
      fprintf(stderr, "[gcore_b200] gk_rmsnorm_bwd_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
      return -3;
    }
    g_noalloc_rms_ptr[dev] = p;
  }
  float* scratch = g_noalloc_rms_ptr[dev];
  int parts = gk_rmsnorm_bwd_parts(T);
  if (parts > GK_NOALLOC_RMSNORM_MAX_PARTS) parts = GK_NOALLOC_RMSNORM_MAX_PARTS;
  return rmsnorm_bwd_launch(g, x, w, rstd, dres, dx, scratch, dw, dw_accumulate, T, H, parts,
                            reinterpret_cast<cudaStream_t>(stream));
}
