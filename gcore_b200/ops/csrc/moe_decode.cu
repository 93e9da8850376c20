// Expert projections of a decode step: a handful of tokens per expert, so the weights of the chosen experts are all that
// counts and HBM bounds the kernel.  y[r] = W[e] x[r] for the rows r of expert e, W [E, N, K], or, with ACT, the gated
// activation silu(gate) * up of the first projection (W [E, 2 F, K], gate rows first).
//
//   * swap-AB: the 128-row tcgen05 tile runs over weight rows (with ACT: 64 gate rows and the 64 up rows that belong to
//     them), an expert's tokens are the MMA N = 16.  Segments are padded to 16 rows, not to the 128 of the general grouped
//     GEMM, whose activations for 16 tokens on 83 experts (10.6 k padded rows) cost more than a tenth of the weights' time
//     and whose zero padding had to be written first.  Columns of padding rows are computed and not stored, so what the
//     padding holds does not matter.
//   * an expert with more than 16 tokens has several segments; they follow one another in the tile order, so that its
//     weights come from L2 the second time.
//   * persistent CTAs, one per SM, with a ring deep enough for 200 KB in flight; tiles in turn.
// Measured, a whole layer of 128 experts, 2048 wide, 768 each, top 8, in a replayed graph, us, through the 128-row grouped GEMM
// -> through this kernel, and the time the chosen experts' weights take from HBM: 1 token 157 -> 42 (12), 4 tokens 219 -> 82
// (45), 16 tokens 314 -> 156 (121), 64 tokens 471 -> 222 (184), 128 tokens 492 -> 232 (186).
// Roles per CTA: warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 epilogue.
#include "ptx.cuh"
#include "host_utils.h"

namespace gkmd {
using namespace gk;

constexpr int BM = 128, BK = 64, UMMA_K = 16, SEG = 16;
constexpr int THREADS = 192, STAGES = 11;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = SEG * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int MAX_EXPERTS = 512;
constexpr int UP_LD = SEG + 1;   // floats between two feature rows of the exchange buffer (odd: no bank conflicts)
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + 64 * UP_LD * 4 + (MAX_EXPERTS + 1) * 4;

struct Params {
  const int* offsets;   // [E + 1] rows, multiples of 16
  const int* counts;    // [E] rows of an expert that hold tokens
  __nv_bfloat16* Y;     // [rows, ldy]
  long long ldy;
  int E, N, K, F;       // F: outputs of an expert (N with ACT is 2 F, else F == N)
  int* err;
};

struct Tile {
  int expert, row0, valid, f;   // f: tile along the outputs
};
__device__ __forceinline__ Tile tile_at(const int* s_off, const Params& p, int tile, int ftiles) {
  Tile t;
  const int seg = tile / ftiles;
  t.f = tile - seg * ftiles;
  t.row0 = seg * SEG;
  int lo = 0, hi = p.E;         // the expert with s_off[lo] <= row0 < s_off[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s_off[mid] <= t.row0) lo = mid; else hi = mid;
  }
  t.expert = lo;
  const int left = p.counts[lo] - (t.row0 - s_off[lo]);
  t.valid = left < SEG ? left : SEG;
  return t;
}

__device__ __forceinline__ bool all_epilogue_warps(bool ok) {
  uint32_t all;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "barrier.red.and.pred q, 1, 128, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(all)
      : "r"(static_cast<uint32_t>(ok))
      : "memory");
  return all != 0;
}

template <bool ACT>
__global__ void __launch_bounds__(THREADS, 1)
moe_decode_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;   // 2
  uint64_t* tempty = tfull + 2;       // 2
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tempty + 2);
  float* s_up = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES + 256);
  int* s_off = reinterpret_cast<int*>(s_up + 64 * UP_LD);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], 128); }
    fence_barrier_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
  }
  if (warp == 2) { tmem_alloc(tmem_holder, 32); tmem_relinquish(); }
  pdl_wait();
  for (int e = threadIdx.x; e <= p.E; e += THREADS) s_off[e] = p.offsets[e];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_holder);
  constexpr int FT = ACT ? 64 : 128;           // outputs per tile
  const int ftiles = (p.F + FT - 1) / FT, ntiles = s_off[p.E] / SEG * ftiles, kbs = (p.K + BK - 1) / BK;

  if (warp == 0) {
    int s = 0, fills = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
      const Tile t = tile_at(s_off, p, tile, ftiles);
      const int w0 = t.expert * p.N + t.f * FT, w1 = ACT ? w0 + p.F : w0 + 64;
      for (int kb = 0; kb < kbs; ++kb) {
        ok = mbar_wait_warp(&empty[s], ph ^ 1, p.err, ERR_WAIT_EMPTY);
        if (!ok) break;
        if (lane == 0) {
          uint8_t* sa = smem + s * STAGE_BYTES;
          mbar_expect_tx(&full[s], STAGE_BYTES);
          tma_load_2d(sa, &tmW, &full[s], kb * BK, w0);
          tma_load_2d(sa + A_BYTES / 2, &tmW, &full[s], kb * BK, w1);
          tma_load_2d(sa + A_BYTES, &tmX, &full[s], kb * BK, t.row0);
        }
        __syncwarp();
        ++fills;
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    for (int j = fills > STAGES ? fills - STAGES : 0; j < fills; ++j) mbar_land(&full[j % STAGES], (j / STAGES) & 1);
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc(BM, SEG, 1, 1, 0, 0);
    int s = 0, n = 0, used = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++n) {
      const int acc = n & 1;
      ok = mbar_wait_warp(&tempty[acc], ((n >> 1) & 1) ^ 1, p.err, ERR_WAIT_TMEM_EMPTY);
      if (!ok) break;
      tc_fence_after();
      for (int kb = 0; kb < kbs; ++kb) {
        ok = mbar_wait_warp(&full[s], ph, p.err, ERR_WAIT_FULL);
        if (!ok) break;
        tc_fence_after();
        if (lane == 0) {
          const uint32_t a = smem_u32(smem + s * STAGE_BYTES), b = a + A_BYTES;
#pragma unroll
          for (int k4 = 0; k4 < BK / UMMA_K; ++k4)
            umma_f16(tmem_base + acc * SEG, make_smem_desc_sw128(a + k4 * (UMMA_K * 2), 16, 1024),
                     make_smem_desc_sw128(b + k4 * (UMMA_K * 2), 16, 1024), idesc, (kb > 0 || k4 > 0) ? 1u : 0u);
          umma_commit(&empty[s]);
          if (kb == kbs - 1) umma_commit(&tfull[acc]);
        }
        __syncwarp();
        ++used;
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    if (used) mbar_land(&empty[(used - 1) % STAGES], ((used - 1) / STAGES) & 1);   // the last products, and all before
  } else {
    const int quad = warp & 3, row = quad * 32 + lane;    // weight row inside the tile = TMEM lane
    int n = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++n) {
      const Tile t = tile_at(s_off, p, tile, ftiles);
      const int acc = n & 1;
      ok = mbar_wait_warp(&tfull[acc], (n >> 1) & 1, p.err, ERR_WAIT_TMEM_FULL);
      if (ACT) ok = all_epilogue_warps(ok);   // the four warps meet at barriers: they leave the loop together
      if (!ok) break;
      tc_fence_after();
      uint32_t r[16];
      tmem_ld16(tmem_base + acc * SEG + (static_cast<uint32_t>(quad * 32) << 16), r);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(&tempty[acc]);
      __nv_bfloat16* y = p.Y + static_cast<long long>(t.row0) * p.ldy;
      if (ACT) {
        if (row >= 64) {
#pragma unroll
          for (int j = 0; j < SEG; ++j) s_up[(row - 64) * UP_LD + j] = __uint_as_float(r[j]);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const int feat = t.f * 64 + row;
        if (row < 64 && feat < p.F) {
#pragma unroll
          for (int j = 0; j < SEG; ++j) {
            if (j < t.valid) {
              const float g = __uint_as_float(r[j]);
              y[j * p.ldy + feat] = __float2bfloat16(g / (1.f + __expf(-g)) * s_up[row * UP_LD + j]);
            }
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");   // the exchange buffer may be written again
      } else {
        const int feat = t.f * 128 + row;
        if (feat < p.F) {
#pragma unroll
          for (int j = 0; j < SEG; ++j)
            if (j < t.valid) y[j * p.ldy + feat] = __float2bfloat16(__uint_as_float(r[j]));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem_base, 32); }
}

}  // namespace gkmd

using namespace gkmd;

// W [E, N, K] and X [rows, K] bf16 row-major, 16-byte aligned, K a multiple of 8; segments of 16 rows (offsets, counts on the
// device).  act: silu(gate) * up of N = 2 F rows, F a multiple of 64.  Y [rows, F].
GK_EXPORT int gk_moe_decode(const void* W, const void* X, void* Y, const int* offsets, const int* counts, int rows, int E,
                            int N, int K, int act, int* err, void* stream) {
  if (E < 1 || E > MAX_EXPERTS || rows < 1 || rows % SEG || N < 1 || K < 8 || K % 8) return -1;
  if (act && N % 128) return -2;
  if ((reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(X) & 15)) return -3;
  if (static_cast<long long>(E) * N > 0x7fffffff) return -2;
  CUtensorMap tmW, tmX;
  if (make_tmap_2d(&tmW, W, 2, static_cast<uint64_t>(E) * N, K, K, 64, BK, true)) return -4;
  if (make_tmap_2d(&tmX, X, 2, rows, K, K, SEG, BK, true)) return -5;
  Params p;
  p.offsets = offsets; p.counts = counts; p.Y = static_cast<__nv_bfloat16*>(Y);
  p.F = act ? N / 2 : N; p.ldy = p.F;
  p.E = E; p.N = N; p.K = K; p.err = err;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(moe_decode_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(moe_decode_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess)
      return -6;
    configured = true;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const dim3 grid(sm_count()), block(THREADS);
  if (act) launch_k(moe_decode_kernel<true>, grid, block, SMEM_BYTES, st, tmW, tmX, p);
  else launch_k(moe_decode_kernel<false>, grid, block, SMEM_BYTES, st, tmW, tmX, p);
  return launch_status();
}
