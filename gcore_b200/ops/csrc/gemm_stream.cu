// Decode-shaped GEMM: y[T, N] = x[T, K] . W[N, K]^T (+ bias) for T <= 128 tokens.  The weight is the only operand of any
// size; what bounds the kernel is HBM, and beside it the fixed cost of a launch in a chain of short dependent kernels.
//
//   * swap-AB: the 128-row tcgen05 tile runs over output features, the token count is the MMA N (16 .. 128).
//   * Few feature tiles (up to half the SMs): every tile is cut along K into as many equal pieces as there are SMs per
//     tile, one piece per CTA.  The pieces of a tile lie in fp32 in a scratch buffer (they stay in L2); each of its CTAs
//     waits for the others' and adds its share of the tile.  The CTAs of a grid usually run at the same time, one per SM
//     at most, and wait a microsecond or two; one that waits long (kernels of other streams hold the SMs) leaves its
//     share to the CTA that brings the last piece, so that nothing depends on all of them being resident.
//   * More tiles: the sequence of (tile, 64-deep k-block) units, tile after tile, is cut into one contiguous run per SM, so
//     that 192 or 296 tiles stream as evenly as a multiple of 148; the CTA that brings a divided tile's last piece adds
//     them up.  (Waiting for the others would cost: a run's first piece belongs to a tile that its neighbour ends with.)
//   * Runs are cut between tiles only where what this leaves idle costs less than adding up the pieces (short K, many tokens).
//   Always the pieces are added in the order of K, so results do not depend on timing.
//   * The weight does not depend on the kernel in front: with programmatic dependent launch the ring's first loads are
//     under way while that kernel still runs.
//
// Roles per CTA: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 epilogue (two per TMEM lane quarter, half of the token
// columns each).  Two accumulators: a piece is drained while the next one is contracted.
#include "ptx.cuh"
#include "host_utils.h"

namespace gkst {
using namespace gk;

constexpr int BM = 128, BK = 64, UMMA_K = 16;
constexpr int EPI_WARPS = 8, EPI_THREADS = EPI_WARPS * 32;
constexpr int THREADS = 64 + EPI_THREADS;
constexpr int MAX_STAGES = 8;
constexpr int A_BYTES = BM * BK * 2;
constexpr int COLS = 8;         // token columns a thread reads from tensor memory at a time

struct StParams {
  int T, Tp, N, K, kbs, units, stages;
  int ks;          // pieces of a tile, one per CTA; 0: contiguous runs
  int tiles;       // > 0: runs are cut between tiles only
  void* Y;
  long long ldy;
  int out_fp32;
  const void* bias;
  int bias_fp32;
  float* ws;       // [CTA][first, last piece][Tp tokens][128 features]
  unsigned long long* counters;   // [tiles]: pieces there | CTAs done << 8 | shares left over << 16, zero between launches
  int share_wait;  // cycles a CTA waits for the others' pieces before it leaves its share of the tile to the last one
  int* err;
};

// CTA c works on units [first_unit(c), first_unit(c + 1))
__device__ __forceinline__ int first_unit(const StParams& p, int c, int ctas) {
  if (p.ks) {
    const int tile = c / p.ks;
    return tile * p.kbs + p.kbs * (c - tile * p.ks) / p.ks;
  }
  if (p.tiles) return static_cast<int>(static_cast<long long>(p.tiles) * c / ctas) * p.kbs;
  return static_cast<int>(static_cast<long long>(p.units) * c / ctas);
}
// the CTAs [lo, hi] that hold pieces of a tile
__device__ __forceinline__ void tile_owners(const StParams& p, int tile, int ctas, int& lo, int& hi) {
  if (p.ks) {
    lo = tile * p.ks;
    hi = lo + p.ks - 1;
  } else {
    lo = static_cast<int>((static_cast<long long>(tile * p.kbs + 1) * ctas - 1) / p.units);
    hi = static_cast<int>((static_cast<long long>((tile + 1) * p.kbs) * ctas - 1) / p.units);
  }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void store_cols(const StParams& p, const float (&v)[COLS], int tok0, int feat) {
  if (feat >= p.N) return;
#pragma unroll
  for (int j = 0; j < COLS; ++j) {
    if (tok0 + j < p.T) {
      const long long at = (tok0 + j) * p.ldy + feat;
      if (p.out_fp32) static_cast<float*>(p.Y)[at] = v[j];
      else static_cast<__nv_bfloat16*>(p.Y)[at] = __float2bfloat16(v[j]);
    }
  }
}

__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long* a) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(a) : "memory");
  return v;
}
constexpr int MAX_PIECES = 48;             // shares of a tile the counter word has a bit for
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Adds up items [i0, i1) of a divided tile, an item being four features of one token.
__device__ __forceinline__ void sum_pieces(const StParams& p, int tile, int lo, int hi, int i0, int i1) {
  for (int i = i0 + static_cast<int>(threadIdx.x) - 64; i < i1; i += EPI_THREADS) {
    const int tok = i >> 5, f4 = (i & 31) * 4, feat = tile * BM + f4;
    const float* src = p.ws + (tok * BM + f4);
    const long long piece = static_cast<long long>(p.Tp) * BM;
    // only the first CTA's piece starts the tile
    float4 v = __ldcg(reinterpret_cast<const float4*>(src + (lo * 2ll + 1) * piece));
    for (int o = lo + 1; o <= hi; o += 6) {
      float4 q[6];
#pragma unroll
      for (int j = 0; j < 6; ++j)
        q[j] = o + j <= hi ? __ldcg(reinterpret_cast<const float4*>(src + (o + j) * 2ll * piece)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 6; ++j) v = add4(v, q[j]);
    }
    const float r[4] = {v.x, v.y, v.z, v.w};
    const long long at = tok * p.ldy + feat;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (feat + e >= p.N) break;
      float b = 0.f;
      if (p.bias)
        b = p.bias_fp32 ? static_cast<const float*>(p.bias)[feat + e]
                        : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[feat + e]);
      if (p.out_fp32) static_cast<float*>(p.Y)[at + e] = r[e] + b;
      else static_cast<__nv_bfloat16*>(p.Y)[at + e] = __float2bfloat16(r[e] + b);
    }
  }
}

// The epilogue warps meet at barriers behind a divided tile: where one of them has given up on a wait, all leave together.
__device__ __forceinline__ bool all_epilogue_warps(bool ok) {
  uint32_t all;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "barrier.red.and.pred q, 1, %2, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(all)
      : "r"(static_cast<uint32_t>(ok)), "n"(EPI_THREADS)
      : "memory");
  return all != 0;
}

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }

// What follows when this CTA's piece of a divided tile lies in the scratch.
__device__ __forceinline__ void finish_piece(const StParams& p, int tile, int ctas, unsigned long long* s_word) {
  int lo, hi;
  tile_owners(p, tile, ctas, lo, hi);
  const int pieces = hi - lo + 1, items = 32 * p.T;
  unsigned long long* word = &p.counters[tile];
  __threadfence();
  epi_sync();
  if (p.ks) {
    const int mine = static_cast<int>(blockIdx.x) - lo;
    if (threadIdx.x == 64) {
      unsigned long long shares = 1ull << mine;     // what this CTA adds up
      const unsigned long long old = atomicAdd(word, 1ull);
      if (static_cast<int>(old & 0xff) == pieces - 1) {
        shares |= old >> 16;
      } else {
        const long long t0 = clock64();
        while (static_cast<int>(load_acquire(word) & 0xff) < pieces) {
          if (clock64() - t0 < p.share_wait) continue;
          // the CTA that brings the last piece sees the bit, unless it came first: then all pieces are there
          if (static_cast<int>(atomicOr(word, shares << 16) & 0xff) < pieces) shares = 0;
          break;
        }
      }
      __threadfence();
      *s_word = shares;
    }
    epi_sync();
    for (unsigned long long shares = *s_word; shares; shares &= shares - 1) {
      const int k = __ffsll(shares) - 1;
      sum_pieces(p, tile, lo, hi, items * k / pieces, items * (k + 1) / pieces);
    }
    // the last CTA to be done leaves the word at zero for the next launch
    if (threadIdx.x == 64 && static_cast<int>((atomicAdd(word, 256ull) >> 8) & 0xff) == pieces - 1) *word = 0;
  } else {
    if (threadIdx.x == 64) {
      *s_word = static_cast<int>(atomicAdd(word, 1ull)) == pieces - 1;
      __threadfence();
    }
    epi_sync();
    if (*s_word) {
      sum_pieces(p, tile, lo, hi, 0, items);
      if (threadIdx.x == 64) *word = 0;
    }
    epi_sync();   // the flag may be written again
  }
}

__global__ void __launch_bounds__(THREADS, 2)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, StParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = A_BYTES + p.Tp * 128;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* tfull = empty + MAX_STAGES;   // 2
  uint64_t* tempty = tfull + 2;           // 2
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tempty + 2);
  unsigned long long* s_word = reinterpret_cast<unsigned long long*>(tmem_holder + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ctas = gridDim.x;
  const int u0 = first_unit(p, blockIdx.x, ctas), u1 = first_unit(p, blockIdx.x + 1, ctas);
  uint32_t tmem_cols = 32;
  while (tmem_cols < 2u * p.Tp) tmem_cols <<= 1;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], EPI_THREADS); }
    fence_barrier_init();
    const int pre = u1 - u0 < p.stages ? u1 - u0 : p.stages;
    for (int i = 0; i < pre; ++i) {
      const int tile = (u0 + i) / p.kbs, kb = (u0 + i) - tile * p.kbs;
      mbar_expect_tx(&full[i], stage_bytes);
      tma_load_2d(smem + i * stage_bytes, &tmW, &full[i], kb * BK, tile * BM);
    }
  }
  if (warp == 2) { tmem_alloc(tmem_holder, tmem_cols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_holder);
  pdl_wait();   // the activations, and what the epilogue writes

  if (warp == 0) {
    const int pre = u1 - u0 < p.stages ? u1 - u0 : p.stages;
    int tile = u0 / p.kbs, kb = u0 - tile * p.kbs;
    int s = 0, i = 0;
    uint32_t ph = 0;
    for (; i < u1 - u0; ++i) {
      if (i >= pre && !mbar_wait_warp(&empty[s], ph ^ 1, p.err, ERR_WAIT_EMPTY)) break;
      if (lane == 0) {
        uint8_t* sa = smem + s * stage_bytes;
        if (i >= pre) {
          mbar_expect_tx(&full[s], stage_bytes);
          tma_load_2d(sa, &tmW, &full[s], kb * BK, tile * BM);
        }
        tma_load_2d(sa + A_BYTES, &tmX, &full[s], kb * BK, 0);
      }
      __syncwarp();
      if (++kb == p.kbs) { kb = 0; ++tile; }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    for (int j = i > p.stages ? i - p.stages : 0; j < i; ++j) mbar_land(&full[j % p.stages], (j / p.stages) & 1);
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc(BM, p.Tp, 1, 1, 0, 0);
    int s = 0, piece = 0, kb = u0 % p.kbs, u = u0;
    uint32_t ph = 0;
    bool fresh = true;
    for (; u < u1; ++u) {
      const int acc = piece & 1;
      if (fresh && !mbar_wait_warp(&tempty[acc], ((piece >> 1) & 1) ^ 1, p.err, ERR_WAIT_TMEM_EMPTY)) break;
      if (!mbar_wait_warp(&full[s], ph, p.err, ERR_WAIT_FULL)) break;
      tc_fence_after();
      const bool ends = kb == p.kbs - 1 || u == u1 - 1;
      if (lane == 0) {
        const uint32_t a_base = smem_u32(smem + s * stage_bytes), b_base = a_base + A_BYTES;
#pragma unroll
        for (int k4 = 0; k4 < BK / UMMA_K; ++k4) {
          umma_f16(tmem_base + acc * p.Tp, make_smem_desc_sw128(a_base + k4 * (UMMA_K * 2), 16, 1024),
                   make_smem_desc_sw128(b_base + k4 * (UMMA_K * 2), 16, 1024), idesc, (!fresh || k4 > 0) ? 1u : 0u);
        }
        umma_commit(&empty[s]);
        if (ends) umma_commit(&tfull[acc]);
      }
      __syncwarp();
      fresh = ends;
      if (ends) ++piece;
      if (++kb == p.kbs) kb = 0;
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    const int last = u - u0 - 1;   // the products of the last k-block, and with them all before
    if (last >= 0) mbar_land(&empty[last % p.stages], (last / p.stages) & 1);
  } else {
    const int quad = warp & 3;
    const int row = quad * 32 + lane;                // output feature inside the tile = TMEM lane
    const int half = (warp - 2) >> 2;                // which token columns
    const int c0 = half * (p.Tp / 2), c1 = c0 + p.Tp / 2;
    int piece = 0;
    for (int u = u0; u < u1; ++piece) {
      const int tile = u / p.kbs, kb0 = u - tile * p.kbs;
      const int next = (tile + 1) * p.kbs < u1 ? (tile + 1) * p.kbs : u1;
      const bool whole = kb0 == 0 && next - u == p.kbs;
      const int acc = piece & 1, feat = tile * BM + row;
      if (!all_epilogue_warps(mbar_wait(&tfull[acc], (piece >> 1) & 1, p.err, ERR_WAIT_TMEM_FULL))) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * p.Tp + (static_cast<uint32_t>(quad * 32) << 16);
      float bias = 0.f;
      if (p.bias && feat < p.N)
        bias = p.bias_fp32 ? static_cast<const float*>(p.bias)[feat]
                           : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[feat]);
      // a CTA's piece that starts inside a tile lies in the first half of its scratch, one that starts a tile in the second
      float* part = p.ws + (blockIdx.x * 2ll + (kb0 == 0)) * (p.Tp * BM) + row;
      for (int c = c0; c < c1 && c < p.T; c += COLS) {
        uint32_t r[COLS];
        tmem_ld8(taddr + c, r);
        tmem_ld_wait();
        if (whole) {
          float v[COLS];
#pragma unroll
          for (int j = 0; j < COLS; ++j) v[j] = __uint_as_float(r[j]) + bias;
          store_cols(p, v, c, feat);
        } else {
#pragma unroll
          for (int j = 0; j < COLS; ++j)
            if (c + j < p.T) __stcg(part + (c + j) * BM, __uint_as_float(r[j]));
        }
      }
      tc_fence_before();
      mbar_arrive(&tempty[acc]);
      if (!whole) finish_piece(p, tile, ctas, s_word);
      u = next;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem_base, tmem_cols); }
}

// Token columns of the accumulators: a multiple of 16 (one half per epilogue warp of a lane quarter, 8 columns at a time).
static int padded_tokens(int T) { return (T + 15) / 16 * 16; }

}  // namespace gkst

using namespace gkst;

// Id of the capture that a stream takes part in, 0 outside of one (or where it cannot be told).
GK_EXPORT unsigned long long gk_capture_id(void* stream) {
  cudaStreamCaptureStatus status;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(reinterpret_cast<cudaStream_t>(stream), &status, &id) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return status == cudaStreamCaptureStatusActive ? id : 0;
}

// Floats of scratch for the pieces of divided tiles.
GK_EXPORT long long gk_gemm_stream_scratch(int T) { return 2ll * sm_count() * padded_tokens(T) * BM; }

// W [N, K] and X [T, K] bf16 row-major (K contiguous, leading dimensions multiples of 8, 16-byte aligned), 1 <= T <= 128.
// counters: two zero ints per 128 features, 8-byte aligned; a launch leaves them at zero, and launches that may run at the
// same time must not share them.  share_wait: cycles a CTA waits for the other pieces of its tile (results do not depend on it).
GK_EXPORT int gk_gemm_stream(const void* W, long long ldw, const void* X, long long ldx, void* Y, long long ldy,
                             int out_fp32, const void* bias, int bias_fp32, int T, int N, int K, float* ws,
                             long long ws_floats, int* counters, long long counter_ints, int share_wait, int* err,
                             void* stream) {
  if (T < 1 || T > 128 || N < 1 || K < 1) return -1;
  if ((ldw & 7) || (ldx & 7) || (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(X) & 15)) return -3;
  StParams p;
  p.T = T; p.Tp = padded_tokens(T); p.N = N; p.K = K;
  const int tiles = (N + BM - 1) / BM;
  p.kbs = (K + BK - 1) / BK;
  if (static_cast<long long>(tiles) * p.kbs > 0x3fffffff) return -2;
  p.units = tiles * p.kbs;
  if (ws_floats < gk_gemm_stream_scratch(T)) return -8;
  if (!counters || counter_ints < 2ll * tiles || (reinterpret_cast<uintptr_t>(counters) & 7)) return -9;
  CUtensorMap tmW, tmX;
  if (make_tmap_2d(&tmW, W, 2, N, K, ldw, BM, BK, true)) return -4;
  if (make_tmap_2d(&tmX, X, 2, T, K, ldx, p.Tp, BK, true)) return -5;
  p.Y = Y; p.ldy = ldy; p.out_fp32 = out_fp32; p.bias = bias; p.bias_fp32 = bias_fp32;
  p.ws = ws; p.counters = reinterpret_cast<unsigned long long*>(counters);
  p.share_wait = share_wait; p.err = err;
  const int sms = sm_count(), stage_bytes = A_BYTES + p.Tp * 128;
  const double weight_us = 2e-6 * N * K / 6.5;   // time the weight takes from HBM
  // Ring: below half of an SM the next GEMM's CTA fits beside this one and has its first loads under way early; that pays
  // while the launch is short (4608 x 3584, 4 tokens: 10.6 against 10.9 us).  Long launches want more in flight than
  // two half rings bring (152064 x 3584, 4 tokens: 173 against 182 us; 37888 x 3584: 45.5 against 47.5 us).
  const int budget = weight_us < 8. ? 104 * 1024 : 200 * 1024;
  p.stages = (budget - 1024 - 256) / stage_bytes;
  if (p.stages < 3) p.stages = 3;
  if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
  // Cuts (measured, us, 4 / 64 tokens).  One piece per CTA where that occupies most SMs: 3584 x 18944 28 / 31 against 28 / 37
  // in runs, 4096 x 14336 26 / 29 against 25 / 33; 7168 x 18432 would leave a quarter of them idle: 57 / 62 against 48 / 58.
  p.ks = p.tiles = 0;
  int grid = p.units < sms ? p.units : sms;
  if (2 * tiles <= sms) {
    int ks = sms / tiles;
    const int most = p.kbs / 3 > 1 ? p.kbs / 3 : 1;   // at least three k-blocks per piece
    const bool full = tiles * ks * 5 >= sms * 4;
    if (ks > most) ks = most;
    if (ks > MAX_PIECES) ks = MAX_PIECES;
    if (full || ks == most || ks == MAX_PIECES || T > 64) { p.ks = ks; grid = tiles * ks; }
  }
  // Adding up divided tiles costs about 1.5 us and 0.1 us per token, with fewer tiles than SMs (where hardly one is whole) 4 us
  // and 0.14; whole tiles leave SMs idle in the last round (runs / whole, us: 32768 x 1024, 64 tokens 22.6 / 18.2; 28672 x 4096,
  // 4 tokens 42 / 52; 10240 x 1024, 4 and 64 tokens 12.5 / 10.7 and 22 / 11.9; 9728 x 5120 24 / 34 and 33 / 36).
  if (!p.ks && 2 * tiles > sms) {
    const double rounds = (tiles + sms - 1) / sms, idle_us = (rounds * sms / tiles - 1.) * weight_us;
    if (idle_us < (tiles < sms ? 4. + 0.14 * T : 1.5 + 0.1 * T)) {
      p.tiles = tiles;
      grid = tiles < sms ? tiles : sms;
    }
  }
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
      return -6;
    cudaFuncSetAttribute(gemm_stream_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    configured = true;
  }
  launch_k(gemm_stream_kernel, dim3(grid), dim3(THREADS), p.stages * stage_bytes + 1024 + 256,
           reinterpret_cast<cudaStream_t>(stream), tmW, tmX, p);
  return launch_status();
}
