// Block-scaled e4m3 linear layer for sm_100a.
//
//   C[m, n] = sum_kb  sa[kb, m] * sb[n / 128, kb] * ( A8[m, kb-block] . B8[n, kb-block] )
//
// A8 [M, K] carries one fp32 scale per row and 128-wide K block ("1 x 128",
// activations / output gradients), B8 [N, K] one per 128 x 128 block (weights).
// Each K block is a separate tcgen05.mma chain (kind::f8f6f4, 4 issues of K=32)
// into its own 128-column TMEM accumulator; the epilogue warps multiply that
// partial product by the two block scales while adding it into fp32 registers,
// so the scales never touch the tensor-core path and a 4-deep ring of TMEM
// accumulators lets the MMAs of block kb+1..kb+3 run under the scaling of kb.
//
// The quantisers produce exactly the operand layouts the GEMM consumes:
//   rows:   bf16 [R, K] -> e4m3 [R, K] + scales [K/128, R]  (optionally the
//           RMSNorm of the row: the cast is fused into the norm that produces
//           the linear's input, the row never round-trips through bf16)
//   blocks: bf16 [N, K] -> e4m3 [N, K] and its transpose [K, N] + scales [N/128, K/128]
//
// The reference's fp8 path is per-tensor scaling around cuBLASLt
// (src/chaoscontrol/kernels/fp8_linear.py:171-265,
//  kernels/_cublaslt/src/cublaslt_fp8_matmul.cpp:281-291); this is the
// finer-grained replacement.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "ccb_api.h"
#include "ptx.cuh"
#include "runtime.h"

namespace ccb {

constexpr float E4M3_MAX = 448.f;

__device__ __forceinline__ uint16_t e4m3x2(float a, float b) {
  return (uint16_t)__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
}

// ---------------------------------------------------------------------------
// Row quantiser (1 x 128 scales), optionally fused with RMSNorm.
// A row is held in registers by one warp (half a warp at K = 128): a lane owns 8 contiguous elements of
// each 8 * LPR-column segment, so a 128-column block is 16 lanes and its amax is 4 shuffles.  Bound by
// HBM; the segment count is a template argument, because a kernel written for the widest row spends its
// registers and its issue slots on segments that are not there: 65 536 rows, K = 256 and K = 1024
// together 107 us with eight segments, 54 with 1 and 4 (4.7 TB/s).
// ---------------------------------------------------------------------------
constexpr int QR_MAXSEG = 8;   // K <= 2048

template <int LPR, int NSEG>
__global__ void __launch_bounds__(256)
fp8_quant_rows_kernel(const __nv_bfloat16* __restrict__ x, long long ldx,
                      const __nv_bfloat16* __restrict__ norm_w, float eps,
                      uint8_t* __restrict__ q, float* __restrict__ s_t, float* __restrict__ inv_rms_out,
                      __nv_bfloat16* __restrict__ y_out, int R, int K) {
  constexpr int RPW = 32 / LPR, SEG = 8 * LPR;
  const int lane = threadIdx.x % LPR;
  const int row = (blockIdx.x * 8 + (threadIdx.x >> 5)) * RPW + (threadIdx.x & 31) / LPR;
  const bool on = row < R;                 // no early exit: the shuffles take the whole warp
  uint4 raw[NSEG];
#pragma unroll
  for (int sgm = 0; sgm < NSEG; ++sgm) {
    const int c = sgm * SEG + lane * 8;
    raw[sgm] = (on && c < K) ? __ldg(reinterpret_cast<const uint4*>(x + (long long)row * ldx + c)) : make_uint4(0u, 0u, 0u, 0u);
  }
  auto unpack = [](const uint4& u, float (&f)[8]) {
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
  };
  float inv_rms = 1.f;
  if (norm_w != nullptr) {
    float ss = 0.f;
#pragma unroll
    for (int sgm = 0; sgm < NSEG; ++sgm) {
      float v[8];
      unpack(raw[sgm], v);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    inv_rms = rsqrtf(ss / (float)K + eps);
    if (on && lane == 0 && inv_rms_out != nullptr) inv_rms_out[row] = inv_rms;
  }
#pragma unroll
  for (int sgm = 0; sgm < NSEG; ++sgm) {
    const int c = sgm * SEG + lane * 8;
    float v[8];
    unpack(raw[sgm], v);
    if (norm_w != nullptr && c < K) {
      float wv[8];
      unpack(__ldg(reinterpret_cast<const uint4*>(norm_w + c)), wv);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = v[i] * inv_rms * wv[i];
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    // 16 lanes = one 128-column block
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (on && c < K) {
      const float scale = fmaxf(amax, 1e-12f) * (1.f / E4M3_MAX);
      const float inv = 1.f / scale;
      uint2 o;
      o.x = (uint32_t)e4m3x2(v[0] * inv, v[1] * inv) | ((uint32_t)e4m3x2(v[2] * inv, v[3] * inv) << 16);
      o.y = (uint32_t)e4m3x2(v[4] * inv, v[5] * inv) | ((uint32_t)e4m3x2(v[6] * inv, v[7] * inv) << 16);
      *reinterpret_cast<uint2*>(q + (long long)row * K + c) = o;
      if ((lane & 15) == 0) s_t[(long long)(c >> 7) * R + row] = scale;
      if (y_out != nullptr) {
        uint4 yo;
        yo.x = pack_bf16x2(v[0], v[1]); yo.y = pack_bf16x2(v[2], v[3]);
        yo.z = pack_bf16x2(v[4], v[5]); yo.w = pack_bf16x2(v[6], v[7]);
        *reinterpret_cast<uint4*>(y_out + (long long)row * K + c) = yo;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Weight quantiser (128 x 128 scales): one CTA per block, writes W8 and W8^T.
// A weight is a handful of blocks on 148 SMs, so the time is one block's latency: VEC (sizes in eights,
// 16-byte aligned) takes 16 elements a thread in two 16-byte loads and writes 8 codes at a time, instead of
// 64 two-byte trips a thread (1024 x 256: 15.6 us before, 4.6 now).  The transposed half reads the tile's
// columns from shared memory; a row stride of 130 elements keeps those reads free of bank conflicts.
// ---------------------------------------------------------------------------
template <bool VEC>
__global__ void __launch_bounds__(1024)
fp8_quant_blocks_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q,
                        uint8_t* __restrict__ qt, float* __restrict__ s, int N, int K) {
  __shared__ __nv_bfloat16 tile[128][130];
  __shared__ float wmax[32];
  const int n0 = blockIdx.y * 128, k0 = blockIdx.x * 128;
  constexpr int STEP = VEC ? 8 : 1;                       // elements of a row a thread takes at once
  constexpr int COLS = 128 / STEP, ROWS = 1024 / COLS;    // threads along and down the tile
  const int tx = threadIdx.x % COLS * STEP, ty = threadIdx.x / COLS;
  uint4 raw[VEC ? 128 / ROWS : 1];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 128 / ROWS; ++j) {
    const int i = ty + j * ROWS, n = n0 + i, k = k0 + tx;
    if constexpr (VEC) {
      raw[j] = (n < N && k < K) ? __ldg(reinterpret_cast<const uint4*>(w + (long long)n * K + k)) : make_uint4(0u, 0u, 0u, 0u);
    } else {
      __nv_bfloat16 v = __float2bfloat16(0.f);
      if (n < N && k < K) v = w[(long long)n * K + k];
      tile[i][tx] = v;
      amax = fmaxf(amax, fabsf(__bfloat162float(v)));
    }
  }
  if constexpr (VEC) {
#pragma unroll
    for (int j = 0; j < 128 / ROWS; ++j) {
      uint32_t* t = reinterpret_cast<uint32_t*>(&tile[ty + j * ROWS][tx]);
      const uint32_t r[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        t[e] = r[e];
        const float2 f = unpack_bf16x2(r[e]);
        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = wmax[0];
#pragma unroll
  for (int i = 1; i < 32; ++i) amax = fmaxf(amax, wmax[i]);
  const float scale = fmaxf(amax, 1e-12f) * (1.f / E4M3_MAX);
  const float inv = 1.f / scale;
  if (threadIdx.x == 0) s[(long long)blockIdx.y * gridDim.x + blockIdx.x] = scale;
  // codes of STEP elements (ROW: along the row, else down the column) of the tile -> 8 bytes or 1
  auto put = [&](uint8_t* dst, int i, int c, bool row) {
    float f[STEP];
#pragma unroll
    for (int e = 0; e < STEP; ++e) f[e] = __bfloat162float(row ? tile[i][c + e] : tile[c + e][i]) * inv;
    if constexpr (VEC) {
      uint2 o;
      o.x = (uint32_t)e4m3x2(f[0], f[1]) | ((uint32_t)e4m3x2(f[2], f[3]) << 16);
      o.y = (uint32_t)e4m3x2(f[4], f[5]) | ((uint32_t)e4m3x2(f[6], f[7]) << 16);
      *reinterpret_cast<uint2*>(dst) = o;
    } else {
      *dst = (uint8_t)__nv_cvt_float_to_fp8(f[0], __NV_SATFINITE, __NV_E4M3);
    }
  };
#pragma unroll
  for (int j = 0; j < 128 / ROWS; ++j) {
    const int i = ty + j * ROWS;
    if (n0 + i < N && k0 + tx < K) put(q + (long long)(n0 + i) * K + k0 + tx, i, tx, true);
    if (qt != nullptr && k0 + i < K && n0 + tx < N) put(qt + (long long)(k0 + i) * N + n0 + tx, i, tx, false);
  }
}

// ---------------------------------------------------------------------------
// Block-scaled GEMM
// ---------------------------------------------------------------------------
constexpr int FB_BM = 128, FB_BN = 128, FB_BK = 128;        // one-byte elements: 128 per swizzle row
constexpr int FB_STAGE = FB_BM * FB_BK;                      // 16 KiB per operand tile
constexpr int FB_SLOTS = 4;                                  // TMEM accumulator ring (4 x 128 columns)
constexpr int FB_EPI_WARPS = 8;
constexpr int FB_THREADS = 64 + 32 * FB_EPI_WARPS;
// bf16 results leave through shared memory and TMA stores: each epilogue warp stages its 32 rows x 64 columns
// (128-byte rows, swizzled).  Storing them from registers, a row to a lane, cost 32 half-used sectors an
// instruction: 65 536 x 256 x 1024 and its input gradient took 116 us, staged 101.
constexpr int FB_STG = 32 * 128;
// RES: the weight tiles of a CTA's columns stay in shared memory (up to 128 KiB) while it walks the rows, and only
// activations stream, a k-block to a stage; a row block's stages serve all of the CTA's column tiles.  With both
// operands streaming, every 128 x 128 tile drags 2 x 128 x K bytes through the L2 -> SM path.  Events, cold L2,
// streaming / resident in us at 65 536 rows: K x N = 256 x 1024 55 / 46, 512 x 1024 89 / 73, 384 x 640 50 / 46,
// 1024 x 1024 155 / 146, 1024 x 256 50 / 46.
template <int RES>
struct FbCfg {
  static constexpr int STAGES = RES ? 4 : 5;
  static constexpr int RES_TILES = RES ? 8 : 0;              // 16 KiB weight tiles kept
  static constexpr int A_OFF = RES_TILES * FB_STAGE;
  static constexpr int STG_OFF = A_OFF + STAGES * (RES ? 1 : 2) * FB_STAGE;
  static constexpr int BAR_OFF = STG_OFF + FB_EPI_WARPS * FB_STG;
  static constexpr int SMEM = 1024 + BAR_OFF + 512;
  static_assert(SMEM <= 227 * 1024, "exceeds the per-CTA shared memory limit");
};

struct FbArgs {
  int M, N, K, kblocks, tiles_m, tiles_n;
  int nt, groups;           // RES: column tiles of a CTA, groups of CTAs that split the columns
  const float* sa_t;        // [K/128, M]
  const float* sb;          // scale of (output column block j, k block kb) at sb[j * sb_so + kb * sb_sk]
  long long sb_so, sb_sk;
  void* C;
  long long ldc;
  int out_fp32, tma_store;
  const __nv_bfloat16* bias;
  int* status;
};

// Work of a CTA: row blocks w, w + nw, ... and, in each, column tiles [nt0, nt1); without RES one tile at a time.
struct FbWalk {
  int unit, step, units, nt0, nt1;
};
template <int RES>
__device__ __forceinline__ FbWalk fb_walk(const FbArgs& p) {
  FbWalk w;
  if (RES) {
    const int g = (int)blockIdx.x % p.groups;
    w.unit = (int)blockIdx.x / p.groups;
    w.step = (int)gridDim.x / p.groups;
    w.units = p.tiles_m;
    w.nt0 = g * p.nt;
    w.nt1 = min(p.tiles_n, w.nt0 + p.nt);
  } else {
    w.unit = blockIdx.x;
    w.step = gridDim.x;
    w.units = p.tiles_m * p.tiles_n;
    w.nt0 = 0;
    w.nt1 = 1;
  }
  return w;
}

template <int RES>
__global__ void __launch_bounds__(FB_THREADS, 1)
fp8_block_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmC, const FbArgs p) {
  using Cfg = FbCfg<RES>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem + Cfg::A_OFF;
  uint8_t* sB = RES ? smem : smem + STAGES * FB_STAGE;      // RES: tile (nt, kb) at ((nt - nt0) * kblocks + kb)
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + FB_SLOTS;
  uint64_t* bres_bar = tempty_bar + FB_SLOTS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bres_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const FbWalk wk = fb_walk<RES>(p);

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    for (int i = 0; i < FB_SLOTS; ++i) { mbar_init(&tfull_bar[i], 1); mbar_init(&tempty_bar[i], FB_EPI_WARPS); }
    mbar_init(bres_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      if (RES && wk.unit < wk.units) {
        mbar_arrive_expect_tx(bres_bar, (uint32_t)((wk.nt1 - wk.nt0) * p.kblocks * FB_STAGE));
        for (int nt = wk.nt0; nt < wk.nt1; ++nt)
          for (int kb = 0; kb < p.kblocks; ++kb)
            tma_load_3d(sB + ((nt - wk.nt0) * p.kblocks + kb) * FB_STAGE, &tmB, bres_bar, kb * FB_BK, nt * FB_BN, 0);
      }
      for (int u = wk.unit; u < wk.units && ok; u += wk.step) {
        const int m0 = (RES ? u : u / p.tiles_n) * FB_BM, n0 = RES ? 0 : (u % p.tiles_n) * FB_BN;
        for (int kb = 0; kb < p.kblocks; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag, p.status)) { ok = false; break; }
          mbar_arrive_expect_tx(&full_bar[stage], (RES ? 1 : 2) * FB_STAGE);
          tma_load_3d(sA + stage * FB_STAGE, &tmA, &full_bar[stage], kb * FB_BK, m0, 0);
          if (!RES) tma_load_3d(sB + stage * FB_STAGE, &tmB, &full_bar[stage], kb * FB_BK, n0, 0);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        // aborting: bounded grace period for loads still in flight
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) { }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_f8(FB_BM, FB_BN, 0, 0);
      uint32_t n_slot = 0, n_ld = 0;
      bool ok = true;
      if (RES && wk.unit < wk.units) {
        ok = mbar_wait(bres_bar, 0u, abort_flag, p.status);
        tc_fence_after_sync();
      }
      for (int u = wk.unit; u < wk.units && ok; u += wk.step, n_ld += (uint32_t)p.kblocks) {
        for (int nt = wk.nt0; nt < wk.nt1 && ok; ++nt) {
          for (int kb = 0; kb < p.kblocks; ++kb, ++n_slot) {
            const int slot = n_slot % FB_SLOTS;
            const uint32_t sph = (n_slot / FB_SLOTS) & 1u;
            const uint32_t ld = n_ld + (uint32_t)kb;
            const int stage = (int)(ld % STAGES);
            if (!mbar_wait(&tempty_bar[slot], sph ^ 1u, abort_flag, p.status)) { ok = false; break; }
            // a row block's stages arrive once and serve every column tile (more than one only while all fit the ring)
            if (nt == wk.nt0 && !mbar_wait(&full_bar[stage], (ld / STAGES) & 1u, abort_flag, p.status)) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t a_base = smem_u32(sA + stage * FB_STAGE);
            const uint32_t b_base = smem_u32(sB + (RES ? (nt - wk.nt0) * p.kblocks + kb : stage) * FB_STAGE);
#pragma unroll
            for (int k = 0; k < FB_BK / 32; ++k) {
              const uint64_t adesc = make_smem_desc(a_base + k * 32, 16, 1024);
              const uint64_t bdesc = make_smem_desc(b_base + k * 32, 16, 1024);
              umma_f8(tmem_base + (uint32_t)(slot * FB_BN), adesc, bdesc, idesc, k > 0 ? 1u : 0u);
            }
            if (nt == wk.nt1 - 1) umma_commit(&empty_bar[stage]);
            umma_commit(&tfull_bar[slot]);
          }
        }
      }
    }
  } else {
    const int q = warp & 3;                    // TMEM lane quadrant
    const int part = (warp - 2) >> 2;          // columns [64 * part, 64 * part + 64) of the tile
    const int row_in_tile = q * 32 + lane;
    uint8_t* my_stage = smem + Cfg::STG_OFF + (warp - 2) * FB_STG;
    uint32_t n_slot = 0;
    bool ok = true;
    // The two block scales of a k-block do not depend on its accumulator: they are requested AHEAD k-blocks early,
    // across tiles.  Fetched as the k-block began, their L2 latency was the k-block's time: 1470 cycles against 256
    // of tensor work (streaming, 65 536 rows: 256 x 1024 66 us -> 55, 1024 x 1024 171 -> 155).
    constexpr int AHEAD = 3;
    float sca[AHEAD], scb[AHEAD];
    int fu = wk.unit, fnt = wk.nt0, fkb = 0;                 // the k-block whose scales are fetched next
    auto fetch_scales = [&](int i) {
      sca[i] = scb[i] = 0.f;
      if (fu >= wk.units) return;
      const int fm = (RES ? fu : fu / p.tiles_n) * FB_BM + row_in_tile, fn = RES ? fnt : fu % p.tiles_n;
      if (fm < p.M) sca[i] = __ldg(p.sa_t + (long long)fkb * p.M + fm);
      scb[i] = __ldg(p.sb + (long long)fn * p.sb_so + (long long)fkb * p.sb_sk);
      if (++fkb == p.kblocks) {
        fkb = 0;
        if (++fnt == wk.nt1) { fnt = wk.nt0; fu += wk.step; }
      }
    };
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) fetch_scales(i);
    for (int u = wk.unit; u < wk.units && ok; u += wk.step)
    for (int nt = wk.nt0; nt < wk.nt1; ++nt) {
      const int m0 = (RES ? u : u / p.tiles_n) * FB_BM, n0 = (RES ? nt : u % p.tiles_n) * FB_BN;
      const int m = m0 + row_in_tile;
      const bool row_ok = m < p.M;
      float out[2][32];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 32; ++i) out[h][i] = 0.f;
      for (int kb = 0; kb < p.kblocks; ++kb, ++n_slot) {
        const int slot = n_slot % FB_SLOTS;
        const uint32_t sph = (n_slot / FB_SLOTS) & 1u;
        const float sc = sca[0] * scb[0];
#pragma unroll
        for (int i = 0; i + 1 < AHEAD; ++i) { sca[i] = sca[i + 1]; scb[i] = scb[i + 1]; }
        fetch_scales(AHEAD - 1);
        {
          const bool w = mbar_wait(&tfull_bar[slot], sph, abort_flag, p.status);
          if (!__all_sync(0xffffffffu, w)) { ok = false; break; }
        }
        tc_fence_after_sync();
        const uint32_t t_addr = tmem_base + (uint32_t)(slot * FB_BN + part * 64) + ((uint32_t)(q * 32) << 16);
        uint32_t r[2][32];
        __syncwarp();
        tmem_ld32(t_addr, r[0]);
        tmem_ld32(t_addr + 32, r[1]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 32; ++i) out[h][i] = fmaf(__uint_as_float(r[h][i]), sc, out[h][i]);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[slot]);
      }
      if (!ok) break;
      if (p.bias != nullptr) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = n0 + part * 64 + h * 32;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (n + i < p.N) out[h][i] += __bfloat162float(__ldg(p.bias + n + i));
        }
      }
      if (p.tma_store) {
        if (lane == 0) tma_store_wait_read<0>();           // this warp's last store has left the staging rows
        __syncwarp();
        uint8_t* srow = my_stage + lane * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int h = j >> 2, e = (j & 3) * 8;
          *reinterpret_cast<uint4*>(srow + (j ^ (lane & 7)) * 16) =
              make_uint4(pack_bf16x2(out[h][e], out[h][e + 1]), pack_bf16x2(out[h][e + 2], out[h][e + 3]),
                         pack_bf16x2(out[h][e + 4], out[h][e + 5]), pack_bf16x2(out[h][e + 6], out[h][e + 7]));
        }
        fence_proxy_async_smem();
        __syncwarp();
        const int col = n0 + part * 64, row = m0 + q * 32;
        if (lane == 0 && col < p.N && row < p.M) {          // the store clips rows and columns past the end
          tma_store_3d(&tmC, my_stage, col, row, 0);
          tma_store_commit();
        }
      } else if (row_ok) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = n0 + part * 64 + h * 32;
          const int nvalid = p.N - n;
          if (nvalid <= 0) continue;
          if (p.out_fp32) {
            float* dst = reinterpret_cast<float*>(p.C) + (long long)m * p.ldc + n;
            if (nvalid >= 32) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                reinterpret_cast<float4*>(dst)[i] = make_float4(out[h][4 * i], out[h][4 * i + 1], out[h][4 * i + 2], out[h][4 * i + 3]);
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (i < nvalid) dst[i] = out[h][i];
            }
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)m * p.ldc + n;
            if (nvalid >= 32) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint4 o;
                o.x = pack_bf16x2(out[h][8 * i + 0], out[h][8 * i + 1]);
                o.y = pack_bf16x2(out[h][8 * i + 2], out[h][8 * i + 3]);
                o.z = pack_bf16x2(out[h][8 * i + 4], out[h][8 * i + 5]);
                o.w = pack_bf16x2(out[h][8 * i + 6], out[h][8 * i + 7]);
                reinterpret_cast<uint4*>(dst)[i] = o;
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (i < nvalid) dst[i] = __float2bfloat16(out[h][i]);
            }
          }
        }
      }
    }
    // this warp's stores must have left shared memory and landed
    if (p.tma_store && lane == 0) tma_store_wait_all<0>();
    __syncwarp();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int RES>
static int launch_block_gemm(int grid, const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC,
                             const FbArgs& p, cudaStream_t stream) {
  static bool attr_set[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 15]) {
    cudaError_t e = cudaFuncSetAttribute(fp8_block_gemm_kernel<RES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         FbCfg<RES>::SMEM);
    if (e != cudaSuccess) return set_error("cudaFuncSetAttribute(fp8_block_gemm): %s", cudaGetErrorString(e));
    attr_set[dev & 15] = true;
  }
  fp8_block_gemm_kernel<RES><<<grid, FB_THREADS, FbCfg<RES>::SMEM, stream>>>(tmA, tmB, tmC, p);
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : set_error("fp8_block_gemm launch: %s", cudaGetErrorString(e));
}

}  // namespace ccb

using namespace ccb;

extern "C" int ccb_fp8_quant_rows(const void* x, int64_t ldx, const void* norm_w, float eps, void* q,
                                  float* s_t, float* inv_rms_out, void* y_out, int64_t R, int64_t K,
                                  void* stream) {
  if (R <= 0) return 0;
  if (K % 128 != 0 || K > 256 * QR_MAXSEG || ldx % 8 != 0)
    return set_error("ccb_fp8_quant_rows: K must be a multiple of 128 and <= %d, rows 16-byte aligned", 256 * QR_MAXSEG);
  auto launch = [&](auto kern, int rows) {
    kern<<<(unsigned)((R + rows - 1) / rows), 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)norm_w, eps, (uint8_t*)q, s_t, inv_rms_out,
        (__nv_bfloat16*)y_out, (int)R, (int)K);
  };
  if (K <= 128) launch(fp8_quant_rows_kernel<16, 1>, 16);
  else if (K <= 256) launch(fp8_quant_rows_kernel<32, 1>, 8);
  else if (K <= 512) launch(fp8_quant_rows_kernel<32, 2>, 8);
  else if (K <= 1024) launch(fp8_quant_rows_kernel<32, 4>, 8);
  else launch(fp8_quant_rows_kernel<32, QR_MAXSEG>, 8);
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : set_error("fp8_quant_rows launch: %s", cudaGetErrorString(e));
}

extern "C" int ccb_fp8_quant_blocks(const void* w, void* q, void* qt, float* s, int64_t N, int64_t K,
                                    void* stream) {
  if (N <= 0 || K <= 0) return 0;
  dim3 grid((unsigned)((K + 127) / 128), (unsigned)((N + 127) / 128));
  const bool vec = N % 8 == 0 && K % 8 == 0 && ((uintptr_t)w & 15) == 0 && (((uintptr_t)q | (uintptr_t)qt) & 7) == 0;
  auto kern = vec ? fp8_quant_blocks_kernel<true> : fp8_quant_blocks_kernel<false>;
  kern<<<grid, 1024, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)w, (uint8_t*)q, (uint8_t*)qt, s, (int)N, (int)K);
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : set_error("fp8_quant_blocks launch: %s", cudaGetErrorString(e));
}

// Column tiles of a CTA in the resident-weight kernel (as many as fit, and as leave every CTA at least two row blocks;
// more than one only while a row block fits the activation ring), or 0: the streaming kernel.  Fewer tiles than SMs: one
// tile a CTA, streaming.  Otherwise what decides is the tiles of the busiest CTA.  Streaming deals single tiles out, the
// resident kernel whole column groups, floor(SMs / groups) CTAs to each: 75 groups of a 9600-wide result leave 73 of 148
// SMs without any.  Its tiles are cheaper, more so where a row block serves several of them.  Measured at 65 536 rows
// (events, cold L2; work = tiles of the busiest CTA, resident / streaming; time = resident / streaming):
//   K = 128 (up to 8 tiles):     work 1.00 time 0.88, 1.16 0.97, 1.24 1.02, 1.29 1.06, 1.60 1.29    -> up to 7/6
//   K = 256 .. 512 (2 or 4):     1.00 0.73-0.85, 1.19 0.89-0.99, 1.32 0.94-0.98, 1.33 0.97-1.09, 1.48 1.25-1.28, 1.97 1.4
//                                                                                                    -> below 4/3
//   K = 640 .. 1024 (1):         1.00 0.89-0.96, 1.06 0.97, 1.15 1.10, 1.18 1.08, 1.48 1.27-1.53, 1.97 1.67 -> up to 17/16
extern "C" int64_t ccb_fp8_block_plan(int64_t M, int64_t N, int64_t K, int64_t sms) {
  const int64_t kb = K / 128, tm = (M + FB_BM - 1) / FB_BM, tn = (N + FB_BN - 1) / FB_BN, total = tm * tn;
  if (kb < 1 || kb > FbCfg<1>::RES_TILES || total <= sms) return 0;
  int64_t nt = kb <= 4 ? FbCfg<1>::RES_TILES / kb : 1;
  if (nt > total / (2 * sms)) nt = total / (2 * sms);
  if (nt < 1) nt = 1;
  const int64_t groups = (tn + nt - 1) / nt;
  if (groups > sms) return 0;
  const int64_t walkers = sms / groups < tm ? sms / groups : tm;
  const int64_t res = (tm + walkers - 1) / walkers * (nt < tn ? nt : tn), str = (total + sms - 1) / sms;
  const bool even = kb == 1 ? 6 * res <= 7 * str : (kb <= 4 ? 3 * res < 4 * str : 16 * res <= 17 * str);
  return even ? nt : 0;
}

extern "C" int ccb_fp8_block_gemm(const void* A8, const float* sa_t, const void* B8, const float* sb,
                                  int64_t sb_so, int64_t sb_sk, void* C, int64_t ldc, int64_t out_fp32,
                                  const void* bias, int64_t M, int64_t N, int64_t K, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (K % 128 != 0) return set_error("ccb_fp8_block_gemm: K must be a multiple of 128 (got %lld)", (long long)K);
  if ((out_fp32 ? ldc % 4 : ldc % 8) != 0) return set_error("ccb_fp8_block_gemm: output rows must be 16-byte aligned");
  CUtensorMap tmA, tmB;
  if (make_tmap_u8_3d(&tmA, A8, (uint64_t)K, (uint64_t)M, 1, (uint64_t)K, 0, 128, FB_BM)) return -1;
  if (make_tmap_u8_3d(&tmB, B8, (uint64_t)K, (uint64_t)N, 1, (uint64_t)K, 0, 128, FB_BN)) return -1;
  FbArgs p;
  // rows and base are on 16-byte boundaries wherever torch allocated the output itself
  CUtensorMap tmC;
  memset(&tmC, 0, sizeof(tmC));
  p.tma_store = !out_fp32 && ((uintptr_t)C & 15) == 0 ? 1 : 0;
  if (p.tma_store && make_tmap_bf16_3d(&tmC, C, (uint64_t)N, (uint64_t)M, 1, (uint64_t)ldc, 0, 64, 32)) return -1;
  p.M = (int)M; p.N = (int)N; p.K = (int)K;
  p.kblocks = (int)(K / 128);
  p.tiles_m = (int)((M + FB_BM - 1) / FB_BM);
  p.tiles_n = (int)((N + FB_BN - 1) / FB_BN);
  p.sa_t = sa_t; p.sb = sb; p.sb_so = sb_so; p.sb_sk = sb_sk;
  p.C = C; p.ldc = ldc; p.out_fp32 = (int)out_fp32;
  p.bias = (const __nv_bfloat16*)bias;
  p.status = ccb_status_ptr();
  const long long total = (long long)p.tiles_m * p.tiles_n;
  const int sms = ccb_num_sms();
  p.nt = (int)ccb_fp8_block_plan(M, N, K, sms);
  p.groups = 1;
  if (p.nt > 0) {
    p.groups = (p.tiles_n + p.nt - 1) / p.nt;
    const long long walkers = sms / p.groups < p.tiles_m ? sms / p.groups : p.tiles_m;
    return launch_block_gemm<1>((int)(walkers * p.groups), tmA, tmB, tmC, p, (cudaStream_t)stream);
  }
  return launch_block_gemm<0>((int)(total < sms ? total : sms), tmA, tmB, tmC, p, (cudaStream_t)stream);
}
