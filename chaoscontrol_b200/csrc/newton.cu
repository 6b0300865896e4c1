// Newton-Schulz orthogonalisation of a batch of small matrices as one launch.
//
// Five quintic iterations X <- aX + (bA + cA^2) X, A = X X^T (tall matrices: A = X^T X and X from the left)
// are fifteen dependent products.  For the trunk's matrices (256 x 256, 512 x 256) each product is a few
// microseconds of latency -- launch, set-up, one tile's loads, its store -- and almost no work: as separate
// launches 16 matrices 256 x 256 took 134 us on the device and eighteen launches on the host; 74 and four here.  A
// cluster of up to eight CTAs owns a matrix for the whole iteration: every CTA computes 128 x 128 tiles of the current
// product (tcgen05, fp32 accumulators in TMEM), results go through L2, and a cluster barrier takes the place of
// a launch.  The arithmetic is that of the separate products (csrc/gemm.cu's store epilogue), bit for bit.
//
// Operands are fetched by all threads with 16-byte cp.async past the L1 (the other CTAs have just written them)
// into the swizzled layout the MMA reads, three 128-wide chunks of the contraction in flight, so no tensor maps
// and no cross-proxy ordering of global memory are involved.  Reference: src/chaoscontrol/optim/muon.py:20-50.
#include "ptx.cuh"
#include "ccb_api.h"
#include "runtime.h"

namespace ccb {

constexpr int NZ_T = 128;                     // tile edge
constexpr int NZ_KC = 128;                    // contraction indices of a stage
constexpr int NZ_KB = 16384;                  // one 64-wide k-block of an operand: 128 rows x 128 bytes
constexpr int NZ_OPER = NZ_KC / 64 * NZ_KB;   // 32 KiB
constexpr int NZ_STAGES = 3;
constexpr int NZ_THREADS = 256;
constexpr int NZ_SMEM = 1024 + NZ_STAGES * 2 * NZ_OPER;

struct NewtonArgs {
  __nv_bfloat16 *X, *Y, *A, *B;               // [G, r, c] twice, [G, k, k] twice, k = min(r, c)
  int r, c, k, tall, steps;
  float ca, cb, cc;
  int* status;
};

// 16 bytes to shared memory, zeros instead when `valid` is false (the address is then not read).
__device__ __forceinline__ void nz_copy16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void nz_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void nz_wait(int pending) {
  if (pending >= 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
  else if (pending == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// 128 rows (K-major: rows of the matrix, NZ_KC columns from k0; MN-major: 128 columns from i0, NZ_KC rows from k0) of
// a row-major [rows, cols] matrix -> swizzled k-blocks; what lies outside the matrix becomes zero.
template <bool MN>
__device__ __forceinline__ void nz_load(uint8_t* dst, const __nv_bfloat16* src, int rows, int cols, int i0, int k0) {
  static_assert(NZ_KC == NZ_T, "both layouts are 128 rows of sixteen 16-byte vectors");
  const uint32_t d = smem_u32(dst);
#pragma unroll
  for (int s = 0; s < NZ_T * 16 / NZ_THREADS; ++s) {
    const int i = threadIdx.x + s * NZ_THREADS, row = i >> 4, v = i & 15, j = v & 7;
    const int gr = (MN ? k0 : i0) + row, gc = (MN ? i0 : k0) + v * 8;
    const int off = MN ? (row >> 6) * NZ_KB + (v >> 3) * 8192 + (row & 63) * 128 : (v >> 3) * NZ_KB + row * 128;
    const bool in = gr < rows && gc < cols;
    nz_copy16(d + off + ((j ^ (row & 7)) << 4), src + (in ? (long long)gr * cols + gc : 0), in);
  }
}

__global__ void __launch_bounds__(NZ_THREADS, 1)
newton_kernel(const NewtonArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cl = (int)gridDim.x, rank = (int)blockIdx.x;       // one cluster spans grid.x
  const long long nx = (long long)p.r * p.c, na = (long long)p.k * p.k, g = blockIdx.y;
  __nv_bfloat16 *X = p.X + g * nx, *Y = p.Y + g * nx, *A = p.A + g * na, *B = p.B + g * na;

  if (threadIdx.x == 0) {
    mbar_init(&done_bar, 1);
    abort_s = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&tmem_slot, NZ_T);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  uint32_t commits = 0;

  // D [m, n] = alpha * opA . opB (+ beta * cin) over kk, tiles dealt to the cluster's CTAs
  auto product = [&](const __nv_bfloat16* a, int ar, int ac, int a_mn, const __nv_bfloat16* b, int br, int bc, int b_mn,
                     const __nv_bfloat16* cin, __nv_bfloat16* d, int m, int n, int kk, float alpha, float beta) {
    const int tn = (n + NZ_T - 1) / NZ_T, tiles = (m + NZ_T - 1) / NZ_T * tn;
    const uint32_t idesc = make_idesc_bf16(NZ_T, NZ_T, a_mn, b_mn);
    const int q = warp & 3, part = warp >> 2;                  // TMEM lane quadrant, 64-column half
    for (int t = rank; t < tiles; t += cl) {
      const int m0 = t / tn * NZ_T, n0 = t % tn * NZ_T;
      const int nch = (kk + NZ_KC - 1) / NZ_KC;
      auto fetch = [&](int ch) {
        uint8_t* sA = smem + ch % NZ_STAGES * 2 * NZ_OPER;
        if (a_mn) nz_load<true>(sA, a, ar, ac, m0, ch * NZ_KC); else nz_load<false>(sA, a, ar, ac, m0, ch * NZ_KC);
        if (b_mn) nz_load<true>(sA + NZ_OPER, b, br, bc, n0, ch * NZ_KC);
        else nz_load<false>(sA + NZ_OPER, b, br, bc, n0, ch * NZ_KC);
        nz_commit();
      };
      int issued = 0;
      for (; issued < nch && issued < NZ_STAGES; ++issued) fetch(issued);
      for (int ch = 0; ch < nch; ++ch) {
        nz_wait(issued - ch - 1);
        fence_proxy_async_smem();                              // the MMA reads what these threads have copied
        __syncthreads();
        if (threadIdx.x == 0) {
          tc_fence_after_sync();
          const uint32_t sA = smem_u32(smem + ch % NZ_STAGES * 2 * NZ_OPER), sB = sA + NZ_OPER;
          const int nkb = min(NZ_KC / 64, (kk - ch * NZ_KC + 63) / 64);
          for (int kb = 0; kb < nkb; ++kb) {
            const uint32_t ab = sA + kb * NZ_KB, bb = sB + kb * NZ_KB;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              const uint64_t ad = a_mn ? make_smem_desc(ab + s * 2048, 8192, 1024) : make_smem_desc(ab + s * 32, 16, 1024);
              const uint64_t bd = b_mn ? make_smem_desc(bb + s * 2048, 8192, 1024) : make_smem_desc(bb + s * 32, 16, 1024);
              umma_bf16(tmem, ad, bd, idesc, (ch > 0 || kb > 0 || s > 0) ? 1u : 0u);
            }
          }
          if (issued < nch || ch == nch - 1) umma_commit(&done_bar);
        }
        if (issued < nch) {                                    // the stage is refilled once its products have been read
          mbar_wait(&done_bar, commits++ & 1u, abort_flag, p.status);
          fetch(issued++);
        }
      }
      // the addend does not depend on the product: requested while the MMAs run
      const int row = m0 + q * 32 + lane, col = n0 + part * 64;
      uint4 cv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        cv[j] = (cin != nullptr && row < m && col + j * 8 < n)
                    ? __ldcg(reinterpret_cast<const uint4*>(cin + (long long)row * n + col + j * 8)) : make_uint4(0u, 0u, 0u, 0u);
      mbar_wait(&done_bar, commits++ & 1u, abort_flag, p.status);
      __syncwarp();
      tc_fence_after_sync();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t acc[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * 64 + h * 32), acc);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 cq = cv[h * 4 + j];
          const float2 c0 = unpack_bf16x2(cq.x), c1 = unpack_bf16x2(cq.y), c2 = unpack_bf16x2(cq.z), c3 = unpack_bf16x2(cq.w);
          const float cf[8] = {c0.x, c0.y, c1.x, c1.y, c2.x, c2.y, c3.x, c3.y};
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            v[e] = __uint_as_float(acc[j * 8 + e]);
            v[e] = cin != nullptr ? fmaf(alpha, v[e], __fmul_rn(beta, cf[e])) : alpha * v[e];
          }
          if (row < m && col + h * 32 + j * 8 < n) {
            uint4 o;
            o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
            o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
            *reinterpret_cast<uint4*>(d + (long long)row * n + col + h * 32 + j * 8) = o;
          }
        }
      }
      tc_fence_before_sync();
      __syncthreads();                                         // the accumulator is free for the next tile
      tc_fence_after_sync();
    }
    // everything written above is visible to the cluster, nothing it reads is replaced before all have read it
    cluster_sync_all();
  };

  for (int s = 0; s < p.steps; ++s) {
    if (p.tall) product(X, p.r, p.c, 1, X, p.r, p.c, 1, nullptr, A, p.k, p.k, p.r, 1.f, 0.f);
    else product(X, p.r, p.c, 0, X, p.r, p.c, 0, nullptr, A, p.k, p.k, p.c, 1.f, 0.f);
    product(A, p.k, p.k, 0, A, p.k, p.k, 0, A, B, p.k, p.k, p.k, p.cc, p.cb);
    if (p.tall) product(X, p.r, p.c, 0, B, p.k, p.k, 0, X, Y, p.r, p.c, p.k, 1.f, p.ca);
    else product(B, p.k, p.k, 0, X, p.r, p.c, 1, X, Y, p.r, p.c, p.k, 1.f, p.ca);
    __nv_bfloat16* t = X;
    X = Y;
    Y = t;
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, NZ_T);
  }
}

// One tile of every product to a CTA (with two, 1 of 512 x 512 took 178 us against 160, 16 of them 357 against 220), and
// not more CTAs than the lines below.  A matrix takes about 75 us whatever the batch, so time goes up by that with
// every round of clusters: 148 SMs hold 14 clusters of eight at once, 36 of four.  Five iterations, one launch /
// fifteen in us (events, cold L2):
//   eight CTAs (512 x 256):  8 matrices 86 / 153, 14 88 / 163, 16 166 / 165, 32 248 / 216    -> 16: 7/8 of the SMs
//   four (256 x 256):        32 80 / 177, 64 154 / 224, 74 225 / 226, 148 373 / 329          -> 74: twice the SMs
//   two (128 x 256):         74 72 / 153, 148 137 / 187          one (128 x 128):  148 70 / 165, 296 131 / 230
// Past its line the gain comes and goes with how full the last wave of clusters is (20 of 512 x 256 168 / 214, 80 of
// 256 x 256 225 / 308).
static bool newton_fits(int64_t G, int64_t tiles, int cl) {
  const int64_t sms = ccb_num_sms();
  return tiles <= cl && G * cl <= (cl == 8 ? sms * 7 / 8 : 2 * sms);
}

}  // namespace ccb

using namespace ccb;

// `steps` iterations on X [G, r, c] (bf16, contiguous); Y like X, A and B [G, k, k] with k = min(r, c) are workspace.
// The result is in X for an even number of steps, else in Y.  Returns 1, launching nothing, for shapes that the
// separate products run better.
extern "C" int ccb_newton_schulz(void* X, void* Y, void* A, void* B, int64_t G, int64_t r, int64_t c, int64_t steps,
                                 float ca, float cb, float cc, void* stream) {
  if (G <= 0 || r <= 0 || c <= 0) return 0;
  const uintptr_t all = (uintptr_t)X | (uintptr_t)Y | (uintptr_t)A | (uintptr_t)B;
  if (r % 8 != 0 || c % 8 != 0 || (all & 15) != 0 || G > 65535 || r > 4096 || c > 4096) return 1;
  const int64_t k = r < c ? r : c, tk = (k + NZ_T - 1) / NZ_T;
  const int64_t tx = ((r + NZ_T - 1) / NZ_T) * ((c + NZ_T - 1) / NZ_T), tiles = tx > tk * tk ? tx : tk * tk;
  int cl = 1;
  while (cl < 8 && cl < tiles) cl *= 2;
  if (!newton_fits(G, tiles, cl)) return 1;
  static bool attr_set[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 15]) {
    cudaError_t e = cudaFuncSetAttribute(newton_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NZ_SMEM);
    if (e != cudaSuccess) return set_error("cudaFuncSetAttribute(newton_schulz): %s", cudaGetErrorString(e));
    attr_set[dev & 15] = true;
  }
  NewtonArgs p;
  p.X = (__nv_bfloat16*)X; p.Y = (__nv_bfloat16*)Y; p.A = (__nv_bfloat16*)A; p.B = (__nv_bfloat16*)B;
  p.r = (int)r; p.c = (int)c; p.k = (int)k; p.tall = r > c ? 1 : 0; p.steps = (int)steps;
  p.ca = ca; p.cb = cb; p.cc = cc;
  p.status = ccb_status_ptr();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cl, (unsigned)G);
  cfg.blockDim = dim3(NZ_THREADS);
  cfg.dynamicSmemBytes = NZ_SMEM;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cl; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, newton_kernel, p);
  count_launch();
  return e == cudaSuccess ? 0 : set_error("newton_schulz launch: %s", cudaGetErrorString(e));
}
