// Fused diagonal-SSM scan, forward and backward.
//
// Input is the packed projection P[r, 4D] = (select | candidate | gate | delta)
// raw GEMM outputs (bf16), r = b*T + t.  The kernel applies the gate
// nonlinearities, builds decay = exp(-max(softplus(delta), 1e-4) * sigmoid(log_a))
// and update = sigmoid(select) * tanh(candidate), runs the recurrence
//   h[t] = decay[t] * h[t-1] + update[t],   h[-1] = h0 (zero when absent)
// in fp32 registers and emits y = sigmoid(gate) * h.  decay / update / gate are
// never written to memory.  One thread owns two adjacent channels of one batch
// row, so every warp-wide access is a full 128-byte line.
//
// Reference semantics: src/chaoscontrol/core.py:492-507 (_diag_terms),
// core.py:26-32 (recurrence), kernels/_ssm_scan/src/ssm_scan_fwd.cu:103-126 and
// ssm_scan_bwd.cu:104-141 (the unfused serial scan these kernels replace).
// Unlike the reference kernels these take an initial state and return the
// final state, so carried-state evaluation never drops to a per-token loop.
#include "ptx.cuh"
#include <cuda_fp16.h>
#include "ccb_api.h"
#include "runtime.h"

namespace ccb {

constexpr int SCAN_THREADS = 128;

struct Gates {
  float decay, sel, cand, gate, sp_sig, delta;  // sp_sig = d softplus / d raw (0 when clamped)
};

// POLY: the two exponentials run on the FMA pipe (exp_nonpos_fma) instead of the special-function
// unit, which the three tanh and the logarithm of every channel step already keep busy.
template <bool POLY>
__device__ __forceinline__ Gates eval_gates(float s_raw, float c_raw, float g_raw, float d_raw,
                                            float a) {
  Gates g;
  g.sel = sigmoidf_fast(s_raw);
  g.cand = tanhf_fast(c_raw);
  g.gate = sigmoidf_fast(g_raw);
  const float e = POLY ? exp_nonpos_fma(-fabsf(d_raw)) : __expf(-fabsf(d_raw));
  float sp = fmaxf(d_raw, 0.f) + __logf(1.f + e);
  // d softplus / dx = sigmoid(x)
  const float inv1pe = rcpf_fast(1.f + e);
  const float sig = d_raw >= 0.f ? inv1pe : e * inv1pe;
  g.sp_sig = sp > 1e-4f ? sig : 0.f;
  g.delta = fmaxf(sp, 1e-4f);
  g.decay = POLY ? exp_nonpos_fma(-g.delta * a) : __expf(-g.delta * a);
  return g;
}

// ---- packed fp32x2 evaluation ------------------------------------------------------------------
// One thread owns two adjacent channels that go through the same arithmetic, and both kernels are
// bound by instruction issue, not by bytes: sm_100's two-wide fp32 instructions (fma / mul / add on a
// register pair) do each step for both channels at once.  Special-function ops stay one per channel.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2s(float a) { return make_float2(a, a); }
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2f(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 sigmoid2(float2 x) {
  const float2 h = __fmul2_rn(x, f2s(0.5f));
  return __ffma2_rn(f2(tanhf_fast(h.x), tanhf_fast(h.y)), f2s(0.5f), f2s(0.5f));
}

struct Gates2 {
  float2 decay, sel, cand, gate, sp_sig, delta;
};

// nal2e = -sigmoid(log_a) * log2(e), per channel: decay = 2^(delta * nal2e)
template <bool WANT_SIG>
__device__ __forceinline__ Gates2 eval_gates2(float2 s_raw, float2 c_raw, float2 g_raw, float2 d_raw,
                                              float2 nal2e) {
  constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
  Gates2 g;
  g.sel = sigmoid2(s_raw);
  g.cand = f2(tanhf_fast(c_raw.x), tanhf_fast(c_raw.y));
  g.gate = sigmoid2(g_raw);
  const float2 t = __fmul2_rn(f2(-fabsf(d_raw.x), -fabsf(d_raw.y)), f2s(LOG2E));
  const float2 e = f2(ex2f(t.x), ex2f(t.y));
  const float2 ope = __fadd2_rn(e, f2s(1.f));
  const float2 sp = __ffma2_rn(f2(lg2f(ope.x), lg2f(ope.y)), f2s(LN2), f2(fmaxf(d_raw.x, 0.f), fmaxf(d_raw.y, 0.f)));
  if (WANT_SIG) {
    const float2 inv = f2(rcpf_fast(ope.x), rcpf_fast(ope.y));
    const float2 einv = __fmul2_rn(e, inv);
    g.sp_sig = f2(sp.x > 1e-4f ? (d_raw.x >= 0.f ? inv.x : einv.x) : 0.f,
                  sp.y > 1e-4f ? (d_raw.y >= 0.f ? inv.y : einv.y) : 0.f);
  }
  g.delta = f2(fmaxf(sp.x, 1e-4f), fmaxf(sp.y, 1e-4f));
  const float2 u = __fmul2_rn(g.delta, nal2e);
  g.decay = f2(ex2f(u.x), ex2f(u.y));
  return g;
}

// grid: (ceil(D/256), B); block: 128 threads, 2 channels per thread.
// MODE 0: scalar arithmetic; 1: scalar with FMA-pipe exponentials; 2: packed fp32x2 arithmetic.
// U time steps are loaded ahead of their arithmetic; MINB resident blocks per SM bound the registers.
template <int MODE, int U = 8, int MINB = 4>
__global__ void __launch_bounds__(SCAN_THREADS, MINB)
scan_fwd_kernel(const __nv_bfloat16* __restrict__ P, long long ldp, const float* __restrict__ log_a,
                const float* __restrict__ h0, __nv_bfloat16* __restrict__ y,
                __nv_bfloat16* __restrict__ hout, float* __restrict__ hT, int T, int D,
                long long la_bstride) {
  constexpr int SCAN_UNROLL = U;
  const int b = blockIdx.y;
  const int d = (blockIdx.x * SCAN_THREADS + threadIdx.x) * 2;
  if (d >= D) return;
  // la_bstride != 0: every batch row has its own decay vector (per-document test-time training)
  const float a0 = sigmoidf_fast(log_a[b * la_bstride + d]);
  const float a1 = sigmoidf_fast(log_a[b * la_bstride + d + 1]);
  const float2 nal2e = f2(-a0 * 1.4426950408889634f, -a1 * 1.4426950408889634f);
  float s0 = 0.f, s1 = 0.f;
  if (h0 != nullptr) {
    s0 = h0[(long long)b * D + d];
    s1 = h0[(long long)b * D + d + 1];
  }
  const uint32_t* Pw = reinterpret_cast<const uint32_t*>(P + (long long)b * T * ldp + d);
  const long long rowstride = ldp / 2;   // in uint32 units
  const int dq = D / 2;
  uint32_t* yw = reinterpret_cast<uint32_t*>(y + ((long long)b * T) * D + d);
  uint32_t* hw = hout ? reinterpret_cast<uint32_t*>(hout + ((long long)b * T) * D + d) : nullptr;

  for (int t0 = 0; t0 < T; t0 += SCAN_UNROLL) {
    uint32_t raw[SCAN_UNROLL][4];
#pragma unroll
    for (int u = 0; u < SCAN_UNROLL; ++u) {
      if (t0 + u < T) {
        const uint32_t* row = Pw + (long long)(t0 + u) * rowstride;
        raw[u][0] = __ldg(row);
        raw[u][1] = __ldg(row + dq);
        raw[u][2] = __ldg(row + 2 * dq);
        raw[u][3] = __ldg(row + 3 * dq);
      }
    }
#pragma unroll
    for (int u = 0; u < SCAN_UNROLL; ++u) {
      if (t0 + u < T) {
        const float2 sr = unpack_bf16x2(raw[u][0]);
        const float2 cr = unpack_bf16x2(raw[u][1]);
        const float2 gr = unpack_bf16x2(raw[u][2]);
        const float2 dr = unpack_bf16x2(raw[u][3]);
        const long long o = (long long)(t0 + u) * dq;
        if (MODE == 2) {
          const Gates2 g = eval_gates2<false>(sr, cr, gr, dr, nal2e);
          const float2 st = __ffma2_rn(g.decay, f2(s0, s1), __fmul2_rn(g.sel, g.cand));
          s0 = st.x;
          s1 = st.y;
          const float2 yv = __fmul2_rn(g.gate, st);
          yw[o] = pack_bf16x2(yv.x, yv.y);
        } else {
          const Gates g0 = eval_gates<MODE == 1>(sr.x, cr.x, gr.x, dr.x, a0);
          const Gates g1 = eval_gates<MODE == 1>(sr.y, cr.y, gr.y, dr.y, a1);
          s0 = g0.decay * s0 + g0.sel * g0.cand;
          s1 = g1.decay * s1 + g1.sel * g1.cand;
          yw[o] = pack_bf16x2(g0.gate * s0, g1.gate * s1);
        }
        if (hw) hw[o] = pack_bf16x2(s0, s1);
      }
    }
  }
  if (hT != nullptr) {
    hT[(long long)b * D + d] = s0;
    hT[(long long)b * D + d + 1] = s1;
  }
}

// Backward.  Walks t from T-1 down to 0 with the carry dh[t] * decay[t].
// Needs the forward states h (bf16) and the raw projections; recomputes the
// gates.  Emits dP (optionally pre-multiplied by the consumer's RMSNorm row
// scale rs[r] = rsqrt(rowss[r] * inv_dim + eps)), per-batch-row partials of
// d log_a, and optionally d h0.
template <int MODE, int U = 8, int MINB = 4>
__global__ void __launch_bounds__(SCAN_THREADS, MINB)
scan_bwd_kernel(const __nv_bfloat16* __restrict__ P, long long ldp, const float* __restrict__ log_a,
                const float* __restrict__ h0, const __nv_bfloat16* __restrict__ hstates,
                const __nv_bfloat16* __restrict__ dy, const float* __restrict__ dhT,
                const float* __restrict__ rowss, float inv_dim, float eps,
                __nv_bfloat16* __restrict__ dP, long long lddp, float* __restrict__ dloga_part,
                float* __restrict__ dh0, int T, int D, long long la_bstride) {
  constexpr int SCAN_UNROLL = U;
  const int b = blockIdx.y;
  const int d = (blockIdx.x * SCAN_THREADS + threadIdx.x) * 2;
  if (d >= D) return;
  const float a0 = sigmoidf_fast(log_a[b * la_bstride + d]);
  const float a1 = sigmoidf_fast(log_a[b * la_bstride + d + 1]);
  const float2 nal2e = f2(-a0 * 1.4426950408889634f, -a1 * 1.4426950408889634f);
  const long long rowbase = (long long)b * T;
  const int dq = D / 2;
  const uint32_t* Pw = reinterpret_cast<const uint32_t*>(P + rowbase * ldp + d);
  const long long prs = ldp / 2;
  uint32_t* dPw = reinterpret_cast<uint32_t*>(dP + rowbase * lddp + d);
  const long long dprs = lddp / 2;
  const uint32_t* hw = reinterpret_cast<const uint32_t*>(hstates + rowbase * D + d);
  const uint32_t* dyw = reinterpret_cast<const uint32_t*>(dy + rowbase * D + d);

  float c0 = 0.f, c1 = 0.f;      // carry: dL/dh[t] contribution from t+1
  if (dhT != nullptr) {
    c0 = dhT[(long long)b * D + d];
    c1 = dhT[(long long)b * D + d + 1];
  }
  float da0 = 0.f, da1 = 0.f;
  float2 hcur = unpack_bf16x2(__ldg(hw + (long long)(T - 1) * dq));

  for (int t1 = T - 1; t1 >= 0; t1 -= SCAN_UNROLL) {
    uint32_t raw[SCAN_UNROLL][4];
    uint32_t hp[SCAN_UNROLL];
    uint32_t dyr[SCAN_UNROLL];
    float rsr[SCAN_UNROLL];
#pragma unroll
    for (int u = 0; u < SCAN_UNROLL; ++u) {
      const int t = t1 - u;
      if (t >= 0) {
        const uint32_t* row = Pw + (long long)t * prs;
        raw[u][0] = __ldg(row);
        raw[u][1] = __ldg(row + dq);
        raw[u][2] = __ldg(row + 2 * dq);
        raw[u][3] = __ldg(row + 3 * dq);
        dyr[u] = __ldg(dyw + (long long)t * dq);
        hp[u] = t > 0 ? __ldg(hw + (long long)(t - 1) * dq) : 0u;
        rsr[u] = rowss ? rsqrtf(__ldg(rowss + rowbase + t) * inv_dim + eps) : 1.f;
      }
    }
#pragma unroll
    for (int u = 0; u < SCAN_UNROLL; ++u) {
      const int t = t1 - u;
      if (t >= 0) {
        const float2 sr = unpack_bf16x2(raw[u][0]);
        const float2 cr = unpack_bf16x2(raw[u][1]);
        const float2 gr = unpack_bf16x2(raw[u][2]);
        const float2 dr = unpack_bf16x2(raw[u][3]);
        const float2 dyv = unpack_bf16x2(dyr[u]);
        float2 hprev;
        if (t > 0) {
          hprev = unpack_bf16x2(hp[u]);
        } else if (h0 != nullptr) {
          hprev = make_float2(h0[(long long)b * D + d], h0[(long long)b * D + d + 1]);
        } else {
          hprev = make_float2(0.f, 0.f);
        }
        const float rs = rsr[u];
        uint32_t* orow = dPw + (long long)t * dprs;
        if (MODE == 2) {
          const Gates2 g = eval_gates2<true>(sr, cr, gr, dr, nal2e);
          const float2 one = f2s(1.f), neg1 = f2s(-1.f), rs2 = f2s(rs);
          // y = gate * h;  h = decay * hprev + sel * cand
          const float2 dgate = __fmul2_rn(dyv, hcur);
          const float2 dh = __ffma2_rn(dyv, g.gate, f2(c0, c1));
          const float2 ddec = __fmul2_rn(dh, hprev);
          const float2 cn = __fmul2_rn(dh, g.decay);
          c0 = cn.x;
          c1 = cn.y;
          const float2 ds = __fmul2_rn(__fmul2_rn(dh, g.cand), __fmul2_rn(g.sel, __ffma2_rn(g.sel, neg1, one)));
          const float2 dc = __fmul2_rn(__fmul2_rn(dh, g.sel), __ffma2_rn(__fmul2_rn(g.cand, neg1), g.cand, one));
          const float2 dg = __fmul2_rn(dgate, __fmul2_rn(g.gate, __ffma2_rn(g.gate, neg1, one)));
          // decay = exp(-delta * a): d/d delta = -a * decay ; d/d a = -delta * decay
          const float2 dd = __fmul2_rn(__fmul2_rn(ddec, __fmul2_rn(f2(-a0, -a1), g.decay)), g.sp_sig);
          const float2 dan = __ffma2_rn(__fmul2_rn(ddec, g.delta), __fmul2_rn(g.decay, neg1), f2(da0, da1));
          da0 = dan.x;
          da1 = dan.y;
          const float2 o0 = __fmul2_rn(ds, rs2), o1 = __fmul2_rn(dc, rs2), o2 = __fmul2_rn(dg, rs2),
                       o3 = __fmul2_rn(dd, rs2);
          orow[0] = pack_bf16x2(o0.x, o0.y);
          orow[dq] = pack_bf16x2(o1.x, o1.y);
          orow[2 * dq] = pack_bf16x2(o2.x, o2.y);
          orow[3 * dq] = pack_bf16x2(o3.x, o3.y);
        } else {
          const Gates g0 = eval_gates<MODE == 1>(sr.x, cr.x, gr.x, dr.x, a0);
          const Gates g1 = eval_gates<MODE == 1>(sr.y, cr.y, gr.y, dr.y, a1);
          // y = gate * h
          const float dgate0 = dyv.x * hcur.x, dgate1 = dyv.y * hcur.y;
          const float dh0_ = dyv.x * g0.gate + c0, dh1_ = dyv.y * g1.gate + c1;
          // h = decay * hprev + sel * cand
          const float ddec0 = dh0_ * hprev.x, ddec1 = dh1_ * hprev.y;
          c0 = dh0_ * g0.decay;
          c1 = dh1_ * g1.decay;
          const float ds0 = dh0_ * g0.cand * g0.sel * (1.f - g0.sel);
          const float ds1 = dh1_ * g1.cand * g1.sel * (1.f - g1.sel);
          const float dc0 = dh0_ * g0.sel * (1.f - g0.cand * g0.cand);
          const float dc1 = dh1_ * g1.sel * (1.f - g1.cand * g1.cand);
          const float dg0 = dgate0 * g0.gate * (1.f - g0.gate);
          const float dg1 = dgate1 * g1.gate * (1.f - g1.gate);
          // decay = exp(-delta * a): d/d delta = -a * decay ; d/d a = -delta * decay
          const float dd0 = ddec0 * (-a0 * g0.decay) * g0.sp_sig;
          const float dd1 = ddec1 * (-a1 * g1.decay) * g1.sp_sig;
          da0 += ddec0 * (-g0.delta * g0.decay);
          da1 += ddec1 * (-g1.delta * g1.decay);
          orow[0] = pack_bf16x2(ds0 * rs, ds1 * rs);
          orow[dq] = pack_bf16x2(dc0 * rs, dc1 * rs);
          orow[2 * dq] = pack_bf16x2(dg0 * rs, dg1 * rs);
          orow[3 * dq] = pack_bf16x2(dd0 * rs, dd1 * rs);
        }
        hcur = hprev;
      }
    }
  }
  if (dloga_part != nullptr) {
    // d a / d log_a = a (1 - a)
    dloga_part[(long long)b * D + d] = da0 * a0 * (1.f - a0);
    dloga_part[(long long)b * D + d + 1] = da1 * a1 * (1.f - a1);
  }
  if (dh0 != nullptr) {
    dh0[(long long)b * D + d] = c0;
    dh0[(long long)b * D + d + 1] = c1;
  }
}

// ---- time-tiled scans for few channels -----------------------------------------------------------
// The kernels above give every channel pair one thread for all T steps, so a batch of B rows keeps only
// B * D / 256 blocks busy and each of them waits for memory and for the special functions of one step
// after the other.  Here the warps of a block share the steps of 64 channels of one row: a tile is
// NW * U steps, warp w takes U of them, evaluates their gates (the expensive part, independent of the
// recurrence) and folds them into one affine map state -> A * state + b; the maps of the tile go through
// shared memory, every warp composes them in order up to its own steps, and then runs its U steps from
// the exact carry with the serial kernels' arithmetic.  One barrier per tile (the maps are double
// buffered); the next tile's operands are requested before it.
// CL > 1: a cluster of CL blocks shares one row's steps the same way, the composed map of each block's
// tile goes to the other blocks' shared memory, so that even one row of 256 channels uses 32 SMs.
// All fp32, as above: only the carry at a warp's first step is rounded differently.
// a * b, except that two non-zero factors never give zero: a product of decays that underflows would turn an
// infinite state into NaN where the serial kernels keep it infinite (the smallest normal number stands in).
__device__ __forceinline__ float2 keep_normal(float2 prod, float2 a, float2 b) {
  if (prod.x == 0.f && a.x != 0.f && b.x != 0.f) prod.x = 1.17549435e-38f;
  if (prod.y == 0.f && a.y != 0.f && b.y != 0.f) prod.y = 1.17549435e-38f;
  return prod;
}
__device__ __forceinline__ void st_cluster_f4(uint32_t addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// The carry of a tile.  In: this warp's map (A, b) and the state at the start of the (cluster's) tile.  Returns
// the state at this warp's first step and leaves the state after the whole tile in `st`.
template <int NW, int CL>
__device__ __forceinline__ float2 tile_carry(float4 (&seg)[NW][32], float4 (&blk)[CL][32], int warp, int lane, int rank,
                                             float4 map, float2& st) {
  seg[warp][lane] = map;
  __syncthreads();
  float2 mine = st;
  if constexpr (CL == 1) {
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      if (w == warp) mine = st;
      const float4 v = seg[w][lane];
      st = __ffma2_rn(f2(v.x, v.y), st, f2(v.z, v.w));
    }
  } else {
    // the block's own composition: up to this warp, and whole
    float2 A = f2s(1.f), bb = f2s(0.f), Am = A, bm = bb;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      if (w == warp) { Am = A; bm = bb; }
      const float4 v = seg[w][lane];
      A = keep_normal(__fmul2_rn(A, f2(v.x, v.y)), A, f2(v.x, v.y));
      bb = __ffma2_rn(f2(v.x, v.y), bb, f2(v.z, v.w));
    }
    if (warp < CL) st_cluster_f4(mapa_shared(smem_u32(&blk[rank][lane]), (uint32_t)warp), make_float4(A.x, A.y, bb.x, bb.y));
    cluster_sync_all();
#pragma unroll
    for (int r = 0; r < CL; ++r) {
      if (r == rank) mine = st;
      const float4 v = blk[r][lane];
      st = __ffma2_rn(f2(v.x, v.y), st, f2(v.z, v.w));
    }
    mine = __ffma2_rn(Am, mine, bm);
  }
  return mine;
}

template <int U, int NW, int MINB, int CL>
__global__ void __launch_bounds__(32 * NW, MINB)
scan_tile_fwd_kernel(const __nv_bfloat16* __restrict__ P, long long ldp, const float* __restrict__ log_a,
                     const float* __restrict__ h0, __nv_bfloat16* __restrict__ y,
                     __nv_bfloat16* __restrict__ hout, float* __restrict__ hT, int T, int D,
                     long long la_bstride) {
  static_assert(CL <= NW, "warp r hands the block's map to block r of the cluster");
  constexpr int TT = U * NW * CL;
  __shared__ float4 seg[2][NW][32];
  __shared__ float4 blk[2][CL][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CL > 1 ? (int)cluster_ctarank() : 0;
  const int first = (rank * NW + warp) * U;        // this warp's first step of a tile
  if (CL > 1) cluster_sync_all();                  // every block runs before any writes to its shared memory
  const int b = blockIdx.y;
  const int d = (blockIdx.x * 32 + lane) * 2;
  const bool on = d < D;
  float2 nal2e = f2s(0.f), st = f2s(0.f);
  if (on) {
    const float* la = log_a + b * la_bstride + d;
    nal2e = f2(-sigmoidf_fast(la[0]) * 1.4426950408889634f, -sigmoidf_fast(la[1]) * 1.4426950408889634f);
    if (h0 != nullptr) st = f2(h0[(long long)b * D + d], h0[(long long)b * D + d + 1]);
  }
  const uint32_t* Pw = reinterpret_cast<const uint32_t*>(P + (long long)b * T * ldp + d);
  const long long rowstride = ldp / 2;
  const int dq = D / 2;
  uint32_t* yw = reinterpret_cast<uint32_t*>(y + ((long long)b * T) * D + d);
  uint32_t* hw = hout ? reinterpret_cast<uint32_t*>(hout + ((long long)b * T) * D + d) : nullptr;

  uint32_t raw[U][4];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (on && t0 + u < T) {
        const uint32_t* row = Pw + (long long)(t0 + u) * rowstride;
        raw[u][0] = __ldg(row);
        raw[u][1] = __ldg(row + dq);
        raw[u][2] = __ldg(row + 2 * dq);
        raw[u][3] = __ldg(row + 3 * dq);
      } else {
        raw[u][0] = raw[u][1] = raw[u][2] = raw[u][3] = 0u;
      }
    }
  };
  fetch(first);
  int buf = 0;
  for (int t0 = 0; t0 < T; t0 += TT, buf ^= 1) {
    const int tw = t0 + first;
    float2 dec[U], upd[U], gate[U];
    float2 A = f2s(1.f), bb = f2s(0.f);
    if (tw < T) {                          // a warp past the end leaves the state as it is
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const Gates2 g = eval_gates2<false>(unpack_bf16x2(raw[u][0]), unpack_bf16x2(raw[u][1]),
                                            unpack_bf16x2(raw[u][2]), unpack_bf16x2(raw[u][3]), nal2e);
        const bool in = tw + u < T;
        dec[u] = in ? g.decay : f2s(1.f);
        upd[u] = in ? __fmul2_rn(g.sel, g.cand) : f2s(0.f);
        gate[u] = g.gate;
        A = __fmul2_rn(A, dec[u]);
        bb = __ffma2_rn(dec[u], bb, upd[u]);
      }
    }
    if (t0 + TT < T) fetch(tw + TT);
    if (A.x == 0.f || A.y == 0.f) {
      A = f2s(1.f);
#pragma unroll
      for (int u = 0; u < U; ++u) A = keep_normal(__fmul2_rn(A, dec[u]), A, dec[u]);
    }
    float2 h = tile_carry<NW, CL>(seg[buf], blk[buf], warp, lane, rank, make_float4(A.x, A.y, bb.x, bb.y), st);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (on && tw + u < T) {
        h = __ffma2_rn(dec[u], h, upd[u]);
        const long long o = (long long)(tw + u) * dq;
        const float2 yv = __fmul2_rn(gate[u], h);
        yw[o] = pack_bf16x2(yv.x, yv.y);
        if (hw) hw[o] = pack_bf16x2(h.x, h.y);
      }
    }
  }
  if (hT != nullptr && rank == 0 && warp == 0 && on) {
    hT[(long long)b * D + d] = st.x;
    hT[(long long)b * D + d + 1] = st.y;
  }
}

// Backward: the same split over t = T-1 .. 0.  The carried quantity c = dL/dh[t] * decay[t] obeys
// c' = decay * (c + dy * gate), again an affine map; with the carry known each warp runs the serial
// kernel's step.  d log_a is summed per warp and joined in warp order.
template <int U, int NW, int MINB, int CL>
__global__ void __launch_bounds__(32 * NW, MINB)
scan_tile_bwd_kernel(const __nv_bfloat16* __restrict__ P, long long ldp, const float* __restrict__ log_a,
                     const float* __restrict__ h0, const __nv_bfloat16* __restrict__ hstates,
                     const __nv_bfloat16* __restrict__ dy, const float* __restrict__ dhT,
                     const float* __restrict__ rowss, float inv_dim, float eps,
                     __nv_bfloat16* __restrict__ dP, long long lddp, float* __restrict__ dloga_part,
                     float* __restrict__ dh0, int T, int D, long long la_bstride) {
  static_assert(CL <= NW, "warp r hands the block's map to block r of the cluster");
  constexpr int TT = U * NW * CL;
  __shared__ float4 seg[2][NW][32];
  __shared__ float4 blk[2][CL][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CL > 1 ? (int)cluster_ctarank() : 0;
  const int first = (rank * NW + warp) * U;        // this warp's first step of a tile
  if (CL > 1) cluster_sync_all();                  // every block runs before any writes to its shared memory
  const int b = blockIdx.y;
  const int d = (blockIdx.x * 32 + lane) * 2;
  const bool on = d < D;
  float2 a = f2s(0.f), carry = f2s(0.f), hinit = f2s(0.f);
  if (on) {
    const float* la = log_a + b * la_bstride + d;
    a = f2(sigmoidf_fast(la[0]), sigmoidf_fast(la[1]));
    if (dhT != nullptr) carry = f2(dhT[(long long)b * D + d], dhT[(long long)b * D + d + 1]);
    if (h0 != nullptr) hinit = f2(h0[(long long)b * D + d], h0[(long long)b * D + d + 1]);
  }
  const float2 nal2e = f2(-a.x * 1.4426950408889634f, -a.y * 1.4426950408889634f);
  const long long rowbase = (long long)b * T;
  const int dq = D / 2;
  const uint32_t* Pw = reinterpret_cast<const uint32_t*>(P + rowbase * ldp + d);
  const long long prs = ldp / 2;
  uint32_t* dPw = reinterpret_cast<uint32_t*>(dP + rowbase * lddp + d);
  const long long dprs = lddp / 2;
  const uint32_t* hw = reinterpret_cast<const uint32_t*>(hstates + rowbase * D + d);
  const uint32_t* dyw = reinterpret_cast<const uint32_t*>(dy + rowbase * D + d);

  uint32_t raw[U][4], dyr[U], hr[U + 1];
  float rsr[U];
  // step u of a tile that starts at position j0 of the reversed order is t = T - 1 - (j0 + u)
  auto fetch = [&](int j0) {
#pragma unroll
    for (int u = 0; u <= U; ++u) {
      const int t = T - 1 - (j0 + u);
      hr[u] = (on && t >= 0) ? __ldg(hw + (long long)t * dq) : 0u;
      if (u == U) break;
      if (on && t >= 0) {
        const uint32_t* row = Pw + (long long)t * prs;
        raw[u][0] = __ldg(row);
        raw[u][1] = __ldg(row + dq);
        raw[u][2] = __ldg(row + 2 * dq);
        raw[u][3] = __ldg(row + 3 * dq);
        dyr[u] = __ldg(dyw + (long long)t * dq);
      } else {
        raw[u][0] = raw[u][1] = raw[u][2] = raw[u][3] = dyr[u] = 0u;
      }
      rsr[u] = (rowss && t >= 0) ? __ldg(rowss + rowbase + t) : 0.f;
    }
  };
  fetch(first);
  float2 da = f2s(0.f);
  int buf = 0;
  for (int j0 = 0; j0 < T; j0 += TT, buf ^= 1) {
    const int jw = j0 + first;
    Gates2 g[U];
    float2 dyv[U], hc[U + 1];
    float rs[U];
    float2 A = f2s(1.f), bb = f2s(0.f);
    hc[U] = unpack_bf16x2(hr[U]);
    if (jw < T) {                          // a warp past the beginning leaves the carry as it is
#pragma unroll
      for (int u = 0; u < U; ++u) {
        g[u] = eval_gates2<true>(unpack_bf16x2(raw[u][0]), unpack_bf16x2(raw[u][1]), unpack_bf16x2(raw[u][2]),
                                 unpack_bf16x2(raw[u][3]), nal2e);
        dyv[u] = unpack_bf16x2(dyr[u]);
        hc[u] = unpack_bf16x2(hr[u]);
        rs[u] = rowss ? rsqrtf(rsr[u] * inv_dim + eps) : 1.f;
        if (jw + u < T) {
          A = __fmul2_rn(A, g[u].decay);
          bb = __fmul2_rn(g[u].decay, __ffma2_rn(dyv[u], g[u].gate, bb));
        }
      }
    }
    if (j0 + TT < T) fetch(jw + TT);
    if (A.x == 0.f || A.y == 0.f) {
      A = f2s(1.f);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (jw + u < T) A = keep_normal(__fmul2_rn(A, g[u].decay), A, g[u].decay);
    }
    float2 c = tile_carry<NW, CL>(seg[buf], blk[buf], warp, lane, rank, make_float4(A.x, A.y, bb.x, bb.y), carry);
    const float2 one = f2s(1.f), neg1 = f2s(-1.f);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = T - 1 - (jw + u);
      if (t >= 0) {
        const float2 hprev = t > 0 ? hc[u + 1] : hinit;
        const float2 rs2 = f2s(rs[u]);
        // y = gate * h;  h = decay * hprev + sel * cand
        const float2 dgate = __fmul2_rn(dyv[u], hc[u]);
        const float2 dh = __ffma2_rn(dyv[u], g[u].gate, c);
        const float2 ddec = __fmul2_rn(dh, hprev);
        c = __fmul2_rn(dh, g[u].decay);
        const float2 ds = __fmul2_rn(__fmul2_rn(dh, g[u].cand), __fmul2_rn(g[u].sel, __ffma2_rn(g[u].sel, neg1, one)));
        const float2 dc = __fmul2_rn(__fmul2_rn(dh, g[u].sel), __ffma2_rn(__fmul2_rn(g[u].cand, neg1), g[u].cand, one));
        const float2 dg = __fmul2_rn(dgate, __fmul2_rn(g[u].gate, __ffma2_rn(g[u].gate, neg1, one)));
        // decay = exp(-delta * a): d/d delta = -a * decay ; d/d a = -delta * decay
        const float2 dd = __fmul2_rn(__fmul2_rn(ddec, __fmul2_rn(f2(-a.x, -a.y), g[u].decay)), g[u].sp_sig);
        da = __ffma2_rn(__fmul2_rn(ddec, g[u].delta), __fmul2_rn(g[u].decay, neg1), da);
        if (on) {
          const float2 o0 = __fmul2_rn(ds, rs2), o1 = __fmul2_rn(dc, rs2), o2 = __fmul2_rn(dg, rs2),
                       o3 = __fmul2_rn(dd, rs2);
          uint32_t* orow = dPw + (long long)t * dprs;
          orow[0] = pack_bf16x2(o0.x, o0.y);
          orow[dq] = pack_bf16x2(o1.x, o1.y);
          orow[2 * dq] = pack_bf16x2(o2.x, o2.y);
          orow[3 * dq] = pack_bf16x2(o3.x, o3.y);
        }
      }
    }
  }
  if (dloga_part != nullptr) {
    __syncthreads();                       // the maps of the last tile have been read
    float2* join = reinterpret_cast<float2*>(&seg[0][0][0]);
    join[warp * 32 + lane] = da;
    __syncthreads();
    float2 t = f2s(0.f);
    if (warp == 0) {
      t = join[lane];
#pragma unroll
      for (int w = 1; w < NW; ++w) t = __fadd2_rn(t, join[w * 32 + lane]);
    }
    if constexpr (CL > 1) {                // block sums to block 0, added in block order
      cluster_sync_all();                  // block 0 has read the maps of its last tile
      if (warp == 0) st_cluster_f4(mapa_shared(smem_u32(&blk[0][rank][lane]), 0u), make_float4(t.x, t.y, 0.f, 0.f));
      cluster_sync_all();
      if (warp == 0 && rank == 0) {
        t = f2(blk[0][0][lane].x, blk[0][0][lane].y);
#pragma unroll
        for (int r = 1; r < CL; ++r) t = __fadd2_rn(t, f2(blk[0][r][lane].x, blk[0][r][lane].y));
      }
    }
    if (warp == 0 && rank == 0 && on) {
      // d a / d log_a = a (1 - a)
      dloga_part[(long long)b * D + d] = t.x * a.x * (1.f - a.x);
      dloga_part[(long long)b * D + d + 1] = t.y * a.y * (1.f - a.y);
    }
  }
  if (dh0 != nullptr && rank == 0 && warp == 0 && on) {
    dh0[(long long)b * D + d] = carry.x;
    dh0[(long long)b * D + d + 1] = carry.y;
  }
}

// Plain recurrence state[t] = decay[t] * state[t-1] + update[t] for the public ssm_scan op, in
// the operand dtypes the reference op accepts without a cast
// (kernels/_ssm_scan/__init__.py:104-113): decay / update = bf16/bf16, bf16/fp16, fp16/fp16,
// fp32/fp32, fp32/bf16, fp32/fp16.  fp32 accumulator; the states are kept in fp32 for backward.
template <typename T> __device__ __forceinline__ float scan_ld(const T* p, long long i);
template <> __device__ __forceinline__ float scan_ld<float>(const float* p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float scan_ld<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
  return __bfloat162float(p[i]);
}
template <> __device__ __forceinline__ float scan_ld<__half>(const __half* p, long long i) { return __half2float(p[i]); }
template <typename T> __device__ __forceinline__ void scan_st(T* p, long long i, float v);
template <> __device__ __forceinline__ void scan_st<float>(float* p, long long i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void scan_st<__nv_bfloat16>(__nv_bfloat16* p, long long i, float v) {
  p[i] = __float2bfloat16(v);
}
template <> __device__ __forceinline__ void scan_st<__half>(__half* p, long long i, float v) { p[i] = __float2half(v); }
//
// Bound by HBM once enough loads are in flight; the recurrence itself is one FMA a step.  So a block's eight
// warps take eight steps each of the same 32 * VEC channels: every warp requests its steps of the next
// 64-step tile, waits for the state from the warp before it (a named barrier and one shared-memory slot),
// runs its eight FMAs in step order, hands the state on and stores.  The sums are those of a serial loop, but
// the loads of 64 steps are in flight instead of one.  bf16, 256 x 512 x 256: forward 60 us = 5.6 TB/s (one
// thread a channel: 97, and 27 to convert the states), backward 83 us = 4.9 TB/s (189); 2 x 129 x 96 in fp32:
// 5 and 5 us (12 and 15).
constexpr int PS_U = 8, PS_NW = 8, PS_TT = PS_U * PS_NW;

// VEC channels of one step as they were loaded.  They stay one register word until they are used: taking a
// pair of 16-bit values apart at the load would wait for each load where it is issued.
template <typename T, int VEC> struct ScanRaw;
template <> struct ScanRaw<float, 1> { using type = float; };
template <> struct ScanRaw<float, 2> { using type = float2; };
template <> struct ScanRaw<__nv_bfloat16, 1> { using type = unsigned short; };
template <> struct ScanRaw<__nv_bfloat16, 2> { using type = unsigned int; };
template <> struct ScanRaw<__half, 1> { using type = unsigned short; };
template <> struct ScanRaw<__half, 2> { using type = unsigned int; };
template <typename T, int VEC> using scan_raw = typename ScanRaw<T, VEC>::type;

template <typename T, int VEC>
__device__ __forceinline__ scan_raw<T, VEC> raw_ld(const T* p) { return __ldg(reinterpret_cast<const scan_raw<T, VEC>*>(p)); }
template <typename T, int VEC>
__device__ __forceinline__ void raw_get(const scan_raw<T, VEC>& q, float (&f)[VEC]) {
  const T* v = reinterpret_cast<const T*>(&q);
#pragma unroll
  for (int i = 0; i < VEC; ++i) f[i] = scan_ld(v, i);
}
template <typename T, int VEC>
__device__ __forceinline__ void raw_st(T* p, const float (&f)[VEC]) {
  scan_raw<T, VEC> q;
  T* v = reinterpret_cast<T*>(&q);
#pragma unroll
  for (int i = 0; i < VEC; ++i) scan_st(v, i, f[i]);
  *reinterpret_cast<scan_raw<T, VEC>*>(p) = q;
}

// The state's way through the warps of a block: warp w receives on barrier 1 + w and hands on to 1 + (w + 1) % 8.
// A barrier takes one warp's arrival and one warp's wait; it is used again only after the state has gone round.
template <int VEC>
__device__ __forceinline__ void chain_recv(const float (&slot)[PS_NW][32 * VEC], int warp, int lane, float (&s)[VEC]) {
  asm volatile("barrier.cta.sync %0, 64;" ::"r"(1 + warp) : "memory");
#pragma unroll
  for (int i = 0; i < VEC; ++i) s[i] = slot[warp][lane * VEC + i];
}
template <int VEC>
__device__ __forceinline__ void chain_send(float (&slot)[PS_NW][32 * VEC], int warp, int lane, const float (&s)[VEC]) {
  const int to = (warp + 1) % PS_NW;
#pragma unroll
  for (int i = 0; i < VEC; ++i) slot[to][lane * VEC + i] = s[i];
  asm volatile("barrier.cta.arrive %0, 64;" ::"r"(1 + to) : "memory");
}

// states (fp32) and out (the update's type) are both optional.
template <typename DT, typename UT, int VEC>
__global__ void __launch_bounds__(32 * PS_NW, VEC * (sizeof(DT) + sizeof(UT)) > 12 ? 2 : 3)
plain_scan_fwd_kernel(const DT* __restrict__ decay, const UT* __restrict__ update,
                      const float* __restrict__ h0, float* __restrict__ states, UT* __restrict__ out, int T, int D) {
  __shared__ float slot[PS_NW][32 * VEC];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.y;
  const int d = (blockIdx.x * 32 + lane) * VEC;
  const bool on = d < D;
  const long long base = (long long)b * T * D + d;
  scan_raw<DT, VEC> dn[PS_U] = {};
  scan_raw<UT, VEC> un[PS_U] = {};
  auto fetch = [&](int t0) {
#pragma unroll
    for (int u = 0; u < PS_U; ++u) {
      if (on && t0 + u < T) {
        dn[u] = raw_ld<DT, VEC>(decay + base + (long long)(t0 + u) * D);
        un[u] = raw_ld<UT, VEC>(update + base + (long long)(t0 + u) * D);
      }
    }
  };
  fetch(warp * PS_U);
  for (int t0 = 0; t0 < T; t0 += PS_TT) {
    const int tw = t0 + warp * PS_U;
    const bool more = t0 + PS_TT < T;
    scan_raw<DT, VEC> dc[PS_U];
    scan_raw<UT, VEC> uc[PS_U];
#pragma unroll
    for (int u = 0; u < PS_U; ++u) { dc[u] = dn[u]; uc[u] = un[u]; }
    if (more) fetch(tw + PS_TT);
    float s[VEC], st[PS_U][VEC];
    if (t0 == 0 && warp == 0) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) s[i] = (h0 && on) ? h0[(long long)b * D + d + i] : 0.f;
    } else {
      chain_recv<VEC>(slot, warp, lane, s);
    }
#pragma unroll
    for (int u = 0; u < PS_U; ++u) {
      if (tw + u < T) {
        float df[VEC], uf[VEC];
        raw_get<DT, VEC>(dc[u], df);
        raw_get<UT, VEC>(uc[u], uf);
#pragma unroll
        for (int i = 0; i < VEC; ++i) s[i] = fmaf(df[i], s[i], uf[i]);
      }
#pragma unroll
      for (int i = 0; i < VEC; ++i) st[u][i] = s[i];
    }
    if (warp < PS_NW - 1 || more) chain_send<VEC>(slot, warp, lane, s);
#pragma unroll
    for (int u = 0; u < PS_U; ++u) {
      if (on && tw + u < T) {
        const long long o = base + (long long)(tw + u) * D;
        if (states) raw_st<float, VEC>(states + o, st[u]);
        if (out) raw_st<UT, VEC>(out + o, st[u]);
      }
    }
  }
}

// gstates / gupdate in the update dtype, gdecay in the decay dtype.
template <typename DT, typename UT, int VEC>
__global__ void __launch_bounds__(32 * PS_NW, VEC == 2 ? 2 : 3)
plain_scan_bwd_kernel(const DT* __restrict__ decay, const float* __restrict__ states,
                      const float* __restrict__ h0, const UT* __restrict__ gstates,
                      DT* __restrict__ gdecay, UT* __restrict__ gupdate,
                      float* __restrict__ gh0, int T, int D) {
  __shared__ float slot[PS_NW][32 * VEC];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.y;
  const int d = (blockIdx.x * 32 + lane) * VEC;
  const bool on = d < D;
  const long long base = (long long)b * T * D + d;
  // `g` (not g * decay) goes from step to step, as in the serial loop's g[t] = go[t] + g[t+1] * decay[t+1]: one
  // rounding a step.  So a warp also reads the decay of the step before its first (dl).
  scan_raw<DT, VEC> dn[PS_U] = {}, dl = {};
  scan_raw<UT, VEC> gn[PS_U] = {};
  scan_raw<float, VEC> pn[PS_U] = {};       // the state before each step
  // step u of the warp whose steps start at position j0 of the reversed order is t = T - 1 - (j0 + u)
  auto fetch = [&](int j0) {
#pragma unroll
    for (int u = 0; u < PS_U; ++u) {
      const int t = T - 1 - (j0 + u);
      if (on && t >= 0) {
        const long long o = base + (long long)t * D;
        dn[u] = raw_ld<DT, VEC>(decay + o);
        gn[u] = raw_ld<UT, VEC>(gstates + o);
        pn[u] = raw_ld<float, VEC>(states + (t > 0 ? o - D : o));     // step 0: replaced by h0 where it is used
      }
    }
    if (on && j0 > 0 && j0 <= T) dl = raw_ld<DT, VEC>(decay + base + (long long)(T - j0) * D);
  };
  fetch(warp * PS_U);
  float g[VEC];                             // dL/d state of the step before (later in time)
#pragma unroll
  for (int i = 0; i < VEC; ++i) g[i] = 0.f;
  for (int j0 = 0; j0 < T; j0 += PS_TT) {
    const int jw = j0 + warp * PS_U;
    const bool more = j0 + PS_TT < T;
    scan_raw<DT, VEC> dc[PS_U], dlc = dl;
    scan_raw<UT, VEC> gc[PS_U];
    scan_raw<float, VEC> pc[PS_U];
#pragma unroll
    for (int u = 0; u < PS_U; ++u) { dc[u] = dn[u]; gc[u] = gn[u]; pc[u] = pn[u]; }
    if (more) fetch(jw + PS_TT);
    if (jw > 0) chain_recv<VEC>(slot, warp, lane, g);
    float gs[PS_U][VEC], dp[VEC];
    raw_get<DT, VEC>(dlc, dp);
#pragma unroll
    for (int u = 0; u < PS_U; ++u) {
      if (jw + u < T) {
        float gf[VEC];
        raw_get<UT, VEC>(gc[u], gf);
#pragma unroll
        for (int i = 0; i < VEC; ++i) g[i] = jw + u > 0 ? fmaf(g[i], dp[i], gf[i]) : gf[i];
        raw_get<DT, VEC>(dc[u], dp);
      }
#pragma unroll
      for (int i = 0; i < VEC; ++i) gs[u][i] = g[i];
    }
    if (warp < PS_NW - 1 || more) chain_send<VEC>(slot, warp, lane, g);
#pragma unroll
    for (int u = 0; u < PS_U; ++u) {
      const int t = T - 1 - (jw + u);
      if (on && t >= 0) {
        const long long o = base + (long long)t * D;
        float gd[VEC], pf[VEC];
        raw_get<float, VEC>(pc[u], pf);
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          if (t == 0) pf[i] = h0 ? h0[(long long)b * D + d + i] : 0.f;
          gd[i] = gs[u][i] * pf[i];
        }
        raw_st<UT, VEC>(gupdate + o, gs[u]);
        raw_st<DT, VEC>(gdecay + o, gd);
        if (gh0 && t == 0) {
          float d0[VEC];
          raw_get<DT, VEC>(dc[u], d0);
#pragma unroll
          for (int i = 0; i < VEC; ++i) gh0[(long long)b * D + d + i] = gs[u][i] * d0[i];
        }
      }
    }
  }
}

// The same recurrence, one thread to VEC channels for all steps: for short sequences, where most warps of the
// kernels above have no step and only pass the state on (the rule is at plain_scan_serial).  Same arithmetic, same bits.
template <typename DT, typename UT, int VEC>
__global__ void __launch_bounds__(SCAN_THREADS)
plain_scan_serial_fwd_kernel(const DT* __restrict__ decay, const UT* __restrict__ update, const float* __restrict__ h0,
                             float* __restrict__ states, UT* __restrict__ out, int T, int D) {
  const int b = blockIdx.y, d = (blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (d >= D) return;
  float s[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) s[i] = h0 ? h0[(long long)b * D + d + i] : 0.f;
  long long o = (long long)b * T * D + d;
  for (int t = 0; t < T; ++t, o += D) {
    float df[VEC], uf[VEC];
    raw_get<DT, VEC>(raw_ld<DT, VEC>(decay + o), df);
    raw_get<UT, VEC>(raw_ld<UT, VEC>(update + o), uf);
#pragma unroll
    for (int i = 0; i < VEC; ++i) s[i] = fmaf(df[i], s[i], uf[i]);
    if (states) raw_st<float, VEC>(states + o, s);
    if (out) raw_st<UT, VEC>(out + o, s);
  }
}

template <typename DT, typename UT, int VEC>
__global__ void __launch_bounds__(SCAN_THREADS)
plain_scan_serial_bwd_kernel(const DT* __restrict__ decay, const float* __restrict__ states,
                             const float* __restrict__ h0, const UT* __restrict__ gstates,
                             DT* __restrict__ gdecay, UT* __restrict__ gupdate, float* __restrict__ gh0, int T, int D) {
  const int b = blockIdx.y, d = (blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (d >= D) return;
  const long long base = (long long)b * T * D + d;
  float g[VEC], dp[VEC];
  for (int t = T - 1; t >= 0; --t) {
    const long long o = base + (long long)t * D;
    float gf[VEC], pf[VEC], gd[VEC];
    raw_get<UT, VEC>(raw_ld<UT, VEC>(gstates + o), gf);
    if (t > 0) {
      raw_get<float, VEC>(raw_ld<float, VEC>(states + o - D), pf);
    } else {
#pragma unroll
      for (int i = 0; i < VEC; ++i) pf[i] = h0 ? h0[(long long)b * D + d + i] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      g[i] = t < T - 1 ? fmaf(g[i], dp[i], gf[i]) : gf[i];
      gd[i] = g[i] * pf[i];
    }
    raw_get<DT, VEC>(raw_ld<DT, VEC>(decay + o), dp);
    raw_st<UT, VEC>(gupdate + o, g);
    raw_st<DT, VEC>(gdecay + o, gd);
  }
  if (gh0) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) gh0[(long long)b * D + d + i] = g[i] * dp[i];
  }
}

}  // namespace ccb

using namespace ccb;

// Arithmetic of the fused scan kernels: 0 scalar fp32; 1 scalar with the gate exponentials as an FMA-pipe
// polynomial (measured slower: the kernels are bound by instruction issue, not by the special-function
// unit); 2 packed fp32x2.  Returns the old value.
static int g_scan_poly_exp = 2;
extern "C" int ccb_scan_poly_exp(int mode) {
  const int old = g_scan_poly_exp;
  if (mode >= 0 && mode <= 2) g_scan_poly_exp = mode;
  return old;
}

template <typename K, typename... A>
static int launch_tile(K kern, int cl, int threads, int64_t B, int64_t D, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((D / 2 + 31) / 32), (unsigned)B, (unsigned)cl);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = (unsigned)cl;
  cfg.attrs = at; cfg.numAttrs = cl > 1 ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  count_launch();
  return e == cudaSuccess ? 0 : set_error("scan launch: %s", cudaGetErrorString(e));
}

template <int U, int NW, int MINB, int CL>
static int launch_tile_fwd(const void* P, int64_t ldp, const float* log_a, const float* h0, void* y, void* hout, float* hT,
                           int64_t B, int64_t T, int64_t D, int64_t la_bstride, cudaStream_t stream) {
  return launch_tile(scan_tile_fwd_kernel<U, NW, MINB, CL>, CL, 32 * NW, B, D, stream, (const __nv_bfloat16*)P,
                     (long long)ldp, log_a, h0, (__nv_bfloat16*)y, (__nv_bfloat16*)hout, hT, (int)T, (int)D,
                     (long long)la_bstride);
}

template <int U, int NW, int MINB, int CL>
static int launch_tile_bwd(const void* P, int64_t ldp, const float* log_a, const float* h0, const void* hstates,
                           const void* dy, const float* dhT, const float* rowss, float inv_dim, float eps, void* dP,
                           int64_t lddp, float* dloga_part, float* dh0, int64_t B, int64_t T, int64_t D,
                           int64_t la_bstride, cudaStream_t stream) {
  return launch_tile(scan_tile_bwd_kernel<U, NW, MINB, CL>, CL, 32 * NW, B, D, stream, (const __nv_bfloat16*)P,
                     (long long)ldp, log_a, h0, (const __nv_bfloat16*)hstates, (const __nv_bfloat16*)dy, dhT, rowss,
                     inv_dim, eps, (__nv_bfloat16*)dP, (long long)lddp, dloga_part, dh0, (int)T, (int)D,
                     (long long)la_bstride);
}

// Which scan.  `warps` = 64-channel warps of the whole batch.  A serial thread needs every SM full of them to
// hide a step's latency; measured on a B200, T = 512, D = 256, serial / time-tiled in us (events, cold L2):
//   forward   B = 1: 117 / 11   64: 126 / 32   256: 146 / 91    512: 189 / 167   1024: 283 / 318
//   backward  B = 1: 181 / 20   64: 191 / 63   256: 228 / 185   512: 318 / 353   1024: 576 / 687
// so the line lies at 16 (forward) and 8 (backward) warps per SM.  Below 64 steps a tile is partly empty and the
// line is nearer.  4 warps per SM: T = 32 15 / 14 and 24 / 20, T = 24 12 / 12 and 20 / 20; T = 16 10 / 12 and 17 / 17,
// T = 1 8 / 10 and 13 / 15.  2 per SM: T = 16 10 / 10 and 17 / 13, T = 8 8 / 8 and 13 / 13.  8 per SM: T = 32 16 / 21 and
// 28 / 28, T = 16 12 / 18 and 19 / 24.
static bool scan_tiled(int64_t warps, int64_t T, int per_sm) {
  return g_scan_poly_exp == 2 && warps <= (int64_t)(T >= 64 ? per_sm : (T >= 24 ? 4 : 2)) * ccb_num_sms();
}
// Blocks of a cluster: while they fit two to an SM and each still has steps (B = 1: 23 us with one block, 11 with
// eight; 16 rows of 256 channels: 25 with one, 17 with four, 19 with eight).
static int scan_cluster(int64_t warps, int64_t T, int tile) {
  int cl = 8;
  while (cl > 1 && (warps * cl > 2 * ccb_num_sms() || (int64_t)tile * (cl / 2) >= T)) cl /= 2;
  return cl;
}

extern "C" int ccb_scan_fwd(const void* P, int64_t ldp, const float* log_a, const float* h0,
                            void* y, void* hout, float* hT, int64_t B, int64_t T, int64_t D,
                            int64_t la_bstride, void* stream) {
  if (B <= 0 || T <= 0) return 0;
  if (D % 8 != 0 || ldp % 2 != 0) return set_error("ccb_scan_fwd: D must be a multiple of 8");
  dim3 grid((unsigned)((D / 2 + SCAN_THREADS - 1) / SCAN_THREADS), (unsigned)B);
  const int64_t warps = B * ((D + 63) / 64);
  if (scan_tiled(warps, T, 16)) {
    auto launch = launch_tile_fwd<8, 8, 2, 1>;
    switch (scan_cluster(warps, T, 64)) {
      case 8: launch = launch_tile_fwd<8, 8, 2, 8>; break;
      case 4: launch = launch_tile_fwd<8, 8, 2, 4>; break;
      case 2: launch = launch_tile_fwd<8, 8, 2, 2>; break;
    }
    return launch(P, ldp, log_a, h0, y, hout, hT, B, T, D, la_bstride, (cudaStream_t)stream);
  }
  // forward: six steps loaded ahead and six resident blocks per SM (72 registers) measured best: 0.286 ms at
  // 524 288 rows against 0.311 ms with eight steps ahead and four blocks
  auto kern = g_scan_poly_exp == 2 ? scan_fwd_kernel<2, 6, 6> : (g_scan_poly_exp == 1 ? scan_fwd_kernel<1> : scan_fwd_kernel<0>);
  kern<<<grid, SCAN_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)P, ldp, log_a, h0, (__nv_bfloat16*)y, (__nv_bfloat16*)hout, hT, (int)T,
      (int)D, (long long)la_bstride);
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : set_error("scan_fwd launch: %s", cudaGetErrorString(e));
}

extern "C" int ccb_scan_bwd(const void* P, int64_t ldp, const float* log_a, const float* h0,
                            const void* hstates, const void* dy, const float* dhT,
                            const float* rowss, float inv_dim, float eps, void* dP, int64_t lddp,
                            float* dloga_part, float* dh0, int64_t B, int64_t T, int64_t D,
                            int64_t la_bstride, void* stream) {
  if (B <= 0 || T <= 0) return 0;
  if (D % 8 != 0) return set_error("ccb_scan_bwd: D must be a multiple of 8");
  dim3 grid((unsigned)((D / 2 + SCAN_THREADS - 1) / SCAN_THREADS), (unsigned)B);
  const int64_t warps = B * ((D + 63) / 64);
  if (scan_tiled(warps, T, 8)) {
    auto launch = launch_tile_bwd<4, 8, 2, 1>;
    switch (scan_cluster(warps, T, 32)) {
      case 8: launch = launch_tile_bwd<4, 8, 2, 8>; break;
      case 4: launch = launch_tile_bwd<4, 8, 2, 4>; break;
      case 2: launch = launch_tile_bwd<4, 8, 2, 2>; break;
    }
    return launch(P, ldp, log_a, h0, hstates, dy, dhT, rowss, inv_dim, eps, dP, lddp, dloga_part, dh0, B, T, D,
                  la_bstride, (cudaStream_t)stream);
  }
  // backward: eight steps ahead, four blocks per SM (116 registers): 0.538 ms; six blocks with six / four steps
  // ahead measured 0.632 / 0.706 ms (fewer loads in flight cost more than the extra warps bring)
  auto kern = g_scan_poly_exp == 2 ? scan_bwd_kernel<2> : (g_scan_poly_exp == 1 ? scan_bwd_kernel<1> : scan_bwd_kernel<0>);
  kern<<<grid, SCAN_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)P, ldp, log_a, h0, (const __nv_bfloat16*)hstates,
      (const __nv_bfloat16*)dy, dhT, rowss, inv_dim, eps, (__nv_bfloat16*)dP, lddp, dloga_part, dh0,
      (int)T, (int)D, (long long)la_bstride);
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : set_error("scan_bwd launch: %s", cudaGetErrorString(e));
}

// dtype codes: 0 = fp32, 1 = bf16, 2 = fp16.  Accepted (decay, update) pairs: (1,1) (1,2) (2,2) (0,0) (0,1) (0,2).
static inline bool plain_scan_combo_ok(int64_t dd, int64_t ud) {
  return (dd == 1 && ud == 1) || (dd == 1 && ud == 2) || (dd == 2 && ud == 2) || (dd == 0 && ud >= 0 && ud <= 2);
}
#define CCB_SCAN_DISPATCH(dd, ud, ...)                                                     \
  do {                                                                                      \
    if (dd == 0 && ud == 0) { using DT = float; using UT = float; __VA_ARGS__; }                   \
    else if (dd == 0 && ud == 1) { using DT = float; using UT = __nv_bfloat16; __VA_ARGS__; }      \
    else if (dd == 0 && ud == 2) { using DT = float; using UT = __half; __VA_ARGS__; }             \
    else if (dd == 1 && ud == 1) { using DT = __nv_bfloat16; using UT = __nv_bfloat16; __VA_ARGS__; } \
    else if (dd == 1 && ud == 2) { using DT = __nv_bfloat16; using UT = __half; __VA_ARGS__; }     \
    else { using DT = __half; using UT = __half; __VA_ARGS__; }                                    \
  } while (0)

// Two channels to a lane where every row starts on a pair's boundary.
static inline bool plain_scan_pairs(int64_t D, int64_t dd, int64_t ud, const void* dec, const void* dec2, const void* upd,
                                    const void* upd2, const float* st) {
  const uintptr_t da = dd == 0 ? 7 : 3, ua = ud == 0 ? 7 : 3;
  return D % 2 == 0 && (((uintptr_t)dec | (uintptr_t)dec2) & da) == 0 && (((uintptr_t)upd | (uintptr_t)upd2) & ua) == 0 &&
         ((uintptr_t)st & 7) == 0;
}

// Whether one thread takes all steps.  A block of the eight-warp kernels costs its hand-over chain whatever the number of
// steps (2 us forward and 3 backward for every 440 of them), the serial kernels cost a step's latency T times.  Measured
// on a B200, D = 256, bf16, eight warps / serial in us, forward and backward (events, cold L2; blocks = B x D / 64):
//   T = 1:  64 rows 8 / 6, 7 / 7         1024 rows 25 / 6, 34 / 6       4096 rows 76 / 8, 117 / 8
//   T = 8:  64 rows 8 / 8, 8 / 11         256 rows 12 / 8, 15 / 12      4096 rows 84 / 20, 139 / 27
//   T = 32: 256 rows 12 / 14, 16 / 25     512 rows 18 / 16, 27 / 27     1024 rows 31 / 20, 45 / 35
//   T = 48: 512 rows 20 / 20, 29 / 39    1024 rows 33 / 29, 51 / 47     2048 rows 57 / 51, 90 / 61
static bool plain_scan_serial(int64_t B, int64_t T, int64_t lanes, int64_t blocks_per_step) {
  return T < PS_TT && B * ((lanes + 31) / 32) > blocks_per_step * T;
}
// Threads of a serial block: narrow rows do not leave warps idle.
static int64_t plain_scan_threads(int64_t lanes) { return lanes < SCAN_THREADS ? (lanes + 31) / 32 * 32 : SCAN_THREADS; }

// states: fp32 (kept for backward), out: the states in the update's dtype; either may be null.
extern "C" int ccb_plain_scan_fwd(const void* decay, int64_t decay_dtype, const void* update,
                                  int64_t update_dtype, const float* h0, float* states, void* out, int64_t B,
                                  int64_t T, int64_t D, void* stream) {
  if (B <= 0 || T <= 0 || D <= 0) return 0;
  if (!plain_scan_combo_ok(decay_dtype, update_dtype))
    return set_error("ccb_plain_scan_fwd: (decay, update) dtype pair (%lld, %lld) is not supported",
                     (long long)decay_dtype, (long long)update_dtype);
  const bool pairs = plain_scan_pairs(D, decay_dtype, update_dtype, decay, decay, update, out ? out : update, states);
  const int64_t lanes = pairs ? D / 2 : D;
  const bool serial = plain_scan_serial(B, T, lanes, 48);
  const int64_t width = serial ? plain_scan_threads(lanes) : 32;       // lanes of a block
  dim3 grid((unsigned)((lanes + width - 1) / width), (unsigned)B);
  CCB_SCAN_DISPATCH(decay_dtype, update_dtype, {
    auto kern = serial ? (pairs ? plain_scan_serial_fwd_kernel<DT, UT, 2> : plain_scan_serial_fwd_kernel<DT, UT, 1>)
                       : (pairs ? plain_scan_fwd_kernel<DT, UT, 2> : plain_scan_fwd_kernel<DT, UT, 1>);
    kern<<<grid, (unsigned)(serial ? width : 32 * PS_NW), 0, (cudaStream_t)stream>>>((const DT*)decay, (const UT*)update, h0, states, (UT*)out, (int)T,
                                                        (int)D);
  });
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : set_error("plain_scan_fwd launch: %s", cudaGetErrorString(e));
}

extern "C" int ccb_plain_scan_bwd(const void* decay, int64_t decay_dtype, const float* states,
                                  const float* h0, const void* gstates, int64_t update_dtype,
                                  void* gdecay, void* gupdate, float* gh0, int64_t B, int64_t T,
                                  int64_t D, void* stream) {
  if (B <= 0 || T <= 0 || D <= 0) return 0;
  if (!plain_scan_combo_ok(decay_dtype, update_dtype))
    return set_error("ccb_plain_scan_bwd: (decay, update) dtype pair (%lld, %lld) is not supported",
                     (long long)decay_dtype, (long long)update_dtype);
  const bool pairs = plain_scan_pairs(D, decay_dtype, update_dtype, decay, gdecay, gstates, gupdate, states);
  const int64_t lanes = pairs ? D / 2 : D;
  const bool serial = plain_scan_serial(B, T, lanes, 80);
  const int64_t width = serial ? plain_scan_threads(lanes) : 32;
  dim3 grid((unsigned)((lanes + width - 1) / width), (unsigned)B);
  CCB_SCAN_DISPATCH(decay_dtype, update_dtype, {
    auto kern = serial ? (pairs ? plain_scan_serial_bwd_kernel<DT, UT, 2> : plain_scan_serial_bwd_kernel<DT, UT, 1>)
                       : (pairs ? plain_scan_bwd_kernel<DT, UT, 2> : plain_scan_bwd_kernel<DT, UT, 1>);
    kern<<<grid, (unsigned)(serial ? width : 32 * PS_NW), 0, (cudaStream_t)stream>>>((const DT*)decay, states, h0, (const UT*)gstates, (DT*)gdecay,
                                                        (UT*)gupdate, gh0, (int)T, (int)D);
  });
  count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : set_error("plain_scan_bwd launch: %s", cudaGetErrorString(e));
}
