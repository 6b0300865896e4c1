// Bandwidth-bound helpers around the GEMMs: embedding gather with fused row
// sum-of-squares, sorted scatter-add embedding backward, split-K reduction with
// the RMSNorm-weight fold, standalone RMSNorm (fwd/bwd) for callers outside
// the fused trunk, optimizer updates (Muon momentum / apply, AdamW, LAMB
// moments), global grad-norm clip, casts and the SGD step used by test-time
// training.  Everything is vectorised to 16-byte accesses where shapes allow.
//
// Reference counterparts: kernels/_lm_head_loss/src/rms_norm.cu:23-112 (RMSNorm),
// optim/muon.py:390-448 and 540-658 (Muon / AdamW updates),
// distributed.py:175-216 (fused grad clip).
#include "ptx.cuh"
#include "ccb_api.h"
#include "runtime.h"
#include <type_traits>

namespace ccb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float block_sum(float v, float* sm) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (l == 0) sm[w] = v;
  __syncthreads();
  float r = (threadIdx.x < nw) ? sm[threadIdx.x] : 0.f;
  if (w == 0) r = warp_sum(r);
  if (threadIdx.x == 0) sm[0] = r;
  __syncthreads();
  return sm[0];
}

// ---------------------------------------------------------------------------
// Embedding forward: x[r, :] = E[tok[r], :], ss[r] = sum x^2.  One warp per row.
// ---------------------------------------------------------------------------
template <typename TokT>
__global__ void embed_fwd_kernel(const TokT* __restrict__ tok, const __nv_bfloat16* __restrict__ E,
                                 __nv_bfloat16* __restrict__ x, float* __restrict__ ss, long long R,
                                 int D, int V) {
  const long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= R) return;
  const int lane = threadIdx.x & 31;
  long long t = (long long)tok[r];
  t = t < 0 ? 0 : (t >= V ? V - 1 : t);
  const uint4* src = reinterpret_cast<const uint4*>(E + t * D);
  uint4* dst = reinterpret_cast<uint4*>(x + r * D);
  float acc = 0.f;
  for (int c = lane; c < D / 8; c += 32) {
    uint4 q = __ldg(src + c);
    dst[c] = q;
    float2 f;
    f = unpack_bf16x2(q.x); acc += f.x * f.x + f.y * f.y;
    f = unpack_bf16x2(q.y); acc += f.x * f.x + f.y * f.y;
    f = unpack_bf16x2(q.z); acc += f.x * f.x + f.y * f.y;
    f = unpack_bf16x2(q.w); acc += f.x * f.x + f.y * f.y;
  }
  acc = warp_sum(acc);
  if (lane == 0 && ss) ss[r] = acc;
}

// ---------------------------------------------------------------------------
// Embedding backward over token-sorted rows, bit-reproducible (no atomics).
//
// Stage 1: each warp owns CH = 32 consecutive sorted positions and sums the
// rows of each run of equal tokens in position order.  A run that lies wholly
// inside the chunk has one owner and is stored straight to dE.  A run that
// continues from the previous chunk or into the next one is written to the
// chunk's boundary slot instead: slot 0 for a run that starts at the chunk's
// first position, slot 1 for a run that starts later and runs off its end.
// Stage 1 also records, per token, the first and the last sorted position it occupies.
// Stage 2: one block per token whose rows span several chunks adds the
// boundary slots of those chunks in chunk order and stores the row of dE.
// The summation order is a function of the sorted token array alone, so two
// runs over the same batch give the same bits (the sort must be stable for
// `perm` itself to be reproducible).  dE must be zeroed by the caller: rows of
// tokens that do not occur are never written.
// ---------------------------------------------------------------------------
constexpr int EMB_CH = 32;

// Sort keys: the token, or -1 / V for one below / above the table (its rows belong to no gradient; the order stays that
// of the tokens).  Two bytes instead of eight leave a radix sort two passes instead of eight.
template <typename TokT>
__global__ void token_keys_kernel(const TokT* __restrict__ tok, short* __restrict__ key, long long R, int V) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < R; i += (long long)gridDim.x * blockDim.x) {
    const long long t = (long long)tok[i];
    key[i] = (short)(t < 0 ? -1 : (t < V ? t : V));
  }
}

template <int VPL, typename TokT>   // VPL uint4 vectors per lane: D = 256 * VPL
__global__ void embed_bwd_runs_kernel(const TokT* __restrict__ sorted_tok,
                                      const long long* __restrict__ perm,
                                      const __nv_bfloat16* __restrict__ dx,
                                      float* __restrict__ dE, float* __restrict__ slots,
                                      long long* __restrict__ first_pos,
                                      long long* __restrict__ last_pos, long long R, int D, int V) {
  const long long chunk = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long p0 = chunk * EMB_CH;
  if (p0 >= R) return;
  const long long p1 = (p0 + EMB_CH < R) ? p0 + EMB_CH : R;
  const int lane = threadIdx.x & 31;
  const int n = (int)(p1 - p0);
  // one coalesced load of the chunk's tokens and row indices, handed round by shuffles
  const long long my_tok = (lane < n) ? (long long)sorted_tok[p0 + lane] : -1;
  const long long my_row = (lane < n) ? perm[p0 + lane] : 0;
  const long long tok_before = (p0 > 0) ? (long long)sorted_tok[p0 - 1] : -1;
  const long long tok_after = (p1 < R) ? (long long)sorted_tok[p1] : -1;
  {
    // token boundaries: where a token's rows begin and end in the sorted order
    long long prev = __shfl_up_sync(0xffffffffu, my_tok, 1);
    long long next = __shfl_down_sync(0xffffffffu, my_tok, 1);
    if (lane == 0) prev = tok_before;
    if (lane == n - 1) next = tok_after;
    if (lane < n && my_tok >= 0 && my_tok < V) {
      if (prev != my_tok) first_pos[my_tok] = p0 + lane;
      if (next != my_tok) last_pos[my_tok] = p0 + lane;
    }
  }
  float acc[VPL][8];
#pragma unroll
  for (int v = 0; v < VPL; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
  long long cur = __shfl_sync(0xffffffffu, my_tok, 0);
  int run_start = 0;
  auto flush = [&](long long tk, int a, int b) {
    // run of token tk over chunk positions [a, b)
    if (tk < 0 || tk >= V) return;
    const bool open_left = (a == 0) && (tok_before == tk);
    const bool open_right = (b == n) && (tok_after == tk);
    float* o;
    if (!open_left && !open_right) o = dE + tk * D;
    else o = slots + (chunk * 2 + (a == 0 ? 0 : 1)) * (long long)D;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      float4* o4 = reinterpret_cast<float4*>(o + (v * 32 + lane) * 8);
      o4[0] = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
      o4[1] = make_float4(acc[v][4], acc[v][5], acc[v][6], acc[v][7]);
    }
  };
  for (int j0 = 0; j0 < n; j0 += 4) {
    // four rows are requested before any is added: the adds stay in position order
    uint4 q[4][VPL];
    long long tk[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u;
      tk[u] = __shfl_sync(0xffffffffu, my_tok, j & 31);
      const long long row = __shfl_sync(0xffffffffu, my_row, j & 31);
      if (j < n) {
        const uint4* src = reinterpret_cast<const uint4*>(dx + row * D);
#pragma unroll
        for (int v = 0; v < VPL; ++v) q[u][v] = __ldg(src + v * 32 + lane);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u;
      if (j >= n) break;
      if (tk[u] != cur) {
        flush(cur, run_start, j);
#pragma unroll
        for (int v = 0; v < VPL; ++v)
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
        cur = tk[u];
        run_start = j;
      }
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        float2 f;
        f = unpack_bf16x2(q[u][v].x); acc[v][0] += f.x; acc[v][1] += f.y;
        f = unpack_bf16x2(q[u][v].y); acc[v][2] += f.x; acc[v][3] += f.y;
        f = unpack_bf16x2(q[u][v].z); acc[v][4] += f.x; acc[v][5] += f.y;
        f = unpack_bf16x2(q[u][v].w); acc[v][6] += f.x; acc[v][7] += f.y;
      }
    }
  }
  flush(cur, run_start, n);
}

// A token's boundary slots k = w, w + 16, ... are added by warp w in order (lane l owns columns
// [l * D/32, (l+1) * D/32)) and the sixteen sums are added in warp order: a fixed tree, wide enough that the most
// frequent token of a Zipf batch (thousands of chunks) does not serialise behind one warp.  Up to sixteen slots the
// tree is a plain sum in slot order, which one warp does by itself.  So a block takes up to JOIN_TOKS tokens, a grid
// apart so that neighbouring ids (frequent ones come together) spread over blocks: its warps take the short ones side
// by side, then all of them each long one.  A block of sixteen warps per token, most of which had nothing to join,
// took 44 us at 32 768 rows and V = 16 384; 10 now.  A small vocabulary has few tokens and all of them long: its blocks
// take fewer, four blocks to an SM.  With 32 tokens to a block 262 144 rows over 256 words ran on 8 SMs (runs and join
// 102 us, one token to a block 53).
// first_pos / last_pos come from stage 1; last_pos is -1 for tokens that do not occur.
constexpr int EMB_JOIN_WARPS = 16, EMB_JOIN_TOKS = 32;
template <int FPL>   // floats per lane: D = 32 * FPL
__global__ void __launch_bounds__(EMB_JOIN_WARPS * 32)
embed_bwd_join_kernel(const long long* __restrict__ first_pos, const long long* __restrict__ last_pos,
                      const float* __restrict__ slots, float* __restrict__ dE, int D, int V, int toks) {
  extern __shared__ float sm_join[];          // [EMB_JOIN_WARPS][D]
  __shared__ long long s_first[EMB_JOIN_TOKS], s_n[EMB_JOIN_TOKS];     // first position; slots to add (0: none)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = lane * FPL;
  if (threadIdx.x < toks) {
    const long long tk = (long long)blockIdx.x + (long long)threadIdx.x * gridDim.x;
    long long s = 0, n = 0;
    if (tk < V) {
      const long long e = last_pos[tk] + 1;
      if (e > 0) {
        s = first_pos[tk];
        const long long cs = s / EMB_CH, ce = (e - 1) / EMB_CH;
        if (cs != ce) n = ce - cs + 1;        // one owner: stored by stage 1
      }
    }
    s_first[threadIdx.x] = s;
    s_n[threadIdx.x] = n;
  }
  __syncthreads();
  // slots of token j: chunk cs (first or second slot), then first slots
  auto slot_ptr = [&](int j, long long k) {
    const long long s = s_first[j], cs = s / EMB_CH;
    return slots + ((cs + k) * 2 + (k == 0 && s % EMB_CH != 0 ? 1 : 0)) * (long long)D + c0;
  };
  float acc[FPL];
  // adds slots k, k + step, ... in order, four in flight
  auto add_slots = [&](int j, long long k, long long n, int step) {
#pragma unroll
    for (int i = 0; i < FPL; ++i) acc[i] = 0.f;
    for (; k + 3 * step < n; k += 4 * step) {
      float4 t[4][FPL / 4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4* p = reinterpret_cast<const float4*>(slot_ptr(j, k + u * step));
#pragma unroll
        for (int i = 0; i < FPL / 4; ++i) t[u][i] = p[i];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < FPL / 4; ++i) {
          acc[4 * i] += t[u][i].x; acc[4 * i + 1] += t[u][i].y;
          acc[4 * i + 2] += t[u][i].z; acc[4 * i + 3] += t[u][i].w;
        }
    }
    for (; k < n; k += step) {
      const float4* p = reinterpret_cast<const float4*>(slot_ptr(j, k));
#pragma unroll
      for (int i = 0; i < FPL / 4; ++i) {
        const float4 v = p[i];
        acc[4 * i] += v.x; acc[4 * i + 1] += v.y; acc[4 * i + 2] += v.z; acc[4 * i + 3] += v.w;
      }
    }
  };
  for (int j = warp; j < toks; j += EMB_JOIN_WARPS) {
    const long long n = s_n[j];
    if (n == 0 || n > EMB_JOIN_WARPS) continue;
    add_slots(j, 0, n, 1);
    float4* o = reinterpret_cast<float4*>(dE + ((long long)blockIdx.x + (long long)j * gridDim.x) * D + c0);
#pragma unroll
    for (int i = 0; i < FPL / 4; ++i) o[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
  }
  for (int j = 0; j < toks; ++j) {
    const long long n = s_n[j];
    if (n <= EMB_JOIN_WARPS) continue;        // the same for the whole block
    add_slots(j, warp, n, EMB_JOIN_WARPS);
#pragma unroll
    for (int i = 0; i < FPL; ++i) sm_join[warp * D + c0 + i] = acc[i];
    __syncthreads();
    const long long tk = (long long)blockIdx.x + (long long)j * gridDim.x;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
      float t = sm_join[c];
#pragma unroll
      for (int w = 1; w < EMB_JOIN_WARPS; ++w) t += sm_join[w * D + c];
      dE[tk * D + c] = t;
    }
    __syncthreads();                          // before the next token's sums replace these
  }
}

// ---------------------------------------------------------------------------
// Split-K reduction.  out[n,k] (+)= colscale[k] * (scale *) sum_s part[s,n,k], stored as fp32 or bf16
// (the parameter's own dtype, so no cast pass follows; `scale`, one fp32 value on the device, multiplies the fp32
// sum); when W is given also emits per-row-block
// partial column sums of sum[n,k] * W[n,k] (the gradient of an RMSNorm weight folded into W),
// reduced by a second tiny kernel so the result is deterministic.
//
// Bound by the latency of the partials' loads (they sit in L2): a weight gradient of the trunk is only
// N x K = 64 K elements with S = 148 / tiles partials each.  So a block is small (8 rows x 64 columns,
// one float4 per thread) and the partials are split over G thread groups, each adding a contiguous range
// of them as a shallow tree; the groups are joined in group order through shared memory: a fixed order.  Error of
// the fp32 sums against 64 bits, relative 2-norm: 15 partials 5.4e-8, 37 6.3e-8, 74 7.6e-8 (added one after the
// other in up to eight groups 5.7, 7.3 and 8.4; without groups 7.4, 11.3 and 15.7).
// A block of 8 full rows with one thread per column (the kernel below, 32 blocks for a 256 x 256 output)
// took 630 of the 4 260 us of a 4-layer training step at 32 768 rows; with this one the step went from
// 4.51 to 4.04 ms, a 131 072-row block's forward and backward from 1.63 to 1.48 ms.
// grid: (ceil(N / 8), ceil(K / 64)); block: 128 * G threads.  K a multiple of 4, 16-byte aligned operands.
// ---------------------------------------------------------------------------
constexpr int SPK_ROWS = 8, SPK_COLS = 64;

__device__ __forceinline__ void store_grad4(float* o, float4 v) { *reinterpret_cast<float4*>(o) = v; }
__device__ __forceinline__ void store_grad4(__nv_bfloat16* o, float4 v) {
  uint2 q;
  q.x = pack_bf16x2(v.x, v.y);
  q.y = pack_bf16x2(v.z, v.w);
  *reinterpret_cast<uint2*>(o) = q;
}
__device__ __forceinline__ void store_grad1(float* o, float v) { *o = v; }
// Where row n of the result goes: one [N, K] tensor, or up to four of `rows` rows each (a packed weight whose parts are
// parameters of their own, with gradients in allocations of their own).
template <typename OT>
struct SpkOut {
  OT* p[4];
  int rows;
  __device__ __forceinline__ OT* row(int n, int K) const {
    OT* q = p[0];                              // rows = N for one tensor
    if (n >= rows) { q = p[1]; n -= rows; }
    if (n >= rows) { q = p[2]; n -= rows; }
    if (n >= rows) { q = p[3]; n -= rows; }
    return q + (long long)n * K;
  }
};
__device__ __forceinline__ void store_grad1(__nv_bfloat16* o, float v) { *o = __float2bfloat16(v); }

template <int G, typename OT>
__global__ void __launch_bounds__(128 * G)
splitk_tile_kernel(const float* __restrict__ part, int S, long long split_stride, int N, int K,
                   const __nv_bfloat16* __restrict__ colscale, const __nv_bfloat16* __restrict__ W,
                   const float* __restrict__ scale, const SpkOut<OT> out, float* __restrict__ colpart) {
  __shared__ float4 join[G > 1 ? (G - 1) * 128 : 1];
  __shared__ float4 colj[128];
  const int slot = threadIdx.x & 127, g = threadIdx.x >> 7;
  const int n = blockIdx.x * SPK_ROWS + (slot >> 4);
  const int k = blockIdx.y * SPK_COLS + (slot & 15) * 4;
  const bool ok = n < N && k < K;
  const long long o = (long long)n * K + k;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add = [&](const float4 v) { acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w; };
  if (ok) {
    const int per = (S + G - 1) / G;
    int sp = g * per;
    const int s1 = min(S, sp + per);
    const float* pp = part + o;
    // up to four at a time, the last eight in even parts, into two sums in turn: a third of the roundings of a serial sum
    float4 odd = make_float4(0.f, 0.f, 0.f, 0.f);
    for (bool even = true; sp < s1; even = !even) {
      const int left = s1 - sp, take = left >= 8 ? 4 : (left > 4 ? (left + 1) / 2 : left);
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        v[u] = u < take ? __ldg(reinterpret_cast<const float4*>(pp + (long long)(sp + u) * split_stride))
                        : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 t = make_float4((v[0].x + v[1].x) + (v[2].x + v[3].x), (v[0].y + v[1].y) + (v[2].y + v[3].y),
                                   (v[0].z + v[1].z) + (v[2].z + v[3].z), (v[0].w + v[1].w) + (v[2].w + v[3].w));
      if (even) add(t); else { odd.x += t.x; odd.y += t.y; odd.z += t.z; odd.w += t.w; }
      sp += take;
    }
    add(odd);
  }
  if (G > 1) {
    if (g > 0) join[(g - 1) * 128 + slot] = acc;
    __syncthreads();
    if (g == 0) {
#pragma unroll
      for (int j = 0; j < G - 1; ++j) add(join[j * 128 + slot]);
    }
  }
  if (g == 0) {
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ok) {
      if (scale != nullptr) {
        const float up = __ldg(scale);
        acc.x *= up; acc.y *= up; acc.z *= up; acc.w *= up;
      }
      if (W != nullptr) {
        const uint2 q = __ldg(reinterpret_cast<const uint2*>(W + o));
        const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y);
        w = make_float4(acc.x * a.x, acc.y * a.y, acc.z * b.x, acc.w * b.y);
      }
      if (colscale != nullptr) {
        const uint2 q = __ldg(reinterpret_cast<const uint2*>(colscale + k));
        const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y);
        acc.x *= a.x; acc.y *= a.y; acc.z *= b.x; acc.w *= b.y;
      }
      store_grad4(out.row(n, K) + k, acc);
    }
    if (colpart != nullptr) colj[slot] = w;
  }
  if (colpart != nullptr) {
    __syncthreads();
    const int c = blockIdx.y * SPK_COLS + threadIdx.x;
    if (threadIdx.x < SPK_COLS && c < K) {
      const float* cj = reinterpret_cast<const float*>(colj);
      float t = 0.f;
#pragma unroll
      for (int r = 0; r < SPK_ROWS; ++r) t += cj[r * SPK_COLS + threadIdx.x];
      colpart[(long long)blockIdx.x * K + c] = t;
    }
  }
}

// Any K and alignment, or accumulation into `out`: one thread per column, 8 rows in turn.
// grid: ceil(N / 8); block: 256 threads striding over k.
template <typename OT>
__global__ void splitk_reduce_kernel(const float* __restrict__ part, int S, long long split_stride,
                                     int N, int K, const __nv_bfloat16* __restrict__ colscale,
                                     const __nv_bfloat16* __restrict__ W, const float* __restrict__ scale,
                                     const SpkOut<OT> out, int accumulate, float* __restrict__ colpart) {
  const float up = scale ? __ldg(scale) : 1.f;
  const int n0 = blockIdx.x * SPK_ROWS;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const float cs = colscale ? __bfloat162float(colscale[k]) : 1.f;
    float cacc = 0.f;
#pragma unroll
    for (int i = 0; i < SPK_ROWS; ++i) {
      const int n = n0 + i;
      if (n < N) {
        float s = 0.f;
        const float* pp = part + (long long)n * K + k;
        int sp = 0;
        // four independent loads in flight, added in index order (the sum keeps its fixed order)
        for (; sp + 4 <= S; sp += 4) {
          const float v0 = pp[(long long)sp * split_stride], v1 = pp[(long long)(sp + 1) * split_stride];
          const float v2 = pp[(long long)(sp + 2) * split_stride], v3 = pp[(long long)(sp + 3) * split_stride];
          s += v0; s += v1; s += v2; s += v3;
        }
        for (; sp < S; ++sp) s += pp[(long long)sp * split_stride];
        s *= up;
        const long long o = (long long)n * K + k;
        if (W) cacc += s * __bfloat162float(W[o]);
        const float val = s * cs;
        OT* dst = out.row(n, K) + k;
        store_grad1(dst, accumulate ? (float)*dst + val : val);
      }
    }
    if (colpart) colpart[(long long)blockIdx.x * K + k] = cacc;
  }
}

// out[k] (+)= sum_b part[b, k].  Block: 32 columns x 32 row groups; group g adds rows g, g+32, ...
// in order, then a warp adds the 32 group sums of a column as a binary tree: a fixed order, so the
// result does not depend on scheduling, with five roundings at the size of the total instead of 31.
constexpr int COLSUM_COLS = 32, COLSUM_GROUPS = 32;
template <typename OT>
__global__ void colsum_kernel(const float* __restrict__ part, int NB, int K, OT* __restrict__ out,
                              int accumulate) {
  __shared__ float sm[COLSUM_GROUPS][COLSUM_COLS + 1];
  const int col = threadIdx.x & (COLSUM_COLS - 1), grp = threadIdx.x / COLSUM_COLS;
  const int k = blockIdx.x * COLSUM_COLS + col;
  float s = 0.f;
  if (k < K) {
    int b = grp;
    for (; b + 3 * COLSUM_GROUPS < NB; b += 4 * COLSUM_GROUPS) {
      const float v0 = part[(long long)b * K + k];
      const float v1 = part[(long long)(b + COLSUM_GROUPS) * K + k];
      const float v2 = part[(long long)(b + 2 * COLSUM_GROUPS) * K + k];
      const float v3 = part[(long long)(b + 3 * COLSUM_GROUPS) * K + k];
      s += v0; s += v1; s += v2; s += v3;
    }
    for (; b < NB; b += COLSUM_GROUPS) s += part[(long long)b * K + k];
  }
  sm[grp][col] = s;
  __syncthreads();
  float t = sm[col][grp];                  // lane = group, warp = column
#pragma unroll
  for (int o = 1; o < COLSUM_GROUPS; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  const int kc = blockIdx.x * COLSUM_COLS + grp;
  if (col == 0 && kc < K) store_grad1(out + kc, accumulate ? (float)out[kc] + t : t);
}

// Partial column sums of a bf16 [R, N] matrix (a bias gradient): part[b, n] over the rows of row block b, which the
// column sum above then adds in block order.  A warp takes 256 columns, 8 to a lane in one 16-byte load, and every
// eighth row of the block, four rows in flight; the warps are joined as a binary tree.  Bound by HBM: 64 095 x 1024
// with the column sum 38 us (an fp32 copy of the matrix and a reduction over it: 262); 8000 x 512 13 (41).  Error of
// the fp32 sums against 64 bits there: rms 1.6e-5 (2.8e-5) and 4.1e-6 (4.5e-6), of sums of the order of 250 and 90; with
// the warps and the groups added one after the other it was 2.8e-5 and 5.7e-6.
// grid: (ceil(N / 256), row blocks); N a multiple of 8, 16-byte aligned rows.
__global__ void __launch_bounds__(256)
colsum_rows_kernel(const __nv_bfloat16* __restrict__ x, long long R, int N, int rows_per_block, float* __restrict__ part) {
  __shared__ float sm[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * 256 + lane * 8;
  const long long r0 = (long long)blockIdx.y * rows_per_block, r1 = r0 + rows_per_block < R ? r0 + rows_per_block : R;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  auto add = [&](const uint4& q) {
    const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), d = unpack_bf16x2(q.z), e = unpack_bf16x2(q.w);
    acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y; acc[4] += d.x; acc[5] += d.y; acc[6] += e.x; acc[7] += e.y;
  };
  if (c < N) {
    const __nv_bfloat16* p = x + c;
    long long r = r0 + warp;
    for (; r + 24 < r1; r += 32) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = __ldg(reinterpret_cast<const uint4*>(p + (r + u * 8) * N));
#pragma unroll
      for (int u = 0; u < 4; ++u) add(q[u]);
    }
    for (; r < r1; r += 8) add(__ldg(reinterpret_cast<const uint4*>(p + r * N)));
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) sm[warp][lane * 8 + i] = acc[i];
  __syncthreads();
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col < N) {
    float t[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) t[w] = sm[w][threadIdx.x];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
      for (int w = 0; w < 8; w += 2 * o) t[w] += t[w + o];
    part[(long long)blockIdx.y * N + col] = t[0];
  }
}

// W'[n,k] = W[n,k] * wn[k]  (bf16), the RMSNorm weight folded into a linear; any width and alignment.
__global__ void fold_colscale_kernel(const __nv_bfloat16* __restrict__ W,
                                     const __nv_bfloat16* __restrict__ wn,
                                     __nv_bfloat16* __restrict__ out, long long N, int K) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N * K) return;
  const int k = (int)(i % K);
  out[i] = __float2bfloat16(__bfloat162float(W[i]) * __bfloat162float(wn[k]));
}
// The same in 16-byte vectors (an LM head of 16 384 x 256: 16 us an element a thread, under 8 like this).
__global__ void __launch_bounds__(256)
fold_colscale_vec_kernel(const uint4* __restrict__ W, const uint4* __restrict__ wn, uint4* __restrict__ out,
                         long long n, int kv) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint4 w = __ldg(W + i), g = __ldg(wn + (int)(i % kv));
  auto mul = [](uint32_t a, uint32_t b) {
    const float2 x = unpack_bf16x2(a), y = unpack_bf16x2(b);
    return pack_bf16x2(x.x * y.x, x.y * y.y);
  };
  out[i] = make_uint4(mul(w.x, g.x), mul(w.y, g.y), mul(w.z, g.z), mul(w.w, g.w));
}

// ---------------------------------------------------------------------------
// Standalone RMSNorm, fp32 statistics: y = x * rsqrt(mean(x^2) + eps) * w.
//
// Bound by HBM.  LPR lanes share a row (a whole warp from 129 channels up, so that narrow rows do not
// leave lanes idle) and hold it in registers, NV 16-byte vectors each: every operand is read once with
// 16-byte loads.  Forward: one row per LPR lanes.  Backward: a warp walks its rows with the next row's
// loads in flight and keeps its columns' weight gradients in registers until the block's rows are done;
// the strips of the warps are then added in warp order and a column sum adds the blocks in block order,
// so the weight gradient is bit-reproducible.  At 100 001 x 512: backward 56 us (5.5 TB/s; 165 us with 4
// bytes a lane, two passes and an accumulator in shared memory), forward 34 us (36 us).
// ---------------------------------------------------------------------------
template <int NV> struct RowVec { uint4 q[NV]; };

template <int LPR, int NV>
__device__ __forceinline__ RowVec<NV> load_row_vec(const __nv_bfloat16* row, int l, int D) {
  RowVec<NV> r;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = (v * LPR + l) * 8;
    r.q[v] = c < D ? __ldg(reinterpret_cast<const uint4*>(row + c)) : make_uint4(0u, 0u, 0u, 0u);
  }
  return r;
}
__device__ __forceinline__ void unpack8(const uint4& q, float (&f)[8]) {
  const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), c = unpack_bf16x2(q.z), d = unpack_bf16x2(q.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
template <int LPR>
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int LPR, int NV>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_vec_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                       __nv_bfloat16* __restrict__ y, float* __restrict__ inv_rms, long long R, int D, float eps) {
  constexpr int RPW = 32 / LPR;                       // rows of a warp
  const int l = threadIdx.x % LPR;
  const long long r = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * RPW + (threadIdx.x & 31) / LPR;
  const bool on = r < R;                              // no early exit: the shuffles take the whole warp
  const RowVec<NV> xr = load_row_vec<LPR, NV>(x + (on ? r : 0) * D, l, D);
  const RowVec<NV> wr = load_row_vec<LPR, NV>(w, l, D);
  float acc = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    float f[8];
    unpack8(xr.q[v], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc += f[i] * f[i];
  }
  const float inv = rsqrtf(row_sum<LPR>(acc) / (float)D + eps);
  if (!on) return;
  if (l == 0 && inv_rms) inv_rms[r] = inv;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = (v * LPR + l) * 8;
    if (c < D) {
      float f[8], g[8];
      unpack8(xr.q[v], f);
      unpack8(wr.q[v], g);
      uint4 o;
      o.x = pack_bf16x2(f[0] * inv * g[0], f[1] * inv * g[1]);
      o.y = pack_bf16x2(f[2] * inv * g[2], f[3] * inv * g[3]);
      o.z = pack_bf16x2(f[4] * inv * g[4], f[5] * inv * g[5]);
      o.w = pack_bf16x2(f[6] * inv * g[6], f[7] * inv * g[7]);
      *reinterpret_cast<uint4*>(y + r * D + c) = o;
    }
  }
}

template <int LPR, int NV>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_vec_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                       const __nv_bfloat16* __restrict__ go, const float* __restrict__ inv_rms,
                       __nv_bfloat16* __restrict__ gx, float* __restrict__ gw_part, long long R, int D,
                       int rows_per_block) {
  extern __shared__ float sm_gw[];   // [8 warps][D]
  constexpr int RPW = 32 / LPR;
  const int l = threadIdx.x % LPR, warp = threadIdx.x >> 5;
  const long long r0 = (long long)blockIdx.x * rows_per_block;
  const long long r1 = r0 + rows_per_block < R ? r0 + rows_per_block : R;
  const RowVec<NV> wr = load_row_vec<LPR, NV>(w, l, D);
  float acc[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
  const float inv_d = 1.f / (float)D;
  long long r = r0 + (long long)warp * RPW + (threadIdx.x & 31) / LPR;
  RowVec<NV> xr, gr;
  float inv = 0.f;
  auto fetch = [&](long long row) {
    const bool on = row < r1;
    xr = load_row_vec<LPR, NV>(x + (on ? row : r0) * D, l, D);
    gr = load_row_vec<LPR, NV>(go + (on ? row : r0) * D, l, D);
    inv = on ? __ldg(inv_rms + row) : 0.f;
  };
  // one row ahead; past 1024 channels the registers hold one row only
  constexpr bool AHEAD = NV <= 4;
  if (AHEAD) fetch(r);
  for (long long base = r0 + (long long)warp * RPW; base < r1; base += 8 * RPW, r += 8 * RPW) {
    if (!AHEAD) fetch(r);
    const RowVec<NV> xc = xr, gc = gr;
    const float ic = inv;
    if (AHEAD && base + 8 * RPW < r1) fetch(r + 8 * RPW);
    float dot = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float xv[8], gv[8], wv[8];
      unpack8(xc.q[v], xv);
      unpack8(gc.q[v], gv);
      unpack8(wr.q[v], wv);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot += gv[i] * wv[i] * (xv[i] * ic);
    }
    dot = row_sum<LPR>(dot) * inv_d;
    if (r < r1) {
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int c = (v * LPR + l) * 8;
        float xv[8], gv[8], wv[8], o[8];
        unpack8(xc.q[v], xv);
        unpack8(gc.q[v], gv);
        unpack8(wr.q[v], wv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xh = xv[i] * ic;
          o[i] = ic * (gv[i] * wv[i] - xh * dot);
          acc[v][i] += gv[i] * xh;
        }
        if (c < D) {
          uint4 q;
          q.x = pack_bf16x2(o[0], o[1]); q.y = pack_bf16x2(o[2], o[3]);
          q.z = pack_bf16x2(o[4], o[5]); q.w = pack_bf16x2(o[6], o[7]);
          *reinterpret_cast<uint4*>(gx + r * D + c) = q;
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int o = LPR; o < 32; o <<= 1) acc[v][i] += __shfl_xor_sync(0xffffffffu, acc[v][i], o);
    }
    const int c = (v * LPR + l) * 8;
    if ((threadIdx.x & 31) < LPR && c < D) {
      float4* s4 = reinterpret_cast<float4*>(sm_gw + warp * D + c);
      s4[0] = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
      s4[1] = make_float4(acc[v][4], acc[v][5], acc[v][6], acc[v][7]);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    float t = sm_gw[c];
#pragma unroll
    for (int k = 1; k < 8; ++k) t += sm_gw[k * D + c];
    gw_part[(long long)blockIdx.x * D + c] = t;
  }
}

// ss[r] = sum_d v^2 with v = a (+ b, rounded to bf16 and stored to `sum`): the row statistics that the trunk's
// GEMM epilogues take, for a residual stream that no kernel of this library produced.  One pass over the
// row, a warp or part of one to a row as above.  (The same through fp32 copies of the tensor: 183 us at
// 131 072 x 256, of 1.44 ms for the block's forward and backward.)
template <int LPR, int NV>
__global__ void __launch_bounds__(256)
row_ss_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
              __nv_bfloat16* __restrict__ sum, float* __restrict__ ss, long long R, int D) {
  constexpr int RPW = 32 / LPR;
  const int l = threadIdx.x % LPR;
  const long long r = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * RPW + (threadIdx.x & 31) / LPR;
  const bool on = r < R;                              // no early exit: the shuffles take the whole warp
  const RowVec<NV> ar = load_row_vec<LPR, NV>(a + (on ? r : 0) * D, l, D);
  RowVec<NV> br;
  if (b) br = load_row_vec<LPR, NV>(b + (on ? r : 0) * D, l, D);
  float acc = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    float f[8];
    unpack8(ar.q[v], f);
    if (b) {
      float g[8];
      unpack8(br.q[v], g);
      uint4 o;
      o.x = pack_bf16x2(f[0] + g[0], f[1] + g[1]); o.y = pack_bf16x2(f[2] + g[2], f[3] + g[3]);
      o.z = pack_bf16x2(f[4] + g[4], f[5] + g[5]); o.w = pack_bf16x2(f[6] + g[6], f[7] + g[7]);
      unpack8(o, f);
      const int c = (v * LPR + l) * 8;
      if (on && c < D) *reinterpret_cast<uint4*>(sum + r * D + c) = o;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) acc += f[i] * f[i];
  }
  acc = row_sum<LPR>(acc);
  if (on && l == 0) ss[r] = acc;
}

// A layer's weights as its GEMMs read them, in one launch: the four [D, D] projections packed (Wp, when
// they are not already) and packed with the norm weight folded in (Wp_f), the feed-forward weight folded
// (Wfc_f), and log_a in fp32.  All a few hundred KB: a launch's latency is what it costs, so one launch
// takes the place of four (a 512-token evaluation chunk of one block spent 9 of its 61 us on them).
struct LayerFold {
  const __nv_bfloat16* w[4];      // select, in, gate, delta  [D, D]
  const __nv_bfloat16 *wn1, *fc, *wn2, *log_a;
  __nv_bfloat16 *Wp, *Wp_f, *Wfc_f;   // Wp may be null
  float* log_a32;
  int D, F;
};
__global__ void __launch_bounds__(256) layer_fold_kernel(const LayerFold p) {
  const long long dd = (long long)p.D * p.D / 8, ff = (long long)p.F * p.D / 8;
  const long long n = 4 * dd + ff + p.D / 8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (i >= 4 * dd + ff) {
      const long long c = (i - 4 * dd - ff) * 8;
      float f[8];
      unpack8(__ldg(reinterpret_cast<const uint4*>(p.log_a + c)), f);
      *reinterpret_cast<float4*>(p.log_a32 + c) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(p.log_a32 + c + 4) = make_float4(f[4], f[5], f[6], f[7]);
      continue;
    }
    const bool proj = i < 4 * dd;
    const long long e = proj ? i % dd : i - 4 * dd;          // 16-byte vector inside its matrix
    const int col = (int)(e * 8 % p.D);
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(proj ? p.w[i / dd] : p.fc) + e);
    float f[8], g[8];
    unpack8(q, f);
    unpack8(__ldg(reinterpret_cast<const uint4*>((proj ? p.wn1 : p.wn2) + col)), g);
    uint4 o;
    o.x = pack_bf16x2(f[0] * g[0], f[1] * g[1]); o.y = pack_bf16x2(f[2] * g[2], f[3] * g[3]);
    o.z = pack_bf16x2(f[4] * g[4], f[5] * g[5]); o.w = pack_bf16x2(f[6] * g[6], f[7] * g[7]);
    if (proj) {
      reinterpret_cast<uint4*>(p.Wp_f)[i] = o;
      if (p.Wp) reinterpret_cast<uint4*>(p.Wp)[i] = q;
    } else {
      reinterpret_cast<uint4*>(p.Wfc_f)[e] = o;
    }
  }
}

// ---------------------------------------------------------------------------
// RMSNorm of any even width and 4-byte alignment (one warp per row), fp32 statistics.
// y = x * rsqrt(mean(x^2) + eps) * w ; optional residual add x = x + res first.
// ---------------------------------------------------------------------------
__global__ void rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                   const __nv_bfloat16* __restrict__ res,
                                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                   __nv_bfloat16* __restrict__ xsum, float* __restrict__ inv_rms,
                                   long long R, int D, float eps) {
  const long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= R) return;
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* xr = x + r * D;
  float acc = 0.f;
  for (int c = lane * 2; c < D; c += 64) {
    float2 f = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(xr + c));
    if (res) {
      float2 g = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(res + r * D + c));
      f.x = __bfloat162float(__float2bfloat16(f.x + g.x));
      f.y = __bfloat162float(__float2bfloat16(f.y + g.y));
      if (xsum) *reinterpret_cast<uint32_t*>(xsum + r * D + c) = pack_bf16x2(f.x, f.y);
    }
    acc += f.x * f.x + f.y * f.y;
  }
  acc = warp_sum(acc);
  const float inv = rsqrtf(acc / (float)D + eps);
  if (lane == 0 && inv_rms) inv_rms[r] = inv;
  for (int c = lane * 2; c < D; c += 64) {
    float2 f = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(xr + c));
    if (res) {
      float2 g = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(res + r * D + c));
      f.x = __bfloat162float(__float2bfloat16(f.x + g.x));
      f.y = __bfloat162float(__float2bfloat16(f.y + g.y));
    }
    float2 ww = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + c));
    *reinterpret_cast<uint32_t*>(y + r * D + c) = pack_bf16x2(f.x * inv * ww.x, f.y * inv * ww.y);
  }
}

// Backward: gx = inv * (go*w - xhat * mean(go*w*xhat)); weight grad as per-block partials
// [gridDim.x, D].  Inside a block every warp adds its rows, in row order, into its own [D] strip of
// shared memory (a lane owns its columns, so no atomics), the strips are added in warp order, and a
// second-stage column sum adds the blocks in order: the weight gradient is bit-reproducible.
__global__ void rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x,
                                   const __nv_bfloat16* __restrict__ w,
                                   const __nv_bfloat16* __restrict__ go,
                                   const float* __restrict__ inv_rms, __nv_bfloat16* __restrict__ gx,
                                   float* __restrict__ gw_part, long long R, int D,
                                   int rows_per_block) {
  extern __shared__ float sm_gw[];   // [warps][D]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* mine = sm_gw + warp * D;
  for (int c = lane; c < D; c += 32) mine[c] = 0.f;
  __syncwarp();
  const long long r0 = (long long)blockIdx.x * rows_per_block;
  for (long long r = r0 + warp; r < r0 + rows_per_block && r < R; r += nw) {
    const float inv = inv_rms[r];
    float dot = 0.f;
    for (int c = lane * 2; c < D; c += 64) {
      float2 xv = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(x + r * D + c));
      float2 gv = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(go + r * D + c));
      float2 wv = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + c));
      dot += gv.x * wv.x * xv.x * inv + gv.y * wv.y * xv.y * inv;
    }
    dot = warp_sum(dot) / (float)D;
    for (int c = lane * 2; c < D; c += 64) {
      float2 xv = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(x + r * D + c));
      float2 gv = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(go + r * D + c));
      float2 wv = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + c));
      const float xh0 = xv.x * inv, xh1 = xv.y * inv;
      *reinterpret_cast<uint32_t*>(gx + r * D + c) =
          pack_bf16x2(inv * (gv.x * wv.x - xh0 * dot), inv * (gv.y * wv.y - xh1 * dot));
      mine[c] += gv.x * xh0;
      mine[c + 1] += gv.y * xh1;
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    float t = sm_gw[c];
    for (int k = 1; k < nw; ++k) t += sm_gw[k * D + c];
    gw_part[(long long)blockIdx.x * D + c] = t;
  }
}

// ---------------------------------------------------------------------------
// Optimizer kernels
// ---------------------------------------------------------------------------
// Muon momentum: buf = mu*buf + g ; dir = nesterov ? g + mu*buf : buf.  Writes dir in bf16 and the
// sum of squares of the bf16-rounded direction of each block's slice to a per-device scratch slot
// (grid: (blocks_per_mat, G); slot = matrix * blocks_per_mat + block).  No atomics: the normalise
// kernel adds a matrix's slots in index order, so the Frobenius norm is reproducible.
constexpr int MUON_PART_SLOTS = 16384;
__device__ float g_muon_part[MUON_PART_SLOTS];

__global__ void muon_momentum_kernel(const float* __restrict__ g, float* __restrict__ buf,
                                     __nv_bfloat16* __restrict__ dir, long long numel_per_mat, float mu,
                                     int nesterov) {
  __shared__ float sm[32];
  const long long base = (long long)blockIdx.y * numel_per_mat;
  float acc = 0.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < numel_per_mat;
       i += (long long)gridDim.x * blockDim.x) {
    const float gv = g[base + i];
    const float b = mu * buf[base + i] + gv;
    buf[base + i] = b;
    const float dv = nesterov ? gv + mu * b : b;
    const __nv_bfloat16 q = __float2bfloat16(dv);
    dir[base + i] = q;
    const float qf = __bfloat162float(q);
    acc += qf * qf;
  }
  acc = block_sum(acc, sm);
  if (threadIdx.x == 0) g_muon_part[blockIdx.y * gridDim.x + blockIdx.x] = acc;
}

// X = dir / (||dir||_F + eps) in bf16, in place; sumsq[matrix] receives the squared norm.
// `nparts` is the momentum kernel's blocks_per_mat.
__global__ void muon_normalize_kernel(__nv_bfloat16* __restrict__ dir, float* __restrict__ sumsq,
                                      int nparts, long long numel_per_mat, float eps) {
  __shared__ float sm[32];
  float tot = 0.f;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) tot += g_muon_part[blockIdx.y * nparts + i];
  tot = block_sum(tot, sm);                    // same fixed tree in every block of the matrix
  if (threadIdx.x == 0 && blockIdx.x == 0) sumsq[blockIdx.y] = tot;
  const long long base = (long long)blockIdx.y * numel_per_mat;
  const float inv = 1.f / (sqrtf(tot) + eps);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < numel_per_mat;
       i += (long long)gridDim.x * blockDim.x)
    dir[base + i] = __float2bfloat16(__bfloat162float(dir[base + i]) * inv);
}

// p = p * (1 - lr*wd) - lr*scale * O   (bf16 params, bf16 orthogonalised update)
__global__ void muon_apply_kernel(__nv_bfloat16* __restrict__ p, const __nv_bfloat16* __restrict__ O,
                                  long long n, float lr_scale, float decay_mul) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = __bfloat162float(p[i]) * decay_mul - lr_scale * __bfloat162float(O[i]);
    p[i] = __float2bfloat16(v);
  }
}

// Decoupled AdamW over a flat range; fp32 moments, bf16 or fp32 params.
template <typename PT>
__global__ void adamw_kernel(PT* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                             float* __restrict__ v, long long n, float lr, float b1, float b2,
                             float eps, float wd, float bias1, float bias2_sqrt,
                             const float* __restrict__ gscale) {
  const float gs = gscale ? *gscale : 1.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float gv = g[i] * gs;
    const float mi = b1 * m[i] + (1.f - b1) * gv;
    const float vi = b2 * v[i] + (1.f - b2) * gv * gv;
    m[i] = mi;
    v[i] = vi;
    float pv = (float)p[i];
    pv *= (1.f - lr * wd);
    pv -= (lr / bias1) * mi / (sqrtf(vi) / bias2_sqrt + eps);
    p[i] = (PT)pv;
  }
}

// Global L2 norm in two stages with a fixed summation order (no atomics): every block writes
// the sum of squares of its grid-stride slice to its own slot of a per-device scratch array, and
// the single-block second stage adds the slots in index order.  Two replicas that hold the same
// gradient bits therefore compute the same clip coefficient.
constexpr int SUMSQ_MAX_BLOCKS = 148 * 8;
__device__ float g_sumsq_part[SUMSQ_MAX_BLOCKS];

__global__ void sumsq_kernel(const float* __restrict__ g, long long n) {
  __shared__ float sm[32];
  float acc = 0.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    acc += g[i] * g[i];
  acc = block_sum(acc, sm);
  if (threadIdx.x == 0) g_sumsq_part[blockIdx.x] = acc;
}

// stat = {sumsq, coef, norm}; coef = min(1, max_norm / (norm + 1e-6)).  One block of 256 threads.
__global__ void clip_coef_kernel(float* __restrict__ stat, int nparts, float max_norm) {
  __shared__ float sm[32];
  float acc = 0.f;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) acc += g_sumsq_part[i];
  acc = block_sum(acc, sm);
  if (threadIdx.x == 0) {
    const float norm = sqrtf(acc);
    stat[0] = acc;
    stat[1] = fminf(1.f, max_norm / (norm + 1e-6f));
    stat[2] = norm;
  }
}
__global__ void scale_by_ptr_kernel(float* __restrict__ g, long long n, const float* __restrict__ coef) {
  const float c = *coef;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    g[i] *= c;
}

// p -= lr * g  (test-time-training SGD), bf16 params, fp32 grads.
__global__ void sgd_kernel(__nv_bfloat16* __restrict__ p, const float* __restrict__ g, long long n,
                           float lr) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    p[i] = __float2bfloat16(__bfloat162float(p[i]) - lr * g[i]);
}

// lse[m] from per-(tile, half) partials (max, sum 2^(z - max)) in the log2 domain;
// partials are laid out [nparts][M], so the lanes of a warp read consecutive rows.  PW warps of a block share 32 rows
// and take the partials w, w + PW, ... of each, merged as they arrive and then across warps in warp order: the
// 128 partials of a 16 384-word vocabulary are one dependent chain when a thread has a row to itself, 26 us for
// the 511 rows of an evaluation chunk whose logits GEMM takes 12; 4 us with sixteen warps.
constexpr int LSC_WARPS = 16;
__device__ __forceinline__ void lse_merge(float2& a, const float2 v) {
  // An empty partial (sum zero) adds nothing, whatever its maximum.  Every other one is merged, so that a sum that is
  // not a number (a NaN logit, or an infinite one: the tile's own inf - inf) makes the row's result one as well.
  if (v.y != 0.f) {
    const float m = fmaxf(a.x, v.x);
    a.y = (a.y != 0.f ? a.y * exp2f(a.x - m) : 0.f) + v.y * exp2f(v.x - m);
    a.x = m;
  }
}
template <int PW>
__global__ void __launch_bounds__(32 * LSC_WARPS)
lse_combine_kernel(const float2* __restrict__ part, int nparts, long long M,
                   const float* __restrict__ zt, float* __restrict__ lse, float* __restrict__ loss) {
  __shared__ float2 join[PW > 1 ? LSC_WARPS : 1][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, w0 = warp % PW;
  const long long m = ((long long)blockIdx.x * (LSC_WARPS / PW) + warp / PW) * 32 + lane;
  float2 a = make_float2(-INFINITY, 0.f);
  if (m < M) {
    int i = w0;
    for (; i + 3 * PW < nparts; i += 4 * PW) {
      float2 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg(&part[(long long)(i + u * PW) * M + m]);
#pragma unroll
      for (int u = 0; u < 4; ++u) lse_merge(a, v[u]);
    }
    for (; i < nparts; i += PW) lse_merge(a, __ldg(&part[(long long)i * M + m]));
  }
  if constexpr (PW > 1) {
    join[warp][lane] = a;
    __syncthreads();
  }
  if (w0 == 0 && m < M) {
#pragma unroll
    for (int w = 1; w < PW; ++w) lse_merge(a, join[warp + w][lane]);
    const float l = (a.x + log2f(a.y)) * 0.6931471805599453f;
    lse[m] = l;
    if (loss != nullptr && zt != nullptr) loss[m] = l - zt[m];
  }
}

__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ s, __nv_bfloat16* __restrict__ d,
                                        long long n, float scale) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    d[i] = __float2bfloat16(s[i] * scale);
}
__global__ void cast_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ s, float* __restrict__ d,
                                        long long n, float scale, int accumulate) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = __bfloat162float(s[i]) * scale;
    d[i] = accumulate ? d[i] + v : v;
  }
}

static inline int grid_for(long long n, int threads, int cap = 148 * 8) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  return (int)(b > cap ? cap : b);
}

}  // namespace ccb

using namespace ccb;
#define CCB_CHECK_LAUNCH(name)                                                   \
  do {                                                                           \
    count_launch();                                                              \
    cudaError_t e__ = cudaGetLastError();                                        \
    if (e__ != cudaSuccess) return set_error(name ": %s", cudaGetErrorString(e__)); \
  } while (0)

extern "C" int ccb_embed_fwd(const void* tok, int64_t tok_is_i64, const void* E, void* x, float* ss,
                             int64_t R, int64_t D, int64_t V, void* stream) {
  if (R <= 0) return 0;
  if (D % 8) return set_error("ccb_embed_fwd: D must be a multiple of 8");
  const int wpb = 8;
  const unsigned grid = (unsigned)((R + wpb - 1) / wpb);
  if (tok_is_i64)
    embed_fwd_kernel<long long><<<grid, wpb * 32, 0, (cudaStream_t)stream>>>(
        (const long long*)tok, (const __nv_bfloat16*)E, (__nv_bfloat16*)x, ss, R, (int)D, (int)V);
  else
    embed_fwd_kernel<int><<<grid, wpb * 32, 0, (cudaStream_t)stream>>>(
        (const int*)tok, (const __nv_bfloat16*)E, (__nv_bfloat16*)x, ss, R, (int)D, (int)V);
  CCB_CHECK_LAUNCH("embed_fwd");
  return 0;
}

// slots: workspace of ccb_embed_bwd_slots(R, D, V) floats, 16-byte aligned: the boundary sums of
// stage 1 followed by the per-token first / last positions (need not be initialised).
extern "C" int64_t ccb_embed_bwd_slots(int64_t R, int64_t D, int64_t V) {
  return ((R + EMB_CH - 1) / EMB_CH) * 2 * D + 4 * V;
}
// key[i] = the token, -1 below or V above the table; V < 32 768.
extern "C" int ccb_token_keys(const void* tok, int64_t tok_is_i64, void* key_i16, int64_t R, int64_t V, void* stream) {
  if (R <= 0) return 0;
  if (V <= 0 || V > 32767) return set_error("ccb_token_keys: V=%lld does not fit 16-bit keys", (long long)V);
  if (tok_is_i64)
    token_keys_kernel<<<grid_for(R, 256), 256, 0, (cudaStream_t)stream>>>((const long long*)tok, (short*)key_i16, R, (int)V);
  else
    token_keys_kernel<<<grid_for(R, 256), 256, 0, (cudaStream_t)stream>>>((const int*)tok, (short*)key_i16, R, (int)V);
  CCB_CHECK_LAUNCH("token_keys");
  return 0;
}

template <int VPL, typename TokT>
static int launch_embed_bwd(const TokT* st, const long long* pm, const __nv_bfloat16* g, float* dE, float* slots,
                            long long* fp, long long* lp, int64_t R, int64_t V, cudaStream_t s) {
  constexpr int D = 256 * VPL, wpb = 4;
  const long long chunks = (R + EMB_CH - 1) / EMB_CH;
  embed_bwd_runs_kernel<VPL, TokT><<<(unsigned)((chunks + wpb - 1) / wpb), wpb * 32, 0, s>>>(
      st, pm, g, dE, slots, fp, lp, R, D, (int)V);
  CCB_CHECK_LAUNCH("embed_bwd_runs");
  constexpr int smem = EMB_JOIN_WARPS * D * (int)sizeof(float);
  // sixteen [1024] strips are 64 KiB of shared memory: above the default limit, opt in
  if (smem > 48 * 1024) cudaFuncSetAttribute(embed_bwd_join_kernel<D / 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const int64_t want = (V + 4 * ccb_num_sms() - 1) / (4 * ccb_num_sms());
  const int toks = (int)(want < EMB_JOIN_TOKS ? want : EMB_JOIN_TOKS);
  embed_bwd_join_kernel<D / 32><<<(unsigned)((V + toks - 1) / toks), EMB_JOIN_WARPS * 32, smem, s>>>(
      fp, lp, slots, dE, D, (int)V, toks);
  CCB_CHECK_LAUNCH("embed_bwd_join");
  return 0;
}

// sorted_tok: int64, or the 16-bit keys of ccb_token_keys (tok_bytes 8 / 2).
extern "C" int ccb_embed_bwd_sorted_as(const void* sorted_tok, int64_t tok_bytes, const int64_t* perm, const void* dx,
                                       float* dE, float* slots, int64_t R, int64_t D, int64_t V, void* stream) {
  if (R <= 0) return 0;
  if (slots == nullptr) return set_error("ccb_embed_bwd_sorted_as: the boundary-slot workspace is required");
  if (tok_bytes != 8 && tok_bytes != 2) return set_error("ccb_embed_bwd_sorted_as: tokens of %lld bytes", (long long)tok_bytes);
  if (D != 256 && D != 512 && D != 1024)
    return set_error("ccb_embed_bwd_sorted_as: D=%lld unsupported (256, 512, 1024)", (long long)D);
  cudaStream_t s = (cudaStream_t)stream;
  const long long* pm = (const long long*)perm;
  const __nv_bfloat16* g = (const __nv_bfloat16*)dx;
  long long* fp = reinterpret_cast<long long*>(slots + (R + EMB_CH - 1) / EMB_CH * 2 * D);
  long long* lp = fp + V;
  cudaMemsetAsync(lp, 0xFF, sizeof(long long) * (size_t)V, s);      // -1: token does not occur
  auto run = [&](auto* st) {
    if (D == 256) return launch_embed_bwd<1>(st, pm, g, dE, slots, fp, lp, R, V, s);
    if (D == 512) return launch_embed_bwd<2>(st, pm, g, dE, slots, fp, lp, R, V, s);
    return launch_embed_bwd<4>(st, pm, g, dE, slots, fp, lp, R, V, s);
  };
  return tok_bytes == 8 ? run((const long long*)sorted_tok) : run((const short*)sorted_tok);
}

static int launch_colsum(const float* part, int64_t NB, int64_t K, void* out, int out_bf16, int64_t accumulate,
                         cudaStream_t s) {
  const unsigned grid = (unsigned)((K + COLSUM_COLS - 1) / COLSUM_COLS), threads = COLSUM_COLS * COLSUM_GROUPS;
  if (out_bf16)
    colsum_kernel<<<grid, threads, 0, s>>>(part, (int)NB, (int)K, (__nv_bfloat16*)out, (int)accumulate);
  else
    colsum_kernel<<<grid, threads, 0, s>>>(part, (int)NB, (int)K, (float*)out, (int)accumulate);
  CCB_CHECK_LAUNCH("colsum");
  return 0;
}

template <typename OT>
static int launch_splitk(const float* part, int64_t S, int64_t split_stride, int64_t N, int64_t K,
                         const __nv_bfloat16* colscale, const __nv_bfloat16* W, const float* scale, void* const* parts,
                         int64_t nparts, int64_t accumulate, float* colpart, cudaStream_t s) {
  SpkOut<OT> out = {};
  uintptr_t outs = 0;
  for (int i = 0; i < nparts; ++i) {
    out.p[i] = (OT*)parts[i];
    outs |= (uintptr_t)parts[i];
  }
  out.rows = (int)(N / nparts);
  const unsigned nb = (unsigned)((N + SPK_ROWS - 1) / SPK_ROWS);
  const uintptr_t wide = (uintptr_t)part | outs;                            // 16-byte accesses
  const uintptr_t half = (uintptr_t)colscale | (uintptr_t)W;                // 8-byte accesses
  const bool tile = !accumulate && K % 4 == 0 && split_stride % 4 == 0 && (wide & 15) == 0 && (half & 7) == 0 &&
                    (K + SPK_COLS - 1) / SPK_COLS <= 65535;
  if (tile) {
    const dim3 grid(nb, (unsigned)((K + SPK_COLS - 1) / SPK_COLS));
    // Groups: as many as make about 1000 blocks' worth of threads, and each keeps at least four partials so that its
    // loads are in flight together.  A result with blocks enough needs none: they then only cost the joins and read each
    // partial in smaller pieces.  us with 1 / 2 / 4 / 8 groups (events, cold L2): 74 partials of 256 x 256 20 / 16 / 14 /
    // 12, 64 of 512 x 256 18 / 16 / 16 / 16, 74 of 1024 x 256 29 / 25 / 31 / 33, 25 of 2048 x 512 31 / 33 / 37 / 47,
    // 15 of 16 384 x 512 102 / 115 / 143 / 313 (one thread a column: 133).
    const int64_t blocks = (int64_t)grid.x * grid.y, most = S <= 4 ? 1 : (S <= 8 ? 2 : (S <= 24 ? 4 : 8));
    int64_t groups = most;
    while (groups > 1 && blocks * groups > 8 * (int64_t)ccb_num_sms()) groups /= 2;
    if (groups == 1) splitk_tile_kernel<1, OT><<<grid, 128, 0, s>>>(part, (int)S, split_stride, (int)N, (int)K, colscale, W, scale, out, colpart);
    else if (groups == 2) splitk_tile_kernel<2, OT><<<grid, 256, 0, s>>>(part, (int)S, split_stride, (int)N, (int)K, colscale, W, scale, out, colpart);
    else if (groups == 4) splitk_tile_kernel<4, OT><<<grid, 512, 0, s>>>(part, (int)S, split_stride, (int)N, (int)K, colscale, W, scale, out, colpart);
    else splitk_tile_kernel<8, OT><<<grid, 1024, 0, s>>>(part, (int)S, split_stride, (int)N, (int)K, colscale, W, scale, out, colpart);
  } else {
    splitk_reduce_kernel<OT><<<nb, 256, 0, s>>>(part, (int)S, split_stride, (int)N, (int)K, colscale, W, scale, out,
                                                (int)accumulate, colpart);
  }
  CCB_CHECK_LAUNCH("splitk_reduce");
  return 0;
}

// The results go to `nout` tensors of N / nout rows (1 to 4); they and `colsum_out` are fp32, or bf16 with out_bf16;
// `scale` (device, may be null) multiplies the sums.
extern "C" int ccb_splitk_reduce_parts(const float* part, int64_t S, int64_t split_stride, int64_t N, int64_t K,
                                       const void* colscale, const void* W, const float* scale, void* const* outs,
                                       int64_t nout, int64_t out_bf16, int64_t accumulate, float* colpart,
                                       void* colsum_out, int64_t colsum_accumulate, void* stream) {
  if (N <= 0 || K <= 0) return 0;
  if (nout < 1 || nout > 4 || N % nout != 0)
    return set_error("ccb_splitk_reduce_parts: %lld rows into %lld tensors", (long long)N, (long long)nout);
  cudaStream_t s = (cudaStream_t)stream;
  const __nv_bfloat16* cs = (const __nv_bfloat16*)colscale;
  const __nv_bfloat16* w = (const __nv_bfloat16*)W;
  float* cp = W ? colpart : nullptr;
  const int rc = out_bf16 ? launch_splitk<__nv_bfloat16>(part, S, split_stride, N, K, cs, w, scale, outs, nout, accumulate, cp, s)
                          : launch_splitk<float>(part, S, split_stride, N, K, cs, w, scale, outs, nout, accumulate, cp, s);
  if (rc) return rc;
  if (cp && colsum_out)
    return launch_colsum(cp, (N + SPK_ROWS - 1) / SPK_ROWS, K, colsum_out, (int)out_bf16, colsum_accumulate, s);
  return 0;
}

extern "C" int ccb_splitk_reduce_as(const float* part, int64_t S, int64_t split_stride, int64_t N, int64_t K,
                                    const void* colscale, const void* W, const float* scale, void* out,
                                    int64_t out_bf16, int64_t accumulate, float* colpart, void* colsum_out,
                                    int64_t colsum_accumulate, void* stream) {
  return ccb_splitk_reduce_parts(part, S, split_stride, N, K, colscale, W, scale, &out, 1, out_bf16, accumulate, colpart,
                                 colsum_out, colsum_accumulate, stream);
}

extern "C" int ccb_colsum_as(const float* part, int64_t NB, int64_t K, void* out, int64_t out_bf16,
                             int64_t accumulate, void* stream) {
  if (K <= 0) return 0;
  return launch_colsum(part, NB, K, out, (int)out_bf16, accumulate, (cudaStream_t)stream);
}
extern "C" int ccb_colsum(const float* part, int64_t NB, int64_t K, float* out, int64_t accumulate,
                          void* stream) {
  return ccb_colsum_as(part, NB, K, out, 0, accumulate, stream);
}

// Row blocks of ccb_colsum_bf16 (part holds that many rows of N floats): about eight blocks to an SM in all.
extern "C" int64_t ccb_colsum_bf16_blocks(int64_t R, int64_t N) {
  const int64_t cols = (N + 255) / 256, want = (8 * (int64_t)ccb_num_sms() + cols - 1) / cols;
  int64_t rows = (R + want - 1) / want;
  rows = rows < 32 ? 32 : (rows + 7) / 8 * 8;
  return (R + rows - 1) / rows;
}
// out[n] = sum_r x[r, n], rounded once.  Returns 1, launching nothing, for rows that are not whole aligned vectors.
extern "C" int ccb_colsum_bf16(const void* x, int64_t R, int64_t N, float* part, void* out, int64_t out_bf16, void* stream) {
  if (R <= 0 || N <= 0) return 1;
  const int64_t nb = ccb_colsum_bf16_blocks(R, N), rows = ((R + nb - 1) / nb + 7) / 8 * 8;
  if (N % 8 != 0 || ((uintptr_t)x & 15) != 0 || nb > 65535) return 1;
  const dim3 grid((unsigned)((N + 255) / 256), (unsigned)nb);
  colsum_rows_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, R, (int)N, (int)rows, part);
  CCB_CHECK_LAUNCH("colsum_bf16");
  return launch_colsum(part, nb, N, out, (int)out_bf16, 0, (cudaStream_t)stream);
}

extern "C" int ccb_fold_colscale(const void* W, const void* wn, void* out, int64_t N, int64_t K,
                                 void* stream) {
  if (N * K <= 0) return 0;
  if (K % 8 == 0 && (((uintptr_t)W | (uintptr_t)wn | (uintptr_t)out) & 15) == 0) {
    const long long n = N * K / 8;
    fold_colscale_vec_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        (const uint4*)W, (const uint4*)wn, (uint4*)out, n, (int)(K / 8));
  } else {
    fold_colscale_kernel<<<(unsigned)((N * K + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)W, (const __nv_bfloat16*)wn, (__nv_bfloat16*)out, N, (int)K);
  }
  CCB_CHECK_LAUNCH("fold_colscale");
  return 0;
}

// Rows of at most 1536 channels in whole 16-byte vectors, all operands 16-byte aligned.
constexpr int RMSNORM_VEC_MAX_DIM = 1536;
static inline bool rmsnorm_vec_ok(int64_t D, const void* a, const void* b, const void* c, const void* d) {
  return D % 8 == 0 && D <= RMSNORM_VEC_MAX_DIM &&
         (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15) == 0;
}
// f(lanes per row, vectors per lane) as integral constants
template <typename F>
static void rmsnorm_dispatch(int64_t D, F f) {
  using std::integral_constant;
  if (D <= 64) f(integral_constant<int, 8>(), integral_constant<int, 1>());
  else if (D <= 128) f(integral_constant<int, 16>(), integral_constant<int, 1>());
  else if (D <= 256) f(integral_constant<int, 32>(), integral_constant<int, 1>());
  else if (D <= 512) f(integral_constant<int, 32>(), integral_constant<int, 2>());
  else if (D <= 768) f(integral_constant<int, 32>(), integral_constant<int, 3>());
  else if (D <= 1024) f(integral_constant<int, 32>(), integral_constant<int, 4>());
  else f(integral_constant<int, 32>(), integral_constant<int, 6>());
}

// ss[r] = sum_d (a (+ b))^2; with b, `sum` receives a + b.  Returns 1, launching nothing, for rows that are not
// whole aligned 16-byte vectors or are wider than 1536.
extern "C" int ccb_row_ss(const void* a, const void* b, void* sum, float* ss, int64_t R, int64_t D, void* stream) {
  if (R <= 0) return 0;
  if (!rmsnorm_vec_ok(D, a, b, sum, nullptr)) return 1;
  rmsnorm_dispatch(D, [&](auto lpr, auto nv) {
    constexpr int LPR = decltype(lpr)::value, NV = decltype(nv)::value;
    const int64_t rows = 8 * (32 / LPR);
    row_ss_kernel<LPR, NV><<<(unsigned)((R + rows - 1) / rows), 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, (__nv_bfloat16*)sum, ss, R, (int)D);
  });
  CCB_CHECK_LAUNCH("row_ss");
  return 0;
}

// See layer_fold_kernel.  Returns 1, launching nothing, for operands that are not 16-byte aligned.
extern "C" int ccb_layer_fold(const void* sel, const void* in, const void* gate, const void* delta, const void* wn1,
                              const void* fc, const void* wn2, const void* log_a, void* Wp, void* Wp_f, void* Wfc_f,
                              float* log_a32, int64_t D, int64_t F, void* stream) {
  if (D <= 0 || F <= 0) return 0;
  const uintptr_t all = (uintptr_t)sel | (uintptr_t)in | (uintptr_t)gate | (uintptr_t)delta | (uintptr_t)wn1 |
                        (uintptr_t)fc | (uintptr_t)wn2 | (uintptr_t)log_a | (uintptr_t)Wp | (uintptr_t)Wp_f |
                        (uintptr_t)Wfc_f | (uintptr_t)log_a32;
  if (D % 8 != 0 || (all & 15) != 0) return 1;
  LayerFold p;
  p.w[0] = (const __nv_bfloat16*)sel; p.w[1] = (const __nv_bfloat16*)in;
  p.w[2] = (const __nv_bfloat16*)gate; p.w[3] = (const __nv_bfloat16*)delta;
  p.wn1 = (const __nv_bfloat16*)wn1; p.fc = (const __nv_bfloat16*)fc;
  p.wn2 = (const __nv_bfloat16*)wn2; p.log_a = (const __nv_bfloat16*)log_a;
  p.Wp = (__nv_bfloat16*)Wp; p.Wp_f = (__nv_bfloat16*)Wp_f; p.Wfc_f = (__nv_bfloat16*)Wfc_f;
  p.log_a32 = log_a32;
  p.D = (int)D; p.F = (int)F;
  layer_fold_kernel<<<grid_for((4 * D * D + F * D + D) / 8, 256), 256, 0, (cudaStream_t)stream>>>(p);
  CCB_CHECK_LAUNCH("layer_fold");
  return 0;
}

extern "C" int ccb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* xsum,
                               float* inv_rms, int64_t R, int64_t D, float eps, void* stream) {
  if (R <= 0) return 0;
  if (D % 2) return set_error("ccb_rmsnorm_fwd: D must be even");
  const int wpb = 8;
  if (res == nullptr && rmsnorm_vec_ok(D, x, w, y, y)) {
    rmsnorm_dispatch(D, [&](auto lpr, auto nv) {
      constexpr int LPR = decltype(lpr)::value, NV = decltype(nv)::value;
      const int64_t rows = wpb * (32 / LPR);
      rmsnorm_fwd_vec_kernel<LPR, NV><<<(unsigned)((R + rows - 1) / rows), 256, 0, (cudaStream_t)stream>>>(
          (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, inv_rms, R, (int)D, eps);
    });
  } else {
    rmsnorm_fwd_kernel<<<(unsigned)((R + wpb - 1) / wpb), wpb * 32, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w, (__nv_bfloat16*)y,
        (__nv_bfloat16*)xsum, inv_rms, R, (int)D, eps);
  }
  CCB_CHECK_LAUNCH("rmsnorm_fwd");
  return 0;
}

// gw_part must hold ccb_rmsnorm_bwd_blocks(R) * D floats.  Eight per-warp [D] strips of shared
// memory bound the channel count (48 KiB without an opt-in).
constexpr int RMSNORM_BWD_MAX_DIM = 1536;
// Rows of a block: whole rounds of the two blocks that an SM holds, at least two rounds and no block of more than 256
// rows; at least one row for each of the eight warps.  256 rows for every size left 9 000 rows on 36 SMs (89 us at 384
// channels, now 7); always two rounds made the blocks of large batches long, and the last ones late: 300 000 x 256
// 124 us (110 in four rounds), 1 000 000 x 66 357 (308 in blocks of 256, which cost 160 000 x 512 a third round: 97 -> 114).
static inline int64_t rmsnorm_bwd_rows(int64_t R) {
  const int64_t round = 2 * (int64_t)ccb_num_sms(), rounds = (R + 256 * round - 1) / (256 * round);
  const int64_t blocks = round * (rounds < 2 ? 2 : rounds), rows = (R + blocks - 1) / blocks;
  return rows < 8 ? 8 : (rows + 7) / 8 * 8;
}
extern "C" int64_t ccb_rmsnorm_bwd_blocks(int64_t R) {
  const int64_t rpb = rmsnorm_bwd_rows(R);
  return (R + rpb - 1) / rpb;
}
static int launch_rmsnorm_bwd(const void* x, const void* w, const void* go, const float* inv_rms, void* gx,
                              float* gw_part, int64_t R, int64_t D, int64_t rpb, cudaStream_t s) {
  const unsigned nb = (unsigned)((R + rpb - 1) / rpb);
  const size_t smem = (size_t)8 * D * sizeof(float);
  if (rmsnorm_vec_ok(D, x, w, go, gx)) {
    rmsnorm_dispatch(D, [&](auto lpr, auto nv) {
      rmsnorm_bwd_vec_kernel<decltype(lpr)::value, decltype(nv)::value><<<nb, 256, smem, s>>>(
          (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)go, inv_rms, (__nv_bfloat16*)gx,
          gw_part, R, (int)D, (int)rpb);
    });
  } else {
    rmsnorm_bwd_kernel<<<nb, 256, smem, s>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
                                             (const __nv_bfloat16*)go, inv_rms, (__nv_bfloat16*)gx, gw_part, R,
                                             (int)D, (int)rpb);
  }
  CCB_CHECK_LAUNCH("rmsnorm_bwd");
  return 0;
}
// gw_out: fp32, or bf16 with gw_bf16; may be null.
extern "C" int ccb_rmsnorm_bwd_as(const void* x, const void* w, const void* go, const float* inv_rms,
                                  void* gx, float* gw_part, void* gw_out, int64_t gw_bf16, int64_t R, int64_t D,
                                  void* stream) {
  if (R <= 0) return 0;
  if (D > RMSNORM_BWD_MAX_DIM) return set_error("ccb_rmsnorm_bwd: D=%lld exceeds %d", (long long)D, RMSNORM_BWD_MAX_DIM);
  const int rc = launch_rmsnorm_bwd(x, w, go, inv_rms, gx, gw_part, R, D, rmsnorm_bwd_rows(R), (cudaStream_t)stream);
  if (rc || !gw_out) return rc;
  return launch_colsum(gw_part, ccb_rmsnorm_bwd_blocks(R), D, gw_out, (int)gw_bf16, 0, (cudaStream_t)stream);
}
extern "C" int ccb_rmsnorm_bwd(const void* x, const void* w, const void* go, const float* inv_rms,
                               void* gx, float* gw_part, float* gw_out, int64_t R, int64_t D,
                               void* stream) {
  return ccb_rmsnorm_bwd_as(x, w, go, inv_rms, gx, gw_part, gw_out, 0, R, D, stream);
}

static inline int muon_blocks_per_mat(int64_t G, int64_t numel_per_mat) {
  int cap = (int)(G >= 16 ? 74 : 1184 / G);
  if ((int64_t)cap * G > MUON_PART_SLOTS) cap = (int)(MUON_PART_SLOTS / G);
  return grid_for(numel_per_mat, 256, cap < 1 ? 1 : cap);
}
// The two calls form one unit: normalize reads the per-block sums the momentum launch left in the
// per-device scratch, so they must run back to back on one stream with the same (G, numel_per_mat).
extern "C" int ccb_muon_momentum(const float* g, float* buf, void* dir, float* sumsq, int64_t G,
                                 int64_t numel_per_mat, float mu, int64_t nesterov, void* stream) {
  if (G <= 0 || numel_per_mat <= 0) return 0;
  if (G > MUON_PART_SLOTS) return set_error("ccb_muon_momentum: at most %d matrices per call", MUON_PART_SLOTS);
  (void)sumsq;
  dim3 grid((unsigned)muon_blocks_per_mat(G, numel_per_mat), (unsigned)G);
  muon_momentum_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(g, buf, (__nv_bfloat16*)dir,
                                                               numel_per_mat, mu, (int)nesterov);
  CCB_CHECK_LAUNCH("muon_momentum");
  return 0;
}
extern "C" int ccb_muon_normalize(void* dir, float* sumsq, int64_t G, int64_t numel_per_mat,
                                  float eps, void* stream) {
  if (G <= 0 || numel_per_mat <= 0) return 0;
  if (G > MUON_PART_SLOTS) return set_error("ccb_muon_normalize: at most %d matrices per call", MUON_PART_SLOTS);
  const int nparts = muon_blocks_per_mat(G, numel_per_mat);
  dim3 grid((unsigned)nparts, (unsigned)G);
  muon_normalize_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)dir, sumsq, nparts,
                                                                numel_per_mat, eps);
  CCB_CHECK_LAUNCH("muon_normalize");
  return 0;
}
extern "C" int ccb_muon_apply(void* p, const void* O, int64_t n, float lr_scale, float decay_mul,
                              void* stream) {
  if (n <= 0) return 0;
  muon_apply_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
      (__nv_bfloat16*)p, (const __nv_bfloat16*)O, n, lr_scale, decay_mul);
  CCB_CHECK_LAUNCH("muon_apply");
  return 0;
}
extern "C" int ccb_adamw(void* p, int64_t p_is_bf16, const float* g, float* m, float* v, int64_t n,
                         float lr, float b1, float b2, float eps, float wd, float bias1,
                         float bias2_sqrt, const float* gscale, void* stream) {
  if (n <= 0) return 0;
  if (p_is_bf16)
    adamw_kernel<__nv_bfloat16><<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
        (__nv_bfloat16*)p, g, m, v, n, lr, b1, b2, eps, wd, bias1, bias2_sqrt, gscale);
  else
    adamw_kernel<float><<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
        (float*)p, g, m, v, n, lr, b1, b2, eps, wd, bias1, bias2_sqrt, gscale);
  CCB_CHECK_LAUNCH("adamw");
  return 0;
}
// stat: 3 floats {sumsq, coef, norm}.  Computes the global L2 norm of g[0:n]
// and multiplies g by min(1, max_norm / (norm + 1e-6)) without a host sync.
extern "C" int ccb_clip_grad_norm(float* g, int64_t n, float max_norm, float* stat, void* stream) {
  if (n <= 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const int nb = grid_for(n, 256, SUMSQ_MAX_BLOCKS);
  sumsq_kernel<<<nb, 256, 0, s>>>(g, n);
  CCB_CHECK_LAUNCH("sumsq");
  clip_coef_kernel<<<1, 256, 0, s>>>(stat, nb, max_norm);
  CCB_CHECK_LAUNCH("clip_coef");
  scale_by_ptr_kernel<<<grid_for(n, 256), 256, 0, s>>>(g, n, stat + 1);
  CCB_CHECK_LAUNCH("scale_by_ptr");
  return 0;
}
extern "C" int ccb_sgd(void* p, const float* g, int64_t n, float lr, void* stream) {
  if (n <= 0) return 0;
  sgd_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)p, g, n, lr);
  CCB_CHECK_LAUNCH("sgd");
  return 0;
}
extern "C" int ccb_lse_combine(const float* part, int64_t nparts, int64_t M, const float* zt, float* lse,
                               float* loss, void* stream) {
  if (M <= 0) return 0;
  // Warps to a row: one while its partials are two rounds of loads, sixteen for long lists of few rows, else four.
  // 1 / 4 / 16 in us (events, cold L2): 65 536 rows of 4 partials 8 / 8 / 16, of 32 14 / 12 / 23, of 128 38 / 22 / 30;
  // 9000 rows of 64 21 / 10 / 10, of 128 33 / 14 / 10; 20 000 rows of 128 33 / 15 / 15; 511 rows of 32 12 / 8 / 8.
  const int pw = nparts <= 8 ? 1 : (nparts > 32 && M <= 16384 ? 16 : 4);
  const long long rows = 32 * (LSC_WARPS / pw);
  auto kern = pw == 1 ? lse_combine_kernel<1> : (pw == 4 ? lse_combine_kernel<4> : lse_combine_kernel<16>);
  kern<<<(unsigned)((M + rows - 1) / rows), 32 * LSC_WARPS, 0, (cudaStream_t)stream>>>(
      (const float2*)part, (int)nparts, (long long)M, zt, lse, loss);
  CCB_CHECK_LAUNCH("lse_combine");
  return 0;
}
extern "C" int ccb_cast_f32_to_bf16(const float* s, void* d, int64_t n, float scale, void* stream) {
  if (n <= 0) return 0;
  cast_f32_to_bf16_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(s, (__nv_bfloat16*)d, n,
                                                                              scale);
  CCB_CHECK_LAUNCH("cast_f32_to_bf16");
  return 0;
}
extern "C" int ccb_cast_bf16_to_f32(const void* s, float* d, int64_t n, float scale,
                                    int64_t accumulate, void* stream) {
  if (n <= 0) return 0;
  cast_bf16_to_f32_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)s, d, n, scale, (int)accumulate);
  CCB_CHECK_LAUNCH("cast_bf16_to_f32");
  return 0;
}

// ---------------------------------------------------------------------------
// Allocation-free RMSNorm backward (declared in ccb_noalloc.h).
// The per-block partial weight gradients live in an array that is part of the
// library image instead of a buffer handed in by the caller.
// ---------------------------------------------------------------------------
#include "ccb_noalloc.h"

namespace {
constexpr int64_t kNoallocRowsPerBlock = 256;
constexpr int64_t kNoallocMaxBlocks = CCB_NOALLOC_RMSNORM_MAX_ROWS / kNoallocRowsPerBlock;
// 256 blocks x 1024 channels x 4 B = 1 MiB, resident on every device that loads the library.
static __device__ __align__(256) float g_noalloc_rmsnorm_part[kNoallocMaxBlocks *
                                                               CCB_NOALLOC_RMSNORM_MAX_DIM];
// In host code the array's name is only a handle; the kernels need the device
// address, looked up once per device with that device current.
static float* g_noalloc_part_ptr[16] = {nullptr};
}  // namespace

extern "C" int ccb_rmsnorm_bwd_noalloc(const void* x, const void* w, const void* go,
                                       const float* inv_rms, void* gx, float* gw_out, int64_t R,
                                       int64_t D, void* stream) {
  if (R <= 0) return 0;
  if (R > CCB_NOALLOC_RMSNORM_MAX_ROWS)
    return set_error("ccb_rmsnorm_bwd_noalloc: R=%lld exceeds the built-in workspace (max %d rows)",
                     (long long)R, CCB_NOALLOC_RMSNORM_MAX_ROWS);
  if (D <= 0 || D > CCB_NOALLOC_RMSNORM_MAX_DIM || (D % 2) != 0)
    return set_error("ccb_rmsnorm_bwd_noalloc: D=%lld unsupported (even, max %d)", (long long)D,
                     CCB_NOALLOC_RMSNORM_MAX_DIM);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_error("cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= 16) return set_error("ccb_rmsnorm_bwd_noalloc: device index %d unsupported", dev);
  if (g_noalloc_part_ptr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_noalloc_rmsnorm_part);
    if (e != cudaSuccess || p == nullptr)
      return set_error("cudaGetSymbolAddress(workspace): %s", cudaGetErrorString(e));
    g_noalloc_part_ptr[dev] = p;
  }
  float* part = g_noalloc_part_ptr[dev];
  const unsigned nb = (unsigned)((R + kNoallocRowsPerBlock - 1) / kNoallocRowsPerBlock);
  cudaStream_t s = (cudaStream_t)stream;
  const int rc = launch_rmsnorm_bwd(x, w, go, inv_rms, gx, part, R, D, kNoallocRowsPerBlock, s);
  if (rc) return rc;
  return launch_colsum(part, nb, D, gw_out, 0, 0, s);
}
