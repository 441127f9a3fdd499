// Gated delta rule (linear-attention recurrence of the Qwen3.5 DeltaNet layers) and the causal
// depthwise conv1d + SiLU in front of it, forward and backward.
//
//   S_t = exp(g_t) S_{t-1};  delta_t = beta_t (v_t - S_t^T k_t);  S_t += k_t delta_t^T;  o_t = S_t^T q_t
//
// Everything is fp32. The columns of the state [DK, DV] never meet in the recurrence, so the two serial passes
// (the state forward, its cotangent backward) give each column to four lanes of a warp, 32 columns to a block and
// DV / 32 blocks to a (batch, head): 64 heads of 128 x 128 then make 1024 warps instead of 256, and a token costs a
// warp one pass over 32 registers and two shuffles. k, q and the block's values arrive 16 tokens at a time by cp.async.
// Bound by the chain of a token (two warps a scheduler, issue slots 36% busy) and the shared-memory pipe (61 - 65%).
//
// What else the backward needs - dq, dk, dg, dbeta - are sums over columns. They leave the serial chain: within a
// 64-token chunk they are products of [64, 64], [64, DK] and [64, DV] tiles with the chunk's boundary states, one block
// per (batch, head, chunk) (`delta_chunk_grads_kernel`). The forward keeps v - (decayed state)^T k per token and the
// state at chunk starts; the backward pass over the cotangent keeps it at chunk ends.
//
// Forward + backward, B 4, T 512, H 16, 128 x 128: 7.62 ms with one thread per column, the state of every token
// written out and read back in the backward, and two passes over shared memory per token;
// 0.76 ms so, errors against 64 bits 1.1e-7 .. 2.6e-7 (1.5e-7 .. 3.2e-7 before).
//
// Replaces the XLA einsum + scan lowering of param_decomp/target_ports/qwen3_5_moe.py:89-158,187-293;
// the torch restatement of the same recurrence (`models/ports.py`) is the oracle.
#include "common.cuh"

namespace {

using pd::f32x2;
using pd::fma2;
using pd::mul2;
using pd::pk2;

constexpr int kChunk = 64;    // tokens between stored states
constexpr int kStage = 16;    // tokens per cp.async stage of the serial passes (divides kChunk)
constexpr int kCols = 32;     // state columns per block of the serial passes
constexpr int kSerialThreads = 128;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(pd::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(pd::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ float sum2(f32x2 v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo + hi;
}
__device__ __forceinline__ float quad_sum(float v) {  // over the four lanes of a column
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// One stage of the serial passes: kStage tokens of k, q, the block's columns of v (or d_o), g and beta.
template <int DK>
struct Stage {
  float k[kStage][DK], q[kStage][DK], val[kStage][kCols];
  float g[kStage], beta[kStage];
  float decay[kStage], kq[kStage];  // exp(g), k . q: filled in after arrival
};

template <int DK>
__device__ __forceinline__ void load_stage(Stage<DK>& s, const float* k, const float* q, const float* val,
                                           const float* g, const float* beta, long long row0, int H, int DV, int col0,
                                           int t0, int n) {
  const int tid = threadIdx.x;
  for (int i = tid; i < n * (DK / 4); i += kSerialThreads) {
    const int r = i / (DK / 4), c = (i % (DK / 4)) * 4;
    const long long at = (row0 + static_cast<long long>(t0 + r) * H) * DK + c;
    cp_async16(&s.k[r][c], k + at);
    cp_async16(&s.q[r][c], q + at);
  }
  for (int i = tid; i < n * (kCols / 4); i += kSerialThreads) {
    const int r = i / (kCols / 4), c = (i % (kCols / 4)) * 4;
    cp_async16(&s.val[r][c], val + (row0 + static_cast<long long>(t0 + r) * H) * DV + col0 + c);
  }
  if (tid < n) {
    cp_async4(&s.g[tid], g + row0 + static_cast<long long>(t0 + tid) * H);
  } else if (tid >= 32 && tid - 32 < n) {
    cp_async4(&s.beta[tid - 32], beta + row0 + static_cast<long long>(t0 + tid - 32) * H);
  }
  cp_async_commit();
}

// exp(g) and k . q of the arrived tokens, a warp per token (with the quad's four parts a dot would cost every warp
// of the block 2 * DK / 8 more instructions per token).
template <int DK>
__device__ __forceinline__ void finish_stage(Stage<DK>& s, int n) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = warp; t < n; t += kSerialThreads / 32) {
    float d = 0.0f;
#pragma unroll
    for (int i = 0; i < DK; i += 32) d = fmaf(s.k[t][i + lane], s.q[t][i + lane], d);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (lane == 0) {
      s.kq[t] = d;
      s.decay[t] = static_cast<float>(exp(static_cast<double>(s.g[t])));
    }
  }
}

// grid (B * H, DV / kCols). A lane holds rows 16 i + 4 part + {0..3} of its column. Both dots of a token read the
// state before its update (o = a S^T q + (k . q) delta), so the token is one pass and one shuffle tree.
// `resid` [B, T, H, DV] (v - a S^T k) and `ckpt` [B * H, chunks, DV, DK] (state at chunk starts) may be null.
template <int DK>
__global__ void __launch_bounds__(kSerialThreads) delta_fwd_kernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ g,
    const float* __restrict__ beta, float* __restrict__ o, float* __restrict__ resid, float* __restrict__ ckpt, int T,
    int H, int DV) {
  __shared__ __align__(16) Stage<DK> stages[2];
  constexpr int NI = DK / 16;  // float4 pieces per lane
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  const int lane = threadIdx.x & 31, part = lane & 3;
  const int cl = (threadIdx.x >> 5) * 8 + (lane >> 2);  // column within the block
  const int col0 = blockIdx.y * kCols, col = col0 + cl;
  const long long row0 = static_cast<long long>(b) * T * H + h;
  const int n_chunks = (T + kChunk - 1) / kChunk;
  f32x2 S[2 * NI];
#pragma unroll
  for (int i = 0; i < 2 * NI; ++i) S[i] = 0ull;
  load_stage(stages[0], k, q, v, g, beta, row0, H, DV, col0, 0, min(kStage, T));
  for (int t0 = 0, buf = 0; t0 < T; t0 += kStage, buf ^= 1) {
    const int n = min(kStage, T - t0);
    Stage<DK>& s = stages[buf];
    cp_async_wait_all();
    __syncthreads();
    finish_stage(s, n);
    __syncthreads();  // also: every warp has left the other buffer
    if (t0 + kStage < T)
      load_stage(stages[buf ^ 1], k, q, v, g, beta, row0, H, DV, col0, t0 + kStage, min(kStage, T - t0 - kStage));
    if (ckpt != nullptr && t0 % kChunk == 0) {
      float* c = ckpt + ((static_cast<long long>(blockIdx.x) * n_chunks + t0 / kChunk) * DV + col) * DK;
#pragma unroll
      for (int i = 0; i < NI; ++i)
        *reinterpret_cast<ulonglong2*>(c + 16 * i + 4 * part) = make_ulonglong2(S[2 * i], S[2 * i + 1]);
    }
#pragma unroll 2
    for (int t = 0; t < n; ++t) {
      f32x2 kk[2 * NI];
      f32x2 m0 = 0ull, m1 = 0ull, p0 = 0ull, p1 = 0ull;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(&s.k[t][16 * i + 4 * part]);
        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(&s.q[t][16 * i + 4 * part]);
        kk[2 * i] = kv.x;
        kk[2 * i + 1] = kv.y;
        m0 = fma2(S[2 * i], kv.x, m0);
        m1 = fma2(S[2 * i + 1], kv.y, m1);
        p0 = fma2(S[2 * i], qv.x, p0);
        p1 = fma2(S[2 * i + 1], qv.y, p1);
      }
      const float a = s.decay[t];
      const float m = quad_sum(sum2(m0) + sum2(m1));
      const float p = quad_sum(sum2(p0) + sum2(p1));
      const float r = fmaf(-a, m, s.val[t][cl]);
      const float delta = r * s.beta[t];
      const f32x2 a2 = pk2(a, a), d2 = pk2(delta, delta);
#pragma unroll
      for (int i = 0; i < 2 * NI; ++i) S[i] = fma2(kk[i], d2, mul2(S[i], a2));
      if (part == 0) {
        const long long at = (row0 + static_cast<long long>(t0 + t) * H) * DV + col;
        o[at] = fmaf(a, p, delta * s.kq[t]);
        if (resid != nullptr) resid[at] = r;
      }
    }
  }
}

// The cotangent G of the state, last token first, split over columns like the forward:
//   d delta_t = (G + q do^T)^T k = G^T k + (k . q) do;   G <- a (G + q do^T - beta k d delta^T)
// `ddelta` [B, T, H, DV]; `gck` [B * H, chunks, DV, DK]: G as it enters each chunk's last token.
template <int DK>
__global__ void __launch_bounds__(kSerialThreads) delta_bwd_state_kernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ d_o,
    const float* __restrict__ g, const float* __restrict__ beta, float* __restrict__ ddelta, float* __restrict__ gck,
    int T, int H, int DV) {
  __shared__ __align__(16) Stage<DK> stages[2];
  constexpr int NI = DK / 16;
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  const int lane = threadIdx.x & 31, part = lane & 3;
  const int cl = (threadIdx.x >> 5) * 8 + (lane >> 2);
  const int col0 = blockIdx.y * kCols, col = col0 + cl;
  const long long row0 = static_cast<long long>(b) * T * H + h;
  const int n_chunks = (T + kChunk - 1) / kChunk;
  f32x2 G[2 * NI];
#pragma unroll
  for (int i = 0; i < 2 * NI; ++i) G[i] = 0ull;
  int t0 = (T - 1) / kStage * kStage;
  load_stage(stages[0], k, q, d_o, g, beta, row0, H, DV, col0, t0, T - t0);
  for (int buf = 0; t0 >= 0; t0 -= kStage, buf ^= 1) {
    const int n = min(kStage, T - t0);
    Stage<DK>& s = stages[buf];
    cp_async_wait_all();
    __syncthreads();
    finish_stage(s, n);
    __syncthreads();
    if (t0 > 0) load_stage(stages[buf ^ 1], k, q, d_o, g, beta, row0, H, DV, col0, t0 - kStage, kStage);
    if ((t0 + n) % kChunk == 0 || t0 + n == T) {
      float* c = gck + ((static_cast<long long>(blockIdx.x) * n_chunks + t0 / kChunk) * DV + col) * DK;
#pragma unroll
      for (int i = 0; i < NI; ++i)
        *reinterpret_cast<ulonglong2*>(c + 16 * i + 4 * part) = make_ulonglong2(G[2 * i], G[2 * i + 1]);
    }
#pragma unroll 2
    for (int t = n - 1; t >= 0; --t) {
      const float a = s.decay[t], dot = s.val[t][cl];
      const f32x2 a2 = pk2(a, a), do2 = pk2(dot, dot);
      f32x2 kk[2 * NI];
      f32x2 m0 = 0ull, m1 = 0ull;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(&s.k[t][16 * i + 4 * part]);
        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(&s.q[t][16 * i + 4 * part]);
        kk[2 * i] = kv.x;
        kk[2 * i + 1] = kv.y;
        m0 = fma2(G[2 * i], kv.x, m0);
        m1 = fma2(G[2 * i + 1], kv.y, m1);
        G[2 * i] = fma2(qv.x, do2, G[2 * i]);
        G[2 * i + 1] = fma2(qv.y, do2, G[2 * i + 1]);
      }
      const float dd = fmaf(s.kq[t], dot, quad_sum(sum2(m0) + sum2(m1)));
      const float dm = -s.beta[t] * dd;
      const f32x2 dm2 = pk2(dm, dm);
#pragma unroll
      for (int i = 0; i < 2 * NI; ++i) G[i] = mul2(a2, fma2(kk[i], dm2, G[i]));
      if (part == 0) ddelta[(row0 + static_cast<long long>(t0 + t) * H) * DV + col] = dd;
    }
  }
}

// ---- gradients of one chunk --------------------------------------------------------------------------------------
// With delta = beta resid, dm = -beta ddelta, D[u, s] = exp(g_{s+1} + .. + g_u), S the state before the chunk, G the
// cotangent after it, L_t = D[t, before the chunk], R_t = D[last, t]:
//   dq_t = L_t S do_t + sum_{s <= t} D[t, s] (do_t . delta_s) k_s
//   dk_t = L_t S dm_t + R_t G delta_t + sum_{u >= t} D[u, t] (do_u . delta_t) q_u
//          + sum_{u > t} D[u, t] (dm_u . delta_t) k_u + sum_{s < t} D[t, s] (dm_t . delta_s) k_s
//   dg_t = <a S_{t-1}, G_t + k_t dm_t^T>, expanded over the same terms: pairs s < t <= u, tokens u >= t against S,
//          tokens s < t against G, and exp(sum g) <S, G>. Every term is added, none is a difference of running sums,
//          so the result keeps the accuracy of a direct sum.
//   dv_t = beta ddelta_t, dbeta_t = ddelta_t . resid_t.
// Decays are differences of a running sum of g kept in 64 bits (in 32 its rounding would show in D), as are the
// exponentials and the few hundred final additions of dg. A g below -10^4 enters the sum as -10^4: exp of either is 0 in
// 32 bits, but with -inf the differences past it would be NaN and with -10^18 the later terms of the sum would be lost.
// 256 threads, a thread owns 4 tokens x DK / 16 columns of dq, dk. 7.3 M FMA per chunk at 128 x 128; the
// operand tiles take 217 KB of shared memory, one block per SM. Two warps a scheduler at 222 registers leave latency bare:
// FMA pipe 35%, shared-memory pipe 39%, issue slots 29% busy.
constexpr int kGradThreads = 256;
constexpr float kMinLogDecay = -1.0e4f;
__device__ __forceinline__ double log_decay(float g) { return g < kMinLogDecay ? kMinLogDecay : g; }
constexpr int kSlice = 16;          // rows of S^T / G^T staged at a time
constexpr int kWPitch = kChunk + 4;

template <int DK, int DV>
struct GradPlan {
  static constexpr int kPK = DK + 4, kPV = DV + 4;  // pitches: 16-byte rows, neighbouring rows in other banks
  static constexpr int kTiles = 2 * kChunk * kPK + 3 * kChunk * kPV;
  static constexpr int kPairs = kChunk * kChunk > 2 * kSlice * DK ? kChunk * kChunk : 2 * kSlice * DK;
  static constexpr int kFloats = kTiles + 2 * kChunk * kWPitch + kPairs + 8 * kChunk + 2 * kChunk /* 64-bit sums */;
  static constexpr int kBytes = kFloats * 4;
};

template <int NP>
__device__ __forceinline__ void load_pairs(const float* row, int tx, f32x2 (&out)[NP]) {
  if constexpr (NP == 1) {
    out[0] = *reinterpret_cast<const f32x2*>(row + 2 * tx);
  } else {
#pragma unroll
    for (int h = 0; h < NP / 2; ++h) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(row + 64 * h + 4 * tx);
      out[2 * h] = v.x;
      out[2 * h + 1] = v.y;
    }
  }
}
template <int NP>
__device__ __forceinline__ void store_pairs(float* row, int tx, const f32x2 (&v)[NP]) {
  if constexpr (NP == 1) {
    *reinterpret_cast<f32x2*>(row + 2 * tx) = v[0];
  } else {
#pragma unroll
    for (int h = 0; h < NP / 2; ++h)
      *reinterpret_cast<ulonglong2*>(row + 64 * h + 4 * tx) = make_ulonglong2(v[2 * h], v[2 * h + 1]);
  }
}

template <int DK, int DV>
__global__ void __launch_bounds__(kGradThreads, 1) delta_chunk_grads_kernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ d_o,
    const float* __restrict__ resid, const float* __restrict__ g, const float* __restrict__ beta,
    const float* __restrict__ ckpt, const float* __restrict__ gck, float* __restrict__ dq, float* __restrict__ dk,
    float* __restrict__ dv /* holds ddelta on entry */, float* __restrict__ dg, float* __restrict__ dbeta, int T,
    int H) {
  using Plan = GradPlan<DK, DV>;
  constexpr int PK = Plan::kPK, PV = Plan::kPV, NP = DK / 32;
  extern __shared__ __align__(16) float smem[];
  float* sQ = smem;
  float* sK = sQ + kChunk * PK;
  float* sDo = sK + kChunk * PK;
  float* sDe = sDo + kChunk * PV;  // delta
  float* sDm = sDe + kChunk * PV;
  float* sW1 = sDm + kChunk * PV;       // [u][s] D (do_u . delta_s), s <= u
  float* sW2 = sW1 + kChunk * kWPitch;  // symmetric: D (dm_u . delta_s) at [u][s] and [s][u], s < u
  float* sM = sW2 + kChunk * kWPitch;   // pair terms of dg, later the S^T / G^T slices
  double* s_cum = reinterpret_cast<double*>(sM + Plan::kPairs);
  float* s_beta = reinterpret_cast<float*>(s_cum + kChunk);
  float* s_L = s_beta + kChunk;
  float* s_R = s_L + kChunk;
  float* s_x = s_R + kChunk;
  float* s_y = s_x + kChunk;
  float* s_rect = s_y + kChunk;
  float* s_db = s_rect + kChunk;
  float* s_red = s_db + kChunk;  // [64]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = tid >> 4, tx = tid & 15;
  const int c = blockIdx.y, n_chunks = gridDim.y;
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  const long long row0 = (static_cast<long long>(b) * T + static_cast<long long>(c) * kChunk) * H + h;
  const int n = min(kChunk, T - c * kChunk);

  if (warp == 0) {  // running sum of g: two tokens per lane
    const double g0 = 2 * lane < n ? log_decay(g[row0 + static_cast<long long>(2 * lane) * H]) : 0.0;
    const double g1 = 2 * lane + 1 < n ? log_decay(g[row0 + static_cast<long long>(2 * lane + 1) * H]) : 0.0;
    double acc = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, acc, o);
      if (lane >= o) acc += up;
    }
    const double total = __shfl_sync(0xffffffffu, acc, 31);
    const double c0 = acc - g1;
    s_cum[2 * lane] = c0;
    s_cum[2 * lane + 1] = acc;
    s_L[2 * lane] = static_cast<float>(exp(c0));
    s_L[2 * lane + 1] = static_cast<float>(exp(acc));
    s_R[2 * lane] = static_cast<float>(exp(total - c0));
    s_R[2 * lane + 1] = static_cast<float>(exp(total - acc));
  } else if (warp < 4) {
    const int t = tid - 32;
    if (t < kChunk) s_beta[t] = t < n ? beta[row0 + static_cast<long long>(t) * H] : 0.0f;
  }
  for (int i = tid; i < kChunk * (DK / 4); i += kGradThreads) {
    const int r = i / (DK / 4), d = (i % (DK / 4)) * 4;
    float4 qv = make_float4(0.f, 0.f, 0.f, 0.f), kv = qv;
    if (r < n) {
      const long long at = (row0 + static_cast<long long>(r) * H) * DK + d;
      qv = *reinterpret_cast<const float4*>(q + at);
      kv = *reinterpret_cast<const float4*>(k + at);
    }
    *reinterpret_cast<float4*>(sQ + r * PK + d) = qv;
    *reinterpret_cast<float4*>(sK + r * PK + d) = kv;
  }
  __syncthreads();
  for (int r = warp; r < kChunk; r += kGradThreads / 32) {  // a warp per token
    const float bt = s_beta[r];
    const long long at = (row0 + static_cast<long long>(r) * H) * DV;
    float db = 0.0f;
#pragma unroll
    for (int j = lane; j < DV; j += 32) {
      float o = 0.0f, rs = 0.0f, dd = 0.0f;
      if (r < n) {
        o = d_o[at + j];
        rs = resid[at + j];
        dd = dv[at + j];
        dv[at + j] = bt * dd;
      }
      sDo[r * PV + j] = o;
      sDe[r * PV + j] = bt * rs;
      sDm[r * PV + j] = -bt * dd;
      db = fmaf(dd, rs, db);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) db += __shfl_xor_sync(0xffffffffu, db, o);
    if (lane == 0) s_db[r] = db;
  }
  __syncthreads();

  // ---- [64, 64] products: this thread's rows u = 4 ty + r, columns s = tx + 16 e ----
  {
    float a1[4][4], a2[4][4];
    f32x2 acc1[4][4], acc2[4][4];
    auto clear = [&]() {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc1[r][e] = acc2[r][e] = 0ull;
    };
    auto grams = [&](const float* A1, const float* A2, const float* Bm, int pitch, int width) {
#pragma unroll 2
      for (int j = 0; j < width; j += 4) {
        ulonglong2 x1[4], x2[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          x1[r] = *reinterpret_cast<const ulonglong2*>(A1 + (4 * ty + r) * pitch + j);
          x2[r] = *reinterpret_cast<const ulonglong2*>(A2 + (4 * ty + r) * pitch + j);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(Bm + (tx + 16 * e) * pitch + j);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            acc1[r][e] = fma2(x1[r].x, y.x, acc1[r][e]);
            acc2[r][e] = fma2(x2[r].x, y.x, acc2[r][e]);
            acc1[r][e] = fma2(x1[r].y, y.y, acc1[r][e]);
            acc2[r][e] = fma2(x2[r].y, y.y, acc2[r][e]);
          }
        }
      }
    };
    clear();
    grams(sDo, sDm, sDe, PV, DV);  // do_u . delta_s, dm_u . delta_s
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a1[r][e] = sum2(acc1[r][e]);
        a2[r][e] = sum2(acc2[r][e]);
      }
    clear();
    grams(sQ, sK, sK, PK, DK);  // q_u . k_s, k_u . k_s
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int u = 4 * ty + r, s = tx + 16 * e;
        float w1 = 0.0f, m = 0.0f;
        if (s <= u) {
          const float d = static_cast<float>(exp(s_cum[u] - s_cum[s]));
          w1 = d * a1[r][e];
          if (s < u) {
            const float w2 = d * a2[r][e];
            m = fmaf(w1, sum2(acc1[r][e]), w2 * sum2(acc2[r][e]));
            sW2[u * kWPitch + s] = w2;
            sW2[s * kWPitch + u] = w2;
          } else {
            sW2[u * kWPitch + u] = 0.0f;
          }
        }
        sW1[u * kWPitch + s] = w1;
        sM[u * kChunk + s] = m;
      }
  }
  __syncthreads();
  {  // pairs s < t <= u of dg_t, four threads per token
    const int t = tid >> 2, part = tid & 3;
    double acc = 0.0;
    for (int u = t; u < kChunk; ++u)
      for (int s = part; s < t; s += 4) acc += sM[u * kChunk + s];
    const float hi = static_cast<float>(acc);
    acc = quad_sum(hi) + quad_sum(static_cast<float>(acc - hi));
    if (part == 0) s_rect[t] = acc;
  }
  __syncthreads();

  // ---- products with the boundary states, 16 value columns at a time ----
  f32x2 p1[4][NP], p2[4][NP], p3[4][NP];  // S do, S dm, G delta
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int p = 0; p < NP; ++p) p1[r][p] = p2[r][p] = p3[r][p] = 0ull;
  const long long state0 = (static_cast<long long>(blockIdx.x) * n_chunks + c) * DK * DV;
  float* sS = sM;
  float* sG = sM + kSlice * DK;
  constexpr int kPieces = (kSlice * DK / 4 + kGradThreads - 1) / kGradThreads;
  float4 nextS[kPieces], nextG[kPieces];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
      const int at = tid + i * kGradThreads;
      if (at < kSlice * DK / 4) {
        nextS[i] = *reinterpret_cast<const float4*>(ckpt + state0 + static_cast<long long>(j0) * DK + 4 * at);
        nextG[i] = *reinterpret_cast<const float4*>(gck + state0 + static_cast<long long>(j0) * DK + 4 * at);
      }
    }
  };
  float z = 0.0f;  // <S, G>
  fetch(0);
  for (int j0 = 0; j0 < DV; j0 += kSlice) {
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
      const int at = tid + i * kGradThreads;
      if (at < kSlice * DK / 4) {
        *reinterpret_cast<float4*>(sS + 4 * at) = nextS[i];
        *reinterpret_cast<float4*>(sG + 4 * at) = nextG[i];
        z = fmaf(nextS[i].x, nextG[i].x, fmaf(nextS[i].y, nextG[i].y, fmaf(nextS[i].z, nextG[i].z, fmaf(nextS[i].w, nextG[i].w, z))));
      }
    }
    __syncthreads();
    if (j0 + kSlice < DV) fetch(j0 + kSlice);
#pragma unroll
    for (int jj = 0; jj < kSlice; jj += 4) {
      float xo[4][4], xm[4][4], xe[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int at = (4 * ty + r) * PV + j0 + jj;
        *reinterpret_cast<float4*>(xo[r]) = *reinterpret_cast<const float4*>(sDo + at);
        *reinterpret_cast<float4*>(xm[r]) = *reinterpret_cast<const float4*>(sDm + at);
        *reinterpret_cast<float4*>(xe[r]) = *reinterpret_cast<const float4*>(sDe + at);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        f32x2 st[NP], gt[NP];
        load_pairs<NP>(sS + (jj + e) * DK, tx, st);
        load_pairs<NP>(sG + (jj + e) * DK, tx, gt);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const f32x2 o2 = pk2(xo[r][e], xo[r][e]), m2 = pk2(xm[r][e], xm[r][e]), e2 = pk2(xe[r][e], xe[r][e]);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            p1[r][p] = fma2(o2, st[p], p1[r][p]);
            p2[r][p] = fma2(m2, st[p], p2[r][p]);
            p3[r][p] = fma2(e2, gt[p], p3[r][p]);
          }
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  if (lane == 0) s_red[warp] = z;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int t = 4 * ty + r;
    const f32x2 L2 = pk2(s_L[t], s_L[t]), R2 = pk2(s_R[t], s_R[t]);
    f32x2 qv[NP], kv[NP], x2 = 0ull, y2 = 0ull;
    load_pairs<NP>(sQ + t * PK, tx, qv);
    load_pairs<NP>(sK + t * PK, tx, kv);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      p1[r][p] = mul2(L2, p1[r][p]);
      p2[r][p] = mul2(L2, p2[r][p]);
      p3[r][p] = mul2(R2, p3[r][p]);
      x2 = fma2(qv[p], p1[r][p], fma2(kv[p], p2[r][p], x2));
      y2 = fma2(kv[p], p3[r][p], y2);
      p2[r][p] = pd::add2(p2[r][p], p3[r][p]);
    }
    float x = sum2(x2), y = sum2(y2);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if (tx == 0) {
      s_x[t] = x;
      s_y[t] = y;
    }
  }
  // ---- pairs of tokens: dq += W1 K, dk += W2 K + W1^T Q ----
  for (int s = 0; s < kChunk; s += 4) {
    float w1[4][4], w2[4][4], wt[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      *reinterpret_cast<float4*>(w1[r]) = *reinterpret_cast<const float4*>(sW1 + (4 * ty + r) * kWPitch + s);
      *reinterpret_cast<float4*>(w2[r]) = *reinterpret_cast<const float4*>(sW2 + (4 * ty + r) * kWPitch + s);
      *reinterpret_cast<float4*>(wt[r]) = *reinterpret_cast<const float4*>(sW1 + (s + r) * kWPitch + 4 * ty);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f32x2 kv[NP], qv[NP];
      load_pairs<NP>(sK + (s + e) * PK, tx, kv);
      load_pairs<NP>(sQ + (s + e) * PK, tx, qv);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const f32x2 a = pk2(w1[r][e], w1[r][e]), bq = pk2(w2[r][e], w2[r][e]), ct = pk2(wt[e][r], wt[e][r]);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          p1[r][p] = fma2(a, kv[p], p1[r][p]);
          p2[r][p] = fma2(bq, kv[p], fma2(ct, qv[p], p2[r][p]));
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int t = 4 * ty + r;
    if (t < n) {
      const long long at = (row0 + static_cast<long long>(t) * H) * DK;
      store_pairs<NP>(dq + at, tx, p1[r]);
      store_pairs<NP>(dk + at, tx, p2[r]);
    }
  }
  __syncthreads();
  if (tid < n) {
    double acc = 0.0;
    for (int w = 0; w < kGradThreads / 32; ++w) acc += s_red[w];
    acc = s_L[kChunk - 1] * acc + s_rect[tid];
    for (int u = tid; u < kChunk; ++u) acc += s_x[u];
    for (int s = 0; s < tid; ++s) acc += s_y[s];
    dg[row0 + static_cast<long long>(tid) * H] = acc;
    dbeta[row0 + static_cast<long long>(tid) * H] = s_db[tid];
  }
}

// ---- causal depthwise conv1d + SiLU: y[b,t,c] = silu(sum_j w[c,j] x[b,t-(K-1)+j,c]) ----
__global__ void conv1d_silu_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                       __nv_bfloat16* __restrict__ y, int B, int T, int D, int K) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long total = static_cast<long long>(B) * T * D;
  if (idx >= total) return;
  const int c = static_cast<int>(idx % D);
  const int t = static_cast<int>((idx / D) % T);
  float acc = 0.0f;
  for (int j = 0; j < K; ++j) {
    const int ts = t - (K - 1) + j;
    if (ts >= 0) acc = fmaf(__bfloat162float(w[c * K + j]), __bfloat162float(x[idx + static_cast<long long>(ts - t) * D]), acc);
  }
  y[idx] = __float2bfloat16(acc / (1.0f + __expf(-acc)));
}

// dx[b,s,c] = sum_j w[c,j] dpre[b,s+(K-1)-j,c];  dw[c,j] += sum_{b,t} dpre[b,t,c] x[b,t-(K-1)+j,c]
__global__ void conv1d_silu_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                       const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx,
                                       float* __restrict__ dw, int B, int T, int D, int K) {
  // one thread per (b, c), walking t: keeps a K-deep window of dpre and x in registers (K <= 8)
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (c >= D) return;
  float wk[8], dwk[8], win_x[8];
  for (int j = 0; j < 8; ++j) {
    wk[j] = j < K ? __bfloat162float(w[c * K + j]) : 0.0f;
    dwk[j] = 0.0f;
    win_x[j] = 0.0f;  // x[t-(K-1)+j]
  }
  const long long base = static_cast<long long>(b) * T * D + c;
  // pass 1 (forward in t): dpre and dw
  for (int t = 0; t < T; ++t) {
    for (int j = 0; j + 1 < K; ++j) win_x[j] = win_x[j + 1];
    win_x[K - 1] = __bfloat162float(x[base + static_cast<long long>(t) * D]);
    float pre = 0.0f;
    for (int j = 0; j < K; ++j) pre = fmaf(wk[j], win_x[j], pre);
    const float sg = 1.0f / (1.0f + __expf(-pre));
    const float dpre = __bfloat162float(dy[base + static_cast<long long>(t) * D]) * sg * (1.0f + pre * (1.0f - sg));
    for (int j = 0; j < K; ++j) dwk[j] = fmaf(dpre, win_x[j], dwk[j]);
  }
  for (int j = 0; j < K; ++j) atomicAdd(dw + c * K + j, dwk[j]);
  // pass 2 (backward in t): dx[s] needs dpre[s .. s+K-1]; recompute dpre on the fly with a second window
  // window of x for recomputing pre at tokens s..s+K-1 would need 2K-1 values: simpler to recompute per token
  for (int s = T - 1; s >= 0; --s) {
    float acc = 0.0f;
    for (int j = 0; j < K; ++j) {
      const int t = s + (K - 1) - j;  // token whose window position j reads x[s]
      if (t >= T) continue;
      float pre = 0.0f;
      for (int jj = 0; jj < K; ++jj) {
        const int ts = t - (K - 1) + jj;
        if (ts >= 0) pre = fmaf(wk[jj], __bfloat162float(x[base + static_cast<long long>(ts) * D]), pre);
      }
      const float sg = 1.0f / (1.0f + __expf(-pre));
      const float dpre = __bfloat162float(dy[base + static_cast<long long>(t) * D]) * sg * (1.0f + pre * (1.0f - sg));
      acc = fmaf(wk[j], dpre, acc);
    }
    dx[base + static_cast<long long>(s) * D] = __float2bfloat16(acc);
  }
}

template <int DK, int DV>
int launch_fwd(const float* q, const float* k, const float* v, const float* g, const float* beta, float* o,
               float* resid, float* ckpt, int B, int T, int H, cudaStream_t st) {
  delta_fwd_kernel<DK><<<dim3(B * H, DV / kCols), kSerialThreads, 0, st>>>(q, k, v, g, beta, o, resid, ckpt, T, H, DV);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}

template <int DK, int DV>
int launch_bwd(const float* q, const float* k, const float* resid, const float* g, const float* beta,
               const float* d_o, const float* ckpt, float* gck, float* dq, float* dk, float* dv, float* dg,
               float* dbeta, int B, int T, int H, cudaStream_t st) {
  using Plan = GradPlan<DK, DV>;
  auto kern = delta_chunk_grads_kernel<DK, DV>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Plan::kBytes) != cudaSuccess) return 300;
  delta_bwd_state_kernel<DK><<<dim3(B * H, DV / kCols), kSerialThreads, 0, st>>>(q, k, d_o, g, beta, dv, gck, T, H, DV);
  kern<<<dim3(B * H, (T + kChunk - 1) / kChunk), kGradThreads, Plan::kBytes, st>>>(q, k, d_o, resid, g, beta, ckpt,
                                                                                gck, dq, dk, dv, dg, dbeta, T, H);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}

}  // namespace

#define PD_DELTA_DISPATCH(FN, ...)                                  \
  if (dk == 64 && dv == 64) return FN<64, 64>(__VA_ARGS__);         \
  if (dk == 128 && dv == 128) return FN<128, 128>(__VA_ARGS__);     \
  if (dk == 64 && dv == 128) return FN<64, 128>(__VA_ARGS__);       \
  if (dk == 32 && dv == 32) return FN<32, 32>(__VA_ARGS__);         \
  return pd::kBadArgument;

// q, k [B,T,H,dk], v, o [B,T,H,dv], g, beta [B,T,H] fp32 contiguous, q / k / v 16-byte aligned; for a backward pass
// resid [B,T,H,dv] and ckpt [B*H, ceil(T/64), dv, dk], else both null
extern "C" int pd_delta_rule_fwd(const float* q, const float* k, const float* v, const float* g, const float* beta,
                                 float* o, float* resid, float* ckpt, int B, int T, int H, int dk, int dv,
                                 void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  PD_DELTA_DISPATCH(launch_fwd, q, k, v, g, beta, o, resid, ckpt, B, T, H, st)
}

// gck: scratch like ckpt; d_o 16-byte aligned
extern "C" int pd_delta_rule_bwd(const float* q, const float* k, const float* resid, const float* g, const float* beta,
                                 const float* d_o, const float* ckpt, float* gck, float* dq, float* dk_, float* dv_,
                                 float* dg, float* dbeta, int B, int T, int H, int dk, int dv, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  PD_DELTA_DISPATCH(launch_bwd, q, k, resid, g, beta, d_o, ckpt, gck, dq, dk_, dv_, dg, dbeta, B, T, H, st)
}

extern "C" int pd_conv1d_silu_fwd(const void* x, const void* w, void* y, int B, int T, int D, int K, void* stream) {
  if (K < 1 || K > 8) return pd::kBadArgument;
  const long long total = static_cast<long long>(B) * T * D;
  conv1d_silu_fwd_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y), B, T,
      D, K);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}

// dw [D, K] fp32 must be zero on entry
extern "C" int pd_conv1d_silu_bwd(const void* x, const void* w, const void* dy, void* dx, float* dw, int B, int T,
                                  int D, int K, void* stream) {
  if (K < 1 || K > 8) return pd::kBadArgument;
  dim3 grid((D + 127) / 128, B);
  conv1d_silu_bwd_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w),
      static_cast<const __nv_bfloat16*>(dy), static_cast<__nv_bfloat16*>(dx), dw, B, T, D, K);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}
