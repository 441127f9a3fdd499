// Flash attention for sm_100a: QK^T and PV (and the five backward products) on tcgen05 with the
// accumulators in TMEM, operands staged by non-multicast TMA into 128-byte-swizzled shared memory.
//
// Layout: q [B, T, H, hd], k / v [B, T, Hkv, hd] (bf16, hd contiguous, hd = 64 or 128), out like q;
// T a multiple of 128. Causal and/or document-segmented (block-diagonal) masks; grouped-query
// attention by head // (H / Hkv). The log-sum-exp is kept per (b, h, t) in base-2 units of the
// scaled scores for the backward.
//
// Forward: CTAs walk the (128 query rows, head, batch) items, longest first, two CTAs to an SM; warps 0-3 = softmax
// (one query row per thread = one TMEM lane), warp 4 = TMA producer, warp 5 = MMA issuer. Keys come 64 at a time:
//     S = Q K_n^T  (TMEM, two buffers)  ->  online softmax in registers  ->  P_n (bf16, TMEM)  ->  O += P_n V_n (TMEM)
// S of the next 64 keys is formed while the softmax warps work on the current ones, also across items, so they wait
// neither for the tensor pipe nor for a new item's first loads. A row's scores are read once into registers; P goes
// back to tensor memory over the scores it came from, as the A operand of P V, and never touches shared memory. O
// stays in TMEM and is rescaled only when a row's maximum grows by more than 2^8 over the one its exponents refer to
// (l, O and the final quotient share that reference, so the result is the same). Tiles off the diagonal of
// unsegmented calls take no mask arithmetic. 256 TMEM columns and at most 98 KB a CTA; K and V halves share one ring in the
// order the tensor pipe takes them. What bounds it is the exponentials (16 lanes a clock: 1024 cycles per 128 x 128).
// B 64, T 512, 12 heads of 64: 152 us with one 128-key S at a time, P through shared memory and O in registers, 88 us
// now; B 4, T 2048, 32 / 8 heads of 128: 440 -> 174 us (790 TFLOP/s). One item per CTA and 128 keys a step: 100, 215 us.
//
// Backward, one CTA per (128 key rows, kv head, batch), looping over the query heads of the group
// and the query tiles that see this key tile:
//     S = Q_i K_j^T, dP = dO_i V_j^T (TMEM) -> P = exp2(S - L), dS = P * (dP - D) * scale (bf16, shared)
//     dV += P^T dO_i, dK += dS^T Q_i (TMEM, across the whole loop), dQ_i = dS K_j (TMEM -> fp32 atomics)
// P and dS are written once, row-major in the key index, and read both as a K-major operand (dQ) and
// as an MN-major operand (the transposed products), which the descriptor's major bits allow.
//
// Every wait is bounded; on a time-out the status word is set and all roles leave.
//
// Replaces the reference's cuDNN fused attention and its tokamax Mosaic alternative
// (param_decomp/attention.py:116-137,148-245).
#include <algorithm>

#include "attention_common.cuh"

namespace {

using namespace pd_attn;

struct AttnArgs {
  int B, T, H, Hkv;
  int causal;
  float scale_log2;       // log2(e) / sqrt(hd)
  float scale;            // 1 / sqrt(hd)
  const int* segment_ids; // [B, T] or null
  __nv_bfloat16* out;     // [B, T, H, hd]
  float* lse;             // [B, H, T] base-2 log-sum-exp of the scaled scores
  // backward only
  const float* delta;     // [B, H, T] rowsum(dO * O)
  float* dq_accum;        // [B, T, H, hd] fp32, zero on entry
  __nv_bfloat16* dk;      // [B, T, Hkv, hd]
  __nv_bfloat16* dv;
  int* status;
};

constexpr int kSub = 64;  // keys per softmax step of the forward

template <int HD>
struct FwdPlan {
  static constexpr int kQBytes = kTile * HD * 2;
  static constexpr int kSlotBytes = kSub * HD * 2;      // 64 rows of K or V
  static constexpr int kSlots = HD == 64 ? 8 : 4;       // 64 KB: a CTA stays under half an SM's shared memory
  static constexpr int kTotal = kQBytes + kSlots * kSlotBytes + 1024 /*align*/ + 256 /*barriers*/ + 4 * kSub * 4 /*segment ids*/;
  static constexpr uint32_t kTmemCols = 256;            // S / P buffers [0, 64) and [64, 128), O [128, 128 + hd)
};
constexpr float kRescaleLog2 = 8.0f;

// The 64-key steps of the items a CTA walks (w, w + stride, ...), in order.
struct StepCursor {
  const AttnArgs& a;
  int w, stride, items, n_qt;
  int j = 0, n_sub = 0, qt = 0, h = 0, b = 0;
  __device__ StepCursor(const AttnArgs& args, int first, int step) : a(args), w(first), stride(step) {
    n_qt = a.T / kTile;
    items = n_qt * a.H * a.B;
    open();
  }
  __device__ bool done() const { return w >= items; }
  __device__ bool last() const { return j + 1 == n_sub; }
  __device__ void open() {  // longest items first; neighbours share K and V of a (batch, kv head)
    if (done()) return;
    const int hb = w % (a.H * a.B);
    qt = n_qt - 1 - w / (a.H * a.B);
    h = hb % a.H;
    b = hb / a.H;
    n_sub = (kTile / kSub) * (a.causal ? qt + 1 : n_qt);
  }
  __device__ void advance() {
    if (++j == n_sub) {
      j = 0;
      w += stride;
      open();
    }
  }
};

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
template <int HD>
__global__ void __launch_bounds__(kFwdThreads, 2) attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                  const __grid_constant__ CUtensorMap tmK,
                                                                  const __grid_constant__ CUtensorMap tmV,
                                                                  const AttnArgs args) {
  using Plan = FwdPlan<HD>;
  constexpr int kSlots = Plan::kSlots;
  constexpr int kKB = HD / 64;  // 64-wide K blocks of the head dimension
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sm_q = base;
  const uint32_t sm_kv = sm_q + Plan::kQBytes;
  const uint32_t sm_bar = sm_kv + kSlots * Plan::kSlotBytes;
  // barriers: q_full, q_empty, slot_full[8], slot_empty[8], s_full[2], p_full[2], o_full, o_empty
  const uint32_t bar_qf = sm_bar, bar_qe = bar_qf + 8;
  const uint32_t bar_f = bar_qe + 8, bar_e = bar_f + 64, bar_s = bar_e + 64, bar_p = bar_s + 16;
  const uint32_t bar_o = bar_p + 16, bar_oe = bar_o + 8;
  const uint32_t tmem_slot = bar_oe + 8;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gbase + (tmem_slot - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + (tmem_slot + 4 - base));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* seg_k = reinterpret_cast<int*>(gbase + (sm_bar + 256 - base)) + (warp & 3) * kSub;  // a softmax warp's ids

  if (threadIdx.x == 0) {
    mbar_init(bar_qf, 1);
    mbar_init(bar_qe, 1);
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(bar_f + 8 * i, 1);
      mbar_init(bar_e + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_s + 8 * i, 1);
      mbar_init(bar_p + 8 * i, kSoftmaxThreads);
    }
    mbar_init(bar_o, 1);
    mbar_init(bar_oe, kSoftmaxThreads);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, Plan::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = *tmem_slot_ptr;
  const uint32_t tmem_o = tmem_s + 2 * kSub;
  const int w0 = static_cast<int>(blockIdx.x), wstep = static_cast<int>(gridDim.x);

  // Producer and MMA issuer walk one sequence of tensor steps: S_0, S_1, then P V_n, S_{n+2} for every n. Each step
  // takes the next slot of the ring (64 rows of K for S, of V for P V).
  if (warp == 4) {
    // ---------------- TMA producer (whole warp walks the loop, one elected lane issues) ----------------
    StepCursor sc(args, w0, wstep), vc(args, w0, wstep);
    uint32_t slot = 0, phase = 0, q_count = 0;
    bool ok = true;
    auto load = [&](const StepCursor& c, const CUtensorMap* tm) {
      ok = mbar_wait_warp(bar_e + 8 * slot, phase ^ 1, abort_flag);
      if (!ok) return;
      if (elect_one_sync()) {
        mbar_expect_tx(bar_f + 8 * slot, Plan::kSlotBytes);
        const int hk = c.h / (args.H / args.Hkv);
        for (int i = 0; i < kKB; ++i)
          tma_load_3d(sm_kv + slot * Plan::kSlotBytes + i * (kSub * 128), tm, bar_f + 8 * slot, hk * HD + 64 * i,
                      c.j * kSub, c.b);
      }
      if (++slot == kSlots) {
        slot = 0;
        phase ^= 1;
      }
    };
    auto next_k = [&]() {
      if (sc.done()) return;
      if (sc.j == 0) {  // a new item: its queries, once the last S of the item before has been formed
        ok = mbar_wait_warp(bar_qe, (q_count & 1) ^ 1, abort_flag);
        if (!ok) return;
        ++q_count;
        if (elect_one_sync()) {
          mbar_expect_tx(bar_qf, Plan::kQBytes);
          for (int i = 0; i < kKB; ++i) tma_load_3d(sm_q + i * (kTile * 128), &tmQ, bar_qf, sc.h * HD + 64 * i, sc.qt * kTile, sc.b);
        }
      }
      load(sc, &tmK);
      sc.advance();
    };
    next_k();
    if (ok) next_k();
    while (ok && !vc.done()) {
      load(vc, &tmV);
      vc.advance();
      if (ok) next_k();
    }
    if (!ok && lane == 0) atomicCAS(args.status, 0, kTimeoutProducer);
  } else if (warp == 5) {
    // ---------------- MMA issuer (whole warp walks the loop, one elected lane issues) ----------------
    constexpr uint32_t idesc_s = make_idesc_bf16(kTile, kSub, 0, 0);
    constexpr uint32_t idesc_o = make_idesc_bf16(kTile, HD, 0, 1);
    StepCursor sc(args, w0, wstep), vc(args, w0, wstep);
    uint32_t slot = 0, phase = 0, q_count = 0, s_count = 0, v_count = 0, o_count = 0;
    bool ok = true;
    auto advance_slot = [&]() {
      if (++slot == kSlots) {
        slot = 0;
        phase ^= 1;
      }
    };
    auto next_s = [&]() {
      if (sc.done()) return;
      if (sc.j == 0) {
        ok = mbar_wait_warp(bar_qf, q_count & 1, abort_flag);
        ++q_count;
      }
      if (ok) ok = mbar_wait_warp(bar_f + 8 * slot, phase, abort_flag);
      if (!ok) return;
      tc_fence_after();
      if (elect_one_sync()) {
        const uint32_t d = tmem_s + (s_count & 1) * kSub;
#pragma unroll
        for (int c = 0; c < kKB; ++c) {
          const uint64_t ad = make_smem_desc(sm_q + c * (kTile * 128), 16, 1024);
          const uint64_t bd = make_smem_desc(sm_kv + slot * Plan::kSlotBytes + c * (kSub * 128), 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(d, ad + k * 2, bd + k * 2, idesc_s, (c > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(bar_e + 8 * slot);
        umma_commit(bar_s + 8 * (s_count & 1));
        if (sc.last()) umma_commit(bar_qe);
      }
      ++s_count;
      advance_slot();
      sc.advance();
    };
    next_s();
    if (ok) next_s();
    while (ok && !vc.done()) {
      // P_n is in tensor memory; the softmax warps are done with S_n and with rescaling O
      const uint32_t buf = v_count & 1;
      ok = mbar_wait_warp(bar_p + 8 * buf, (v_count >> 1) & 1, abort_flag) &&
           mbar_wait_warp(bar_f + 8 * slot, phase, abort_flag);
      if (ok && vc.j == 0) {  // O of the item before has been read out
        ok = mbar_wait_warp(bar_oe, (o_count & 1) ^ 1, abort_flag);
        ++o_count;
      }
      if (!ok) break;
      tc_fence_after();
      if (elect_one_sync()) {
        const uint64_t vd = make_smem_desc(sm_kv + slot * Plan::kSlotBytes, kSub * 128, 1024);
#pragma unroll
        for (int k = 0; k < kSub / 16; ++k)  // 16 keys: eight columns of P, two 8-row groups of V
          umma_bf16_ts(tmem_o, tmem_s + buf * kSub + 8 * k, vd + k * (2048 >> 4), idesc_o, (vc.j > 0 || k > 0) ? 1u : 0u);
        umma_commit(bar_e + 8 * slot);
        umma_commit(bar_o);
      }
      advance_slot();
      vc.advance();
      if (!sc.done()) {  // S_{n+2} overwrites P_n: P V_n has read it
        ok = mbar_wait_warp(bar_o, v_count & 1, abort_flag);
        if (ok) next_s();
      }
      ++v_count;
    }
    if (!ok && lane == 0) atomicCAS(args.status, 0, kTimeoutMma);
  } else {
    // ---------------- softmax + output (one query row per thread) ----------------
    const int row = threadIdx.x;  // 0..127 = TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const f32x2 scale2 = pk2(args.scale_log2, args.scale_log2);
    uint32_t n = 0;  // steps so far: S buffer n & 1
    bool ok = true;
    StepCursor sc(args, w0, wstep);
    while (ok && !sc.done()) {
      const int q_idx = sc.qt * kTile + row;
      const int* seg_row = args.segment_ids ? args.segment_ids + static_cast<long long>(sc.b) * args.T : nullptr;
      const int seg_q = seg_row ? seg_row[q_idx] : 0;
      float m_ref = -INFINITY;  // the maximum the exponents of l and O refer to
      f32x2 l2 = 0ull;
      const int diag_j = args.causal ? sc.qt * (kTile / kSub) : 0x7FFFFFFF;  // steps from here on cross the diagonal
      for (int j = 0; j < sc.n_sub; ++j, ++n) {
        if (seg_row) {  // the warp's own copy of the step's ids
          __syncwarp();
#pragma unroll
          for (int c = 0; c < kSub / 32; ++c) seg_k[c * 32 + lane] = seg_row[j * kSub + c * 32 + lane];
          __syncwarp();
        }
        const uint32_t buf = n & 1;
        if (!mbar_wait_warp(bar_s + 8 * buf, (n >> 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_sp = tmem_s + buf * kSub + lane_base;
        uint32_t r[2][32];
#pragma unroll
        for (int c = 0; c < 2; ++c) tmem_ld_32x32(tmem_sp + c * 32, r[c]);
        tmem_ld_wait();
        constexpr uint32_t kNegInf = 0xFF800000u;
        if (j >= diag_j) {
          const int lim = row - (j - diag_j) * kSub;  // last key column this row sees
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > lim) r[c][i] = kNegInf;
        }
        if (seg_row) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const int4 id = *reinterpret_cast<const int4*>(seg_k + c * 32 + i);
              if (id.x != seg_q) r[c][i] = kNegInf;
              if (id.y != seg_q) r[c][i + 1] = kNegInf;
              if (id.z != seg_q) r[c][i + 2] = kNegInf;
              if (id.w != seg_q) r[c][i + 3] = kNegInf;
            }
        }
        float mx[4];  // four chains of the row maximum (the scale is positive)
#pragma unroll
        for (int c = 0; c < 4; ++c) mx[c] = __uint_as_float(r[c >> 1][(c & 1) * 16]);
#pragma unroll
        for (int i = 1; i < 16; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) mx[c] = fmaxf(mx[c], __uint_as_float(r[c >> 1][(c & 1) * 16 + i]));
        const float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * args.scale_log2;
        const bool grow = j == 0 ? m_tile > -INFINITY : m_tile > m_ref + kRescaleLog2;
        if (j == 0) {
          if (grow) m_ref = m_tile;
        } else if (__any_sync(0xffffffffu, grow)) {
          const float alpha = grow ? fast_exp2(m_ref - m_tile) : 1.0f;  // 0 where nothing was seen before
          if (grow) m_ref = m_tile;
          l2 = mul2(l2, pk2(alpha, alpha));
          if (!mbar_wait_warp(bar_o, (n - 1) & 1, abort_flag)) { ok = false; break; }
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < HD / 16; ++c) {
            uint32_t o[16];
            tmem_ld_16(tmem_o + lane_base + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_16(tmem_o + lane_base + c * 16, o);
          }
        }
        const float m_sub = m_ref == -INFINITY ? 0.0f : -m_ref;  // a row with nothing kept yet: exp2(-inf) = 0
        const f32x2 m2 = pk2(m_sub, m_sub);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t packed[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = unpack2(fma2(pk2u(r[c][2 * i], r[c][2 * i + 1]), scale2, m2));
            packed[i] = pack_bf16(fast_exp2(x.x), fast_exp2(x.y));
            l2 = add2(l2, unpack_bf16_2(packed[i]));  // the sum uses the rounded values the tensor core will see
          }
          tmem_st_16(tmem_sp + c * 16, packed);
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(bar_p + 8 * buf);
      }
      if (!ok) break;
      // both of the last two P V may still run, and a parity only tells neighbouring phases apart: wait for each
      if (!mbar_wait_warp(bar_o, (n - 2) & 1, abort_flag) || !mbar_wait_warp(bar_o, (n - 1) & 1, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const float2 lp = unpack2(l2);
      const float l_run = lp.x + lp.y;
      const float inv = 1.0f / l_run;
      __nv_bfloat16* dst = args.out + ((static_cast<long long>(sc.b) * args.T + q_idx) * args.H + sc.h) * HD;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem_o + lane_base + c * 32, o);
        tmem_ld_wait();
        if (c == HD / 32 - 1) {  // the tensor pipe may start on the next item's O
          tc_fence_before();
          mbar_arrive(bar_oe);
        }
        float f[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(o[i]) * inv;
#pragma unroll
        for (int g = 0; g < 4; ++g)
          *reinterpret_cast<uint4*>(dst + c * 32 + 8 * g) =
              make_uint4(pack_bf16(f[8 * g], f[8 * g + 1]), pack_bf16(f[8 * g + 2], f[8 * g + 3]),
                         pack_bf16(f[8 * g + 4], f[8 * g + 5]), pack_bf16(f[8 * g + 6], f[8 * g + 7]));
      }
      if (args.lse) args.lse[(static_cast<long long>(sc.b) * args.H + sc.h) * args.T + q_idx] = m_ref + log2f(l_run);
      sc.j = sc.n_sub - 1;
      sc.advance();
    }
    if (!ok) atomicCAS(args.status, 0, kTimeoutEpilogue);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem_s, Plan::kTmemCols);
}

// ------------------------------------------------------------------------------------------------
// backward
// ------------------------------------------------------------------------------------------------
// D[b, h, t] = sum_d dO * O  (one warp per row)
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                  float* __restrict__ delta, int B, int T, int H, int hd) {
  const long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);  // (b, t, h)
  if (row >= static_cast<long long>(B) * T * H) return;
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* po = o + row * hd;
  const __nv_bfloat16* pd = d_o + row * hd;
  float acc = 0.0f;
  for (int i = lane * 2; i < hd; i += 64) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(po + i));
    const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(pd + i));
    acc += a.x * g.x + a.y * g.y;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (lane == 0) {
    const long long bt = row / H;
    const int h = static_cast<int>(row % H);
    const long long b = bt / T, t = bt % T;
    delta[(b * H + h) * T + t] = acc;
  }
}

__global__ void attn_dq_cast_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, long long n) {
  for (long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x * 4) {
    const float4 v = *reinterpret_cast<const float4*>(acc + i);
    uint2 o;
    o.x = pack_bf16(v.x, v.y);
    o.y = pack_bf16(v.z, v.w);
    *reinterpret_cast<uint2*>(dq + i) = o;
  }
}

template <int HD>
struct BwdPlan {
  static constexpr int kTileBytes = kTile * HD * 2;  // K, V, Q or dO tile
  static constexpr int kStages = HD == 64 ? 2 : 1;   // Q / dO ring
  static constexpr int kPBytes = kTile * kTile * 2;
  static constexpr int kTotal = 2 * kTileBytes + 2 * kStages * kTileBytes + 2 * kPBytes + 1024 + 1024;
  // TMEM: [0,128) S, later dQ; [128,256) dP; [256,256+HD) dV; [256+HD, 256+2HD) dK
  static constexpr uint32_t kTmemCols = 512;
};

template <int HD>
__global__ void __launch_bounds__(kFwdThreads, 1) attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                   const __grid_constant__ CUtensorMap tmK,
                                                                   const __grid_constant__ CUtensorMap tmV,
                                                                   const __grid_constant__ CUtensorMap tmdO,
                                                                   const AttnArgs args) {
  using Plan = BwdPlan<HD>;
  constexpr int kStages = Plan::kStages;
  constexpr int kKB = HD / 64;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sm_k = base;
  const uint32_t sm_v = sm_k + Plan::kTileBytes;
  const uint32_t sm_q = sm_v + Plan::kTileBytes;
  const uint32_t sm_do = sm_q + kStages * Plan::kTileBytes;
  const uint32_t sm_p = sm_do + kStages * Plan::kTileBytes;
  const uint32_t sm_ds = sm_p + Plan::kPBytes;
  const uint32_t sm_bar = sm_ds + Plan::kPBytes;
  // barriers: kv_full, qdo_full[2], qdo_empty[2], sdp_full, pds_full, dq_full, dq_empty, final
  const uint32_t bar_kv = sm_bar;
  const uint32_t bar_qf = bar_kv + 8, bar_qe = bar_qf + 16;
  const uint32_t bar_sdp = bar_qe + 16, bar_pds = bar_sdp + 8, bar_dqf = bar_pds + 8, bar_dqe = bar_dqf + 8;
  const uint32_t bar_fin = bar_dqe + 8;
  const uint32_t tmem_slot = bar_fin + 8;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gbase + (tmem_slot - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + (tmem_slot + 4 - base));
  int* seg_k = reinterpret_cast<int*>(gbase + (sm_bar + 256 - base));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_qt = args.T / kTile;
  const int kt = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
  const int group = args.H / args.Hkv;
  const int qt_lo = args.causal ? kt : 0;
  const int per_head = n_qt - qt_lo;
  const int n_it = per_head * group;  // iteration it -> head hk*group + it / per_head, q tile qt_lo + it % per_head

  if (threadIdx.x == 0) {
    mbar_init(bar_kv, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_qf + 8 * s, 1);
      mbar_init(bar_qe + 8 * s, 1);
    }
    mbar_init(bar_sdp, 1);
    mbar_init(bar_pds, kSoftmaxThreads);
    mbar_init(bar_dqf, 1);
    mbar_init(bar_dqe, kSoftmaxThreads);
    mbar_init(bar_fin, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, Plan::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = *tmem_slot_ptr;
  const uint32_t tmem_dp = tmem_s + 128;
  const uint32_t tmem_dv = tmem_s + 256;
  const uint32_t tmem_dk = tmem_dv + HD;

  if (warp == 4) {
    if (elect_one_sync()) {
      mbar_expect_tx(bar_kv, 2 * Plan::kTileBytes);
      for (int c = 0; c < kKB; ++c) {
        tma_load_3d(sm_k + c * (kTile * 128), &tmK, bar_kv, hk * HD + 64 * c, kt * kTile, b);
        tma_load_3d(sm_v + c * (kTile * 128), &tmV, bar_kv, hk * HD + 64 * c, kt * kTile, b);
      }
    }
    for (int it = 0; it < n_it; ++it) {
      const int st = it % kStages;
      const uint32_t ph = static_cast<uint32_t>((it / kStages) & 1);
      if (!mbar_wait_warp(bar_qe + 8 * st, ph ^ 1, abort_flag)) {
        if (lane == 0) atomicCAS(args.status, 0, kTimeoutProducer);
        break;
      }
      const int h = hk * group + it / per_head;
      const int qt = qt_lo + it % per_head;
      if (elect_one_sync()) {
        mbar_expect_tx(bar_qf + 8 * st, 2 * Plan::kTileBytes);
        for (int c = 0; c < kKB; ++c) {
          tma_load_3d(sm_q + st * Plan::kTileBytes + c * (kTile * 128), &tmQ, bar_qf + 8 * st, h * HD + 64 * c,
                      qt * kTile, b);
          tma_load_3d(sm_do + st * Plan::kTileBytes + c * (kTile * 128), &tmdO, bar_qf + 8 * st, h * HD + 64 * c,
                      qt * kTile, b);
        }
      }
    }
  } else if (warp == 5) {
    {
      constexpr uint32_t idesc_s = make_idesc_bf16(kTile, kTile, 0, 0);   // Q K^T, dO V^T
      constexpr uint32_t idesc_t = make_idesc_bf16(kTile, HD, 1, 1);      // P^T dO, dS^T Q
      constexpr uint32_t idesc_q = make_idesc_bf16(kTile, HD, 0, 1);      // dS K
      bool ok = mbar_wait_warp(bar_kv, 0, abort_flag);
      for (int it = 0; it < n_it && ok; ++it) {
        const int st = it % kStages;
        if (!mbar_wait_warp(bar_qf + 8 * st, static_cast<uint32_t>((it / kStages) & 1), abort_flag)) { ok = false; break; }
        // the softmax warps have read dQ of the previous iteration out of the S columns
        if (!mbar_wait_warp(bar_dqe, static_cast<uint32_t>((it & 1) ^ 1), abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t q_s = sm_q + st * Plan::kTileBytes, do_s = sm_do + st * Plan::kTileBytes;
        if (elect_one_sync()) {
#pragma unroll
          for (int c = 0; c < kKB; ++c) {
            const uint64_t qd = make_smem_desc(q_s + c * (kTile * 128), 16, 1024);
            const uint64_t kd = make_smem_desc(sm_k + c * (kTile * 128), 16, 1024);
            const uint64_t dod = make_smem_desc(do_s + c * (kTile * 128), 16, 1024);
            const uint64_t vd = make_smem_desc(sm_v + c * (kTile * 128), 16, 1024);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              umma_bf16(tmem_s, qd + k * 2, kd + k * 2, idesc_s, (c > 0 || k > 0) ? 1u : 0u);
              umma_bf16(tmem_dp, dod + k * 2, vd + k * 2, idesc_s, (c > 0 || k > 0) ? 1u : 0u);
            }
          }
          umma_commit(bar_sdp);
        }
        if (!mbar_wait_warp(bar_pds, static_cast<uint32_t>(it & 1), abort_flag)) { ok = false; break; }
        tc_fence_after();
        if (elect_one_sync()) {
          // transposed products: A = P or dS read MN-major (K = query rows), B = dO or Q read MN-major
          const uint64_t pt = make_smem_desc(sm_p, kTile * 128, 1024);
          const uint64_t dst = make_smem_desc(sm_ds, kTile * 128, 1024);
          const uint64_t dob = make_smem_desc(do_s, kTile * 128, 1024);
          const uint64_t qb = make_smem_desc(q_s, kTile * 128, 1024);
#pragma unroll
          for (int k = 0; k < kTile / 16; ++k) {
            umma_bf16(tmem_dv, pt + k * (2048 >> 4), dob + k * (2048 >> 4), idesc_t, (it > 0 || k > 0) ? 1u : 0u);
            umma_bf16(tmem_dk, dst + k * (2048 >> 4), qb + k * (2048 >> 4), idesc_t, (it > 0 || k > 0) ? 1u : 0u);
          }
          // dQ_i = dS K_j: A = dS K-major in the key index, B = K_j read MN-major (K = key rows)
          const uint64_t kb_ = make_smem_desc(sm_k, kTile * 128, 1024);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint64_t dsd = make_smem_desc(sm_ds + c * (kTile * 128), 16, 1024);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_bf16(tmem_s, dsd + k * 2, kb_ + (c * 4 + k) * (2048 >> 4), idesc_q, (c > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit(bar_qe + 8 * st);
          umma_commit(bar_dqf);
        }
      }
      if (ok && elect_one_sync()) umma_commit(bar_fin);
      if (!ok && lane == 0) atomicCAS(args.status, 0, kTimeoutMma);
    }
  } else {
    const int row = threadIdx.x;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    if (args.segment_ids) seg_k[row] = args.segment_ids[b * args.T + kt * kTile + row];
    named_barrier_softmax();
    bool ok = true;
    uint32_t r[32], g[32];
    for (int it = 0; it < n_it && ok; ++it) {
      const int h = hk * group + it / per_head;
      const int qt = qt_lo + it % per_head;
      const int q_idx = qt * kTile + row;
      const long long stat = (static_cast<long long>(b) * args.H + h) * args.T + q_idx;
      const float L = args.lse[stat];
      const float Dq = args.delta[stat];
      const int seg_q = args.segment_ids ? args.segment_ids[b * args.T + q_idx] : 0;
      const bool diag = args.causal && qt == kt;
      if (!mbar_wait(bar_sdp, static_cast<uint32_t>(it & 1), abort_flag)) { ok = false; break; }
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        tmem_ld_32x32(tmem_s + lane_base + c * 32, r);
        tmem_ld_32x32(tmem_dp + lane_base + c * 32, g);
        tmem_ld_wait();
        uint32_t pp[16], dd[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float p2[2], d2[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int col = c * 32 + i + e;  // key index inside the tile
            const bool keep = (!diag || col <= row) && (!args.segment_ids || seg_k[col] == seg_q);
            const float p = keep ? fast_exp2(__uint_as_float(r[i + e]) * args.scale_log2 - L) : 0.0f;
            p2[e] = p;
            d2[e] = p * (__uint_as_float(g[i + e]) - Dq) * args.scale;
          }
          pp[i >> 1] = pack_bf16(p2[0], p2[1]);
          dd[i >> 1] = pack_bf16(d2[0], d2[1]);
        }
        const uint32_t off = (c >> 1) * (kTile * 128);
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const uint32_t a = swz(row, (c & 1) * 4 + q4);
          st_shared_v4(sm_p + off + a, make_uint4(pp[4 * q4], pp[4 * q4 + 1], pp[4 * q4 + 2], pp[4 * q4 + 3]));
          st_shared_v4(sm_ds + off + a, make_uint4(dd[4 * q4], dd[4 * q4 + 1], dd[4 * q4 + 2], dd[4 * q4 + 3]));
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      mbar_arrive(bar_pds);
      // dQ_i tile -> fp32 accumulation buffer (other key tiles add to the same rows)
      if (!mbar_wait(bar_dqf, static_cast<uint32_t>(it & 1), abort_flag)) { ok = false; break; }
      tc_fence_after();
      float* dq_row = args.dq_accum + ((static_cast<long long>(b) * args.T + q_idx) * args.H + h) * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        tmem_ld_32x32(tmem_s + lane_base + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          atomicAdd(reinterpret_cast<float4*>(dq_row + c * 32 + i),
                    make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]),
                                __uint_as_float(r[i + 3])));
      }
      tc_fence_before();
      mbar_arrive(bar_dqe);
    }
    if (ok) {
      if (n_it > 0) {
        if (!mbar_wait(bar_fin, 0, abort_flag)) ok = false;
      }
      if (ok) {
        tc_fence_after();
        const long long krow = ((static_cast<long long>(b) * args.T + kt * kTile + row) * args.Hkv + hk) * HD;
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          __nv_bfloat16* dst = (which == 0 ? args.dv : args.dk) + krow;
          const uint32_t src = (which == 0 ? tmem_dv : tmem_dk) + lane_base;
#pragma unroll 1
          for (int c = 0; c < HD / 32; ++c) {
            if (n_it > 0) {
              tmem_ld_32x32(src + c * 32, r);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0u;
            }
#pragma unroll
            for (int q8 = 0; q8 < 4; ++q8) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(r[8 * q8]), __uint_as_float(r[8 * q8 + 1]));
              v.y = pack_bf16(__uint_as_float(r[8 * q8 + 2]), __uint_as_float(r[8 * q8 + 3]));
              v.z = pack_bf16(__uint_as_float(r[8 * q8 + 4]), __uint_as_float(r[8 * q8 + 5]));
              v.w = pack_bf16(__uint_as_float(r[8 * q8 + 6]), __uint_as_float(r[8 * q8 + 7]));
              *reinterpret_cast<uint4*>(dst + c * 32 + 8 * q8) = v;
            }
          }
        }
      }
    }
    if (!ok) atomicCAS(args.status, 0, kTimeoutEpilogue);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem_s, Plan::kTmemCols);
}

template <int HD>
int launch_fwd(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const AttnArgs& a, cudaStream_t st) {
  auto kern = attn_fwd_kernel<HD>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdPlan<HD>::kTotal) != cudaSuccess)
      return 300;
    configured = true;
  }
  const long long items = static_cast<long long>(a.T / kTile) * a.H * a.B;
  if (items > 0x3FFFFFFF) return kBadArgument;
  kern<<<static_cast<unsigned>(std::min<long long>(items, 2 * 148)), kFwdThreads, FwdPlan<HD>::kTotal, st>>>(q, k, v, a);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}

template <int HD>
int launch_bwd(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& d_o,
               const AttnArgs& a, cudaStream_t st) {
  auto kern = attn_bwd_kernel<HD>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdPlan<HD>::kTotal) != cudaSuccess)
      return 300;
    configured = true;
  }
  dim3 grid(a.T / kTile, a.Hkv, a.B);
  kern<<<grid, kFwdThreads, BwdPlan<HD>::kTotal, st>>>(q, k, v, d_o, a);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}

}  // namespace

extern "C" int pd_flash_attention_fwd(const void* q, const void* k, const void* v, void* out, float* lse,
                                      const int* segment_ids, int B, int T, int H, int Hkv, int hd, int causal,
                                      int* status, void* stream) {
  if (bad_shape(B, T, H, Hkv, hd) || status == nullptr) return pd::kBadArgument;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = encode_bthd(&tq, q, B, T, H, hd)) != 0) return 1000 + rc;
  if ((rc = encode_bthd(&tk, k, B, T, Hkv, hd, kSub)) != 0) return 1000 + rc;
  if ((rc = encode_bthd(&tv, v, B, T, Hkv, hd, kSub)) != 0) return 1000 + rc;
  AttnArgs a{};
  a.B = B; a.T = T; a.H = H; a.Hkv = Hkv; a.causal = causal;
  a.scale = 1.0f / sqrtf(static_cast<float>(hd));
  a.scale_log2 = a.scale * kLog2e;
  a.segment_ids = segment_ids;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.lse = lse;
  a.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return hd == 64 ? launch_fwd<64>(tq, tk, tv, a, st) : launch_fwd<128>(tq, tk, tv, a, st);
}

// `delta` [B, H, T] fp32 and `dq_accum` [B, T, H, hd] fp32 are scratch supplied by the caller;
// `dq_accum` must be zero on entry.
extern "C" int pd_flash_attention_bwd(const void* q, const void* k, const void* v, const void* out, const void* d_out,
                                      const float* lse, float* delta, float* dq_accum, void* dq, void* dk, void* dv,
                                      const int* segment_ids, int B, int T, int H, int Hkv, int hd, int causal,
                                      int* status, void* stream) {
  if (bad_shape(B, T, H, Hkv, hd) || status == nullptr) return pd::kBadArgument;
  CUtensorMap tq, tk, tv, tdo;
  int rc;
  if ((rc = encode_bthd(&tq, q, B, T, H, hd)) != 0) return 1000 + rc;
  if ((rc = encode_bthd(&tk, k, B, T, Hkv, hd)) != 0) return 1000 + rc;
  if ((rc = encode_bthd(&tv, v, B, T, Hkv, hd)) != 0) return 1000 + rc;
  if ((rc = encode_bthd(&tdo, d_out, B, T, H, hd)) != 0) return 1000 + rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long rows = static_cast<long long>(B) * T * H;
  attn_delta_kernel<<<static_cast<unsigned>((rows + 7) / 8), 256, 0, st>>>(
      static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out), delta, B, T, H, hd);
  AttnArgs a{};
  a.B = B; a.T = T; a.H = H; a.Hkv = Hkv; a.causal = causal;
  a.scale = 1.0f / sqrtf(static_cast<float>(hd));
  a.scale_log2 = a.scale * kLog2e;
  a.segment_ids = segment_ids;
  a.lse = const_cast<float*>(lse);
  a.delta = delta;
  a.dq_accum = dq_accum;
  a.dk = static_cast<__nv_bfloat16*>(dk);
  a.dv = static_cast<__nv_bfloat16*>(dv);
  a.status = status;
  rc = hd == 64 ? launch_bwd<64>(tq, tk, tv, tdo, a, st) : launch_bwd<128>(tq, tk, tv, tdo, a, st);
  if (rc != 0) return rc;
  const long long n = rows * hd;
  attn_dq_cast_kernel<<<static_cast<unsigned>(std::min<long long>((n / 4 + 255) / 256, 148 * 16)), 256, 0, st>>>(
      dq_accum, static_cast<__nv_bfloat16*>(dq), n);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}
