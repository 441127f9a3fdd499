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
// back to tensor memory over the scores it came from, as the A operand of P V, and never touches shared memory (steps of
// published kernels: the online softmax of FlashAttention, P in tensor memory as in CUTLASS's Blackwell attention example). O
// stays in TMEM; a warp rescales its rows there when the maximum of one has grown. The exponents always refer to the
// running maximum: with an older one as reference (rescaling only past a growth of 2^8) a row's largest probability is a
// rounded number instead of exactly 1 and the error against 64 bits is 1.5 to 3% larger (forward 93 and 173 us so, 99 and
// 198 us as it is). Tiles off the diagonal of
// unsegmented calls take no mask arithmetic. 256 TMEM columns and at most 98 KB a CTA; K and V halves share one ring in the
// order the tensor pipe takes them. What bounds it is a warp's chain of load, maximum, exponentials and
// store per step: tensor pipe 26 / 51% (width 64 / 128), exponentials 39 / 41%, issue slots 43 / 48% busy.
// B 64, T 512, 12 heads of 64: 99 us (152 us with one 128-key S at a time, P through shared memory and O in registers);
// B 4, T 2048, 32 / 8 heads of 128: 198 us, 695 TFLOP/s (440 us).
//
// Backward, one CTA per (128 key rows, kv head, batch), looping over the query heads of the group
// and the query tiles that see this key tile:
//     S = Q_i K_j^T, dP = dO_i V_j^T (TMEM) -> P = exp2(S - L), dS = P * (dP - D) * scale (bf16, shared)
//     dV += P^T dO_i, dK += dS^T Q_i (TMEM, across the whole loop), dQ_i = dS K_j (TMEM -> fp32 reductions)
// P and dS are written once, row-major in the key index, and read both as a K-major operand (dQ) and
// as an MN-major operand (the transposed products), which the descriptor's major bits allow.
// Eight elementwise warps, two per TMEM lane quarter, take half of a tile's keys each; four more move dQ out (the
// reductions of a 128 x 128 dQ keep a warp's load-store path busy for 2000 cycles). The tensor pipe does not wait for a
// whole tile: S_{i+1} is issued once P_i is stored, dP_{i+1} once dS_i is (hd 64) or once dQ_i, which shares its
// columns, has been read out (hd 128, 512 TMEM columns). dQ sums in a scratch laid out [b, h, q tile][hd / 4][128 rows][4], so that a warp's 16-byte
// reductions are one contiguous 512-byte run; a last pass casts it to bf16 rows. The pass over dO and O that forms D
// also clears that scratch. With one warpgroup that took every step in turn and 16-byte atomics at row pitch, B 64,
// T 512, 12 heads of 64 took 420 us and B 4, T 2048, 32 / 8 heads of 128 995 us (D, scratch and cast included);
// now 289 and 580 us. What is left is the chain S -> P -> dP -> dS -> dQ of a tile, of which 512 columns hold one: tensor
// pipe 25 / 49% busy, every other unit less.
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
  float* dq_accum;        // [B, H, T / 128][hd / 4][128][4] fp32
  __nv_bfloat16* dk;      // [B, T, Hkv, hd]
  __nv_bfloat16* dv;
  int* status;
};

constexpr int kSub = 64;  // keys per softmax step of the forward
// P V_n reports on barrier n % kOutBars. A parity wait only tells neighbouring phases apart. When a softmax warp waits for
// P V_n, P V_{n-1} may be running or may have ended, P V_n may have ended too, and nothing later has been issued: with one
// barrier the state is one of three phases, with two it is "before" or "after".
constexpr int kOutBars = 2;

template <int HD>
struct FwdPlan {
  static constexpr int kQBytes = kTile * HD * 2;
  static constexpr int kSlotBytes = kSub * HD * 2;      // 64 rows of K or V
  static constexpr int kSlots = HD == 64 ? 8 : 4;       // 64 KB: a CTA stays under half an SM's shared memory
  static constexpr int kTotal = kQBytes + kSlots * kSlotBytes + 1024 /*align*/ + 256 /*barriers*/ + 4 * kSub * 4 /*segment ids*/;
  static constexpr uint32_t kTmemCols = 256;            // S / P buffers [0, 64) and [64, 128), O [128, 128 + hd)
};

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
  // barriers: q_full, q_empty, slot_full[8], slot_empty[8], s_full[2], p_full[2], o_full[2], o_empty
  const uint32_t bar_qf = sm_bar, bar_qe = bar_qf + 8;
  const uint32_t bar_f = bar_qe + 8, bar_e = bar_f + 64, bar_s = bar_e + 64, bar_p = bar_s + 16;
  const uint32_t bar_o = bar_p + 16, bar_oe = bar_o + 8 * kOutBars;
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
    for (int i = 0; i < kOutBars; ++i) mbar_init(bar_o + 8 * i, 1);
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
  auto wait_out = [&](uint32_t n) {  // until P V_n has ended
    return mbar_wait_warp(bar_o + 8 * (n % kOutBars), (n / kOutBars) & 1, abort_flag);
  };

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
        umma_commit(bar_o + 8 * (v_count % kOutBars));
      }
      advance_slot();
      vc.advance();
      if (!sc.done()) {  // S_{n+2} overwrites P_n: P V_n has read it
        ok = wait_out(v_count);
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
      float m_ref = -INFINITY;  // the row's running maximum, which the exponents of l and O refer to
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
        const float m_new = fmaxf(m_ref, m_tile);
        const float alpha = m_new > m_ref ? fast_exp2(m_ref - m_new) : 1.0f;  // 0 where nothing was seen before
        const bool rescale = j > 0 && __any_sync(0xffffffffu, m_new > m_ref);
        m_ref = m_new;
        l2 = mul2(l2, pk2(alpha, alpha));
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
        if (rescale) {  // last, so that P V_{n-1} has run beside the exponentials
          if (!wait_out(n - 1)) { ok = false; break; }
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
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(bar_p + 8 * buf);
      }
      if (!ok) break;
      if (!wait_out(n - 1)) {  // the pipe runs them in order: all of the item's P V have ended
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
// D[b, h, t] = sum_d dO * O, hd / 8 lanes per row; clears the dQ scratch on the way (as many floats as dO has values).
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                  float* __restrict__ delta, float* __restrict__ dq_accum, int B, int T, int H, int hd) {
  const long long rows = static_cast<long long>(B) * T * H, pieces = rows * (hd / 8);
  const int lpr = hd / 8;  // 8 or 16: a row never straddles a warp
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;  // 8 values
  float acc = 0.0f;
  if (i < pieces) {
    const uint4 a = *reinterpret_cast<const uint4*>(o + 8 * i), g = *reinterpret_cast<const uint4*>(d_o + 8 * i);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, gw[4] = {g.x, g.y, g.z, g.w};
    f32x2 t = 0ull;
#pragma unroll
    for (int k = 0; k < 4; ++k) t = fma2(unpack_bf16_2(aw[k]), unpack_bf16_2(gw[k]), t);
    const float2 t2 = unpack2(t);
    acc = t2.x + t2.y;
    reinterpret_cast<float4*>(dq_accum)[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f);
    reinterpret_cast<float4*>(dq_accum)[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int s = lpr / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (i < pieces && i % lpr == 0) {
    const long long row = i / lpr, bt = row / H;
    const int h = static_cast<int>(row % H);
    delta[(bt / T * H + h) * T + bt % T] = acc;
  }
}

// [b, h, q tile][hd / 4][128][4] fp32 -> bf16 [B, T, H, hd]: a thread gathers 32 columns of its row; the rows leave
// through shared memory so that four lanes write a row's 64 bytes together (16 bytes a row and store took 1.6x as long).
__global__ void __launch_bounds__(kTile) attn_dq_cast_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq,
                                                             int T, int H, int hd) {
  __shared__ uint4 rows[kTile][4];
  const int n_qt = T / kTile, groups = hd / 32;
  const int cg = static_cast<int>(blockIdx.x % groups);
  const long long item = blockIdx.x / groups;  // (b, h, qt)
  const int qt = static_cast<int>(item % n_qt), t = threadIdx.x;
  const long long bh = item / n_qt;
  const float4* src = reinterpret_cast<const float4*>(acc) + (item * (hd / 4) + cg * 8) * kTile + t;
  float4 v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = src[c * kTile];
#pragma unroll
  for (int c = 0; c < 4; ++c)
    rows[t][c ^ ((t >> 1) & 3)] = make_uint4(pack_bf16(v[2 * c].x, v[2 * c].y), pack_bf16(v[2 * c].z, v[2 * c].w),
                                             pack_bf16(v[2 * c + 1].x, v[2 * c + 1].y), pack_bf16(v[2 * c + 1].z, v[2 * c + 1].w));
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = k * 32 + (t >> 2), c = t & 3;
    __nv_bfloat16* dst = dq + ((bh / H * T + qt * kTile + r) * H + bh % H) * hd + cg * 32 + 8 * c;
    *reinterpret_cast<uint4*>(dst) = rows[r][c ^ ((r >> 1) & 3)];
  }
}

constexpr int kBwdEwThreads = 256;                     // two elementwise warps per TMEM lane quarter
constexpr int kBwdDqThreads = 128;                     // four warps that move dQ out
constexpr int kBwdThreads = kBwdEwThreads + kBwdDqThreads + 64;  // then the producer and the MMA issuer

template <int HD>
struct BwdPlan {
  static constexpr int kTileBytes = kTile * HD * 2;  // K, V, Q or dO tile
  static constexpr int kDoStages = HD == 64 ? 2 : 1;
  static constexpr int kPBytes = kTile * kTile * 2;
  static constexpr int kTotal = (2 + 2 /*Q ring*/ + kDoStages) * kTileBytes + 2 * kPBytes + 1024 /*align*/ + 1024 /*barriers, ids*/;
  static constexpr uint32_t kTmemCols = 512;
  // S [0, 128), dP [128, 256), dV, dK, then dQ in columns of its own (hd 64) or over dP (hd 128)
  static constexpr bool kOwnDq = HD == 64;
  static constexpr uint32_t kDv = 256, kDk = 256 + HD, kDq = kOwnDq ? 384 : 128;
};

template <int HD>
__global__ void __launch_bounds__(kBwdThreads, 1) attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                   const __grid_constant__ CUtensorMap tmK,
                                                                   const __grid_constant__ CUtensorMap tmV,
                                                                   const __grid_constant__ CUtensorMap tmdO,
                                                                   const AttnArgs args) {
  using Plan = BwdPlan<HD>;
  constexpr int kDoStages = Plan::kDoStages;
  constexpr int kKB = HD / 64;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sm_k = base;
  const uint32_t sm_v = sm_k + Plan::kTileBytes;
  const uint32_t sm_q = sm_v + Plan::kTileBytes;
  const uint32_t sm_do = sm_q + 2 * Plan::kTileBytes;
  const uint32_t sm_p = sm_do + kDoStages * Plan::kTileBytes;
  const uint32_t sm_ds = sm_p + Plan::kPBytes;
  const uint32_t sm_bar = sm_ds + Plan::kPBytes;
  const uint32_t bar_kv = sm_bar;
  const uint32_t bar_qf = bar_kv + 8, bar_qe = bar_qf + 16;    // Q ring full / empty [2]
  const uint32_t bar_gf = bar_qe + 16, bar_ge = bar_gf + 16;   // dO ring full / empty [2]
  const uint32_t bar_s = bar_ge + 16, bar_dp = bar_s + 8;      // S, dP formed
  const uint32_t bar_pf = bar_dp + 8, bar_pe = bar_pf + 8;     // P stored (S read) / consumed
  const uint32_t bar_df = bar_pe + 8, bar_de = bar_df + 8;     // dS stored (dP read) / consumed
  const uint32_t bar_dqf = bar_de + 8, bar_dqe = bar_dqf + 8;  // dQ formed / read out
  const uint32_t bar_fin = bar_dqe + 8;
  const uint32_t tmem_slot = bar_fin + 8;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gbase + (tmem_slot - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + (tmem_slot + 4 - base));
  int* seg_k = reinterpret_cast<int*>(gbase + (sm_bar + 256 - base));  // [128]

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
      mbar_init(bar_gf + 8 * s, 1);
      mbar_init(bar_ge + 8 * s, 1);
    }
    mbar_init(bar_s, 1);
    mbar_init(bar_dp, 1);
    mbar_init(bar_pf, kBwdEwThreads);
    mbar_init(bar_pe, 1);
    mbar_init(bar_df, kBwdEwThreads);
    mbar_init(bar_de, 1);
    mbar_init(bar_dqf, 1);
    mbar_init(bar_dqe, kBwdDqThreads);
    mbar_init(bar_fin, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (threadIdx.x < kTile && args.segment_ids)
    seg_k[threadIdx.x] = args.segment_ids[static_cast<long long>(b) * args.T + kt * kTile + threadIdx.x];
  if (warp == 13) {
    tmem_alloc(tmem_slot, Plan::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = *tmem_slot_ptr;
  const uint32_t tmem_dp = tmem_s + 128;
  const uint32_t tmem_dv = tmem_s + Plan::kDv, tmem_dk = tmem_s + Plan::kDk, tmem_dq = tmem_s + Plan::kDq;

  if (warp == 12) {
    // ---------------- TMA producer ----------------
    if (elect_one_sync()) {
      mbar_expect_tx(bar_kv, 2 * Plan::kTileBytes);
      for (int c = 0; c < kKB; ++c) {
        tma_load_3d(sm_k + c * (kTile * 128), &tmK, bar_kv, hk * HD + 64 * c, kt * kTile, b);
        tma_load_3d(sm_v + c * (kTile * 128), &tmV, bar_kv, hk * HD + 64 * c, kt * kTile, b);
      }
    }
    for (int it = 0; it < n_it; ++it) {
      const int h = hk * group + it / per_head, qt = qt_lo + it % per_head;
      auto load = [&](uint32_t full, uint32_t empty, uint32_t dst, const CUtensorMap* tm, int stages) {
        const int st = it % stages;
        if (!mbar_wait_warp(empty + 8 * st, static_cast<uint32_t>((it / stages) & 1) ^ 1, abort_flag)) return false;
        if (elect_one_sync()) {
          mbar_expect_tx(full + 8 * st, Plan::kTileBytes);
          for (int c = 0; c < kKB; ++c)
            tma_load_3d(dst + st * Plan::kTileBytes + c * (kTile * 128), tm, full + 8 * st, h * HD + 64 * c, qt * kTile, b);
        }
        return true;
      };
      if (!load(bar_qf, bar_qe, sm_q, &tmQ, 2) || !load(bar_gf, bar_ge, sm_do, &tmdO, kDoStages)) {
        if (lane == 0) atomicCAS(args.status, 0, kTimeoutProducer);
        break;
      }
    }
  } else if (warp == 13) {
    // ---------------- MMA issuer ----------------
    constexpr uint32_t idesc_s = make_idesc_bf16(kTile, kTile, 0, 0);   // Q K^T, dO V^T
    constexpr uint32_t idesc_t = make_idesc_bf16(kTile, HD, 1, 1);      // P^T dO, dS^T Q
    constexpr uint32_t idesc_q = make_idesc_bf16(kTile, HD, 0, 1);      // dS K
    auto wait = [&](uint32_t bar, int count) { return mbar_wait_warp(bar, static_cast<uint32_t>(count & 1), abort_flag); };
    // D = A B^T of two K-major tiles (S and dP)
    auto issue_nt = [&](uint32_t d, uint32_t a_s, uint32_t b_s, uint32_t done) {
      if (elect_one_sync()) {
#pragma unroll
        for (int c = 0; c < kKB; ++c) {
          const uint64_t ad = make_smem_desc(a_s + c * (kTile * 128), 16, 1024);
          const uint64_t bd = make_smem_desc(b_s + c * (kTile * 128), 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(d, ad + k * 2, bd + k * 2, idesc_s, (c > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(done);
      }
    };
    // D (+)= A^T B: A = P or dS read MN-major (K = query rows), B = dO or Q read MN-major
    auto issue_tn = [&](uint32_t d, uint32_t a_s, uint32_t b_s, bool first) {
      const uint64_t ad = make_smem_desc(a_s, kTile * 128, 1024), bd = make_smem_desc(b_s, kTile * 128, 1024);
#pragma unroll
      for (int k = 0; k < kTile / 16; ++k)
        umma_bf16(d, ad + k * (2048 >> 4), bd + k * (2048 >> 4), idesc_t, (!first || k > 0) ? 1u : 0u);
    };
    auto issue_s = [&](int it) {
      if (!mbar_wait_warp(bar_qf + 8 * (it & 1), static_cast<uint32_t>((it >> 1) & 1), abort_flag)) return false;
      tc_fence_after();
      issue_nt(tmem_s, sm_q + (it & 1) * Plan::kTileBytes, sm_k, bar_s);
      return true;
    };
    auto issue_dp = [&](int it) {
      const int st = it % kDoStages;
      if (!mbar_wait_warp(bar_gf + 8 * st, static_cast<uint32_t>((it / kDoStages) & 1), abort_flag)) return false;
      tc_fence_after();
      issue_nt(tmem_dp, sm_do + st * Plan::kTileBytes, sm_v, bar_dp);
      return true;
    };
    bool ok = mbar_wait_warp(bar_kv, 0, abort_flag);
    if (n_it > 0) ok = ok && issue_s(0) && issue_dp(0);
    for (int it = 0; it < n_it && ok; ++it) {
      const uint32_t q_s = sm_q + (it & 1) * Plan::kTileBytes;
      const int g_st = it % kDoStages;
      ok = wait(bar_pf, it);
      if (!ok) break;
      tc_fence_after();
      if (it + 1 < n_it && !issue_s(it + 1)) { ok = false; break; }
      if (elect_one_sync()) {
        issue_tn(tmem_dv, sm_p, sm_do + g_st * Plan::kTileBytes, it == 0);
        umma_commit(bar_pe);
        umma_commit(bar_ge + 8 * g_st);
      }
      ok = wait(bar_df, it);
      if (!ok) break;
      tc_fence_after();
      if (Plan::kOwnDq) {
        if (it + 1 < n_it && !issue_dp(it + 1)) { ok = false; break; }
        if (it > 0 && !wait(bar_dqe, it - 1)) { ok = false; break; }
        tc_fence_after();
      }
      if (elect_one_sync()) {
        // dQ_i = dS K_j: A = dS K-major in the key index, B = K_j read MN-major (K = key rows)
        const uint64_t kb_ = make_smem_desc(sm_k, kTile * 128, 1024);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint64_t dsd = make_smem_desc(sm_ds + c * (kTile * 128), 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16(tmem_dq, dsd + k * 2, kb_ + (c * 4 + k) * (2048 >> 4), idesc_q, (c > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(bar_dqf);
        issue_tn(tmem_dk, sm_ds, q_s, it == 0);
        umma_commit(bar_de);
        umma_commit(bar_qe + 8 * (it & 1));
      }
      if (!Plan::kOwnDq && it + 1 < n_it && (!wait(bar_dqe, it) || !issue_dp(it + 1))) { ok = false; break; }
    }
    if (ok && elect_one_sync()) umma_commit(bar_fin);
    if (!ok && lane == 0) atomicCAS(args.status, 0, kTimeoutMma);
  } else if (warp >= 8) {
    // ---------------- dQ -> fp32 scratch (other key tiles add to the same rows) ----------------
    const int row = threadIdx.x - kBwdEwThreads;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    int item = (b * args.H + hk * group) * n_qt + qt_lo, qi = 0;  // (b, h, q tile), and the tile's count in this head
    for (int it = 0; it < n_it; ++it) {
      float4* dst = reinterpret_cast<float4*>(args.dq_accum) + static_cast<long long>(item) * (HD / 4) * kTile + row;
      if (++qi == per_head) {  // next head of the group
        qi = 0;
        item += qt_lo;
      }
      ++item;
      if (!mbar_wait_warp(bar_dqf, static_cast<uint32_t>(it & 1), abort_flag)) {
        if (lane == 0) atomicCAS(args.status, 0, kTimeoutEpilogue);
        break;
      }
      tc_fence_after();
      uint32_t r[HD / 32][32];
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) tmem_ld_32x32(tmem_dq + lane_base + c * 32, r[c]);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(bar_dqe);
#pragma unroll
      for (int c = 0; c < HD / 32; ++c)
#pragma unroll
        for (int i = 0; i < 8; ++i)
          asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + (c * 8 + i) * kTile),
                       "f"(__uint_as_float(r[c][4 * i])), "f"(__uint_as_float(r[c][4 * i + 1])),
                       "f"(__uint_as_float(r[c][4 * i + 2])), "f"(__uint_as_float(r[c][4 * i + 3]))
                       : "memory");
    }
  } else {
    // ---------------- elementwise: query row = TMEM lane, `half` picks 64 keys of the tile ----------------
    const int row = threadIdx.x & (kTile - 1), half = warp >> 2;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    bool ok = true;
    auto wait = [&](uint32_t bar, int count) {
      ok = mbar_wait_warp(bar, static_cast<uint32_t>(count & 1), abort_flag);
      return ok;
    };
    const f32x2 scale_log2 = pk2(args.scale_log2, args.scale_log2), scale = pk2(args.scale, args.scale);
    const uint32_t blk_p = sm_p + half * (kTile * 128), blk_ds = sm_ds + half * (kTile * 128);
    float next_L = 0.0f, next_D = 0.0f;
    int next_seg = 0;
    const long long stat_h = (static_cast<long long>(b) * args.H + hk * group) * args.T + row;
    const int* seg_q_row = args.segment_ids ? args.segment_ids + static_cast<long long>(b) * args.T + row : nullptr;
    auto load_stats = [&](int head, int tile) {  // an iteration ahead: their latency stays off the chain
      const long long stat = stat_h + static_cast<long long>(head) * args.T + tile * kTile;
      next_L = args.lse[stat];
      next_D = args.delta[stat];
      if (seg_q_row) next_seg = seg_q_row[tile * kTile];
    };
    int head_n = 0, qt_n = qt_lo;  // of the next iteration
    load_stats(0, qt_n);
    for (int it = 0; it < n_it; ++it) {
      const int qt = qt_n, seg_q = next_seg;
      const f32x2 negL = pk2(-next_L, -next_L), negD = pk2(-next_D, -next_D);
      if (++qt_n == n_qt) {
        qt_n = qt_lo;
        ++head_n;
      }
      if (it + 1 < n_it) load_stats(head_n, qt_n);
      if (!wait(bar_s, it)) break;
      tc_fence_after();
      uint32_t r[2][32];  // scores, then probabilities
#pragma unroll
      for (int c = 0; c < 2; ++c) tmem_ld_32x32(tmem_s + lane_base + half * 64 + c * 32, r[c]);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 x = unpack2(fma2(pk2u(r[c][i], r[c][i + 1]), scale_log2, negL));
          r[c][i] = __float_as_uint(fast_exp2(x.x));
          r[c][i + 1] = __float_as_uint(fast_exp2(x.y));
        }
      if (args.causal && qt == kt) {
        const int lim = row - half * 64;  // last key column of this half that the row sees
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > lim) r[c][i] = 0u;
      }
      if (args.segment_ids) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const int4 id = *reinterpret_cast<const int4*>(seg_k + half * 64 + c * 32 + i);
            if (id.x != seg_q) r[c][i] = 0u;
            if (id.y != seg_q) r[c][i + 1] = 0u;
            if (id.z != seg_q) r[c][i + 2] = 0u;
            if (id.w != seg_q) r[c][i + 3] = 0u;
          }
      }
      if (it > 0 && !wait(bar_pe, it - 1)) break;
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        const uint32_t* v = &r[g >> 2][(g & 3) * 8];
        st_shared_v4(blk_p + swz(row, g), make_uint4(pack_bf16_2(pk2u(v[0], v[1])), pack_bf16_2(pk2u(v[2], v[3])),
                                                     pack_bf16_2(pk2u(v[4], v[5])), pack_bf16_2(pk2u(v[6], v[7]))));
      }
      tc_fence_before();
      fence_proxy_async_smem();
      mbar_arrive(bar_pf);
      if (!wait(bar_dp, it)) break;
      tc_fence_after();
      if (it > 0 && !wait(bar_de, it - 1)) break;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t g[32];
        tmem_ld_32x32(tmem_dp + lane_base + half * 64 + c * 32, g);
        tmem_ld_wait();
        uint32_t d[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          d[i] = pack_bf16_2(mul2(mul2(pk2u(r[c][2 * i], r[c][2 * i + 1]), add2(pk2u(g[2 * i], g[2 * i + 1]), negD)), scale));
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4)
          st_shared_v4(blk_ds + swz(row, c * 4 + q4), make_uint4(d[4 * q4], d[4 * q4 + 1], d[4 * q4 + 2], d[4 * q4 + 3]));
      }
      tc_fence_before();
      fence_proxy_async_smem();
      mbar_arrive(bar_df);
    }
    if (ok && n_it > 0) wait(bar_fin, 0);
    if (ok) {  // dV by the first four warps, dK by the others
      tc_fence_after();
      const long long krow = ((static_cast<long long>(b) * args.T + kt * kTile + row) * args.Hkv + hk) * HD;
      __nv_bfloat16* dst = (half == 0 ? args.dv : args.dk) + krow;
      const uint32_t src = (half == 0 ? tmem_dv : tmem_dk) + lane_base;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(src + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g)
          *reinterpret_cast<uint4*>(dst + c * 32 + 8 * g) =
              make_uint4(pack_bf16_2(pk2u(r[8 * g], r[8 * g + 1])), pack_bf16_2(pk2u(r[8 * g + 2], r[8 * g + 3])),
                         pack_bf16_2(pk2u(r[8 * g + 4], r[8 * g + 5])), pack_bf16_2(pk2u(r[8 * g + 6], r[8 * g + 7])));
      }
    }
    if (!ok) atomicCAS(args.status, 0, kTimeoutEpilogue);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) tmem_dealloc(tmem_s, Plan::kTmemCols);
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
  kern<<<grid, kBwdThreads, BwdPlan<HD>::kTotal, st>>>(q, k, v, d_o, a);
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

// `delta` [B, H, T] fp32 and `dq_accum` (B T H hd floats) are scratch supplied by the caller, contents irrelevant;
// out, d_out and dq_accum on 16-byte boundaries.
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
  const long long rows = static_cast<long long>(B) * T * H, pieces = rows * (hd / 8);
  if ((pieces + 255) / 256 > 0x7FFFFFFF || rows / kTile > 0x3FFFFFFF) return kBadArgument;
  attn_delta_kernel<<<static_cast<unsigned>((pieces + 255) / 256), 256, 0, st>>>(
      static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out), delta, dq_accum, B, T, H, hd);
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
  attn_dq_cast_kernel<<<static_cast<unsigned>(rows / kTile * (hd / 32)), kTile, 0, st>>>(
      dq_accum, static_cast<__nv_bfloat16*>(dq), T, H, hd);
  return cudaGetLastError() == cudaSuccess ? 0 : 400;
}
