// Vocabulary KL and its gradient, one row of logits pair per position:
//   kl[row] = KL(softmax(lc[row]) || softmax(lm[row]));  dlm[row] = softmax(lm) - softmax(lc)
// (the caller scales by the upstream gradient / number of positions inside the next GEMM).
// Rows are `ld` elements apart (padded to a multiple of 8); V valid columns.
#include <algorithm>

#include "common.cuh"

namespace {

using namespace pd;

__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Rows too long for the shared memory of a cluster: one block per row, three passes over global memory.
__global__ void vocab_kl_streamed_kernel(const __nv_bfloat16* __restrict__ lc, const __nv_bfloat16* __restrict__ lm,
                                __nv_bfloat16* __restrict__ dlm, float* __restrict__ kl, int V, long long ld) {
  const long long row = blockIdx.x;
  const __nv_bfloat16* a = lc + row * ld;
  const __nv_bfloat16* b = lm + row * ld;
  __shared__ float red[4][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // pass 1: row maxima
  float ma = -INFINITY, mb = -INFINITY;
  for (int i = threadIdx.x * 8; i < V; i += blockDim.x * 8) {
    const uint4 qa = *reinterpret_cast<const uint4*>(a + i), qb = *reinterpret_cast<const uint4*>(b + i);
    const __nv_bfloat16* ha = reinterpret_cast<const __nv_bfloat16*>(&qa);
    const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&qb);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (i + k < V) { ma = fmaxf(ma, __bfloat162float(ha[k])); mb = fmaxf(mb, __bfloat162float(hb[k])); }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ma = fmaxf(ma, __shfl_xor_sync(0xffffffffu, ma, o));
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, o));
  }
  if (lane == 0) { red[0][warp] = ma; red[1][warp] = mb; }
  __syncthreads();
  ma = red[0][0]; mb = red[1][0];
  for (int w = 1; w < nw; ++w) { ma = fmaxf(ma, red[0][w]); mb = fmaxf(mb, red[1][w]); }
  __syncthreads();
  // pass 2: partition functions and the cross term sum exp(a - ma) * (a - b)
  float sa = 0.f, sb = 0.f, cross = 0.f;
  for (int i = threadIdx.x * 8; i < V; i += blockDim.x * 8) {
    const uint4 qa = *reinterpret_cast<const uint4*>(a + i), qb = *reinterpret_cast<const uint4*>(b + i);
    const __nv_bfloat16* ha = reinterpret_cast<const __nv_bfloat16*>(&qa);
    const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&qb);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (i + k < V) {
        const float x = __bfloat162float(ha[k]), y = __bfloat162float(hb[k]);
        const float ea = __expf(x - ma);
        sa += ea; sb += __expf(y - mb); cross += ea * (x - y);
      }
    }
  }
  sa = warp_total(sa); sb = warp_total(sb); cross = warp_total(cross);
  if (lane == 0) { red[0][warp] = sa; red[1][warp] = sb; red[2][warp] = cross; }
  __syncthreads();
  sa = 0.f; sb = 0.f; cross = 0.f;
  for (int w = 0; w < nw; ++w) { sa += red[0][w]; sb += red[1][w]; cross += red[2][w]; }
  const float lsa = ma + __logf(sa), lsb = mb + __logf(sb);
  // KL = sum p_a (a - lsa - b + lsb) = cross / sa - lsa + lsb
  if (threadIdx.x == 0) kl[row] = cross / sa - lsa + lsb;
  // pass 3: gradient wrt the masked logits
  if (dlm != nullptr) {
    __nv_bfloat16* d = dlm + row * ld;
    const float ia = 1.f / sa, ib = 1.f / sb;
    for (int i = threadIdx.x * 8; i < V; i += blockDim.x * 8) {
      const uint4 qa = *reinterpret_cast<const uint4*>(a + i), qb = *reinterpret_cast<const uint4*>(b + i);
      const __nv_bfloat16* ha = reinterpret_cast<const __nv_bfloat16*>(&qa);
      const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&qb);
      __nv_bfloat16 o[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float x = __bfloat162float(ha[k]), y = __bfloat162float(hb[k]);
        o[k] = __float2bfloat16(i + k < V ? __expf(y - mb) * ib - __expf(x - ma) * ia : 0.f);
      }
      *reinterpret_cast<uint4*>(d + i) = *reinterpret_cast<uint4*>(o);
    }
  }
}

// ---- rows held in shared memory ----------------------------------------------------------------------------------
// A cluster of 1, 2, 4 or 8 CTAs owns a row pair: each CTA brings its slice of both rows into shared memory with bulk
// copies (one 16-byte group per thread and piece), reads it there for the sums and again for the gradient, so every
// logit crosses HBM once. A thread keeps its own running maximum and sums relative to it; partial results are combined
// over the warp, the block and (through distributed shared memory, one cluster barrier per row) the cluster. Clusters
// walk the rows; a piece of the next row is requested as soon as the gradient pass has read the current one out of it.
// Slices are kept below half an SM's shared memory where 8 CTAs allow it, so that one CTA's copies run beside
// another's arithmetic. 6 bytes of HBM traffic and four exponentials (16 lanes a clock) per logit pair take about the
// same time and overlap in part: DRAM 40%, exponential unit 62% busy. 8192 rows of 50,277: 900 us in three passes over
// global memory, 652 us so.
struct RowSums {
  float ma, mb, sa, sb, cross;  // maxima; sums of exp(a - ma), exp(b - mb), exp(a - ma) (a - b)
};
// Floor of a thread's maximum: a thread that holds only masked logits (-inf or the type's lowest) adds nothing, instead of
// sums of differences near the end of the range that its zero weight would turn into NaN.
constexpr float kMinMax = -1.0e30f;
constexpr float kLowest = -3.3895313892515355e38f;  // lowest finite bf16
constexpr float kLog2E = 1.4426950408889634f;

__device__ __forceinline__ RowSums merge(const RowSums& x, const RowSums& y) {
  RowSums r;
  r.ma = fmaxf(x.ma, y.ma);
  r.mb = fmaxf(x.mb, y.mb);
  const float xa = ex2((x.ma - r.ma) * kLog2E), ya = ex2((y.ma - r.ma) * kLog2E);
  r.sa = x.sa * xa + y.sa * ya;
  r.cross = x.cross * xa + y.cross * ya;
  r.sb = x.sb * ex2((x.mb - r.mb) * kLog2E) + y.sb * ex2((y.mb - r.mb) * kLog2E);
  return r;
}
__device__ __forceinline__ RowSums shuffle_xor(const RowSums& x, int o) {
  return RowSums{__shfl_xor_sync(0xffffffffu, x.ma, o), __shfl_xor_sync(0xffffffffu, x.mb, o),
                 __shfl_xor_sync(0xffffffffu, x.sa, o), __shfl_xor_sync(0xffffffffu, x.sb, o),
                 __shfl_xor_sync(0xffffffffu, x.cross, o)};
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void store_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r =
      __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}

constexpr int kMaxPieces = 32;

__global__ void __launch_bounds__(512) vocab_kl_rows_kernel(const __nv_bfloat16* __restrict__ lc,
                                                            const __nv_bfloat16* __restrict__ lm,
                                                            __nv_bfloat16* __restrict__ dlm, float* __restrict__ kl,
                                                            long long rows, int V, long long ld, int slice_groups,
                                                            int cs, int* __restrict__ status) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) unsigned long long bars[kMaxPieces];
  __shared__ RowSums red[16], xch[2][8];
  __shared__ int abort_flag;
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int rank = cs > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int g_first = rank * slice_groups;                                       // in groups of 8 logits
  const int n_groups = max(0, min(slice_groups, (V + 7) / 8 - g_first));
  const int pieces = (n_groups + nt - 1) / nt;
  uint8_t* buf_a = smem;
  uint8_t* buf_b = smem + static_cast<long long>(slice_groups) * 16;
  const uint32_t bar0 = smem_u32(bars);
  // columns past V in this thread's last group (0 for every thread but the one that holds the row's last group)
  const int my_over = n_groups > 0 && tid == (n_groups - 1) % nt ? max(0, 8 * (g_first + n_groups) - V) : 0;
  if (tid == 0) {
    for (int i = 0; i < pieces; ++i) mbar_init(bar0 + 8 * i, 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  const long long first = blockIdx.x / cs, step = gridDim.x / cs;
  auto request = [&](long long row, int piece) {  // one thread; nothing new once a wait has run out
    if (*static_cast<volatile int*>(&abort_flag)) return;
    const int g0 = piece * nt, n = min(nt, n_groups - g0);
    const long long at = row * ld + 8ll * (g_first + g0);
    mbar_expect_tx(bar0 + 8 * piece, 32u * n);
    bulk_load(smem_u32(buf_a + 16 * g0), lc + at, 16u * n, bar0 + 8 * piece);
    bulk_load(smem_u32(buf_b + 16 * g0), lm + at, 16u * n, bar0 + 8 * piece);
  };
  if (tid == 0 && first < rows)
    for (int i = 0; i < pieces; ++i) request(first, i);
  if (cs > 1) cluster_sync_all();  // every CTA of the cluster runs before another one stores to its shared memory
  const f32x2 l2e = pk2(kLog2E, kLog2E), neg1 = pk2(-1.0f, -1.0f);
  int turn = 0, exchange = 0;
  for (long long row = first; row < rows; row += step, ++turn) {
    // this thread's maxima
    uint32_t wa = 0xFF80FF80u, wb = 0xFF80FF80u;  // -inf pairs
    for (int i = 0; i < pieces; ++i) {
      if (!mbar_wait(bar0 + 8 * i, turn & 1, &abort_flag) && status != nullptr) atomicCAS(status, 0, kTimeoutProducer);
      const int g = i * nt + tid;
      if (g >= n_groups) break;
      uint4 a = *reinterpret_cast<const uint4*>(buf_a + 16 * g), b = *reinterpret_cast<const uint4*>(buf_b + 16 * g);
      const int over = 8 * (g_first + g + 1) - V;  // columns past V in the row's last group: equal and as low as can be
      if (over > 0) {
        __nv_bfloat16* ta = reinterpret_cast<__nv_bfloat16*>(buf_a + 16 * g);
        __nv_bfloat16* tb = reinterpret_cast<__nv_bfloat16*>(buf_b + 16 * g);
        for (int k = 8 - over; k < 8; ++k) ta[k] = tb[k] = __ushort_as_bfloat16(0xFF7Fu);
        fence_proxy_async_smem();  // before the next row's bulk copy writes here
        a = *reinterpret_cast<const uint4*>(buf_a + 16 * g);
        b = *reinterpret_cast<const uint4*>(buf_b + 16 * g);
      }
      wa = max_bf16x2(wa, max_bf16x2(max_bf16x2(a.x, a.y), max_bf16x2(a.z, a.w)));
      wb = max_bf16x2(wb, max_bf16x2(max_bf16x2(b.x, b.y), max_bf16x2(b.z, b.w)));
    }
    const float max_a = fmaxf(__uint_as_float(wa << 16), __uint_as_float(wa & 0xFFFF0000u));
    const float max_b = fmaxf(__uint_as_float(wb << 16), __uint_as_float(wb & 0xFFFF0000u));
    // One pass, sums relative to the thread's own maxima. A row whose logits all lie below the floor comes out with a
    // sum of zero: two more passes, one for the row's true maxima and one for sums relative to them.
    RowSums t;
    float ref_a = fmaxf(kMinMax, max_a), ref_b = fmaxf(kMinMax, max_b);
    for (int pass = 0;; ++pass) {
      t = RowSums{ref_a, ref_b, 0.0f, 0.0f, 0.0f};
      if (pass != 1) {
        const f32x2 na = pk2(-ref_a, -ref_a), nb = pk2(-ref_b, -ref_b);
        f32x2 sa = 0ull, sb = 0ull, cr = 0ull;
        for (int g = tid; g < n_groups; g += nt) {
          const uint4 a = *reinterpret_cast<const uint4*>(buf_a + 16 * g), b = *reinterpret_cast<const uint4*>(buf_b + 16 * g);
          const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const f32x2 x = unpack_bf16_2(aw[k]), y = unpack_bf16_2(bw[k]);
            const float2 dx = unpack2(mul2(add2(x, na), l2e)), dy = unpack2(mul2(add2(y, nb), l2e));
            const f32x2 ea = pk2(ex2(dx.x), ex2(dx.y));
            sa = add2(sa, ea);
            sb = add2(sb, pk2(ex2(dy.x), ex2(dy.y)));
            cr = fma2(ea, fma2(y, neg1, x), cr);
          }
        }
        const float2 s0 = unpack2(sa), s1 = unpack2(sb), s2 = unpack2(cr);
        t.sa = s0.x + s0.y;
        t.sb = s1.x + s1.y;
        t.cross = s2.x + s2.y;
        if (pass == 2 && my_over > 0) {  // the columns past V hold the lowest value, which counts here
          t.sa -= my_over * ex2((kLowest - ref_a) * kLog2E);
          t.sb -= my_over * ex2((kLowest - ref_b) * kLog2E);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t = merge(t, shuffle_xor(t, o));
      if (lane == 0) red[warp] = t;
      __syncthreads();
      if (warp == 0) {
        t = red[lane < nt / 32 ? lane : 0];
        if (lane >= nt / 32) t.sa = t.sb = t.cross = 0.0f;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) t = merge(t, shuffle_xor(t, o));
        if (lane < cs) {  // to every CTA of the cluster
          const uint32_t local = smem_u32(&xch[exchange & 1][rank]);
          const uint32_t at = cs > 1 ? mapa_shared(local, lane) : local;
          store_cluster_f32(at, t.ma);
          store_cluster_f32(at + 4, t.mb);
          store_cluster_f32(at + 8, t.sa);
          store_cluster_f32(at + 12, t.sb);
          store_cluster_f32(at + 16, t.cross);
        }
      }
      if (cs > 1)
        cluster_sync_all();
      else
        __syncthreads();
      t = xch[exchange & 1][0];
      for (int r = 1; r < cs; ++r) t = merge(t, xch[exchange & 1][r]);
      ++exchange;
      if (pass == 0 && (t.sa == 0.0f || t.sb == 0.0f)) {  // the same verdict in every thread of the cluster
        ref_a = fmaxf(kLowest, max_a);
        ref_b = fmaxf(kLowest, max_b);
      } else if (pass == 1) {
        ref_a = t.ma;
        ref_b = t.mb;
      } else {
        if (pass == 2 && my_over > 0) {  // and take no part in the gradient
          const int g = n_groups - 1;
          __nv_bfloat16* ta = reinterpret_cast<__nv_bfloat16*>(buf_a + 16 * g);
          __nv_bfloat16* tb = reinterpret_cast<__nv_bfloat16*>(buf_b + 16 * g);
          for (int k = 8 - my_over; k < 8; ++k) ta[k] = tb[k] = __ushort_as_bfloat16(0xFF80u);
          fence_proxy_async_smem();
        }
        break;
      }
    }
    // KL = sum p_a (a - lsa - b + lsb) = cross / sa - lsa + lsb
    if (rank == 0 && tid == 0) kl[row] = t.cross / t.sa - (t.ma + __logf(t.sa)) + (t.mb + __logf(t.sb));
    const bool more = row + step < rows;
    if (dlm != nullptr) {
      const f32x2 na = pk2(-t.ma, -t.ma), nb = pk2(-t.mb, -t.mb);
      const float ia = -1.0f / t.sa, ib = 1.0f / t.sb;
      const f32x2 ia2 = pk2(ia, ia), ib2 = pk2(ib, ib);
      __nv_bfloat16* d = dlm + row * ld + 8ll * g_first;
      for (int i = 0; i < pieces; ++i) {
        const int g = i * nt + tid;
        if (g < n_groups) {
          const uint4 a = *reinterpret_cast<const uint4*>(buf_a + 16 * g), b = *reinterpret_cast<const uint4*>(buf_b + 16 * g);
          const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
          uint32_t o[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 dx = unpack2(mul2(add2(unpack_bf16_2(aw[k]), na), l2e));
            const float2 dy = unpack2(mul2(add2(unpack_bf16_2(bw[k]), nb), l2e));
            o[k] = pack_bf16_2(fma2(pk2(ex2(dx.x), ex2(dx.y)), ia2, mul2(pk2(ex2(dy.x), ex2(dy.y)), ib2)));
          }
          *reinterpret_cast<uint4*>(d + 8ll * g) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        if (more) {
          __syncthreads();  // the piece has been read
          if (tid == 0) request(row + step, i);
        }
      }
    } else if (more) {
      __syncthreads();
      if (tid == 0)
        for (int i = 0; i < pieces; ++i) request(row + step, i);
    }
  }
}

}  // namespace

extern "C" int pd_vocab_kl(const void* lc, const void* lm, void* dlm, float* kl, long long rows, int V,
                           long long ld, int* status, void* stream) {
  if (ld % 8 != 0 || rows <= 0) return 5;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const auto* a = static_cast<const __nv_bfloat16*>(lc);
  const auto* b = static_cast<const __nv_bfloat16*>(lm);
  auto* d = static_cast<__nv_bfloat16*>(dlm);
  // Smallest cluster whose slices (32 bytes per group of 8 columns) leave room for two CTAs on an SM; past that, up to
  // one CTA per SM; longer rows stream through global memory.
  constexpr int kHalfSm = 108 * 1024, kWholeSm = 220 * 1024;
  const long long groups = (static_cast<long long>(V) + 7) / 8;
  int cs = 1;
  while (cs < 8 && (groups + cs - 1) / cs * 32 > kHalfSm) cs *= 2;
  const long long slice = (groups + cs - 1) / cs;
  if (slice * 32 > kWholeSm) {
    vocab_kl_streamed_kernel<<<static_cast<unsigned>(rows), 512, 0, st>>>(a, b, d, kl, V, ld);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
  }
  const int smem = static_cast<int>(slice * 32);
  // short rows: fewer threads, so that every thread has a group and more rows share an SM
  const int nt = slice >= 1024 ? 512 : slice >= 256 ? 256 : 128;
  auto kern = vocab_kl_rows_kernel;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm) != cudaSuccess) return 2;
  const int per_sm = std::max(1, std::min(2048 / nt / 2, 227 * 1024 / (smem + 3 * 1024)));
  const long long clusters = std::min<long long>(rows, 148ll * per_sm / cs);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(clusters * cs));
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a, b, d, kl, rows, V, ld, static_cast<int>(slice), cs, status);
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : 1;
}
