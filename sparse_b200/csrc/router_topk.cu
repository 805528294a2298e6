// Router: logits (fixed fp32 summation order) -> softmax (fp32) -> top-k.
//
// Replaces `_routing_router` of the reference (utils/eval_core.py:9519-9520,
// 9591-9595) plus the scalar gate of the shared expert
// (utils/eval_core.py:9461-9462).
//
// Summation order of one logit (bit-exact contract with the CPU oracle): the H
// inputs are cut into groups of 8; lane l of a warp takes groups l, l+32, l+64,
// ... in increasing order and keeps two partial sums, one over the even and one
// over the odd elements of its groups, elements in increasing order, each step
// p = fl(p + fl(x*w)) (for bf16 inputs the product is exact, so a fused
// multiply-add gives the same bits); the lane sum is fl(p_even + p_odd); the 32
// lane sums are combined by an xor-butterfly with offsets 16, 8, 4, 2, 1; the
// bias is added in fp32 and the result is rounded once to the model dtype.
//
// Work split: one CTA owns TB tokens whose activations sit in shared memory; each
// of its 8 warps streams groups of RW router rows from L2 and dots them with all
// TB tokens, so a weight row is fetched once per CTA.  HBM traffic is one read of
// x plus the outputs; above a thousand tokens the kernel is bound by the fp32 FMA
// pipe and the L2 reads of the router rows (2*T*E*H flops on CUDA cores), below by
// latency: there a cluster of CS CTAs shares a token tile, each takes 1/CS of the
// router rows and hands every token's logits to the CTA that finishes the token.
#include "sb_common.cuh"

namespace sb {
namespace {

constexpr int kRouterThreads = 256;
constexpr int kRouterWarps = kRouterThreads / 32;
constexpr int kMaxExperts = 256;
constexpr int kMaxK = 8;

template <typename IN> struct Load8;

template <> struct Load8<__nv_bfloat16> {
  static constexpr bool kExactProduct = true;
  __device__ static void from(const uint4 *p, float (&v)[8]) {
    uint4 r = *p;
    v[0] = bf16_lo(r.x); v[1] = bf16_hi(r.x); v[2] = bf16_lo(r.y); v[3] = bf16_hi(r.y);
    v[4] = bf16_lo(r.z); v[5] = bf16_hi(r.z); v[6] = bf16_lo(r.w); v[7] = bf16_hi(r.w);
  }
  __device__ static void from_global(const __nv_bfloat16 *base, size_t elem, float (&v)[8]) {
    uint4 r = __ldg(reinterpret_cast<const uint4 *>(base + elem));
    v[0] = bf16_lo(r.x); v[1] = bf16_hi(r.x); v[2] = bf16_lo(r.y); v[3] = bf16_hi(r.y);
    v[4] = bf16_lo(r.z); v[5] = bf16_hi(r.z); v[6] = bf16_lo(r.w); v[7] = bf16_hi(r.w);
  }
  __device__ static float round_model(float f) { return round_bf16(f); }
  __device__ static void store(__nv_bfloat16 *p, float f) { *p = __float2bfloat16_rn(f); }
  __device__ static float load(const __nv_bfloat16 *p) { return __bfloat162float(*p); }
};

template <> struct Load8<float> {
  static constexpr bool kExactProduct = false;
  __device__ static void from(const uint4 *p, float (&v)[8]) {
    uint4 a = p[0], b = p[1];
    v[0] = __uint_as_float(a.x); v[1] = __uint_as_float(a.y);
    v[2] = __uint_as_float(a.z); v[3] = __uint_as_float(a.w);
    v[4] = __uint_as_float(b.x); v[5] = __uint_as_float(b.y);
    v[6] = __uint_as_float(b.z); v[7] = __uint_as_float(b.w);
  }
  __device__ static void from_global(const float *base, size_t elem, float (&v)[8]) {
    const uint4 *p = reinterpret_cast<const uint4 *>(base + elem);
    uint4 a = __ldg(p), b = __ldg(p + 1);
    v[0] = __uint_as_float(a.x); v[1] = __uint_as_float(a.y);
    v[2] = __uint_as_float(a.z); v[3] = __uint_as_float(a.w);
    v[4] = __uint_as_float(b.x); v[5] = __uint_as_float(b.y);
    v[6] = __uint_as_float(b.z); v[7] = __uint_as_float(b.w);
  }
  __device__ static float round_model(float f) { return f; }
  __device__ static void store(float *p, float f) { *p = f; }
  __device__ static float load(const float *p) { return *p; }
};

__device__ __forceinline__ float butterfly_sum(float v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ float butterfly_max(float v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// Sums of 32 values over the 32 lanes at once: lane i returns the warp-wide sum of
// v[i].  Each step halves the values a lane still carries (it keeps the half that
// its lane-id bit selects and hands the other half to its partner), so this takes
// 31 shuffles instead of 32 x 5.  The additions pair the same lanes at the same
// offsets (16, 8, 4, 2, 1) as butterfly_sum, and fp32 addition is commutative:
// the result has the bits butterfly_sum gives for that value on every lane.
__device__ __forceinline__ float warp_sum_each(float (&v)[32], int lane) {
#pragma unroll
  for (int half = 16; half >= 1; half >>= 1) {
    const bool upper = (lane & half) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = upper ? v[i + half] : v[i];
      const float send = upper ? v[i] : v[i + half];
      v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, half));
    }
  }
  return v[0];
}

// One warp: softmax over E model-dtype logits (given as fp32 values) and top-k.
// `lg` points at this token's E logits in shared memory.
template <typename IN>
__device__ void warp_softmax_topk(const float *lg, int E, int K, int renorm, int lane,
                                  int32_t *out_idx, IN *out_w) {
  constexpr int kPerLane = kMaxExperts / 32;
  float p[kPerLane];
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < kPerLane; ++i) {
    int e = lane + 32 * i;
    p[i] = (e < E) ? lg[e] : -INFINITY;
    m = fmaxf(m, p[i]);
  }
  m = butterfly_max(m);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < kPerLane; ++i) {
    int e = lane + 32 * i;
    if (e < E) { p[i] = expf(p[i] - m); s = __fadd_rn(s, p[i]); } else { p[i] = -1.f; }
  }
  s = butterfly_sum(s);
#pragma unroll
  for (int i = 0; i < kPerLane; ++i)
    if (p[i] >= 0.f) p[i] = __fdiv_rn(p[i], s);
  // A row with a NaN or an infinite logit has NaN probabilities.  torch.topk ranks
  // NaN above every number (utils/eval_core.py:9591-9595 calls it); here NaN gets
  // the key 3 for the selection, so that the indices written are always expert
  // ids, and the weight written for it is NaN again.
#pragma unroll
  for (int i = 0; i < kPerLane; ++i)
    if (p[i] != p[i]) p[i] = 3.f;

  float sel_v[kMaxK];
  int sel_i[kMaxK];
#pragma unroll
  for (int k = 0; k < kMaxK; ++k) {
    if (k >= K) break;
    // lane-local best: larger probability, then smaller expert id
    float bv = -2.f; int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
      int e = lane + 32 * i;
      if (p[i] > bv) { bv = p[i]; bi = e; }   // ascending e: first max wins
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, bv, off);
      int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    sel_v[k] = bv > 2.f ? __int_as_float(0x7fc00000) : bv; sel_i[k] = bi;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i)
      if (lane + 32 * i == bi) p[i] = -1.f;
  }
  if (lane == 0) {
    float denom = 1.f;
    if (renorm) {
      float t = 0.f;
      for (int k = 0; k < K; ++k) t = __fadd_rn(t, sel_v[k]);
      denom = fmaxf(t, 1e-12f);
    }
#pragma unroll
    for (int k = 0; k < kMaxK; ++k) {
      if (k >= K) break;
      float v = renorm ? __fdiv_rn(sel_v[k], denom) : sel_v[k];
      out_idx[k] = sel_i[k];
      Load8<IN>::store(out_w + k, v);
    }
  }
}

// Two running partial sums (even / odd elements) packed for the two-wide FMA.
struct Acc2 {
  unsigned long long v;
  __device__ static Acc2 zero() { Acc2 a; a.v = 0ull; return a; }
  __device__ float lane_sum() const {
    return __fadd_rn(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
  }
  template <typename P> __device__ void fma(const P &x, const P &w, int i) { x.fma_into(v, w, i); }
};

// Eight consecutive elements as four (even, odd) pairs.
template <typename IN> struct Pair4;

template <> struct Pair4<__nv_bfloat16> {
  unsigned long long p[4];
  __device__ static unsigned long long widen(uint32_t word) {      // bf16x2 -> {f32 lo, f32 hi}
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(word << 16), "r"(word & 0xffff0000u));
    return r;
  }
  __device__ void load(const uint4 *src) {
    const uint4 q = *src;
    p[0] = widen(q.x); p[1] = widen(q.y); p[2] = widen(q.z); p[3] = widen(q.w);
  }
  // products of bf16 values are exact in fp32, so the fused form equals mul-then-add
  __device__ void fma_into(unsigned long long &acc, const Pair4 &w, int i) const {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(p[i]), "l"(w.p[i]));
  }
};

template <> struct Pair4<float> {
  float e[8];
  __device__ void load(const uint4 *src) {
    const uint4 a = src[0], b = src[1];
    e[0] = __uint_as_float(a.x); e[1] = __uint_as_float(a.y); e[2] = __uint_as_float(a.z);
    e[3] = __uint_as_float(a.w); e[4] = __uint_as_float(b.x); e[5] = __uint_as_float(b.y);
    e[6] = __uint_as_float(b.z); e[7] = __uint_as_float(b.w);
  }
  // fp32 inputs: multiply and add round separately (the order the CPU check emulates)
  __device__ void fma_into(unsigned long long &acc, const Pair4 &w, int i) const {
    float lo = __uint_as_float((uint32_t)acc), hi = __uint_as_float((uint32_t)(acc >> 32));
    lo = __fadd_rn(lo, __fmul_rn(e[2 * i], w.e[2 * i]));
    hi = __fadd_rn(hi, __fmul_rn(e[2 * i + 1], w.e[2 * i + 1]));
    acc = ((unsigned long long)__float_as_uint(hi) << 32) | (unsigned long long)__float_as_uint(lo);
  }
};

__device__ __forceinline__ uint32_t router_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// a float into the same shared-memory place of CTA `rank` of this cluster
__device__ __forceinline__ void store_to_cta(float *place, uint32_t rank, float v) {
  uint32_t addr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(addr) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(place))), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// all CTAs that share a token tile
template <int CS>
__device__ __forceinline__ void sync_tile() {
  if constexpr (CS == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

template <typename IN, int TB, int RW, int CS, int REGS>
__global__ void __launch_bounds__(kRouterThreads) __maxnreg__(REGS)
router_kernel(const IN *__restrict__ x, const IN *__restrict__ wg, const float *__restrict__ bias,
              const IN *__restrict__ wsg, int T, int H, int E, int K, int renorm, int fp32_logits,
              int32_t *__restrict__ out_idx, IN *__restrict__ out_w,
              void *__restrict__ out_logits, IN *__restrict__ out_shared) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kVecPerGroup = sizeof(IN) == 2 ? 1 : 2;      // uint4 per 8 elements
  const int G = H / 8;
  uint4 *sx = reinterpret_cast<uint4 *>(smem_raw);            // [TB][G*kVecPerGroup]
  float *slog = reinterpret_cast<float *>(sx + (size_t)TB * G * kVecPerGroup);  // [TB][E+1]
  const int NR = E + (wsg != nullptr ? 1 : 0);
  const int ldl = E + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CS == 1 ? 0 : (int)router_cluster_rank();
  const int t0 = blockIdx.x / CS * TB;     // this tile's tokens: t0 .. t0 + TB - 1, zeros past the last

  // stage the activation tile
  const int vec_per_tok = G * kVecPerGroup;
  for (int i = threadIdx.x; i < TB * vec_per_tok; i += kRouterThreads) {
    int t = i / vec_per_tok, v = i - t * vec_per_tok;
    uint4 val = make_uint4(0, 0, 0, 0);
    if (t0 + t < T)
      val = __ldg(reinterpret_cast<const uint4 *>(x + (size_t)(t0 + t) * H) + v);
    sx[i] = val;
  }
  sync_tile<CS>();

  // RW router rows per warp pass: one shared-memory read of a token's 8 activations
  // feeds 8 * RW multiply-adds, issued as two-wide fp32 FMAs (`fma.rn.f32x2`: two
  // independent IEEE FMAs per instruction, so the bits are those of scalar FMAs).
  // Each lane therefore keeps TWO partial sums per logit, one over the even and one
  // over the odd elements of its groups.  AHEAD steps of weight vectors are fetched
  // before their math: one step beside the current one where the math covers a
  // fetch, several steps at once where it does not.
  constexpr int AHEAD = TB >= 4 ? 1 : sizeof(IN) == 2 ? 4 : 2;
  const int steps = (G + 31) / 32;
  const int groups = (NR + RW - 1) / RW;
  const bool whole = (G & 31) == 0;        // a hidden size of whole 256-element steps needs no lane guards
  for (int grp = rank * kRouterWarps + warp; grp < groups; grp += CS * kRouterWarps) {
    const IN *wp[RW];                      // rows past the last read row 0's weights; their sums are never stored
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      const int row = grp * RW + r;
      wp[r] = (row < E || row >= NR) ? wg + (size_t)(row < E ? row : 0) * H : wsg;
    }
    Acc2 acc[TB][RW];
#pragma unroll
    for (int t = 0; t < TB; ++t)
#pragma unroll
      for (int r = 0; r < RW; ++r) acc[t][r] = Acc2::zero();
    uint4 cur[AHEAD][RW][kVecPerGroup];
    const auto fetch = [&](uint4 (&dst)[RW][kVecPerGroup], int j) {
      const int g = j * 32 + lane;
#pragma unroll
      for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int v = 0; v < kVecPerGroup; ++v) {
          dst[r][v] = make_uint4(0, 0, 0, 0);
          if (j < steps && (whole || g < G)) dst[r][v] = __ldg(reinterpret_cast<const uint4 *>(wp[r] + (size_t)g * 8) + v);
        }
    };
    const auto step = [&](const uint4 (&src)[RW][kVecPerGroup], int j) {
      const int g = j * 32 + lane;
      if (!whole && g >= G) return;
      Pair4<IN> w[RW];
#pragma unroll
      for (int r = 0; r < RW; ++r) w[r].load(&src[r][0]);
#pragma unroll
      for (int t = 0; t < TB; ++t) {
        Pair4<IN> xv;
        xv.load(sx + ((size_t)t * G + g) * kVecPerGroup);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int r = 0; r < RW; ++r) acc[t][r].fma(xv, w[r], i);
      }
    };
    if constexpr (AHEAD == 1) {
      uint4 nxt[RW][kVecPerGroup];
      fetch(cur[0], 0);
#pragma unroll 1
      for (int j = 0; j < steps; ++j) {
        fetch(nxt, j + 1);
        step(cur[0], j);
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int v = 0; v < kVecPerGroup; ++v) cur[0][r][v] = nxt[r][v];
      }
    } else {
#pragma unroll 1
      for (int j = 0; j < steps; j += AHEAD) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) fetch(cur[u], j + u);
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
          if (j + u < steps) step(cur[u], j + u);
      }
    }
    const auto deliver = [&](int t, int row, float sum) {
      if (row >= NR) return;
      if (row < E && bias != nullptr) sum = __fadd_rn(sum, bias[row]);
      // the shared gate's logit (row E) is always a model-dtype linear output
      const float v = (fp32_logits && row < E) ? sum : Load8<IN>::round_model(sum);
      if constexpr (CS == 1) slog[t * ldl + row] = v;
      else store_to_cta(slog + t * ldl + row, t % CS, v);
    };
    if constexpr (TB * RW > 4) {
      // lane t*RW + r ends up with the logit of (token t, row r of this group)
      float part[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) part[i] = 0.f;
#pragma unroll
      for (int t = 0; t < TB; ++t)
#pragma unroll
        for (int r = 0; r < RW; ++r) part[t * RW + r] = acc[t][r].lane_sum();
      const float sum = warp_sum_each(part, lane);
      if (lane / RW < TB) deliver(lane / RW, grp * RW + lane % RW, sum);
    } else {
#pragma unroll
      for (int t = 0; t < TB; ++t)
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const float sum = butterfly_sum(acc[t][r].lane_sum());
          if (lane == 0) deliver(t, grp * RW + r, sum);
        }
    }
  }
  sync_tile<CS>();

  for (int t = rank + CS * warp; t < TB; t += CS * kRouterWarps) {
    const int tok = t0 + t;
    if (tok >= T) continue;
    const float *lg = slog + t * ldl;
    if (out_logits != nullptr) {
      if (fp32_logits)
        for (int e = lane; e < E; e += 32) static_cast<float *>(out_logits)[(size_t)tok * E + e] = lg[e];
      else
        for (int e = lane; e < E; e += 32)
          Load8<IN>::store(static_cast<IN *>(out_logits) + (size_t)tok * E + e, lg[e]);
    }
    if (wsg != nullptr && lane == 0) {
      float v = lg[E];
      float sg = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-v)));
      Load8<IN>::store(out_shared + tok, sg);
    }
    warp_softmax_topk<IN>(lg, E, K, renorm, lane, out_idx + (size_t)tok * K,
                          out_w + (size_t)tok * K);
  }
}

template <typename LT, typename IN>
__global__ void __launch_bounds__(kRouterThreads)
softmax_topk_kernel(const LT *__restrict__ logits, int ld_logits, int T, int E, int K, int renorm,
                    int32_t *__restrict__ out_idx, IN *__restrict__ out_w) {
  __shared__ float slog[kRouterWarps][kMaxExperts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tok = blockIdx.x * kRouterWarps + warp;
  if (tok >= T) return;
  for (int e = lane; e < E; e += 32) slog[warp][e] = Load8<LT>::load(logits + (size_t)tok * ld_logits + e);
  __syncwarp();
  warp_softmax_topk<IN>(slog[warp], E, K, renorm, lane, out_idx + (size_t)tok * K,
                        out_w + (size_t)tok * K);
}

// Decode-sized router: one warp per (token, router row), so a single token's 61
// rows are streamed by 61 warps on 8 SMs instead of by one CTA.  Same per-lane
// summation order as router_kernel (groups lane, lane+32, ...; even/odd partial
// sums; butterfly), hence the same bits.  Logits go to `ws` as fp32 values
// already rounded to the model dtype (unless fp32_logits); softmax_topk_kernel
// finishes the job.
template <typename IN>
__global__ void __launch_bounds__(kRouterThreads)
router_rows_kernel(const IN *__restrict__ x, const IN *__restrict__ wg, const float *__restrict__ bias,
                   const IN *__restrict__ wsg, int T, int H, int E, int fp32_logits,
                   float *__restrict__ ws, void *__restrict__ out_logits, IN *__restrict__ out_shared) {
  constexpr int kVecPerGroup = sizeof(IN) == 2 ? 1 : 2;
  pdl_launch_dependents();
  pdl_wait();
  const int NR = E + (wsg != nullptr ? 1 : 0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tok = blockIdx.x;
  const int row = blockIdx.y * kRouterWarps + warp;
  if (row >= NR) return;
  const IN *wrow = (row < E) ? wg + (size_t)row * H : wsg;
  const IN *xrow = x + (size_t)tok * H;
  const int G = H / 8;
  Acc2 acc = Acc2::zero();
  for (int g0 = 0; g0 < G; g0 += 32 * 4) {
    uint4 wq[4][kVecPerGroup], xq[4][kVecPerGroup];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < kVecPerGroup; ++v) {
        const int g = g0 + u * 32 + lane;
        wq[u][v] = make_uint4(0, 0, 0, 0); xq[u][v] = make_uint4(0, 0, 0, 0);
        if (g < G) {
          wq[u][v] = __ldg(reinterpret_cast<const uint4 *>(wrow + (size_t)g * 8) + v);
          xq[u][v] = __ldg(reinterpret_cast<const uint4 *>(xrow + (size_t)g * 8) + v);
        }
      }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (g0 + u * 32 + lane < G) {
        Pair4<IN> wv, xv;
        wv.load(&wq[u][0]);
        xv.load(&xq[u][0]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc.fma(xv, wv, i);
      }
    }
  }
  float sum = butterfly_sum(acc.lane_sum());
  if (lane == 0) {
    if (row < E) {
      if (bias != nullptr) sum = __fadd_rn(sum, bias[row]);
      const float lg = fp32_logits ? sum : Load8<IN>::round_model(sum);
      ws[(size_t)tok * E + row] = lg;
      if (out_logits != nullptr) {
        if (fp32_logits) static_cast<float *>(out_logits)[(size_t)tok * E + row] = lg;
        else Load8<IN>::store(static_cast<IN *>(out_logits) + (size_t)tok * E + row, lg);
      }
    } else {
      const float v = Load8<IN>::round_model(sum);
      Load8<IN>::store(out_shared + tok, __fdiv_rn(1.f, __fadd_rn(1.f, expf(-v))));
    }
  }
}

template <typename IN, int TB, int RW, int CS, int REGS = 128>
int32_t launch_router_tile(const void *x, const void *wg, const float *bias, const void *wsg, int T,
                           int H, int E, int K, int renorm, int fp32_logits, int32_t *out_idx,
                           void *out_w, void *out_logits, void *out_shared, cudaStream_t stream) {
  const size_t smem = (size_t)TB * H * sizeof(IN) + (size_t)TB * (E + 1) * sizeof(float);
  auto kern = router_kernel<IN, TB, RW, CS, REGS>;
  if (smem > 48 * 1024)
    SB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // The largest shared-memory split, the one a GEMM CTA needs: the two can then share an SM.
  SB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((T + TB - 1) / TB * CS));
  cfg.blockDim = dim3(kRouterThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  SB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, static_cast<const IN *>(x), static_cast<const IN *>(wg), bias,
                                   static_cast<const IN *>(wsg), T, H, E, K, renorm, fp32_logits, out_idx,
                                   static_cast<IN *>(out_w), out_logits, static_cast<IN *>(out_shared)));
  SB_LAUNCH_CHECK();
  return SB_OK;
}

// Tile shapes.  Up to seven tokens per CTA: 28 running sums of two per lane, for which 128
// registers are just too few (24 to 28 bytes a thread are spilled, 40 to 56 in the
// six-token tiles of 112 registers, about 180 in fp32); fewer tokens per tile, and the
// router rows split over a cluster, while that is what it takes to give every SM two CTAs
// (148 SMs):
//   T <= 74    1 token,  2 rows a pass, 4 CTAs per tile    T <= 592   4 tokens, 2 CTAs
//   T <= 296   2 tokens, 4 rows a pass, 2 CTAs             T <= 1036  7 tokens, 2 CTAs
//   above      7 tokens, 1 CTA
// A tile of a wide hidden size gives up tokens until it fits 100 KB.
// `beside` a GEMM, above 592 tokens: six tokens and 112 registers.  The GEMM CTA's ten
// warps of 96 registers are three on one scheduler, and that is what they leave two router
// warps.  At 128 registers the router waits for the GEMM to end (4096 tokens 696 us per
// layer against 680 us, 16384 tokens 2249 us against 2178 us); alone the wider tile is the
// faster one (51 us against 59 us at 4096 tokens, 187 us against 207 us at 16384).  Up to 1024
// tokens the shared pass holds 32 SMs and not all, and the layer's time is the same with
// either tile (277 against 279 us at 1003 tokens, within the spread of its runs).
template <typename IN>
int32_t launch_router_t(const void *x, const void *wg, const float *bias, const void *wsg, int T,
                        int H, int E, int K, int renorm, int fp32_logits, int32_t *out_idx,
                        void *out_w, void *out_logits, void *out_shared, cudaStream_t stream, bool beside) {
  const int slots = 2 * (sb_device_sm_count() > 0 ? sb_device_sm_count() : 148);
  const size_t row = (size_t)H * sizeof(IN) + (size_t)(E + 1) * sizeof(float), room = 100 * 1024;
  auto launch = launch_router_tile<IN, 1, 2, 4>;
  if (T > slots / 4 && 2 * row <= room) launch = launch_router_tile<IN, 2, 4, 2>;
  if (T > slots && 4 * row <= room) launch = launch_router_tile<IN, 4, 4, 2>;
  if (T > 2 * slots && 7 * row <= room) launch = launch_router_tile<IN, 7, 4, 2>;
  if (T > 7 * slots / 2 && 7 * row <= room) launch = launch_router_tile<IN, 7, 4, 1>;
  if constexpr (sizeof(IN) == 2) {       // (the layer pass, which asks for it, is bf16)
    if (beside && T > 2 * slots && 6 * row <= room)
      launch = T > 3 * slots ? launch_router_tile<IN, 6, 4, 1, 112> : launch_router_tile<IN, 6, 4, 2, 112>;
  }
  return launch(x, wg, bias, wsg, T, H, E, K, renorm, fp32_logits, out_idx, out_w, out_logits, out_shared, stream);
}

}  // namespace

int32_t launch_router(const void *x, const void *wg, const float *bias, const void *wsg, int T,
                      int H, int E, int K, int renorm, int dtype, int fp32_logits, int32_t *out_idx,
                      void *out_w, void *out_logits, void *out_shared_scale, cudaStream_t stream, bool beside) {
  if (T < 0 || H <= 0 || H % 8 != 0 || E < 1 || E > kMaxExperts || K < 1 || K > kMaxK || K > E)
    return fail(SB_E_INVALID_ARG, "sb_router_topk: need H%%8==0, 1<=K<=8, K<=E<=256 (T=%d H=%d E=%d K=%d)",
                T, H, E, K);
  if (T == 0) return SB_OK;
  if (!x || !wg || !out_idx || !out_w) return fail(SB_E_INVALID_ARG, "sb_router_topk: null pointer");
  if ((wsg != nullptr) != (out_shared_scale != nullptr))
    return fail(SB_E_INVALID_ARG, "sb_router_topk: w_shared_gate and out_shared_scale go together");
  if (!aligned(x, 16) || !aligned(wg, 16) || (wsg && !aligned(wsg, 16)))
    return fail(SB_E_INVALID_ARG, "sb_router_topk: x, wg, w_shared_gate must be 16-byte aligned");
  if ((size_t)H * (dtype == SB_DTYPE_F32 ? 4 : 2) + (E + 1) * 4 > 200 * 1024)
    return fail(SB_E_UNSUPPORTED, "sb_router_topk: hidden size %d too large for the token tile", H);
  if (dtype == SB_DTYPE_BF16)
    return launch_router_t<__nv_bfloat16>(x, wg, bias, wsg, T, H, E, K, renorm, fp32_logits, out_idx,
                                          out_w, out_logits, out_shared_scale, stream, beside);
  if (dtype == SB_DTYPE_F32)
    return launch_router_t<float>(x, wg, bias, wsg, T, H, E, K, renorm, fp32_logits, out_idx, out_w,
                                  out_logits, out_shared_scale, stream, beside);
  return fail(SB_E_INVALID_ARG, "sb_router_topk: unknown dtype %d", dtype);
}

namespace {

// Decode-sized softmax/top-k AND expert sort in one CTA: warp t finishes token
// t (same arithmetic as softmax_topk_kernel), then the T*K items (at most 128)
// are ranked by (expert id, item index) with an all-pairs count, which yields
// the same stable expert-sorted order, offsets and tile table as the permute
// kernels.
constexpr int kSmallMaxItems = 16 * kMaxK;

__global__ void __launch_bounds__(512)
route_sort_small_kernel(const float *__restrict__ logits, int T, int E, int K, int renorm, int tile_rows,
                        int tile_cap, int32_t *__restrict__ out_idx, __nv_bfloat16 *__restrict__ out_w,
                        int32_t *__restrict__ expert_offsets, int32_t *__restrict__ slot_of_item,
                        int32_t *__restrict__ item_of_slot, __nv_bfloat16 *__restrict__ slot_scale,
                        int32_t *__restrict__ tile_table) {
  __shared__ float slog[16][kMaxExperts];
  __shared__ int s_exp[kSmallMaxItems];
  __shared__ int s_off[kMaxExperts + 1];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < T) {
    for (int e = lane; e < E; e += 32) slog[warp][e] = logits[(size_t)warp * E + e];
    __syncwarp();
    warp_softmax_topk<__nv_bfloat16>(slog[warp], E, K, renorm, lane, out_idx + (size_t)warp * K,
                                     out_w + (size_t)warp * K);
  }
  __syncthreads();                       // this CTA's global writes are visible to all its threads
  const int n = T * K;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int e = out_idx[i];
    s_exp[i] = (e >= 0 && e < E) ? e : -1;
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) {
    int below = 0;
    for (int j = 0; j < n; ++j) below += (s_exp[j] >= 0 && s_exp[j] < e) ? 1 : 0;
    s_off[e] = below;
    expert_offsets[e] = below;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int e = s_exp[i];
    int slot = -1;
    if (e >= 0) {
      slot = 0;
      for (int j = 0; j < n; ++j) slot += (s_exp[j] >= 0 && (s_exp[j] < e || (s_exp[j] == e && j < i))) ? 1 : 0;
      item_of_slot[slot] = i;
      slot_scale[slot] = out_w[i];
    }
    slot_of_item[i] = slot;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int ts = 0;                          // tiles of the experts below e
    for (int j = 0; j < e; ++j) ts += (s_off[j + 1] - s_off[j] + tile_rows - 1) / tile_rows;
    const int cnt = s_off[e + 1] - s_off[e];
    const int nt = (cnt + tile_rows - 1) / tile_rows;
    for (int m = 0; m < nt; ++m) {
      const int ti = ts + m;
      if (ti >= tile_cap) break;
      int32_t *ent = tile_table + kTileHeaderInts + (size_t)ti * kTileEntryInts;
      const int rb = s_off[e] + m * tile_rows;
      ent[0] = e; ent[1] = rb; ent[2] = min(s_off[e + 1], rb + tile_rows); ent[3] = 0;
    }
    if (e == E - 1) {
      const int all = ts + nt;
      tile_table[0] = all < tile_cap ? all : tile_cap;
      tile_table[1] = s_off[E];
      tile_table[2] = tile_rows; tile_table[3] = 0;
    }
  }
}

}  // namespace

int32_t launch_router_decode(const void *x, const void *wg, const float *bias, const void *wsg, int T, int H,
                             int E, int K, int renorm, int fp32_logits, float *ws, int32_t *out_idx,
                             void *out_w, void *out_logits, void *out_shared_scale, int32_t *expert_offsets,
                             int32_t *slot_of_item, int32_t *item_of_slot, void *slot_scale, int32_t *tile_table,
                             cudaStream_t stream) {
  if (T <= 0) return SB_OK;
  if (H % 8 != 0 || E < 1 || E > kMaxExperts || K < 1 || K > kMaxK || K > E || !ws)
    return fail(SB_E_INVALID_ARG, "router (decode): bad arguments");
  if (!aligned(x, 16) || !aligned(wg, 16) || (wsg && !aligned(wsg, 16)))
    return fail(SB_E_INVALID_ARG, "router (decode): x, wg, w_shared_gate must be 16-byte aligned");
  const int NR = E + (wsg ? 1 : 0);
  dim3 grid(T, (NR + kRouterWarps - 1) / kRouterWarps);
  SB_CUDA_CHECK(launch_pdl(router_rows_kernel<__nv_bfloat16>, grid, dim3(kRouterThreads), 0, stream,
                           static_cast<const __nv_bfloat16 *>(x), static_cast<const __nv_bfloat16 *>(wg), bias,
                           static_cast<const __nv_bfloat16 *>(wsg), T, H, E, fp32_logits, ws, out_logits,
                           static_cast<__nv_bfloat16 *>(out_shared_scale)));
  SB_LAUNCH_CHECK();
  if (tile_table != nullptr) {
    // softmax/top-k and the expert sort in one single-CTA launch
    if (T > 16 || !expert_offsets || !slot_of_item || !item_of_slot || !slot_scale)
      return fail(SB_E_INVALID_ARG, "router (decode): sort outputs need T <= 16 and all tables");
    const int warps = T > 4 ? 16 : 4;
    SB_CUDA_CHECK(launch_pdl(route_sort_small_kernel, dim3(1), dim3(warps * 32), 0, stream,
                             static_cast<const float *>(ws), T, E, K, renorm, sb_tile_rows(),
                             T * K / SB_TILE_M + E, out_idx, static_cast<__nv_bfloat16 *>(out_w), expert_offsets,
                             slot_of_item, item_of_slot, static_cast<__nv_bfloat16 *>(slot_scale), tile_table));
    SB_LAUNCH_CHECK();
    return SB_OK;
  }
  softmax_topk_kernel<float, __nv_bfloat16><<<(T + kRouterWarps - 1) / kRouterWarps, kRouterThreads, 0, stream>>>(
      ws, E, T, E, K, renorm, out_idx, static_cast<__nv_bfloat16 *>(out_w));
  SB_LAUNCH_CHECK();
  return SB_OK;
}

int32_t launch_softmax_topk(const void *logits, int T, int E, int K, int renorm, int dtype,
                            int32_t *out_idx, void *out_w, cudaStream_t stream) {
  if (T < 0 || E < 1 || E > kMaxExperts || K < 1 || K > kMaxK || K > E)
    return fail(SB_E_INVALID_ARG, "sb_softmax_topk: need 1<=K<=8, K<=E<=256 (T=%d E=%d K=%d)", T, E, K);
  if (T == 0) return SB_OK;
  if (!logits || !out_idx || !out_w) return fail(SB_E_INVALID_ARG, "sb_softmax_topk: null pointer");
  int blocks = (T + kRouterWarps - 1) / kRouterWarps;
  if (dtype == SB_DTYPE_BF16)
    softmax_topk_kernel<__nv_bfloat16, __nv_bfloat16><<<blocks, kRouterThreads, 0, stream>>>(
        static_cast<const __nv_bfloat16 *>(logits), E, T, E, K, renorm, out_idx,
        static_cast<__nv_bfloat16 *>(out_w));
  else if (dtype == SB_DTYPE_F32)
    softmax_topk_kernel<float, float><<<blocks, kRouterThreads, 0, stream>>>(
        static_cast<const float *>(logits), E, T, E, K, renorm, out_idx, static_cast<float *>(out_w));
  else
    return fail(SB_E_INVALID_ARG, "sb_softmax_topk: unknown dtype %d", dtype);
  SB_LAUNCH_CHECK();
  return SB_OK;
}

}  // namespace sb
