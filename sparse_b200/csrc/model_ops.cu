// The small kernels of the decode loop around the MoE layers: RMSNorm with the
// residual add folded in, rotary embedding + KV-cache append, and decode-time
// attention (one query per sequence against the cache).
//
// The reference runs these through the Transformers model classes
// (utils/eval_core.py:17807-17829 loads them, the loop at 18464-18607 calls
// them once per generated token); here they are plain CUDA so that one decode
// step -- every layer's attention, norms and MoE block -- can be captured in a
// single CUDA graph.  All three are HBM-bound: the norm reads and writes its
// rows once, the attention reads each cached key and value exactly once.
//
// Arithmetic contract (matched by the fp32 PyTorch restatement in the tests
// within bf16 tolerance): sums and softmax in fp32; bf16 rounding of the
// residual sum, of the normalised row before the weight multiply, and of the
// outputs.
#include "sb_common.cuh"

namespace sb {
namespace {

constexpr int kNormThreads = 256;
constexpr int kMaxNormRow = 16384;    // eight 16-byte vectors a thread

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// One CTA per row.  h = bf16(residual + delta) (or residual alone); the row is
// written back to `residual` when a delta was added; out = weight * bf16(h * rsqrt(mean(h^2) + eps)).
//
// HBM-bound at prefill: a row is read once as 16-byte vectors, stays in registers
// (NV vectors a thread; a bf16 copy in shared memory for the sum of squares) and is
// written once, residual and normalised.
// (2-byte accesses and a row in shared memory: 17 us for 4096 rows of 2048, whose
// bytes take 10 us.)  At a decode step's few rows it is one load round trip.
template <int NV>
__global__ void __launch_bounds__(kNormThreads)
add_rmsnorm_vec_kernel(__nv_bfloat16 *__restrict__ residual, size_t res_stride,
                       const __nv_bfloat16 *__restrict__ delta, const __nv_bfloat16 *__restrict__ delta2,
                       const __nv_bfloat16 *__restrict__ weight, float eps, int H, __nv_bfloat16 *__restrict__ out) {
  __shared__ float part[kNormThreads / 32];
  __shared__ uint4 row[NV * kNormThreads];
  pdl_launch_dependents();
  pdl_wait();
  const int vecs = H >> 3;
  const size_t base = (size_t)blockIdx.x * vecs;
  uint4 *res = reinterpret_cast<uint4 *>(residual + blockIdx.x * res_stride);
  const uint4 *d1 = reinterpret_cast<const uint4 *>(delta) + base, *d2 = reinterpret_cast<const uint4 *>(delta2) + base;
  uint4 r[NV], a[NV], b[NV], w[NV];
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int i = threadIdx.x + n * kNormThreads;
    r[n] = a[n] = b[n] = w[n] = make_uint4(0, 0, 0, 0);
    if (i < vecs) {
      r[n] = res[i];
      if (delta != nullptr) a[n] = __ldg(d1 + i);
      if (delta2 != nullptr) b[n] = __ldg(d2 + i);
      if (out != nullptr) w[n] = __ldg(reinterpret_cast<const uint4 *>(weight) + i);
    }
  }
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int i = threadIdx.x + n * kNormThreads;
    uint32_t *rv = reinterpret_cast<uint32_t *>(&r[n]);
    const uint32_t *av = reinterpret_cast<const uint32_t *>(&a[n]), *bv = reinterpret_cast<const uint32_t *>(&b[n]);
    if (delta != nullptr) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float lo = round_bf16(bf16_lo(rv[k]) + bf16_lo(av[k])), hi = round_bf16(bf16_hi(rv[k]) + bf16_hi(av[k]));
        if (delta2 != nullptr) {
          lo = round_bf16(lo + bf16_lo(bv[k]));
          hi = round_bf16(hi + bf16_hi(bv[k]));
        }
        rv[k] = pack_bf16x2(lo, hi);
      }
      if (i < vecs) res[i] = r[n];
    }
    if (i < vecs) row[i] = r[n];
  }
  if (out == nullptr) return;
  // The squares are summed in element order t, t + 256, ... per thread, as the
  // kernel for ragged rows below does: the same bits whatever the row's alignment.
  __syncthreads();
  const __nv_bfloat16 *elem = reinterpret_cast<const __nv_bfloat16 *>(row);
  float ss = 0.f;
#pragma unroll 8
  for (int i = threadIdx.x; i < H; i += kNormThreads) {
    const float v = __bfloat162float(elem[i]);
    ss += v * v;
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) tot += part[i];
  const float inv = rsqrtf(tot / (float)H + eps);
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int i = threadIdx.x + n * kNormThreads;
    const uint32_t *rv = reinterpret_cast<const uint32_t *>(&r[n]), *wv = reinterpret_cast<const uint32_t *>(&w[n]);
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      o[k] = pack_bf16x2(bf16_lo(wv[k]) * round_bf16(bf16_lo(rv[k]) * inv), bf16_hi(wv[k]) * round_bf16(bf16_hi(rv[k]) * inv));
    if (i < vecs) reinterpret_cast<uint4 *>(out)[base + i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// The same for rows that are no whole 16-byte vectors (or not aligned to them).
__global__ void __launch_bounds__(kNormThreads)
add_rmsnorm_kernel(__nv_bfloat16 *__restrict__ residual, size_t res_stride, const __nv_bfloat16 *__restrict__ delta,
                   const __nv_bfloat16 *__restrict__ delta2, const __nv_bfloat16 *__restrict__ weight, float eps,
                   int H, __nv_bfloat16 *__restrict__ out) {
  extern __shared__ float row[];                 // H floats
  __shared__ float part[kNormThreads / 32];
  const size_t base = (size_t)blockIdx.x * H;
  residual += blockIdx.x * res_stride;
  float ss = 0.f;
  for (int i = threadIdx.x; i < H; i += kNormThreads) {
    float v = __bfloat162float(residual[i]);
    if (delta != nullptr) {
      v = round_bf16(v + __bfloat162float(delta[base + i]));
      if (delta2 != nullptr) v = round_bf16(v + __bfloat162float(delta2[base + i]));
      residual[i] = __float2bfloat16_rn(v);
    }
    row[i] = v;
    ss += v * v;
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < kNormThreads / 32; ++w) tot += part[w];
  const float inv = rsqrtf(tot / (float)H + eps);
  if (out != nullptr)
    for (int i = threadIdx.x; i < H; i += kNormThreads)
      out[base + i] = __float2bfloat16_rn(__bfloat162float(weight[i]) * round_bf16(row[i] * inv));
}

int32_t launch_add_rmsnorm(void *residual, int res_stride, const void *delta, const void *delta2, const void *weight,
                           float eps, int T, int H, void *out, cudaStream_t stream) {
  __nv_bfloat16 *res = static_cast<__nv_bfloat16 *>(residual), *oo = static_cast<__nv_bfloat16 *>(out);
  const __nv_bfloat16 *d1 = static_cast<const __nv_bfloat16 *>(delta), *d2 = static_cast<const __nv_bfloat16 *>(delta2);
  const __nv_bfloat16 *ww = static_cast<const __nv_bfloat16 *>(weight);
  if (H % 8 == 0 && res_stride % 8 == 0 && aligned(res, 16) && aligned(d1, 16) && aligned(d2, 16) && aligned(ww, 16) &&
      aligned(oo, 16)) {
    const int nv = (H / 8 + kNormThreads - 1) / kNormThreads;
    auto kern = nv == 1 ? add_rmsnorm_vec_kernel<1> : nv == 2 ? add_rmsnorm_vec_kernel<2>
                        : nv <= 4 ? add_rmsnorm_vec_kernel<4> : add_rmsnorm_vec_kernel<8>;
    SB_CUDA_CHECK(launch_pdl(kern, dim3(T), dim3(kNormThreads), 0, stream, res, (size_t)res_stride, d1, d2, ww, eps, H, oo));
  } else {
    if ((size_t)H * sizeof(float) > 47 * 1024)          // (with the partial sums more than the 48 KB of any launch)
      SB_CUDA_CHECK(cudaFuncSetAttribute(add_rmsnorm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kMaxNormRow * (int)sizeof(float)));
    add_rmsnorm_kernel<<<T, kNormThreads, (size_t)H * sizeof(float), stream>>>(res, (size_t)res_stride, d1, d2, ww, eps,
                                                                               H, oo);
  }
  SB_LAUNCH_CHECK();
  return SB_OK;
}

// Rotates the first `rope_dim` elements of every q and k head (pairs
// (i, i + rope_dim/2), angle pos * theta^(-2i/rope_dim)), writes q back in place
// and k, v into the cache row of (sequence, position).
//
// A token's angles are the same for every head: the CTA works out its
// rope_dim/2 sines and cosines once, in shared memory, and the heads then move
// as W-element vectors (W = 8: 16 bytes), all of a thread's loads independent.
// HBM-bound at prefill (q, k, v read and written once); at a decode step's few
// tokens it is the length of the chain position -> angle -> rows, so the token's
// vectors are spread over `gridDim.y` CTAs.  (One sincosf per rotated element and
// 2-byte accesses: 18 us at 8 tokens, 91 us at 4096 tokens of 16 heads of 128.)
// W = 1 serves head widths, strides and addresses that are no whole vectors.
constexpr int kRopeThreads = 256;
constexpr int kRopeTable = 1024;      // angles kept in shared memory; wider heads compute them per element

struct RopeSource {                   // element (token t, head h, i) at base + t*token + h*head + i
  const __nv_bfloat16 *base;
  int token, head;
  __device__ __forceinline__ const __nv_bfloat16 *at(int t, int h) const {
    return base + (size_t)t * token + (size_t)h * head;
  }
};

__device__ __forceinline__ float2 rope_cos_sin(int pos, int j, float log_theta, int rope_dim) {
  const float ang = (float)pos * __expf(-log_theta * (2.0f * (float)j / (float)rope_dim));
  float sn, cs;
  sincosf(ang, &sn, &cs);
  return make_float2(round_bf16(cs), round_bf16(sn));
}

template <int W> struct RopeVec { uint32_t w[W / 2]; };
template <> struct RopeVec<1> { unsigned short w; };

template <int W>
__device__ __forceinline__ RopeVec<W> rope_load(const __nv_bfloat16 *p) {
  RopeVec<W> r;
  if constexpr (W == 8) {
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    r.w[0] = q.x; r.w[1] = q.y; r.w[2] = q.z; r.w[3] = q.w;
  } else {
    r.w = *reinterpret_cast<const unsigned short *>(p);
  }
  return r;
}
template <int W>
__device__ __forceinline__ void rope_store(__nv_bfloat16 *p, const RopeVec<W> &r) {
  if constexpr (W == 8) *reinterpret_cast<uint4 *>(p) = make_uint4(r.w[0], r.w[1], r.w[2], r.w[3]);
  else *reinterpret_cast<unsigned short *>(p) = r.w;
}
__device__ __forceinline__ float2 rope_pair(float a, float b, float2 cs) {
  return make_float2(round_bf16(a * cs.x) + round_bf16(-b * cs.y), round_bf16(b * cs.x) + round_bf16(a * cs.y));
}

// src (lo half at src, hi half at src + half) rotated into dst, W pairs from pair j on
template <int W>
__device__ __forceinline__ void rope_rotate(const __nv_bfloat16 *src, __nv_bfloat16 *dst, int j, int half, int pos,
                                            float log_theta, int rope_dim, const float2 *table) {
  const RopeVec<W> lo = rope_load<W>(src + j), hi = rope_load<W>(src + j + half);
  RopeVec<W> rl, rh;
  if constexpr (W == 8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 e = rope_pair(bf16_lo(lo.w[i]), bf16_lo(hi.w[i]), table[j + 2 * i]);
      const float2 o = rope_pair(bf16_hi(lo.w[i]), bf16_hi(hi.w[i]), table[j + 2 * i + 1]);
      rl.w[i] = pack_bf16x2(e.x, o.x);
      rh.w[i] = pack_bf16x2(e.y, o.y);
    }
  } else {
    const float2 cs = half <= kRopeTable ? table[j] : rope_cos_sin(pos, j, log_theta, rope_dim);
    const float2 e = rope_pair(__bfloat162float(__ushort_as_bfloat16(lo.w)),
                               __bfloat162float(__ushort_as_bfloat16(hi.w)), cs);
    rl.w = __bfloat16_as_ushort(__float2bfloat16_rn(e.x));
    rh.w = __bfloat16_as_ushort(__float2bfloat16_rn(e.y));
  }
  rope_store<W>(dst + j, rl);
  rope_store<W>(dst + j + half, rh);
}

template <int W>
__global__ void __launch_bounds__(kRopeThreads)
rope_append_kernel(__nv_bfloat16 *__restrict__ q, int q_stride, RopeSource k_rot, RopeSource k_rest, RopeSource v,
                   const int32_t *__restrict__ seq_of_token, const int32_t *__restrict__ pos_of_token, int n_q,
                   int n_kv, int dk, int dv, int rope_dim, float theta, int s_max,
                   __nv_bfloat16 *__restrict__ cache_k, __nv_bfloat16 *__restrict__ cache_v) {
  __shared__ float2 table[kRopeTable];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int pos = pos_of_token[t], seq = seq_of_token[t];
  const int half = rope_dim >> 1;
  const float log_theta = __logf(theta);
  if (half <= kRopeTable)
    for (int j = threadIdx.x; j < half; j += kRopeThreads) table[j] = rope_cos_sin(pos, j, log_theta, rope_dim);
  __syncthreads();
  const bool cached = pos >= 0 && pos < s_max;
  __nv_bfloat16 *ck = cache_k + ((size_t)seq * s_max + pos) * n_kv * dk;
  __nv_bfloat16 *cv = cache_v + ((size_t)seq * s_max + pos) * n_kv * dv;
  // the token's vectors in one line: rotated q, rotated k, rest of k, v
  const int per_rot = half / W, per_rest = (dk - rope_dim) / W, per_v = dv / W;
  const int end_q = n_q * per_rot, end_k = end_q + n_kv * per_rot, end_rest = end_k + n_kv * per_rest;
  const int end = cached ? end_rest + n_kv * per_v : end_q;
  for (int i = blockIdx.y * kRopeThreads + threadIdx.x; i < end; i += gridDim.y * kRopeThreads) {
    if (i < end_q) {
      const int h = i / per_rot, j = (i - h * per_rot) * W;
      __nv_bfloat16 *p = q + (size_t)t * q_stride + (size_t)h * dk;
      rope_rotate<W>(p, p, j, half, pos, log_theta, rope_dim, table);
    } else if (i < end_k) {
      const int n = i - end_q, h = n / per_rot, j = (n - h * per_rot) * W;
      rope_rotate<W>(k_rot.at(t, h), ck + (size_t)h * dk, j, half, pos, log_theta, rope_dim, table);
    } else if (i < end_rest) {
      const int n = i - end_k, h = n / per_rest, j = (n - h * per_rest) * W;
      rope_store<W>(ck + (size_t)h * dk + rope_dim + j, rope_load<W>(k_rest.at(t, h) + j));
    } else {
      const int n = i - end_rest, h = n / per_v, j = (n - h * per_v) * W;
      rope_store<W>(cv + (size_t)h * dv + j, rope_load<W>(v.at(t, h) + j));
    }
  }
}

int32_t launch_rope(__nv_bfloat16 *q, int q_stride, RopeSource k_rot, RopeSource k_rest, RopeSource v,
                    const int32_t *seq_of_token, const int32_t *pos_of_token, int T, int n_q, int n_kv, int dk, int dv,
                    int rope_dim, float theta, int s_max, void *cache_k, void *cache_v, cudaStream_t stream) {
  const auto whole = [](const RopeSource &s) { return aligned(s.base, 16) && s.token % 8 == 0 && s.head % 8 == 0; };
  const bool vec = dk % 8 == 0 && dv % 8 == 0 && rope_dim % 16 == 0 && rope_dim <= 2 * kRopeTable && q_stride % 8 == 0 &&
                   aligned(q, 16) && whole(k_rot) && whole(k_rest) && whole(v) && aligned(cache_k, 16) && aligned(cache_v, 16);
  // at most two waves of CTAs: more would only repeat the angle table
  const int sms = sb_device_sm_count() > 0 ? sb_device_sm_count() : 148;
  const int items = (n_q * (rope_dim / 2) + n_kv * (dk - rope_dim / 2 + dv)) / (vec ? 8 : 1);
  const int wanted = (items + kRopeThreads - 1) / kRopeThreads, room = (2 * sms + T - 1) / T;
  const dim3 grid(T, wanted < 1 ? 1 : wanted < room ? wanted : room);
  auto kern = vec ? rope_append_kernel<8> : rope_append_kernel<1>;
  SB_CUDA_CHECK(launch_pdl(kern, grid, dim3(kRopeThreads), 0, stream, q, q_stride, k_rot, k_rest, v, seq_of_token,
                           pos_of_token, n_q, n_kv, dk, dv, rope_dim, theta, s_max,
                           static_cast<__nv_bfloat16 *>(cache_k), static_cast<__nv_bfloat16 *>(cache_v)));
  SB_LAUNCH_CHECK();
  return SB_OK;
}

// Decode attention, split over the keys.  grid = (sequences * query heads,
// splits).  HBM-bound: every cached key and value is read once, so what counts is
// bytes in flight and instructions per byte.  Eight lanes share a key: lane i of
// them owns the 16-byte vectors i, i + 8, ... of the key and of the value, so a
// warp's load covers four keys in whole 128-byte lines, the score needs three
// shuffles for four keys, and each of the 16 groups of a CTA keeps its own running
// maximum; groups, then warps, then splits are merged by their maxima.
// (One key per warp with 8-byte loads and five shuffles a key: 30 us for the
// 137 MB of 8 sequences of 2049 positions with 16 heads of 128.)  Seven CTAs per
// SM, where the head width lets the registers: the splits are cut for six.
constexpr int kAttnThreads = 128;
constexpr int kAttnLanes = 8;                                   // lanes per key
constexpr int kAttnGroups = kAttnThreads / kAttnLanes;

// 8 elements as fp32; A16: the address is a multiple of 16 bytes (else of 4)
template <bool A16>
__device__ __forceinline__ uint4 load_vec8(const __nv_bfloat16 *p) {
  if (A16) return __ldg(reinterpret_cast<const uint4 *>(p));
  const uint32_t *w = reinterpret_cast<const uint32_t *>(p);
  return make_uint4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
}

template <int DK, int DV, bool A16>
__global__ void __launch_bounds__(kAttnThreads, DK <= 128 ? 7 : 5)
attn_decode_kernel(const __nv_bfloat16 *__restrict__ q, int q_stride, const __nv_bfloat16 *__restrict__ cache_k,
                   const __nv_bfloat16 *__restrict__ cache_v, const int32_t *__restrict__ seq_lens, int n_q,
                   int n_kv, int s_max, float scale, int n_split, float *__restrict__ part) {
  constexpr int NK = DK / 64, NV = DV / 64;   // vectors a lane owns of a key / of a value
  constexpr int U = 2;                        // keys a group has in flight per iteration
  pdl_launch_dependents();
  pdl_wait();
  const int bh = blockIdx.x, split = blockIdx.y;
  const int b = bh / n_q, h = bh - b * n_q;
  const int hk = h / (n_q / n_kv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = threadIdx.x / kAttnLanes, li = threadIdx.x % kAttnLanes;
  const int len = min(seq_lens[b], s_max);
  const int per = (len + n_split - 1) / n_split;
  const int j0 = split * per, j1 = min(len, j0 + per);
  float qv[NK * 8];
#pragma unroll
  for (int e = 0; e < NK * 8; ++e)
    qv[e] = __bfloat162float(q[(size_t)b * q_stride + (size_t)h * DK + ((e >> 3) * kAttnLanes + li) * 8 + (e & 7)]) * scale;
  float m = -INFINITY, l = 0.f, acc[NV * 8];
#pragma unroll
  for (int e = 0; e < NV * 8; ++e) acc[e] = 0.f;
  const __nv_bfloat16 *kb = cache_k + ((size_t)b * s_max * n_kv + hk) * DK + li * 8;
  const __nv_bfloat16 *vb = cache_v + ((size_t)b * s_max * n_kv + hk) * DV + li * 8;
  for (int base = j0; base < j1; base += kAttnGroups * U) {
    uint4 kv[U][NK], vv[U][NV];
    float s[U];
    bool ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = base + u * kAttnGroups + group;
      ok[u] = j < j1;
      const int jj = min(j, j1 - 1);          // clamped: a line its neighbours read too, masked below
#pragma unroll
      for (int n = 0; n < NK; ++n) kv[u][n] = load_vec8<A16>(kb + (size_t)jj * n_kv * DK + n * kAttnLanes * 8);
#pragma unroll
      for (int n = 0; n < NV; ++n) vv[u][n] = load_vec8<A16>(vb + (size_t)jj * n_kv * DV + n * kAttnLanes * 8);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float even = 0.f, odd = 0.f;
#pragma unroll
      for (int n = 0; n < NK; ++n) {
        const uint32_t w[4] = {kv[u][n].x, kv[u][n].y, kv[u][n].z, kv[u][n].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          even += qv[n * 8 + 2 * i] * bf16_lo(w[i]);
          odd += qv[n * 8 + 2 * i + 1] * bf16_hi(w[i]);
        }
      }
      s[u] = even + odd;
    }
#pragma unroll
    for (int off = kAttnLanes / 2; off >= 1; off >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
    float m_new = m;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (ok[u]) m_new = fmaxf(m_new, s[u]);
    // a group that has seen no key yet, or only scores of -inf, keeps its zero sums: those
    // keys have the weight exp(-inf - 0) = 0
    const float m_ref = m_new == -INFINITY ? 0.f : m_new;
    const float corr = m == m_new ? 1.f : __expf(m - m_ref);
    l *= corr;
#pragma unroll
    for (int e = 0; e < NV * 8; ++e) acc[e] *= corr;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!ok[u]) continue;                   // a masked key adds nothing, whatever its clamped row holds
      const float p = __expf(s[u] - m_ref);
      l += p;
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const uint32_t w[4] = {vv[u][n].x, vv[u][n].y, vv[u][n].z, vv[u][n].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[n * 8 + 2 * i] += p * bf16_lo(w[i]);
          acc[n * 8 + 2 * i + 1] += p * bf16_hi(w[i]);
        }
      }
    }
    m = m_new;
  }
  // merge the four groups of a warp, then the four warps
#pragma unroll
  for (int off = kAttnLanes; off <= 16; off <<= 1) {
    const float mm = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    const float c = m == -INFINITY ? 0.f : __expf(m - mm);
    l *= c;
    l += __shfl_xor_sync(0xffffffffu, l, off);
#pragma unroll
    for (int e = 0; e < NV * 8; ++e) {
      acc[e] *= c;
      acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], off);
    }
    m = mm;
  }
  __shared__ float sm[4], sl[4], sacc[4][DV];
  if (lane == 0) { sm[warp] = m; sl[warp] = l; }
  if (lane < kAttnLanes) {
#pragma unroll
    for (int e = 0; e < NV * 8; ++e) sacc[warp][((e >> 3) * kAttnLanes + li) * 8 + (e & 7)] = acc[e];
  }
  __syncthreads();
  float *dst = part + ((size_t)bh * n_split + split) * (DV + 2);
  const float mm = fmaxf(fmaxf(sm[0], sm[1]), fmaxf(sm[2], sm[3]));
  float c[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) c[w] = sm[w] == -INFINITY ? 0.f : __expf(sm[w] - mm);
  if (threadIdx.x < DV)
    dst[2 + threadIdx.x] = sacc[0][threadIdx.x] * c[0] + sacc[1][threadIdx.x] * c[1] + sacc[2][threadIdx.x] * c[2] +
                           sacc[3][threadIdx.x] * c[3];
  if (threadIdx.x == 0) {
    dst[0] = mm;
    dst[1] = sl[0] * c[0] + sl[1] * c[1] + sl[2] * c[2] + sl[3] * c[3];
  }
}

// One CTA of DV threads per (sequence, head).  The first warp turns the splits'
// maxima into weights, so the sum over the splits is a run of independent loads
// (with the weights worked out by every thread in the loop: 7.6 us at 56 splits).
constexpr int kMaxSplit = 256;
template <int DV>
__global__ void __launch_bounds__(DV)
attn_merge_kernel(const float *__restrict__ part, int n_split, __nv_bfloat16 *__restrict__ out) {
  __shared__ float weight[kMaxSplit];
  __shared__ float total;
  pdl_launch_dependents();
  pdl_wait();
  const int bh = blockIdx.x;
  const float *src = part + (size_t)bh * n_split * (DV + 2);
  if (threadIdx.x < 32) {
    float ms[kMaxSplit / 32], ls[kMaxSplit / 32], mm = -INFINITY, ll = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxSplit / 32; ++i) {
      const int s = threadIdx.x + 32 * i;
      ms[i] = -INFINITY; ls[i] = 0.f;
      if (s < n_split) { ms[i] = src[(size_t)s * (DV + 2)]; ls[i] = src[(size_t)s * (DV + 2) + 1]; }
      mm = fmaxf(mm, ms[i]);
    }
    mm = warp_max(mm);
#pragma unroll
    for (int i = 0; i < kMaxSplit / 32; ++i) {
      const float c = ms[i] == -INFINITY ? 0.f : __expf(ms[i] - mm);
      ll += ls[i] * c;
      if (threadIdx.x + 32 * i < n_split) weight[threadIdx.x + 32 * i] = c;
    }
    ll = warp_sum(ll);
    if (threadIdx.x == 0) total = ll;
  }
  __syncthreads();
  float acc = 0.f;
#pragma unroll 8
  for (int s = 0; s < n_split; ++s) acc += src[(size_t)s * (DV + 2) + 2 + threadIdx.x] * weight[s];
  out[(size_t)bh * DV + threadIdx.x] = __float2bfloat16_rn(total > 0.f ? acc / total : 0.f);
}

template <int DK, int DV>
int32_t launch_attn_decode(const __nv_bfloat16 *q, int q_stride, const __nv_bfloat16 *cache_k,
                           const __nv_bfloat16 *cache_v, const int32_t *seq_lens, int B, int n_q, int n_kv, int s_max,
                           float scale, int n_split, float *part, __nv_bfloat16 *out, cudaStream_t stream) {
  auto kern = aligned(cache_k, 16) && aligned(cache_v, 16) ? attn_decode_kernel<DK, DV, true>
                                                           : attn_decode_kernel<DK, DV, false>;
  SB_CUDA_CHECK(launch_pdl(kern, dim3(B * n_q, n_split), dim3(kAttnThreads), 0, stream, q, q_stride, cache_k, cache_v,
                           seq_lens, n_q, n_kv, s_max, scale, n_split, part));
  SB_LAUNCH_CHECK();
  SB_CUDA_CHECK(launch_pdl(attn_merge_kernel<DV>, dim3(B * n_q), dim3(DV), 0, stream,
                           static_cast<const float *>(part), n_split, out));
  SB_LAUNCH_CHECK();
  return SB_OK;
}

// Greedy token of every row of logits: the index of the largest value, the first
// one among equals, NaN above every number (torch.argmax's rules).  A cluster of
// eight CTAs per row: each reads its eighth of the vocabulary as 16-byte vectors and
// the leader takes the best of the eight through distributed shared memory.
// Latency-bound: one row of 102400 is 200 KB (a library reduction over an fp32 copy
// of the row took 25 + 5 us, on one CTA).
constexpr int kArgmaxThreads = 512;
constexpr int kArgmaxCtas = 8;

// values as keys in their order; index in the low half so that of equal values the first wins
__device__ __forceinline__ unsigned long long argmax_key(uint32_t bf16_bits, uint32_t index) {
  const uint32_t mag = bf16_bits & 0x7fffu;
  uint32_t ord = bf16_bits & 0x8000u ? 0x8000u - mag : 0x8000u + mag;       // -0 and +0 give the same
  if (mag > 0x7f80u) ord = 0x10000u;                                        // NaN
  return ((unsigned long long)ord << 32) | (0xffffffffu - index);
}
__device__ __forceinline__ unsigned long long key_max(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

__global__ void __cluster_dims__(kArgmaxCtas, 1, 1) __launch_bounds__(kArgmaxThreads)
argmax_rows_kernel(const __nv_bfloat16 *__restrict__ logits, int V, int vec, int64_t *__restrict__ out) {
  __shared__ unsigned long long best_of_warp[kArgmaxThreads / 32];
  __shared__ unsigned long long best_of_cta[kArgmaxCtas];
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x / kArgmaxCtas;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const unsigned short *src = reinterpret_cast<const unsigned short *>(logits) + (size_t)row * V;
  unsigned long long best = 0;
  if (vec) {
    const uint4 *v = reinterpret_cast<const uint4 *>(src);
#pragma unroll 4
    for (int i = rank * kArgmaxThreads + threadIdx.x; i < V / 8; i += kArgmaxCtas * kArgmaxThreads) {
      const uint4 q = __ldg(v + i);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        best = key_max(best, argmax_key(w[k] & 0xffffu, 8 * i + 2 * k));
        best = key_max(best, argmax_key(w[k] >> 16, 8 * i + 2 * k + 1));
      }
    }
  } else {
    for (int i = rank * kArgmaxThreads + threadIdx.x; i < V; i += kArgmaxCtas * kArgmaxThreads)
      best = key_max(best, argmax_key(src[i], i));
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) best = key_max(best, __shfl_xor_sync(0xffffffffu, best, off));
  if ((threadIdx.x & 31) == 0) best_of_warp[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = threadIdx.x < kArgmaxThreads / 32 ? best_of_warp[threadIdx.x] : 0;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) best = key_max(best, __shfl_xor_sync(0xffffffffu, best, off));
  }
  // (the first arrive also says that every CTA of the cluster has started)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x == 0) {
    uint32_t addr;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;"
                 : "=r"(addr) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(best_of_cta + rank))));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(best) : "memory");
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank == 0 && threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < kArgmaxCtas; ++c) best = key_max(best, best_of_cta[c]);
    out[row] = (int64_t)(0xffffffffu - (uint32_t)best);
  }
}

}  // namespace
}  // namespace sb

using namespace sb;

extern "C" {

int32_t sb_add_rmsnorm(void *residual, const void *delta, const void *delta2, const void *weight, float eps,
                       int32_t T, int32_t H, void *out, void *stream) {
  if (T < 0 || H <= 0 || H > kMaxNormRow) return fail(SB_E_INVALID_ARG, "sb_add_rmsnorm: bad shape (T=%d H=%d)", T, H);
  if (T == 0) return SB_OK;
  if (!residual || (!out && !delta) || (out && !weight) || (delta2 && !delta))
    return fail(SB_E_INVALID_ARG, "sb_add_rmsnorm: null pointer");
  return launch_add_rmsnorm(residual, H, delta, delta2, weight, eps, T, H, out, static_cast<cudaStream_t>(stream));
}

int32_t sb_rmsnorm_rows(const void *rows, int32_t row_stride, const void *weight, float eps, int32_t T, int32_t H,
                        void *out, void *stream) {
  if (T < 0 || H <= 0 || H > kMaxNormRow || row_stride < H)
    return fail(SB_E_INVALID_ARG, "sb_rmsnorm_rows: bad shape (T=%d H=%d stride=%d)", T, H, row_stride);
  if (T == 0) return SB_OK;
  if (!rows || !weight || !out) return fail(SB_E_INVALID_ARG, "sb_rmsnorm_rows: null pointer");
  // (without a delta the kernel does not write to its source rows)
  return launch_add_rmsnorm(const_cast<void *>(rows), row_stride, nullptr, nullptr, weight, eps, T, H, out,
                            static_cast<cudaStream_t>(stream));
}

int32_t sb_rope_append(void *q, const void *k, const void *v, const int32_t *seq_of_token,
                       const int32_t *pos_of_token, int32_t T, int32_t n_q, int32_t n_kv, int32_t dk, int32_t dv,
                       int32_t rope_dim, float theta, int32_t s_max, void *cache_k, void *cache_v, int32_t q_stride,
                       int32_t k_stride, int32_t v_stride, void *stream) {
  if (q_stride == 0) q_stride = n_q * dk;
  if (k_stride == 0) k_stride = n_kv * dk;
  if (v_stride == 0) v_stride = n_kv * dv;
  if (q_stride < n_q * dk || k_stride < n_kv * dk || v_stride < n_kv * dv)
    return fail(SB_E_INVALID_ARG, "sb_rope_append: a token stride is smaller than the token");
  if (T < 0 || n_q < 1 || n_kv < 1 || dk < 2 || dv < 1 || rope_dim < 0 || rope_dim > dk || (rope_dim & 1) || s_max < 1)
    return fail(SB_E_INVALID_ARG, "sb_rope_append: bad shape");
  if (T == 0) return SB_OK;
  if (!q || !k || !v || !seq_of_token || !pos_of_token || !cache_k || !cache_v)
    return fail(SB_E_INVALID_ARG, "sb_rope_append: null pointer");
  const __nv_bfloat16 *kk = static_cast<const __nv_bfloat16 *>(k);
  return launch_rope(static_cast<__nv_bfloat16 *>(q), q_stride, RopeSource{kk, k_stride, dk},
                     RopeSource{kk + rope_dim, k_stride, dk}, RopeSource{static_cast<const __nv_bfloat16 *>(v), v_stride, dv},
                     seq_of_token, pos_of_token, T, n_q, n_kv, dk, dv, rope_dim, theta, s_max, cache_k, cache_v,
                     static_cast<cudaStream_t>(stream));
}

int32_t sb_rope_append_mla(void *q, const void *k_pe, const void *kv, const int32_t *seq_of_token,
                           const int32_t *pos_of_token, int32_t T, int32_t n_heads, int32_t rope_dim, int32_t nope_dim,
                           int32_t dv, float theta, int32_t s_max, void *cache_k, void *cache_v, int32_t q_stride,
                           int32_t k_pe_stride, int32_t kv_stride, void *stream) {
  const int dk = rope_dim + nope_dim;
  if (T < 0 || n_heads < 1 || rope_dim < 0 || (rope_dim & 1) || nope_dim < 0 || dk < 2 || dv < 1 || s_max < 1)
    return fail(SB_E_INVALID_ARG, "sb_rope_append_mla: bad shape");
  if (q_stride < n_heads * dk || k_pe_stride < rope_dim || kv_stride < n_heads * (nope_dim + dv))
    return fail(SB_E_INVALID_ARG, "sb_rope_append_mla: a token stride is smaller than the token");
  if (T == 0) return SB_OK;
  if (!q || !k_pe || !kv || !seq_of_token || !pos_of_token || !cache_k || !cache_v)
    return fail(SB_E_INVALID_ARG, "sb_rope_append_mla: null pointer");
  const __nv_bfloat16 *rest = static_cast<const __nv_bfloat16 *>(kv);
  return launch_rope(static_cast<__nv_bfloat16 *>(q), q_stride,
                     RopeSource{static_cast<const __nv_bfloat16 *>(k_pe), k_pe_stride, 0},
                     RopeSource{rest, kv_stride, nope_dim + dv}, RopeSource{rest + nope_dim, kv_stride, nope_dim + dv},
                     seq_of_token, pos_of_token, T, n_heads, n_heads, dk, dv, rope_dim, theta, s_max, cache_k, cache_v,
                     static_cast<cudaStream_t>(stream));
}

int32_t sb_argmax_rows(const void *logits, int32_t B, int32_t V, int64_t *out, void *stream) {
  if (B < 0 || V < 1 || B > (1 << 24) || V > (1 << 30))
    return fail(SB_E_INVALID_ARG, "sb_argmax_rows: bad shape (B=%d V=%d)", B, V);
  if (B == 0) return SB_OK;
  if (!logits || !out) return fail(SB_E_INVALID_ARG, "sb_argmax_rows: null pointer");
  SB_CUDA_CHECK(launch_pdl(argmax_rows_kernel, dim3(B * kArgmaxCtas), dim3(kArgmaxThreads), 0,
                           static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16 *>(logits), V,
                           V % 8 == 0 && aligned(logits, 16) ? 1 : 0, out));
  SB_LAUNCH_CHECK();
  return SB_OK;
}

size_t sb_attn_decode_workspace_bytes(int32_t B, int32_t n_q, int32_t dv, int32_t n_split) {
  if (B < 0 || n_q < 1 || dv < 1 || n_split < 1) return 0;
  return (size_t)B * n_q * n_split * (dv + 2) * sizeof(float);
}

int32_t sb_attn_decode(const void *q, int32_t q_stride, const void *cache_k, const void *cache_v,
                       const int32_t *seq_lens, int32_t B, int32_t n_q, int32_t n_kv, int32_t dk, int32_t dv,
                       int32_t s_max, float scale, int32_t n_split, void *ws, size_t ws_bytes, void *out,
                       void *stream) {
  if (q_stride == 0) q_stride = n_q * dk;
  if (q_stride < n_q * dk) return fail(SB_E_INVALID_ARG, "sb_attn_decode: q_stride smaller than a token's heads");
  if (B < 0 || n_q < 1 || n_kv < 1 || n_q % n_kv != 0 || s_max < 1 || n_split < 1 || n_split > 256)
    return fail(SB_E_INVALID_ARG, "sb_attn_decode: bad shape");
  if (B == 0) return SB_OK;
  if (!q || !cache_k || !cache_v || !seq_lens || !ws || !out) return fail(SB_E_INVALID_ARG, "sb_attn_decode: null pointer");
  if (!aligned(cache_k, 4) || !aligned(cache_v, 4) || !aligned(ws, 4))
    return fail(SB_E_INVALID_ARG, "sb_attn_decode: cache_k, cache_v, ws must be 4-byte aligned");
  if (ws_bytes < sb_attn_decode_workspace_bytes(B, n_q, dv, n_split))
    return fail(SB_E_WORKSPACE, "sb_attn_decode: workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *qq = static_cast<const __nv_bfloat16 *>(q);
  const __nv_bfloat16 *kk = static_cast<const __nv_bfloat16 *>(cache_k);
  const __nv_bfloat16 *vv = static_cast<const __nv_bfloat16 *>(cache_v);
  float *part = static_cast<float *>(ws);
  __nv_bfloat16 *oo = static_cast<__nv_bfloat16 *>(out);
  if (dk == 128 && dv == 128)
    return launch_attn_decode<128, 128>(qq, q_stride, kk, vv, seq_lens, B, n_q, n_kv, s_max, scale, n_split, part, oo, st);
  if (dk == 192 && dv == 128)
    return launch_attn_decode<192, 128>(qq, q_stride, kk, vv, seq_lens, B, n_q, n_kv, s_max, scale, n_split, part, oo, st);
  if (dk == 64 && dv == 64)
    return launch_attn_decode<64, 64>(qq, q_stride, kk, vv, seq_lens, B, n_q, n_kv, s_max, scale, n_split, part, oo, st);
  return fail(SB_E_UNSUPPORTED, "sb_attn_decode: head dims (%d,%d) not built (128/128, 192/128, 64/64)", dk, dv);
}

}  // extern "C"
