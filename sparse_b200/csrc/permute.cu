// Expert-sorted token permutation: a stable counting sort of the flat
// (token, slot) items by expert id, the gather of activation rows into that
// order, and the row-tile table for the grouped GEMM.
//
// Replaces expand/argsort/gather/bincount of the reference's dispatch
// (utils/eval_core.py:14873-14882) and the re-sort by expert in the local
// executor (utils/eval_core.py:13240-13253).  Integer work is exact: the slot of
// an item is (number of items of smaller expert id) + (number of earlier items
// of the same expert), which is what a stable sort by expert id yields.
//
// Above kFusedMaxItems items four launches: count (per 128-item chunk histogram) -> scan (per-expert
// prefix over chunks, expert offsets, tile table) -> scatter (ranks inside a
// chunk by warp match) -> gather (one warp per output row, 16-byte vectors).
// The gather is the only HBM-heavy part: it reads T*H*2 bytes (re-reads of a
// row hit L2) and writes n_items*H*2.
#include <atomic>

#include "sb_common.cuh"

namespace sb {
namespace {

constexpr int kChunk = 128;          // items per warp-chunk
constexpr int kWarpsPerBlock = 8;
constexpr int kMaxExperts = 256;

__global__ void __launch_bounds__(kWarpsPerBlock * 32)
permute_count_kernel(const int32_t *__restrict__ item_expert, int n_items, int E, int nchunks,
                     int32_t *__restrict__ counts) {
  __shared__ int hist[kWarpsPerBlock][kMaxExperts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = blockIdx.x * kWarpsPerBlock + warp;
  for (int e = lane; e < E; e += 32) hist[warp][e] = 0;
  __syncwarp();
  if (chunk < nchunks) {
#pragma unroll
    for (int r = 0; r < kChunk / 32; ++r) {
      int i = chunk * kChunk + r * 32 + lane;
      if (i < n_items) {
        int e = item_expert[i];
        if (e >= 0 && e < E) atomicAdd(&hist[warp][e], 1);
      }
    }
    __syncwarp();
    for (int e = lane; e < E; e += 32) counts[(size_t)chunk * E + e] = hist[warp][e];
  }
}

// One CTA.  counts[c][e] becomes the number of items of expert e in chunks < c.
__global__ void __launch_bounds__(1024)
permute_scan_kernel(int32_t *__restrict__ counts, int nchunks, int E, int tile_cap, int tile_rows,
                    int32_t *__restrict__ expert_offsets, int32_t *__restrict__ tile_table) {
  __shared__ int total[kMaxExperts];
  __shared__ int offs[kMaxExperts + 1];
  __shared__ int tile_start[kMaxExperts + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = warp; e < E; e += 32) {
    int running = 0;
    for (int c0 = 0; c0 < nchunks; c0 += 32) {
      int c = c0 + lane;
      int v = (c < nchunks) ? counts[(size_t)c * E + e] : 0;
      int incl = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        int o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += o;
      }
      if (c < nchunks) counts[(size_t)c * E + e] = running + incl - v;
      running += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) total[e] = running;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int o = 0, ts = 0;
    for (int e = 0; e < E; ++e) {
      offs[e] = o; tile_start[e] = ts;
      o += total[e];
      ts += (total[e] + tile_rows - 1) / tile_rows;
    }
    offs[E] = o; tile_start[E] = ts;
    tile_table[0] = ts < tile_cap ? ts : tile_cap;
    tile_table[1] = o;          // total rows
    tile_table[2] = tile_rows; tile_table[3] = 0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) expert_offsets[e] = offs[e];
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int nt = tile_start[e + 1] - tile_start[e];
    for (int m = 0; m < nt; ++m) {
      int ti = tile_start[e] + m;
      if (ti >= tile_cap) break;
      int32_t *ent = tile_table + kTileHeaderInts + (size_t)ti * kTileEntryInts;
      int rb = offs[e] + m * tile_rows;
      int re = offs[e + 1] < rb + tile_rows ? offs[e + 1] : rb + tile_rows;
      ent[0] = e; ent[1] = rb; ent[2] = re; ent[3] = 0;
    }
  }
}

__global__ void __launch_bounds__(kWarpsPerBlock * 32)
permute_scatter_kernel(const int32_t *__restrict__ item_expert,
                       const __nv_bfloat16 *__restrict__ item_scale, int n_items, int E,
                       int nchunks, const int32_t *__restrict__ chunk_base,
                       const int32_t *__restrict__ expert_offsets,
                       int32_t *__restrict__ slot_of_item, int32_t *__restrict__ item_of_slot,
                       __nv_bfloat16 *__restrict__ slot_scale) {
  __shared__ int base[kWarpsPerBlock][kMaxExperts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = blockIdx.x * kWarpsPerBlock + warp;
  if (chunk >= nchunks) return;
  for (int e = lane; e < E; e += 32)
    base[warp][e] = expert_offsets[e] + chunk_base[(size_t)chunk * E + e];
  __syncwarp();
#pragma unroll
  for (int r = 0; r < kChunk / 32; ++r) {
    int i = chunk * kChunk + r * 32 + lane;
    int e = -1;
    if (i < n_items) { e = item_expert[i]; if (e < 0 || e >= E) e = -1; }
    unsigned peers = __match_any_sync(0xffffffffu, e);
    int rank = __popc(peers & ((1u << lane) - 1u));
    int slot = -1;
    if (e >= 0) slot = base[warp][e] + rank;
    __syncwarp();
    if (e >= 0 && rank == 0) base[warp][e] += __popc(peers);
    __syncwarp();
    if (i < n_items) {
      slot_of_item[i] = slot;
      if (slot >= 0) {
        item_of_slot[slot] = i;
        if (slot_scale != nullptr) slot_scale[slot] = item_scale[i];
      }
    }
  }
}

// Count, scan and scatter in ONE launch of one cluster, up to kFusedMaxItems items
// (16384 tokens with top-8 routing are 131072).  Bound by latency, not by bytes: the
// routed GEMM waits for it.  Each warp of the CS CTAs owns a contiguous range of
// items and ranks them among its own in one pass (warp match, running counts in
// shared memory), leaving the rank where the slot will go; the CTAs hand each other
// their totals through distributed shared memory; one warp per CTA scans the
// experts; the second pass only adds the base of (expert, warp range).  Loads run
// eight rounds of 32 items ahead, so a round does not wait for its own.  Same result
// as the three-kernel path; the workspace is not touched.
// 16 warps per CTA whatever the item count, so that a few hundred items are one
// round (one warp per 512 items took 9 us for 256, 15 us for 1800); not 32, so that
// a CTA finds room on an SM beside a GEMM CTA of another stream.  Eight CTAs above
// kOneCtaItems: one CTA took 66 us for 30000 items beside a GEMM.
constexpr int kFusedMaxItems = 262144;
constexpr int kFusedWarps = 16;
constexpr int kFusedCtas = 8;
constexpr int kOneCtaItems = 2048;

template <int CS>
__global__ void __launch_bounds__(kFusedWarps * 32)
permute_fused_kernel(const int32_t *__restrict__ item_expert, const __nv_bfloat16 *__restrict__ item_scale,
                     int n_items, int E, int tile_cap, int tile_rows, int32_t *__restrict__ expert_offsets,
                     int32_t *__restrict__ slot_of_item, int32_t *__restrict__ item_of_slot,
                     __nv_bfloat16 *__restrict__ slot_scale, int32_t *__restrict__ tile_table) {
  extern __shared__ int fused_smem[];
  int *hist = fused_smem;                    // [kFusedWarps][E] counts, then bases
  int *offs = hist + kFusedWarps * E;        // [E+1]
  int *tile_start = offs + (E + 1);          // [E+1]
  int *cta_tot = tile_start + (E + 1);       // [CS][E] items of every CTA of the cluster
  constexpr int kBatch = 8;
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t cta = 0;
  if constexpr (CS > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cta));
  constexpr int kWarps = CS * kFusedWarps;
  const int per_warp = ((n_items + kWarps - 1) / kWarps + 31) & ~31;     // items per warp, multiple of 32
  const int begin = min(n_items, ((int)cta * kFusedWarps + warp) * per_warp);
  const int end = min(n_items, begin + per_warp);
  int *mine = hist + warp * E;
  for (int e = lane; e < E; e += 32) mine[e] = 0;
  __syncwarp();
  for (int b0 = begin; b0 < end; b0 += 32 * kBatch) {
    int ev[kBatch];
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      const int i = b0 + r * 32 + lane;
      ev[r] = i < end ? item_expert[i] : -1;
    }
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      const int i = b0 + r * 32 + lane;
      const int e = ev[r] >= 0 && ev[r] < E ? ev[r] : -1;
      if (b0 + r * 32 >= end) break;         // (uniform over the warp)
      const unsigned peers = __match_any_sync(0xffffffffu, e);
      const int rank = __popc(peers & ((1u << lane) - 1u));
      const int before = e >= 0 ? mine[e] : 0;
      __syncwarp();
      if (e >= 0 && rank == 0) mine[e] = before + __popc(peers);
      __syncwarp();
      if (i < end) slot_of_item[i] = before + rank;
    }
  }
  if constexpr (CS > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // this CTA runs
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int c[kFusedWarps], run = 0;
#pragma unroll
    for (int w = 0; w < kFusedWarps; ++w) c[w] = hist[w * E + e];
#pragma unroll
    for (int w = 0; w < kFusedWarps; ++w) { hist[w * E + e] = run; run += c[w]; }
    cta_tot[cta * E + e] = run;
  }
  __syncthreads();
  if constexpr (CS > 1) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int i = threadIdx.x; i < CS * E; i += blockDim.x) {
      const uint32_t to = (uint32_t)(i / E);
      int *place = cta_tot + cta * E + (i - (int)to * E);
      if (to == cta) continue;
      uint32_t addr;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                   : "=r"(addr) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(place))), "r"(to));
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(*place) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (warp == 0) {
    // lane l scans experts 8l .. 8l+7
    constexpr int kPerLane = kMaxExperts / 32;
    int cnt[kPerLane], rows = 0, tiles = 0;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
      const int e = lane * kPerLane + i;
      cnt[i] = 0;
      if (e < E)
        for (int c = 0; c < CS; ++c) cnt[i] += cta_tot[c * E + e];
      rows += cnt[i];
      tiles += (cnt[i] + tile_rows - 1) / tile_rows;
    }
    int o = rows, ts = tiles;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int po = __shfl_up_sync(0xffffffffu, o, off), pt = __shfl_up_sync(0xffffffffu, ts, off);
      if (lane >= off) { o += po; ts += pt; }
    }
    if (lane == 31) {
      offs[E] = o; tile_start[E] = ts;
      if (cta == 0) {
        tile_table[0] = ts < tile_cap ? ts : tile_cap;
        tile_table[1] = o;
        tile_table[2] = tile_rows; tile_table[3] = 0;
      }
    }
    o -= rows; ts -= tiles;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
      const int e = lane * kPerLane + i;
      if (e < E) { offs[e] = o; tile_start[e] = ts; }
      o += cnt[i];
      ts += (cnt[i] + tile_rows - 1) / tile_rows;
    }
  }
  __syncthreads();
  // base of (expert, warp range): the expert's rows, the earlier CTAs' and the earlier warps' items
  for (int i = threadIdx.x; i < kFusedWarps * E; i += blockDim.x) {
    const int e = i % E;
    int base = offs[e];
    for (int c = 0; c < (int)cta; ++c) base += cta_tot[c * E + e];
    hist[i] += base;
  }
  if (cta == 0) {
    for (int e = threadIdx.x; e <= E; e += blockDim.x) expert_offsets[e] = offs[e];
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
      const int nt = tile_start[e + 1] - tile_start[e];
      for (int m = 0; m < nt; ++m) {
        const int ti = tile_start[e] + m;
        if (ti >= tile_cap) break;
        int32_t *ent = tile_table + kTileHeaderInts + (size_t)ti * kTileEntryInts;
        const int rb = offs[e] + m * tile_rows;
        const int re = offs[e + 1] < rb + tile_rows ? offs[e + 1] : rb + tile_rows;
        ent[0] = e; ent[1] = rb; ent[2] = re; ent[3] = 0;
      }
    }
  }
  // The gather's CTAs may take their places from here on, not earlier: waiting for
  // the whole sort they would keep a GEMM CTA of another stream off their SMs.
  pdl_launch_dependents();
  __syncthreads();
  for (int b0 = begin; b0 < end; b0 += 32 * kBatch) {
    int ev[kBatch], rk[kBatch];
    __nv_bfloat16 sv[kBatch];
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      const int i = b0 + r * 32 + lane;
      ev[r] = -1;
      if (i < end) {
        ev[r] = item_expert[i];
        rk[r] = slot_of_item[i];             // this lane wrote it
        if (slot_scale != nullptr) sv[r] = item_scale[i];
      }
    }
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      const int i = b0 + r * 32 + lane;
      if (i < end) {
        const int e = ev[r];
        const int slot = e >= 0 && e < E ? mine[e] + rk[r] : -1;
        slot_of_item[i] = slot;
        if (slot >= 0) {
          item_of_slot[slot] = i;
          if (slot_scale != nullptr) slot_scale[slot] = sv[r];
        }
      }
    }
  }
}

template <int CS>
cudaError_t launch_permute_fused(const int32_t *item_expert, const void *item_scale, int n_items, int E, int tile_cap,
                                 int32_t *expert_offsets, int32_t *slot_of_item, int32_t *item_of_slot,
                                 void *slot_scale, int32_t *tile_table, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CS);
  cfg.blockDim = dim3(kFusedWarps * 32);
  cfg.dynamicSmemBytes = ((size_t)(kFusedWarps + CS) * E + 2 * (size_t)(E + 1)) * sizeof(int);    // at most 27 KB
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CS; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CS > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, permute_fused_kernel<CS>, item_expert, static_cast<const __nv_bfloat16 *>(item_scale),
                            n_items, E, tile_cap, (int)sb_tile_rows(), expert_offsets, slot_of_item, item_of_slot,
                            static_cast<__nv_bfloat16 *>(slot_scale), tile_table);
}

// One warp per output row.
__global__ void __launch_bounds__(256)
permute_gather_kernel(const uint4 *__restrict__ x, const int32_t *__restrict__ item_of_slot,
                      const int32_t *__restrict__ expert_offsets, int E, int items_per_row,
                      int vec_per_row, uint4 *__restrict__ out_rows) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int n_rows = expert_offsets[E];
  const int warps_total = gridDim.x * (blockDim.x >> 5);
  for (int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); slot < n_rows;
       slot += warps_total) {
    int src = item_of_slot[slot] / items_per_row;
    const uint4 *s = x + (size_t)src * vec_per_row;
    uint4 *d = out_rows + (size_t)slot * vec_per_row;
    for (int v = lane; v < vec_per_row; v += 32) d[v] = __ldg(s + v);
  }
}

}  // namespace

static inline int num_chunks(int n_items) { return (n_items + kChunk - 1) / kChunk; }

int32_t launch_permute(const void *x, const int32_t *item_expert, const void *item_scale,
                       int n_items, int items_per_row, int H, int E, void *ws, size_t ws_bytes,
                       void *out_rows, int32_t *expert_offsets, int32_t *slot_of_item,
                       int32_t *item_of_slot, void *slot_scale, int32_t *tile_table,
                       cudaStream_t stream) {
  if (n_items < 0 || items_per_row < 1 || H <= 0 || H % 8 != 0 || E < 1 || E > kMaxExperts)
    return fail(SB_E_INVALID_ARG, "sb_permute: need H%%8==0, 1<=E<=256, items_per_row>=1 (n=%d H=%d E=%d)",
                n_items, H, E);
  if (!expert_offsets || !tile_table || !ws)
    return fail(SB_E_INVALID_ARG, "sb_permute: null pointer");
  // out_rows == NULL: sort only, no row gather (x may then be NULL as well)
  if (n_items > 0 && (!item_expert || !slot_of_item || !item_of_slot || (out_rows && !x)))
    return fail(SB_E_INVALID_ARG, "sb_permute: null pointer");
  if ((slot_scale != nullptr) != (item_scale != nullptr))
    return fail(SB_E_INVALID_ARG, "sb_permute: item_scale and slot_scale go together");
  if (ws_bytes < sb_permute_workspace_bytes(n_items, E))
    return fail(SB_E_WORKSPACE, "sb_permute: workspace %zu < %zu bytes", ws_bytes,
                sb_permute_workspace_bytes(n_items, E));
  if (!aligned(x, 16) || !aligned(out_rows, 16))
    return fail(SB_E_INVALID_ARG, "sb_permute: rows must be 16-byte aligned");
  const int nchunks = num_chunks(n_items);
  int32_t *counts = static_cast<int32_t *>(ws);
  const int tile_cap = n_items / SB_TILE_M + E;
  if (n_items > 0 && n_items <= kFusedMaxItems) {
    const auto sort = n_items > kOneCtaItems ? launch_permute_fused<kFusedCtas> : launch_permute_fused<1>;
    SB_CUDA_CHECK(sort(item_expert, item_scale, n_items, E, tile_cap, expert_offsets, slot_of_item, item_of_slot,
                       slot_scale, tile_table, stream));
    SB_LAUNCH_CHECK();
    if (out_rows != nullptr) {
      int gblocks = (n_items + 7) / 8;
      const int max_blocks = sb_device_sm_count() * 8;
      if (gblocks > max_blocks) gblocks = max_blocks;
      SB_CUDA_CHECK(launch_pdl(permute_gather_kernel, dim3(gblocks), dim3(256), 0, stream,
                               static_cast<const uint4 *>(x), static_cast<const int32_t *>(item_of_slot),
                               static_cast<const int32_t *>(expert_offsets), E, items_per_row, H / 8,
                               static_cast<uint4 *>(out_rows)));
      SB_LAUNCH_CHECK();
    }
    return SB_OK;
  }
  if (nchunks > 0) {
    int blocks = (nchunks + kWarpsPerBlock - 1) / kWarpsPerBlock;
    permute_count_kernel<<<blocks, kWarpsPerBlock * 32, 0, stream>>>(item_expert, n_items, E,
                                                                    nchunks, counts);
    SB_LAUNCH_CHECK();
  }
  permute_scan_kernel<<<1, 1024, 0, stream>>>(counts, nchunks, E, tile_cap, sb_tile_rows(), expert_offsets,
                                              tile_table);
  SB_LAUNCH_CHECK();
  if (nchunks > 0) {
    int blocks = (nchunks + kWarpsPerBlock - 1) / kWarpsPerBlock;
    permute_scatter_kernel<<<blocks, kWarpsPerBlock * 32, 0, stream>>>(
        item_expert, static_cast<const __nv_bfloat16 *>(item_scale), n_items, E, nchunks, counts,
        expert_offsets, slot_of_item, item_of_slot, static_cast<__nv_bfloat16 *>(slot_scale));
    SB_LAUNCH_CHECK();
    if (out_rows != nullptr) {
      int rows_per_block = 8;
      int gblocks = (n_items + rows_per_block - 1) / rows_per_block;
      int max_blocks = sb_device_sm_count() * 8;
      if (gblocks > max_blocks) gblocks = max_blocks;
      SB_CUDA_CHECK(launch_pdl(permute_gather_kernel, dim3(gblocks), dim3(256), 0, stream,
                               static_cast<const uint4 *>(x), static_cast<const int32_t *>(item_of_slot),
                               static_cast<const int32_t *>(expert_offsets), E, items_per_row, H / 8,
                               static_cast<uint4 *>(out_rows)));
      SB_LAUNCH_CHECK();
    }
  }
  return SB_OK;
}

}  // namespace sb

// ---- sb_permute_noalloc: the same sort with library-owned scratch -----------------
//
// Scratch for the per-chunk histograms of sb_permute, reserved in the library's
// own device image instead of being passed in.  512 KiB; every GPU that loads
// the library carries it until the process exits.
constexpr int kStaticScratchInts = 131072;
static __device__ __align__(256) int32_t g_permute_scratch[kStaticScratchInts];

// Device address of g_permute_scratch per device ordinal (0 = not looked up yet).
// In host code the symbol's name is only a handle; the address a kernel can use
// has to be asked for, with that device current.
// Two host threads making the first call on a device both store the same value;
// the atomic makes that a defined (relaxed) access instead of a data race.
static std::atomic<int32_t *> g_permute_scratch_addr[64];

extern "C" int32_t sb_permute_noalloc(const void *x, const int32_t *item_expert,
                                      const void *item_scale, int32_t n_items,
                                      int32_t items_per_row, int32_t H, int32_t E, void *out_rows,
                                      int32_t *expert_offsets, int32_t *slot_of_item,
                                      int32_t *item_of_slot, void *slot_scale,
                                      int32_t *tile_table, void *stream) {
  if (n_items < 0 || E < 1 || E > sb::kMaxExperts)
    return sb::fail(SB_E_INVALID_ARG, "sb_permute_noalloc: need n_items>=0 and 1<=E<=256 (n=%d E=%d)",
                    n_items, E);
  const size_t need_ints = (size_t)sb::num_chunks(n_items) * (size_t)E;
  if (need_ints > (size_t)kStaticScratchInts)
    return sb::fail(SB_E_WORKSPACE,
                    "sb_permute_noalloc: %d items over %d experts need %zu scratch ints, the built-in "
                    "scratch holds %d (ceil(n_items/128)*E must not exceed it); use sb_permute with a "
                    "caller-provided workspace",
                    n_items, E, need_ints, kStaticScratchInts);
  int dev = -1;
  SB_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return sb::fail(SB_E_UNSUPPORTED, "sb_permute_noalloc: device ordinal %d", dev);
  int32_t *scratch = g_permute_scratch_addr[dev].load(std::memory_order_relaxed);
  if (scratch == nullptr) {
    int32_t *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_permute_scratch);
    if (e != cudaSuccess || p == nullptr)
      return sb::fail(SB_E_CUDA, "sb_permute_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
                      cudaGetErrorString(e));
    g_permute_scratch_addr[dev].store(p, std::memory_order_relaxed);
    scratch = p;
  }
  // Nothing in the scratch has to start at zero: the count pass overwrites every
  // histogram cell the later passes read, so stale contents of an earlier call
  // are never observed.
  return sb::launch_permute(x, item_expert, item_scale, n_items, items_per_row, H, E,
                            scratch,
                            (size_t)kStaticScratchInts * sizeof(int32_t), out_rows, expert_offsets,
                            slot_of_item, item_of_slot, slot_scale, tile_table,
                            static_cast<cudaStream_t>(stream));
}

extern "C" size_t sb_permute_workspace_bytes(int32_t n_items, int32_t E) {
  size_t n = (size_t)sb::num_chunks(n_items < 0 ? 0 : n_items) * (size_t)(E < 1 ? 1 : E) * sizeof(int32_t);
  return n < 256 ? 256 : ((n + 255) / 256) * 256;
}

extern "C" size_t sb_tile_table_ints(int32_t n_items, int32_t E) {
  size_t tiles = (size_t)(n_items < 0 ? 0 : n_items) / SB_TILE_M + (size_t)(E < 1 ? 1 : E);
  return sb::kTileHeaderInts + tiles * sb::kTileEntryInts;
}
