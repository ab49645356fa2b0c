// Token permutation: a STABLE counting sort of the T*k (token,slot) pairs by expert id, the tile list
// that the grouped GEMMs walk, and the row gather + 1x128 e4m3 activation quantisation.
//
// The sort reproduces the reference device kernel's per-expert `nonzero` (my_ops/fusedMoE.pl:737-755):
// inside one expert the flat pair ids t*k+j ascend.  It is deterministic (no atomics decide order):
//   hist    : chunk c (1024 pairs) counts its pairs per expert            -> chunk_cnt[c][e]
//   scan    : per expert a running sum over chunks, then a scan over experts -> chunk_base, offsets
//   scatter : position = offsets[e] + chunk_base[c][e] + (pairs of e in earlier warps of the chunk)
//             + (pairs of e in lower lanes of the warp)
// For P <= 1024 all three steps run in one single-CTA kernel, up to 8192 in one cluster of CTAs.
#include "internal.h"

namespace {

constexpr int kChunk = 1024;  // pairs per CTA (32 warps)
constexpr int kMaxE = 1024;
constexpr int kMaxDevices = 64;  // per-device caches below are indexed by the CUDA device ordinal

// Per-warp histogram of this chunk in shared memory: wh[w*E + e].  Returns the pair's expert (or -1)
// and its rank among equal experts in lower lanes of its warp.
__device__ __forceinline__ int chunk_hist(const int32_t* ids, int64_t P, int E, int64_t p,
                                          int* wh, int& rank_in_warp, int32_t* status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < 32 * E; i += blockDim.x) wh[i] = 0;
  __syncthreads();
  int e = -1;
  if (p < P) {
    e = ids[p];
    if (e < 0 || e >= E) {
      e = -1;
      if (status) atomicOr(status, B200MOE_STATUS_BAD_EXPERT);
    }
  }
  unsigned peers = __match_any_sync(0xffffffffu, e);
  rank_in_warp = __popc(peers & ((1u << lane) - 1u));
  if (e >= 0 && rank_in_warp == 0) wh[warp * E + e] = __popc(peers);
  __syncthreads();
  return e;
}

__global__ void __launch_bounds__(kChunk)
permute_hist_kernel(const int32_t* ids, int64_t P, int E, int32_t* __restrict__ chunk_cnt,
                    int32_t* status) {
  pdl_begin();
  extern __shared__ int wh[];
  int rank;
  chunk_hist(ids, P, E, (int64_t)blockIdx.x * kChunk + threadIdx.x, wh, rank, status);
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int s = 0;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) s += wh[w * E + e];
    chunk_cnt[(int64_t)blockIdx.x * E + e] = s;
  }
}

// exclusive scan of the threads' counts (thread t < E: expert t) by one CTA of 1024 threads; result in offs[0..E], valid
// after the next __syncthreads
__device__ __forceinline__ void block_exclusive_scan(int my, int E, int32_t* offs, int* tmp /* [32] */) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int v = t < E ? my : 0;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += u;
  }
  __syncthreads();  // tmp of the scan before is read
  if (lane == 31) tmp[warp] = v;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += tmp[w];
  if (t < E) offs[t + 1] = before + v;
  if (t == 0) offs[0] = 0;
}

// what the grouped GEMMs walk, written by one CTA from the expert offsets in shared memory: {expert, first row} per 128
// rows of an expert, their number, and zeros in the counters of shared tiles
__device__ __forceinline__ void write_mtiles(const int* soffs, int E, int* toffs, int* tmp, int32_t* __restrict__ mtiles,
                                             int32_t* __restrict__ num_mtiles, int max_mtiles, int32_t* split_cnt) {
  moe_clear_counters(split_cnt);
  const int t = threadIdx.x;
  const int b = t < E ? soffs[t] : 0;
  const int n = t < E ? (soffs[t + 1] - b + kTileM - 1) / kTileM : 0;
  block_exclusive_scan(n, E, toffs, tmp);
  __syncthreads();
  for (int i = 0; i < n && toffs[t] + i < max_mtiles; ++i) {
    mtiles[2 * (toffs[t] + i)] = t;
    mtiles[2 * (toffs[t] + i) + 1] = b + i * kTileM;
  }
  if (t == 0) *num_mtiles = min(toffs[E], max_mtiles);
}

__global__ void __launch_bounds__(kChunk)
permute_scan_kernel(int32_t* __restrict__ chunk_cnt, int nchunks, int E, int32_t* __restrict__ offsets,
                    int32_t* __restrict__ mtiles, int32_t* __restrict__ num_mtiles, int max_mtiles, int32_t* split_cnt) {
  pdl_begin();
  __shared__ int tmp[32], soffs[kMaxE + 1], toffs[kMaxE + 1];
  int total = 0;
  if ((int)threadIdx.x < E) {
    // eight counts are requested before the first is used: walked one by one, every chunk costs an L2 round trip
    // (64 chunks of a 65536-pair batch: 20 us for this one block)
    for (int c0 = 0; c0 < nchunks; c0 += 8) {
      int v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = c0 + i < nchunks ? chunk_cnt[(int64_t)(c0 + i) * E + threadIdx.x] : 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (c0 + i < nchunks) chunk_cnt[(int64_t)(c0 + i) * E + threadIdx.x] = total;  // becomes chunk_base
        total += v[i];
      }
    }
  }
  block_exclusive_scan(total, E, soffs, tmp);
  __syncthreads();
  for (int i = threadIdx.x; i <= E; i += blockDim.x) offsets[i] = soffs[i];
  if (mtiles) write_mtiles(soffs, E, toffs, tmp, mtiles, num_mtiles, max_mtiles, split_cnt);
}

__global__ void __launch_bounds__(kChunk)
permute_scatter_kernel(const int32_t* ids, int64_t P, int E,
                       const int32_t* chunk_base, const int32_t* offsets,
                       int32_t* __restrict__ sorted_pair, int32_t* __restrict__ pos_of) {
  pdl_begin();
  extern __shared__ int wh[];
  int rank;
  const int64_t p = (int64_t)blockIdx.x * kChunk + threadIdx.x;
  int e = chunk_hist(ids, P, E, p, wh, rank, nullptr);
  for (int x = threadIdx.x; x < E; x += blockDim.x) {  // warp histogram -> exclusive prefix over warps
    int s = 0;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) {
      int v = wh[w * E + x];
      wh[w * E + x] = s;
      s += v;
    }
  }
  __syncthreads();
  int pos = -1;
  if (e >= 0) {
    pos = offsets[e] + chunk_base[(int64_t)blockIdx.x * E + e] + wh[(threadIdx.x >> 5) * E + e] + rank;
    sorted_pair[pos] = (int32_t)p;
  }
  if (pos_of && p < P) pos_of[p] = pos;
  // Pairs whose id was out of range have no position: the tail [offsets[E], P) is filled with -1 so that no consumer
  // ever indexes with an unwritten entry (valid positions all lie below offsets[E], so this does not race with them).
  if (p < P && p >= offsets[E]) sorted_pair[p] = -1;
}

// P <= 1024: histogram, scan and scatter in one CTA
__global__ void __launch_bounds__(kChunk)
permute_small_kernel(const int32_t* ids, int64_t P, int E, int32_t* __restrict__ offsets,
                     int32_t* __restrict__ sorted_pair, int32_t* status, int32_t* __restrict__ mtiles,
                     int32_t* __restrict__ num_mtiles, int max_mtiles, int32_t* __restrict__ pos_of,
                     int32_t* split_cnt) {
  pdl_begin();
  extern __shared__ int wh[];
  __shared__ int tmp[32], soffs[kMaxE + 1], toffs[kMaxE + 1];
  int rank;
  int e = chunk_hist(ids, P, E, threadIdx.x, wh, rank, status);
  int total = 0;
  if ((int)threadIdx.x < E) {
#pragma unroll 8
    for (int w = 0; w < 32; ++w) {
      int v = wh[w * E + threadIdx.x];
      wh[w * E + threadIdx.x] = total;
      total += v;
    }
  }
  block_exclusive_scan(total, E, soffs, tmp);
  __syncthreads();
  for (int i = threadIdx.x; i <= E; i += blockDim.x) offsets[i] = soffs[i];
  int pos = -1;
  if (e >= 0) {
    pos = soffs[e] + wh[(threadIdx.x >> 5) * E + e] + rank;
    sorted_pair[pos] = (int32_t)threadIdx.x;
  }
  if (pos_of && (int64_t)threadIdx.x < P) pos_of[threadIdx.x] = pos;
  if ((int64_t)threadIdx.x < P && (int)threadIdx.x >= soffs[E]) sorted_pair[threadIdx.x] = -1;  // dropped pairs: see above
  if (mtiles) write_mtiles(soffs, E, toffs, tmp, mtiles, num_mtiles, max_mtiles, split_cnt);
}

// 1024 < P <= 8192: the same with one cluster, a chunk of 1024 pairs per CTA; the CTAs read one another's counts through
// distributed shared memory (6216 pairs: 7 us for the one launch, 12.7 us for the general form's three and 3.5 for the
// list)
constexpr int kMaxCluster = 8;  // portable cluster size
__global__ void __launch_bounds__(kChunk)
permute_cluster_kernel(const int32_t* ids, int64_t P, int E, int32_t* __restrict__ offsets,
                       int32_t* __restrict__ sorted_pair, int32_t* status, int32_t* __restrict__ mtiles,
                       int32_t* __restrict__ num_mtiles, int max_mtiles, int32_t* __restrict__ pos_of, int32_t* split_cnt) {
  pdl_begin();
  extern __shared__ int wh[];
  __shared__ int tmp[32], soffs[kMaxE + 1], toffs[kMaxE + 1], cnt[kMaxE], base[kMaxE];
  const int me = blockIdx.y, chunks = gridDim.y, t = threadIdx.x;
  const int64_t p = (int64_t)me * kChunk + t;
  int rank;
  const int e = chunk_hist(ids, P, E, p, wh, rank, status);
  if (t < E) {
    int total = 0;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) {
      int v = wh[w * E + t];
      wh[w * E + t] = total;
      total += v;
    }
    cnt[t] = total;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  int total = 0;
  if (t < E) {
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(cnt + t);
    int before = 0;
    for (int c = 0; c < chunks; ++c) {
      uint32_t remote;
      int v;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(c));
      asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
      if (c < me) before += v;
      total += v;
    }
    base[t] = before;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // done with the others' counts
  block_exclusive_scan(total, E, soffs, tmp);
  __syncthreads();
  int pos = -1;
  if (e >= 0) {
    pos = soffs[e] + base[e] + wh[(t >> 5) * E + e] + rank;
    sorted_pair[pos] = (int32_t)p;
  }
  if (p < P) {
    if (pos_of) pos_of[p] = pos;
    if (p >= soffs[E]) sorted_pair[p] = -1;  // dropped pairs: see above
  }
  if (me == 0) {
    for (int i = t; i <= E; i += blockDim.x) offsets[i] = soffs[i];
    if (mtiles) write_mtiles(soffs, E, toffs, tmp, mtiles, num_mtiles, max_mtiles, split_cnt);
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while its counts are read
}

__global__ void gather_scatter_index_kernel(int32_t* __restrict__ gather_index,
                                            int32_t* __restrict__ scatter_index,
                                            int32_t* __restrict__ num_per_expert,
                                            const int32_t* sorted_pair,
                                            const int32_t* offsets, int64_t T, int k) {
  pdl_begin();
  const int e = blockIdx.x;
  const int b = offsets[e], n = offsets[e + 1] - b;
  if (threadIdx.x == 0) num_per_expert[e] = n;
  for (int i = threadIdx.x; i < n && i < T; i += blockDim.x) {
    int pr = sorted_pair[b + i];
    scatter_index[(int64_t)e * T + i] = pr;
    gather_index[(int64_t)e * T + i] = pr / k;
  }
}

// ---- row gather + 1x128 e4m3 quantisation -------------------------------------------------------
// A warp owns `cpw` consecutive 256-column chunks of one output row: a lane owns 8 consecutive bf16 (one 16-byte
// load), 16 lanes own one 128-column group.  The groups of a row are independent, so with few rows (decode sizes)
// they are spread over warps (cpw = 1: the kernel is one load-and-store deep instead of H/256); with many rows one
// warp walks a whole row (fewer blocks, the row's gather index read once).
__global__ void __launch_bounds__(256)
quant_rows_kernel(uint8_t* __restrict__ q, float* __restrict__ s_t, int64_t ld,
                  const __nv_bfloat16* x, const int32_t* row_map, int div,
                  int64_t rows, int H, int cpw, int warps_per_row, MoeIdentityLists lists) {
  pdl_begin();
  if (lists.offsets && blockIdx.x == 0) moe_write_identity_lists(lists, (int)rows);
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int64_t r = w / warps_per_row;
  if (r >= rows) return;
  const int c_begin = (int)(w - r * warps_per_row) * cpw * 256;
  if (row_map && row_map[r] < 0) return;  // position of a dropped pair (id out of range): no row
  const int64_t src = row_map ? (int64_t)(row_map[r] / div) : r;
  const __nv_bfloat16* xr = x + src * H;
  const int c_end = min(c_begin + cpw * 256, H);
  // Four 256-column chunks at a time, their loads issued before the first is used: taken one by one, every chunk of a
  // row costs the warp a whole round trip to L2 (Qwen3 shape, 65536 rows of 2048: 73 us for 400 MB).
  for (int c0 = c_begin; c0 < c_end; c0 += 4 * 256) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = c0 + u * 256 + lane * 8;
      raw[u] = c < c_end ? *reinterpret_cast<const uint4*>(xr + c) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = c0 + u * 256 + lane * 8;
      if (c0 + u * 256 >= c_end) break;  // uniform over the warp
      float v[8];
      float amax = 0.f;
      const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 f = __bfloat1622float2(b2[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      if (c < c_end) {
        amax = fmaxf(amax, kAmaxFloor);
        const float inv = kFp8Max / amax;
        uint2 out;
        out.x = moe_f32x4_to_e4m3x4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv);
        out.y = moe_f32x4_to_e4m3x4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv);
        *reinterpret_cast<uint2*>(q + r * H + c) = out;
        if ((lane & 15) == 0) s_t[(int64_t)(c >> 7) * ld + r] = amax / kFp8Max;
      }
    }
  }
}

// The routed rows of a layer, token by token: a token is read and quantised ONCE and its e4m3 bytes are stored to the
// positions of its k (token,slot) pairs (pos_of, the inverse of the permutation; -1 = dropped).  Walking the sorted rows
// instead reads and converts every token k times: Qwen3 shape, 8192 tokens x 8 slots: 72 us, bound by the conversions
// and k-fold reads, for 134 MB of output that the copy bandwidth writes in 20 us; now 31 us.  DeepSeek shape, 2048
// tokens 62 -> 28 us, Mixtral shape, 4096 tokens 21 -> 13 us.
// A lane owns 16 consecutive columns (eight lanes one 128-column group), so a store instruction puts down 512 bytes of a
// row; a warp takes `cpw` 512-column chunks of a token, their loads issued together.
constexpr int QT_CPW = 2;
__global__ void __launch_bounds__(256)
quant_tokens_kernel(uint8_t* __restrict__ q, float* __restrict__ s_t, int64_t ld, const __nv_bfloat16* x,
                    const int32_t* pos_of, int64_t T, int k, int H, int cpw, int warps_per_tok,
                    float* __restrict__ acc32) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int64_t t = w / warps_per_tok;
  if (t >= T) return;  // uniform over the warp
  const int c0 = (int)(w - t * warps_per_tok) * cpw * 512 + lane * 16;
  uint4 raw[QT_CPW][2];
#pragma unroll
  for (int u = 0; u < QT_CPW; ++u) {
    const int c = c0 + u * 512;
    const bool on = u < cpw && c < H;
    raw[u][0] = on ? *reinterpret_cast<const uint4*>(x + t * H + c) : make_uint4(0, 0, 0, 0);
    raw[u][1] = on ? *reinterpret_cast<const uint4*>(x + t * H + c + 8) : make_uint4(0, 0, 0, 0);
  }
  if (acc32) {  // the token's fp32 row of the fused combine starts from zero
#pragma unroll
    for (int u = 0; u < QT_CPW; ++u)
      if (u < cpw && c0 + u * 512 < H)
#pragma unroll
        for (int i = 0; i < 4; ++i) reinterpret_cast<float4*>(acc32 + t * H + c0 + u * 512)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  int32_t my_pos = lane < k ? pos_of[t * k + lane] : -1;
  uint4 out[QT_CPW];
  float sc[QT_CPW];
#pragma unroll
  for (int u = 0; u < QT_CPW; ++u) {
    float v[16], amax = 0.f;
    const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&raw[u][0]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 f = __bfloat1622float2(b2[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
      amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    amax = fmaxf(amax, kAmaxFloor);
    const float inv = kFp8Max / amax;
    sc[u] = amax / kFp8Max;
    out[u].x = moe_f32x4_to_e4m3x4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv);
    out[u].y = moe_f32x4_to_e4m3x4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv);
    out[u].z = moe_f32x4_to_e4m3x4(v[8] * inv, v[9] * inv, v[10] * inv, v[11] * inv);
    out[u].w = moe_f32x4_to_e4m3x4(v[12] * inv, v[13] * inv, v[14] * inv, v[15] * inv);
  }
  for (int j0 = 0; j0 < k; j0 += 32) {
    if (j0 > 0) my_pos = j0 + lane < k ? pos_of[t * k + j0 + lane] : -1;
    const int n = min(32, k - j0);
    for (int j = 0; j < n; ++j) {
      const int64_t p = __shfl_sync(0xffffffffu, my_pos, j);
      if (p < 0) continue;
#pragma unroll
      for (int u = 0; u < QT_CPW; ++u) {
        const int c = c0 + u * 512;
        if (u < cpw && c < H) {
          *reinterpret_cast<uint4*>(q + p * H + c) = out[u];
          if ((lane & 7) == 0) s_t[(int64_t)(c >> 7) * ld + p] = sc[u];
        }
      }
    }
  }
}

}  // namespace

extern "C" size_t b200moe_permute_scratch_ints(int64_t P, int64_t E) {
  if (P <= kChunk) return 1;
  return (size_t)((P + kChunk - 1) / kChunk) * (size_t)E;
}

// b200moe_permute; with `pos_of` != NULL the inverse map too (pos_of[pair] = its position, -1 = dropped); with `mtiles` != NULL the
// GEMMs' m-tile list too
int moe_permute_impl(int32_t* sorted_pair, int32_t* expert_offsets, const int32_t* ids, int64_t T, int64_t k, int64_t E,
                     int32_t* scratch, int32_t* status, int32_t* pos_of, int32_t* mtiles, int32_t* num_mtiles,
                     int max_mtiles, int32_t* split_cnt, void* stream) {
  MOE_CHECK_ARG(sorted_pair && expert_offsets && ids && T >= 0 && k > 0 && E > 0);
  const int64_t P = T * k;
  MOE_CHECK_SHAPE(E <= kMaxE && P < (1 << 24));
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = (size_t)32 * E * sizeof(int);
  // The dynamic shared-memory cap of a kernel is a per-DEVICE attribute: set it once on every device that comes here.
  static bool attr_done[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200MOE_EDRIVER;
  if (!attr_done[dev]) {
    cudaFuncSetAttribute(permute_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * kMaxE * 4);
    cudaFuncSetAttribute(permute_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * kMaxE * 4);
    cudaFuncSetAttribute(permute_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * kMaxE * 4);
    cudaFuncSetAttribute(permute_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * kMaxE * 4);
    attr_done[dev] = true;
  }
  if (P <= kChunk) {
    return moe_launch(permute_small_kernel, 1, kChunk, smem, st, ids, P, (int)E, expert_offsets, sorted_pair, status, mtiles,
                      num_mtiles, max_mtiles, pos_of, split_cnt);
  }
  MOE_CHECK_ARG(scratch);
  const int nchunks = (int)((P + kChunk - 1) / kChunk);
  if (nchunks <= kMaxCluster)
    return moe_launch_as(true, nchunks, permute_cluster_kernel, dim3(1, nchunks), kChunk, smem, st, ids, P, (int)E,
                              expert_offsets, sorted_pair, status, mtiles, num_mtiles, max_mtiles, pos_of, split_cnt);
  int rc = moe_launch(permute_hist_kernel, nchunks, kChunk, smem, st, ids, P, (int)E, scratch, status);
  if (!rc) rc = moe_launch(permute_scan_kernel, 1, kChunk, 0, st, scratch, nchunks, (int)E, expert_offsets, mtiles, num_mtiles,
                            max_mtiles, split_cnt);
  if (!rc)
    rc = moe_launch(permute_scatter_kernel, nchunks, kChunk, smem, st, ids, P, (int)E, scratch, expert_offsets, sorted_pair,
                    pos_of);
  return rc;
}

extern "C" int b200moe_permute(int32_t* sorted_pair, int32_t* expert_offsets, const int32_t* ids, int64_t T,
                               int64_t k, int64_t E, int32_t* scratch, int32_t* status, void* stream) {
  return moe_permute_impl(sorted_pair, expert_offsets, ids, T, k, E, scratch, status, nullptr, nullptr, nullptr, 0,
                          nullptr, stream);
}

extern "C" int b200moe_gather_scatter_index(int32_t* gather_index, int32_t* scatter_index,
                                            int32_t* num_per_expert, const int32_t* sorted_pair,
                                            const int32_t* expert_offsets, int64_t T, int64_t k, int64_t E,
                                            void* stream) {
  MOE_CHECK_ARG(gather_index && scatter_index && num_per_expert && sorted_pair && expert_offsets);
  MOE_CHECK_ARG(T >= 0 && k > 0 && E > 0);
  if (T == 0) return B200MOE_OK;
  return moe_launch(gather_scatter_index_kernel, (unsigned)E, 256, 0, (cudaStream_t)stream, gather_index, scatter_index,
                    num_per_expert, sorted_pair, expert_offsets, T, (int)k);
}

namespace {
int launch_quant_rows(uint8_t* q, float* s_t, int64_t ld, const void* x, const int32_t* row_map, int64_t div, int64_t rows,
                      int64_t H, const MoeIdentityLists& lists, cudaStream_t st) {
  const int chunks = (int)((H + 255) / 256);
  const int cpw = rows >= 2048 ? chunks : 1;
  const int warps_per_row = (chunks + cpw - 1) / cpw;
  return moe_launch(quant_rows_kernel, (unsigned)((rows * warps_per_row + 7) / 8), 256, 0, st, q, s_t, ld,
                    reinterpret_cast<const __nv_bfloat16*>(x), row_map, (int)div, rows, (int)H, cpw, warps_per_row, lists);
}
}  // namespace

extern "C" int b200moe_quant_rows(uint8_t* q, float* s_t, int64_t ld, const void* x, const int32_t* row_map,
                                  int64_t div, int64_t rows, int64_t H, void* stream) {
  MOE_CHECK_ARG(q && s_t && x && rows >= 0 && H > 0 && div > 0 && ld >= rows);
  MOE_CHECK_SHAPE(H % kBlock == 0);
  if (!moe_aligned16(x) || !moe_aligned16(q)) return B200MOE_EALIGN;
  if (rows == 0) return B200MOE_OK;
  return launch_quant_rows(q, s_t, ld, x, row_map, div, rows, H, MoeIdentityLists{}, (cudaStream_t)stream);
}

int moe_quant_identity(uint8_t* q, float* s_t, int64_t ld, const void* x, int64_t rows, int64_t H,
                       const MoeIdentityLists& lists, cudaStream_t st) {
  return launch_quant_rows(q, s_t, ld, x, nullptr, 1, rows, H, lists, st);
}

int moe_quant_tokens(uint8_t* q, float* s_t, int64_t ld, const void* x, const int32_t* pos_of, int64_t T, int64_t k,
                     int64_t H, float* acc32, cudaStream_t st) {
  const int64_t chunks = (H + 511) / 512;
  // two chunks per warp once that still leaves every SM its full set of warps
  const int cpw = T * chunks >= (int64_t)QT_CPW * 64 * moe_device_sm_count() ? QT_CPW : 1;
  const int64_t wpt = (chunks + cpw - 1) / cpw;
  return moe_launch(quant_tokens_kernel, (unsigned)((T * wpt + 7) / 8), 256, 0, st, q, s_t, ld,
                    reinterpret_cast<const __nv_bfloat16*>(x), pos_of, T, (int)k, (int)H, cpw, (int)wpt, acc32);
}

// ---- permutation without caller-provided scratch ---------------------------------------------------
// For hosts that must not (or cannot) allocate device memory around the call - a serving process whose
// memory pool is fixed at start-up, a plugin that is only handed input and output buffers.  The chunk-count table that b200moe_permute takes from the caller lives here in
// a fixed array inside the library image instead; every GPU that loads the library holds these 256 KB until
// the process exits.
constexpr size_t kStaticScratchInts = 64 * 1024;  // 256 KB: e.g. 65536 pairs x 1024 experts, 262144 pairs x 256
static __device__ __align__(256) int32_t g_permute_scratch[kStaticScratchInts];

namespace {
// In host code `g_permute_scratch` is only a handle for the runtime, not a device address, so the address the
// kernels need is looked up once per device, with that device current.
int static_scratch_ptr(int32_t** out) {
  static int32_t* ptrs[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return B200MOE_ESHAPE;
  if (!ptrs[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_permute_scratch);
    if (e != cudaSuccess) return (int)e;
    ptrs[dev] = reinterpret_cast<int32_t*>(p);
  }
  *out = ptrs[dev];
  return B200MOE_OK;
}
}  // namespace

extern "C" size_t b200moe_permute_static_max_scratch_ints(void) { return kStaticScratchInts; }

extern "C" int b200moe_permute_static(int32_t* sorted_pair, int32_t* expert_offsets, const int32_t* ids,
                                      int64_t T, int64_t k, int64_t E, int32_t* status, void* stream) {
  MOE_CHECK_ARG(T >= 0 && k > 0 && E > 0);
  if (b200moe_permute_scratch_ints(T * k, E) > kStaticScratchInts) return B200MOE_ESHAPE;
  int32_t* scratch = nullptr;
  int rc = static_scratch_ptr(&scratch);
  if (rc != B200MOE_OK) return rc;
  // The table is written in full by the histogram step before it is read, so nothing has to be cleared.
  return b200moe_permute(sorted_pair, expert_offsets, ids, T, k, E, scratch, status, stream);
}
