// Routing kernels: plain / grouped top-k on given scores, the fused score->select->normalise chain,
// and the router GEMM.  One warp owns one row; element e of the row lives in lane e%32, register e/32,
// so loads are coalesced and every selection step is a register scan plus two warp reductions.
//
// Tie rule everywhere: among equal values the LOWEST index wins (the reference leaves tie order open:
// aten::topk on its CPU path and an index-perturbation on its device path, native_ops/Topk.pl:82-100).
#include <float.h>
#include <limits.h>
#include <math.h>

#include "internal.h"

namespace {

constexpr int kWarpsPerBlock = 4;

__device__ __forceinline__ void warp_argmax(float& v, int& idx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float ov = __shfl_xor_sync(0xffffffffu, v, o);
    int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) {
      v = ov;
      idx = oi;
    }
  }
}

// A float as an unsigned number of the same order (-0 counts as +0, NaN above everything), so that a warp's maximum is
// one redux instruction.
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t b = __float_as_uint(v + 0.0f);
  return b ^ ((int32_t)b < 0 ? 0xffffffffu : 0x80000000u);
}

// Top-k of a row held as v[j] <-> element lane + 32*j (elements >= n are not candidates).
// Lane j (< k) returns the j-th result in (rv, ri).  Every round is a scan of the lane's registers and two warp
// reductions (largest key, then the lowest index that has it): an argmax by shuffles is five dependent steps of two
// shuffles each, and k rounds of it were most of this kernel's time (with the divisions of group_mask: 256 experts in 8
// groups, 64 tokens 14.7 -> 7.8 us, 2048 tokens 18.7 -> 10.0 us).
template <int VPT>
__device__ __forceinline__ void warp_topk(const float (&v)[VPT], int n, int k, int lane, float& rv,
                                          int& ri) {
  uint32_t key[VPT];  // 0 = no candidate (below every key: the key of -inf is 0x007fffff)
#pragma unroll
  for (int j = 0; j < VPT; ++j) key[j] = lane + 32 * j < n ? order_key(v[j]) : 0u;
  rv = -INFINITY;
  ri = 0;
  for (int it = 0; it < k; ++it) {
    uint32_t bk = 0;
    float bv = -INFINITY;
    int bi = INT_MAX;
#pragma unroll
    for (int j = 0; j < VPT; ++j)
      if (key[j] > bk) bk = key[j], bv = v[j], bi = lane + 32 * j;  // ascending inside a lane: the first maximum wins
    const uint32_t best = __reduce_max_sync(0xffffffffu, bk);
    const int idx = (int)__reduce_min_sync(0xffffffffu, bk == best ? (uint32_t)bi : (uint32_t)INT_MAX);
    if (idx == INT_MAX) break;  // (uniform) no candidate left
    bv = __shfl_sync(0xffffffffu, bv, idx & 31);
#pragma unroll
    for (int j = 0; j < VPT; ++j)
      if (lane + 32 * j == idx) key[j] = 0u;
    if (lane == it) rv = bv, ri = idx;
  }
}

// Group-limited masking (python/regression/test_llm/test_noaux_tc_topk.py:10-35): group score = sum of
// the two largest members (formed in `dtype`), keep `topk_groups` groups, mask the rest to -inf.
template <int VPT>
__device__ __forceinline__ void group_mask(float (&v)[VPT], int n, int n_groups, int topk_groups,
                                           int dtype, int lane) {
  const int gsz = n / n_groups;
  // e / gsz for e < 1024 as a multiplication (the error of the rounded-up reciprocal stays below 1023 / 2^20 < 1 / gsz),
  // once per element: a division per element and group was most of the time of a grouped selection
  const uint32_t inv = ((1u << 20) + gsz - 1) / gsz;
  int grp[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) grp[j] = lane + 32 * j < n ? (int)(((uint32_t)(lane + 32 * j) * inv) >> 20) : -1;
  float my_gs = -INFINITY;  // lane g holds the score of group g
  for (int g = 0; g < n_groups; ++g) {
    float a1 = -INFINITY, a2 = -INFINITY;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      if (grp[j] == g) {
        float x = v[j];
        if (x > a1) {
          a2 = a1;
          a1 = x;
        } else if (x > a2) {
          a2 = x;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float b1 = __shfl_xor_sync(0xffffffffu, a1, o);
      float b2 = __shfl_xor_sync(0xffffffffu, a2, o);
      float hi = fmaxf(a1, b1);
      float lo = fmaxf(fminf(a1, b1), fmaxf(a2, b2));
      a1 = hi;
      a2 = lo;
    }
    float gs = gsz > 1 ? moe_add_in_dtype(a1, a2, dtype) : a1;
    if (lane == g) my_gs = gs;
  }
  uint32_t keep = 0;
  bool used = false;
  for (int it = 0; it < topk_groups; ++it) {
    float bv = (lane < n_groups && !used) ? my_gs : -INFINITY;
    int bi = (lane < n_groups && !used) ? lane : INT_MAX;
    warp_argmax(bv, bi);
    if (bi != INT_MAX) {
      keep |= 1u << bi;
      if (bi == lane) used = true;
    }
  }
#pragma unroll
  for (int j = 0; j < VPT; ++j)
    if (grp[j] >= 0 && !((keep >> grp[j]) & 1u)) v[j] = -INFINITY;
}

template <int VPT>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
topk_kernel(void* __restrict__ values, int32_t* __restrict__ indices, const void* scores,
            int dtype, int64_t batch, int n, int n_groups, int topk_groups, int k) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= batch) return;
  float v[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    int e = lane + 32 * j;
    v[j] = e < n ? moe_load_as_f32(scores, row * n + e, dtype) : -INFINITY;
  }
  if (n_groups > 1) group_mask<VPT>(v, n, n_groups, topk_groups, dtype, lane);
  float rv;
  int ri;
  warp_topk<VPT>(v, n, k, lane, rv, ri);
  if (lane < k) {
    moe_store_from_f32(values, row * k + lane, dtype, rv);
    indices[row * k + lane] = ri;
  }
}

struct RouteArgs {
  int32_t* ids;
  float* w;
  __nv_bfloat16* w_bf16;
  const float* logit_bias;
  const float* bias;
  int k, score_func, n_groups, topk_groups, renorm;
  float scale;
};

// One row by one warp: s[j] = logit of element lane + 32*j (elements >= n are not candidates).
template <int VPT>
__device__ __forceinline__ void route_row(float (&s)[VPT], const RouteArgs& a, int64_t row, int n, int lane) {
  const int k = a.k;
  float sel[VPT];  // selection scores; s becomes the un-biased scores
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    int e = lane + 32 * j;
    s[j] = e < n ? (a.logit_bias ? s[j] + a.logit_bias[e] : s[j]) : -INFINITY;
  }
  if (a.score_func == B200MOE_SCORE_SOFTMAX) {
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < VPT; ++j) m = fmaxf(m, s[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      int e = lane + 32 * j;
      s[j] = e < n ? expf(s[j] - m) : 0.f;
      sum += s[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
    for (int j = 0; j < VPT; ++j) s[j] = s[j] / sum;
  } else {
#pragma unroll
    for (int j = 0; j < VPT; ++j) s[j] = 1.0f / (1.0f + expf(-s[j]));
  }
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    int e = lane + 32 * j;
    sel[j] = e < n ? (a.bias ? s[j] + a.bias[e] : s[j]) : -INFINITY;
  }
  if (a.n_groups > 1) group_mask<VPT>(sel, n, a.n_groups, a.topk_groups, B200MOE_F32, lane);
  float rv;
  int ri;
  warp_topk<VPT>(sel, n, k, lane, rv, ri);
  // gather the un-biased score of the chosen expert: it lives in lane ri%32, register ri/32
  float wv = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    // every lane publishes register j; lane `it` picks the one it needs
    float cand = __shfl_sync(0xffffffffu, s[j], ri & 31);
    if ((ri >> 5) == j) wv = cand;
  }
  if (lane >= k) wv = 0.f;
  if (a.renorm) {
    float sum = wv;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    wv = wv / sum;
  }
  wv = wv * a.scale;
  if (lane < k) {
    a.ids[row * k + lane] = ri;
    a.w[row * k + lane] = wv;
    if (a.w_bf16) a.w_bf16[row * k + lane] = __float2bfloat16_rn(wv);
  }
}

template <int VPT>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
route_kernel(const float* logits, int64_t T, int n, const RouteArgs a) {
  pdl_begin();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= T) return;
  float s[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    int e = lane + 32 * j;
    s[j] = e < n ? logits[row * n + e] : -INFINITY;
  }
  route_row<VPT>(s, a, row, n, lane);
}

// ---- router GEMM ---------------------------------------------------------------------------------
// logits[t,e] = sum_h x[t,h] * wr[e,h]; bf16 operands, fp32 accumulation on the warp-level tensor path
// (mma.sync m16n8k16).  It is ~0.5 % of the layer's FLOPs and bound by the copies of x and wr on their way to shared
// memory and by the chain of MMAs over K.  That chain is never cut: a logit is the same number whatever the tile and the
// batch size (K in order), so that a token's experts do not depend on them - cutting it moves logits by 1e-6, which gave
// one token in a few thousand other experts.  So the batch decides the tile instead, the largest that gives most SMs a
// block; stages are four or eight 64-column chunks deep.  Against 32 x 64 tiles and three stages for every batch: DeepSeek
// shape 64 tokens 42 -> 25 us (8 blocks became 64), 2048 tokens 57 -> 52, Qwen3 shape 8192 tokens 34 -> 27.
constexpr int RG_BK = 64, RG_LD = RG_BK + 8;  // +8 bf16: conflict-free ldmatrix
template <int BM_, int BN_, int WM_, int WN_, int STAGES_>
struct RgTile {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, STAGES = STAGES_;  // WM x WN warps
  static constexpr int THREADS = 32 * WM * WN, MT = BM / WM / 16, NT = BN / WN / 8;
  static constexpr int STAGE_ELEMS = (BM + BN) * RG_LD;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_ELEMS * sizeof(__nv_bfloat16);
  static_assert(BM == WM * MT * 16 && BN == WN * NT * 8 && (NT == 1 || NT % 2 == 0) && (BM + BN) * 8 % THREADS == 0, "");
};
using RgLarge = RgTile<64, 128, 2, 4, 4>;
using RgMedium = RgTile<32, 64, 2, 2, 4>;
using RgSmall = RgTile<16, 16, 1, 2, 8>;

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldmatrix_x2(uint32_t& r0, uint32_t& r1, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r0), "=r"(r1)
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// 16-byte asynchronous copy global -> shared; bytes = 0 writes zeros (rows / columns past the end)
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)),
               "l"(gsrc), "r"(bytes)
               : "memory");
}

// grid (ceil(T / BM), ceil(E / BN))
template <class C>
__global__ void __launch_bounds__(C::THREADS)
router_gemm_kernel(float* __restrict__ logits, const __nv_bfloat16* x,
                   const __nv_bfloat16* wr, int64_t T, int64_t H, int64_t E) {
  pdl_begin();
  extern __shared__ __align__(16) uint8_t rg_smem[];
  __nv_bfloat16* const stages = reinterpret_cast<__nv_bfloat16*>(rg_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row_w = (warp % C::WM) * (C::MT * 16), col_w = (warp / C::WM) * (C::NT * 8);  // the warp's part of the tile
  const int64_t t0 = (int64_t)blockIdx.x * C::BM, e0 = (int64_t)blockIdx.y * C::BN;
  const int nk = (int)((H + RG_BK - 1) / RG_BK);
  float acc[C::MT][C::NT][4];
#pragma unroll
  for (int m = 0; m < C::MT; ++m)
#pragma unroll
    for (int i = 0; i < C::NT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[m][i][j] = 0.f;
  auto load_stage = [&](int kt) {
    __nv_bfloat16* const st = stages + (size_t)(kt % C::STAGES) * C::STAGE_ELEMS;
    const int64_t k0 = (int64_t)kt * RG_BK;
#pragma unroll
    for (int i = 0; i < (C::BM + C::BN) * 8 / C::THREADS; ++i) {  // rows of x, then rows of wr; 8 chunks of 16 B each
      const int c = tid + i * C::THREADS;
      const int r = c >> 3, cc = (c & 7) * 8;
      const bool is_x = r < C::BM;
      const int64_t row = is_x ? t0 + r : e0 + r - C::BM;
      const bool on = k0 + cc < H && row < (is_x ? T : E);
      const __nv_bfloat16* src = (is_x ? x : wr) + (on ? row * H + k0 + cc : 0);
      cp_async16(st + r * RG_LD + cc, src, on ? 16 : 0);
    }
  };
  // one commit group per chunk, empty where there is no chunk left, so that "all but the newest groups are complete"
  // always means "chunk kt has landed"
#pragma unroll
  for (int s = 0; s < C::STAGES - 1; ++s) {
    if (s < nk) load_stage(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(C::STAGES - 2) : "memory");
    __syncthreads();  // chunk kt is there for everyone, and everyone is done with the stage that is filled next
    if (kt + C::STAGES - 1 < nk) load_stage(kt + C::STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const __nv_bfloat16* sA = stages + (size_t)(kt % C::STAGES) * C::STAGE_ELEMS;
    const __nv_bfloat16* sB = sA + C::BM * RG_LD;
#pragma unroll
    for (int kk = 0; kk < RG_BK; kk += 16) {
      uint32_t a[C::MT][4], b[C::NT][2];
#pragma unroll
      for (int m = 0; m < C::MT; ++m)  // rows 0-7 / 8-15 at k, then the same at k + 8
        ldmatrix_x4(a[m], sA + (row_w + m * 16 + (lane & 15)) * RG_LD + kk + (lane >> 4) * 8);
      if (C::NT == 1) {
        ldmatrix_x2(b[0][0], b[0][1], sB + (col_w + (lane & 7)) * RG_LD + kk + ((lane >> 3) & 1) * 8);
      } else {
#pragma unroll
        for (int p = 0; p < C::NT / 2; ++p) {  // columns 0-7 at k, k + 8, then columns 8-15
          uint32_t r[4];
          ldmatrix_x4(r, sB + (col_w + p * 16 + (lane & 7) + ((lane >> 4) << 3)) * RG_LD + kk + ((lane >> 3) & 1) * 8);
          b[2 * p][0] = r[0], b[2 * p][1] = r[1];
          b[(2 * p + 1) % C::NT][0] = r[2], b[(2 * p + 1) % C::NT][1] = r[3];
        }
      }
#pragma unroll
      for (int m = 0; m < C::MT; ++m)
#pragma unroll
        for (int nb = 0; nb < C::NT; ++nb) mma_bf16_16816(acc[m][nb], a[m], b[nb][0], b[nb][1]);
    }
  }
  const int g = lane >> 2, tq = lane & 3;
#pragma unroll
  for (int m = 0; m < C::MT; ++m)
#pragma unroll
    for (int nb = 0; nb < C::NT; ++nb)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t r = t0 + row_w + m * 16 + g + (i >> 1) * 8, c = e0 + col_w + nb * 8 + tq * 2 + (i & 1);
        if (r < T && c < E) logits[r * E + c] = acc[m][nb][i];
      }
}

// Small-T variant (decode): one block per expert row; its 4 warps split H (16-byte loads) and dot the slice with up
// to RV_MAXT token rows; the warps' partial sums are added in warp order (deterministic).  The grid covers all
// experts, so the read of the router weights is spread over many SMs and only H/1024 loads deep.
constexpr int RV_MAXT = 8;
__global__ void __launch_bounds__(128)
router_gemv_kernel(float* __restrict__ logits, const __nv_bfloat16* x,
                   const __nv_bfloat16* wr, int64_t T, int64_t H, int64_t E) {
  pdl_begin();
  __shared__ float part[4][RV_MAXT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t e = blockIdx.x;
  const int64_t t0 = (int64_t)blockIdx.y * RV_MAXT;
  float acc[RV_MAXT];
#pragma unroll
  for (int t = 0; t < RV_MAXT; ++t) acc[t] = 0.f;
  for (int64_t h = (int64_t)threadIdx.x * 8; h < H; h += 1024) {
    uint4 wv = *reinterpret_cast<const uint4*>(wr + e * H + h);
    const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
    for (int t = 0; t < RV_MAXT; ++t) {
      if (t0 + t < T) {
        uint4 xv = *reinterpret_cast<const uint4*>(x + (t0 + t) * H + h);
        const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 a = __bfloat1622float2(w2[i]), b = __bfloat1622float2(x2[i]);
          acc[t] = fmaf(a.x, b.x, acc[t]);
          acc[t] = fmaf(a.y, b.y, acc[t]);
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < RV_MAXT; ++t) {
    float v = acc[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) part[warp][t] = v;
  }
  __syncthreads();
  if (threadIdx.x < RV_MAXT && t0 + threadIdx.x < T)
    logits[(t0 + threadIdx.x) * E + e] = part[0][threadIdx.x] + part[1][threadIdx.x] + part[2][threadIdx.x] + part[3][threadIdx.x];
}

constexpr int RS_TOK = 4, RS_WARPS = 8;
// Few-experts variant (E <= 16, e.g. 8 for Mixtral): the 64x64 tensor-core tile would be mostly padding, and the
// op is a read of x.  A block owns RS_TOK tokens and its 8 warps split H between them (interleaved 256-column
// slices, 16-byte loads of x and of the L2-resident router weights), so that decode-size batches still fill more
// than a handful of SMs; the per-warp partial sums meet in shared memory and are added in warp order, so the
// result does not depend on timing.  With ROUTE the block goes on to route its tokens, one warp each, from the logits it
// has just formed: one launch less in front of the experts (Mixtral shape, 32 tokens: 6.6 + 3.5 us as two kernels).
template <int EP, bool ROUTE>
__global__ void __launch_bounds__(RS_WARPS * 32)
router_small_e_kernel(float* __restrict__ logits, const __nv_bfloat16* x,
                       const __nv_bfloat16* wr, int64_t T, int64_t H, int E, const RouteArgs ra) {
  pdl_begin();
  __shared__ float sums[RS_TOK][EP];
  __shared__ float part[RS_WARPS][RS_TOK][EP];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t0 = (int64_t)blockIdx.x * RS_TOK;
  float acc[RS_TOK][EP];
#pragma unroll
  for (int i = 0; i < RS_TOK; ++i)
#pragma unroll
    for (int e = 0; e < EP; ++e) acc[i][e] = 0.f;
  for (int64_t col = (int64_t)(warp * 32 + lane) * 8; col < H; col += RS_WARPS * 256) {
    float xv[RS_TOK][8];
#pragma unroll
    for (int i = 0; i < RS_TOK; ++i) {
      uint4 raw = make_uint4(0, 0, 0, 0);
      if (t0 + i < T) raw = *reinterpret_cast<const uint4*>(x + (t0 + i) * H + col);
      const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f = __bfloat1622float2(b2[j]);
        xv[i][2 * j] = f.x;
        xv[i][2 * j + 1] = f.y;
      }
    }
#pragma unroll
    for (int e = 0; e < EP; ++e) {
      uint4 raw = make_uint4(0, 0, 0, 0);
      if (e < E) raw = *reinterpret_cast<const uint4*>(wr + (int64_t)e * H + col);
      const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f = __bfloat1622float2(b2[j]);
#pragma unroll
        for (int i = 0; i < RS_TOK; ++i) {
          acc[i][e] = fmaf(xv[i][2 * j], f.x, acc[i][e]);
          acc[i][e] = fmaf(xv[i][2 * j + 1], f.y, acc[i][e]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RS_TOK; ++i)
#pragma unroll
    for (int e = 0; e < EP; ++e) {
      float v = acc[i][e];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) part[warp][i][e] = v;
    }
  __syncthreads();
  if (threadIdx.x < RS_TOK * EP) {
    const int i = threadIdx.x / EP, e = threadIdx.x % EP;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) v += part[w][i][e];
    if (t0 + i < T && e < E) logits[(t0 + i) * E + e] = v;
    if (ROUTE) sums[i][e] = v;
  }
  if (ROUTE) {
    __syncthreads();
    if (warp < RS_TOK && t0 + warp < T) {
      float s[1] = {lane < EP ? sums[warp][lane] : 0.f};  // (elements >= E are masked by route_row)
      route_row<1>(s, ra, t0 + warp, E, lane);
    }
  }
}

template <class C>
int launch_router_gemm(float* logits, const __nv_bfloat16* x, const __nv_bfloat16* wr, int64_t T, int64_t H, int64_t E,
                       cudaStream_t st) {
  constexpr int kMaxDevices = 64;
  static bool attr_done[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200MOE_EDRIVER;
  if (!attr_done[dev]) {  // per-device attribute
    cudaFuncSetAttribute(router_gemm_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    attr_done[dev] = true;
  }
  return moe_launch(router_gemm_kernel<C>, dim3((unsigned)((T + C::BM - 1) / C::BM), (unsigned)((E + C::BN - 1) / C::BN)),
                    C::THREADS, C::SMEM, st, logits, x, wr, T, H, E);
}

template <typename F>
int dispatch_vpt(int64_t n, F&& f) {
  if (n <= 32) return f(std::integral_constant<int, 1>{});
  if (n <= 64) return f(std::integral_constant<int, 2>{});
  if (n <= 128) return f(std::integral_constant<int, 4>{});
  if (n <= 256) return f(std::integral_constant<int, 8>{});
  if (n <= 512) return f(std::integral_constant<int, 16>{});
  return f(std::integral_constant<int, 32>{});
}

int launch_topk(void* values, int32_t* indices, const void* scores, int dtype, int64_t batch, int64_t n,
                int64_t n_groups, int64_t topk_groups, int64_t k, void* stream) {
  MOE_CHECK_ARG(values && indices && scores);
  MOE_CHECK_ARG(dtype == B200MOE_F32 || dtype == B200MOE_BF16 || dtype == B200MOE_F16);
  MOE_CHECK_ARG(batch >= 0 && n > 0 && k > 0);
  MOE_CHECK_SHAPE(n <= 1024 && k <= 32 && k <= n);
  if (n_groups > 1) {
    MOE_CHECK_SHAPE(n_groups <= 32 && n % n_groups == 0 && topk_groups >= 1 && topk_groups <= n_groups);
    MOE_CHECK_SHAPE(k <= topk_groups * (n / n_groups));
  }
  if (batch == 0) return B200MOE_OK;
  dim3 grid((unsigned)((batch + kWarpsPerBlock - 1) / kWarpsPerBlock));
  return dispatch_vpt(n, [&](auto vpt) {
    return moe_launch(topk_kernel<decltype(vpt)::value>, grid, kWarpsPerBlock * 32, 0, (cudaStream_t)stream, values, indices,
                      scores, dtype, batch, (int)n, (int)n_groups, (int)topk_groups, (int)k);
  });
}

}  // namespace

extern "C" int b200moe_noaux_tc_topk(void* values, int32_t* indices, const void* scores, int dtype,
                                     int64_t batch, int64_t n_experts, int64_t n_groups,
                                     int64_t topk_groups, int64_t top_k, void* stream) {
  MOE_CHECK_ARG(n_groups >= 1);
  return launch_topk(values, indices, scores, dtype, batch, n_experts, n_groups, topk_groups, top_k, stream);
}

extern "C" int b200moe_topk(void* values, int32_t* indices, const void* x, int dtype, int64_t batch,
                            int64_t n, int64_t k, void* stream) {
  return launch_topk(values, indices, x, dtype, batch, n, 1, 1, k, stream);
}

namespace {
int check_route(const void* ids, const void* w, const void* logits, int64_t T, int64_t E, int64_t k, int score_func,
                int64_t n_groups, int64_t topk_groups) {
  MOE_CHECK_ARG(ids && w && logits && T >= 0 && E > 0 && k > 0);
  MOE_CHECK_ARG(score_func == B200MOE_SCORE_SOFTMAX || score_func == B200MOE_SCORE_SIGMOID);
  MOE_CHECK_SHAPE(E <= 1024 && k <= 32 && k <= E);
  if (n_groups > 1) {
    MOE_CHECK_SHAPE(n_groups <= 32 && E % n_groups == 0 && topk_groups >= 1 && topk_groups <= n_groups);
    MOE_CHECK_SHAPE(k <= topk_groups * (E / n_groups));
  }
  return B200MOE_OK;
}
RouteArgs route_args(int32_t* ids, float* w, void* w_bf16, const float* logit_bias, const float* bias, int64_t k,
                     int score_func, int64_t n_groups, int64_t topk_groups, int renorm, float scale) {
  return RouteArgs{ids, w, reinterpret_cast<__nv_bfloat16*>(w_bf16), logit_bias, bias, (int)k, score_func,
                   (int)(n_groups > 1 ? n_groups : 1), (int)topk_groups, renorm, scale};
}
}  // namespace

extern "C" int b200moe_route(int32_t* ids, float* w, void* w_bf16, const float* logits,
                             const float* logit_bias, const float* bias, int64_t T, int64_t E, int64_t k, int score_func, int64_t n_groups,
                             int64_t topk_groups, int renorm, float scale, void* stream) {
  const int rc = check_route(ids, w, logits, T, E, k, score_func, n_groups, topk_groups);
  if (rc) return rc;
  if (T == 0) return B200MOE_OK;
  const RouteArgs a = route_args(ids, w, w_bf16, logit_bias, bias, k, score_func, n_groups, topk_groups, renorm, scale);
  dim3 grid((unsigned)((T + kWarpsPerBlock - 1) / kWarpsPerBlock));
  return dispatch_vpt(E, [&](auto vpt) {
    return moe_launch(route_kernel<decltype(vpt)::value>, grid, kWarpsPerBlock * 32, 0, (cudaStream_t)stream, logits, T,
                      (int)E, a);
  });
}

extern "C" int b200moe_router_route(float* logits, int32_t* ids, float* w, void* w_bf16, const void* x, const void* wr,
                                    const float* logit_bias, const float* bias, int64_t T, int64_t H, int64_t E, int64_t k,
                                    int score_func, int64_t n_groups, int64_t topk_groups, int renorm, float scale,
                                    void* stream) {
  int rc = check_route(ids, w, logits, T, E, k, score_func, n_groups, topk_groups);
  if (rc) return rc;
  // One kernel where the few-experts variant forms the logits, which holds all of a token's in one block, and its blocks
  // (one to an SM with the selection's registers) fit the SMs at once: Mixtral shape, 512 tokens 7.3 us against
  // 6.5 + 3.9, but 4096 tokens 35.1 against 21.5 + 4.6.  The other variants, and the small batches that spread every
  // expert row over a block, route in a second kernel.
  if (E > 16 || T <= 2 * RV_MAXT || T > (int64_t)RS_TOK * moe_device_sm_count()) {
    rc = b200moe_router_logits(logits, x, wr, T, H, E, stream);
    if (rc) return rc;
    return b200moe_route(ids, w, w_bf16, logits, logit_bias, bias, T, E, k, score_func, n_groups, topk_groups, renorm, scale,
                         stream);
  }
  MOE_CHECK_ARG(x && wr && H > 0);
  MOE_CHECK_SHAPE(H % 8 == 0);
  if (!moe_aligned16(x) || !moe_aligned16(wr)) return B200MOE_EALIGN;
  const RouteArgs a = route_args(ids, w, w_bf16, logit_bias, bias, k, score_func, n_groups, topk_groups, renorm, scale);
  return moe_launch(E <= 8 ? router_small_e_kernel<8, true> : router_small_e_kernel<16, true>,
                    dim3((unsigned)((T + RS_TOK - 1) / RS_TOK)), RS_WARPS * 32, 0, (cudaStream_t)stream, logits,
                    reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(wr), T, H, (int)E, a);
}

extern "C" int b200moe_router_logits(float* logits, const void* x, const void* wr, int64_t T, int64_t H,
                                     int64_t E, void* stream) {
  MOE_CHECK_ARG(logits && x && wr && T >= 0 && H > 0 && E > 0);
  MOE_CHECK_SHAPE(H % 8 == 0);
  if (!moe_aligned16(x) || !moe_aligned16(wr)) return B200MOE_EALIGN;
  if (T == 0) return B200MOE_OK;
  auto xb = reinterpret_cast<const __nv_bfloat16*>(x);
  auto wb = reinterpret_cast<const __nv_bfloat16*>(wr);
  if (T <= 2 * RV_MAXT) {
    return moe_launch(router_gemv_kernel, dim3((unsigned)E, (unsigned)((T + RV_MAXT - 1) / RV_MAXT)), 128, 0,
                      (cudaStream_t)stream, logits, xb, wb, T, H, E);
  } else if (E <= 16) {
    return moe_launch(E <= 8 ? router_small_e_kernel<8, false> : router_small_e_kernel<16, false>, dim3((unsigned)((T + RS_TOK - 1) / RS_TOK)),
                      RS_WARPS * 32, 0, (cudaStream_t)stream, logits, xb, wb, T, H, (int)E, RouteArgs{});
  } else {
    // the larger tile where it still gives most SMs a block
    auto blocks = [&](int bm, int bn) { return ((T + bm - 1) / bm) * ((E + bn - 1) / bn); };
    const int64_t enough = moe_device_sm_count() * 4 / 5;
    if (blocks(RgLarge::BM, RgLarge::BN) >= enough) return launch_router_gemm<RgLarge>(logits, xb, wb, T, H, E, (cudaStream_t)stream);
    if (blocks(RgMedium::BM, RgMedium::BN) >= enough) return launch_router_gemm<RgMedium>(logits, xb, wb, T, H, E, (cudaStream_t)stream);
    return launch_router_gemm<RgSmall>(logits, xb, wb, T, H, E, (cudaStream_t)stream);
  }
}
