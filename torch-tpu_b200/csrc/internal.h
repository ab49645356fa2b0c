// Launchers shared between the translation units of libb200moe (not part of the C ABI).
#pragma once
#include "common.cuh"

constexpr int kTileM = 128;  // rows of one m-tile of the grouped GEMMs

// Workspace of tiles that several CTAs share (schedule.h): partial sums, one slot per part, and one counter per shared
// tile, zero when the launch starts and zero again when it ends.
constexpr int kMaxSplitCtas = 160;
constexpr int kSplitCounters = kMaxSplitCtas;
struct MoeSplitBuffers {
  float* part;
  int32_t* cnt;
};
// floats of one slot: the row quarters of a 128 x 256 tile that a problem of P rows can have
inline int moe_split_slot_floats(int64_t P) { return (int)(P < kTileM ? (P + 31) / 32 : kTileM / 32) * 32 * 256; }
inline size_t moe_split_part_bytes(int64_t P) { return (size_t)kMaxSplitCtas * moe_split_slot_floats(P) * sizeof(float); }

// One grouped-GEMM problem: rows [0,P) sorted by expert, m-tiles built from expert_offsets.
struct MoeGemmArgs {
  // activations
  const uint8_t* aq;        // W8A8: e4m3 [P,K]
  const float* as_t;        // W8A8: scales [K/128, ld]
  int64_t ld;               // leading dimension of transposed scale arrays
  const __nv_bfloat16* a16; // W8A16: bf16 rows; gemm1: x [T,H] gathered through row_map/div; gemm2: h [P,I]
  const int32_t* row_map;   // sorted_pair (flat t*k+j) or nullptr for identity
  int div;                  // k (pair -> token)
  // weights of this problem ([E,I,H] e4m3, scales [E,I/128,H/128])
  const uint8_t* w0;        // gemm1: gate; gemm2: down
  const uint8_t* w1;        // gemm1: up
  const void* s0;
  const void* s1;
  int scale_dtype;
  int w_bf16;               // weights are bf16 (no scales): W8A16 tensor-core kernels only
  // tiling
  const int32_t* mtiles;    // int2 {expert, row0} per m-tile
  const int32_t* num_mtiles;
  const int32_t* offsets;   // expert_offsets[E+1]
  int max_mtiles;
  int max_ctas;             // 0 = all SMs; else the cap on the tensor-core kernels' persistent grid
  int64_t P;
  int H, I, E;
  // outputs
  uint8_t* hq;              // gemm1 W8A8: e4m3 [P,I]
  float* hs_t;              // gemm1 W8A8: [I/128, ld]
  __nv_bfloat16* h16;       // gemm1 W8A16: bf16 [P,I]
  __nv_bfloat16* out;       // gemm2: bf16 rows of H, row index = row_map ? row_map[r] : r
  int ksplit;               // gemm2 (tensor-core path): > 1 splits K over CTAs, partial sums added into out32
  float* out32;             // fp32 [rows,H], zero on entry, same row indexing as out (needed when ksplit > 1)
  MoeSplitBuffers split;    // lets CTAs share tiles (part NULL = they may not)
  // gemm2 with the weighted combine fused in (tensor-core path only): row r adds comb_w[pair] * y[r,:] into
  // comb32[pair / div, :], pair = row_map ? row_map[r] : r; comb32 fp32 [T,H], zero on entry; comb_w NULL = weight 1
  float* comb32;
  const void* comb_w;
  int comb_wdt;
  // gemm2 over peer memory (tensor-core path only): row r goes to rank (row_src[r] >> 24), row (row_src[r] & 0xFFFFFF)
  // of that rank's buffer out_tbl[rank] (bf16 rows of H); overrides out/row_map
  const int32_t* row_src;
  const uint64_t* out_tbl;
  int hold_next;            // tensor-core kernels: the kernel behind this one starts after it and not beside it (see pdl_next)
  int lists_ready;          // mtiles / num_mtiles / offsets are older than the launch's direct predecessor (see pdl_wait)
  int32_t* status;
};

// May a GEMM of NT n-tiles and K columns on `grid` CTAs start early (common.cuh)?  The host knows the rows that the
// buffers hold; the number of m-tiles is estimated from them, half a tile on top for each expert that can have rows.
// With a few rows per expert the GEMM streams weights and its first requests go out early (DeepSeek shape, without / with:
// 64 tokens, 2 rows, 1778 / 1768 us; 256 tokens, 8 rows, 2174 / 2148; 1023 tokens, 32 rows, 2404 / 2457).
inline bool moe_gemm_overlaps(const MoeGemmArgs& g, int NT, int64_t K, int grid) {
  if (g.P <= kOverlapMaxRowsPerExpert * g.E) return true;
  const int64_t half_tiles = 2 * g.P / kTileM + (g.E < g.P ? g.E : g.P) + 1;
  return half_tiles * NT * (K / kBlock) <= 2 * kOverlapMaxKBlocks * grid;
}

// lists of an identity problem (one expert, rows 0..rows): offsets = {0, rows} and its m-tiles; offsets NULL = none
struct MoeIdentityLists {
  int32_t* offsets;
  int32_t* mtiles;
  int32_t* num_mtiles;
  int32_t* split_cnt;  // kSplitCounters counters to clear, or NULL
};
#ifdef __CUDACC__
__device__ __forceinline__ void moe_clear_counters(int32_t* cnt) {
  if (cnt)
    for (int i = threadIdx.x; i < kSplitCounters; i += blockDim.x) cnt[i] = 0;
}
// by the threads of one block
__device__ __forceinline__ void moe_write_identity_lists(const MoeIdentityLists& l, int rows) {
  const int n = (rows + kTileM - 1) / kTileM;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    l.mtiles[2 * i] = 0;
    l.mtiles[2 * i + 1] = i * kTileM;
  }
  moe_clear_counters(l.split_cnt);
  if (threadIdx.x == 0) l.offsets[0] = 0, l.offsets[1] = rows, *l.num_mtiles = n;
}
#endif

// b200moe_permute that also writes the inverse map (pos_of, may be NULL) and the m-tile list (mtiles, may be NULL)
int moe_permute_impl(int32_t* sorted_pair, int32_t* expert_offsets, const int32_t* ids, int64_t T, int64_t k, int64_t E,
                     int32_t* scratch, int32_t* status, int32_t* pos_of, int32_t* mtiles, int32_t* num_mtiles,
                     int max_mtiles, int32_t* split_cnt, void* stream);
// quantised rows of x at the positions of every token's k pairs (and zeros to acc32 [T,H], may be NULL); quantised rows 0..rows with the identity lists
int moe_quant_tokens(uint8_t* q, float* s_t, int64_t ld, const void* x, const int32_t* pos_of, int64_t T, int64_t k,
                     int64_t H, float* acc32, cudaStream_t st);
int moe_quant_identity(uint8_t* q, float* s_t, int64_t ld, const void* x, int64_t rows, int64_t H,
                       const MoeIdentityLists& lists, cudaStream_t st);
// tiles of rows [offsets[e], offsets[e+1]) clipped to max_rows; at most max_mtiles entries are written; clears the
// counters of shared tiles (split_cnt, may be NULL)
int moe_build_mtiles(int32_t* mtiles, int32_t* num_mtiles, const int32_t* offsets, int E, int64_t max_rows,
                     int max_mtiles, int32_t* split_cnt, cudaStream_t st);
int moe_identity_lists(const MoeIdentityLists& lists, int64_t rows, cudaStream_t st);

int moe_gemm1_simple(const MoeGemmArgs& a, int act_mode, cudaStream_t st);
int moe_gemm2_simple(const MoeGemmArgs& a, int act_mode, cudaStream_t st);
int moe_gemm1_tc(const MoeGemmArgs& a, cudaStream_t st);
int moe_gemm2_tc(const MoeGemmArgs& a, cudaStream_t st);
// plain linear layer: out[r, :I] = A[r, :H] * w0^T, w0 [E*I, H] K-major with scales s0 [E, ceil(I/128), H/128]; bf16 rows of I
int moe_linear_tc(const MoeGemmArgs& a, cudaStream_t st);
// the reference arithmetic (bf16 activations, weights dequantised to bf16) on the tensor cores; a16 = rows in sorted order
int moe_gemm1_w8a16_tc(const MoeGemmArgs& a, cudaStream_t st);
int moe_gemm2_w8a16_tc(const MoeGemmArgs& a, cudaStream_t st);
int moe_gather_rows_bf16(__nv_bfloat16* dst, const __nv_bfloat16* x, const int32_t* row_map, int div, int64_t rows,
                         int H, cudaStream_t st);
int moe_f32_rows_to_bf16(__nv_bfloat16* out, const float* in, int64_t n, cudaStream_t st);
int moe_device_sm_count();
bool moe_tc_available();
