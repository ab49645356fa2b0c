// Shared device/host helpers of the fused-MoE kernels (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/b200moe.h"

#define B200MOE_STATUS_BAD_EXPERT 1
#define B200MOE_STATUS_WAIT_TIMEOUT 2
#define B200MOE_STATUS_PEER_TIMEOUT 4
#define B200MOE_STATUS_PEER_OVERFLOW 8

constexpr int kBlock = 128;          // quantisation block (columns per activation scale, weight tile edge)
constexpr float kFp8Max = 448.0f;    // largest finite e4m3 value
constexpr float kAmaxFloor = 1e-12f; // floor of a group's max|x| before the scale is formed

#define MOE_CHECK_ARG(cond)            \
  do {                                 \
    if (!(cond)) return B200MOE_EINVAL; \
  } while (0)
#define MOE_CHECK_SHAPE(cond)          \
  do {                                 \
    if (!(cond)) return B200MOE_ESHAPE; \
  } while (0)

static inline int moe_launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? B200MOE_OK : (int)e;
}

static inline bool moe_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ---- launches that overlap the end of the kernel before them -----------------------------------------------------
// A call is a chain of short kernels, and at decode sizes the gaps between them (drain, launch, set-up of the next) cost
// as much as the kernels.  moe_launch starts a kernel while its predecessor on the stream still runs (programmatic stream
// serialisation).  The rules that make this safe: every kernel launched this way executes pdl_wait() in every thread
// before it touches memory that an earlier kernel of the stream writes or reads (it returns when the predecessor has
// completed and its writes are visible), and pdl_next(), which lets the successor start, comes after it.  So when a
// kernel starts, everything before its direct predecessor is complete.  Launched after anything else than such a
// kernel, pdl_wait() finds its predecessor complete.  Such a kernel reads through plain pointers: `const __restrict__`
// would promise that the data does not change while the kernel runs (and allow the read-only load path), and it runs
// while its predecessor still writes.
// A kernel whose SMs are meant to be shared with another stream's leaves pdl_next() out (the GEMMs' hold_next): started
// early, the blocks behind it take SMs and wait there.  With 98 CTAs the gate/up GEMM of one Mixtral expert, 4096 tokens,
// held a permutation of another stream until its own end: it ended 758 us after the call's start, 88 us without (the call
// itself 1.16 and 1.14 ms).  DeepSeek shape, 1 token, the shared expert's GEMMs on the side stream: 136 -> 115 us; 8 to 64
// tokens the same with either.
// Not for large launches: what an early start saves is a gap of two or three microseconds, whatever the size, and beside
// a long kernel it costs more than that.  Layer times in us, without / with the early start:
//   GEMMs, by the K blocks (0.5 to 0.6 us each) that a CTA of the gate/up GEMM walks: 15 (small layer, 4096 tokens) 69.9 /
//   63.9; 83 (Qwen3 shape, 1024) 113.4 / 110.5; 125 (2048) 192.9 / 186.2; 208 (4096) 332 / 331; 303 (Mixtral shape, 512)
//   428 / 430; 496 (1024) 635 / 641; 884 (2048) 1103 / 1124; 1647 (4095) 1976 / 2024.
//   Other kernels, by their blocks: up to 256 (small layer, 512 tokens) 36.9 / 34.8; 2048 (combine, small layer, 4096
//   tokens) 63.9 / 62.8 and (Qwen3 shape, 2048) 186.2 / 183.5; 4096 (Qwen3 shape, 4096) 331 / 335.
constexpr long long kOverlapMaxBlocks = 2048;
constexpr int64_t kOverlapMaxKBlocks = 256;  // per CTA of a GEMM
constexpr int64_t kOverlapMaxRowsPerExpert = 16;
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_next();
}
template <typename... KArgs, typename... Args>
inline int moe_launch_as(bool overlap, int cluster_y, void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem,
                         cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = at[1].val.clusterDim.z = 1;
  at[1].val.clusterDim.y = (unsigned)cluster_y;
  cfg.attrs = at;
  cfg.numAttrs = cluster_y > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return (int)e;
  }
  return B200MOE_OK;
}
template <typename... KArgs, typename... Args>
inline int moe_launch(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, Args&&... args) {
  const bool overlap = (long long)grid.x * grid.y * grid.z <= kOverlapMaxBlocks;
  return moe_launch_as(overlap, 1, kernel, grid, block, smem, st, static_cast<Args&&>(args)...);
}
#endif

// ---- scalar loads of score / scale tensors in their storage dtype -----------------------------
__device__ __forceinline__ float moe_load_as_f32(const void* p, int64_t i, int dtype) {
  if (dtype == B200MOE_F32) return reinterpret_cast<const float*>(p)[i];
  if (dtype == B200MOE_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return __half2float(reinterpret_cast<const __half*>(p)[i]);
}
__device__ __forceinline__ void moe_store_from_f32(void* p, int64_t i, int dtype, float v) {
  if (dtype == B200MOE_F32) reinterpret_cast<float*>(p)[i] = v;
  else if (dtype == B200MOE_BF16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
}
// a + b rounded into `dtype` (what an add of two tensors of that dtype yields)
__device__ __forceinline__ float moe_add_in_dtype(float a, float b, int dtype) {
  float s = a + b;
  if (dtype == B200MOE_BF16) return __bfloat162float(__float2bfloat16_rn(s));
  if (dtype == B200MOE_F16) return __half2float(__float2half_rn(s));
  return s;
}

// ---- e4m3 conversion ---------------------------------------------------------------------------
__device__ __forceinline__ float moe_e4m3_to_f32(uint8_t v) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(v, __NV_E4M3);
  return __half2float(__half(h));
}
// two floats -> two e4m3 bytes (RNE, saturating to +-448); low byte = a
__device__ __forceinline__ uint16_t moe_f32x2_to_e4m3x2(float a, float b) {
  return __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ uint32_t moe_f32x4_to_e4m3x4(float a, float b, float c, float d) {
  return (uint32_t)moe_f32x2_to_e4m3x2(a, b) | ((uint32_t)moe_f32x2_to_e4m3x2(c, d) << 16);
}

__device__ __forceinline__ float moe_bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// SiLU in fp32: x * 1/(1+exp(-x))
__device__ __forceinline__ float moe_silu(float x) { return x / (1.0f + expf(-x)); }
