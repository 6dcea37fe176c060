// Shared device helpers for the D2DMoE sm_100a kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/d2dmoe.h"

namespace d2d {

using bf16 = __nv_bfloat16;

// ---- dtype traits --------------------------------------------------------
template <typename T> struct DT;
template <> struct DT<float> {
  static __device__ __forceinline__ float to_f(float v) { return v; }
  static __device__ __forceinline__ float from_f(float v) { return v; }
  // value after being materialised as a tensor of this dtype
  static __device__ __forceinline__ float round(float v) { return v; }
};
template <> struct DT<bf16> {
  static __device__ __forceinline__ float to_f(bf16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ bf16 from_f(float v) { return __float2bfloat16_rn(v); }
  static __device__ __forceinline__ float round(float v) {
    return __bfloat162float(__float2bfloat16_rn(v));
  }
};

// four consecutive elements as floats (16-byte load for float, 8-byte for bf16)
__device__ __forceinline__ float4 load4(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// ---- programmatic dependent launch ----------------------------------------
// A kernel launched with launch_pdl may start while the previous kernel of the stream is
// still running; it must call grid_dependency_wait() before it touches memory written by
// earlier kernels.  grid_launch_dependents() lets the next such kernel be scheduled early.
// Both are no-ops for kernels launched the ordinary way.
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// cluster > 0: in clusters of that many CTAs.
template <typename... KArgs, typename... Args>
inline int launch_pdl_cluster(int cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block,
                              size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster > 0) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  if (cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...) == cudaSuccess) return D2D_OK;
  cudaGetLastError();
  return D2D_ERR_LAUNCH;
}

template <typename... KArgs, typename... Args>
inline int launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                      cudaStream_t s, Args... args) {
  return launch_pdl_cluster(0, kernel, grid, block, smem, s, args...);
}

// ---- device status word ---------------------------------------------------
// First error wins; kernels return early after reporting, they never trap.
__device__ __forceinline__ void report(int* dev_status, int code) {
  if (dev_status) atomicCAS(dev_status, 0, code);
}

// ---- activations ----------------------------------------------------------
// relu, exact-erf gelu, tanh, leaky relu (slope 0.01), tanh-form gelu.
__device__ __forceinline__ float activate(float h, int act) {
  switch (act) {
    case D2D_RELU: return fmaxf(h, 0.0f);
    case D2D_GELU: return h * 0.5f * (1.0f + erff(h * 0.70710678118654752440f));
    case D2D_TANH: return tanhf(h);
    case D2D_LEAKY_RELU: return h >= 0.0f ? h : 0.01f * h;
    case D2D_GELU_TANH: {
      const float k = 0.79788456080286535588f;
      return 0.5f * h * (1.0f + tanhf(k * (h + 0.044715f * h * h * h)));
    }
    default: return h;
  }
}

// ---- vector reductions into global memory ---------------------------------
// fp32: one 16-byte red per 4 values.  bf16: packed pairs, 8 bytes per red.
__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void red_add_v4(bf16* p, float a, float b, float c, float d) {
  uint32_t lo = pack_bf16x2(a, b), hi = pack_bf16x2(c, d);
  asm volatile("red.global.add.noftz.v2.bf16x2 [%0], {%1, %2};" ::"l"(p), "r"(lo), "r"(hi)
               : "memory");
}
// eight bf16 sums in pairs, each rounded once
__device__ __forceinline__ uint4 add_bf16x8(uint4 a, uint4 b) {
  uint4 r;
  const __nv_bfloat162* x = reinterpret_cast<const __nv_bfloat162*>(&a);
  const __nv_bfloat162* y = reinterpret_cast<const __nv_bfloat162*>(&b);
  __nv_bfloat162* z = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) z[i] = __hadd2_rn(x[i], y[i]);
  return r;
}
__device__ __forceinline__ void red_add_1(float* p, float a) { atomicAdd(p, a); }
__device__ __forceinline__ void red_add_1(bf16* p, float a) { atomicAdd(p, __float2bfloat16_rn(a)); }

// bits i (even experts) and 16 + i (odd experts) -> bits 2i and 2i + 1
__device__ __forceinline__ uint32_t interleave16(uint32_t v) {
  uint32_t t = (v ^ (v >> 8)) & 0x0000ff00u;
  v ^= t ^ (t << 8);
  t = (v ^ (v >> 4)) & 0x00f000f0u;
  v ^= t ^ (t << 4);
  t = (v ^ (v >> 2)) & 0x0c0c0c0cu;
  v ^= t ^ (t << 2);
  t = (v ^ (v >> 1)) & 0x22222222u;
  return v ^ t ^ (t << 1);
}

// 32 x 32 bit matrix, one row per lane, turned over: bit i of lane b's result = bit b of lane i's
// word (block swaps of size 16, 8, 4, 2, 1)
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) == 0 ? (x & m) | ((y & m) << j) : (x & ~m) | ((y >> j) & m);
    m ^= m << (j >> 1);
  }
  return x;
}

__host__ __device__ __forceinline__ int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ __forceinline__ int64_t ceil_div64(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace d2d

// ---- internal launch interface (host side, used by d2d_abi.cu) -------------
namespace d2d {

// Optional by-product of the expert kernels: per (expert, token) vector norms over the last
// dimension of what the expert computes for that token, norms[e * N + token] in the tensor
// dtype (the labels router training captures with forward hooks upstream, utils.py:353-369).
struct NormCapture {
  void* norms = nullptr;   // [E, N]; entries of pairs outside the token lists are left alone
  int layer = 0;           // 0 none, D2D_NORM_OF_INTERMEDIATE, D2D_NORM_OF_OUTPUT
  int ord = 2;             // 1 (sum of magnitudes) or 2 (Euclidean)
};

int launch_router_mask_simt(const void* x, const void* wa, const void* wb, float mult,
                            uint32_t* mask_bits, void* scores, const void* last_bias,
                            int add_residual, void* out_init, int64_t N, int d, int R, int E,
                            int dtype, int* dev_status, cudaStream_t s, void* rt_out = nullptr);
int launch_gate_rule(const void* scores, int rule, int k, float tau, uint32_t* mask_bits,
                     int64_t N, int E, int dtype, cudaStream_t s);
int launch_mask_from_scores(const void* scores, float mult, uint32_t* mask_bits, int64_t N, int E,
                            int dtype, int* dev_status, cudaStream_t s);
// rule 0: dynk_max with threshold multiplier mult; D2D_RULE_TOPK (k), D2D_RULE_DYNK (tau).
// direct: initial rows only of tokens not kept by exactly one expert.  *lists: in, token_idx and
// offsets may be written here as well (short calls); out, they were
struct ListsOut {
  int32_t* token_idx = nullptr;
  int32_t* offsets = nullptr;
  bool written = false;
  void* table = nullptr;       // in: memory for a mask table that may be written instead (long calls)
  bool tabled = false;         // out: it was
};

// What an expert kernel that makes its own lists reads: the counts table of the compaction, and the mask
// turned over, per 128-token tile and expert the four words whose bit t says that token 32 q + t of the
// tile keeps the expert.  A tile's entries lie together: whole sectors are written at once.
struct MaskTable {
  uint8_t* counts;             // [ntiles][EP]
  uint4* words;                // [ntiles][E]
  int ntiles, EP;
};
constexpr int TABLE_CHUNKS = 15;                       // parts in which its readers count it,
constexpr int64_t TABLE_MAX_TILES = 511 * TABLE_CHUNKS;    // each with 16-bit sums
MaskTable mask_table(void* mem, int64_t N, int E);
size_t mask_table_bytes(int64_t N, int E);
int launch_gate_scores_fused(const void* scores, int rule, int k, float tau, float mult,
                             uint32_t* mask_bits, void* rt, int32_t* tile_counts, const void* x,
                             const void* last_bias, int add_residual, void* out, bool direct,
                             int64_t N, int d, int E, int dtype, cudaStream_t s, ListsOut* lists);
int launch_all_experts(uint32_t* mask_bits, void* rt, int32_t* token_idx, int32_t* offsets,
                       const void* x, const void* last_bias, int add_residual, void* out,
                       int64_t N, int d, int E, int dtype, cudaStream_t s);
int launch_init_out(const void* x, const void* last_bias, int add_residual, void* out, int64_t N,
                    int d, int dtype, cudaStream_t s);
int launch_prenorm_init(const void* x, const void* gamma, const void* beta, float eps, int kind,
                        float gamma_offset, const void* last_bias, void* xn, void* out, int64_t N,
                        int d, int dtype, cudaStream_t s);
int launch_expand_mask(const uint32_t* mask_bits, void* rt, int64_t N, int E, int dtype,
                       cudaStream_t s);
int launch_pack_mask(const void* rt, uint32_t* mask_bits, int64_t N, int E, int dtype,
                     cudaStream_t s);
// SM count of the current device, and the dynamic shared memory opt-in of `kernel` on it (both
// hold per device and are looked up once; safe from several host threads)
int device_launch_facts(const void* kernel, size_t smem, int* sms);
size_t compact_workspace_bytes(int64_t n_max, int E);
int compact_row_cells(int E);      // cells (bytes) per row of the compaction's counts table
bool compact_counts_itself(int64_t N, int E);   // no count kernel needed
// counts_ready: the byte table counts_ws[tile of 128 tokens][compact_row_cells(E)] is already
// filled (by the router kernel); otherwise a count kernel fills it first
int launch_compact(const uint32_t* mask_bits, int32_t* token_idx, int32_t* offsets, int64_t N,
                   int E, int32_t* counts_ws, int* dev_status, cudaStream_t s,
                   bool counts_ready);
// fp32 with 16-byte vectors everywhere, else D2D_ERR_UNSUPPORTED
int launch_router_fp32(const void* x, const void* wa, const void* wb, float mult,
                       uint32_t* mask_bits, void* scores, void* rt, const void* last_bias,
                       int add_residual, void* out_init, int64_t N, int d, int R, int E,
                       cudaStream_t s);
int launch_experts_fp32(const void* x, const int32_t* token_idx, const int32_t* offsets,
                        const void* w1, const void* b1, const void* w2, void* out, int64_t N, int d,
                        int E, int H, int act, int* dev_status, cudaStream_t s, int kept);
// kept: experts that a token keeps, 0 where the rule leaves it open
int launch_experts_simt(const void* x, const int32_t* token_idx, const int32_t* offsets,
                        const void* w1, const void* b1, const void* w_up, const void* w2,
                        void* out, int64_t N, int d, int E, int H, int act, int dtype,
                        int* dev_status, cudaStream_t s, NormCapture nc = NormCapture(), int kept = 0);

}  // namespace d2d
