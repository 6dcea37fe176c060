// What the tensor-core expert kernels share: the packed weights' layout, the hidden epilogue's
// arithmetic and the output instruction.
#pragma once
#include "d2d_umma_api.cuh"
#include "d2d_umma_ptx.cuh"

namespace d2d {
namespace umma {

constexpr int MAX_E = 128;
constexpr int NS_MAX = 8, NS2_MAX = 8;        // stages of the two rings (upper bounds)
constexpr int SMEM_TILES = 212 * 1024;        // both rings

struct Geo {
  int kc1;         // d / 64
  int w1_stage;    // W1 (and W_up) bytes per 64-deep slice
  int kc2;         // ceil(H / 64)
  int nd, nc;      // output columns per step of the second product, steps
  int ns, ns2;     // ring stages
  int a_slot;      // bytes of a stage's rows of x
  int stage;       // bytes of a stage of the first ring: a_slot, then w1_stage
  int w2_piece;    // W2 bytes of a step's 64-deep slice (one stage of the second ring)
  long long w1_bytes, bias_off, stride;   // packed layout per expert
};

// n: tokens of the call.  A list has at most n rows, so with n <= 32 (64) a tile needs only the first
// quarter (half) of its 16 KB of x: the MMA still reads 128 rows, but what stands in the other
// rows' place reaches only accumulator rows nobody reads.  A decode step of the gated form keeps
// four stages of weights in flight instead of three.
inline Geo experts_geo(int d, int H, bool glu, long long n) {
  Geo g;
  g.kc1 = d / 64;
  g.w1_stage = (glu ? 2 : 1) * H * 128;
  g.kc2 = (H + 63) / 64;
  g.nd = !glu && d % 128 == 0 ? 128 : 64;
  g.nc = d / g.nd;
  g.a_slot = n <= 32 ? SLOT / 4 : n <= 64 ? SLOT / 2 : SLOT;
  g.stage = g.a_slot + g.w1_stage;
  g.w2_piece = g.nd * 128;
  // 48 KB of W2 pieces, then as many stages of the first ring as fit, the rest for W2
  const int ns = (SMEM_TILES - 48 * 1024) / g.stage;
  g.ns = ns < NS_MAX ? ns : NS_MAX;
  const int ns2 = (SMEM_TILES - g.ns * g.stage) / g.w2_piece;
  g.ns2 = ns2 < NS2_MAX ? ns2 : NS2_MAX;
  g.w1_bytes = (long long)g.kc1 * g.w1_stage;
  g.bias_off = g.w1_bytes + (long long)g.nc * g.kc2 * g.w2_piece;
  g.stride = (g.bias_off + 512 + 1023) / 1024 * 1024;
  return g;
}

// 16 hidden columns as 8 packed bf16 pairs, with the upstream rounding points
// (T(x W1), + b1, activation, x T(x W_up)) done in packed bf16 arithmetic: one
// float->bf16x2 conversion per pair instead of one conversion per rounding point.
// NORM: nacc also collects the row's norm terms of the activation (before the gating
// product), 1 = magnitudes, 2 = squares.
template <int ACT, bool GLU, bool NORM>
__device__ __forceinline__ void ep1_pairs(const uint32_t* v, const uint32_t* u, const uint32_t* bp,
                                          uint32_t* w, float& nacc, int nord) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    __nv_bfloat162 h =
        __floats2bfloat162_rn(__uint_as_float(v[2 * q]), __uint_as_float(v[2 * q + 1]));
    h = __hadd2_rn(h, *reinterpret_cast<const __nv_bfloat162*>(&bp[q]));
    if (ACT == D2D_RELU) {
      h = __hmax2(h, __float2bfloat162_rn(0.f));
    } else {
      const float2 f = __bfloat1622float2(h);
      h = __floats2bfloat162_rn(activate(f.x, ACT), activate(f.y, ACT));
    }
    if (NORM) {
      const float2 f = __bfloat1622float2(h);
      nacc += nord == 1 ? fabsf(f.x) + fabsf(f.y) : fmaf(f.x, f.x, f.y * f.y);
    }
    if (GLU) {
      const __nv_bfloat162 uu =
          __floats2bfloat162_rn(__uint_as_float(u[2 * q]), __uint_as_float(u[2 * q + 1]));
      h = __hmul2_rn(h, uu);
    }
    w[q] = *reinterpret_cast<uint32_t*>(&h);
  }
}

// Row n of a packed W2 piece holds this output column of the piece: in each block of 32 the two 2-bit
// fields above the lowest bit change places, so that column 8 f + 2 l + i of the accumulator, which
// the fragment loads give to lane l of a row, is output column 8 l + 2 f + i.
__host__ __device__ __forceinline__ int out_column(int n) {
  return (n & ~30) | ((n & 6) << 2) | ((n >> 2) & 6);
}

// t >= 0: add; t < -1: store; -1: nothing (predicated, no branch)
__device__ __forceinline__ void put_row(void* p, int t, uint4 add, uint4 st) {
  asm volatile(
      "{\n\t.reg .pred a, b;\n\t"
      "setp.ge.s32 a, %1, 0;\n\t"
      "setp.lt.s32 b, %1, -1;\n\t"
      "@a red.global.add.noftz.v4.bf16x2 [%0], {%2, %3, %4, %5};\n\t"
      "@b st.global.v4.b32 [%0], {%6, %7, %8, %9};\n\t}" ::"l"(p),
      "r"(t), "r"(add.x), "r"(add.y), "r"(add.z), "r"(add.w), "r"(st.x), "r"(st.y), "r"(st.z),
      "r"(st.w)
      : "memory");
}

// t >= 0: add
__device__ __forceinline__ void add_row(void* p, int t, uint4 v) {
  asm volatile(
      "{\n\t.reg .pred a;\n\t"
      "setp.ge.s32 a, %1, 0;\n\t"
      "@a red.global.add.noftz.v4.bf16x2 [%0], {%2, %3, %4, %5};\n\t}" ::"l"(p),
      "r"(t), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
      : "memory");
}

}  // namespace umma

// Short calls (d2d_experts_short.cu)
bool experts_short_supported(int64_t N, int d, int E, int H, bool glu, int kept);
int launch_experts_short(const void* x, const int32_t* token_idx, const int32_t* offsets,
                         const void* packed, void* out, int64_t N, int d, int E, int H, bool glu,
                         int act, int* dev_status, cudaStream_t s, DirectRows dr);

}  // namespace d2d
