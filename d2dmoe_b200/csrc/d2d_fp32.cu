// fp32 kernels of the layer for aligned shapes: router + dynk_max rule, and expert FFN.
//
// True fp32 products (upstream forbids TF32 there, architectures/moe/moe_impls.py:153,288), on the FMA
// units.  What bounds them at the sizes fp32 is used at (1576 tokens: 0.16 + 0.47 GFMA, 17 us of the chip's
// rate) is, beside the start-up of each kernel, what a warp issues besides FMAs and how evenly items fall on 148
// SMs.  Both kernels are made of one product: 16 (32) rows x 32 hidden columns over all of d, 128 threads, the
// four warps and the two halves of each splitting every 64-deep chunk of d eightfold, 4 (8) x 8 outputs per lane.
//   * Every warp copies its own 16-deep part of a chunk into stages of its own: no barrier in the loop, and the
//     ring goes on from W1 to W2 (read directly, the second product waited for L2 24 times an item).
//   * FMAs are packed pairs (fma.rn.f32x2: each half rounded as fmaf is).  With both operands in registers
//     they reach 108 FMAs a clock and SM from one warp a scheduler on; scalar ones 91, held up by register ports.
//     The router's pairs are even and odd k, the experts' two neighbouring columns.
//   * A shared-memory read of 16 bytes a lane takes 2 clocks where no four neighbouring lanes want more than
//     two vectors, else 4, whatever is the same across the rest of the warp: hence the lanes' order.
//   router   a cluster of four CTAs has 16 tokens; each takes every fourth slice of 32 hidden
//            columns and the scores' share of it; the shares meet through distributed shared memory
//   experts  an item is (expert, 16 or 32 rows of its list, 32 hidden columns); it adds its share of the
//            second product to the output rows.  In fp32 nothing is rounded between the
//            slices, so no exchange is needed; the price is one add of the output rows per slice.
// Measured (24 experts x 768 x 128, router 128, graph replays, stages that a CTA shares -> this): 50 tokens
// 54.1 -> 29.8, 197 57.1 -> 33.8, 788 70.8 -> 52.0, 1576 74.6 -> 54.7 (router 24.5 -> 17.0, experts 49.7 -> 35.5),
// 6304 209 -> 171.
#include <cooperative_groups.h>

#include <algorithm>

#include "d2d_common.cuh"

namespace d2d {
namespace {

namespace cg = cooperative_groups;

constexpr int NT = 128;
constexpr int TH = 32;             // hidden columns of an item
constexpr int KC = 64;             // depth of a chunk: 16 for each warp
constexpr int KW = 16;
constexpr int ST = 3;              // stages of a warp
constexpr int W2_ROWS = 8;         // second product: rows of W2 in a stage, 64 columns of each
constexpr int CLUSTER = 4;
constexpr int MAX_E = 256;
constexpr int CP = TH + 4;         // row pitch of Wb's columns

// MR: rows of a lane in either product, a quarter of an item's
template <int MR>
struct Tiling {
  static constexpr int TR = 4 * MR;                       // rows of an item
  static constexpr int A_FLOATS = TR * KW;
  static constexpr int STAGE = A_FLOATS + KW * TH;        // floats of a warp's stage
  static constexpr int PART = TR * TH;                    // a warp's sums
  static constexpr int FLOATS = 4 * (ST * STAGE + PART);  // of a CTA
  // CTAs per SM of the experts' grid.  (16 rows: the tables of 64 experts and more leave room for four at a time; the
  // fifth then follows the first that is done.  A grid of four, us, five / four: 64 experts 197 tokens 48.6 / 46.2,
  // 1576 74.6 / 77.3, 6304 205 / 198, 12 608 358 / 370; 96 experts x 32 197 tokens 32.1 / 34.6; 128 experts 788 69.8 / 82.5;
  // 64 of d = 2048 4096 tokens 383 / 420.)
  static constexpr int CTAS = MR == 4 ? 5 : 3;
  static_assert(W2_ROWS * 64 <= STAGE, "a stage holds a piece of W2");
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp16(uint32_t dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// 16 bytes, or zeros where !ok
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// two fp32 FMAs in one instruction: (c.lo + a.lo b.lo, c.hi + a.hi b.hi), each rounded once as fmaf is
using pair = unsigned long long;
__device__ __forceinline__ pair fma2(pair a, pair b, pair c) {
  pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ pair twice(float a) {
  pair d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
  return d;
}
__device__ __forceinline__ float2 halves(pair a) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(a));
  return f;
}
__device__ __forceinline__ void ld_pairs(uint32_t p, pair* v) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "r"(p) : "memory");
}
__device__ __forceinline__ void ld_vec(uint32_t p, float* v) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(p)
               : "memory");
}
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Where the 16-byte vector v of a row is: [row][16 k] tiles (lanes read four rows' vectors 2 j and 2 j + 1 at
// once: eight bank groups) and [row][32 columns] tiles of sums.
__device__ __forceinline__ int at_k(int row, int v) { return row * KW + 4 * (v ^ (row & 2)); }
__device__ __forceinline__ int at_h(int row, int v) { return row * TH + 4 * (v ^ (row & 7)); }
// row r of a [column][16 k] tile: a lane's rows cg + 4 j are columns 16 (j / 4) + 4 cg + j % 4
__device__ __forceinline__ int b_col(int r) { return 16 * (r >> 4) + 4 * (r & 3) + ((r >> 2) & 3); }

// A warp's stages: shared-memory addresses of the one that is read and the one that is filled.  The ring goes on
// from the first product to the second one.
template <int MR>
struct Ring {
  static constexpr uint32_t BYTES = 4 * Tiling<MR>::STAGE;
  uint32_t first, cur, fill;
  __device__ __forceinline__ explicit Ring(const float* base)
      : first(smem_addr(base)), cur(first), fill(first) {}
  __device__ __forceinline__ uint32_t after(uint32_t a) const {
    return a == first + (ST - 1) * BYTES ? first : a + BYTES;
  }
};

// Sums of the TR x 32 product, thread t: row t / (32 / MR), columns MR (t % (32 / MR)) .. + MR - 1.  issue(stage, s)
// copies this warp's part of chunk s to that address (s >= chunks: what the caller wants next).  BT: the B tile is
// [column][k] (b_col) instead of [k][column].
template <int MR, bool BT, typename Issue>
__device__ __forceinline__ void product(Ring<MR>& r, float* part, int chunks, Issue issue, float* sum) {
  using T = Tiling<MR>;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int kh = lane >> 4, rg = (lane >> 1 & 1) | (lane >> 2 & 2), cg = (lane & 1) | (lane >> 1 & 2);
  // BT: pairs of even and odd k; else of two columns
  pair sums[MR][BT ? 8 : 4];
#pragma unroll
  for (int i = 0; i < MR; ++i)
#pragma unroll
    for (int j = 0; j < (BT ? 8 : 4); ++j) sums[i][j] = 0;
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) {
    issue(r.fill, s);
    r.fill = r.after(r.fill);
    cp_commit();
  }
  // (vectors 2 kk + kh: the swizzle leaves the low bit alone)
  const uint32_t a0 = 4 * at_k(rg, kh), a1 = 4 * at_k(rg, 2 + kh);
  const uint32_t b0 = 4 * T::A_FLOATS + 4 * (BT ? at_k(cg, kh) : 4 * kh * TH + 4 * (cg + 4 * kh));
  const uint32_t b1 = 4 * T::A_FLOATS + 4 * (BT ? at_k(cg, 2 + kh) : 4 * kh * TH + 4 * (cg + 4 - 4 * kh));
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    cp_wait<ST - 2>();
    __syncwarp();                      // chunk c is here, the warp is done with chunk c - 1
    issue(r.fill, c + ST - 1);
    r.fill = r.after(r.fill);
    cp_commit();
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {   // this lane's k: 8 kk + 4 kh .. + 3
      const uint32_t pa = r.cur + (kk ? a1 : a0);
      if (BT) {
        const uint32_t pb = r.cur + (kk ? b1 : b0);
        pair a[MR][2];
#pragma unroll
        for (int i = 0; i < MR; ++i) ld_pairs(pa + 16 * KW * i, a[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          pair b[2];
          ld_pairs(pb + 16 * KW * j, b);
#pragma unroll
          for (int i = 0; i < MR; ++i) sums[i][j] = fma2(a[i][0], b[0], sums[i][j]);
#pragma unroll
          for (int i = 0; i < MR; ++i) sums[i][j] = fma2(a[i][1], b[1], sums[i][j]);
        }
      } else {
        float a[MR][4];
#pragma unroll
        for (int i = 0; i < MR; ++i) ld_vec(pa + 16 * KW * i, a[i]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          pair b[4];
          ld_pairs(r.cur + b0 + 4 * TH * (8 * kk + q), b);
          ld_pairs(r.cur + b1 + 4 * TH * (8 * kk + q), b + 2);
#pragma unroll
          for (int i = 0; i < MR; ++i) {
            const pair av = twice(a[i][q]);
#pragma unroll
            for (int j = 0; j < 4; ++j) sums[i][j] = fma2(av, b[j], sums[i][j]);
          }
        }
      }
    }
    r.cur = r.after(r.cur);
  }
  float acc[MR][8];
#pragma unroll
  for (int i = 0; i < MR; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 f = halves(sums[i][BT ? j : j / 2]);
      acc[i][j] = BT ? f.x + f.y : j % 2 ? f.y : f.x;
    }
  // the two halves of a warp (each keeps half of the rows), then the four warps
#pragma unroll
  for (int i = 0; i < MR / 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float give = kh ? acc[i][j] : acc[i + MR / 2][j];
      const float keep = kh ? acc[i + MR / 2][j] : acc[i][j];
      acc[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
  float* P = part + w * T::PART;
#pragma unroll
  for (int i = 0; i < MR / 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<float4*>(P + at_h(rg + 4 * (i + kh * (MR / 2)), 4 * j + cg)) =
          make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
  __syncthreads();
  const int row = tid / (32 / MR), v0 = (MR / 4) * (tid % (32 / MR));
#pragma unroll
  for (int u = 0; u < MR / 4; ++u) {
    float* o = sum + 4 * u;
    o[0] = o[1] = o[2] = o[3] = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 p = *reinterpret_cast<const float4*>(part + k * T::PART + at_h(row, v0 + u));
      o[0] += p.x; o[1] += p.y; o[2] += p.z; o[3] += p.w;
    }
  }
}

__device__ __forceinline__ float nanmax(float a, float b) {
  return (a != a || b != b) ? __int_as_float(0x7fc00000) : fmaxf(a, b);
}

// ---------------------------------------------------------------------------
// router
// ---------------------------------------------------------------------------
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(NT, 3)
router_fp32_kernel(const float* __restrict__ x, const float* __restrict__ wa,
                   const float* __restrict__ wb, float mult, uint32_t* __restrict__ mask_bits,
                   float* __restrict__ scores, float* __restrict__ rt,
                   const float* __restrict__ last_bias, int add_residual,
                   float* __restrict__ out_init, int64_t N, int d, int R, int E) {
  constexpr int MR = 4;
  using T = Tiling<MR>;
  constexpr int TR = T::TR, TS = TR / CLUSTER;            // rows of the tile, rows this CTA settles
  extern __shared__ __align__(16) float sm[];
  float* hs = sm + 4 * ST * T::STAGE;         // sums, then [TR][TH] hidden slice in the first warp's
  float* share = sm + T::FLOATS;              // [TR][EP] this CTA's share of the scores
  const int EP = E + 1;
  float* wbs = share + ((TR * EP + 3) & ~3);  // [E][CP] the slice's columns of Wb
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t t0 = (int64_t)(blockIdx.x / CLUSTER) * TR;
  grid_launch_dependents();
  grid_dependency_wait();
  for (int i = tid; i < TR * EP; i += NT) share[i] = 0.f;
  const int slices = (R + TH - 1) / TH, chunks = (d + KC - 1) / KC;
  const int lr = lane >> 2, kl = w * KW + 4 * (lane & 3), dst = at_k(lr, lane & 3);
  for (int sl = rank; sl < slices; sl += CLUSTER) {
    // Wb's columns of the slice, with the first chunk (8 vectors per expert; past R: zeros)
    for (int i = tid; i < E * 8; i += NT) {
      const int c = sl * TH + (i & 7) * 4;
      cp16(smem_addr(wbs + (i >> 3) * CP + (i & 7) * 4), c < R ? wb + (int64_t)(i >> 3) * R + c : wb,
           c < R);
    }
    // the rows and columns this lane copies, one chunk after another (in the place of what is not there: the
    // first ones, whose sums nobody uses)
    const float *xr[TR / 8], *wr[TH / 8];
#pragma unroll
    for (int u = 0; u < TR / 8; ++u) {
      const int64_t t = t0 + lr + 8 * u;
      xr[u] = x + (t < N ? t * d : 0) + kl;
    }
#pragma unroll
    for (int u = 0; u < TH / 8; ++u) {
      const int c = sl * TH + b_col(lr + 8 * u);
      wr[u] = wa + (c < R ? (int64_t)c * d : 0) + kl;
    }
    auto issue = [&](uint32_t stage, int s) {
      const uint32_t to = stage + 4 * dst;
      if (s * KC + KC <= d) {
#pragma unroll
        for (int u = 0; u < TR / 8; ++u) cp16(to + 32 * KW * u, xr[u]);
#pragma unroll
        for (int u = 0; u < TH / 8; ++u) cp16(to + 4 * T::A_FLOATS + 32 * KW * u, wr[u]);
      } else if (s < chunks) {
        const bool in = s * KC + kl < d;
#pragma unroll
        for (int u = 0; u < TR / 8; ++u) cp16(to + 32 * KW * u, in ? xr[u] : x, in);
#pragma unroll
        for (int u = 0; u < TH / 8; ++u)
          cp16(to + 4 * T::A_FLOATS + 32 * KW * u, in ? wr[u] : wa, in);
      }
#pragma unroll
      for (int u = 0; u < TR / 8; ++u) xr[u] += KC;
#pragma unroll
      for (int u = 0; u < TH / 8; ++u) wr[u] += KC;
    };
    float h[MR];
    Ring<MR> ring(sm + w * ST * T::STAGE);
    product<MR, true>(ring, hs, chunks, issue, h);
    cp_wait<0>();                              // (Wb)
    const int row = tid / (32 / MR), v0 = (MR / 4) * (tid % (32 / MR));
#pragma unroll
    for (int u = 0; u < MR / 4; ++u) {
      const bool in = sl * TH + 4 * (v0 + u) < R;              // (R is a multiple of 4)
      *reinterpret_cast<float4*>(hs + at_h(row, v0 + u)) =
          in ? make_float4(fmaxf(h[4 * u], 0.f), fmaxf(h[4 * u + 1], 0.f), fmaxf(h[4 * u + 2], 0.f),
                           fmaxf(h[4 * u + 3], 0.f))
             : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    // scores of the slice: the threads of a row share its experts (columns past R are zero)
    float4 hv[TH / 4];
#pragma unroll
    for (int q = 0; q < TH / 4; ++q)
      hv[q] = *reinterpret_cast<const float4*>(hs + at_h(row, q));
    for (int e = tid % (32 / MR); e < E; e += 32 / MR) {
      const float* wr = wbs + e * CP;
      float a[2] = {0.f, 0.f};
#pragma unroll
      for (int q = 0; q < TH / 4; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(wr + 4 * q);
        a[q & 1] = fmaf(hv[q].x, v.x, a[q & 1]);
        a[q & 1] = fmaf(hv[q].y, v.y, a[q & 1]);
        a[q & 1] = fmaf(hv[q].z, v.z, a[q & 1]);
        a[q & 1] = fmaf(hv[q].w, v.w, a[q & 1]);
      }
      share[row * EP + e] += a[0] + a[1];
    }
    __syncthreads();
  }
  cluster.sync();
  // CTA r settles tokens TS r .. + TS - 1 of the tile, a warp SU of them, lane = expert (+ 32 j)
  constexpr int SU = TS / 4;
  const int nw = (E + 31) / 32;
  const float* part[CLUSTER];
#pragma unroll
  for (int c = 0; c < CLUSTER; ++c) part[c] = cluster.map_shared_rank(share, c);
  float sc[SU][MAX_E / 32];            // every token's shares are read before one is settled
#pragma unroll
  for (int j = 0; j < MAX_E / 32; ++j) {
    if (j >= nw) break;
    const int e = lane + 32 * j;
    float v[SU][CLUSTER];
#pragma unroll
    for (int u = 0; u < SU; ++u)
#pragma unroll
      for (int c = 0; c < CLUSTER; ++c)
        v[u][c] = e < E ? part[c][(TS * rank + SU * w + u) * EP + e] : 0.f;
#pragma unroll
    for (int u = 0; u < SU; ++u) sc[u][j] = fabsf(((v[u][0] + v[u][1]) + v[u][2]) + v[u][3]);
  }
  static_assert(CLUSTER == 4, "sum of the shares");
#pragma unroll
  for (int u = 0; u < SU; ++u) {
    const int64_t t = t0 + TS * rank + SU * w + u;
    if (t >= N) break;                 // warp-uniform
    const float* s = sc[u];
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < MAX_E / 32; ++j) {
      if (j >= nw) break;
      const int e = lane + 32 * j;
      if (e < E) {
        m = nanmax(m, s[j]);
        if (scores) scores[t * E + e] = s[j];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = nanmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float thr = __fmul_rn(m, mult);
#pragma unroll
    for (int j = 0; j < MAX_E / 32; ++j) {
      if (j >= nw) break;
      const int e = lane + 32 * j;
      const bool keep = e < E && s[j] >= thr;
      const uint32_t word = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) mask_bits[t * nw + j] = word;
      if (rt && e < E) rt[t * E + e] = keep ? 1.f : 0.f;
    }
  }
  if (out_init) {
    for (int i = tid; i < TS * (d / 4); i += NT) {
      const int64_t t = t0 + TS * rank + i / (d / 4);
      const int c = i % (d / 4);
      if (t >= N) break;
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
      if (last_bias) o = __ldg(reinterpret_cast<const float4*>(last_bias) + c);
      if (add_residual) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(x + t * d) + c);
        o = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
      }
      *(reinterpret_cast<float4*>(out_init + t * d) + c) = o;
    }
  }
  cluster.sync();                      // the others may still read this CTA's shares
}

// ---------------------------------------------------------------------------
// experts
// ---------------------------------------------------------------------------
template <int MR>
__global__ void __launch_bounds__(NT, Tiling<MR>::CTAS)
experts_fp32_kernel(const float* __restrict__ x, const int32_t* __restrict__ token_idx,
                    const int32_t* __restrict__ offsets, const float* __restrict__ w1,
                    const float* __restrict__ b1, const float* __restrict__ w2,
                    float* __restrict__ out, int64_t N, int d, int E, int H, int act,
                    int* dev_status) {
  using T = Tiling<MR>;
  constexpr int TR = T::TR;
  extern __shared__ __align__(16) float sm[];
  float* hs = sm + 4 * ST * T::STAGE;         // sums, then [TR][TH] hidden slice in the first warp's
  int* off = reinterpret_cast<int*>(sm + T::FLOATS);      // [E + 1]
  int* tstart = off + E + 1;                              // [E + 1] first tile of each expert
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  grid_launch_dependents();
  grid_dependency_wait();
  for (int e = tid; e <= E; e += NT) off[e] = offsets[e];
  __syncthreads();
  if (w == 0) {                        // lane has experts 8 lane .. + 7
    int c[MAX_E / 32], sum = 0;
#pragma unroll
    for (int q = 0; q < MAX_E / 32; ++q) {
      const int e = lane * (MAX_E / 32) + q;
      const bool bad =
          e < E && (off[e + 1] < off[e] || off[e] < 0 || off[e + 1] > N * (int64_t)E);
      if (bad) report(dev_status, D2D_ERR_INDEX_RANGE);
      c[q] = e < E && !bad ? (off[e + 1] - off[e] + TR - 1) / TR : 0;      // a bad list is dropped
      sum += c[q];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    int run = incl - sum;
#pragma unroll
    for (int q = 0; q < MAX_E / 32; ++q) {
      const int e = lane * (MAX_E / 32) + q;
      if (e <= E) tstart[e] = run;
      run += c[q];
    }
    if (lane == 31) tstart[E] = incl;
  }
  __syncthreads();
  const int slices = (H + TH - 1) / TH, chunks = (d + KC - 1) / KC, total = tstart[E] * slices;
  const int lr = lane >> 2, kl = w * KW + 4 * (lane & 3), dst = at_k(lr, lane & 3);
#pragma unroll 1
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    const int tile = item / slices, h0 = (item - tile * slices) * TH;
    int lo = 0, hi = E;                // last e with tstart[e] <= tile
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tstart[mid] <= tile) lo = mid; else hi = mid;
    }
    const int e = lo, r0 = off[e] + (tile - tstart[e]) * TR;
    const int nrows = min(TR, off[e + 1] - r0);
    int tok = lane < nrows ? token_idx[r0 + lane] : -1;   // every warp has the item's rows
    if (lane < nrows && (tok < 0 || tok >= N)) {
      if (w == 0) report(dev_status, D2D_ERR_INDEX_RANGE);
      tok = -1;
    }
    // the rows of x and the columns of the weights this lane copies, one chunk after another (in the place of
    // what is not there: the first ones, whose sums nobody uses)
    const float* xr[TR / 8];
#pragma unroll
    for (int u = 0; u < TR / 8; ++u)
      xr[u] = x + (int64_t)max(__shfl_sync(0xffffffffu, tok, lr + 8 * u), 0) * d + kl;
    const int kn = min(TH, H - h0), pieces = (kn + W2_ROWS - 1) / W2_ROWS;
    const float* w1r = w1 + ((int64_t)e * d + w * KW + (lane >> 3)) * H + h0 +
                       (4 * (lane & 7) < kn ? 4 * (lane & 7) : 0);
    const float* const w2s = w2 + ((int64_t)e * H + h0 + (lane >> 4)) * d;
    const float* w2r = w2s + min(64 * w + 4 * (lane & 15), d - 4);
    const uint32_t dst1 = 4 * (T::A_FLOATS + (lane >> 3) * TH + 4 * (lane & 7)),
                   dst1x = 4 * (T::A_FLOATS + (lane >> 3) * TH + 4 * ((lane & 7) ^ 4)),
                   dst2 = 4 * ((lane >> 4) * 64 + 4 * (lane & 15));
    int p_next = 0, k_next = 0;        // columns and rows of W2 that are copied next
    auto issue = [&](uint32_t stage, int s) {
      if (s < chunks) {
        const float* row = w1r;
        const int64_t four = 4 * (int64_t)H;
        if (s * KC + KC <= d) {
#pragma unroll
          for (int u = 0; u < TR / 8; ++u) cp16(stage + 4 * dst + 32 * KW * u, xr[u]);
#pragma unroll
          for (int u = 0; u < 4; ++u, row += four)     // k = 64 s + 16 w + 4 u + lane / 8
            cp16(stage + 16 * TH * u + (u & 1 ? dst1x : dst1), row);
        } else {
          const bool in = s * KC + kl < d;
#pragma unroll
          for (int u = 0; u < TR / 8; ++u) cp16(stage + 4 * dst + 32 * KW * u, in ? xr[u] : x, in);
#pragma unroll
          for (int u = 0; u < 4; ++u, row += four) {   // (d is a multiple of 4)
            const bool there = s * KC + w * KW + 4 * u < d;
            cp16(stage + 16 * TH * u + (u & 1 ? dst1x : dst1), there ? row : w1, there);
          }
        }
#pragma unroll
        for (int u = 0; u < TR / 8; ++u) xr[u] += KC;
        w1r += (int64_t)KC * H;
      } else if (p_next < d) {
        const float* row = w2r;
        const int64_t two = 2 * (int64_t)d;
        if (k_next + W2_ROWS <= kn) {
#pragma unroll
          for (int u = 0; u < W2_ROWS / 2; ++u, row += two) cp16(stage + dst2 + 512 * u, row);
        } else {
#pragma unroll
          for (int u = 0; u < W2_ROWS / 2; ++u, row += two) {
            const bool there = k_next + 2 * u + (lane >> 4) < kn;
            cp16(stage + dst2 + 512 * u, there ? row : w2, there);
          }
        }
        w2r += W2_ROWS * (int64_t)d;
        k_next += W2_ROWS;
        if (k_next >= kn) {
          k_next = 0;
          p_next += 256;
          w2r = w2s + min(p_next + 64 * w + 4 * (lane & 15), d - 4);
        }
      }
    };
    float h[MR];
    Ring<MR> ring(sm + w * ST * T::STAGE);
    product<MR, false>(ring, hs, chunks, issue, h);
    const int row = tid / (32 / MR), v0 = (MR / 4) * (tid % (32 / MR));
#pragma unroll
    for (int u = 0; u < MR / 4; ++u) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = h0 + 4 * (v0 + u) + q;
        float v = 0.f;
        if (c < H)
          v = activate(b1 ? h[4 * u + q] + __ldg(b1 + (int64_t)e * H + c) : h[4 * u + q], act);
        h[4 * u + q] = v;
      }
      *reinterpret_cast<float4*>(hs + at_h(row, v0 + u)) =
          make_float4(h[4 * u], h[4 * u + 1], h[4 * u + 2], h[4 * u + 3]);
    }
    __syncthreads();
    // second product: TR rows x 256 columns per pass, K = 32; a warp has 64 columns, a lane MR x 8
    const uint32_t hs0 = smem_addr(hs);
    const int rg = (lane >> 1 & 1) | (lane >> 3 & 2), cgp = (lane & 1) | (lane >> 1 & 6);
#pragma unroll 1
    for (int p0 = 0; p0 < d; p0 += 256) {
      pair sums[MR][4];
#pragma unroll
      for (int i = 0; i < MR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sums[i][j] = 0;
#pragma unroll 1
      for (int kp = 0; kp < pieces; ++kp) {
        cp_wait<ST - 2>();
        __syncwarp();
        issue(ring.fill, chunks);
        ring.fill = ring.after(ring.fill);
        cp_commit();
        const uint32_t pb = ring.cur + 16 * cgp;
#pragma unroll
        for (int kk = 0; kk < W2_ROWS / 4; ++kk) {
          float a[MR][4];
#pragma unroll
          for (int i = 0; i < MR; ++i)
            ld_vec(hs0 + 4 * at_h(rg + 4 * i, kp * (W2_ROWS / 4) + kk), a[i]);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            pair b[4];
            ld_pairs(pb + 256 * (4 * kk + q), b);
            ld_pairs(pb + 256 * (4 * kk + q) + 128, b + 2);
#pragma unroll
            for (int i = 0; i < MR; ++i) {
              const pair av = twice(a[i][q]);
#pragma unroll
              for (int j = 0; j < 4; ++j) sums[i][j] = fma2(av, b[j], sums[i][j]);
            }
          }
        }
        ring.cur = ring.after(ring.cur);
      }
      const int c0 = p0 + 64 * w + 4 * cgp;
#pragma unroll
      for (int i = 0; i < MR; ++i) {
        const int t = __shfl_sync(0xffffffffu, tok, rg + 4 * i);
        if (t < 0) continue;
        float* o = out + (int64_t)t * d + c0;
        const float2 f0 = halves(sums[i][0]), f1 = halves(sums[i][1]);
        const float2 f2 = halves(sums[i][2]), f3 = halves(sums[i][3]);
        if (c0 < d) red_add_v4(o, f0.x, f0.y, f1.x, f1.y);
        if (c0 + 32 < d) red_add_v4(o + 32, f2.x, f2.y, f3.x, f3.y);
      }
    }
    __syncthreads();                   // the hidden slice has been read
  }
}

bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int MR>
int launch_experts(const float* x, const int32_t* token_idx, const int32_t* offsets, const float* w1,
                   const float* b1, const float* w2, float* out, int64_t N, int d, int E, int H,
                   int act, int* dev_status, int sms, cudaStream_t s) {
  using T = Tiling<MR>;
  const size_t smem = sizeof(float) * (size_t)T::FLOATS + 2 * sizeof(int) * (size_t)(E + 1);
  const int rc = device_launch_facts((const void*)experts_fp32_kernel<MR>, smem, nullptr);
  if (rc != D2D_OK) return rc;
  // at most one item per TR rows of an expert and slice, plus a partial one
  const int64_t most = (ceil_div64(N * (int64_t)E, T::TR) + E) * ceil_div(H, TH);
  const int64_t ctas = (int64_t)T::CTAS * sms, grid = most < ctas ? most : ctas;
  return launch_pdl(experts_fp32_kernel<MR>, dim3((unsigned)grid), dim3(NT), smem, s, x, token_idx,
                    offsets, w1, b1, w2, out, N, d, E, H, act, dev_status);
}

}  // namespace

// Both take 16-byte vectors of x and the weights; D2D_ERR_UNSUPPORTED otherwise (the general-shape
// kernels then run).
int launch_router_fp32(const void* x, const void* wa, const void* wb, float mult,
                       uint32_t* mask_bits, void* scores, void* rt, const void* last_bias,
                       int add_residual, void* out_init, int64_t N, int d, int R, int E,
                       cudaStream_t s) {
  if (d % 4 || R % 4 || E > MAX_E || !al16(x) || !al16(wa) || !al16(wb) || !al16(last_bias) ||
      !al16(out_init))
    return D2D_ERR_UNSUPPORTED;
  using T = Tiling<4>;
  const int64_t tiles = ceil_div64(N, T::TR);
  if (tiles * CLUSTER > 0x7fffffffLL) return D2D_ERR_UNSUPPORTED;
  const size_t smem =
      sizeof(float) * ((size_t)T::FLOATS + (size_t)T::TR * (E + 1) + 4 + (size_t)E * CP);
  const int rc = device_launch_facts((const void*)router_fp32_kernel, smem, nullptr);
  if (rc != D2D_OK) return rc;
  return launch_pdl(router_fp32_kernel, dim3((unsigned)(tiles * CLUSTER)), dim3(NT), smem, s,
                    (const float*)x, (const float*)wa, (const float*)wb, mult, mask_bits,
                    (float*)scores, (float*)rt, (const float*)last_bias, add_residual,
                    (float*)out_init, N, d, R, E);
}

// Rows of an item: 16, which is what spreads a small call over the SMs, or 32 (halves the weights' way from L2 and
// what a warp reads per FMA) where lists are long or, if kept is known (experts a token keeps; 0: the threshold's
// 1.5), where 32 rows take fewer rounds of the CTAs that run at a time (such a round takes a tenth longer).
// Layer of 24 experts, us, 16 / 32 rows, mean length of a list in brackets:
//   threshold    1576 tokens (98) 53.7 / 57.8, 3152 (197) 102 / 107, 4700 (294) 147 / 134, 6304 (394) 184 / 170
//   top-2        1200 (100) 56 / 62, 1576 (131) 85 / 66, 1900 (158) 82 / 86, 2700 (225) 99 / 107, 3152 (263) 122 / 109
//   top-4        700 (117) 54 / 59, 1200 (200) 89 / 96, 1576 (263) 112 / 97, 2700 (450) 165 / 162, 5200 (867) 298 / 270
//   all experts  200 65 / 72, 260 90 / 75, 330 99 / 101, 400 111 / 108, 788 218 / 206, 4000 1028 / 936
int launch_experts_fp32(const void* x, const int32_t* token_idx, const int32_t* offsets,
                        const void* w1, const void* b1, const void* w2, void* out, int64_t N, int d,
                        int E, int H, int act, int* dev_status, cudaStream_t s, int kept) {
  if (d % 4 || H % 4 || E > MAX_E || !al16(x) || !al16(w1) || !al16(w2) || !al16(out))
    return D2D_ERR_UNSUPPORTED;
  int sms = 0;
  const int rc = device_launch_facts(nullptr, 0, &sms);
  if (rc != D2D_OK) return rc;
  const int64_t pairs = kept ? N * kept : N * 3 / 2;
  auto rounds = [&](int rows, int ctas) {      // half a tile more for each list; a twentieth left over is none
    const int64_t tiles = kept == E ? E * ceil_div64(N, rows) : pairs / rows + E / 2;
    const int64_t slots = (int64_t)ctas * sms, items = tiles * ceil_div(H, TH);
    return std::max<int64_t>(ceil_div64(items - slots / 20, slots), 1);
  };
  const bool rows32 = kept ? pairs >= 400 * (int64_t)E ||
                                 11 * rounds(32, Tiling<8>::CTAS) <= 10 * rounds(16, Tiling<4>::CTAS)
                           : pairs >= 288 * (int64_t)E;
  auto launch = rows32 ? launch_experts<8> : launch_experts<4>;
  return launch((const float*)x, token_idx, offsets, (const float*)w1, (const float*)b1,
                (const float*)w2, (float*)out, N, d, E, H, act, dev_status, sms, s);
}

}  // namespace d2d
