// fp32 kernels of the layer for aligned shapes: router + dynk_max rule, and expert FFN.
//
// True fp32 products (upstream forbids TF32 there, architectures/moe/moe_impls.py:153,288), so
// FFMA.  What bounds them at the sizes fp32 is used at (1576 tokens: 0.16 + 0.47 GFMA, 17 us of the
// chip's FFMA rate) is how evenly the work spreads over 148 SMs and what a warp reads from shared
// memory per FMA.  Both kernels are made of one product: 32 rows x 32 hidden columns over all of d,
// 128 threads, the four warps and the two halves of each splitting every 64-deep chunk of d
// eightfold, 8 x 8 outputs per lane: 16 vector reads per 256 FMAs (the general-shape kernels' 4 x 4
// tiles need 32, which is what bounds them), and 4 times as many work items as with all of a
// 128-wide hidden layer in one.
//   router   a cluster of four CTAs has 32 tokens; each takes every fourth slice of 32 hidden
//            columns and the scores' share of it; the shares meet through distributed shared memory
//   experts  an item is (expert, 32 rows of its list, 32 hidden columns); it adds its share of the
//            second product to the output rows.  In fp32 nothing is rounded between the
//            slices, so no exchange is needed; the price is one add of the output rows per slice.
// Measured (1576 tokens x 768, 24 experts x 128, router 128): router 23.7, experts 52.9 us, the layer 78.5
// as a graph replay; with the general-shape kernels 34.2, 80.5 and 115.
#include <cooperative_groups.h>

#include "d2d_common.cuh"

namespace d2d {
namespace {

namespace cg = cooperative_groups;

constexpr int NT = 128;
constexpr int TR = 32;             // rows of an item
constexpr int TH = 32;             // hidden columns of an item
constexpr int KC = 64;             // depth of a staged chunk
constexpr int KP = KC + 4;         // row pitch of [row][k] tiles: 8 rows, 8 bank groups
constexpr int CP = TH + 4;         // row pitch of [.][column] tiles
constexpr int ST = 3;              // stages
constexpr int CLUSTER = 4;
constexpr int MAX_E = 256;
constexpr int A_FLOATS = TR * KP;
constexpr int B_FLOATS = KC * CP > TH * KP ? KC * CP : TH * KP;
constexpr int STAGE_FLOATS = A_FLOATS + B_FLOATS;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// 16 bytes, or zeros where !ok
__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
               "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Sums of the 32 x 32 product, thread t: row t / 4, columns 8 (t % 4) .. + 7.
// load(stage, chunk) issues this thread's copies of one chunk; BT: the B tile is [column][k] (its
// rows permuted by b_row) instead of [k][column].
__device__ __forceinline__ int b_row(int col) {      // column 16 j + 4 cg + c -> row cg + 4 (4 j + c)
  return ((col >> 2) & 3) + 4 * (4 * (col >> 4) + (col & 3));
}
template <bool BT, typename Load>
__device__ __forceinline__ void product32(float* sm, int chunks, Load load, float* sum) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int kh = lane >> 4, rg = (lane >> 2) & 3, cgp = lane & 3;
  const int k0 = (w * 2 + kh) * 8;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) {
    if (s < chunks) load(sm + s * STAGE_FLOATS, s);
    cp_commit();
  }
  int st = 0;
  for (int c = 0; c < chunks; ++c) {
    cp_wait<ST - 2>();
    __syncthreads();                   // chunk c is here; everybody is done with chunk c - 1
    int nst = st + ST - 1;
    if (nst >= ST) nst -= ST;
    if (c + ST - 1 < chunks) load(sm + nst * STAGE_FLOATS, c + ST - 1);
    cp_commit();
    const float* A = sm + st * STAGE_FLOATS;
    const float* B = A + A_FLOATS;
#pragma unroll
    for (int kk = 0; kk < 8; kk += 4) {
      const int k = k0 + kk;
      float4 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        a[i] = *reinterpret_cast<const float4*>(A + (rg + 4 * i) * KP + k);
      if (BT) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 b = *reinterpret_cast<const float4*>(B + (cgp + 4 * j) * KP + k);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
            acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
            acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
            acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 b0 = *reinterpret_cast<const float4*>(B + (k + q) * CP + 4 * cgp);
          const float4 b1 = *reinterpret_cast<const float4*>(B + (k + q) * CP + 16 + 4 * cgp);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float av = q == 0 ? a[i].x : q == 1 ? a[i].y : q == 2 ? a[i].z : a[i].w;
            acc[i][0] = fmaf(av, b0.x, acc[i][0]);
            acc[i][1] = fmaf(av, b0.y, acc[i][1]);
            acc[i][2] = fmaf(av, b0.z, acc[i][2]);
            acc[i][3] = fmaf(av, b0.w, acc[i][3]);
            acc[i][4] = fmaf(av, b1.x, acc[i][4]);
            acc[i][5] = fmaf(av, b1.y, acc[i][5]);
            acc[i][6] = fmaf(av, b1.z, acc[i][6]);
            acc[i][7] = fmaf(av, b1.w, acc[i][7]);
          }
        }
      }
    }
    st = st + 1 == ST ? 0 : st + 1;
  }
  cp_wait<0>();
  // the two halves of a warp, then the four warps (partials in the stage area)
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] += __shfl_xor_sync(0xffffffffu, acc[i][j], 16);
  __syncthreads();
  float* P = sm + w * TR * CP;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if ((i >> 2) != kh) continue;      // each half writes four of the eight rows
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<float4*>(P + (rg + 4 * i) * CP + 16 * j + 4 * cgp) =
          make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
  }
  __syncthreads();
  const int row = tid >> 2, c0 = 8 * (tid & 3);
#pragma unroll
  for (int q = 0; q < 8; ++q) sum[q] = 0.f;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const float4 p0 = *reinterpret_cast<const float4*>(sm + (v * TR + row) * CP + c0);
    const float4 p1 = *reinterpret_cast<const float4*>(sm + (v * TR + row) * CP + c0 + 4);
    sum[0] += p0.x; sum[1] += p0.y; sum[2] += p0.z; sum[3] += p0.w;
    sum[4] += p1.x; sum[5] += p1.y; sum[6] += p1.z; sum[7] += p1.w;
  }
}
static_assert(4 * TR * CP <= ST * STAGE_FLOATS, "partials fit the stage area");

__device__ __forceinline__ float nanmax(float a, float b) {
  return (a != a || b != b) ? __int_as_float(0x7fc00000) : fmaxf(a, b);
}

// ---------------------------------------------------------------------------
// router
// ---------------------------------------------------------------------------
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(NT, 2)
router_fp32_kernel(const float* __restrict__ x, const float* __restrict__ wa,
                   const float* __restrict__ wb, float mult, uint32_t* __restrict__ mask_bits,
                   float* __restrict__ scores, float* __restrict__ rt,
                   const float* __restrict__ last_bias, int add_residual,
                   float* __restrict__ out_init, int64_t N, int d, int R, int E) {
  extern __shared__ __align__(16) float sm[];
  float* hs = sm + ST * STAGE_FLOATS;         // [TR][CP] hidden slice
  float* share = hs + TR * CP;                // [TR][EP] this CTA's share of the scores
  const int EP = E + 1;
  float* wbs = share + ((TR * EP + 3) & ~3);  // [E][CP] the slice's columns of Wb
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t t0 = (int64_t)(blockIdx.x / CLUSTER) * TR;
  grid_launch_dependents();
  grid_dependency_wait();
  for (int i = tid; i < TR * EP; i += NT) share[i] = 0.f;
  const int slices = (R + TH - 1) / TH;
  for (int sl = rank; sl < slices; sl += CLUSTER) {
    // Wb's columns of the slice, with the first chunk (8 vectors per expert; past R: zeros)
    for (int i = tid; i < E * 8; i += NT) {
      const int c = sl * TH + (i & 7) * 4;
      cp16(wbs + (i >> 3) * CP + (i & 7) * 4, c < R ? wb + (int64_t)(i >> 3) * R + c : wb, c < R);
    }
    auto load = [&](float* stage, int chunk) {
      float* A = stage;
      float* B = stage + A_FLOATS;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + NT * u, r = i >> 4, kq = (i & 15) * 4, k = chunk * KC + kq;
        const int64_t t = t0 + r;
        const bool okx = t < N && k < d, okw = sl * TH + r < R && k < d;
        cp16(A + r * KP + kq, okx ? x + t * d + k : x, okx);
        cp16(B + b_row(r) * KP + kq, okw ? wa + (int64_t)(sl * TH + r) * d + k : wa, okw);
      }
    };
    float h[8];
    product32<true>(sm, (d + KC - 1) / KC, load, h);
    const int row = tid >> 2, c0 = 8 * (tid & 3);
#pragma unroll
    for (int q = 0; q < 8; ++q) hs[row * CP + c0 + q] = fmaxf(h[q], 0.f);
    __syncthreads();
    // scores of the slice: thread = row, experts tid % 4, + 4, ... (columns past R are zero)
    float4 hv[TH / 4];
#pragma unroll
    for (int q = 0; q < TH / 4; ++q)
      hv[q] = *reinterpret_cast<const float4*>(hs + row * CP + 4 * q);
    for (int e = tid & 3; e < E; e += 4) {
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
  // CTA r settles tokens 8 r .. 8 r + 7 of the tile, a warp two of them, lane = expert (+ 32 j)
  const int nw = (E + 31) / 32;
  const float* part[CLUSTER];
#pragma unroll
  for (int c = 0; c < CLUSTER; ++c) part[c] = cluster.map_shared_rank(share, c);
  float sc[2][MAX_E / 32];             // both tokens' shares are read before either is settled
#pragma unroll
  for (int j = 0; j < MAX_E / 32; ++j) {
    if (j >= nw) break;
    const int e = lane + 32 * j;
    float v[2][CLUSTER];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int c = 0; c < CLUSTER; ++c)
        v[u][c] = e < E ? part[c][(8 * rank + 2 * w + u) * EP + e] : 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) sc[u][j] = fabsf(((v[u][0] + v[u][1]) + v[u][2]) + v[u][3]);
  }
  static_assert(CLUSTER == 4, "sum of the shares");
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int64_t t = t0 + 8 * rank + 2 * w + u;
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
    for (int i = tid; i < 8 * (d / 4); i += NT) {
      const int64_t t = t0 + 8 * rank + i / (d / 4);
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
__global__ void __launch_bounds__(NT, 3)
experts_fp32_kernel(const float* __restrict__ x, const int32_t* __restrict__ token_idx,
                    const int32_t* __restrict__ offsets, const float* __restrict__ w1,
                    const float* __restrict__ b1, const float* __restrict__ w2,
                    float* __restrict__ out, int64_t N, int d, int E, int H, int act,
                    int* dev_status) {
  extern __shared__ __align__(16) float sm[];
  float* hs = sm + ST * STAGE_FLOATS;         // [TR][CP]
  __shared__ int off[MAX_E + 1], tstart[MAX_E + 1], rows[TR];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  grid_launch_dependents();
  grid_dependency_wait();
  for (int e = tid; e <= E; e += NT) off[e] = offsets[e];
  __syncthreads();
  if (w == 0) {                        // first tile of each expert: lane has experts 8 lane .. + 7
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
  const int slices = (H + TH - 1) / TH, total = tstart[E] * slices;
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    const int tile = item / slices, h0 = (item - tile * slices) * TH;
    int lo = 0, hi = E;                // last e with tstart[e] <= tile
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tstart[mid] <= tile) lo = mid; else hi = mid;
    }
    const int e = lo, r0 = off[e] + (tile - tstart[e]) * TR;
    const int nrows = min(TR, off[e + 1] - r0);
    __syncthreads();                   // rows, hs and the stage area of the previous item are free
    if (tid < TR) {
      int t = tid < nrows ? token_idx[r0 + tid] : -1;
      if (tid < nrows && (t < 0 || t >= N)) {
        report(dev_status, D2D_ERR_INDEX_RANGE);
        t = -1;
      }
      rows[tid] = t;
    }
    __syncthreads();
    const float* w1e = w1 + (int64_t)e * d * H + h0;
    const float* w2e = w2 + ((int64_t)e * H + h0) * d;
    auto load = [&](float* stage, int chunk) {
      float* A = stage;
      float* B = stage + A_FLOATS;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + NT * u;
        const int r = i >> 4, kq = (i & 15) * 4, k = chunk * KC + kq;      // 32 rows x 16 vectors
        const int t = rows[r];
        const bool okx = t >= 0 && k < d;
        cp16(A + r * KP + kq, okx ? x + (int64_t)t * d + k : x, okx);
        const int kr = i >> 3, cq = (i & 7) * 4, kw = chunk * KC + kr;     // 64 k x 8 vectors
        const bool okw = kw < d && h0 + cq < H;
        cp16(B + kr * CP + cq, okw ? w1e + (int64_t)kw * H + cq : w1, okw);
      }
    };
    float h[8];
    product32<false>(sm, (d + KC - 1) / KC, load, h);
    {
      const int row = tid >> 2, c0 = 8 * (tid & 3);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int c = h0 + c0 + q;
        float v = 0.f;
        if (c < H) v = activate(b1 ? h[q] + __ldg(b1 + (int64_t)e * H + c) : h[q], act);
        hs[row * CP + c0 + q] = v;
      }
    }
    __syncthreads();
    // second product: 32 rows x 256 columns per pass, K = 32; a warp has 64 columns, a lane 8 x 8
    const int rg = lane >> 3, cgp = lane & 7;
    const int kn = min(TH, H - h0);    // a multiple of 4
    for (int p0 = 0; p0 < d; p0 += 256) {
      const int c0 = p0 + 64 * w + 4 * cgp;
      const bool ok0 = c0 < d, ok1 = c0 + 32 < d;
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      float acc[8][8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
      float4 nb[4][2];                 // the next four rows of W2: each is read once per CTA
      auto fetch = [&](int k) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float* wr = w2e + (int64_t)(k + q) * d + c0;
          nb[q][0] = ok0 ? __ldg(reinterpret_cast<const float4*>(wr)) : z;
          nb[q][1] = ok1 ? __ldg(reinterpret_cast<const float4*>(wr + 32)) : z;
        }
      };
      fetch(0);
#pragma unroll 1
      for (int k = 0; k < kn; k += 4) {
        float4 b[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          b[q][0] = nb[q][0];
          b[q][1] = nb[q][1];
        }
        if (k + 4 < kn) fetch(k + 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(hs + (rg + 4 * i) * CP + k);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float av = q == 0 ? a.x : q == 1 ? a.y : q == 2 ? a.z : a.w;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              acc[i][4 * j] = fmaf(av, b[q][j].x, acc[i][4 * j]);
              acc[i][4 * j + 1] = fmaf(av, b[q][j].y, acc[i][4 * j + 1]);
              acc[i][4 * j + 2] = fmaf(av, b[q][j].z, acc[i][4 * j + 2]);
              acc[i][4 * j + 3] = fmaf(av, b[q][j].w, acc[i][4 * j + 3]);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = rows[rg + 4 * i];
        if (t < 0) continue;
        float* o = out + (int64_t)t * d + c0;
        if (ok0) red_add_v4(o, acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if (ok1) red_add_v4(o + 32, acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      }
    }
  }
}

bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

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
  const int64_t tiles = ceil_div64(N, TR);
  if (tiles * CLUSTER > 0x7fffffffLL) return D2D_ERR_UNSUPPORTED;
  const size_t smem = sizeof(float) * ((size_t)ST * STAGE_FLOATS + TR * CP + (size_t)TR * (E + 1) + 4 +
                                       (size_t)E * CP);
  const int rc = device_launch_facts((const void*)router_fp32_kernel, smem, nullptr);
  if (rc != D2D_OK) return rc;
  return launch_pdl(router_fp32_kernel, dim3((unsigned)(tiles * CLUSTER)), dim3(NT), smem, s,
                    (const float*)x, (const float*)wa, (const float*)wb, mult, mask_bits,
                    (float*)scores, (float*)rt, (const float*)last_bias, add_residual,
                    (float*)out_init, N, d, R, E);
}

int launch_experts_fp32(const void* x, const int32_t* token_idx, const int32_t* offsets,
                        const void* w1, const void* b1, const void* w2, void* out, int64_t N, int d,
                        int E, int H, int act, int* dev_status, cudaStream_t s) {
  if (d % 4 || H % 4 || E > MAX_E || !al16(x) || !al16(w1) || !al16(w2) || !al16(out))
    return D2D_ERR_UNSUPPORTED;
  const size_t smem = sizeof(float) * ((size_t)ST * STAGE_FLOATS + TR * CP);
  int sms = 0;
  const int rc = device_launch_facts((const void*)experts_fp32_kernel, smem, &sms);
  if (rc != D2D_OK) return rc;
  // three CTAs per SM; at most one item per 32 rows of an expert and slice, plus a partial one
  const int64_t most = (ceil_div64(N * (int64_t)E, TR) + E) * ceil_div(H, TH);
  const int64_t grid = most < 3 * sms ? most : 3 * sms;
  return launch_pdl(experts_fp32_kernel, dim3((unsigned)grid), dim3(NT), smem, s, (const float*)x,
                    token_idx, offsets, (const float*)w1, (const float*)b1, (const float*)w2,
                    (float*)out, N, d, E, H, act, dev_status);
}

}  // namespace d2d
