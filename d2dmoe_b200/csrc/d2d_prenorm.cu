// Pre-norm fused with the block's residual: the pass in front of the MoE-FFN layer.
//
// An upstream transformer block runs   y = ln_2(x);  y = mlp(y);  return x + y
// (architectures/moe/moe_models.py:69-76 ViT, :91-100 GPT, :148-156 Gemma with RMSNorm), i.e.
// a normalisation pass over [N, d] before the layer and a residual-add pass after it.  Here
// ONE pass reads x once and writes both
//     xn[t,:]  = T(norm(x[t,:]))                       the layer's input (router and expert gather)
//     out[t,:] = T(x[t,:] + last_bias)                 the layer output's initial value,
// after which the layer only adds the expert contributions to `out`
// (d2d_moe_forward with add_residual = D2D_OUT_PREINITIALISED): the separate residual pass and the
// router's initial-value writes disappear.
//
//   kind 0  LayerNorm: (x - mean) * rsqrt(var + eps) * gamma + beta   (biased variance)
//   kind 1  RMSNorm:   x * rsqrt(mean(x^2) + eps) * (gamma_offset + gamma)
//           (gamma_offset = 1 for the Gemma form, transformers GemmaRMSNorm; 0 for the plain form)
// Statistics and the affine map are evaluated in fp32, one rounding to T at the end, like the
// framework kernels they replace.  One warp per row; the row stays in registers between the
// statistics and the output (x is read once).
#include <algorithm>

#include "d2d_common.cuh"

namespace d2d {
namespace {

constexpr int NT = 256;
constexpr int MAXV = 16;      // 16-byte vectors per lane: d <= 32 * 16 * (16 / sizeof(T))

// Where gamma, beta and last_bias are when a row's statistics are there: L2, the warp's registers, or shared
// memory.  Registers save a barrier in front of the first row; they cost three vectors a lane and vector of x,
// and with them resident blocks (of bf16 d = 768 three become two, of d = 1024 one: 15 % at 7289 rows).
enum Parameters { IN_L2, IN_REGISTERS, IN_SHARED };

// MAXV_ = vectors a lane holds (the register footprint, hence the number of resident warps and
// the bytes in flight per SM, follows the row length instead of the longest row supported).
template <typename T, int MAXV_, Parameters PAR>
__global__ void __launch_bounds__(NT, PAR != IN_SHARED ? 0 : MAXV_ <= 2 || (MAXV_ == 3 && sizeof(T) == 4) ? 4 : 3)
prenorm_init_kernel(const T* __restrict__ x, const T* __restrict__ gamma,
                    const T* __restrict__ beta, float eps, int kind, float gamma_offset,
                    const T* __restrict__ last_bias, T* __restrict__ xn, T* __restrict__ out,
                    int64_t N, int d) {
  constexpr int V = 16 / sizeof(T);
  grid_launch_dependents();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int dv = d / V;                       // vectors per row
  const int nv = (dv + 31) / 32;              // vectors per lane (<= MAXV_)
  const int64_t warps = (int64_t)gridDim.x * (NT / 32);
  // Short rows (<= 4 vectors per lane) keep the NEXT row's loads in flight while the current
  // row is reduced and written: one row per warp at a time leaves too few bytes in flight.  gamma, beta and
  // last_bias are loaded once, with the first row instead of behind its statistics (Parameters).
  constexpr bool PREFETCH = PAR != IN_L2;
  uint4 raw[MAXV_], nxt[PREFETCH ? MAXV_ : 1];
  constexpr int KEPT = PAR == IN_REGISTERS ? MAXV_ : 1;
  uint4 pg[KEPT], pb[KEPT], pl[KEPT];
  __shared__ uint4 par[3][PAR == IN_SHARED ? 32 * MAXV_ : 1];
  int64_t row = (int64_t)blockIdx.x * (NT / 32) + (threadIdx.x >> 5);
  if (PREFETCH) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * d);
#pragma unroll
    for (int i = 0; i < MAXV_; ++i) {
      const int c = lane + 32 * i;
      if (row < N && i < nv && c < dv) raw[i] = __ldg(xr + c);
    }
  }
  if (PAR == IN_SHARED) {
    const int c = threadIdx.x;
    if (c < dv) {                             // (at most 128 vectors)
      const uint4 z = make_uint4(0u, 0u, 0u, 0u);
      const uint4 g = __ldg(reinterpret_cast<const uint4*>(gamma) + c);
      const uint4 b = beta ? __ldg(reinterpret_cast<const uint4*>(beta) + c) : z;
      const uint4 l = last_bias ? __ldg(reinterpret_cast<const uint4*>(last_bias) + c) : z;
      par[0][c] = g, par[1][c] = b, par[2][c] = l;
    }
    __syncthreads();
  }
  if (PAR == IN_REGISTERS) {
#pragma unroll
    for (int i = 0; i < MAXV_; ++i) {
      const int c = lane + 32 * i;
      pb[i] = pl[i] = make_uint4(0u, 0u, 0u, 0u);
      if (i < nv && c < dv) {
        pg[i] = __ldg(reinterpret_cast<const uint4*>(gamma) + c);
        if (beta) pb[i] = __ldg(reinterpret_cast<const uint4*>(beta) + c);
        if (last_bias) pl[i] = __ldg(reinterpret_cast<const uint4*>(last_bias) + c);
      }
    }
  }
  for (; row < N; row += warps) {
    if (PREFETCH) {
      if (row + warps < N) {
        const uint4* xr = reinterpret_cast<const uint4*>(x + (row + warps) * d);
#pragma unroll
        for (int i = 0; i < MAXV_; ++i) {
          const int c = lane + 32 * i;
          if (i < nv && c < dv) nxt[i] = __ldg(xr + c);
        }
      }
    } else {
      const uint4* xr = reinterpret_cast<const uint4*>(x + row * d);
#pragma unroll
      for (int i = 0; i < MAXV_; ++i) {
        const int c = lane + 32 * i;
        if (i < nv && c < dv) raw[i] = __ldg(xr + c);
      }
    }
    float sum = 0.f, sq = 0.f;
#pragma unroll
    for (int i = 0; i < MAXV_; ++i) {
      const int c = lane + 32 * i;
      if (i < nv && c < dv) {
        const T* e = reinterpret_cast<const T*>(&raw[i]);
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const float v = DT<T>::to_f(e[q]);
          sum += v;
          sq += v * v;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
    }
    float mean = 0.f, rstd;
    if (kind == 0) {
      mean = sum / (float)d;
      float var = 0.f;                        // second pass over the registers: sum (x - mean)^2
#pragma unroll
      for (int i = 0; i < MAXV_; ++i) {
        const int c = lane + 32 * i;
        if (i < nv && c < dv) {
          const T* e = reinterpret_cast<const T*>(&raw[i]);
#pragma unroll
          for (int q = 0; q < V; ++q) {
            const float dlt = DT<T>::to_f(e[q]) - mean;
            var += dlt * dlt;
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) var += __shfl_xor_sync(0xffffffffu, var, o);
      rstd = rsqrtf(var / (float)d + eps);
    } else {
      rstd = rsqrtf(sq / (float)d + eps);
    }
#pragma unroll
    for (int i = 0; i < MAXV_; ++i) {
      const int c = lane + 32 * i;
      if (i < nv && c < dv) {
        uint4 gv, bv = make_uint4(0u, 0u, 0u, 0u), lb = make_uint4(0u, 0u, 0u, 0u);
        if (PAR == IN_REGISTERS) {
          gv = pg[i], bv = pb[i], lb = pl[i];
        } else if (PAR == IN_SHARED) {
          gv = par[0][c], bv = par[1][c], lb = par[2][c];
        } else {
          gv = __ldg(reinterpret_cast<const uint4*>(gamma) + c);
          if (beta) bv = __ldg(reinterpret_cast<const uint4*>(beta) + c);
          if (last_bias) lb = __ldg(reinterpret_cast<const uint4*>(last_bias) + c);
        }
        const T* e = reinterpret_cast<const T*>(&raw[i]);
        const T* g = reinterpret_cast<const T*>(&gv);
        const T* b = reinterpret_cast<const T*>(&bv);
        const T* l = reinterpret_cast<const T*>(&lb);
        T yn[V], yo[V];
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const float v = DT<T>::to_f(e[q]);
          const float nrm = (v - mean) * rstd;
          yn[q] = DT<T>::from_f(kind == 0 ? nrm * DT<T>::to_f(g[q]) + DT<T>::to_f(b[q])
                                          : nrm * (gamma_offset + DT<T>::to_f(g[q])));
          yo[q] = DT<T>::from_f(v + DT<T>::to_f(l[q]));
        }
        *(reinterpret_cast<uint4*>(xn + row * d) + c) = *reinterpret_cast<const uint4*>(yn);
        if (out) *(reinterpret_cast<uint4*>(out + row * d) + c) = *reinterpret_cast<const uint4*>(yo);
      }
    }
    if (PREFETCH) {
#pragma unroll
      for (int i = 0; i < MAXV_; ++i) raw[i] = nxt[i];
    }
  }
}

// Rows of at most four vectors a lane.  Parameters in registers where four blocks fit an SM with them (one vector;
// two of fp32) or there are one and a half blocks an SM at most, else in shared memory.  The grid is four blocks
// per SM, so that a warp has several rows for one reading; six from three rows a warp on in the form that holds
// three or four; and 16 where the hardware spreads many rows better (the lines differ by type, see `many`).
// Half a block, 24 experts x 128, replayed, us: parameters from L2 for each row in 16 blocks per SM / in registers in
// four / by this rule.
//   bf16 d       197 rows             1576               7289               17 730              50 432
//     512   18.4 / 18.3 / 18.2  23.5 / 22.7 / 22.7  31.2 / 31.1 / 29.9  45.1 / 44.1 / 43.2  92.3 / 91.8 / 90.3
//     768   21.0 / 20.7 / 20.7  27.3 / 27.0 / 26.8  39.6 / 39.1 / 38.2  60.3 / 56.2 / 56.3   133 / 127 / 128
//    1024   24.0 / 23.4 / 23.1  31.9 / 30.2 / 30.4  47.5 / 49.1 / 45.4  74.8 / 76.0 / 70.7   174 / 172 / 167
// This kernel alone, fp32, 100 352 rows: d = 64 20.8 / 21.9 / 19.5, 256 50.2 / 55.5 / 49.6, 512 96.5 / 106 / 96.8.
template <typename T, int NV>
int launch_rows(int64_t blocks, int sms, cudaStream_t s, const T* x, const T* gamma, const T* beta, float eps,
                int kind, float gamma_offset, const T* last_bias, T* xn, T* out, int64_t N, int d) {
  auto launch = [&](auto kernel, int64_t grid) {
    return launch_pdl(kernel, dim3((unsigned)grid), dim3(NT), 0, s, x, gamma, beta, eps, kind, gamma_offset,
                      last_bias, xn, out, N, d);
  };
  const int64_t spread = std::min<int64_t>(blocks, 16 * (int64_t)sms);
  if constexpr (NV > 4) {
    return launch(prenorm_init_kernel<T, NV, IN_L2>, spread);
  } else {
    constexpr bool f32 = sizeof(T) == 4;
    constexpr bool one_form = NV == 1 || (f32 && NV == 2);
    const int64_t rows = blocks / (4 * (int64_t)sms);        // of a warp, four blocks per SM
    const bool many = NV == 1 ? f32 && rows >= 8 : rows >= (f32 ? 4 : 8);
    auto grid = [&](int per_sm) { return many ? spread : std::min<int64_t>(blocks, per_sm * (int64_t)sms); };
    if constexpr (!one_form)
      if (2 * blocks > 3 * (int64_t)sms)
        return launch(prenorm_init_kernel<T, NV, IN_SHARED>, grid(rows >= 3 ? 6 : 4));
    return launch(prenorm_init_kernel<T, NV, IN_REGISTERS>, grid(4));
  }
}

}  // namespace

int launch_prenorm_init(const void* x, const void* gamma, const void* beta, float eps, int kind,
                        float gamma_offset, const void* last_bias, void* xn, void* out, int64_t N,
                        int d, int dtype, cudaStream_t s) {
  const int V = dtype == D2D_F32 ? 4 : 8;
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (d % V != 0 || d / V > 32 * MAXV) return D2D_ERR_UNSUPPORTED;
  if (!al16(x) || !al16(gamma) || !al16(beta) || !al16(last_bias) || !al16(xn) || !al16(out))
    return D2D_ERR_BAD_ARG;
  int sms = 0;
  const int rc = device_launch_facts(nullptr, 0, &sms);
  if (rc != D2D_OK) return rc;
  const int nv = (d / V + 31) / 32;
  const int64_t blocks = std::max<int64_t>(ceil_div64(N, NT / 32), 1);      // a row for each warp
#define D2D_PRENORM_CASE(T_, NV_)                                                               \
  return launch_rows<T_, NV_>(blocks, sms, s, (const T_*)x, (const T_*)gamma, (const T_*)beta,  \
                              eps, kind, gamma_offset, (const T_*)last_bias, (T_*)xn, (T_*)out, N, d)
#define D2D_PRENORM_BY_NV(T_)                                                                  \
  do {                                                                                         \
    if (nv <= 1) D2D_PRENORM_CASE(T_, 1);                                                      \
    else if (nv <= 2) D2D_PRENORM_CASE(T_, 2);                                                 \
    else if (nv <= 3) D2D_PRENORM_CASE(T_, 3);                                                 \
    else if (nv <= 4) D2D_PRENORM_CASE(T_, 4);                                                 \
    else if (nv <= 8) D2D_PRENORM_CASE(T_, 8);                                                 \
    else D2D_PRENORM_CASE(T_, MAXV);                                                           \
  } while (0)
  if (dtype == D2D_F32) D2D_PRENORM_BY_NV(float);
  else D2D_PRENORM_BY_NV(bf16);
#undef D2D_PRENORM_BY_NV
#undef D2D_PRENORM_CASE
}

}  // namespace d2d
