// The top-k and cumulative-share rules on one token's scores, in one thread's registers:
//   D2D_RULE_TOPK      k times the first largest of the scores not yet taken
//   D2D_RULE_DYNK      the same on the shares, until their running sum reaches tau
// (order of equal values, NaN, summation and rounding as in gate_rule_kernel).
#pragma once
#include "d2d_common.cuh"

namespace d2d {

template <typename T> struct Acc { typedef float type; };
template <> struct Acc<float> { typedef double type; };

// sv[EMAX], the first E of them scores; sets the bits of the kept experts in word[2].  All lanes of
// the warp call it.
template <typename T, int EMAX, int RULE>
__device__ __forceinline__ void ranked_words(const T* sv, int E, int k, float tau, uint32_t* word) {
  float v[EMAX];
#pragma unroll
  for (int e = 0; e < EMAX; ++e) v[e] = DT<T>::to_f(sv[e]);
  bool negative = false;
  if (RULE == D2D_RULE_DYNK) {
    float s[32];                     // the balanced sum a warp's butterfly makes of 32 lanes
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      s[l] = 0.f;
#pragma unroll
      for (int e = l; e < EMAX; e += 32)
        if (e < E) s[l] += v[e];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int l = 0; l < o; ++l) s[l] += s[l + o];
    const float tot = DT<T>::round(s[0]);
#pragma unroll
    for (int e = 0; e < EMAX; ++e) {
      v[e] = DT<T>::round(v[e] / tot);
      negative |= e < E && v[e] < 0.f;
    }
  }
  const float tau_t = DT<T>::round(tau);
  const int most = RULE == D2D_RULE_TOPK ? k : E;
  uint32_t taken[2] = {0u, 0u};
  typename Acc<T>::type acc = 0;
  bool more = true;                  // the expert of the next rank is kept
  for (int r = 0; r < most; ++r) {
    float m = 0.f;
    int best = -1;
#pragma unroll
    for (int e = 0; e < EMAX; ++e) {
      const bool free = e < E && !((taken[e >> 5] >> (e & 31)) & 1u);
      if (free && (best < 0 || v[e] > m || (v[e] != v[e] && m == m))) {
        m = v[e];
        best = e;
      }
    }
    const uint32_t b0 = best < 32 ? 1u << (best & 31) : 0u;
    const uint32_t b1 = best >= 32 ? 1u << (best & 31) : 0u;
    taken[0] |= b0;
    taken[1] |= b1;
    if (more) {
      word[0] |= b0;
      word[1] |= b1;
    }
    if (RULE == D2D_RULE_DYNK) {
      acc += m;
      more = DT<T>::round((float)acc) < tau_t;
      // without negative shares the running sum only grows
      if (!__any_sync(0xffffffffu, more || negative)) break;
    }
  }
}

}  // namespace d2d
