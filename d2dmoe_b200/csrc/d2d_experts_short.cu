// Experts of short calls (bf16, tcgen05 + TMEM): few rows per expert, so that a call is the time to
// stream the chosen experts' weights through the SMs, not products.  Same result as
// d2d_experts_umma.cu (architectures/moe/moe_impls.py:93-180, 244-301).
//
// What bounds it: the weight stream (an SM takes 64 bytes per clock) and, in the form for long lists,
// instructions whose 128 rows are mostly padding: N / 2 cycles for K = 16 whatever the rows,
// N = 2 H of a gated expert, repeated by every CTA that has a share of the output columns.  Hence
//   * both products are transposed: the WEIGHTS are the 128 rows of the instruction and the (up to
//     32) tokens its columns, 48 cycles (some 70 issued); the packed images serve as the A operand as they are;
//   * a cluster of C CTAs has an expert: each takes H / C of its hidden columns over all of d,
//     pushes its hidden slice into the others' shared memory and then takes its share of
//     the output columns with the whole hidden tile.  No weight is read twice, no partial sum is
//     rounded;
//   * gated form: gate and up rows alternate by 16, so that a warp has both of a hidden
//     column (lanes i and i + 16 trade half of their tokens);
//   * about 100 KB per CTA, two CTAs per SM: as many clusters at once as a call has experts.
//
// Warps: 0-3 both epilogues (thread = weight row = TMEM lane); 4-5 gather the token rows; 6 issues the
// products; 7 streams weights.  Tensor memory (256 columns): accumulator 1 of item i at 32 (i & 1),
// six accumulator-2 buffers from 64 on.
//
// Every wait is bounded, as in d2d_experts_umma.cu; a CTA that gave up still takes part in the last
// cluster barrier, so none leaves while another writes to it.
#include "d2d_experts_common.cuh"

namespace d2d {
using namespace umma;
namespace {

constexpr int NT = 256;
constexpr int TN = 32;                        // tokens of an item
constexpr int XB = TN * 128;                  // bytes of a stage's token rows
constexpr int RINGS = 92 * 1024;              // both rings
constexpr int S1_MAX = 10, S2 = 2;            // stages (ring 2: 16 KB each)
constexpr int HID = 2 * XB;                   // hidden tile, H <= 128
constexpr int OUTB = 4 * 2048;                // transposition blocks of the epilogue warps
constexpr int NACC2 = 6;
constexpr int TM_COLS = 256;

struct ShortParams {
  const bf16* x;
  long long N;
  int d, E, H, C;
  const uint8_t* packed;
  Geo g;
  int hs, wrows, ns, stage;        // hidden columns of a CTA, weight rows, stages and bytes of ring 1
  const int32_t* token_idx;
  const int32_t* offsets;
  bf16* out;
  const uint32_t* mask_bits;
  const bf16* last_bias;
  int* dev_status;
  uint32_t wait_limit;
  int withhold;
};

struct ShortCtl {
  unsigned long long full[S1_MAX], empty[S1_MAX], full2[S2], empty2[S2];
  unsigned long long acc1_full[2], acc1_free[2], acc2_full[NACC2], acc2_empty[NACC2];
  unsigned long long hid_full, hid_free;
  uint32_t tmem_base;
  int abort_flag;
  int wait_limit;                  // must follow abort_flag
  int total;                       // items
  int first[MAX_E];                // items before expert e
  int off[MAX_E], n[MAX_E];        // its list
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t peer(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_cluster() {
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

struct Item {
  int e, r0, rows;
};
// the expert whose items contain i (first[] ascends, an empty expert has the next one's value)
__device__ Item find_item(const ShortCtl* c, int E, int i) {
  int lo = 0, hi = E;
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (c->first[m] <= i) lo = m; else hi = m;
  }
  const int t = (i - c->first[lo]) * TN;
  const int left = c->n[lo] - t;
  return {lo, c->off[lo] + t, left < TN ? left : TN};
}
__device__ __forceinline__ int token(const ShortParams& p, int i) {
  const int t = p.token_idx[i];
  if (t >= 0 && t < p.N) return t;
  report(p.dev_status, D2D_ERR_INDEX_RANGE);
  return -1;
}

// Warps 4-5: a thread has piece t & 7 of rows t / 8 + 8 i.  Rows past the list's end stay as they
// are: what they hold reaches only accumulator columns nobody reads.
__device__ void short_gather(const ShortParams& p, ShortCtl* c, uint32_t ring, int cl, int ncl, int t) {
  volatile int* af = &c->abort_flag;
  const int j = t & 7, r8 = t >> 3;
  RingPos r = {0, 0};
  for (int it = cl; it < c->total; it += ncl) {
    const Item m = find_item(c, p.E, it);
    const bf16* src[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = r8 + 8 * i;
      const int v = row < m.rows ? token(p, m.r0 + row) : -1;
      src[i] = v < 0 ? nullptr : p.x + (size_t)v * p.d + j * 8;
    }
    for (int kc = 0; kc < p.g.kc1; ++kc) {
      if (!mbar_wait_warp(smem_u32(&c->empty[r.s]), r.ph ^ 1, af, p.dev_status)) return;
      const uint32_t dst = ring + r.s * p.stage + p.wrows * 128 + r8 * 128 + ((j ^ r8) << 4);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (src[i]) cp_async16(dst + i * 1024, src[i] + kc * 64);
      cp_async_arrive_noinc(smem_u32(&c->full[r.s]));
      r.next(p.ns);
    }
  }
}

// Warp 7: all lanes wait, lane 0 announces the bytes, the first lanes issue a copy each.
template <bool GLU>
__device__ void short_weights(const ShortParams& p, ShortCtl* c, uint32_t ring, uint32_t ring2, int cl,
                              int ncl, int rank, int s0, int s1, int lane) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  bool withheld = (p.withhold & 1) != 0 && blockIdx.x == 0;
  // ring 1: my hidden columns' rows of a slice; gated: 16 gate rows, 16 up rows, ...
  const int n1 = GLU ? p.wrows >> 4 : 1;
  const uint32_t bytes1 = GLU ? 2048 : p.wrows * 128;
  const int row1 = GLU ? ((lane & 1) ? p.H : 0) + rank * p.hs + 16 * (lane >> 1) : rank * p.hs;
  const uint32_t dst1 = GLU ? lane * 2048 : 0;
  // ring 2: 128 output columns of a 64-deep slice; two pieces where those have 64 columns
  const int n2 = 128 / g.nd;
  RingPos r1 = {0, 0}, r2 = {0, 0};
  const uint8_t* wprev = nullptr;        // the item before: its W2 follows this one's W1
  for (int it = cl; it - ncl < c->total; it += ncl) {
    const bool more = it < c->total;
    const uint8_t* w = p.packed + (more ? (long long)find_item(c, p.E, it).e * g.stride : 0);
    for (int kc = 0; more && kc < g.kc1; ++kc) {
      const uint32_t bar = smem_u32(&c->full[r1.s]);
      if (!mbar_wait_warp(smem_u32(&c->empty[r1.s]), r1.ph ^ 1, af, p.dev_status)) return;
      if (lane == 0) mbar_arrive_expect_tx(bar, p.wrows * 128);
      __syncwarp();
      if (lane < n1 && !withheld)
        bulk_g2s(ring + r1.s * p.stage + dst1, w + (long long)kc * g.w1_stage + row1 * 128, bytes1,
                 bar);
      withheld = false;                  // test hook: that stage never fills, its wait runs out
      r1.next(p.ns);
    }
    for (int s = s0; wprev && s < s1; ++s)
      for (int k2 = 0; k2 < g.kc2; ++k2) {
        const uint32_t bar = smem_u32(&c->full2[r2.s]);
        if (!mbar_wait_warp(smem_u32(&c->empty2[r2.s]), r2.ph ^ 1, af, p.dev_status)) return;
        if (lane == 0) mbar_arrive_expect_tx(bar, SLOT);
        __syncwarp();
        if (lane < n2)
          bulk_g2s(ring2 + r2.s * SLOT + lane * g.w2_piece,
                   wprev + g.w1_bytes + (long long)((s * n2 + lane) * g.kc2 + k2) * g.w2_piece,
                   g.w2_piece, bar);
        r2.next(S2);
      }
    wprev = w;
  }
}

// Warp 6, one thread.  The instruction reads 128 weight rows of a stage; where a CTA has fewer, the
// rest is whatever follows in the rings and reaches only accumulator rows nobody reads.
__device__ void short_mma(const ShortParams& p, ShortCtl* c, uint32_t ring, uint32_t ring2, uint32_t hid,
                          uint32_t tmem, int cl, int ncl, int s0, int s1) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const uint32_t idesc = instr_desc(TILE_M, TN);
  const uint64_t d0 = smem_desc(ring);
  const uint64_t hi = (d0 >> 32) << 32;
  const uint32_t lo0 = (uint32_t)d0, lo2 = (uint32_t)smem_desc(ring2), loh = (uint32_t)smem_desc(hid);
  RingPos r = {0, 0}, r2 = {0, 0}, b2 = {0, 0};
  uint32_t ctx = 0, ph = 0, hph = 0;
  // one item ahead: the first product of the next item runs while this one's hidden slices travel
  for (int it = cl; it - ncl < c->total; it += ncl) {
    if (it < c->total) {
      if (!mbar_wait_fast(smem_u32(&c->acc1_free[ctx]), ph ^ 1, af, p.dev_status)) return;
      tc_fence_after();
      for (int kc = 0; kc < g.kc1; ++kc) {
        if (!mbar_wait_fast(smem_u32(&c->full[r.s]), r.ph, af, p.dev_status)) return;
        fence_proxy_async();             // (the token rows are cp.async writes)
        tc_fence_after();
        const uint32_t alo = lo0 + r.s * ((uint32_t)p.stage >> 4), blo = alo + ((uint32_t)p.wrows << 3);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
          umma_bf16(tmem + 32 * ctx, hi | (alo + 2 * k), hi | (blo + 2 * k), idesc, (kc | k) != 0);
        umma_commit(smem_u32(&c->empty[r.s]));
        r.next(p.ns);
      }
      umma_commit(smem_u32(&c->acc1_full[ctx]));
      ph ^= ctx;
      ctx ^= 1;
    }
    // (A CTA without output columns, d < 128 C, reads no hidden tile.  Nothing would hold hid_full back
    // until it had seen a phase: its own warps hand the tile on at once, and the others may then
    // complete the next phase as well, which has the parity of the one before.)
    if (it == cl || s0 == s1) continue;
    if (!mbar_wait_fast(smem_u32(&c->hid_full), hph, af, p.dev_status)) return;
    hph ^= 1;
    fence_cluster();
    fence_proxy_all();
    for (int s = s0; s < s1; ++s) {
      if (!mbar_wait_fast(smem_u32(&c->acc2_empty[b2.s]), b2.ph ^ 1, af, p.dev_status)) return;
      for (int k2 = 0; k2 < g.kc2; ++k2) {
        if (!mbar_wait_fast(smem_u32(&c->full2[r2.s]), r2.ph, af, p.dev_status)) return;
        tc_fence_after();
        const uint32_t alo = lo2 + r2.s * (SLOT >> 4), blo = loh + k2 * (XB >> 4);
        const int ks = min(4, (p.H >> 4) - 4 * k2);
        for (int k = 0; k < ks; ++k)
          umma_bf16(tmem + 64 + 32 * b2.s, hi | (alo + 2 * k), hi | (blo + 2 * k), idesc, (k2 | k) != 0);
        umma_commit(smem_u32(&c->empty2[r2.s]));
        r2.next(S2);
      }
      umma_commit(smem_u32(&c->acc2_full[b2.s]));
      b2.next(NACC2);
    }
  }
}

// Warps 0-3: hidden slice out of accumulator 1 into every CTA's hidden tile, then the output rows
// of my columns.
template <int ACT, bool GLU>
__device__ void short_epilogues(const ShortParams& p, ShortCtl* c, uint32_t hid, uint32_t outb,
                                uint32_t tmem, int cl, int ncl, int rank, int s0, int s1, int q4,
                                int lane) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const int nw = (p.E + 31) >> 5;
  const uint32_t lanes = (uint32_t)(q4 * 32) << 16;
  constexpr int HW = GLU ? 16 : 32;                     // hidden columns of a warp
  const int h0 = rank * p.hs + q4 * HW;                 // the first of mine
  const int nh = max(0, min(HW, p.hs - q4 * HW));
  const int hl = lane & (HW - 1);                       // my thread's
  const uint32_t blk = outb + q4 * 2048;
  RingPos b2 = {0, 0};
  uint32_t ctx = 0, ph = 0, hph = 0;
  for (int it = cl; it < c->total; it += ncl) {
    const Item m = find_item(c, p.E, it);
    const int tok = lane < m.rows ? token(p, m.r0 + lane) : -1;
    int kept = 0;
    if (p.mask_bits && tok >= 0)
      for (int q = 0; q < nw; ++q) kept += __popc(p.mask_bits[(long long)tok * nw + q]);
    const bool direct = __any_sync(0xffffffffu, kept == 1);
    const int enc = kept == 1 ? (int)((uint32_t)tok | 0x80000000u) : tok;   // see put_row
    const float b1 =
        hl < nh ? __ldg(reinterpret_cast<const float*>(p.packed + (long long)m.e * g.stride +
                                                       g.bias_off) + h0 + hl)
                : 0.f;
    uint32_t bb[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) bb[q] = pack_bf16x2(b1, b1);

    if (!mbar_wait_warp(smem_u32(&c->acc1_full[ctx]), ph, af, p.dev_status)) return;
    tc_fence_after();
    uint32_t v[32];
    tmem_ld32(tmem + 32 * ctx + lanes, v);
    tmem_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&c->acc1_free[ctx]));
    ph ^= ctx;
    ctx ^= 1;
    // the hidden tile of every CTA has been read by its second product of the item before
    if (!mbar_wait_warp(smem_u32(&c->hid_free), hph ^ 1, af, p.dev_status)) return;
    hph ^= 1;
    fence_cluster();
    if (nh > 0) {                        // (warp-uniform; the last warp's lanes may be partly idle)
      const int h = h0 + hl;
      const uint32_t col = hid + (h >> 6) * XB;
      float none = 0.f;
      if (GLU) {
        // lanes 0-15 have the gate rows, 16-31 the up rows: each keeps half of the tokens
        const bool low = lane < 16;
        uint32_t gate[16], up[16], w[8];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const uint32_t got = __shfl_xor_sync(0xffffffffu, low ? v[16 + k] : v[k], 16);
          gate[k] = low ? v[k] : got;
          up[k] = low ? got : v[16 + k];
        }
        ep1_pairs<ACT, true, false>(gate, up, bb, w, none, 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int t = (low ? 0 : 16) + 2 * k;
          asm volatile("st.shared.b16 [%0], %1;" ::"r"(col + swz(t, h & 63)), "h"((uint16_t)w[k]) : "memory");
          asm volatile("st.shared.b16 [%0], %1;" ::"r"(col + swz(t + 1, h & 63)), "h"((uint16_t)(w[k] >> 16)) : "memory");
        }
      } else {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t w[8];
          ep1_pairs<ACT, false, false>(v + 16 * hf, nullptr, bb, w, none, 0);
          if (hl < nh) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int t = 16 * hf + 2 * k;
              asm volatile("st.shared.b16 [%0], %1;" ::"r"(col + swz(t, h & 63)), "h"((uint16_t)w[k]) : "memory");
              asm volatile("st.shared.b16 [%0], %1;" ::"r"(col + swz(t + 1, h & 63)), "h"((uint16_t)(w[k] >> 16)) : "memory");
            }
          }
        }
      }
      __syncwarp();
      for (int h8 = h0; h8 < h0 + nh; h8 += 8) {        // lane = token, 16 bytes
        const uint32_t a = hid + (h8 >> 6) * XB + swz(lane, h8 & 63);
        const uint4 q = ld_shared_v4(a);
        for (int k = 0; k < p.C; ++k)
          if (k != rank)
            asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(peer(a, k)),
                         "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w)
                         : "memory");
      }
      fence_proxy_all();
    }
    __syncwarp();
    if (lane < p.C) arrive_cluster(peer(smem_u32(&c->hid_full), lane));

    for (int s = s0; s < s1; ++s) {
      const int cw = s * 128 + q4 * 32;                 // my warp's columns
      uint4 bz = make_uint4(0u, 0u, 0u, 0u);
      const int col = cw + (lane & 3) * 8;
      if (direct && p.last_bias) bz = __ldg(reinterpret_cast<const uint4*>(p.last_bias + col));
      if (!mbar_wait_warp(smem_u32(&c->acc2_full[b2.s]), b2.ph, af, p.dev_status)) return;
      tc_fence_after();
      tmem_ld32(tmem + 64 + 32 * b2.s + lanes, v);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c->acc2_empty[b2.s]));
      b2.next(NACC2);
#pragma unroll
      for (int t = 0; t < 32; ++t)
        asm volatile("st.shared.b16 [%0], %1;" ::"r"(blk + t * 64 + out_column(lane) * 2),
                     "h"((uint16_t)pack_bf16x2(__uint_as_float(v[t]), 0.f))
                     : "memory");
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = 8 * i + (lane >> 2);
        const uint4 val = ld_shared_v4(blk + row * 64 + (lane & 3) * 16);
        const int t = __shfl_sync(0xffffffffu, enc, row);
        put_row(p.out + (size_t)(t & 0x7fffffff) * p.d + col, t, val, add_bf16x8(bz, val));
      }
      __syncwarp();
    }
    // (the last accumulator's commit covers every product before it)
    if (q4 == 0 && lane < p.C) arrive_cluster(peer(smem_u32(&c->hid_free), lane));
  }
}

template <bool GLU, int ACT>
__global__ void __launch_bounds__(NT, 2) experts_short_kernel(const ShortParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  const uint32_t ring2 = ring + p.ns * p.stage;
  const uint32_t hid = ring2 + S2 * SLOT;
  const uint32_t outb = hid + HID;
  ShortCtl* c = reinterpret_cast<ShortCtl*>(smem_raw + (outb - raw) + OUTB);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank(), cl = blockIdx.x / p.C, ncl = gridDim.x / p.C;
  const int steps = p.d >> 7, s0 = rank * steps / p.C, s1 = (rank + 1) * steps / p.C;

  if (tid == 0) {
    for (int i = 0; i < S1_MAX; ++i) {
      mbar_init(smem_u32(&c->full[i]), 65);             // 64 gather threads, the weights
      mbar_init(smem_u32(&c->empty[i]), 1);
    }
    for (int i = 0; i < S2; ++i) {
      mbar_init(smem_u32(&c->full2[i]), 1);
      mbar_init(smem_u32(&c->empty2[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c->acc1_full[i]), 1);
      mbar_init(smem_u32(&c->acc1_free[i]), 4);
    }
    for (int i = 0; i < NACC2; ++i) {
      mbar_init(smem_u32(&c->acc2_full[i]), 1);
      mbar_init(smem_u32(&c->acc2_empty[i]), 4);
    }
    mbar_init(smem_u32(&c->hid_full), 4 * p.C);
    mbar_init(smem_u32(&c->hid_free), p.C);
    c->abort_flag = 0;
    c->wait_limit = (int)p.wait_limit;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == 6) tmem_alloc(smem_u32(&c->tmem_base), TM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_barrier();
  tc_fence_after();
  const uint32_t tmem = c->tmem_base;

  // Only now: another CTA fits beside this one, and a kernel that waits for this grid must not
  // take the columns that this grid still needs.
  grid_launch_dependents();
  grid_dependency_wait();
  if (warp == 0) {                       // lists and items of the experts 4 lane .. + 3
    int off[5], nt[4], sum = 0;
#pragma unroll
    for (int q = 0; q < 5; ++q) off[q] = 4 * lane + q <= p.E ? p.offsets[4 * lane + q] : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = 4 * lane + q;
      const bool bad = off[q + 1] < off[q] || off[q] < 0 || off[q + 1] > p.N * (long long)p.E;
      const int n = e < p.E && !bad ? off[q + 1] - off[q] : 0;
      if (e < p.E && bad) report(p.dev_status, D2D_ERR_INDEX_RANGE);
      c->off[e] = off[q];
      c->n[e] = n;
      nt[q] = (n + TN - 1) / TN;
      sum += nt[q];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    int at = incl - sum;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      c->first[4 * lane + q] = at;
      at += nt[q];
    }
    if (lane == 31) c->total = incl;
  }
  __syncthreads();

  if (warp < 4) {
    short_epilogues<ACT, GLU>(p, c, hid, outb, tmem, cl, ncl, rank, s0, s1, warp, lane);
  } else if (warp < 6) {
    short_gather(p, c, ring, cl, ncl, tid - 128);
    cp_async_wait_all();
  } else if (warp == 6) {
    if (elect_one()) short_mma(p, c, ring, ring2, hid, tmem, cl, ncl, s0, s1);
    __syncwarp();
  } else {
    short_weights<GLU>(p, c, ring, ring2, cl, ncl, rank, s0, s1, lane);
  }

  // after giving up: see experts_tiles_kernel
  if (*reinterpret_cast<volatile int*>(&c->abort_flag) != 0)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == 6) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, TM_COLS);
  }
  __syncwarp();
  cluster_barrier();                     // the others may still write to this CTA's shared memory
}

// CTAs per expert: four, two where the hidden slices would not be whole 8-row groups (gated: 16 rows
// of gate and up each).  Four instead of two: 21.2 instead of 28.7 us for 32 tokens, d 2048, 128
// gated experts x 128 (two CTAs an SM leave a CTA three stages of 20 KB; one CTA an SM: 24.7).
int cluster_of(int H, bool glu) { return H % (glu ? 64 : 32) == 0 ? 4 : 2; }

// Items that a call is taken to have, from what the host knows: every expert's last tile, and the
// full ones.  kept: experts per token; where the rule does not fix it (0), four, more than a threshold
// rule keeps in use (1.3 to 2.3 at tau_cfg 0.9), so that the items rather fit than not.
long long items_of(int64_t N, int E, int kept) {
  const long long pairs = N * (long long)(kept > 0 ? kept : 4);
  return (pairs < E ? pairs : E) + pairs / TN;
}

// Up to 70 clusters of four run at once with two CTAs an SM (a cluster's SMs are one GPC's): 128 tokens,
// 128 gated experts take 54.3 us with 66, 68, 69 or 70 clusters and 58.4 with 71, 72 or 74, where one
// waits for a place.  Calls that may have an item for every cluster launch 69.  Those that do not launch
// 74, of which the last ones find nothing to do, whichever waits (197 tokens, 24 experts, us per layer:
// 19.3 instead of 20.4).
constexpr int ALL_CLUSTERS = 74, SAFE_CLUSTERS = 69, FEW_ITEMS = 64;

template <bool GLU>
int launch(const ShortParams& p, int act, bool few, cudaStream_t s) {
  int sms = 0;
  auto kernel = act == D2D_RELU         ? experts_short_kernel<GLU, D2D_RELU>
                : act == D2D_GELU       ? experts_short_kernel<GLU, D2D_GELU>
                : act == D2D_TANH       ? experts_short_kernel<GLU, D2D_TANH>
                : act == D2D_LEAKY_RELU ? experts_short_kernel<GLU, D2D_LEAKY_RELU>
                                        : experts_short_kernel<GLU, D2D_GELU_TANH>;
  const size_t smem = 1024 + (size_t)p.ns * p.stage + S2 * SLOT + HID + OUTB + sizeof(ShortCtl) + 64;
  const int rc = device_launch_facts((const void*)kernel, smem, &sms);
  if (rc != D2D_OK) return rc;
  const long long items = (long long)p.E * ((p.N + TN - 1) / TN);
  const long long most =
      p.C == 2 ? sms : (few ? ALL_CLUSTERS : SAFE_CLUSTERS) * (long long)sms / 148;
  const long long n = items < most ? items : most > 0 ? most : 1;
  return launch_pdl_cluster(p.C, kernel, dim3((unsigned)(n * p.C)), dim3(NT), smem, s, p);
}

}  // namespace

// Which calls.  One round of clusters is faster than the form for long lists, a second round of small
// experts is not: the items have to fit.  Layer, us, long form -> this one:
//   24 experts x 128, d 768 (0.4 MB an expert):  32 tokens 21.3 -> 17.8, 256 24.1 -> 19.5
//   96 of them:                   32 tokens 24.2 -> 20.5, 128 27.8 -> 25.9, 256 30.5 -> 31.1, 512 30.4 -> 31.8
// Experts of a megabyte and more are bound by their stream, which is read by every CTA that has a
// share of a list's output there and once here: up to four tokens per expert (two kept each), however
// many items.  Per layer, 64 experts:
//   gated 2048 x 128 (1.5 MB):  32 tokens 40.1 -> 31.8, 256 60.2 -> 42.8, 512 62.5 -> 59.1
//   2048 x 128 (1.0 MB):        32 tokens 32.1 -> 27.3, 256 41.1 -> 33.5, 512 41.1 -> 45.1
//   below the line, gated 1024 x 128 (0.75 MB): 32 tokens 31.2 -> 24.0, 256 37.0 -> 27.9, 512 39.7 -> 36.2
// It would pay for smaller experts too: the line is on the safe side.
bool experts_short_supported(int64_t N, int d, int E, int H, bool glu, int kept) {
  if (N < 1 || N > 512 || d % 128 != 0 || H % 32 != 0 || H > 128) return false;
  if (items_of(N, E, kept) <= ALL_CLUSTERS) return true;
  return experts_geo(d, H, glu, TILE_M).stride >= (1 << 20) && N * (kept > 0 ? kept : 2) <= 8LL * E;
}

int launch_experts_short(const void* x, const int32_t* token_idx, const int32_t* offsets,
                         const void* packed, void* out, int64_t N, int d, int E, int H, bool glu,
                         int act, int* dev_status, cudaStream_t s, DirectRows dr) {
  ShortParams p = {};
  p.x = (const bf16*)x;
  p.N = N;
  p.d = d;
  p.E = E;
  p.H = H;
  p.C = cluster_of(H, glu);
  p.packed = (const uint8_t*)packed;
  p.g = experts_geo(d, H, glu, TILE_M);
  p.hs = H / p.C;
  p.wrows = (glu ? 2 : 1) * p.hs;
  p.stage = p.wrows * 128 + XB;
  p.ns = (RINGS - S2 * SLOT) / p.stage;
  if (p.ns > S1_MAX) p.ns = S1_MAX;
  p.token_idx = token_idx;
  p.offsets = offsets;
  p.out = (bf16*)out;
  p.mask_bits = dr.mask_bits;
  p.last_bias = (const bf16*)dr.last_bias;
  p.dev_status = dev_status;
  umma_debug_read(&p.wait_limit, &p.withhold);
  const bool few = items_of(N, E, dr.kept) <= FEW_ITEMS;
  return glu ? launch<true>(p, act, few, s) : launch<false>(p, act, few, s);
}

}  // namespace d2d
