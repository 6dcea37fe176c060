// Router of the layer on the tensor cores (bf16): per 128 consecutive tokens
//     s = |bf16(relu(bf16(x Wa^T)) Wb^T)|,  keep e iff s_e >= bf16(max s * mult)
// (architectures/moe/moefication.py:328-330 and :80-85), written as mask bits, the 0/1 routing
// tensor and the compaction's counts table; the same CTA writes the initial rows of the layer
// output that the expert kernel will add to (where few SMs have a tile: the others, help_init_rows).
//
// One persistent CTA per SM, 16 warps, one 128-token tile after another:
//   warp 10     one thread loads stages (a 128-row x 64-column TMA box of x and the matching 64-deep
//               slice of Wa, one barrier for both) and, once, the whole of Wb
//   warp  8     one thread issues x Wa^T (tcgen05, N = R in one instruction) into accumulator 1
//   warps 0-3   accumulator 1 -> relu, bf16 -> hidden tile in TENSOR memory
//   warp  9     one thread issues hidden Wb^T, its A operand read from tensor memory
//   warps 4-7   scores -> row maximum, threshold, mask words, routing rows, counts
//   warps 12-15 the tile's initial output rows
//
// Bound: HBM.  A layer reads x once; the initial rows are written only for tokens whose row
// the expert kernel has to ADD to (more than one expert, or none): a token kept by exactly
// one expert gets its row from that expert's store.  The two epilogues are different warps, so
// that the second one does not sit between two tiles.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "d2d_cluster_compact.cuh"
#include "d2d_ranked.cuh"
#include "d2d_tmap.cuh"
#include "d2d_umma_api.cuh"
#include "d2d_umma_ptx.cuh"

namespace d2d {
using namespace umma;
namespace {

constexpr int NTHREADS = 512;
constexpr int WARP_MMA1 = 8, WARP_MMA2 = 9, WARP_LOAD = 10, WARP_INIT0 = 12;
constexpr int NS_MAX = 8;                    // stages (upper bound)
constexpr int MAX_E = 128;
constexpr size_t SMEM_TILES = 220 * 1024;    // stages + Wb
constexpr uint32_t TM_HID = 256, TM_ACC2 = 384;   // tensor-memory columns (accumulator 1 at 0)

struct Geo {
  int kc1;                  // d / 64
  int nsub, nsubw;          // Wa packed as nsub blocks of nsubw rows per 64-deep slice
  int kc2;                  // ceil(R / 64): 64-deep slices of Wb
  int nd;                   // E rounded up to 16
  int ns;                   // stages
  int wa_bytes;             // Wa bytes per stage
  long long w1_bytes, stride;
};

Geo router_geo(int d, int R, int E) {
  Geo g;
  g.kc1 = d / 64;
  g.nsub = R > 128 ? 2 : 1;
  g.nsubw = R / g.nsub;
  g.kc2 = (R + 63) / 64;
  g.nd = (E + 15) / 16 * 16;
  g.wa_bytes = R * 128;
  g.w1_bytes = (long long)g.kc1 * g.wa_bytes;
  const long long wb = (long long)g.kc2 * g.nd * 128;
  g.stride = (g.w1_bytes + wb + 512 + 1023) / 1024 * 1024;
  const int ns = (int)((SMEM_TILES - wb) / (SLOT + (g.wa_bytes + 1023) / 1024 * 1024));
  g.ns = ns < NS_MAX ? ns : NS_MAX;
  return g;
}

struct Params {
  long long N;
  int d, R, E;
  const uint8_t* packed;
  Geo g;
  float mult;
  int k;                    // ranked rules
  float tau;
  uint32_t* mask_bits;
  bf16* scores;             // optional [N, E]
  bf16* rt_out;             // optional: 0/1 routing tensor [N, E]
  uint8_t* tile_counts;     // optional: bytes [tiles][EP], kept tokens per expert
  int32_t* token_idx;       // optional (one tile per CTA, all CTAs one cluster): the token lists
  int32_t* offsets;
  int EP;
  MaskTable mt;             // words null: none
  bf16* out_init;           // optional: initial output rows last_bias (+ resid)
  const bf16* last_bias;
  const bf16* resid;
  int init_all;             // every row; 0: rows not kept by exactly one expert
  int ctas;                 // that take tiles
  bf16* help_init;          // optional: every initial row, by the CTAs behind those (then out_init is null)
  int* dev_status;
  uint32_t wait_limit;
  int withhold;             // test hook: CTA 0 never loads its first weight slice
};

struct Ctl {
  unsigned long long full[NS_MAX], empty[NS_MAX];
  unsigned long long wb_full, acc1_full[2], acc1_empty[2], hid_full, g2_done, acc2_empty;
  unsigned long long init_full[2], init_empty[2], cnt_full;
  uint32_t tmem_base;
  int abort_flag;
  int wait_limit;           // must follow abort_flag (mbar_wait reads abort_flag[1])
  int cnt[2][4][MAX_E];     // per expert, the tokens of a 32-token row group that keep it: number or bits
  uint32_t init_rows[2][4];
};

// WARM: a role's first pass is without effect.  Where the kernel also writes the lists (up to eight tiles,
// one each) there is none: the previous call's kernels are over too soon for it, and its branches alone
// make a call whose code is executed once longer (single calls, 197 tokens 21.2 -> 22.4 us per layer).  Long calls
// gain by it (queued, 12608 tokens x 24 52.3 -> 48.2, 50432 80.0 -> 77.3, 65536 x 96 114.4 -> 106.1), and so do short ones
// that leave the lists to other kernels, which are there to be waited for (replayed, without / with it: 24
// experts stage by stage 1024 tokens 26.5 / 25.0, 256 21.5 / 20.4, 64 19.6 / 20.4, 32 19.0 / 18.5; top-4 of 96 1024 tokens
// 62.7 / 61.4, 128 59.4 / 58.0, 64 55.0 / 55.6; nothing but routers one after another 5.5 / 5.8).
template <bool WARM>
__device__ __forceinline__ bool first_run() {
  if (WARM) return first_pass();
  grid_dependency_wait();
  return true;
}
template <bool WARM>
__device__ __forceinline__ bool next_run() {
  return WARM ? in_earnest() : true;
}

template <bool WARM>
__device__ void role_load(const Params& p, Ctl* c, const CUtensorMap* tmx, uint32_t ring,
                          uint32_t wb, uint32_t stage_bytes) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const int tiles = (int)((p.N + TILE_M - 1) / TILE_M);
  const uint32_t wb_bytes = (uint32_t)(g.kc2 * g.nd * 128);
  bool withheld = (p.withhold & 1) != 0 && blockIdx.x == 0;
  RingPos r = {0, 0};
  bool first = true, run = first_run<WARM>();
  for (int tile = blockIdx.x; tile < tiles;) {
    const int slices = run ? g.kc1 : 1;
    for (int kc = 0; kc < slices; ++kc) {
      if (run && !mbar_wait_fast(smem_u32(&c->empty[r.s]), r.ph ^ 1, af, p.dev_status)) return;
      const uint32_t bar = smem_u32(&c->full[r.s]), dst = ring + r.s * stage_bytes;
      mbar_arrive_expect_tx(bar, SLOT + g.wa_bytes, run);
      tma_load_2d(dst, tmx, kc * 64, tile * TILE_M, bar, run);
      bulk_g2s(dst + SLOT, p.packed + (long long)kc * g.wa_bytes, g.wa_bytes, bar, run && !withheld);
      if (run) {
        withheld = false;
        r.next(g.ns);
      }
    }
    if (first) {           // after the first tile's stages: Wb is needed only behind its hidden tile
      first = !run;
      const uint32_t bar = smem_u32(&c->wb_full);
      mbar_arrive_expect_tx(bar, wb_bytes, run);
      bulk_g2s(wb, p.packed + g.w1_bytes, wb_bytes, bar, run);
    }
    if (run) {
      tile += p.ctas;
    } else {
      grid_dependency_wait();
      run = next_run<WARM>();
    }
  }
}

template <bool WARM>
__device__ void role_mma1(const Params& p, Ctl* c, uint32_t ring, uint32_t stage_bytes,
                          uint32_t tmem) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const int tiles = (int)((p.N + TILE_M - 1) / TILE_M);
  const uint32_t idesc = instr_desc(TILE_M, p.R);
  const uint64_t d0 = smem_desc(ring);
  const uint32_t hi = (uint32_t)(d0 >> 32), lo0 = (uint32_t)d0;
  const int nacc = p.R <= 128 ? 2 : 1;
  RingPos r = {0, 0}, a = {0, 0};
  bool run = first_run<WARM>();
  for (int tile = blockIdx.x; tile < tiles;) {
    if (run && !mbar_wait_fast(smem_u32(&c->acc1_empty[a.s]), a.ph ^ 1, af, p.dev_status)) return;
    tc_fence_after();
    const uint32_t acc = tmem + a.s * 128;
    const int slices = run ? g.kc1 : 1;
    for (int kc = 0; kc < slices; ++kc) {
      if (run && !mbar_wait_fast(smem_u32(&c->full[r.s]), r.ph, af, p.dev_status)) return;
      tc_fence_after();
      const uint32_t alo = lo0 + r.s * (stage_bytes >> 4), blo = alo + (SLOT >> 4);
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k)
        umma_bf16(acc, ((uint64_t)hi << 32) | (alo + 2 * k), ((uint64_t)hi << 32) | (blo + 2 * k),
                  idesc, (kc | k) != 0, run);
      umma_commit(smem_u32(&c->empty[r.s]), run);
      if (run) r.next(g.ns);
    }
    umma_commit(smem_u32(&c->acc1_full[a.s]), run);
    if (run) {
      a.next(nacc);
      tile += p.ctas;
    } else {
      grid_dependency_wait();
      run = next_run<WARM>();
    }
  }
}

template <bool WARM>
__device__ void role_mma2(const Params& p, Ctl* c, uint32_t wb, uint32_t tmem) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const int tiles = (int)((p.N + TILE_M - 1) / TILE_M);
  const uint32_t idesc = instr_desc(TILE_M, g.nd);
  const uint64_t d0 = smem_desc(wb);
  const uint32_t hi = (uint32_t)(d0 >> 32), lo0 = (uint32_t)d0;
  const int ksteps = p.R >> 4;
  uint32_t ph = 0;
  bool run = first_run<WARM>();
  for (int tile = blockIdx.x; tile < tiles;) {
    if (run) {
      if (tile == (int)blockIdx.x &&
          !mbar_wait_fast(smem_u32(&c->wb_full), 0, af, p.dev_status))
        return;
      if (!mbar_wait_fast(smem_u32(&c->acc2_empty), ph ^ 1, af, p.dev_status)) return;
      if (!mbar_wait_fast(smem_u32(&c->hid_full), ph, af, p.dev_status)) return;
    }
    tc_fence_after();
    for (int k = 0; k < ksteps; ++k)
      umma_bf16_ta(tmem + TM_ACC2, tmem + TM_HID + 8 * k,
                   ((uint64_t)hi << 32) | (lo0 + (uint32_t)(k >> 2) * (g.nd * 8) + 2 * (k & 3)),
                   idesc, k != 0, run);
    umma_commit(smem_u32(&c->g2_done), run);
    if (run) {
      tile += p.ctas;
      ph ^= 1;
    } else {
      grid_dependency_wait();
      run = next_run<WARM>();
    }
  }
}

// 16 hidden columns as 8 packed bf16 pairs: relu(T(x Wa^T))
__device__ __forceinline__ void relu_pairs(const uint32_t* v, uint32_t* w) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    __nv_bfloat162 h =
        __floats2bfloat162_rn(__uint_as_float(v[2 * q]), __uint_as_float(v[2 * q + 1]));
    h = __hmax2(h, __float2bfloat162_rn(0.f));
    w[q] = *reinterpret_cast<uint32_t*>(&h);
  }
}

// warps 0-3, thread = tile row = TMEM lane: hidden tile = bf16 relu of accumulator 1
template <bool WARM>
__device__ void role_hidden(const Params& p, Ctl* c, uint32_t tmem, int et) {
  volatile int* af = &c->abort_flag;
  const int tiles = (int)((p.N + TILE_M - 1) / TILE_M);
  const uint32_t lane_base = (uint32_t)(et & ~31) << 16;
  const int nacc = p.R <= 128 ? 2 : 1;
  RingPos a = {0, 0};
  uint32_t ph = 0;
  bool run = first_run<WARM>();
#pragma unroll 1
  for (int tile = blockIdx.x; tile < tiles;) {
    if (run) {
      if (!mbar_wait_warp(smem_u32(&c->acc1_full[a.s]), a.ph, af, p.dev_status)) return;
      // the previous tile's second product has read the hidden tile
      if (!mbar_wait_warp(smem_u32(&c->g2_done), ph ^ 1, af, p.dev_status)) return;
    }
    tc_fence_after();
    const uint32_t src = tmem + lane_base + a.s * 128, dst = tmem + lane_base + TM_HID;
    for (int c0 = 0; c0 < p.R; c0 += 16) {
      uint32_t v[16], w[8];
      tmem_ld16(src + c0, v);
      tmem_wait_ld();
      relu_pairs(v, w);
      tmem_st8(dst + (c0 >> 1), w);
    }
    tmem_wait_st();
    tc_fence_before();
    mbar_arrive(smem_u32(&c->acc1_empty[a.s]), run);
    mbar_arrive(smem_u32(&c->hid_full), run);
    if (run) {
      a.next(nacc);
      tile += p.ctas;
      ph ^= 1;
    } else {
      grid_dependency_wait();
      run = next_run<WARM>();
    }
  }
}

// one row of E bf16 values held as packed pairs
template <int NB>
__device__ __forceinline__ void store_row(bf16* dst, const uint32_t* s, int E) {
  if ((E & 7) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
    for (int h = 0; h < NB * 2; ++h)
      if (8 * h < E)
        *reinterpret_cast<uint4*>(dst + 8 * h) =
            make_uint4(s[4 * h], s[4 * h + 1], s[4 * h + 2], s[4 * h + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < NB * 8; ++q) {
      if (2 * q < E) dst[2 * q] = __ushort_as_bfloat16((unsigned short)(s[q] & 0xffff));
      if (2 * q + 1 < E) dst[2 * q + 1] = __ushort_as_bfloat16((unsigned short)(s[q] >> 16));
    }
  }
}

// warps 4-7, thread = tile row: the row's scores stay in registers as packed bf16 pairs
// (NB blocks of 16 experts), so tensor memory is read once and handed back at once
template <int NB, int RULE, bool WARM>
__device__ void role_gate(const Params& p, Ctl* c, uint32_t tmem, int et) {
  volatile int* af = &c->abort_flag;
  const int tiles = (int)((p.N + TILE_M - 1) / TILE_M);
  const int lane = et & 31, q4 = et >> 5, E = p.E;
  constexpr int NW = (NB + 1) / 2;                    // mask words that can be non-zero
  const int nw = (E + 31) >> 5;                       // == NW
  const uint32_t lane_base = (uint32_t)(et & ~31) << 16;
  uint32_t ph = 0, buf = 0, ibuf_ph = 0;
  bool run = first_run<WARM>();                    // first pass: as if no row were there
#pragma unroll 1
  for (int tile = blockIdx.x; tile < tiles;) {
    const long long trow = (long long)tile * TILE_M + et;
    const bool live = run && trow < p.N;
    if (run && !mbar_wait_warp(smem_u32(&c->g2_done), ph, af, p.dev_status)) return;
    tc_fence_after();
    uint32_t s[NB * 8];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      uint32_t v[16];
      tmem_ld16(tmem + lane_base + TM_ACC2 + 16 * b, v);
      tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const __nv_bfloat162 h = __habs2(
            __floats2bfloat162_rn(__uint_as_float(v[2 * q]), __uint_as_float(v[2 * q + 1])));
        s[8 * b + q] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    tc_fence_before();
    mbar_arrive(smem_u32(&c->acc2_empty), run);
    // columns past E have zero weights, hence score 0: no effect on a maximum of magnitudes
    __nv_bfloat162 m2 = *reinterpret_cast<const __nv_bfloat162*>(&s[0]);
#pragma unroll
    for (int q = 1; q < NB * 8; ++q)
      m2 = __hmax2_nan(m2, *reinterpret_cast<const __nv_bfloat162*>(&s[q]));
    const float m = nanmax(__low2float(m2), __high2float(m2));
    const __nv_bfloat162 thr = __float2bfloat162_rn(__fmul_rn(m, p.mult));
    if (p.scores && live) store_row<NB>(p.scores + trow * E, s, E);
    uint32_t word[RULE != 0 ? 2 : NW];
#pragma unroll
    for (int j = 0; j < (RULE != 0 ? 2 : NW); ++j) word[j] = 0u;
    if (RULE != 0) {
      ranked_words<bf16, NB * 16, RULE>(reinterpret_cast<const bf16*>(s), run ? E : 1, run ? p.k : 1, p.tau,
                                        word);
#pragma unroll
      for (int q = 0; q < NB * 8; ++q)
        s[q] = ((word[0] >> (2 * q)) & 1u ? 0x3f80u : 0u) |
               ((word[0] >> (2 * q + 1)) & 1u ? 0x3f800000u : 0u);
    } else {
#pragma unroll
      for (int q = 0; q < NB * 8; ++q) {
        const uint32_t k = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&s[q]), thr);
        word[q >> 4] |= k & (0x00010001u << (q & 15));
        s[q] = k & 0x3f803f80u;                       // the routing entries: bf16 1.0 or 0
      }
    }
    int kept = 0;
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      if (RULE == 0) word[j] = interleave16(word[j]);
      if (32 * j + 32 > E) word[j] &= (1u << (E - 32 * j)) - 1u;      // E > 32 j
      if (!live) word[j] = 0u;
      kept += __popc(word[j]);
      if (live) p.mask_bits[trow * nw + j] = word[j];
    }
    if (p.out_init && !p.init_all) {
      const bool todo = live && kept != 1;
      const uint32_t rows = __ballot_sync(0xffffffffu, todo);
      if (run && !mbar_wait_warp(smem_u32(&c->init_empty[buf]), ibuf_ph ^ 1, af, p.dev_status)) return;
      if (lane == 0) {
        c->init_rows[buf][q4] = rows;
        mbar_arrive(smem_u32(&c->init_full[buf]), run);
      }
      __syncwarp();
      if (run) ibuf_ph ^= buf;
    }
    if (p.token_idx) {         // (the only tile: both halves of cnt are free)
#pragma unroll
      for (int j = 0; j < NW; ++j)
        c->cnt[0][q4][32 * j + lane] = (int)transpose32(word[j], lane);
    } else if (p.tile_counts) {
#pragma unroll
      for (int j = 0; j < NW; ++j) {
        const uint32_t col = transpose32(word[j], lane);
        c->cnt[buf][q4][32 * j + lane] = WARM && p.mt.words ? (int)col : __popc(col);
      }
      // one barrier per tile: the other half of cnt is written before anybody passes it again (an
      // mbarrier, because a warp that gave up never comes)
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c->cnt_full), run);
      if (run && !mbar_wait_warp(smem_u32(&c->cnt_full), ph, af, p.dev_status)) return;
      if (et < p.EP) {
        int n = 0;
        if (et < E) {
          const int a = c->cnt[buf][0][et], b = c->cnt[buf][1][et], cc = c->cnt[buf][2][et],
                    dd = c->cnt[buf][3][et];
          if (WARM && p.mt.words) {
            if (run) p.mt.words[(long long)tile * E + et] = make_uint4(a, b, cc, dd);
            n = __popc(a) + __popc(b) + __popc(cc) + __popc(dd);
          } else {
            n = a + b + cc + dd;
          }
        }
        if (run) p.tile_counts[(long long)tile * p.EP + et] = (uint8_t)n;
      }
    }
    if (p.rt_out && live) store_row<NB>(p.rt_out + trow * E, s, E);
    if (run) {
      tile += p.ctas;
      ph ^= 1;
      buf ^= 1;
    } else {
      grid_dependency_wait();
      run = next_run<WARM>();
    }
  }
}

// warps 12-15 where every row is initialised with the layer's own input: out of the stages of the first
// product, which then wait for these warps as well.  Warp w has rows 32 w .. + 31.  (Read
// again from memory, eight rows at a time: 12608 x 768 took 26 thousand cycles, twice the rest of the tile.)
template <bool WARM>
__device__ void role_init_stages(const Params& p, Ctl* c, uint32_t ring, uint32_t stage_bytes, int w,
                                 int lane) {
  volatile int* af = &c->abort_flag;
  const int tiles = (int)((p.N + TILE_M - 1) / TILE_M), j = lane & 7, r4 = lane >> 3;
  RingPos r = {0, 0};
  bool run = first_run<WARM>();
#pragma unroll 1
  for (int tile = blockIdx.x; tile < tiles;) {
    const long long row0 = (long long)tile * TILE_M + 32 * w + r4;
    const int slices = run ? p.g.kc1 : 1;
#pragma unroll 1
    for (int kc = 0; kc < slices; ++kc) {
      uint4 bz = make_uint4(0u, 0u, 0u, 0u), v[8];
      if (run) {
        if (p.last_bias) bz = __ldg(reinterpret_cast<const uint4*>(p.last_bias) + kc * 8 + j);
        if (!mbar_wait_warp(smem_u32(&c->full[r.s]), r.ph, af, p.dev_status)) return;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = 32 * w + 4 * i + r4;
        v[i] = ld_shared_v4(ring + r.s * stage_bytes + (row >> 3) * 1024 + (row & 7) * 128 +
                            ((j ^ (row & 7)) << 4));
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (run && row0 + 4 * i < p.N)
          *(reinterpret_cast<uint4*>(p.out_init + (row0 + 4 * i) * p.d) + kc * 8 + j) =
              add_bf16x8(bz, v[i]);
      // behind the stores, which have waited for what was loaded: an arrival does not wait for loads under way;
      // and the next copy into the stage is the async proxy's
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c->empty[r.s]), run);
      if (run) r.next(p.g.ns);
    }
    if (run) {
      tile += p.ctas;
    } else {
      grid_dependency_wait();
      run = next_run<WARM>();
    }
  }
}

// warps 12-15: the initial rows of the tile's tokens that ask for one.  Warp w has rows 32 w .. + 31;
// where only the first 32 have any (a call of few tokens) the warps share a row instead, every
// fourth 512-byte piece each (32 tokens x 2048: 12 -> 4 us).
template <bool WARM>
__device__ void role_init(const Params& p, Ctl* c, int w, int lane) {
  volatile int* af = &c->abort_flag;
  const int tiles = (int)((p.N + TILE_M - 1) / TILE_M);
  const int v8 = p.d >> 3;
  uint32_t ph = 0, buf = 0;
  bool run = first_run<WARM>();                    // first pass: one row that is neither read nor written
#pragma unroll 1
  for (int tile = blockIdx.x; tile < tiles;) {
    bool share = false;
    int q = w;
    uint32_t rows;
    if (!run) {
      rows = 1u;
    } else if (p.init_all) {           // no need to know what the gate says
      const long long left = p.N - (long long)tile * TILE_M;
      share = left <= 32;
      q = share ? 0 : w;
      const long long n = left - 32 * q;
      rows = n >= 32 ? 0xffffffffu : n > 0 ? (1u << n) - 1u : 0u;
    } else {
      if (!mbar_wait_warp(smem_u32(&c->init_full[buf]), ph, af, p.dev_status)) return;
      share = (c->init_rows[buf][1] | c->init_rows[buf][2] | c->init_rows[buf][3]) == 0u;
      q = share ? 0 : w;
      rows = c->init_rows[buf][q];
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c->init_empty[buf]));
    }
    const long long row0 = (long long)tile * TILE_M + 32 * q;
    const int step = share ? 128 : 32, c8n = rows == 0u ? 0 : run ? v8 : 32;
#pragma unroll 1
    for (int c8 = lane + (share ? 32 * w : 0); c8 < c8n; c8 += step) {
      uint4 bz = make_uint4(0u, 0u, 0u, 0u);
      if (p.last_bias && run) bz = __ldg(reinterpret_cast<const uint4*>(p.last_bias) + c8);
      if (!p.resid) {
        for (uint32_t m = rows; m != 0u; m &= m - 1)
          if (run) *(reinterpret_cast<uint4*>(p.out_init + (row0 + __ffs(m) - 1) * p.d) + c8) = bz;
        continue;
      }
      for (uint32_t m = rows; m != 0u;) {
        uint4 xv[8];
        int rr[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {        // eight rows in flight
          rr[u] = m != 0u && run ? __ffs(m) - 1 : -1;
          m &= m - 1;
          if (rr[u] >= 0)
            xv[u] = __ldg(reinterpret_cast<const uint4*>(p.resid + (row0 + rr[u]) * p.d) + c8);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (rr[u] >= 0)
            *(reinterpret_cast<uint4*>(p.out_init + (row0 + rr[u]) * p.d) + c8) =
                add_bf16x8(bz, xv[u]);
      }
    }
    if (run) {
      tile += p.ctas;
      ph ^= buf;
      buf ^= 1;
    } else {
      grid_dependency_wait();
      run = next_run<WARM>();
    }
  }
}

// Calls of few tiles: the other CTAs of the grid write every initial row while the tiles are computed.  A tile's
// own CTA knows only behind its gate which rows want one, and 47 rows (of 128, 24 experts at 0.9) at an SM's 30
// bytes a clock then keep the next kernel waiting (197 tokens 19.4 -> 17.4 us).  That the expert kernel stores some of
// these rows again costs what it costs to write them: the rule's line follows their share.  These CTAs hold an SM
// each, with the tiles' shared memory, while they wait for the previous kernel and write: two streams of 1100-token
// layers take 33.5 instead of 32.0 us a pair (197 tokens 19.2 instead of 21.4; beside a gated layer of 32 768 no
// difference).
__device__ __forceinline__ void help_init_rows(const Params& p) {
  const int v8 = p.d >> 3, helpers = (int)gridDim.x - p.ctas, h = (int)blockIdx.x - p.ctas;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row0 = p.N * h / helpers, row1 = p.N * (h + 1) / helpers;
  grid_dependency_wait();
  for (int c8 = lane; c8 < v8; c8 += 32) {
    uint4 bz = make_uint4(0u, 0u, 0u, 0u);
    if (p.last_bias) bz = __ldg(reinterpret_cast<const uint4*>(p.last_bias) + c8);
    if (!p.resid) {
      for (long long t = row0 + warp; t < row1; t += NTHREADS / 32)
        *(reinterpret_cast<uint4*>(p.help_init + t * p.d) + c8) = bz;
      continue;
    }
    for (long long t = row0 + warp; t < row1; t += 4 * (NTHREADS / 32)) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)          // four rows in flight
        if (t + u * (NTHREADS / 32) < row1)
          v[u] = __ldg(reinterpret_cast<const uint4*>(p.resid + (t + u * (NTHREADS / 32)) * p.d) + c8);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (t + u * (NTHREADS / 32) < row1)
          *(reinterpret_cast<uint4*>(p.help_init + (t + u * (NTHREADS / 32)) * p.d) + c8) =
              add_bf16x8(bz, v[u]);
    }
  }
}

// Initial rows: by warps of the tile's CTA, by those out of the stages of the first product, or by CTAs of their
// own.  Kernels of their own, because a call of few tiles executes the code once: as a branch in one kernel
// the second form cost the calls without it 0.4 us (197 tokens 19.5 -> 20.0), the third one as much.
enum { INIT_TILE, INIT_STAGES, INIT_OTHERS };

// RULE: 0, or D2D_RULE_TOPK / D2D_RULE_DYNK (E <= 32).  WARM: see first_run
template <int RULE, bool WARM, int INIT>
__global__ void __launch_bounds__(NTHREADS, 1)
router_tiles_kernel(const Params p, const __grid_constant__ CUtensorMap tmx) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t stage_bytes = SLOT + (uint32_t)(p.g.wa_bytes + 1023) / 1024 * 1024;
  const uint32_t wb = base + p.g.ns * stage_bytes;
  const uint32_t wb_bytes = (uint32_t)(p.g.kc2 * p.g.nd * 128);
  Ctl* c = reinterpret_cast<Ctl*>(smem_raw + (wb - raw) + (wb_bytes + 1023) / 1024 * 1024);
  const int tid = threadIdx.x, warp = tid >> 5;
  // Programmatic dependent launch: the next kernel of the stream may be scheduled while this one
  // runs (it waits for this grid before it reads anything); this CTA initialises its barriers
  // while the previous kernel drains and reads global memory only after the wait below.
  grid_launch_dependents();
  if (INIT == INIT_OTHERS && (int)blockIdx.x >= p.ctas) {
    help_init_rows(p);
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < NS_MAX; ++i) {
      mbar_init(smem_u32(&c->full[i]), 1);
      mbar_init(smem_u32(&c->empty[i]), INIT == INIT_STAGES ? 5 : 1);
    }
    mbar_init(smem_u32(&c->wb_full), 1);
    mbar_init(smem_u32(&c->hid_full), 128);
    mbar_init(smem_u32(&c->g2_done), 1);
    mbar_init(smem_u32(&c->acc2_empty), 128);
    mbar_init(smem_u32(&c->cnt_full), 4);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c->acc1_full[i]), 1);
      mbar_init(smem_u32(&c->acc1_empty[i]), 128);
      mbar_init(smem_u32(&c->init_full[i]), 4);
      mbar_init(smem_u32(&c->init_empty[i]), 4);
    }
    c->abort_flag = 0;
    c->wait_limit = (int)p.wait_limit;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == WARP_MMA1) tmem_alloc(smem_u32(&c->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c->tmem_base;

  // (every role waits for the previous kernel behind its first pass: its bounded waits count from there on)
  if (warp < 4) {
    role_hidden<WARM>(p, c, tmem, tid);
  } else if (warp < 8) {
    if (RULE != 0) {
      if (p.g.nd == 16) role_gate<1, RULE, WARM>(p, c, tmem, tid - 128);
      else role_gate<2, RULE, WARM>(p, c, tmem, tid - 128);
    } else {
      switch (p.g.nd >> 4) {
        case 1: role_gate<1, 0, WARM>(p, c, tmem, tid - 128); break;
        case 2: role_gate<2, 0, WARM>(p, c, tmem, tid - 128); break;
        case 3: role_gate<3, 0, WARM>(p, c, tmem, tid - 128); break;
        case 4: role_gate<4, 0, WARM>(p, c, tmem, tid - 128); break;
        case 5: role_gate<5, 0, WARM>(p, c, tmem, tid - 128); break;
        case 6: role_gate<6, 0, WARM>(p, c, tmem, tid - 128); break;
        case 7: role_gate<7, 0, WARM>(p, c, tmem, tid - 128); break;
        default: role_gate<8, 0, WARM>(p, c, tmem, tid - 128); break;
      }
    }
  } else if (warp == WARP_MMA1) {
    if (elect_one()) role_mma1<WARM>(p, c, base, stage_bytes, tmem);
    __syncwarp();
  } else if (warp == WARP_MMA2) {
    if (elect_one()) role_mma2<WARM>(p, c, wb, tmem);
    __syncwarp();
  } else if (warp == WARP_LOAD) {
    if (elect_one()) role_load<WARM>(p, c, &tmx, base, wb, stage_bytes);
    __syncwarp();
  } else if (INIT != INIT_OTHERS && warp >= WARP_INIT0 && p.out_init) {
    if (INIT == INIT_STAGES)
      role_init_stages<WARM>(p, c, base, stage_bytes, warp - WARP_INIT0, tid & 31);
    else
      role_init<WARM>(p, c, warp - WARP_INIT0, tid & 31);
  }

  // A launch that gave up may still have copies and MMAs in flight that use this CTA's
  // shared and tensor memory: give them time to land before both are released.
  if (*reinterpret_cast<volatile int*>(&c->abort_flag) != 0)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (p.token_idx) {
    grid_dependency_wait();
    uint32_t* rows = reinterpret_cast<uint32_t*>(&c->cnt[0][0][0]);
    if (*reinterpret_cast<volatile int*>(&c->abort_flag) != 0) {     // nothing a list may rely on
      for (int i = tid; i < 4 * MAX_E; i += NTHREADS) rows[i] = 0u;
      __syncthreads();
    }
    cluster_compact<NTHREADS>(rows, MAX_E, reinterpret_cast<int*>(smem_raw + (base - raw)), p.E,
                              (int64_t)blockIdx.x * TILE_M, p.token_idx, p.offsets);
  }
}

// ---------------------------------------------------------------------------
// few tokens, large router
// ---------------------------------------------------------------------------
// A call of at most a few tiles leaves the chip idle above: one CTA streams all of Wa (1 MB for
// 2048 x 256) through its own 64 bytes per clock, 15 us for 32 tokens.  Here a cluster of eight
// CTAs has a tile: each takes an eighth of the hidden columns (all of d, an eighth of Wa), their
// share of the scores (K = R / 8), and after an exchange through distributed shared memory every
// eighth row of the tile.  A row's score is the fp32 sum of eight shares, rounded once.
// Warps 0-3: accumulators (thread = row), then all eight warps settle rows; 4: loads; 5: MMAs.
constexpr int CL = 8, CL_THREADS = 256, CL_NS = 8;

struct ClCtl {
  unsigned long long full[CL_NS], empty[CL_NS];
  unsigned long long wb_full, acc1_full, hid_full, acc2_full;
  uint32_t tmem_base;
  int abort_flag;
  int wait_limit;           // must follow abort_flag
};

__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CL_THREADS, 1)
router_cluster_kernel(const Params p, const __grid_constant__ CUtensorMap tmx) {
  extern __shared__ uint8_t smem_raw[];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  const Geo& g = p.g;
  const int cw = p.R / CL;                              // my hidden columns
  const uint32_t wa_bytes = cw * 128, stage_bytes = SLOT + (wa_bytes + 1023) / 1024 * 1024;
  const uint32_t wb = ring + CL_NS * stage_bytes;       // the 64-deep slice of Wb that has my columns
  const uint32_t wb_bytes = g.nd * 128;
  ClCtl* c = reinterpret_cast<ClCtl*>(smem_raw + (wb - raw) + wb_bytes);
  float* share = reinterpret_cast<float*>(smem_raw + (ring - raw));   // [128][E + 1], over the ring
  const int EP = p.E + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster.block_rank(), tile = blockIdx.x / CL;
  volatile int* af = &c->abort_flag;
  grid_launch_dependents();
  if (tid == 0) {
    for (int i = 0; i < CL_NS; ++i) {
      mbar_init(smem_u32(&c->full[i]), 1);
      mbar_init(smem_u32(&c->empty[i]), 1);
    }
    mbar_init(smem_u32(&c->wb_full), 1);
    mbar_init(smem_u32(&c->acc1_full), 1);
    mbar_init(smem_u32(&c->hid_full), 128);
    mbar_init(smem_u32(&c->acc2_full), 1);
    c->abort_flag = 0;
    c->wait_limit = (int)p.wait_limit;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == 5) tmem_alloc(smem_u32(&c->tmem_base), 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_dependency_wait();
  const uint32_t tmem = c->tmem_base;                   // accumulator 1 / hidden at 0, 2 at 128

  if (warp == 4) {
    if (elect_one()) {
      bool withheld = (p.withhold & 1) != 0 && blockIdx.x == 0;
      const uint8_t* wa = p.packed + rank * wa_bytes;
      mbar_arrive_expect_tx(smem_u32(&c->wb_full), wb_bytes);
      bulk_g2s(wb, p.packed + g.w1_bytes + (long long)(rank * cw / 64) * wb_bytes, wb_bytes,
               smem_u32(&c->wb_full));
      RingPos r = {0, 0};
      for (int kc = 0; kc < g.kc1; ++kc) {
        if (!mbar_wait_fast(smem_u32(&c->empty[r.s]), r.ph ^ 1, af, p.dev_status)) break;
        const uint32_t bar = smem_u32(&c->full[r.s]), dst = ring + r.s * stage_bytes;
        mbar_arrive_expect_tx(bar, SLOT + wa_bytes);
        tma_load_2d(dst, &tmx, kc * 64, tile * TILE_M, bar);
        if (withheld) withheld = false;
        else bulk_g2s(dst + SLOT, wa + (long long)kc * g.wa_bytes, wa_bytes, bar);
        r.next(CL_NS);
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    if (elect_one()) {
      const uint64_t d0 = smem_desc(ring), dw = smem_desc(wb);
      const uint64_t hi = (d0 >> 32) << 32;
      const uint32_t lo0 = (uint32_t)d0, id1 = instr_desc(TILE_M, cw), id2 = instr_desc(TILE_M, g.nd);
      RingPos r = {0, 0};
      bool ok = true;
      for (int kc = 0; ok && kc < g.kc1; ++kc) {
        ok = mbar_wait_fast(smem_u32(&c->full[r.s]), r.ph, af, p.dev_status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t alo = lo0 + r.s * (stage_bytes >> 4), blo = alo + (SLOT >> 4);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
          umma_bf16(tmem, hi | (alo + 2 * k), hi | (blo + 2 * k), id1, (kc | k) != 0);
        umma_commit(smem_u32(&c->empty[r.s]));
        r.next(CL_NS);
      }
      if (ok) umma_commit(smem_u32(&c->acc1_full));
      ok = ok && mbar_wait_fast(smem_u32(&c->wb_full), 0, af, p.dev_status) &&
           mbar_wait_fast(smem_u32(&c->hid_full), 0, af, p.dev_status);
      if (ok) {
        tc_fence_after();
        const uint32_t b0 = (uint32_t)dw + 2 * ((rank * cw & 63) >> 4);
        for (int k = 0; k < (cw >> 4); ++k)
          umma_bf16_ta(tmem + 128, tmem + 8 * k, hi | (b0 + 2 * k), id2, k != 0);
        umma_commit(smem_u32(&c->acc2_full));
      }
    }
    __syncwarp();
  } else if (warp < 4) {
    const uint32_t lb = (uint32_t)(tid & ~31) << 16;
    bool ok = mbar_wait_warp(smem_u32(&c->acc1_full), 0, af, p.dev_status);
    if (ok) {
      tc_fence_after();
      for (int c0 = 0; c0 < cw; c0 += 16) {
        uint32_t v[16], w[8];
        tmem_ld16(tmem + lb + c0, v);
        tmem_wait_ld();
        relu_pairs(v, w);
        tmem_st8(tmem + lb + (c0 >> 1), w);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(smem_u32(&c->hid_full));
      ok = mbar_wait_warp(smem_u32(&c->acc2_full), 0, af, p.dev_status);
    }
    if (ok) {                    // (both products are done: the ring is free)
      tc_fence_after();
      for (int c0 = 0; c0 < p.E; c0 += 16) {
        uint32_t v[16];
        tmem_ld16(tmem + lb + 128 + c0, v);
        tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 16; ++q)
          if (c0 + q < p.E) share[tid * EP + c0 + q] = __uint_as_float(v[q]);
      }
      tc_fence_before();
    }
  }
  // (a CTA that gave up takes part in both cluster barriers all the same)
  if (*af != 0)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  __syncthreads();
  tc_fence_after();
  if (warp == 5) tmem_dealloc(tmem, 256);
  cluster.sync();

  const int nw = (p.E + 31) >> 5, v8 = p.d >> 3;
  const int nrows = (int)min((long long)TILE_M, p.N - (long long)tile * TILE_M);
  const float* part[CL];
#pragma unroll
  for (int k = 0; k < CL; ++k) part[k] = cluster.map_shared_rank(share, k);
  for (int row = rank + CL * warp; row < nrows; row += CL * (CL_THREADS / 32)) {
    const long long t = (long long)tile * TILE_M + row;
    float sc[MAX_E / 32], m = -INFINITY;
#pragma unroll
    for (int j = 0; j < MAX_E / 32; ++j) {
      const int e = lane + 32 * j;
      sc[j] = 0.f;
      if (e < p.E) {
        float a[CL];
#pragma unroll
        for (int k = 0; k < CL; ++k) a[k] = part[k][row * EP + e];
        sc[j] = fabsf(bfr(((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]))));
        m = nanmax(m, sc[j]);
        if (p.scores) p.scores[t * p.E + e] = __float2bfloat16_rn(sc[j]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = nanmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float thr = bfr(__fmul_rn(m, p.mult));
    int kept = 0;
#pragma unroll
    for (int j = 0; j < MAX_E / 32; ++j) {
      if (j >= nw) break;
      const int e = lane + 32 * j;
      const bool keep = e < p.E && sc[j] >= thr;
      const uint32_t word = __ballot_sync(0xffffffffu, keep);
      kept += __popc(word);
      if (lane == 0) p.mask_bits[t * nw + j] = word;
      if (p.rt_out && e < p.E) p.rt_out[t * p.E + e] = __float2bfloat16_rn(keep ? 1.f : 0.f);
    }
    if (p.out_init && (p.init_all || kept != 1)) {
      for (int c8 = lane; c8 < v8; c8 += 32) {
        uint4 o = make_uint4(0u, 0u, 0u, 0u);
        if (p.last_bias) o = __ldg(reinterpret_cast<const uint4*>(p.last_bias) + c8);
        if (p.resid)
          o = add_bf16x8(o, __ldg(reinterpret_cast<const uint4*>(p.resid + t * p.d) + c8));
        *(reinterpret_cast<uint4*>(p.out_init + t * p.d) + c8) = o;
      }
    }
  }
  cluster.sync();                // the others may still read this CTA's shares
  if (p.token_idx && rank == 0) {
    // one tile: its lists from the mask words that the cluster has written (visible since the
    // barrier), 32 tokens a warp
    uint32_t* rows = reinterpret_cast<uint32_t*>(smem_raw + (ring - raw));      // [4][MAX_E]
    int* off = reinterpret_cast<int*>(rows + 4 * MAX_E);
    if (warp < 4) {
      const long long t = 32 * warp + lane;
#pragma unroll
      for (int j = 0; j < MAX_E / 32; ++j) {
        const uint32_t word =
            j < nw && t < p.N ? *const_cast<volatile uint32_t*>(p.mask_bits + t * nw + j) : 0u;
        rows[warp * MAX_E + 32 * j + lane] = transpose32(word, lane);
      }
    }
    __syncthreads();
    if (warp == 0) {             // four experts per lane
      int v[4], s = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int e = 4 * lane + k;
        v[k] = 0;
        if (e < p.E)
          for (int q = 0; q < 4; ++q) v[k] += __popc(rows[q * MAX_E + e]);
        s += v[k];
      }
      int incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      int run = incl - s;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int e = 4 * lane + k;
        if (e < p.E) off[e] = p.offsets[e] = run;
        run += v[k];
      }
      if (lane == 31) p.offsets[p.E] = incl;
    }
    __syncthreads();
    for (int i = tid; i < 4 * p.E; i += CL_THREADS) {
      const int q = i / p.E, e = i - q * p.E;
      int at = off[e];
      for (int k = 0; k < q; ++k) at += __popc(rows[k * MAX_E + e]);
      for (uint32_t m = rows[q * MAX_E + e]; m != 0u; m &= m - 1)
        p.token_idx[at++] = 32 * q + __ffs(m) - 1;
    }
  }
}

__global__ void prepack_router_kernel(const bf16* __restrict__ wa, const bf16* __restrict__ wb,
                                      uint8_t* __restrict__ packed, Geo g, int d, int R, int E) {
  const long long n1 = (long long)g.kc1 * g.nsub * g.nsubw * 64;
  const long long n2 = (long long)g.kc2 * g.nd * 64;
  const bf16 zero = __float2bfloat16_rn(0.f);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n1 + n2;
       i += (long long)gridDim.x * blockDim.x) {
    if (i < n1) {
      const int k = (int)(i % 64);
      const int n = (int)((i / 64) % g.nsubw);
      const int sub = (int)((i / (64LL * g.nsubw)) % g.nsub);
      const int kc = (int)(i / (64LL * g.nsubw * g.nsub));
      const bf16 v = wa[(long long)(sub * g.nsubw + n) * d + kc * 64 + k];
      *reinterpret_cast<bf16*>(packed + (long long)(kc * g.nsub + sub) * g.nsubw * 128 +
                               swz(n, k)) = v;
    } else {
      const long long q = i - n1;
      const int k = (int)(q % 64);
      const int n = (int)((q / 64) % g.nd);
      const int k2 = (int)(q / (64LL * g.nd));
      const int kk = k2 * 64 + k;
      const bf16 v = (n < E && kk < R) ? wb[(long long)n * R + kk] : zero;
      *reinterpret_cast<bf16*>(packed + g.w1_bytes + (long long)k2 * g.nd * 128 + swz(n, k)) = v;
    }
  }
}

size_t smem_bytes(const Geo& g) {
  const size_t stage = SLOT + (size_t)(g.wa_bytes + 1023) / 1024 * 1024;
  const size_t wb = (size_t)(g.kc2 * g.nd * 128 + 1023) / 1024 * 1024;
  return 1024 + g.ns * stage + wb + sizeof(Ctl) + 64;
}

static_assert(1024 + SMEM_TILES + 1024 + sizeof(Ctl) + 64 <= 232448,
              "shared-memory plan exceeds the 227 KB a CTA may use");

}  // namespace

bool umma_router_supported(int d, int R, int E, int dtype) {
  return dtype == D2D_BF16 && d >= 64 && d % 64 == 0 && R >= 16 && R % 16 == 0 &&
         (R <= 128 || R == 256) && E >= 1 && E <= MAX_E;
}

size_t umma_router_packed_bytes(int d, int R, int E) { return (size_t)router_geo(d, R, E).stride; }

int launch_prepack_router(const void* wa, const void* wb, void* packed, int d, int R, int E,
                          cudaStream_t s) {
  const Geo g = router_geo(d, R, E);
  prepack_router_kernel<<<64, 256, 0, s>>>((const bf16*)wa, (const bf16*)wb, (uint8_t*)packed, g, d,
                                           R, E);
  return cudaGetLastError() == cudaSuccess ? D2D_OK : D2D_ERR_LAUNCH;
}

// The cluster form: one cluster of eight per tile, and a Wa worth splitting; it writes no counts table,
// so the mask has to be short enough for the scatter kernel to count itself.  Fifteen clusters run at
// once (the SMs of a cluster are one GPC's); a sixteenth waits for one to end, which only the largest
// Wa still pay for.  Layer of 24 experts x 32, us, one CTA per tile -> cluster:
//   2048 x 256 (512 K values):    32 tokens 30.5 -> 25.6, 1024 46.2 -> 37.4, 1800 54.4 -> 44.8, 2048 54.8 -> 55.1
//                                 (128 gated experts x 128, 2048 tokens: 121 -> 116)
//   2048 x 128 / 1024 x 256 (256 K): 32 tokens 25.8 -> 25.4 / 20.8 -> 18.1, 1024 41.6 -> 37.0 / 30.7 -> 26.8,
//                                    2048 50.3 -> 55.0 / 35.4 -> 38.1; 1536 x 256 with 2048 45.0 -> 46.5
//   below the line: 768 x 256 (192 K) 32 tokens 18.8 -> 16.7, 1024 26.4 -> 23.9; 768 x 128 (96 K) 18.9 -> 19.0
//   with 197, 24.2 -> 23.6 with 1024.  It would pay from about 128 K on.
bool umma_router_splits(int64_t N, int d, int R, int E) {
  const int64_t wa = (int64_t)d * R;
  return wa >= 256 * 1024 && N <= (wa >= 512 * 1024 ? 16 : 15) * TILE_M && R % (16 * CL) == 0 &&
         compact_counts_itself(N, E);
}

// The ranked rules without a launch of their own (layer of 24 experts x 128, us, own launch -> in the
// router): 197 tokens, topk 1 21.8 -> 20.6; 12608 tokens, topk 2 47.2 -> 45.3, topk 8 88.8 -> 83.2,
// dynk 71.1 -> 69.2; 25216 tokens, topk 4 92.6 -> 88.4.  Beyond 32 scores a thread's registers would
// not hold them beside their shares.
bool umma_router_ranks(int64_t N, int d, int R, int E) {
  return E <= 32 && !umma_router_splits(N, d, R, E);
}

int launch_router_mask_umma(const void* x, const void* packed, float mult, uint32_t* mask_bits,
                            void* scores, void* rt_out, const void* last_bias, const void* resid,
                            void* out_init, bool init_all, int32_t* tile_counts, int64_t N, int d,
                            int R, int E, int* dev_status, cudaStream_t s, ListsOut* lists,
                            int rule, int k, float tau) {
  Params p = {};
  p.N = N;
  p.d = d;
  p.R = R;
  p.E = E;
  p.packed = (const uint8_t*)packed;
  p.g = router_geo(d, R, E);
  p.mult = mult;
  p.k = k;
  p.tau = tau;
  p.mask_bits = mask_bits;
  p.scores = (bf16*)scores;
  p.rt_out = (bf16*)rt_out;
  p.tile_counts = reinterpret_cast<uint8_t*>(tile_counts);
  p.EP = compact_row_cells(E);
  p.out_init = (bf16*)out_init;
  p.last_bias = (const bf16*)last_bias;
  p.resid = (const bf16*)resid;
  p.init_all = init_all ? 1 : 0;
  p.dev_status = dev_status;
  umma_debug_read(&p.wait_limit, &p.withhold);
  const int64_t tiles = (N + TILE_M - 1) / TILE_M;
  // x as boxes of 64 columns x 128 consecutive rows; rows past the last token arrive as zeros
  alignas(64) CUtensorMap tmx;
  int rc = encode_tmap_2d_b16(&tmx, x, (uint64_t)d, (uint64_t)N, (uint64_t)d * 2, 64, TILE_M, true);
  if (rc != D2D_OK) return rc == D2D_ERR_BAD_ARG ? D2D_ERR_LAUNCH : rc;
  const bool split = umma_router_splits(N, d, R, E);
  if (lists && lists->table && !split && tiles > CLUSTER_TILES) {
    p.mt = mask_table(lists->table, N, E);
    p.tile_counts = p.mt.counts;
    lists->tabled = true;
  }
  if (lists && tiles <= (split ? 1 : CLUSTER_TILES)) {
    p.token_idx = lists->token_idx;
    p.offsets = lists->offsets;
    lists->written = true;
  }
  if (split) {
    const size_t wa_stage = SLOT + (size_t)(R / CL * 128 + 1023) / 1024 * 1024;
    const size_t smem = 1024 + CL_NS * wa_stage + (size_t)p.g.nd * 128 + sizeof(ClCtl) + 64;
    static_assert((TILE_M * (MAX_E + 1)) * 4 <= CL_NS * SLOT, "shares fit the ring");
    rc = device_launch_facts((const void*)router_cluster_kernel, smem, nullptr);
    if (rc != D2D_OK) return rc;
    return launch_pdl(router_cluster_kernel, dim3((unsigned)(tiles * CL)), dim3(CL_THREADS), smem, s,
                      p, tmx);
  }
  const size_t smem = smem_bytes(p.g);
  int sms = 0;
  rc = device_launch_facts(nullptr, 0, &sms);
  if (rc != D2D_OK) return rc;
  const int64_t ctas = tiles < sms ? tiles : sms;
  p.ctas = (int)ctas;
  // Initial rows by the SMs that have no tile, see help_init_rows.  They write every row, the tile's own CTAs those of
  // tokens with several experts alone: the line follows the share of tokens that may be expected to have
  // them, 1 - E^(-2 (1 - mult)) for normal scores (the gap of the two largest of E is exponential).  Layer, us,
  // by the tiles' own CTAs / by others; 24 experts at mult 0.9 (share 0.47): 197 tokens 19.4 / 17.4, 1100 24.3 / 21.0,
  // 6304 28.1 / 26.0, 12 608 36.8 / 36.7, 14 171 (111 tiles) 37.7 / 37.9; at 0.95 (0.27): 11 483 (90) 30.2 / 29.2, 12 635
  // (99) 30.6 / 31.3; at 0.995 (0.03): 5723 (45) 25.8 / 25.8, 9435 (74) 27.6 / 28.3, 14 171 30.2 / 32.3; 96 experts at 0.9
  // (0.60): 14 171 45.7 / 44.5; 16 of d = 1536 at 0.9 (0.43): 12 635 58.9 / 57.8, 14 171 60.5 / 63.9; 16 of d = 4096 there:
  // 11 483 116.0 / 112.7, 12 635 140.6 / 144.3 (longer rows, written twice, no longer stay in L2); with 123 tiles 38.7 /
  // 44.0.  Half of the SMs if the rows of x are read for them: 788 21.9 / 19.3, 9456 26.6 / 24.5, 12 608 29.1 / 29.7.
  // An eighth where every row starts from last_bias (ranked rules: the tile's own warps write those before its
  // gate).  Top-k: 591 23.3 / 20.7, 985 26.9 / 24.5, 2167 27.1 / 26.5, 5319 35.0 / 35.3, 12 608 47.3 / 48.4.
  // (Short calls, one cluster: up to six more clusters, which are all there at once.)
  const int64_t more = p.token_idx ? tiles * std::min<int64_t>((sms - tiles) / tiles, 6) : sms - ctas;
  const double share = 1.0 - std::pow((double)E, -2.0 * (1.0 - mult));
  const double line = resid ? 0.5 : init_all ? 0.125 : std::min(0.75, 0.3 + share - d / 65536.0);
  const bool help = out_init && more > 0 && (double)tiles <= line * sms;
  if (help) {
    p.help_init = p.out_init;
    p.out_init = nullptr;
  }
  const bool warm = !p.token_idx, stages = warm && p.out_init && init_all && resid;
#define D2D_ROUTER_OF(RULE)                                                    \
  (help ? (warm ? router_tiles_kernel<RULE, true, INIT_OTHERS>                 \
                : router_tiles_kernel<RULE, false, INIT_OTHERS>)               \
        : stages ? router_tiles_kernel<RULE, true, INIT_STAGES>                \
                 : (warm ? router_tiles_kernel<RULE, true, INIT_TILE>          \
                         : router_tiles_kernel<RULE, false, INIT_TILE>))
  auto kernel = rule == D2D_RULE_TOPK   ? D2D_ROUTER_OF(D2D_RULE_TOPK)
                : rule == D2D_RULE_DYNK ? D2D_ROUTER_OF(D2D_RULE_DYNK)
                                        : D2D_ROUTER_OF(0);
#undef D2D_ROUTER_OF
  rc = device_launch_facts((const void*)kernel, smem, nullptr);
  if (rc != D2D_OK) return rc;
  return launch_pdl_cluster(p.token_idx ? (int)tiles : 0, kernel, dim3((unsigned)(ctas + (help ? more : 0))),
                            dim3(NTHREADS), smem, s, p, tmx);
}

}  // namespace d2d
