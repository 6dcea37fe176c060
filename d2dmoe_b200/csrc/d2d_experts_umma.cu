// Experts of the layer on the tensor cores (bf16, tcgen05 + TMEM): per (expert e, up to 128 rows
// of its token list)
//     h   = act(bf16(x[rows] W1[e]) + b1[e]) (* bf16(x[rows] W_up[e]))
//     out[rows] += bf16(h W2[e])
// fusing architectures/moe/moe_impls.py:93-180 (gathered first layer) and :244-301 (second layer +
// atomic add); h never leaves the SM's tensor memory.
//
// What bounds it: latency, not a unit.  A hand-over from the tensor pipe to a waiting thread
// (commit, mbarrier, wake-up) takes about 300 cycles and one back to the issuing thread as much
// again, an M = 128, K = 16 instruction N/2 + 43 cycles with A in shared memory and N/2 + 10 with
// A in tensor memory.  The previous form (hidden tile in shared memory, two accumulator-2
// buffers, separate draining and writing warps) ran 21k cycles per tile with no pipe above 30 %.
// Hence here
//   * the hidden tile replaces accumulator 1 in place: the second product reads its A operand
//     from tensor memory, and no shared memory is spent on it (rings of 128 + 48 KB);
//   * two tiles are in work at once: the first product of one runs while the second product of
//     the other runs and is written out;
//   * accumulator 2 has four 64-column buffers (gated form: two per tile), so that the
//     commit -> drain -> release -> issue loop of a buffer passes while the others are in use;
//   * eight warps drain accumulator 2, each on its own (convert, transpose through its own 4 KB,
//     add or store), in straight-line code: with twenty warps in eight different loops,
//     instruction fetch is what a branch costs;
//   * the lists are cut into equal tiles of a size that fills the last round of the persistent
//     grid; where there are fewer tiles than SMs the output columns are split as well.
//
// Tensor memory (512 columns).  Two-layer form: accumulator 1 / hidden of tile t at 128 (t & 1),
// accumulator-2 buffers at 256 + 64 b.  Gated form: a tile has a half (256 columns): gate at 0,
// up at H, hidden in place at 0, and once epilogue 1 is done two accumulator-2 buffers at 64
// and 192.
//
// Warps: 0-3 epilogue 1; 4-7 and 8-11 drain groups 0 and 1 (even and odd steps); 12-15 row gather
// (cp.async); 16 first product; 17 second product; 18 W1 tiles, 19 W2 tiles (bulk copies).
//
// Every wait is bounded: when one runs out the kernel records D2D_ERR_TIMEOUT in the status word,
// all roles leave their loops, TMEM is freed and the kernel returns.
#include <atomic>

#include "d2d_umma_api.cuh"
#include "d2d_umma_ptx.cuh"

namespace d2d {
using namespace umma;
namespace {

constexpr int NTHREADS = 640;
constexpr int WARP_DRAIN0 = 4, WARP_GATHER0 = 12, WARP_MMA1 = 16, WARP_MMA2 = 17, WARP_W1 = 18,
              WARP_W2 = 19;
constexpr int MAX_E = 128;
constexpr int NS_MAX = 8, NS2_MAX = 8;        // stages of the two rings (upper bounds)
constexpr int ND = 64;                        // output columns per step of the second product
constexpr int STG = 8 * 4096;                 // transposition blocks of the drain warps
constexpr int SMEM_TILES = 220 * 1024;        // both rings + STG

struct Geo {
  int kc1;         // d / 64
  int w1_stage;    // W1 (and W_up) bytes per 64-deep slice
  int kc2;         // ceil(H / 64)
  int nc;          // d / 64: steps of the second product
  int ns, ns2;     // ring stages
  int stage;       // bytes of a stage of the first ring: rows of x (16 KB), then w1_stage
  int w2_stage;    // W2 bytes per step: 64 output columns x kc2 slices
  long long w1_bytes, bias_off, stride;   // packed layout per expert
};

Geo experts_geo(int d, int H, bool glu) {
  Geo g;
  g.kc1 = d / 64;
  g.w1_stage = (glu ? 2 : 1) * H * 128;
  g.kc2 = (H + 63) / 64;
  g.nc = d / ND;
  g.stage = SLOT + g.w1_stage;
  g.w2_stage = g.kc2 * ND * 128;
  // at least three steps of W2, then as many stages of the first ring as fit, the rest for W2
  const int ns = (SMEM_TILES - STG - 3 * g.w2_stage) / g.stage;
  g.ns = ns < NS_MAX ? ns : NS_MAX;
  const int ns2 = (SMEM_TILES - STG - g.ns * g.stage) / g.w2_stage;
  g.ns2 = ns2 < NS2_MAX ? ns2 : NS2_MAX;
  g.w1_bytes = (long long)g.kc1 * g.w1_stage;
  g.bias_off = g.w1_bytes + (long long)g.nc * g.w2_stage;
  g.stride = (g.bias_off + 512 + 1023) / 1024 * 1024;
  return g;
}

struct Params {
  const bf16* x;
  long long N;
  int d, E, H, act;
  const uint8_t* packed;
  Geo g;
  const int32_t* token_idx;
  const int32_t* offsets;
  bf16* out;
  const uint32_t* mask_bits;   // optional: see DirectRows
  const bf16* last_bias;
  int* dev_status;
  uint32_t wait_limit;         // polls per bounded wait
  int withhold;                // test hook: CTA 0 never loads its first weight tile
  bf16* norms;                 // optional: [E, N] norms of each computed pair's activations
  int norm_layer, norm_ord;    // D2D_NORM_OF_INTERMEDIATE / D2D_NORM_OF_OUTPUT (0: none); 1 or 2
};

struct Ctl {
  unsigned long long full[NS_MAX], empty[NS_MAX], full2[NS2_MAX], empty2[NS2_MAX];
  unsigned long long acc1_full[2], ctx_free[2], hid_full[2], acc2_full[4], acc2_empty[4];
  unsigned long long list_full[2], list_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int wait_limit;                  // must follow abort_flag (mbar_wait reads abort_flag[1])
  int total_tiles;                 // tiles x column parts
  int parts;                       // column parts per tile
  int dense_e;                     // > 0: every expert lists all N tokens (number of experts)
  alignas(16) uint32_t bias_s[2][64];   // b1 of the tile's expert as bf16 pairs
  int list[2][128];                // the tile's tokens; sign bit: row is stored; -1: no row
  float npart[128];                // row norm terms of drain group 1
  int off[MAX_E + 1];              // list offsets
  int tstart[MAX_E + 1];           // first tile of each expert
  int rows[MAX_E];                 // rows per tile of each expert
};

// columns of tile t's tensor memory, and of its accumulator-2 buffer b
template <bool GLU>
__device__ __forceinline__ uint32_t tm_tile(uint32_t tmem, uint32_t ctx) {
  return tmem + ctx * (GLU ? 256 : 128);
}
template <bool GLU>
__device__ __forceinline__ uint32_t tm_acc2(uint32_t tmem, uint32_t b) {
  return GLU ? tmem + (b >> 1) * 256 + (b & 1) * 128 + 64 : tmem + 256 + b * 64;
}

struct Tile {
  int e, r0, nrows, n0, n1;        // rows of the token list, steps of the second product
};

__device__ __forceinline__ Tile tile_info(const Params& p, const Ctl* c, int tile) {
  Tile t;
  int part = 0;
  const int parts = c->parts;
  if (parts > 1) {
    part = tile % parts;
    tile /= parts;
  }
  t.n0 = part * p.g.nc / parts;
  t.n1 = (part + 1) * p.g.nc / parts;
  int k;
  if (c->dense_e > 0) {
    // Every expert runs on every token (mode 'all' upstream: router training, label capture):
    // window-major order, the E tiles of one window of tokens next to each other, so that the
    // window's rows of x and out stay in L2.
    k = tile / p.E;
    t.e = tile - k * p.E;
  } else {
    int lo = 0, hi = p.E;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (c->tstart[mid] <= tile) lo = mid; else hi = mid;
    }
    t.e = lo;
    k = tile - c->tstart[lo];
  }
  t.r0 = c->off[t.e] + k * c->rows[t.e];
  t.nrows = min(c->rows[t.e], c->off[t.e + 1] - t.r0);
  return t;
}

// ---------------------------------------------------------------------------
// roles
// ---------------------------------------------------------------------------
// Warps 12-15: rows of x by 16-byte cp.async (4 rows x 128 bytes per warp instruction, software
// swizzle; a TMA gather spends a request per 128-byte row and was 1.6 times slower).  Inside
// a warp's 32 rows those that are stored come first, so that an output instruction (4 rows)
// mostly does one thing.  Rows past the list's end are not loaded: whatever their slots hold
// reaches only accumulator rows nobody reads.
__device__ void role_gather(const Params& p, Ctl* c, uint32_t ring, int w, int lane) {
  volatile int* af = &c->abort_flag;
  const int j = lane & 7, nw = (p.E + 31) >> 5, total = c->total_tiles;
  uint32_t dstoff[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = w * 32 + i * 4 + (lane >> 3);
    dstoff[i] = (row >> 3) * 1024 + (row & 7) * 128 + ((j ^ (row & 7)) << 4);
  }
  int tok = -1, kept = 0;
  bool mine = false;
  auto fetch = [&](int tile) {           // token of my row, -1: none
    tok = -1;
    mine = false;
    if (tile >= total) return;
    const Tile t = tile_info(p, c, tile);
    mine = w * 32 + lane < t.nrows;
    if (mine) tok = p.token_idx[t.r0 + w * 32 + lane];
  };
  auto fetch_kept = [&]() {              // how many experts keep it
    kept = 0;
    if (mine && (tok < 0 || tok >= p.N)) {
      report(p.dev_status, D2D_ERR_INDEX_RANGE);
      tok = -1;
    }
    if (p.mask_bits && tok >= 0)
      for (int q = 0; q < nw; ++q) kept += __popc(p.mask_bits[(long long)tok * nw + q]);
  };
  fetch(blockIdx.x);
  fetch_kept();
  RingPos r = {0, 0};
  uint32_t b = 0, ph = 0;
  for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
    if (!mbar_wait_fast(smem_u32(&c->list_empty[b]), ph ^ 1, af, p.dev_status)) return;
    int* list = c->list[b] + w * 32;
    {
      const bool direct = kept == 1;
      const uint32_t dm = __ballot_sync(0xffffffffu, direct), lt = (1u << lane) - 1u;
      const uint32_t live = __ballot_sync(0xffffffffu, tok >= 0) & ~dm;
      const uint32_t none = ~(dm | live);
      const int slot = direct     ? __popc(dm & lt)
                       : tok >= 0 ? __popc(dm) + __popc(live & lt)
                                  : __popc(dm | live) + __popc(none & lt);
      list[slot] = tok < 0 ? -1 : direct ? (int)((uint32_t)tok | 0x80000000u) : tok;
      __syncwarp();
    }
    const bf16* src[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int v = list[i * 4 + (lane >> 3)];
      src[i] = v == -1 ? nullptr : p.x + (size_t)(v & 0x7fffffff) * p.d + j * 8;
    }
    mbar_arrive(smem_u32(&c->list_full[b]));
    ph ^= b;
    b ^= 1;
    fetch(tile + gridDim.x);             // in flight while this tile's rows are gathered
    const int kmask = p.g.kc1 > 2 ? 2 : p.g.kc1 - 1;
    for (int kc = 0; kc < p.g.kc1; ++kc) {
      if (!mbar_wait_fast(smem_u32(&c->empty[r.s]), r.ph ^ 1, af, p.dev_status)) return;
      const uint32_t base = ring + r.s * p.g.stage;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (src[i]) cp_async16(base + dstoff[i], src[i] + kc * 64);
      cp_async_arrive_noinc(smem_u32(&c->full[r.s]));
      r.next(p.g.ns);
      if (kc == kmask) fetch_kept();
    }
  }
}

// The four roles below each run in ONE thread of their warp for the whole launch: their loops are
// chains of dependent instructions, votes and re-convergence would only lengthen the chain.
__device__ void role_w1(const Params& p, Ctl* c, uint32_t ring) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  bool withheld = (p.withhold & 1) != 0 && blockIdx.x == 0;
  RingPos r = {0, 0};
  for (int tile = blockIdx.x; tile < c->total_tiles; tile += gridDim.x) {
    const uint8_t* src = p.packed + (long long)tile_info(p, c, tile).e * g.stride;
    for (int kc = 0; kc < g.kc1; ++kc, src += g.w1_stage) {
      if (!mbar_wait_fast(smem_u32(&c->empty[r.s]), r.ph ^ 1, af, p.dev_status)) return;
      const uint32_t bar = smem_u32(&c->full[r.s]);
      mbar_arrive_expect_tx(bar, g.w1_stage);
      if (withheld) withheld = false;    // test hook: this stage never fills, its wait runs out
      else bulk_g2s(ring + r.s * g.stage + SLOT, src, g.w1_stage, bar);
      r.next(g.ns);
    }
  }
}

__device__ void role_w2(const Params& p, Ctl* c, uint32_t ring2) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  RingPos r = {0, 0};
  for (int tile = blockIdx.x; tile < c->total_tiles; tile += gridDim.x) {
    const Tile t = tile_info(p, c, tile);
    const uint8_t* src = p.packed + (long long)t.e * g.stride + g.w1_bytes;
    for (int n = t.n0; n < t.n1; ++n) {
      if (!mbar_wait_fast(smem_u32(&c->empty2[r.s]), r.ph ^ 1, af, p.dev_status)) return;
      const uint32_t bar = smem_u32(&c->full2[r.s]);
      mbar_arrive_expect_tx(bar, g.w2_stage);
      bulk_g2s(ring2 + r.s * g.w2_stage, src + (long long)n * g.w2_stage, g.w2_stage, bar);
      r.next(g.ns2);
    }
  }
}

// first product (N = H, gated form N = 2 H in one instruction).  Only the low word of a
// shared-memory descriptor changes (16-byte units; one k-step = 2).
template <bool GLU>
__device__ void role_mma1(const Params& p, Ctl* c, uint32_t ring, uint32_t tmem) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const uint32_t idesc = instr_desc(TILE_M, g.w1_stage >> 7);
  const uint64_t d0 = smem_desc(ring);
  const uint64_t hi = (d0 >> 32) << 32;
  const uint32_t lo0 = (uint32_t)d0;
  RingPos r = {0, 0};
  uint32_t ctx = 0, ph = 0;
  for (int tile = blockIdx.x; tile < c->total_tiles; tile += gridDim.x) {
    const uint32_t acc = tm_tile<GLU>(tmem, ctx);
    if (!mbar_wait_fast(smem_u32(&c->ctx_free[ctx]), ph ^ 1, af, p.dev_status)) return;
    tc_fence_after();
    for (int kc = 0; kc < g.kc1; ++kc) {
      if (!mbar_wait_fast(smem_u32(&c->full[r.s]), r.ph, af, p.dev_status)) return;
      tc_fence_after();
      const uint32_t alo = lo0 + r.s * ((uint32_t)g.stage >> 4), blo = alo + (SLOT >> 4);
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k)
        umma_bf16(acc, hi | (alo + 2 * k), hi | (blo + 2 * k), idesc, (kc | k) != 0);
      umma_commit(smem_u32(&c->empty[r.s]));
      r.next(g.ns);
    }
    umma_commit(smem_u32(&c->acc1_full[ctx]));
    ph ^= ctx;
    ctx ^= 1;
  }
}

// second product: one 64-column step after another, each into the next accumulator-2 buffer
template <bool GLU>
__device__ void role_mma2(const Params& p, Ctl* c, uint32_t ring2, uint32_t tmem) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const uint32_t idesc = instr_desc(TILE_M, ND);
  const uint64_t d0 = smem_desc(ring2);
  const uint64_t hi = (d0 >> 32) << 32;
  const uint32_t lo0 = (uint32_t)d0;
  const int ks = p.H >> 4;
  RingPos r = {0, 0};
  uint32_t ctx = 0, ph = 0, step = 0, uses = 0;   // uses: bit b = parity of buffer b's uses so far
  for (int tile = blockIdx.x; tile < c->total_tiles; tile += gridDim.x) {
    const Tile t = tile_info(p, c, tile);
    const uint32_t hid = tm_tile<GLU>(tmem, ctx);
    if (GLU) step = 0;
    if (!mbar_wait_fast(smem_u32(&c->hid_full[ctx]), ph, af, p.dev_status)) return;
    for (int n = t.n0; n < t.n1; ++n, ++step) {
      const uint32_t b = GLU ? 2 * ctx + (step & 1) : step & 3;
      if (!mbar_wait_fast(smem_u32(&c->full2[r.s]), r.ph, af, p.dev_status)) return;
      if (!mbar_wait_fast(smem_u32(&c->acc2_empty[b]), ((uses >> b) & 1) ^ 1, af, p.dev_status))
        return;
      uses ^= 1u << b;
      tc_fence_after();
      const uint32_t acc = tm_acc2<GLU>(tmem, b), blo = lo0 + r.s * ((uint32_t)g.w2_stage >> 4);
      umma_bf16_ta(acc, hid, hi | blo, idesc, 0);
#pragma unroll
      for (int k = 1; k < 8; ++k)
        if (k < ks)
          umma_bf16_ta(acc, hid + 8 * k, hi | (blo + (k >> 2) * (ND * 8) + 2 * (k & 3)), idesc, 1);
      umma_commit(smem_u32(&c->acc2_full[b]));
      umma_commit(smem_u32(&c->empty2[r.s]));
      r.next(g.ns2);
    }
    // the hidden tile has been read (gated form: the drain warps free the tile's columns)
    if (!GLU) umma_commit(smem_u32(&c->ctx_free[ctx]));
    ph ^= ctx;
    ctx ^= 1;
  }
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

// Warps 0-3, thread = tile row = TMEM lane: accumulator 1 -> bias, activation (x
// up-projection) -> bf16 hidden tile over the columns already read.
template <int ACT, bool GLU, bool NORM>
__device__ void role_ep1(const Params& p, Ctl* c, uint32_t tmem, int et) {
  volatile int* af = &c->abort_flag;
  const uint32_t lane_base = (uint32_t)(et & ~31) << 16;
  const int nord = p.norm_ord;
  uint32_t ctx = 0, ph = 0;
  for (int tile = blockIdx.x; tile < c->total_tiles; tile += gridDim.x) {
    const Tile t = tile_info(p, c, tile);
    // two copies of the bias alternate: a warp already on the next tile never overwrites pairs
    // another warp still reads
    uint32_t* bp = c->bias_s[ctx];
    if (et < (p.H >> 1)) {
      const float2 b = __ldg(reinterpret_cast<const float2*>(p.packed + (long long)t.e * p.g.stride +
                                                             p.g.bias_off) + et);
      bp[et] = pack_bf16x2(b.x, b.y);
    }
    asm volatile("bar.sync 2, 128;" ::: "memory");
    // labels by-product (intermediate layer): this thread's row, its token loaded up front
    float nacc = 0.f;
    int ntok = -1;
    if (NORM) {
      if (!mbar_wait_fast(smem_u32(&c->list_full[ctx]), ph, af, p.dev_status)) return;
      ntok = c->list[ctx][et];
    }
    if (!mbar_wait_fast(smem_u32(&c->acc1_full[ctx]), ph, af, p.dev_status)) return;
    tc_fence_after();
    const uint32_t acc = tm_tile<GLU>(tmem, ctx) + lane_base;
    for (int c0 = 0; c0 < p.H; c0 += 16) {
      uint32_t v[16], u[16], w[8], bb[8];
      tmem_ld16(acc + c0, v);
      if (GLU) tmem_ld16(acc + p.H + c0, u);
      const uint4 q0 = *reinterpret_cast<const uint4*>(bp + (c0 >> 1));
      const uint4 q1 = *reinterpret_cast<const uint4*>(bp + (c0 >> 1) + 4);
      bb[0] = q0.x; bb[1] = q0.y; bb[2] = q0.z; bb[3] = q0.w;
      bb[4] = q1.x; bb[5] = q1.y; bb[6] = q1.z; bb[7] = q1.w;
      tmem_wait_ld();
      ep1_pairs<ACT, GLU, NORM>(v, u, bb, w, nacc, nord);
      tmem_st8(acc + (c0 >> 1), w);
    }
    tmem_wait_st();
    tc_fence_before();
    mbar_arrive(smem_u32(&c->hid_full[ctx]));
    if (NORM && ntok != -1)
      p.norms[(long long)t.e * p.N + (ntok & 0x7fffffff)] =
          __float2bfloat16_rn(nord == 1 ? nacc : sqrtf(nacc));
    ph ^= ctx;
    ctx ^= 1;
  }
}

// t >= 0: add; t < -1: store; -1: nothing (predicated, no branch)
__device__ __forceinline__ void put_row(bf16* p, int t, uint4 add, uint4 st) {
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

template <bool GLU, bool NORM>
__device__ __forceinline__ void role_ep1_act(const Params& p, Ctl* c, uint32_t tmem, int et) {
  switch (p.act) {         // one loop per activation: no branch inside
    case D2D_RELU: role_ep1<D2D_RELU, GLU, NORM>(p, c, tmem, et); break;
    case D2D_GELU: role_ep1<D2D_GELU, GLU, NORM>(p, c, tmem, et); break;
    case D2D_TANH: role_ep1<D2D_TANH, GLU, NORM>(p, c, tmem, et); break;
    case D2D_LEAKY_RELU: role_ep1<D2D_LEAKY_RELU, GLU, NORM>(p, c, tmem, et); break;
    default: role_ep1<D2D_GELU_TANH, GLU, NORM>(p, c, tmem, et); break;
  }
}

// Warps 4-11: drain group j takes every other step; warp q4 of it rows 32 q4 .. +31.
// Thread = row out of tensor memory; through the warp's own 4 KB the 64 columns are turned into
// 8 lanes per row, so that one instruction covers 4 whole 128-byte lines of the output.
// The loop is straight-line code: with the norm terms and the store / add choice as branches inside
// it, a step of some 150 instructions took 2900 cycles, most of them waiting for instructions
// (twenty warps in eight different loops share the instruction caches).
template <bool GLU, bool NORM>
__device__ void role_drain(const Params& p, Ctl* c, uint32_t stg, uint32_t tmem, int j, int q4,
                           int lane) {
  volatile int* af = &c->abort_flag;
  const uint32_t lane_base = (uint32_t)(q4 * 32) << 16;
  const uint32_t blk = stg + (j * 4 + q4) * 4096;
  const uint32_t wr = blk + lane * 128, x7 = lane & 7;
  const int rl = lane >> 3, pl = lane & 7;
  const int nord = p.norm_ord;
  uint32_t ctx = 0, ph = 0, step = 0, uses = 0;    // uses: bit b = parity of buffer b's uses so far
  for (int tile = blockIdx.x; tile < c->total_tiles; tile += gridDim.x) {
    const Tile t = tile_info(p, c, tile);
    if (!mbar_wait_fast(smem_u32(&c->list_full[ctx]), ph, af, p.dev_status)) return;
    const int* list = c->list[ctx] + q4 * 32;
    int rt[8];
#pragma unroll
    for (int it = 0; it < 8; ++it) rt[it] = list[it * 4 + rl];
    const int mine = list[lane];
    const bool any_direct = __any_sync(0xffffffffu, mine < -1);
    // (epilogue 1 reads the list as well where it collects norms: keep it until the tile is done)
    __syncwarp();
    if (lane == 0 && p.norm_layer == 0) mbar_arrive(smem_u32(&c->list_empty[ctx]));
    float nacc = 0.f;
    if (GLU) step = 0;
    const int first = t.n0 + ((step + j) & 1);       // my first step of this tile
    const uint32_t step0 = step;
    step += t.n1 - t.n0;
    for (int n = first; n < t.n1; n += 2) {
      const uint32_t q = step0 + (n - t.n0), b = GLU ? 2 * ctx + (q & 1) : q & 3;
      bf16* o = p.out + n * ND + pl * 8;
      uint4 bz = make_uint4(0u, 0u, 0u, 0u);
      if (any_direct && p.last_bias)
        bz = __ldg(reinterpret_cast<const uint4*>(p.last_bias + n * ND + pl * 8));
      if (!mbar_wait_fast(smem_u32(&c->acc2_full[b]), (uses >> b) & 1, af, p.dev_status)) return;
      uses ^= 1u << b;
      tc_fence_after();
      uint32_t v[64];
      const uint32_t acc = tm_acc2<GLU>(tmem, b) + lane_base;
      tmem_ld32(acc, v);
      tmem_ld32(acc + 32, v + 32);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c->acc2_empty[b]));
#pragma unroll
      for (int pc = 0; pc < 8; ++pc) {      // piece XOR row: conflict-free 16-byte stores
        uint32_t ww[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ww[k] = pack_bf16x2(__uint_as_float(v[8 * pc + 2 * k]),
                              __uint_as_float(v[8 * pc + 2 * k + 1]));
        st_shared_v4(wr + ((pc ^ x7) << 4), ww[0], ww[1], ww[2], ww[3]);
        if (NORM) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float lo = __uint_as_float(ww[k] << 16), hi = __uint_as_float(ww[k] & 0xffff0000u);
            nacc += nord == 1 ? fabsf(lo) + fabsf(hi) : fmaf(lo, lo, hi * hi);
          }
        }
      }
      __syncwarp();
      uint4 val[8];
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int rr = it * 4 + rl;
        val[it] = ld_shared_v4(blk + rr * 128 + ((pl ^ (rr & 7)) << 4));
      }
      __syncwarp();
      if (any_direct) {
#pragma unroll
        for (int it = 0; it < 8; ++it)
          put_row(o + (size_t)(rt[it] & 0x7fffffff) * p.d, rt[it], val[it],
                  add_bf16x8(bz, val[it]));
      } else {
#pragma unroll
        for (int it = 0; it < 8; ++it)
          put_row(o + (size_t)(rt[it] & 0x7fffffff) * p.d, rt[it], val[it], val[it]);
      }
    }
    // every read of this context's tensor memory by this warp is done
    __syncwarp();
    if (lane == 0) {
      if (GLU) mbar_arrive(smem_u32(&c->ctx_free[ctx]));
      if (p.norm_layer != 0) mbar_arrive(smem_u32(&c->list_empty[ctx]));
    }
    if (NORM) {
      // the other group saw the other steps of the same rows
      if (j == 1) c->npart[q4 * 32 + lane] = nacc;
      asm volatile("bar.sync 3, 256;" ::: "memory");
      if (j == 0) nacc += c->npart[q4 * 32 + lane];
      asm volatile("bar.sync 3, 256;" ::: "memory");
      if (mine != -1 && j == 0)
        p.norms[(long long)t.e * p.N + (mine & 0x7fffffff)] =
            __float2bfloat16_rn(nord == 1 ? nacc : sqrtf(nacc));
    }
    ph ^= ctx;
    ctx ^= 1;
  }
}

// ---------------------------------------------------------------------------
// kernel
// ---------------------------------------------------------------------------
// One warp cuts the lists into tiles.  Candidate sizes are eighths of the largest tile; a tile
// costs its weights plus its rows' bytes, and the launch as many tiles as the fullest CTA
// gets, so the size that fills the last round of the grid wins (524 rows per SM: five tiles of
// 105 rows instead of four of 128 and one of 12).  Rates: 64 bytes per clock and SM for loads, 24 for the
// output, measured on an SM's memory interface alone.
__device__ void cut_tiles(const Params& p, Ctl* c, int lane) {
  const int E = p.E, unit = TILE_M / 8;
  int off[5], n[4];
  bool all_n = true;                     // every expert of this lane lists exactly N tokens
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const int e = 4 * lane + q;
    off[q] = e <= E ? p.offsets[e] : 0;
    if (e <= E) c->off[e] = off[q];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = 4 * lane + q;
    n[q] = e < E ? off[q + 1] - off[q] : 0;
    if (e < E && n[q] != p.N) all_n = false;
    if (e < E && (n[q] < 0 || off[q] < 0 || off[q + 1] > p.N * (long long)E)) {
      report(p.dev_status, D2D_ERR_INDEX_RANGE);
      n[q] = 0;
    }
    n[q] = max(n[q], 0);
  }
  const unsigned grid = gridDim.x;
  const unsigned fixed = (unsigned)(p.g.bias_off >> 6) + 2000, per_row = (unsigned)p.d / 8;
  unsigned best_cost = 0xffffffffu, tiles = 0;
  int best = 8;
  for (int k = 8; k >= 1; --k) {
    unsigned mine = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) mine += (unsigned)(n[q] + k * unit - 1) / (unsigned)(k * unit);
    const unsigned T = __reduce_add_sync(0xffffffffu, mine);
    const unsigned cost = ((T + grid - 1) / grid) * (fixed + k * unit * per_row);
    if (cost < best_cost) {
      best_cost = cost;
      best = k;
      tiles = T;
    }
  }
  const int size = best * unit;
  int sum = 0, nt[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = 4 * lane + q;
    nt[q] = (n[q] + size - 1) / size;
    if (e < E) c->rows[e] = nt[q] > 0 ? (n[q] + nt[q] - 1) / nt[q] : 1;   // equal tiles
    sum += nt[q];
  }
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  int run = incl - sum;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = 4 * lane + q;
    if (e <= E) c->tstart[e] = run;
    run += nt[q];
  }
  const bool dense = __all_sync(0xffffffffu, all_n) && E > 1;
  if (lane == 0) {
    // fewer than half as many tiles as CTAs: split the output columns (the first product is
    // repeated, the second product, W2 and the output are shared out)
    int parts = tiles > 0 ? (int)(grid / tiles) : 1;
    parts = max(1, min(parts, p.g.nc));
    if (p.norm_layer != 0) parts = 1;
    c->parts = parts;
    c->total_tiles = (int)tiles * parts;
    c->dense_e = dense ? E : 0;
  }
}

// NORM: 0 none, D2D_NORM_OF_INTERMEDIATE, D2D_NORM_OF_OUTPUT
template <bool GLU, int NORM>
__global__ void __launch_bounds__(NTHREADS, 1) experts_tiles_kernel(const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  const uint32_t ring2 = ring + p.g.ns * p.g.stage;
  const uint32_t stg = ring2 + p.g.ns2 * p.g.w2_stage;
  Ctl* c = reinterpret_cast<Ctl*>(smem_raw + (stg - raw) + STG);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Programmatic dependent launch: see router_tiles_kernel.
  grid_launch_dependents();

  if (tid == 0) {
    for (int i = 0; i < NS_MAX; ++i) {
      mbar_init(smem_u32(&c->full[i]), 129);          // 128 gather threads, one weight copy
      mbar_init(smem_u32(&c->empty[i]), 1);
    }
    for (int i = 0; i < NS2_MAX; ++i) {
      mbar_init(smem_u32(&c->full2[i]), 1);
      mbar_init(smem_u32(&c->empty2[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c->acc1_full[i]), 1);
      mbar_init(smem_u32(&c->ctx_free[i]), GLU ? 8 : 1);
      mbar_init(smem_u32(&c->hid_full[i]), 128);
      mbar_init(smem_u32(&c->list_full[i]), 128);
      mbar_init(smem_u32(&c->list_empty[i]), 8);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&c->acc2_full[i]), 1);
      mbar_init(smem_u32(&c->acc2_empty[i]), 4);
    }
    c->abort_flag = 0;
    c->wait_limit = (int)p.wait_limit;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == WARP_MMA1) tmem_alloc(smem_u32(&c->tmem_base), 512);
  grid_dependency_wait();
  if (warp == 1) cut_tiles(p, c, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c->tmem_base;

  if (warp < WARP_DRAIN0) {
    role_ep1_act<GLU, NORM == D2D_NORM_OF_INTERMEDIATE>(p, c, tmem, tid);
  } else if (warp < WARP_GATHER0) {
    const int w = warp - WARP_DRAIN0;
    role_drain<GLU, NORM == D2D_NORM_OF_OUTPUT>(p, c, stg, tmem, w >> 2, w & 3, lane);
  } else if (warp < WARP_MMA1) {
    role_gather(p, c, ring, warp - WARP_GATHER0, lane);
    cp_async_wait_all();
  } else if (warp == WARP_MMA1) {
    if (elect_one()) role_mma1<GLU>(p, c, ring, tmem);
    __syncwarp();
  } else if (warp == WARP_MMA2) {
    if (elect_one()) role_mma2<GLU>(p, c, ring2, tmem);
    __syncwarp();
  } else if (warp == WARP_W1) {
    if (elect_one()) role_w1(p, c, ring);
    __syncwarp();
  } else {
    if (elect_one()) role_w2(p, c, ring2);
    __syncwarp();
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
}

// Weights packed once into exactly the shared-memory images the MMA reads (K-major, 128-byte
// swizzle), so that a stage's weights are one contiguous bulk copy: per expert the 64-deep slices
// of W1 (gated form: H gate rows, then H up rows), the 64-column x 64-deep pieces of W2, b1 in fp32.
__global__ void prepack_experts_kernel(const bf16* __restrict__ w1, const bf16* __restrict__ b1,
                                       const bf16* __restrict__ w_up, const bf16* __restrict__ w2,
                                       uint8_t* __restrict__ packed, Geo g, int d, int E, int H) {
  const int e = blockIdx.y;
  uint8_t* pe = packed + (long long)e * g.stride;
  const int rows1 = g.w1_stage >> 7;
  const long long n1 = (long long)g.kc1 * rows1 * 64;
  const long long n2 = (long long)g.nc * g.kc2 * ND * 64;
  const bf16 zero = __float2bfloat16_rn(0.f);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n1 + n2 + H;
       i += (long long)gridDim.x * blockDim.x) {
    if (i < n1) {
      // consecutive threads: consecutive hidden columns (the contiguous direction of W1)
      const int n = (int)(i % rows1);
      const int k = (int)((i / rows1) % 64);
      const int kc = (int)(i / (64LL * rows1));
      const bf16* src = n < H ? w1 : w_up;
      const bf16 v = src[((long long)e * d + kc * 64 + k) * H + (n < H ? n : n - H)];
      *reinterpret_cast<bf16*>(pe + (long long)kc * g.w1_stage + swz(n, k)) = v;
    } else if (i < n1 + n2) {
      const long long q = i - n1;
      const int n = (int)(q % ND);
      const int k = (int)((q / ND) % 64);
      const int k2 = (int)((q / (64LL * ND)) % g.kc2);
      const int nci = (int)(q / (64LL * ND * g.kc2));
      const int kk = k2 * 64 + k;
      const bf16 v = kk < H ? w2[((long long)e * H + kk) * d + nci * ND + n] : zero;
      *reinterpret_cast<bf16*>(pe + g.w1_bytes + (long long)(nci * g.kc2 + k2) * (ND * 128) +
                               swz(n, k)) = v;
    } else {
      const int h = (int)(i - n1 - n2);
      reinterpret_cast<float*>(pe + g.bias_off)[h] =
          b1 ? __bfloat162float(b1[(long long)e * H + h]) : 0.f;
    }
  }
}

// test hooks (d2d_debug_configure): process-wide, read at launch
std::atomic<uint32_t> g_wait_limit{WAIT_LIMIT};
std::atomic<int> g_withhold{0};

static_assert(1024 + SMEM_TILES + sizeof(Ctl) + 64 <= 232448,
              "shared-memory plan exceeds the 227 KB a CTA may use");

}  // namespace

// ---------------------------------------------------------------------------
// host interface
// ---------------------------------------------------------------------------
bool umma_experts_supported(int d, int E, int H, bool glu, int dtype) {
  (void)glu;
  return dtype == D2D_BF16 && d >= 64 && d % 64 == 0 && H >= 16 && H <= 128 && H % 16 == 0 &&
         E >= 1 && E <= MAX_E;
}

size_t umma_experts_packed_bytes(int d, int E, int H, bool glu) {
  return (size_t)experts_geo(d, H, glu).stride * (size_t)E;
}

int launch_prepack_experts(const void* w1, const void* b1, const void* w_up, const void* w2,
                           void* packed, int d, int E, int H, cudaStream_t s) {
  const Geo g = experts_geo(d, H, w_up != nullptr);
  dim3 grid(64, E);
  prepack_experts_kernel<<<grid, 256, 0, s>>>((const bf16*)w1, (const bf16*)b1, (const bf16*)w_up,
                                              (const bf16*)w2, (uint8_t*)packed, g, d, E, H);
  return cudaGetLastError() == cudaSuccess ? D2D_OK : D2D_ERR_LAUNCH;
}

int launch_experts_umma(const void* x, const int32_t* token_idx, const int32_t* offsets,
                        const void* packed, void* out, int64_t N, int d, int E, int H, bool glu,
                        int act, int* dev_status, cudaStream_t s, NormCapture nc, DirectRows dr) {
  Params p = {};
  p.x = (const bf16*)x;
  p.N = N;
  p.d = d;
  p.E = E;
  p.H = H;
  p.act = act;
  p.packed = (const uint8_t*)packed;
  p.g = experts_geo(d, H, glu);
  p.token_idx = token_idx;
  p.offsets = offsets;
  p.out = (bf16*)out;
  p.mask_bits = dr.mask_bits;
  p.last_bias = (const bf16*)dr.last_bias;
  p.dev_status = dev_status;
  p.norms = (bf16*)nc.norms;
  p.norm_layer = nc.norms ? nc.layer : 0;
  p.norm_ord = nc.ord;
  umma_debug_read(&p.wait_limit, &p.withhold);
  const size_t smem =
      1024 + (size_t)p.g.ns * p.g.stage + (size_t)p.g.ns2 * p.g.w2_stage + STG + sizeof(Ctl) + 64;
  auto kernel = glu ? (p.norm_layer == 0                          ? experts_tiles_kernel<true, 0>
                       : p.norm_layer == D2D_NORM_OF_INTERMEDIATE ? experts_tiles_kernel<true, 1>
                                                                  : experts_tiles_kernel<true, 2>)
                    : (p.norm_layer == 0                          ? experts_tiles_kernel<false, 0>
                       : p.norm_layer == D2D_NORM_OF_INTERMEDIATE ? experts_tiles_kernel<false, 1>
                                                                  : experts_tiles_kernel<false, 2>);
  static_assert(D2D_NORM_OF_INTERMEDIATE == 1 && D2D_NORM_OF_OUTPUT == 2, "template arguments");
  int sms = 0;
  const int rc = device_launch_facts((const void*)kernel, smem, &sms);
  if (rc != D2D_OK) return rc;
  // at most one tile per kept pair, and column parts of it
  const long long most = N * (long long)E * p.g.nc;
  const long long grid = most < sms ? most : sms;
  return launch_pdl(kernel, dim3((unsigned)grid), dim3(NTHREADS), smem, s, p);
}

// one way of gathering rows is left; kept for callers of the entry point
void umma_debug_select_experts_kernel(int which) { (void)which; }

void umma_debug_read(uint32_t* wait_limit, int* withhold) {
  *wait_limit = g_wait_limit.load();
  *withhold = g_withhold.load();
}

void umma_debug_configure(int wait_limit_log2, int withhold_weight_tile) {
  g_wait_limit.store(wait_limit_log2 >= 4 && wait_limit_log2 <= 22 ? 1u << wait_limit_log2
                                                                    : WAIT_LIMIT);
  g_withhold.store(withhold_weight_tile ? 1 : 0);
}

}  // namespace d2d
