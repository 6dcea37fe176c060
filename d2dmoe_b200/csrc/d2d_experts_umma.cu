// Experts of the layer on the tensor cores (bf16, tcgen05 + TMEM): per (expert e, up to 128 rows
// of its token list)
//     h   = act(bf16(x[rows] W1[e]) + b1[e]) (* bf16(x[rows] W_up[e]))
//     out[rows] += bf16(h W2[e])
// fusing architectures/moe/moe_impls.py:93-180 (gathered first layer) and :244-301 (second layer +
// atomic add); h never leaves the SM's tensor memory.
//
// What bounds it: two chains of nearly the same length, no unit at its rate (the tensor pipe and DRAM are busy below
// 30 % of the time).  For 128 output columns of a tile the drain takes 1850 cycles (see role_drain) and the products
// 1450: an M = 128, K = 16 instruction takes 64 cycles at N = 128, but a role's wait, four of them and a
// commit 280, and a hand-over from the tensor pipe to a waiting thread (commit, mbarrier, wake-up) about 300, one
// back to the issuing thread as much again.  Hence
//   * the hidden tile replaces accumulator 1 in place: the second product reads its A operand
//     from tensor memory, and no shared memory is spent on it (rings of 160 + 48 KB);
//   * two tiles are in work at once: the first product of one runs while the second product of
//     the other runs and is written out;
//   * the second product works in steps of 128 output columns (64 where d or the tensor memory
//     does not allow it) over two or more accumulator-2 buffers: a step costs its issuing thread
//     some 300 cycles besides the products, so few and large ones;
//   * eight warps drain accumulator 2, each 64 columns of its 32 rows and on its own, from
//     registers to whole 128-byte lines of the output;
//   * the lists are cut into equal tiles of a size that fills the last round of the persistent
//     grid; where there are fewer tiles than SMs the output columns are split as well;
//   * on long calls there are no lists before this kernel: the gather warps find a tile's rows in a table
//     that the router leaves (single calls: 50432 tokens 95.1 -> 88.4 us per layer, 12608 x 12 narrow experts
//     39.6 -> 35.6; 131072 gated tokens gain nothing: scatter 12.3 -> 0, this kernel 587 -> 601, see role_gather);
//   * where the weights of all experts stay in L2, the tiles are taken window by window of the
//     token range, all experts of a window next to each other, so that a row of x is read and
//     a row of out is added to in L2 by every expert but the first; last window first, because
//     its rows are what the router has left in L2.
//
// Tensor memory (512 columns).  Two-layer form: accumulator 1 / hidden of tile t at 128 (t & 1),
// accumulator-2 buffers from 256 on (two of 128 or four of 64 columns).  Gated form: a tile has a
// half (256 columns): gate at 0, up at H, hidden in place at 0, and once epilogue 1 is done
// three 64-column accumulator-2 buffers from 64 on.
//
// Warps: 0-3 epilogue 1; 4-11 drain; 12-15 a tile's rows: tokens and gather (cp.async); 16 first product;
// 17 second product; 18 weights (bulk copies); 19 cuts the lists into tiles.  On calls with a mask table 0-11
// and 16-18 count it first.
//
// Every wait is bounded: when one runs out the kernel records D2D_ERR_TIMEOUT in the status word,
// all roles leave their loops, TMEM is freed and the kernel returns.
#include <atomic>

#include "d2d_experts_common.cuh"

namespace d2d {
using namespace umma;
namespace {

constexpr int NTHREADS = 640;
constexpr int WARP_DRAIN0 = 4, WARP_GATHER0 = 12, WARP_MMA1 = 16, WARP_MMA2 = 17, WARP_W = 18;
constexpr int TILE_RING = 4;                  // tiles known ahead of the slowest role
constexpr int TILE_READERS = 4 + 8 + 4 + 1 + 1 + 2;   // warps 0-15, both products, both weight streams
// Weights up to this size are taken to stay in L2 beside a window's rows.  Layer, us, windows / one
// window: up to 48 MB of weights the two are alike on 32768 and 65536 tokens (66.6 / 66.2 with 9 MB,
// 94.9 / 93.7 with 48) and windows win on 131072 (243.7 / 263.9 with 48 MB); from 96 MB on one window
// wins (432 / 412 on 131072 tokens, 273 / 248 on 32768 with 192 MB).  Where between 48 and 96 MB they
// meet has not been measured.
constexpr long long L2_WEIGHTS = 32 << 20;

struct Params {
  const bf16* x;
  long long N;
  int d, E, H, act;
  const uint8_t* packed;
  Geo g;
  int32_t* token_idx;
  int32_t* offsets;
  MaskTable mt;                // words null: the lists are there; else they are made here from the table
  bf16* out;
  const uint32_t* mask_bits;   // optional: see DirectRows
  const bf16* last_bias;
  int* dev_status;
  uint32_t wait_limit;         // polls per bounded wait
  int withhold;                // test hook: CTA 0 never loads its first weight tile
  bool warm;                   // list and gather warps: a first pass without data, see role_list
  bf16* norms;                 // optional: [E, N] norms of each computed pair's activations
  int norm_layer, norm_ord;    // D2D_NORM_OF_INTERMEDIATE / D2D_NORM_OF_OUTPUT (0: none); 1 or 2
};

struct Tile {
  int e;                           // expert; -1: no more tiles
  int n0, n1;                      // steps of the second product
  int r0, nrows;                   // its part of token_idx
  int first, from, seen;           // mask table: place in the expert's list, tile and count to look from
  uint32_t direct[4];              // rows that are stored instead of added to
  int list[TILE_M];                // tokens, -1: no row
  uint32_t bias[64];               // b1 of the expert as bf16 pairs
};

struct Ctl {
  unsigned long long full[NS_MAX], empty[NS_MAX], full2[NS2_MAX], empty2[NS2_MAX];
  unsigned long long acc1_full[2], ctx_free[2], hid_full[2], acc2_full[6], acc2_empty[6];
  unsigned long long tile_full[TILE_RING], bias_full[TILE_RING], rows_full[TILE_RING], tile_empty[TILE_RING];
  unsigned long long np_full[4], np_empty[4], tot_full;
  uint32_t tmem_base;
  int abort_flag;
  int wait_limit;                  // must follow abort_flag (mbar_wait reads abort_flag[1])
  float npart[TILE_M];             // norm terms that the other drain group saw
  alignas(16) int chunk[TABLE_CHUNKS][MAX_E];   // mask table: tokens per expert of a fifteenth of the tiles
  alignas(16) int tot[MAX_E];                   // and of all
  alignas(16) Tile tile[TILE_RING];
};

// columns of a tile's tensor memory
template <bool GLU>
__device__ __forceinline__ uint32_t tm_tile(uint32_t tmem, uint32_t ctx) {
  return tmem + ctx * (GLU ? 256 : 128);
}

// Accumulator-2 buffers in rotation: one ring for all tiles, gated form one per context.
template <bool GLU>
struct Acc2Ring {
  RingPos r0 = {0, 0}, r1 = {0, 0};
  __device__ __forceinline__ RingPos at(uint32_t ctx) const { return GLU && ctx ? r1 : r0; }
  __device__ __forceinline__ uint32_t slot(uint32_t ctx) const {       // barrier index
    return GLU ? 3 * ctx + at(ctx).s : r0.s;
  }
  __device__ __forceinline__ uint32_t column(uint32_t tmem, uint32_t ctx, int nd) const {
    return GLU ? tmem + 256 * ctx + 64 + 64 * at(ctx).s : tmem + 256 + nd * r0.s;
  }
  __device__ __forceinline__ void next(uint32_t ctx, int nd) {
    if (GLU) {
      if (ctx) r1.next(3); else r0.next(3);
    } else {
      r0.next(nd == 128 ? 2 : 4);
    }
  }
};

// ---------------------------------------------------------------------------
// roles
// ---------------------------------------------------------------------------
__device__ __forceinline__ int chunk_start(const MaskTable& t, int w) { return w * t.ntiles / TABLE_CHUNKS; }

// Warps 0-11 and 16-18: tokens per expert in the warp's fifteenth of the counts table.  A lane has 16 cells of every
// so many rows, summed as pairs of 16-bit halves (a chunk has at most 511 tiles of 128 tokens).  (Called
// without `live` before the table is there: see role_list.)
__device__ __forceinline__ void count_chunk(const Params& p, Ctl* c, int w, int lane, bool live) {
  const MaskTable& t = p.mt;
  const int per = t.EP >> 4, step = 32 / per, g = lane & (per - 1);      // lanes per row, rows at once
  const int t1 = chunk_start(t, w + 1);
  uint32_t acc[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll 1
  for (int t0 = chunk_start(t, w) + lane / per; t0 < t1; t0 += 4 * step) {
    uint4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x[u] = make_uint4(0u, 0u, 0u, 0u);
      if (live && t0 + u * step < t1)
        x[u] = *(reinterpret_cast<const uint4*>(t.counts + (size_t)(t0 + u * step) * t.EP) + g);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t v[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        acc[2 * k] += v[k] & 0x00ff00ffu;
        acc[2 * k + 1] += (v[k] >> 8) & 0x00ff00ffu;
      }
    }
  }
#pragma unroll 1
  for (int o = 16; o >= per; o >>= 1)
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
  if (lane < per)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int4 v = make_int4(acc[2 * k] & 0xffff, acc[2 * k + 1] & 0xffff, acc[2 * k] >> 16,
                               acc[2 * k + 1] >> 16);
      int* tot = &c->tot[16 * g + 4 * k];
      *reinterpret_cast<int4*>(&c->chunk[w][16 * g + 4 * k]) = v;
      if (!live) continue;
      if (v.x) atomicAdd(tot, v.x);
      if (v.y) atomicAdd(tot + 1, v.y);
      if (v.z) atomicAdd(tot + 2, v.z);
      if (v.w) atomicAdd(tot + 3, v.w);
    }
  __syncwarp();
  if (live && lane == 0) mbar_arrive(smem_u32(&c->tot_full));
}

__device__ __forceinline__ int warp_scan(int v, int lane) {      // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// position of the r-th one of m
__device__ __forceinline__ int select_bit(uint32_t m, int r) {
  int at = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const int n = __popc((m >> at) & ((1u << s) - 1u));
    if (r >= n) {
      r -= n;
      at += s;
    }
  }
  return at;
}

// Where token `first` of expert e's list is: the counted chunk says from which tile on to look and how many
// tokens come before it.
__device__ __forceinline__ void find_chunk(const MaskTable& t, const Ctl* c, int e, int first, int lane,
                                           bool live, int& tile, int& seen) {
  const int n = live && lane < TABLE_CHUNKS ? c->chunk[lane][e] : 0, incl = warp_scan(n, lane);
  const uint32_t past = __ballot_sync(0xffffffffu, incl > first);
  const int w = past != 0u ? __ffs(past) - 1 : TABLE_CHUNKS;
  seen = __shfl_sync(0xffffffffu, incl - n, w & 31);
  tile = chunk_start(t, w);
}
// the same to the tile, from the counts table
__device__ __forceinline__ void find_tile(const MaskTable& t, int e, int first, int lane, int& tile, int& seen) {
#pragma unroll 1
  for (; tile < t.ntiles; tile += 32) {
    const int n = tile + lane < t.ntiles ? t.counts[(size_t)(tile + lane) * t.EP + e] : 0;
    const int incl = warp_scan(n, lane);
    const uint32_t past = __ballot_sync(0xffffffffu, seen + incl > first);
    const int w = past != 0u ? __ffs(past) - 1 : 31;
    seen += __shfl_sync(0xffffffffu, past != 0u ? incl - n : incl, w);
    if (past != 0u) {
      tile += w;
      return;
    }
  }
}
// expert e's words of 96 tiles, three per lane
constexpr int LOOK = 3;
__device__ __forceinline__ void load_words(const MaskTable& t, int E, int e, int tile, int lane, bool live,
                                           uint4* x) {
#pragma unroll
  for (int k = 0; k < LOOK; ++k) {
    x[k] = make_uint4(0u, 0u, 0u, 0u);
    if (live && tile + 32 * k + lane < t.ntiles)
      x[k] = t.words[(size_t)(tile + 32 * k + lane) * E + e];
  }
}

// Row `row` of a tile out of the mask table, -1 where it is none (row >= nrows).  A lane has one tile's words
// (x: those of the 96 tiles from t->from on), and a row looks for the lane, the word and the bit that it
// is: no loop over bits, as many steps for one token in a hundred as for one in four.  A table that is
// not the mask's, left by a router that gave up, gives -1.
__device__ __forceinline__ int find_token(const Params& p, const Tile* t, uint4* x, int row, int lane, bool live) {
  const MaskTable& mt = p.mt;
  // (first pass: one row from the table's start on, whatever the list warp is writing meanwhile)
  const int first = live ? t->first : 0, end = live ? first + t->nrows : 1;
  int tile = live ? t->from : 0, seen = live ? t->seen : 0, tok = -1;
#pragma unroll 1
  for (;;) {
#pragma unroll 1
    for (int k = 0; k < LOOK && tile < mt.ntiles && seen < end; ++k, tile += 32) {
      const uint4 y = k == 0 ? x[0] : k == 1 ? x[1] : x[2];
      const int c0 = __popc(y.x), c1 = c0 + __popc(y.y), c2 = c1 + __popc(y.z), n = c2 + __popc(y.w);
      const int incl = warp_scan(n, lane), all = __shfl_sync(0xffffffffu, incl, 31);
      int r = first + row - seen, at = 0;
      const bool mine = r >= 0 && r < all && first + row < end;
      seen += all;
      if (live && !__any_sync(0xffffffffu, mine)) continue;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1)   // lanes whose tokens all come before r
        if (__shfl_sync(0xffffffffu, incl, at + s - 1) <= r) at += s;
      at = min(at, 31);
      const int en = __shfl_sync(0xffffffffu, c0 | c1 << 8 | c2 << 16, at);      // (at most 96 each)
      r -= __shfl_sync(0xffffffffu, incl - n, at);
      const int e0 = en & 255, e1 = en >> 8 & 255, e2 = en >> 16;
      const uint32_t w0 = __shfl_sync(0xffffffffu, y.x, at), w1 = __shfl_sync(0xffffffffu, y.y, at),
                     w2 = __shfl_sync(0xffffffffu, y.z, at), w3 = __shfl_sync(0xffffffffu, y.w, at);
      const int q = (r >= e0) + (r >= e1) + (r >= e2);
      const uint32_t w = q == 0 ? w0 : q == 1 ? w1 : q == 2 ? w2 : w3;
      r -= q == 0 ? 0 : q == 1 ? e0 : q == 2 ? e1 : e2;
      if (mine) tok = (tile + at) * 128 + 32 * q + select_bit(w, r);
    }
    if (!live || tile >= mt.ntiles || seen >= end) return tok;
    load_words(mt, p.E, t->e, tile, lane, live, x);
  }
}

// Warp 19: cuts the lists into tiles and hands the ones of this CTA to the other roles: expert, part of the
// list, then its bias.  The rows themselves are found by the gather warps.  Without lists (the mask table in
// their place) the experts' totals are counted here; a launch of its own for the lists took 4.3 us
// (8.5 for 50432 tokens).
//
// Tiles have S rows at most, S as small as the number of rounds of the grid allows:
// T = sum ceil(n_e / S) <= rows / S + E, so R rounds of G CTAs are enough for S = rows / (R G - E),
// and R is the least with S <= 128.  (524 rows per SM: five tiles of about 109 rows per CTA
// instead of four of 128 and one of 12.)  An expert's tiles are equal.
// Where the previous kernel lets this one start early (router, rule on given scores, scatter: p.warm) a first
// pass runs, while that drains, up to the first tile of a list of one row: instructions that are executed
// for the first time cost some 20 cycles each, and everything waits for the first tile.  So do the first
// passes of count_chunk and of the gather warps.  Queued calls: behind a router 50432 tokens 80.2 -> 76.9 us per
// layer; replayed: behind a scatter 1024 tokens x 128 gated 83.8 -> 79.3, 50432 84.7 -> 81.3, 1920 tokens x 64
// of 2048 x 128 56.7 -> 52.4.  Behind a kernel that is over before, it only comes later: mode 'all' 50.6 -> 52.7, behind
// the routing tensor's own kernel 61.0 -> 62.5 (top-4 of 96, 1024 tokens).  (The other roles' code is warm
// too late: with such passes of theirs 79.7.)
__device__ void role_list(const Params& p, Ctl* c, int lane, bool one_window) {
  volatile int* af = &c->abort_flag;
  const int E = p.E, G = gridDim.x;
  const bool tabled = p.mt.words != nullptr;
#pragma unroll 1
  for (bool live = p.warm ? first_pass() : in_earnest(), last = live;; live = in_earnest(), last = true) {
    if (live) grid_dependency_wait();
    int off[5], n[4], nt[4];             // experts 4 lane .. + 3
    if (tabled) {
      if (live && !mbar_wait_warp(smem_u32(&c->tot_full), 0, af, p.dev_status)) return;
      // (first pass: nothing that the counting warps are adding meanwhile)
      int4 v = make_int4(0, 0, 0, 0);
      if (live) v = *reinterpret_cast<const int4*>(&c->tot[4 * lane]);
      n[0] = 4 * lane < E ? v.x : 0;
      n[1] = 4 * lane + 1 < E ? v.y : 0;
      n[2] = 4 * lane + 2 < E ? v.z : 0;
      n[3] = 4 * lane + 3 < E ? v.w : 0;
      const int sum = n[0] + n[1] + n[2] + n[3];
      off[0] = warp_scan(sum, lane) - sum;
#pragma unroll
      for (int q = 0; q < 4; ++q) off[q + 1] = off[q] + n[q];
    } else {
#pragma unroll
      for (int q = 0; q < 5; ++q) off[q] = live && 4 * lane + q <= E ? p.offsets[4 * lane + q] : 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = 4 * lane + q;
        const bool bad = off[q + 1] < off[q] || off[q] < 0 || off[q + 1] > p.N * (long long)E;
        n[q] = e < E && !bad ? off[q + 1] - off[q] : 0;
        if (e < E && bad) report(p.dev_status, D2D_ERR_INDEX_RANGE);
      }
    }
    if (!live) n[0] = lane == 0 ? 1 : 0;
    int rows = 0, used = 0;
    bool all_n = true;                   // every expert of this lane lists exactly N tokens
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      all_n = all_n && (4 * lane + q >= E || n[q] == p.N);
      rows += n[q];
      used += n[q] > 0 ? 1 : 0;
    }
    rows = __reduce_add_sync(0xffffffffu, rows);
    used = __reduce_add_sync(0xffffffffu, used);
    const float R = ceilf(__fdividef((float)rows * (1.0f / TILE_M) + (float)used, (float)G));
    const int S =                        // (never more rows than a stage has room for)
        max(32, min(p.g.a_slot >> 7,
                    (int)ceilf(__fdividef((float)rows, fmaxf(R * (float)G - (float)used, 1.0f)))));
    const uint32_t inv = 0xffffffffu / (uint32_t)S + 1u;      // ceil(2^32 / S)
    int sum = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {        // ceil(n / S): n < 2^31, so at most one too many
      nt[q] = (int)__umulhi((uint32_t)n[q] + (uint32_t)S - 1u, inv);
      if (nt[q] > 0 && (uint32_t)(nt[q] - 1) * (uint32_t)S >= (uint32_t)n[q]) --nt[q];
      sum += nt[q];
    }
    const int total = __reduce_add_sync(0xffffffffu, sum);
    // windows: one per round of the grid, or a single one (expert by expert) where each window
    // would stream all the weights again; with every expert on every token they pay all the same
    const int rounds = one_window && !__all_sync(0xffffffffu, all_n) ? 1 : max(1, (int)R);
    // fewer than half as many tiles as CTAs: split the output columns (the first product is
    // repeated, the second product, W2 and the output are shared out)
    int parts = 1;
    if (total > 0 && 2 * total <= G && p.norm_layer == 0) parts = min(G / total, p.g.nc);
    const float inv_rounds = __fdividef(1.0f, (float)rounds);

    // the current window's tiles of my experts: lo .. hi - 1
    int lo[4], hi[4], w = rounds, start = 0, count = 0, incl = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) lo[q] = nt[q];
    RingPos r = {0, 0};
#pragma unroll 1
    for (int u = live ? blockIdx.x : 0;; u += G, r.next(TILE_RING)) {
      const int tile = parts == 1 ? u : u / parts, part = parts == 1 ? 0 : u - tile * parts;
      Tile* t = &c->tile[r.s];
      if (tile >= total) {
        if (!mbar_wait_warp(smem_u32(&c->tile_empty[r.s]), r.ph ^ 1, af, p.dev_status)) return;
        if (lane == 0) t->e = -1;
        __syncwarp();
        mbar_arrive(smem_u32(&c->tile_full[r.s]));
        break;
      }
      while (tile >= start + count) {
        start += count;
        --w;
        int mine = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          hi[q] = lo[q];
          lo[q] = w == 0 ? 0 : min(hi[q], (int)((float)nt[q] * ((float)w * inv_rounds)));
          mine += hi[q] - lo[q];
        }
        incl = warp_scan(mine, lane);
        count = __shfl_sync(0xffffffffu, incl, 31);
      }
      const int owner = __ffs(__ballot_sync(0xffffffffu, incl > tile - start)) - 1;
      int e = 0, first = 0, r0 = 0, nrows = 0;
      if (lane == owner) {
        int k = tile - start - (incl - (hi[0] + hi[1] + hi[2] + hi[3] - lo[0] - lo[1] - lo[2] - lo[3]));
        int len = 0, tiles = 1;
        bool found = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int m = hi[q] - lo[q];
          if (!found && k < m) {
            found = true;
            e = 4 * lane + q;
            first = lo[q] + k;
            len = n[q];
            tiles = nt[q];
            r0 = off[q];
          }
          if (!found) k -= m;
        }
        const int size = (len + tiles - 1) / tiles;
        first *= size;
        r0 += first;
        nrows = min(size, len - first);  // (may be negative where the last tiles are empty)
      }
      e = __shfl_sync(0xffffffffu, e, owner);
      first = __shfl_sync(0xffffffffu, first, owner);
      int from = 0, seen = 0;
      if (tabled) {
        find_chunk(p.mt, c, e, first, lane, live, from, seen);
        if (u != (int)blockIdx.x && live) find_tile(p.mt, e, first, lane, from, seen);   // (not urgent)
      }
      if (live && !mbar_wait_warp(smem_u32(&c->tile_empty[r.s]), r.ph ^ 1, af, p.dev_status)) return;
      if (lane == owner) {
        t->e = e;
        t->n0 = part * p.g.nc / parts;
        t->n1 = (part + 1) * p.g.nc / parts;
        t->r0 = r0;
        t->nrows = nrows;
        t->first = first;
        t->from = from;
        t->seen = seen;
      }
      __syncwarp();
      if (live) mbar_arrive(smem_u32(&c->tile_full[r.s]));
      const float4 b1 = live && 4 * lane < p.H         // (no global read before the wait)
                            ? __ldg(reinterpret_cast<const float4*>(
                                  p.packed + (long long)e * p.g.stride + p.g.bias_off) + lane)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
      t->bias[2 * lane] = pack_bf16x2(b1.x, b1.y);
      t->bias[2 * lane + 1] = pack_bf16x2(b1.z, b1.w);
      if (!live) break;
      mbar_arrive(smem_u32(&c->bias_full[r.s]));
    }
    if (tabled && live && blockIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (4 * lane + q < E) p.offsets[4 * lane + q] = off[q];
      if (lane == 31) p.offsets[E] = off[4];
      if (lane == 31 && off[4] > p.N * (long long)E) report(p.dev_status, D2D_ERR_INDEX_RANGE);
    }
    if (last) return;
  }
}

// Warps 12-15: warp w has rows 32 w .. + 31 of a tile.  It finds their tokens (the list's, or out of the
// mask table, whose part of the list it then writes), says which of them are stored, and copies their
// rows of x by 16-byte cp.async (4 rows x 128 bytes per warp instruction, software swizzle; a TMA
// gather spends a request per 128-byte row and was 1.6 times slower).  Rows past
// the list's end repeat the 32-row group's first one, a group without rows loads nothing: what
// their slots hold reaches only accumulator rows nobody reads.
// (Beside the traffic of the kernel a load takes some thousand cycles: the mask words of a tile travel
// while its rows are copied, and so do the next tile's table words where that tile is known by then.  The
// selection itself stands between two tiles' copies: a gated expert with two rows per 128-token tile makes it
// search 64 of those for one of its own.)
__device__ void role_gather(const Params& p, Ctl* c, uint32_t ring, int w, int lane) {
  volatile int* af = &c->abort_flag;
  const int j = lane & 7, row = w * 32 + lane;
  const int nw = (p.E + 31) >> 5;
  const bool tabled = p.mt.words != nullptr;
  uint32_t dstoff[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int rr = w * 32 + i * 4 + (lane >> 3);
    dstoff[i] = (rr >> 3) * 1024 + (rr & 7) * 128 + ((j ^ (rr & 7)) << 4);
  }
  RingPos r = {0, 0}, q = {0, 0};
  uint4 x[LOOK];
  x[0] = x[1] = x[2] = make_uint4(0u, 0u, 0u, 0u);
  bool live = p.warm ? first_pass() : in_earnest();
  bool ahead = p.warm;                   // this tile's first loads are on their way (none in a first pass)
  if (live) grid_dependency_wait();
#pragma unroll 1
  for (;;) {
    Tile* t = &c->tile[q.s];
    if (live) {
      if (!mbar_wait_warp(smem_u32(&c->tile_full[q.s]), q.ph, af, p.dev_status)) return;
      if (t->e < 0) return;
    }
    const int e = live ? t->e : 0, nrows = live ? t->nrows : 0, at = live ? t->r0 + row : 0;
    if (!ahead) {
      if (tabled) load_words(p.mt, p.E, e, t->from, lane, live, x);
      else x[0].x = row < nrows ? p.token_idx[at] : 0;
    }
    int tok = (int)x[0].x;
    if (tabled) tok = find_token(p, t, x, row, lane, live);
    if (row < nrows && (tok < 0 || tok >= p.N)) {
      report(p.dev_status, D2D_ERR_INDEX_RANGE);
      tok = -1;
    }
    if (row >= nrows) tok = -1;
    if (live) t->list[row] = tok;
    // (in bounds whatever the table says)
    if (tabled && tok >= 0 && t->n0 == 0 && (uint32_t)at < (uint32_t)(p.N * p.E)) p.token_idx[at] = tok;
    uint32_t mask[4] = {0u, 0u, 0u, 0u};
    if (p.mask_bits && tok >= 0)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < nw) mask[k] = p.mask_bits[(long long)tok * nw + k];
    const int v0 = __shfl_sync(0xffffffffu, tok, 0);
    const bf16* src[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int v = __shfl_sync(0xffffffffu, tok, i * 4 + (lane >> 3));
      src[i] = p.x + (size_t)max(v < 0 ? v0 : v, 0) * p.d + j * 8;
    }
    if (!live) {                         // the previous kernel's results from here on
      grid_dependency_wait();
      live = in_earnest();
      ahead = false;
      continue;
    }
    const RingPos q0 = q;
    q.next(TILE_RING);
    ahead = false;
    if (__all_sync(0xffffffffu, mbar_test_wait(smem_u32(&c->tile_full[q.s]), q.ph))) {
      const Tile* t1 = &c->tile[q.s];
      if (t1->e >= 0) {
        ahead = true;
        if (tabled) load_words(p.mt, p.E, t1->e, t1->from, lane, true, x);
        else x[0].x = row < t1->nrows ? p.token_idx[t1->r0 + row] : 0;
      }
    }
    const bool rows = v0 >= 0;           // warp-uniform
#pragma unroll 1
    for (int kc = 0; kc < p.g.kc1; ++kc) {
      if (!mbar_wait_warp(smem_u32(&c->empty[r.s]), r.ph ^ 1, af, p.dev_status)) return;
      if (rows) {
        const uint32_t base = ring + r.s * p.g.stage;
#pragma unroll
        for (int i = 0; i < 8; ++i) cp_async16(base + dstoff[i], src[i] + kc * 64);
      }
      cp_async_arrive_noinc(smem_u32(&c->full[r.s]));
      r.next(p.g.ns);
    }
    const uint32_t d = __ballot_sync(
        0xffffffffu, __popc(mask[0]) + __popc(mask[1]) + __popc(mask[2]) + __popc(mask[3]) == 1);
    if (lane == 0) c->tile[q0.s].direct[w] = d;
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(smem_u32(&c->rows_full[q0.s]));
      mbar_arrive(smem_u32(&c->tile_empty[q0.s]));
    }
  }
}

// The three roles below each run in ONE thread of their warp for the whole launch: their loops are
// chains of dependent instructions, votes and re-convergence would only lengthen the chain.

// Weights of both rings.  The two streams (W1 slices, W2 steps) advance independently: whichever
// ring has a free stage gets its next piece.
__device__ void role_weights(const Params& p, Ctl* c, uint32_t ring, uint32_t ring2) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  bool withheld = (p.withhold & 1) != 0 && blockIdx.x == 0;
  RingPos r1 = {0, 0}, r2 = {0, 0}, q1 = {0, 0}, q2 = {0, 0};
  int j1 = 0, j2 = 0;                    // pieces left of the current tile; -1: no more tiles
  const uint8_t *s1 = nullptr, *s2 = nullptr;
  uint32_t idle = 0;
  while (j1 >= 0 || j2 >= 0) {
    bool progress = false;
    if (j1 == 0 && mbar_test_wait(smem_u32(&c->tile_full[q1.s]), q1.ph)) {
      const int e = c->tile[q1.s].e;
      j1 = e < 0 ? -1 : g.kc1;
      s1 = p.packed + (long long)e * g.stride;
      mbar_arrive(smem_u32(&c->tile_empty[q1.s]));
      q1.next(TILE_RING);
      progress = true;
    }
    if (j1 > 0 && mbar_test_wait(smem_u32(&c->empty[r1.s]), r1.ph ^ 1)) {
      const uint32_t bar = smem_u32(&c->full[r1.s]);
      mbar_arrive_expect_tx(bar, g.w1_stage);
      if (withheld) withheld = false;    // test hook: this stage never fills, its wait runs out
      else bulk_g2s(ring + r1.s * g.stage + g.a_slot, s1, g.w1_stage, bar);
      s1 += g.w1_stage;
      r1.next(g.ns);
      --j1;
      progress = true;
    }
    if (j2 == 0 && mbar_test_wait(smem_u32(&c->tile_full[q2.s]), q2.ph)) {
      const Tile* t = &c->tile[q2.s];
      const int e = t->e;
      j2 = e < 0 ? -1 : (t->n1 - t->n0) * g.kc2;
      s2 = p.packed + (long long)e * g.stride + g.w1_bytes + (long long)t->n0 * g.kc2 * g.w2_piece;
      mbar_arrive(smem_u32(&c->tile_empty[q2.s]));
      q2.next(TILE_RING);
      progress = true;
    }
    if (j2 > 0 && mbar_test_wait(smem_u32(&c->empty2[r2.s]), r2.ph ^ 1)) {
      const uint32_t bar = smem_u32(&c->full2[r2.s]);
      mbar_arrive_expect_tx(bar, g.w2_piece);
      bulk_g2s(ring2 + r2.s * g.w2_piece, s2, g.w2_piece, bar);
      s2 += g.w2_piece;
      r2.next(g.ns2);
      --j2;
      progress = true;
    }
    if (progress) {
      idle = 0;
    } else {
      if (++idle > 64) __nanosleep(idle > 4096 ? 256 : 32);
      if ((idle & 63) == 0 && *af != 0) return;
      if (idle >= p.wait_limit) {
        *af = 1;
        report(p.dev_status, D2D_ERR_TIMEOUT);
        return;
      }
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
  RingPos r = {0, 0}, q = {0, 0};
  uint32_t ctx = 0, ph = 0;
  for (;; q.next(TILE_RING)) {
    if (!mbar_wait_fast(smem_u32(&c->tile_full[q.s]), q.ph, af, p.dev_status)) return;
    if (c->tile[q.s].e < 0) return;
    mbar_arrive(smem_u32(&c->tile_empty[q.s]));
    const uint32_t acc = tm_tile<GLU>(tmem, ctx);
    if (!mbar_wait_fast(smem_u32(&c->ctx_free[ctx]), ph ^ 1, af, p.dev_status)) return;
    tc_fence_after();
    for (int kc = 0; kc < g.kc1; ++kc) {
      if (!mbar_wait_fast(smem_u32(&c->full[r.s]), r.ph, af, p.dev_status)) return;
      fence_proxy_async();               // (the token rows are cp.async writes)
      tc_fence_after();
      const uint32_t alo = lo0 + r.s * ((uint32_t)g.stage >> 4), blo = alo + ((uint32_t)g.a_slot >> 4);
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

// second product: one step after another, each into the next accumulator-2 buffer
template <bool GLU>
__device__ void role_mma2(const Params& p, Ctl* c, uint32_t ring2, uint32_t tmem) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const uint32_t idesc = instr_desc(TILE_M, g.nd);
  const uint64_t d0 = smem_desc(ring2);
  const uint64_t hi = (d0 >> 32) << 32;
  const uint32_t lo0 = (uint32_t)d0;
  RingPos r = {0, 0}, q = {0, 0};
  Acc2Ring<GLU> ar;
  uint32_t ctx = 0, ph = 0;
  for (;; q.next(TILE_RING)) {
    if (!mbar_wait_fast(smem_u32(&c->tile_full[q.s]), q.ph, af, p.dev_status)) return;
    if (c->tile[q.s].e < 0) return;
    const int n0 = c->tile[q.s].n0, n1 = c->tile[q.s].n1;
    mbar_arrive(smem_u32(&c->tile_empty[q.s]));
    const uint32_t hid = tm_tile<GLU>(tmem, ctx);
    if (!mbar_wait_fast(smem_u32(&c->hid_full[ctx]), ph, af, p.dev_status)) return;
    for (int n = n0; n < n1; ++n) {
      const uint32_t b = ar.slot(ctx), acc = ar.column(tmem, ctx, g.nd);
      if (!mbar_wait_fast(smem_u32(&c->acc2_empty[b]), ar.at(ctx).ph ^ 1, af, p.dev_status)) return;
      for (int k2 = 0; k2 < g.kc2; ++k2) {
        if (!mbar_wait_fast(smem_u32(&c->full2[r.s]), r.ph, af, p.dev_status)) return;
        tc_fence_after();
        const uint32_t blo = lo0 + r.s * ((uint32_t)g.w2_piece >> 4), ha = hid + 32 * k2;
        const int ks = (p.H >> 4) - 4 * k2;
        umma_bf16_ta(acc, ha, hi | blo, idesc, k2);
        if (ks > 1) umma_bf16_ta(acc, ha + 8, hi | (blo + 2), idesc, 1);
        if (ks > 2) umma_bf16_ta(acc, ha + 16, hi | (blo + 4), idesc, 1);
        if (ks > 3) umma_bf16_ta(acc, ha + 24, hi | (blo + 6), idesc, 1);
        umma_commit(smem_u32(&c->empty2[r.s]));
        r.next(g.ns2);
      }
      umma_commit(smem_u32(&c->acc2_full[b]));
      ar.next(ctx, g.nd);
    }
    // the hidden tile has been read (gated form: the drain warps free the tile's columns)
    if (!GLU) umma_commit(smem_u32(&c->ctx_free[ctx]));
    ph ^= ctx;
    ctx ^= 1;
  }
}

// Warps 0-3, thread = tile row = TMEM lane: accumulator 1 -> bias, activation (x
// up-projection) -> bf16 hidden tile over the columns already read.
template <int ACT, bool GLU, bool NORM>
__device__ void role_ep1(const Params& p, Ctl* c, uint32_t tmem, int et) {
  volatile int* af = &c->abort_flag;
  const uint32_t lane_base = (uint32_t)(et & ~31) << 16;
  const int nord = p.norm_ord;
  RingPos q = {0, 0};
  uint32_t ctx = 0, ph = 0;
  for (;; q.next(TILE_RING)) {
    if (!mbar_wait_warp(smem_u32(&c->tile_full[q.s]), q.ph, af, p.dev_status)) return;
    const Tile* t = &c->tile[q.s];
    const int e = t->e;
    if (e < 0) return;
    if (!mbar_wait_warp(smem_u32(&c->bias_full[q.s]), q.ph, af, p.dev_status)) return;
    const uint32_t* bp = t->bias;
    // labels by-product (intermediate layer): this thread's row
    float nacc = 0.f;
    if (NORM && !mbar_wait_warp(smem_u32(&c->rows_full[q.s]), q.ph, af, p.dev_status)) return;
    const int ntok = NORM ? t->list[et] : -1;
    if (!mbar_wait_warp(smem_u32(&c->acc1_full[ctx]), ph, af, p.dev_status)) return;
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
    __syncwarp();
    if ((et & 31) == 0) mbar_arrive(smem_u32(&c->tile_empty[q.s]));
    mbar_arrive(smem_u32(&c->hid_full[ctx]));
    if (NORM && ntok != -1)
      p.norms[(long long)e * p.N + ntok] =
          __float2bfloat16_rn(nord == 1 ? nacc : sqrtf(nacc));
    ph ^= ctx;
    ctx ^= 1;
  }
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

// 16 rows x 64 columns of fragments as bf16 pairs: w[row rl or rl + 8][block of 32 columns][4 pairs]
template <bool NORM>
__device__ __forceinline__ void frag_pairs(const uint32_t* v, uint32_t (&w)[2][2][4], float* nacc, int nord) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t* f = v + 16 * k + 4 * h + 2 * i;
        w[i][k][h] = pack_bf16x2(__uint_as_float(f[0]), __uint_as_float(f[1]));
        if (NORM) {
          const float lo = __uint_as_float(w[i][k][h] << 16),
                      hi = __uint_as_float(w[i][k][h] & 0xffff0000u);
          nacc[i] += nord == 1 ? fabsf(lo) + fabsf(hi) : fmaf(lo, lo, hi * hi);
        }
      }
}

// The lanes of an even row give its second block for the first one of the next row: eight lanes have a
// row's 128 bytes (even rows' lanes the first block's).  All exchanges come before the first write.
template <bool DIRECT>
__device__ __forceinline__ void put_rows(uint32_t (&w)[2][2][4], const int* rt, uint8_t* o,
                                         uint32_t row_bytes, uint4 bz, int odd) {
  uint32_t got[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int h = 0; h < 4; ++h)
      got[i][h] = __shfl_xor_sync(0xffffffffu, odd ? w[i][0][h] : w[i][1][h], 4);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int k = 0; k < 2; ++k) {        // k = 0: the even row
      uint32_t x[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) x[h] = odd == k ? w[i][k][h] : got[i][h];
      const uint4 val = make_uint4(x[0], x[1], x[2], x[3]);
      const int r = rt[2 * i + k];
      uint8_t* const row = o + (uint64_t)((uint32_t)r & 0x7fffffffu) * row_bytes;
      if (DIRECT) put_row(row, r, val, add_bf16x8(bz, val));
      else add_row(row, r, val);
    }
}

// Warps 4-11: warp q4 of group j has rows 32 q4 .. +31 and 64 columns: with 128-column steps the two
// groups share each one, with 64-column steps they take every other one.
// The loads take the accumulator as fragments of 8 rows x 8 columns (four lanes a row, two columns
// each); W2's columns are packed in the order (out_column) that gives a lane eight neighbouring
// ones of each 32-column block, and the lanes of two rows trade a block, so that eight of them have
// 128 bytes of one row: whole lines leave an SM at 25 bytes per clock where they are added, half lines at
// 20 (stored: 32 and 29; 148 CTAs, rows of 1536 bytes).  A transposition through shared memory took 1.7 times as
// long, alone and with nothing written.
// A tile of the two-layer form is bound by this role, and close behind it by the products (1450 cycles): a
// 128-column step takes 1850 cycles, 1700 with no rows and weights coming in, 1530 with nothing written, whether
// those come in or not (vit_256; BERT's 1850, 1750, 1530).  Of the 1530 a warp spends 1080 on its own instructions,
// 780 of them the exchanges and selections of put_rows, and 450 on the loop and the wait for the next
// accumulator; writes add 280 to put_rows.  Rows leave at 18 bytes a clock and SM: 26, mixed, is the way's rate.
// A register that spills here waits behind the writes.
// DIRECT: rows of tokens with one expert are stored, see DirectRows
template <bool GLU, bool NORM, bool DIRECT>
__device__ void role_drain(const Params& p, Ctl* c, uint32_t tmem, int j, int q4, int lane) {
  volatile int* af = &c->abort_flag;
  const Geo& g = p.g;
  const int rl = lane >> 2, ql = lane & 3, odd = rl & 1;
  const int nord = p.norm_ord;
  const bool wide = g.nd == 128;
  const int col0 = wide ? 64 * j : 0;                // my columns of a step
  const uint32_t row_bytes = 2 * (uint32_t)p.d;
  const uint32_t src0 = ((uint32_t)(q4 * 32) << 16) + col0;
  Acc2Ring<GLU> ar;
  RingPos q = {0, 0};
  uint32_t ctx = 0;
  int turn = wide ? j : 0;                           // group whose step is next
  uint32_t nph = 0;
  for (;; q.next(TILE_RING)) {
    if (!mbar_wait_warp(smem_u32(&c->tile_full[q.s]), q.ph, af, p.dev_status)) return;
    const Tile* t = &c->tile[q.s];
    const int e = t->e, n0 = t->n0, n1 = t->n1;
    if (e < 0) return;
    if (!mbar_wait_warp(smem_u32(&c->rows_full[q.s]), q.ph, af, p.dev_status)) return;
    const uint32_t direct = DIRECT ? t->direct[q4] : 0u;
    int rt[8];                           // rows 8 (i / 2) + (rl & ~1) + i % 2; sign bit: stored
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 8 * (i >> 1) + (rl & 6) + (i & 1);
      rt[i] = (int)((uint32_t)t->list[q4 * 32 + r] | (((direct >> r) & 1u) << 31));
    }
    const int mine = NORM ? t->list[q4 * 32 + 8 * ql + rl] : -1;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&c->tile_empty[q.s]));
    float nacc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int n = n0; n < n1; ++n) {
      const bool skip = turn != j;
      if (!wide) turn ^= 1;
      if (skip) {
        ar.next(ctx, g.nd);
        continue;
      }
      const int col = n * g.nd + col0 + 32 * odd + 8 * ql;
      uint8_t* const o = reinterpret_cast<uint8_t*>(p.out + col);
      uint4 bz = make_uint4(0u, 0u, 0u, 0u);
      if (DIRECT && p.last_bias)
        bz = __ldg(reinterpret_cast<const uint4*>(p.last_bias + col));
      const uint32_t b = ar.slot(ctx);
      if (!mbar_wait_warp(smem_u32(&c->acc2_full[b]), ar.at(ctx).ph, af, p.dev_status)) return;
      tc_fence_after();
      const uint32_t acc = ar.column(tmem, ctx, g.nd) + src0;
      ar.next(ctx, g.nd);
      // 16 rows at a time (64 values more would spill): the second half's load runs while the first
      // half is written out
      uint32_t v[32], w[2][2][4];
      tmem_ld_frag64(acc, v);
      tmem_wait_ld32(v);
      frag_pairs<NORM>(v, w, nacc, nord);
      tmem_ld_frag64(acc + (16u << 16), v);
      put_rows<DIRECT>(w, rt, o, row_bytes, bz, odd);
      tmem_wait_ld32(v);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c->acc2_empty[b]));
      frag_pairs<NORM>(v, w, nacc + 2, nord);
      put_rows<DIRECT>(w, rt + 4, o, row_bytes, bz, odd);
    }
    // every read of this tile's tensor memory by this warp is done
    if (GLU) {
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c->ctx_free[ctx]));
    }
    if (NORM) {
      // a row's four lanes, then the other group, which saw the other columns: lane = row 8 ql + rl
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        nacc[i] += __shfl_xor_sync(0xffffffffu, nacc[i], 1);
        nacc[i] += __shfl_xor_sync(0xffffffffu, nacc[i], 2);
        if (ql == i) sum = nacc[i];
      }
      const uint32_t nf = smem_u32(&c->np_full[q4]), ne = smem_u32(&c->np_empty[q4]);
      if (j == 1) {
        if (!mbar_wait_warp(ne, nph ^ 1, af, p.dev_status)) return;
        c->npart[q4 * 32 + lane] = sum;
        mbar_arrive(nf);
      } else {
        if (!mbar_wait_warp(nf, nph, af, p.dev_status)) return;
        sum += c->npart[q4 * 32 + lane];
        mbar_arrive(ne);
        if (mine != -1)
          p.norms[(long long)e * p.N + mine] =
              __float2bfloat16_rn(nord == 1 ? sum : sqrtf(sum));
      }
      nph ^= 1;
    }
    ctx ^= 1;
  }
}

// ---------------------------------------------------------------------------
// kernel
// ---------------------------------------------------------------------------
// NORM: 0 none, D2D_NORM_OF_INTERMEDIATE, D2D_NORM_OF_OUTPUT
template <bool GLU, int NORM>
__global__ void __launch_bounds__(NTHREADS, 1) experts_tiles_kernel(const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  const uint32_t ring2 = ring + p.g.ns * p.g.stage;
  Ctl* c = reinterpret_cast<Ctl*>(smem_raw + (ring2 - raw) + p.g.ns2 * p.g.w2_piece);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Programmatic dependent launch: see router_tiles_kernel.
  grid_launch_dependents();

  if (tid < MAX_E) c->tot[tid] = 0;
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
    }
    for (int i = 0; i < TILE_RING; ++i) {
      mbar_init(smem_u32(&c->tile_full[i]), 32);
      mbar_init(smem_u32(&c->bias_full[i]), 32);
      mbar_init(smem_u32(&c->rows_full[i]), 4);
      mbar_init(smem_u32(&c->tile_empty[i]), TILE_READERS);
      mbar_init(smem_u32(&c->np_full[i]), 32);
      mbar_init(smem_u32(&c->np_empty[i]), 32);
    }
    static_assert(TILE_RING == 4, "np barriers: one per row quarter");
    mbar_init(smem_u32(&c->tot_full), TABLE_CHUNKS);
    for (int i = 0; i < 6; ++i) {
      mbar_init(smem_u32(&c->acc2_full[i]), 1);
      mbar_init(smem_u32(&c->acc2_empty[i]), p.g.nd >> 4);    // four warps per 64 columns
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
  // (the list and gather warps wait for the previous kernel in their roles)
  if (warp < WARP_GATHER0 || (warp >= WARP_MMA1 && warp <= WARP_W)) {
    const int w = warp < WARP_GATHER0 ? warp : warp - (WARP_MMA1 - WARP_GATHER0);
    if (p.mt.words) {
      bool live = first_pass();
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass, live = in_earnest()) {
        if (live) grid_dependency_wait();
        count_chunk(p, c, w, lane, live);
      }
    } else {
      grid_dependency_wait();
    }
  }

  if (warp < WARP_DRAIN0) {
    role_ep1_act<GLU, NORM == D2D_NORM_OF_INTERMEDIATE>(p, c, tmem, tid);
  } else if (warp < WARP_GATHER0) {
    const int w = warp - WARP_DRAIN0;
    if (NORM != D2D_NORM_OF_OUTPUT && p.mask_bits)
      role_drain<GLU, false, true>(p, c, tmem, w >> 2, w & 3, lane);
    else
      role_drain<GLU, NORM == D2D_NORM_OF_OUTPUT, false>(p, c, tmem, w >> 2, w & 3, lane);
  } else if (warp < WARP_MMA1) {
    role_gather(p, c, ring, warp - WARP_GATHER0, lane);
    cp_async_wait_all();
  } else if (warp == WARP_MMA1) {
    if (elect_one()) role_mma1<GLU>(p, c, ring, tmem);
    __syncwarp();
  } else if (warp == WARP_MMA2) {
    if (elect_one()) role_mma2<GLU>(p, c, ring2, tmem);
    __syncwarp();
  } else if (warp == WARP_W) {
    if (elect_one()) role_weights(p, c, ring, ring2);
    __syncwarp();
  } else {
    role_list(p, c, lane, (long long)p.E * p.g.stride > L2_WEIGHTS);
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
// of W1 (gated form: H gate rows, then H up rows), the nd-column x 64-deep pieces of W2, b1 in fp32.
__global__ void prepack_experts_kernel(const bf16* __restrict__ w1, const bf16* __restrict__ b1,
                                       const bf16* __restrict__ w_up, const bf16* __restrict__ w2,
                                       uint8_t* __restrict__ packed, Geo g, int d, int E, int H) {
  const int e = blockIdx.y;
  uint8_t* pe = packed + (long long)e * g.stride;
  const int rows1 = g.w1_stage >> 7;
  const long long n1 = (long long)g.kc1 * rows1 * 64;
  const long long n2 = (long long)g.nc * g.kc2 * g.nd * 64;
  const bf16 zero = __float2bfloat16_rn(0.f);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n1 + n2 + H;
       i += (long long)gridDim.x * blockDim.x) {
    if (i < n1) {
      // consecutive threads: consecutive k, the contiguous direction of the image; the strided reads
      // hit the cache.  (Along W1's own direction a warp's 2-byte stores go to 32 rows of the image:
      // 24 experts 768 x 128 53 us instead of 37, 128 gated experts 2048 x 128 825 instead of 504.)
      const int k = (int)(i % 64);
      const int n = (int)((i / 64) % rows1);
      const int kc = (int)(i / (64LL * rows1));
      const bf16* src = n < H ? w1 : w_up;
      const bf16 v = src[((long long)e * d + kc * 64 + k) * H + (n < H ? n : n - H)];
      *reinterpret_cast<bf16*>(pe + (long long)kc * g.w1_stage + swz(n, k)) = v;
    } else if (i < n1 + n2) {
      const long long q = i - n1;
      const int k = (int)(q % 64);
      const int n = (int)((q / 64) % g.nd);
      const int k2 = (int)((q / (64LL * g.nd)) % g.kc2);
      const int nci = (int)(q / (64LL * g.nd * g.kc2));
      const int kk = k2 * 64 + k;
      const bf16 v = kk < H ? w2[((long long)e * H + kk) * d + nci * g.nd + out_column(n)] : zero;
      *reinterpret_cast<bf16*>(pe + g.w1_bytes + (long long)(nci * g.kc2 + k2) * g.w2_piece +
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
  return (size_t)experts_geo(d, H, glu, TILE_M).stride * (size_t)E;
}

int launch_prepack_experts(const void* w1, const void* b1, const void* w_up, const void* w2,
                           void* packed, int d, int E, int H, cudaStream_t s) {
  const Geo g = experts_geo(d, H, w_up != nullptr, TILE_M);
  dim3 grid(64, E);
  prepack_experts_kernel<<<grid, 256, 0, s>>>((const bf16*)w1, (const bf16*)b1, (const bf16*)w_up,
                                              (const bf16*)w2, (uint8_t*)packed, g, d, E, H);
  return cudaGetLastError() == cudaSuccess ? D2D_OK : D2D_ERR_LAUNCH;
}

int launch_experts_umma(const void* x, int32_t* token_idx, int32_t* offsets,
                        const void* packed, void* out, int64_t N, int d, int E, int H, bool glu,
                        int act, int* dev_status, cudaStream_t s, NormCapture nc, DirectRows dr,
                        const MaskTable* mt) {
  if (!nc.norms && !mt && experts_short_supported(N, d, E, H, glu, dr.kept))
    return launch_experts_short(x, token_idx, offsets, packed, out, N, d, E, H, glu, act, dev_status,
                                s, dr);
  Params p = {};
  p.x = (const bf16*)x;
  p.N = N;
  p.d = d;
  p.E = E;
  p.H = H;
  p.act = act;
  p.packed = (const uint8_t*)packed;
  p.g = experts_geo(d, H, glu, N);
  p.token_idx = token_idx;
  p.offsets = offsets;
  if (mt) p.mt = *mt;
  p.warm = dr.warm;
  p.out = (bf16*)out;
  p.mask_bits = dr.mask_bits;
  p.last_bias = (const bf16*)dr.last_bias;
  p.dev_status = dev_status;
  p.norms = (bf16*)nc.norms;
  p.norm_layer = nc.norms ? nc.layer : 0;
  p.norm_ord = nc.ord;
  umma_debug_read(&p.wait_limit, &p.withhold);
  const size_t smem =
      1024 + (size_t)p.g.ns * p.g.stage + (size_t)p.g.ns2 * p.g.w2_piece + sizeof(Ctl) + 64;
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
