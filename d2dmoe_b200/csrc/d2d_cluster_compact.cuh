// Compaction inside the kernel that applies the routing rule, for calls of at most eight 128-token
// tiles (1024 tokens): the tiles are one cluster, whose CTAs exchange their per-expert counts through
// distributed shared memory and write their own part of the lists.  It takes the place of the
// scatter launch, which such a call spends more time on (about 4 us with the kernel boundary) than
// on its router.
#pragma once
#include <cooperative_groups.h>

#include "d2d_common.cuh"

namespace d2d {

constexpr int CLUSTER_TILES = 8;

// rows[q * stride + e]: which of the tokens 32 q .. 32 q + 31 of this CTA's tile keep expert e;
// scratch: 3 * 256 ints; first: the tile's first token.  All threads of all CTAs of the cluster call
// it, E <= 256; ends with a cluster barrier.
template <int NTHREADS>
__device__ __forceinline__ void cluster_compact(const uint32_t* rows, int stride, int* scratch, int E,
                                                int64_t first, int32_t* token_idx,
                                                int32_t* offsets) {
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31;
  const int rank = (int)cluster.block_rank(), n = (int)cluster.num_blocks();
  int *mine = scratch, *off = scratch + 256, *pre = scratch + 512;
  for (int e = tid; e < E; e += NTHREADS)
    mine[e] = __popc(rows[e]) + __popc(rows[stride + e]) + __popc(rows[2 * stride + e]) +
              __popc(rows[3 * stride + e]);
  cluster.sync();
  for (int e = tid; e < E; e += NTHREADS) {
    int v[CLUSTER_TILES], total = 0, before = 0;
#pragma unroll
    for (int r = 0; r < CLUSTER_TILES; ++r) v[r] = r < n ? cluster.map_shared_rank(mine, r)[e] : 0;
#pragma unroll
    for (int r = 0; r < CLUSTER_TILES; ++r) {
      total += v[r];
      before += r < rank ? v[r] : 0;
    }
    off[e] = total;
    pre[e] = before;
  }
  __syncthreads();
  if (tid < 32) {                      // exclusive scan of the totals, eight experts per lane
    int v[8], s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k] = 8 * lane + k < E ? off[8 * lane + k] : 0;
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
    for (int k = 0; k < 8; ++k) {
      const int e = 8 * lane + k;
      if (e < E) {
        off[e] = run;
        if (rank == 0) offsets[e] = run;
      }
      run += v[k];
    }
    if (rank == 0 && lane == 31) offsets[E] = incl;
  }
  __syncthreads();
  for (int i = tid; i < 4 * E; i += NTHREADS) {
    const int q = i / E, e = i - q * E;
    uint32_t m = rows[q * stride + e];
    if (m == 0u) continue;
    int at = off[e] + pre[e];
    for (int k = 0; k < q; ++k) at += __popc(rows[k * stride + e]);
    for (; m != 0u; m &= m - 1) token_idx[at++] = (int32_t)(first + 32 * q + __ffs(m) - 1);
  }
  cluster.sync();                      // the others may still read `mine`
}

}  // namespace d2d
