// Host-side interface of the tcgen05 (bf16) kernels, used by d2d_abi.cu.
#pragma once
#include "d2d_common.cuh"

namespace d2d {

bool umma_experts_supported(int d, int E, int H, bool glu, int dtype);
size_t umma_experts_packed_bytes(int d, int E, int H, bool glu);
int launch_prepack_experts(const void* w1, const void* b1, const void* w_up, const void* w2,
                           void* packed, int d, int E, int H, cudaStream_t s);
// Rows the expert kernel may store instead of adding to: tokens whose mask has exactly one bit
// get  last_bias + expert output, the others are added to rows that are initialised.
struct DirectRows {
  const uint32_t* mask_bits = nullptr;   // null: every row is added to
  const void* last_bias = nullptr;
  int kept = 0;                          // experts a token keeps, where the rule fixes it
  bool warm = false;                     // the previous kernel lets this one start early: see role_list
};
// mt: there are no lists yet; the kernel makes them from the table and writes them as well
int launch_experts_umma(const void* x, int32_t* token_idx, int32_t* offsets,
                        const void* packed, void* out, int64_t N, int d, int E, int H, bool glu,
                        int act, int* dev_status, cudaStream_t s,
                        NormCapture nc = NormCapture(), DirectRows dr = DirectRows(),
                        const MaskTable* mt = nullptr);

bool umma_router_supported(int d, int R, int E, int dtype);
size_t umma_router_packed_bytes(int d, int R, int E);
int launch_prepack_router(const void* wa, const void* wb, void* packed, int d, int R, int E,
                          cudaStream_t s);
// true: the launch below writes no tile_counts for this size
bool umma_router_splits(int64_t N, int d, int R, int E);
// out_init: initial output rows last_bias (+ resid), every row (init_all) or only those of tokens
// not kept by exactly one expert (the expert kernel stores the others, see DirectRows)
int launch_router_mask_umma(const void* x, const void* packed, float mult, uint32_t* mask_bits,
                            void* scores, void* rt_out, const void* last_bias, const void* resid,
                            void* out_init, bool init_all, int32_t* tile_counts, int64_t N, int d,
                            int R, int E, int* dev_status, cudaStream_t s,
                            ListsOut* lists = nullptr, int rule = 0, int k = 0, float tau = 0.f);
// whether it applies the ranked rules (rule: D2D_RULE_TOPK with k, D2D_RULE_DYNK with tau) itself: a
// token's scores are one thread's registers, which ranks up to 32 of them
bool umma_router_ranks(int64_t N, int d, int R, int E);

// test hooks: poll limit of the bounded device waits (2^log2, out of range = default) and
// a flag that makes CTA 0 of the next launches skip its first weight tile
void umma_debug_configure(int wait_limit_log2, int withhold_weight_tile);
void umma_debug_read(uint32_t* wait_limit, int* withhold);

}  // namespace d2d
