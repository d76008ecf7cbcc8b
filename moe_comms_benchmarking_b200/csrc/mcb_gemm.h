// Argument blocks of the expert path: routing (pair lists, row tiles) and grouped GEMMs.
// Mirrored with ctypes in ops/_ext.py.
#pragma once
#include <stdint.h>

#include "mcb_ctx.h"

#define MCB_GEMM_FC1 0          // gate/up projection + SwiGLU epilogue
#define MCB_GEMM_FC2 1          // down projection + per-row scale epilogue
// Tensor maps of the fused FFN: token rows (gathered four at a time), gate/up and down tiles (16 KB, then 32 KB), and
// activations in boxes of 4, 8, ... 32 rows.
#define MCB_FFN_MAP_X 0
#define MCB_FFN_MAP_W1 1
#define MCB_FFN_MAP_W2 2
#define MCB_FFN_MAP_ACT 5
#define MCB_FFN_TMAPS 13
#define MCB_GEMM_ERR_TIMEOUT 5  // status code: a bounded mbarrier wait ran out

#ifdef __cplusplus
extern "C" {
#endif

// One grouped GEMM: out[row, :] = epilogue(A[row_index[row], :] . W[expert(row)]^T).
typedef struct {
  const void* a_base;          // A rows, bf16, K contiguous
  uint64_t a_row_bytes;
  const int32_t* row_index;    // pair row -> A row (NULL: identity)
  const float* row_scale;      // FC2: factor per pair row (NULL: 1)
  void* out;                   // bf16 [pair rows, n_out]
  uint64_t out_row_bytes;
  const int32_t* tile_expert;  // per row tile: local expert
  const int32_t* tile_row0;    //               first pair row
  const int32_t* tile_rows;    //               rows in the tile (1..128)
  const int32_t* num_m_tiles;  // device scalar
  int32_t n_total;             // weight rows per expert (FC1: 2*I, gate rows then up rows; FC2: H)
  int32_t k_total;             // reduction length (FC1: H; FC2: I)
  uint32_t* status;            // status words (may be NULL)
  uint64_t timeout_ns;
} McbGemmArgs;

// Grouped SwiGLU FFN with the weights as the M operand (mcb_ffn.cuh): both projections in one
// persistent kernel over the pair lists written by the routing.
typedef struct {
  const void* x;               // gathered tokens [T, hidden] bf16
  const int32_t* pair_token;   // [P] pair row -> gathered token
  const float* pair_prob;      // [P] routing weight of each pair row (NULL: 1)
  const int32_t* expert_offset;  // [E_loc + 1] first pair row of each local expert
  const int32_t* max_rows;     // device scalar: largest pair count of one expert
  void* act;                   // [P, intermediate] bf16 (written by the gate/up blocks, read by the down blocks)
  void* y;                     // [P, hidden] bf16 = prob * (act . Wd^T)
  int32_t* ffn_done;           // [E_loc] warp shares of gate/up blocks finished (zeroed by the routing)
  int32_t num_local_experts;
  int32_t hidden;              // multiple of 256
  int32_t intermediate;        // multiple of 128
  int32_t reserved0;
  uint32_t* status;
  uint64_t timeout_ns;
  const void* w1;              // packed interleaved gate/up matrix (E * 2I rows, hidden columns), see mcb_ffn.cuh
  const void* w2;              // packed down matrix (E * hidden rows, I columns)
  // MCB_FFN_TMAPS tensor maps of 128 bytes, 64-byte aligned (mcb_make_ffn_tmaps): in host memory, from where a launch copies
  // them into its parameters; for ranks emulated inside one launch in device memory.
  const void* tmaps;
} McbFfnArgs;

// Routing of the gathered tokens to this rank's experts.
typedef struct {
  const int64_t* topk_idx;     // gathered [T, topk]
  const float* topk_w;         // gathered [T, topk]
  const int32_t* num_tokens;   // device scalar T (step_meta[0])
  int32_t topk;
  int32_t expert_begin;        // first expert owned by this rank
  int32_t num_local_experts;
  int32_t max_tokens;          // capacity of the gathered buffers (bounds check)
  int32_t* expert_count;       // [E_loc]        (scratch, zero between launches)
  int32_t* expert_offset;      // [E_loc + 1]    first pair row of each expert
  int32_t* pair_token;         // [P] gathered-token index of each pair row
  float* pair_prob;            // [P] routing weight of each pair row
  int32_t* pair_pos;           // [T, topk] pair row of (token, k), -1 if the expert is not local
  int32_t* tile_expert;        // row-tile table consumed by the grouped GEMMs
  int32_t* tile_row0;
  int32_t* tile_rows;
  int32_t* num_m_tiles;        // device scalar
  int32_t* sync;               // [4] zero between launches: blocks that have counted, blocks that have left, -, -
  int32_t max_pairs;           // capacity of the pair arrays
  int32_t max_tiles;           // capacity of the tile table
  uint32_t* status;
  uint64_t timeout_ns;
  int32_t* max_rows;           // device scalar: largest number of pair rows of one expert (may be NULL)
  int32_t* ffn_done;           // [E_loc] gate/up blocks finished per expert, set to zero here (may be NULL)
} McbRouteArgs;

// Local pre-sum of each token's expert outputs + cross-rank reduce-scatter.
typedef struct {
  const void* y;               // [P, hidden] bf16, already scaled by the routing weight
  const int32_t* pair_pos;     // [T, topk]
  uint64_t partial_off;        // heap: [T_cap, hidden] bf16 per-rank partial sums
  void* out;                   // local [cap, hidden] bf16
  const int32_t* n_local;
  const int32_t* step_meta;    // [valid, offset, max, epoch]
  int32_t hidden;
  int32_t topk;
  int32_t cap;                 // per-rank capacity
  int32_t site;
  // Bytes between two copies of the partial-sum buffer (0 = one copy).  With two, a caller that runs
  // layers back to back alternates between them, so a rank that is already writing the partial sums of
  // the next layer cannot disturb a peer that is still reducing this one (the barrier inside every
  // combine keeps ranks within one layer of each other).
  uint64_t partial_par_stride;
} McbCombineArgs;

#ifdef __cplusplus
}
#endif

#ifdef MCB_WITH_LAYER_ARGS
// Everything one MoE layer needs, as ONE kernel parameter (or one element of a device array when
// several ranks are emulated inside one launch): the context and the argument blocks of the four phases.
typedef struct alignas(64) {
  McbCtx ctx;
  McbAgvArgs agv;
  // World of one only: where the rows of route.topk_idx and route.topk_w (null: weight 1) come from, if agv is what gathers
  // them and agv.step_meta is what counts them; local_ids null: the routing reads the gathered rows.
  const int64_t* local_ids;
  const float* local_probs;
  McbRouteArgs route;
  McbFfnArgs ffn;
  McbCombineArgs cmb;
  // Optional phase trace (null = off): block 0 stores the global timer (ns) at kernel entry and after
  // dispatch, grid barrier, routing, grid barrier, experts, grid barrier, combine (8 words).  No barrier stands between
  // routing and experts: that phase is empty, and the wait for the other blocks' pair lists is part of the experts.
  unsigned long long* trace;
  unsigned long long reserved0;
} McbLayerArgs;

#define MCB_STEP_SETS 16        // weight sets of one launch (four tensor maps each, in its parameters)
#define MCB_STEP_SYNC_WORDS 160 // counters of a step, 128 bytes apart

// Several layers of a world of one as ONE launch (moe_step.cu).  `layer` is what a layer kernel takes, of any weight set; the
// buffers that layers in flight do not share come three times (pair lists and counters) or twice: [0] those of the last layer,
// which are layer.route's and layer.ffn's own.
typedef struct alignas(64) {
  McbLayerArgs layer;
  const int64_t* ids;            // expert ids, weights (null: 1) and rows of this rank's tokens where the all-gather reads them
  const float* probs;
  const void* x;
  int32_t* pair_token[3];
  float* pair_prob[3];
  int32_t* pair_pos[3];
  int32_t* ffn_done[3];
  void* act[2];                  // the second ones hold two_rows pair rows; larger steps use one buffer for all layers
  void* y[2];
  int64_t two_rows;
  int32_t* expert_count;         // [3][E_loc], zero between launches
  int32_t* sync;                 // [MCB_STEP_SYNC_WORDS], zero between launches
  alignas(64) unsigned long long map_x[16];    // token rows
  unsigned long long map_act[2][8][16];        // activations, by box
} McbMoeStepArgs;
#endif
