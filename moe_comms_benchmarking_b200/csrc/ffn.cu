// The expert path of a MoE layer for sm_100a: the grouped SwiGLU FFN with the weights as the M
// operand (mcb_ffn.cuh) as a kernel of its own, and the WHOLE layer as one cooperative kernel:
//
//   dispatch    every CTA pushes its share of the local tokens to all ranks (multimem.st + cross-GPU
//               barrier, or flagged packets for small steps)                          mcb_dense.cuh
//   routing     counts -> offsets -> pair lists for this rank's experts                  mcb_route.cuh
//   experts     gate/up and down units, one persistent weight stream                      mcb_ffn.cuh
//   combine     per-token pre-sum of the local expert outputs into the symmetric buffer, block-matched
//               cross-GPU barrier, multimem.ld_reduce of the rows this rank owns       mcb_combine.cuh
//
// The launch is cooperative: all CTAs are resident.  A grid-wide barrier follows the dispatch (not in a world of one that
// routes by its own inputs) and the experts, and one falls inside the routing of many entries.  None stands between routing
// and experts: every CTA works out the experts' offsets itself and starts its weight stream at once, and only the roles
// that read pair lists or token rows wait for the other CTAs.  The reference
// stops at the identity expert (bench_nvls.py:109-121); its dispatch and combine are the first and the
// last phase here.  EMU = true runs several ranks inside one launch (gridDim.y = world, each y-slice
// with its own argument block in device memory), which is how the cross-rank protocol of this kernel
// is tested on a single GPU.
#include <cuda.h>
#include <cuda_runtime.h>

#define MCB_WITH_LAYER_ARGS
#include "mcb_combine.cuh"
#include "mcb_dense.cuh"
#include "mcb_ffn.cuh"
#include "mcb_gemm.h"
#include "mcb_launch.h"
#include "mcb_launchers.h"
#include "mcb_route.cuh"
#include "mcb_tmap.h"

namespace mcb {

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFfnThreads, 1) expert_ffn_kernel(const __grid_constant__ McbFfnArgs a,
                                                                                              const __grid_constant__ FfnMaps maps) {
  ffn_setup<false>(maps.map);
  pdl_wait();
  pdl_launch_dependents();
  ffn_device(a, maps.map);
  ffn_teardown();
}

template <bool EMU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFfnThreads, 1)
moe_layer_kernel(const __grid_constant__ McbLayerArgs p_, const __grid_constant__ FfnMaps maps_, const McbLayerArgs* eargs) {
  const McbLayerArgs& p = EMU ? eargs[blockIdx.y] : p_;
  const CUtensorMap* maps = EMU ? reinterpret_cast<const CUtensorMap*>(p.ffn.tmaps) : maps_.map;
  const McbCtx& c = p.ctx;
  uint32_t ll_launch = 0;
  const bool tracing = p.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0;
  auto stamp = [&](int i) { if (tracing) p.trace[i] = globaltimer_ns(); };
  // Grid-wide barriers count up a word that is back at zero whenever a launch has ended (its last block resets it).
  uint32_t* arrivals = epoch_ptr(c, MCB_SITE_LAYER, 1);
  uint32_t target = 0;
  auto meet = [&] { grid_sync(c, arrivals, target += gridDim.x); };
  stamp(0);
  ffn_setup<EMU>(maps);
  const GatheredRows got = agv_device<MCB_SITE_FC1_FUSED>(c, p.agv, ll_launch);      // waits for the previous kernel first
  stamp(1);
  // Routing needs the ids and weights that its arguments name, of all gathered tokens.  In a world of one these are usually
  // rows that this all-gather copies: then they are read where they come from, and nobody waits for the copy.
  const bool alone = c.world == 1 && p.local_ids && got.offset == 0 && got.valid <= got.n;
  const int64_t* ids = alone ? p.local_ids : p.route.topk_idx;
  const float* probs = alone ? p.local_probs : p.route.topk_w;
  if (!alone) meet();
  stamp(2);
  const FfnSmem sm;
  RouteSmem m(reinterpret_cast<int*>(sm.pipe));              // the pipeline is not in use yet
  m.off = sm.off;
  const RouteShare share = route_share(p.route, (int)blockIdx.x, (int)gridDim.x);
  const BlockGroup all;
  if (route_counts_all(all, share)) {
    route_count<true>(all, p.route, ids, m, 0, share.entries, share.lo);
  } else {
    route_count<false>(all, p.route, ids, m, share.lo, share.hi, 0);
    route_publish(all, p.route.num_local_experts, p.route.expert_count, m);
    meet();
    route_collect(all, p.route.num_local_experts, p.route.expert_count, m);
  }
  const int max_rows = route_offsets(all, p.route, m, blockIdx.x == 0);
  route_place(all, p.route, ids, probs, m, share);
  // This block's pair rows (and gathered rows, when alone) are there.  Nobody waits here: the weight stream starts at
  // once, the roles that read rows or lists wait for all blocks.
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(arrivals, 1u);
  }
  target += gridDim.x;
  stamp(3);
  stamp(4);                                                  // an empty phase, see McbLayerArgs::trace
  ffn_run(p.ffn, maps, max_rows, FfnReady{arrivals, (int)target});
  ffn_teardown();
  stamp(5);
  meet();                                                   // every y row is written before any is summed
  stamp(6);
  if (blockIdx.x == gridDim.x - 1)                          // every block has read the counters of the routing
    for (int e = threadIdx.x; e < p.route.num_local_experts; e += blockDim.x) p.route.expert_count[e] = 0;
  combine_body<false>(c, p.cmb, ll_launch);      // partial sums alternate between two buffers, layer by layer
  stamp(7);
  launch_end(c, MCB_SITE_FC1_FUSED, ll_launch, arrivals);
}

}  // namespace mcb

using namespace mcb;

extern "C" {

int mcb_sizeof_ffn_args() { return (int)sizeof(McbFfnArgs); }
int mcb_sizeof_layer_args() { return (int)sizeof(McbLayerArgs); }
int mcb_ffn_smem_bytes() { return kFfnSmemBytes; }
int mcb_ffn_threads() { return kFfnThreads; }

static bool configure_ffn_kernels() {
  static int state = 0;   // 0 = not tried, 1 = ok, -1 = failed
  if (state == 0) {
    cudaError_t e1 = cudaFuncSetAttribute(expert_ffn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFfnSmemBytes);
    cudaError_t e2 = cudaFuncSetAttribute(moe_layer_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFfnSmemBytes);
    cudaError_t e3 = cudaFuncSetAttribute(moe_layer_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFfnSmemBytes);
    state = (e1 == cudaSuccess && e2 == cudaSuccess && e3 == cudaSuccess) ? 1 : -1;
  }
  return state == 1;
}

static int check_ffn_args(const McbFfnArgs* a) {
  if (!a || !a->x || !a->pair_token || !a->expert_offset || !a->max_rows || !a->act || !a->y || !a->ffn_done) return 1;
  if (!a->w1 || !a->w2 || (reinterpret_cast<uintptr_t>(a->w1) & 15) || (reinterpret_cast<uintptr_t>(a->w2) & 15)) return 1;
  if (a->num_local_experts < 1 || a->num_local_experts > kFfnMaxExperts) return 1;
  if (a->hidden < 256 || a->hidden % 256 || a->intermediate < 128 || a->intermediate % 128) return 1;
  if (!a->tmaps || (reinterpret_cast<uintptr_t>(a->tmaps) & 63)) return 1;
  return 0;
}

// The kernels run in CTA pairs: an odd grid is rounded down, one CTA is rounded up.
static int pair_grid(int grid) { return grid < 2 ? 2 : grid & ~1; }

// The tensor maps of one FFN launch (MCB_FFN_TMAPS x 128 bytes) into 64-byte aligned host memory.  x: token rows; act: activations;
// w1, w2: the packed weights.
int mcb_make_ffn_tmaps(void* out, const void* x, uint64_t x_rows, const void* act, uint64_t pair_rows, const void* w1, const void* w2,
                       int experts, int hidden, int intermediate) {
  uint8_t* o = reinterpret_cast<uint8_t*>(out);
  const uint64_t E = experts, H = hidden, I = intermediate;
  if (!out || experts < 1 || hidden % 256 || intermediate % 128) return (int)cudaErrorInvalidValue;
  int err = make_tmap_bf16(o + MCB_FFN_MAP_X * 128, x, x_rows, H, 1);
  for (int b = 0; b < kFfnMaxGroups && !err; ++b)
    err = make_tmap_bf16(o + (MCB_FFN_MAP_ACT + b) * 128, act, pair_rows, I, 4 * (b + 1));
  for (int d = 0; d < 2 && !err; ++d) {
    err = make_tmap_flat(o + (MCB_FFN_MAP_W1 + 2 * d) * 128, w1, E * 2 * I * H * 2, 8 * (d + 1));
    if (!err) err = make_tmap_flat(o + (MCB_FFN_MAP_W2 + 2 * d) * 128, w2, E * H * I * 2, 8 * (d + 1));
  }
  return err;
}

// Gate/up + SwiGLU + down over the pair lists of a routing, as one persistent launch.
int mcb_launch_expert_ffn(const McbFfnArgs* args, int grid, int pdl, cudaStream_t stream) {
  if (grid < 1 || check_ffn_args(args)) return cudaErrorInvalidValue;
  if (!configure_ffn_kernels()) return cudaErrorUnknown;
  // A down block waits for gate/up blocks that other CTAs compute: all CTAs must be resident.
  return launch_kernel(expert_ffn_kernel, dim3(pair_grid(grid)), dim3(kFfnThreads), kFfnSmemBytes, stream, pdl, true, *args,
                       *reinterpret_cast<const FfnMaps*>(args->tmaps));
}

static int check_layer_args(const McbLayerArgs* p, int grid) {
  if (!p || grid < 1 || grid > MCB_MAX_BLOCKS || check_ffn_args(&p->ffn)) return 1;
  if (p->route.num_local_experts < 1 || p->route.num_local_experts > kMaxLocalExperts) return 1;
  if (p->cmb.hidden % 8) return 1;
  return 0;
}

// One whole MoE layer (dispatch, routing, experts, combine) as one cooperative launch.
int mcb_launch_moe_layer(const McbLayerArgs* p, int grid, int pdl, cudaStream_t stream) {
  if (check_layer_args(p, grid)) return cudaErrorInvalidValue;
  if (!configure_ffn_kernels()) return cudaErrorUnknown;
  return launch_kernel(moe_layer_kernel<false>, dim3(pair_grid(grid)), dim3(kFfnThreads), kFfnSmemBytes, stream, pdl, true, *p,
                       *reinterpret_cast<const FfnMaps*>(p->ffn.tmaps), (const McbLayerArgs*)nullptr);
}

// One decode step with real experts, issued natively: the count exchange, then num_layers layers; layer l uses the argument
// block (weight set) l % num_sets.  With `step` (mcb_prepare_moe_step, over the same argument blocks) several layers share a
// launch, without it each is a layer kernel.
int mcb_launch_moe_step(const McbMoeStepArgs* p, const McbLayerArgs* sets, int num_sets, int first, int num_layers, int grid, int pdl,
                        cudaStream_t stream);                                                        // moe_step.cu

int mcb_moe_decode_step(const McbCtx* ctx, const McbMetaArgs* meta, const McbLayerArgs* layers, int num_sets,
                        int num_layers, int grid, int pdl, const McbMoeStepArgs* step, cudaStream_t stream) {
  if (!ctx || !meta || !layers || num_sets < 1 || num_layers < 0) return cudaErrorInvalidValue;
  for (int s = 0; s < num_sets; ++s)
    if (check_layer_args(&layers[s], grid)) return cudaErrorInvalidValue;
  int err = mcb_launch_metadata(ctx, meta, pdl, stream);
  const int together = !step || num_layers < 2 ? 1 : num_sets <= MCB_STEP_SETS ? num_layers : MCB_STEP_SETS;
  for (int l = 0; l < num_layers && err == 0; l += together) {
    const int n = num_layers - l < together ? num_layers - l : together;
    err = n > 1 ? mcb_launch_moe_step(step, layers, num_sets, l, n, grid, pdl, stream)
                : mcb_launch_moe_layer(&layers[l % num_sets], grid, pdl, stream);
  }
  return err;
}

int mcb_emu_moe_layer(const McbLayerArgs* d_args, const McbLayerArgs* h_args0, int world, int grid,
                      cudaStream_t stream) {
  if (!d_args || world < 1 || check_layer_args(h_args0, grid)) return cudaErrorInvalidValue;
  if (!configure_ffn_kernels()) return cudaErrorUnknown;
  McbLayerArgs dummy{};
  FfnMaps no_maps{};
  return launch_kernel(moe_layer_kernel<true>, dim3(pair_grid(grid), world), dim3(kFfnThreads), kFfnSmemBytes, stream, 0, true,
                       dummy, no_maps, d_args);
}

}  // extern "C"
