// Library-wide exports: struct sizes (checked by the Python binding), error strings and
// small device-memory utilities.
#include <cuda_runtime.h>

#include "mcb_launchers.h"

extern "C" {

int mcb_sizeof_launch() { return (int)sizeof(McbLaunch); }

int mcb_launch(const McbLaunch* l, cudaStream_t stream) {
  if (!l) return (int)cudaErrorInvalidValue;
  const int g = l->grid, t = l->threads, pdl = l->pdl;
  switch (l->op) {
    case MCB_OP_METADATA:     return mcb_launch_metadata(l->ctx, static_cast<const McbMetaArgs*>(l->args), pdl, stream);
    case MCB_OP_AGV:          return mcb_launch_agv(l->ctx, static_cast<const McbAgvArgs*>(l->args), g, t, pdl, stream);
    case MCB_OP_RSV:          return mcb_launch_rsv(l->ctx, static_cast<const McbRsvArgs*>(l->args), g, t, pdl, stream);
    case MCB_OP_DENSE_STEP:   return mcb_launch_dense_step(l->ctx, static_cast<const McbDenseStepArgs*>(l->args), g, t, pdl, stream);
    case MCB_OP_A2A_DISPATCH: return mcb_launch_a2a_dispatch(l->ctx, static_cast<const McbA2ADispatchArgs*>(l->args), g, t, pdl, stream);
    case MCB_OP_A2A_COMBINE:  return mcb_launch_a2a_combine(l->ctx, static_cast<const McbA2ACombineArgs*>(l->args), g, t, pdl, stream);
    case MCB_OP_A2A_STEP:     return mcb_launch_a2a_step(l->ctx, static_cast<const McbA2AStepArgs*>(l->args), g, t, pdl, stream);
    case MCB_OP_COMBINE:      return mcb_launch_combine(l->ctx, static_cast<const McbCombineArgs*>(l->args), g, t, pdl, stream);
  }
  return (int)cudaErrorInvalidValue;
}

// Name of an operation, null behind the last one: a caller that numbers them too compares.
const char* mcb_op_name(int op) {
  switch (op) {
    case MCB_OP_METADATA:     return "metadata";
    case MCB_OP_AGV:          return "all_gather_v";
    case MCB_OP_RSV:          return "reduce_scatter_v";
    case MCB_OP_DENSE_STEP:   return "dense_step";
    case MCB_OP_A2A_DISPATCH: return "a2a_dispatch";
    case MCB_OP_A2A_COMBINE:  return "a2a_combine";
    case MCB_OP_A2A_STEP:     return "a2a_step";
    case MCB_OP_COMBINE:      return "expert_combine";
  }
  return nullptr;
}

int mcb_sizeof_ctx() { return (int)sizeof(McbCtx); }
int mcb_sizeof_meta_args() { return (int)sizeof(McbMetaArgs); }
int mcb_sizeof_agv_args() { return (int)sizeof(McbAgvArgs); }
int mcb_sizeof_rsv_args() { return (int)sizeof(McbRsvArgs); }
int mcb_sizeof_a2a_dispatch_args() { return (int)sizeof(McbA2ADispatchArgs); }
int mcb_sizeof_a2a_combine_args() { return (int)sizeof(McbA2ACombineArgs); }
int mcb_sizeof_norm_args() { return (int)sizeof(McbNormArgs); }

const char* mcb_error_string(int err) { return cudaGetErrorString((cudaError_t)err); }

int mcb_max_ranks() { return MCB_MAX_RANKS; }
int mcb_max_blocks() { return MCB_MAX_BLOCKS; }
int mcb_num_sites() { return MCB_NUM_SITES; }

}  // extern "C"
