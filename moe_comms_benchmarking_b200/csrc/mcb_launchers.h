// Launch functions that are defined in one source file and called from another.
#pragma once
#include <cuda_runtime.h>

#include "mcb_gemm.h"

#ifdef __cplusplus
extern "C" {
#endif

int mcb_launch_metadata(const McbCtx* ctx, const McbMetaArgs* args, int pdl, cudaStream_t stream);
int mcb_launch_agv(const McbCtx* ctx, const McbAgvArgs* args, int grid, int threads, int pdl, cudaStream_t stream);
int mcb_launch_rsv(const McbCtx* ctx, const McbRsvArgs* args, int grid, int threads, int pdl, cudaStream_t stream);
int mcb_launch_dense_step(const McbCtx* ctx, const McbDenseStepArgs* args, int grid, int threads, int pdl, cudaStream_t stream);
int mcb_launch_a2a_dispatch(const McbCtx* ctx, const McbA2ADispatchArgs* args, int grid, int threads, int pdl, cudaStream_t stream);
int mcb_launch_a2a_combine(const McbCtx* ctx, const McbA2ACombineArgs* args, int grid, int threads, int pdl, cudaStream_t stream);
int mcb_launch_a2a_step(const McbCtx* ctx, const McbA2AStepArgs* args, int grid, int threads, int pdl, cudaStream_t stream);
int mcb_launch_combine(const McbCtx* ctx, const McbCombineArgs* args, int grid, int threads, int pdl, cudaStream_t stream);

#ifdef __cplusplus
}
#endif
