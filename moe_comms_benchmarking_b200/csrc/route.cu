// Expert path glue for sm_100a: (1) routing of the gathered tokens to this rank's experts
// (histogram -> offsets -> pair lists -> row-tile table for the grouped GEMMs), and (2) the
// combine that sums each token's local expert outputs and reduce-scatters the partial sums
// across ranks in the same kernel.
//
// The reference defers the permute "to the GEMM" and never performs it (its expert is the
// identity; the only trace is the routing mask in bench_nvls.py:195).  Here the permute is an
// index list: the FC1 kernel gathers token rows through pair_token[], so no token is copied.
#include <cuda_runtime.h>

#include <atomic>

#include "mcb_barrier.cuh"
#include "mcb_combine.cuh"
#include "mcb_gemm.h"
#include "mcb_route.cuh"
#include "mcb_launch.h"
#include "mcb_launchers.h"

namespace mcb {

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) route_kernel(const __grid_constant__ McbRouteArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ int s_route[kRouteSmemWords];
  route_device(a, s_route, THREADS != kRouteThreads ? kRouteAllPerThread : a.num_local_experts > 512 ? kRouteAllMany : kRouteAllAlone);
}

// ------------------------------------------------------------------------------------------------
// Combine as a kernel of its own (mcb_combine.cuh): a block owns slices of the rows of gathered tokens, the same on EVERY
// rank; it sums the local pairs of its slices, meets the matching block of every rank, and reduces across the ranks what
// this rank owns.
// ------------------------------------------------------------------------------------------------
template <bool EMU>
__global__ void __launch_bounds__(512) combine_kernel(const __grid_constant__ McbCtx ctx_p,
                                                      const __grid_constant__ McbCombineArgs args_p,
                                                      const McbCtx* ectx, const McbCombineArgs* eargs) {
  const McbCtx& c = EMU ? ectx[blockIdx.y] : ctx_p;
  const McbCombineArgs& a = EMU ? eargs[blockIdx.y] : args_p;
  pdl_wait();
  pdl_launch_dependents();
  combine_body<true>(c, a);
}

// The same in a world of one where rows allow packs of 32 bytes, by two blocks for each of the chip's 148 SMs.  With fewer blocks it is slower than the
// kernel above at large batches: 4096 tokens of 22 ids, an eighth local, by 148 / 64 / 16 blocks 7.1 / 11.7 / 36.7 us (7.2 / 10.9 / 30.5 above, 5.8 by 296),
// 8 ids and rows of 7168 34.8 / 63.3 / 207 (29.9 / 49.5 / 149, 24.1); so callers that ask for fewer get that one.
constexpr int kCombineAloneBlocks = 2 * 148;
__global__ void __launch_bounds__(512, 2) combine_alone_kernel(const __grid_constant__ McbCombineArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int offset = a.step_meta[1], T = a.step_meta[0];
  int n = *a.n_local;
  n = n < 0 ? 0 : n > a.cap ? a.cap : n;
  const int begin = offset < 0 ? 0 : offset, end = T - offset < n ? T : offset + n;
  if (begin >= end) return;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  if ((long long)(end - begin) * ((a.hidden + 255) / 256) <= warps) combine_alone_items<16, 8>(a, begin, end, offset);
  else combine_alone_items<32, 2>(a, begin, end, offset);
}

}  // namespace mcb

using namespace mcb;

extern "C" {

int mcb_sizeof_route_args() { return (int)sizeof(McbRouteArgs); }
int mcb_sizeof_combine_args() { return (int)sizeof(McbCombineArgs); }

// Blocks of a routing launch: as many as the caller asks for, but they wait for one another, so no more than the device holds at once; 0: refused.
int mcb_route_blocks(int grid, int resident) {
  if (grid < 1 || grid > 128) return 0;
  return grid < resident ? grid : resident > 1 ? resident : 1;
}

// Threads of its blocks (see kRouteBlocks).
int mcb_route_threads(const McbRouteArgs* args, int grid) {
  const long long entries = (long long)args->max_tokens * args->topk;
  return grid < kRouteBlocks && entries > (long long)kRouteKept * kRouteThreads * grid ? kRouteWideThreads : kRouteThreads;
}

int mcb_launch_route(const McbRouteArgs* args, int grid, int pdl, cudaStream_t stream) {
  if (mcb_route_blocks(grid, grid) == 0 || args->num_local_experts > kMaxLocalExperts || args->num_local_experts < 1)
    return cudaErrorInvalidValue;
  const int threads = mcb_route_threads(args, grid);
  auto kernel = threads == kRouteThreads ? route_kernel<kRouteThreads> : route_kernel<kRouteWideThreads>;
  // What the device holds does not change: asked for once per device and kernel.
  static std::atomic<int> known[2][64];
  int dev = 0, resident = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return (int)err;
  std::atomic<int>* slot = dev < 64 ? &known[threads == kRouteThreads][dev] : nullptr;
  if (slot) resident = slot->load(std::memory_order_relaxed);
  if (resident == 0) {
    int sms = 0, per_sm = 0;
    if ((err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return (int)err;
    if ((err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0)) != cudaSuccess) return (int)err;
    resident = sms * per_sm;
    if (slot) slot->store(resident, std::memory_order_relaxed);
  }
  return launch_kernel(kernel, dim3(mcb_route_blocks(grid, resident)), dim3(threads), 0, stream, pdl, false, *args);
}

int mcb_launch_combine(const McbCtx* ctx, const McbCombineArgs* args, int grid, int threads, int pdl,
                       cudaStream_t stream) {
  if (grid < 1 || grid > MCB_MAX_BLOCKS || threads < 32 || threads > 512 || (threads & 31) || args->hidden % 8)
    return cudaErrorInvalidValue;
  if (grid >= kCombineAloneBlocks && ctx->world == 1 && args->hidden % 16 == 0 &&
      !((reinterpret_cast<uintptr_t>(args->y) | reinterpret_cast<uintptr_t>(args->out)) & 31))
    return launch_kernel(combine_alone_kernel, dim3(grid), dim3(threads), 0, stream, pdl, false, *args);
  return launch_kernel(combine_kernel<false>, dim3(grid), dim3(threads), 0, stream, pdl, false, *ctx, *args,
                       (const McbCtx*)nullptr, (const McbCombineArgs*)nullptr);
}

int mcb_emu_combine(const McbCtx* d_ctx, const McbCombineArgs* d_args, int world, int grid, int threads,
                    cudaStream_t stream) {
  if (grid < 1 || grid > MCB_MAX_BLOCKS || threads < 32 || threads > 512 || (threads & 31)) return cudaErrorInvalidValue;
  McbCtx dummy{};
  McbCombineArgs dargs{};
  return launch_kernel(combine_kernel<true>, dim3(grid, world), dim3(threads), 0, stream, 0, true, dummy, dargs,
                       d_ctx, d_args);
}

}  // extern "C"
