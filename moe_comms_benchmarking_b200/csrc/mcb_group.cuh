// The threads that run a block-wide device function together: the whole block, or some of its warps behind a named barrier.
#pragma once

namespace mcb {

struct BlockGroup {
  __device__ __forceinline__ int tid() const { return (int)threadIdx.x; }
  __device__ __forceinline__ unsigned size() const { return blockDim.x; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
};
// The WARPS warps of the block from warp FIRST on, with named barrier BAR of their own.
template <int FIRST, int WARPS, int BAR>
struct WarpGroup {
  __device__ __forceinline__ int tid() const { return (int)threadIdx.x - 32 * FIRST; }
  __device__ __forceinline__ unsigned size() const { return 32u * WARPS; }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" :: "n"(BAR), "n"(32 * WARPS) : "memory"); }
};

}  // namespace mcb
