// One step's inputs into a dispatcher's persistent buffers: hidden rows, routing, weights and the token count in ONE
// launch, from device memory or straight from pinned host memory (which the GPU reads over PCIe).  As three copies and a
// fill this was four launches of about 4 us of host time each, more than the kernels of a small layer take.
#include <cuda_runtime.h>

#include "mcb_ctx.h"
#include "mcb_launch.h"
#include "mcb_ptx.cuh"

namespace mcb {

constexpr int kLoadThreads = 256;

__device__ __forceinline__ uint4 load_pack(const uint8_t* p, bool aligned) {
  if (aligned) return ld_v4_stream(p);
  return make_uint4(ld_b32(p), ld_b32(p + 4), ld_b32(p + 8), ld_b32(p + 12));
}

__global__ void __launch_bounds__(kLoadThreads) load_batch_kernel(const __grid_constant__ McbLoadArgs a) {
  pdl_wait();                 // an earlier step may still be reading the buffers
  pdl_launch_dependents();
  // The three ranges end to end as 16-byte packs, so that all loads of a thread are in flight together.
  long long end[3];
  bool aligned[3];
  long long run = 0;
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    run += (long long)(a.bytes[t] >> 4);
    end[t] = run;
    aligned[t] = (reinterpret_cast<uintptr_t>(a.src[t]) & 15) == 0;
  }
  const long long first = (long long)blockIdx.x * kLoadThreads + threadIdx.x, stride = (long long)gridDim.x * kLoadThreads;
  for (long long i0 = first; i0 < run; i0 += stride * 4) {
    uint4 v[4];
    uint8_t* dst[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * stride;
      dst[u] = nullptr;
      if (i < run) {
        const int t = (i >= end[0]) + (i >= end[1]);
        const long long off = (i - (t == 0 ? 0 : (t == 1 ? end[0] : end[1]))) * 16;
        const void* src = t == 0 ? a.src[0] : (t == 1 ? a.src[1] : a.src[2]);
        void* d = t == 0 ? a.dst[0] : (t == 1 ? a.dst[1] : a.dst[2]);
        v[u] = load_pack(reinterpret_cast<const uint8_t*>(src) + off, t == 0 ? aligned[0] : (t == 1 ? aligned[1] : aligned[2]));
        dst[u] = reinterpret_cast<uint8_t*>(d) + off;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (dst[u]) st_v4(dst[u], v[u]);
  }
  if (blockIdx.x == gridDim.x - 1) {          // what is left behind the last whole pack of a range, and the count
    const int t = threadIdx.x >> 2, w = threadIdx.x & 3;
    if (t < 3 && w < (int)(a.bytes[t] & 15) >> 2) {
      const uint64_t off = (a.bytes[t] & ~15ull) + w * 4;
      st_b32(reinterpret_cast<uint8_t*>(a.dst[t]) + off, ld_b32(reinterpret_cast<const uint8_t*>(a.src[t]) + off));
    }
    if (threadIdx.x == kLoadThreads - 1) *a.n_local = a.n;
  }
}

}  // namespace mcb

using namespace mcb;

extern "C" {

int mcb_sizeof_load_args() { return (int)sizeof(McbLoadArgs); }

int mcb_launch_load_batch(const McbLoadArgs* a, int pdl, cudaStream_t stream) {
  if (!a || !a->n_local || a->n < 0) return cudaErrorInvalidValue;
  uint64_t packs = 0;
  for (int t = 0; t < 3; ++t) {
    if (a->bytes[t] & 3) return cudaErrorInvalidValue;
    if (a->bytes[t] && (!a->src[t] || !a->dst[t] || (reinterpret_cast<uintptr_t>(a->src[t]) & 3) ||
                        (reinterpret_cast<uintptr_t>(a->dst[t]) & 15)))
      return cudaErrorInvalidValue;
    packs += a->bytes[t] >> 4;
  }
  uint64_t grid = (packs + kLoadThreads - 1) / kLoadThreads;
  grid = grid < 1 ? 1 : (grid > 592 ? 592 : grid);         // four blocks per SM hold 64 KB of loads in flight
  return launch_kernel(load_batch_kernel, dim3((unsigned)grid), dim3(kLoadThreads), 0, stream, pdl, false, *a);
}

}  // extern "C"
