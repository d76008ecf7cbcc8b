// Combine body shared by the stand-alone combine kernel and the fused kernels.
//
// The work is cut into items, a slice of the row of one gathered token; block b owns the items i with i % nact == b on
// EVERY rank.
//   phase A  partial[item] = sum over the local (token, k) pairs of y[pair]       (this rank's heap)
//   barrier  block b of every rank has written its items' partial sums
//   phase B  for the items of block b whose token this rank owns: out = sum over ranks of partial
//            (multimem.ld_reduce in the switch, or peer loads).
// A world of one writes phase A's sums straight to the output.  A warp serves an item with 1, 2 or 4 16-byte packs per
// lane (32, 64 or 128 packs per item), as many as still give every warp of the grid an item.  With one or two packs it keeps
// eight or four pair rows in flight: with one token and two rows in flight the sum over 22 rows was a chain of eleven trips
// to L2 (7.9 us of a layer, now 2), with one warp per token 190 rows of 7168 values occupied an eighth of the chip (46 us,
// now 9).  With four packs every warp has an item and memory is the limit; what is best there depends on the kernel around:
//   combine_kernel (ALONE)  one row at a time, with ordinary loads.  4096 rows of 1024 values, 8 pairs each: 9.5 us (18.4 with
//                           four rows in flight and streaming loads, 28 with two, 11.4 with four and ordinary loads); 22 pairs
//                           each, 184 MB of them: 39.6 (53, 90, 61).  A world of one comes here with rows that are no multiple of 32 bytes,
//                           with y or out off a 32-byte boundary, and with fewer blocks than combine_alone_kernel takes;
//   behind the experts      two rows, with streaming loads.  The combine of the layer kernel at 4096 / 2048 tokens of 22 pairs:
//                           41 / 24 us (44 / 26 with four rows, 59 / 37 with one and ordinary loads, 53 / 32 with one).
// Call from all threads of the block (any size that is a multiple of 32), or in a world of one from `nwarps` of its warps.
#pragma once
#include <type_traits>

#include "mcb_barrier.cuh"
#include "mcb_gemm.h"

namespace mcb {

__device__ __forceinline__ void acc_row(float (&acc)[8], uint4 v) {
  acc[0] += bf16_lo(v.x); acc[1] += bf16_hi(v.x);
  acc[2] += bf16_lo(v.y); acc[3] += bf16_hi(v.y);
  acc[4] += bf16_lo(v.z); acc[5] += bf16_hi(v.z);
  acc[6] += bf16_lo(v.w); acc[7] += bf16_hi(v.w);
}

// Sum over ranks of one 16-byte pack of the partial buffers (phase B).
__device__ __forceinline__ uint4 combine_reduce_pack(const McbCtx& c, uint64_t off) {
  if (c.transport == MCB_TRANSPORT_MULTIMEM) return mm_ld_reduce_bf16x8(c.heap_mc + off);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < c.world; k0 += 8) {       // eight peers' loads in flight
    uint4 w[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      int q = c.rank + k0 + u;
      if (q >= c.world) q -= c.world;
      w[u] = k0 + u < c.world ? ld_v4_stream(c.heap_peer[q] + off) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) acc_row(acc, w[u]);
  }
  return make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]),
                    pack_bf16x2(acc[4], acc[5]), pack_bf16x2(acc[6], acc[7]));
}

struct CombineShape {
  int T, offset, n;             // gathered tokens, first own one, own ones
  int packs, slices, nact;
  uint64_t row_bytes, partial_off;
};

// PL = packs per lane.
template <int PL, bool ALONE>
__device__ __forceinline__ void combine_items(const McbCtx& c, const McbCombineArgs& a, const CombineShape& s, uint32_t ep, int warp,
                                              int nwarps) {
  constexpr int R = PL == 1 ? 8 : PL == 2 ? 4 : (ALONE ? 1 : 2);       // pair rows in flight
  const int lane = threadIdx.x & 31, bid = blockIdx.x;
  const uint8_t* y = reinterpret_cast<const uint8_t*>(a.y);
  const bool alone = c.world == 1;
  uint8_t* partial = c.heap_local + s.partial_off;
  uint8_t* out = reinterpret_cast<uint8_t*>(a.out);
  const long long items = (long long)s.T * s.slices;
  const long long first = bid + (long long)warp * s.nact, step = (long long)s.nact * nwarps;
  for (long long i = first; i < items; i += step) {
    const int t = (int)(i / s.slices);
    const int p0 = (int)(i - (long long)t * s.slices) * 32 * PL + lane;
    float acc[PL][8];
#pragma unroll
    for (int u = 0; u < PL; ++u)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[u][j] = 0.f;
    for (int k0 = 0; k0 < a.topk; k0 += 32) {
      // lanes read the token's routing slots in parallel, then the warp walks only the local ones
      const int k = k0 + lane;
      const int my_pos = k < a.topk ? a.pair_pos[(long long)t * a.topk + k] : -1;
      uint32_t have = __ballot_sync(0xffffffffu, my_pos >= 0);
      while (have) {
        uint4 v[R][PL];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool live = have != 0;
          const int pos = __shfl_sync(0xffffffffu, my_pos, live ? __ffs(have) - 1 : 0);
          have &= have - 1;
#pragma unroll
          for (int u = 0; u < PL; ++u) {
            const int p = p0 + u * 32;
            const uint8_t* at = y + (uint64_t)pos * s.row_bytes + (uint64_t)p * 16;
            v[r][u] = live && p < s.packs ? (PL == 4 && ALONE ? ld_v4(at) : ld_v4_stream(at)) : make_uint4(0, 0, 0, 0);
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int u = 0; u < PL; ++u) acc_row(acc[u], v[r][u]);
      }
    }
    if (alone && (t < s.offset || t >= s.offset + s.n)) continue;
    uint8_t* dst = alone ? out + (uint64_t)(t - s.offset) * s.row_bytes : partial + (uint64_t)t * s.row_bytes;
#pragma unroll
    for (int u = 0; u < PL; ++u) {
      const int p = p0 + u * 32;
      if (p < s.packs)
        st_v4(dst + (uint64_t)p * 16, make_uint4(pack_bf16x2(acc[u][0], acc[u][1]), pack_bf16x2(acc[u][2], acc[u][3]),
                                                 pack_bf16x2(acc[u][4], acc[u][5]), pack_bf16x2(acc[u][6], acc[u][7])));
    }
  }
  if (alone) return;
  block_barrier_all(c, a.site, bid, ep);
  for (long long i = first; i < items; i += step) {
    const int t = (int)(i / s.slices);
    if (t < s.offset || t >= s.offset + s.n) continue;
    const int p0 = (int)(i - (long long)t * s.slices) * 32 * PL + lane;
    uint4 v[PL];
#pragma unroll
    for (int u = 0; u < PL; ++u)
      if (p0 + u * 32 < s.packs)
        v[u] = combine_reduce_pack(c, s.partial_off + (uint64_t)t * s.row_bytes + (uint64_t)(p0 + u * 32) * 16);
#pragma unroll
    for (int u = 0; u < PL; ++u)
      if (p0 + u * 32 < s.packs) st_v4(out + (uint64_t)(t - s.offset) * s.row_bytes + (uint64_t)(p0 + u * 32) * 16, v[u]);
  }
}

// The sums of a launch of its own in a world of one (combine_alone_kernel), where rows allow packs of 32 bytes: a warp takes 32 packs of BYTES of
// a row, R pair rows in flight.  As long as every slice of 512 bytes has a warp of its own, latency is the limit: packs of 16 bytes, eight rows.
// Beyond that the rate of loads from L2 is, which for 32 bytes per lane is twice that for 16 (copies of 16 MB, 16.4 against 8.2 TB/s), and the warps:
// without the buffers of the sums over ranks the kernel has two blocks per SM.  One B200, us a launch in a row of them, before (one block per SM,
// slices of 512, 1024 and 2048 bytes of 16 per lane) -> now, an eighth of 512 experts, rows of 1024 values:
//   64 / 1024 / 2048 / 4096 / 8191 tokens of top-22, 2.75 pairs each   2.7 / 4.4 / 5.0 / 7.1 / 10.9 -> 2.3 / 3.7 / 4.1 / 5.6 / 8.9
//   half of the experts, 512 / 2000 / 4096 tokens, 11 pairs each       4.5 / 10.6 / 20.8 -> 3.7 / 6.4 / 14.1
//   8 of 64 experts, rows of 7168, 64 / 512 / 4096 tokens of top-8     3.9 / 6.4 / 29.2 -> 3.2 / 4.8 / 24.3
// One row in flight instead of two 5.6 -> 6.5 (4096 tokens), three the same, four 6.0; three blocks per SM 6.8; 16 bytes per lane throughout 7.5.
template <int BYTES, int R>
__device__ __forceinline__ void combine_alone_items(const McbCombineArgs& a, int begin, int end, int offset) {
  static_assert(BYTES == 16 || BYTES == 32, "a pack");
  using Pack = typename std::conditional<BYTES == 32, Pack32, uint4>::type;
  const int lane = threadIdx.x & 31, row_bytes = a.hidden * 2, slices = (row_bytes + 32 * BYTES - 1) / (32 * BYTES);
  const long long items = (long long)(end - begin) * slices, step = (long long)gridDim.x * (blockDim.x >> 5);
  const uint8_t* y = reinterpret_cast<const uint8_t*>(a.y);
  uint8_t* out = reinterpret_cast<uint8_t*>(a.out);
  for (long long i = blockIdx.x + (long long)(threadIdx.x >> 5) * gridDim.x; i < items; i += step) {
    const int t = (int)(i / slices), at = ((int)(i - (long long)t * slices) * 32 + lane) * BYTES;
    const bool live = at < row_bytes;
    float acc[BYTES / 16][8] = {};
    for (int k0 = 0; k0 < a.topk; k0 += 32) {
      const int k = k0 + lane;
      const int my_pos = k < a.topk ? a.pair_pos[(long long)(begin + t) * a.topk + k] : -1;
      uint32_t have = __ballot_sync(0xffffffffu, my_pos >= 0);
      while (have) {
        Pack v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool row = have != 0;
          const int pos = __shfl_sync(0xffffffffu, my_pos, row ? __ffs(have) - 1 : 0);
          have &= have - 1;
          const uint8_t* p = y + (long long)pos * row_bytes + at;
          if constexpr (BYTES == 32) v[r] = row && live ? ld_v8_stream(p) : Pack32{};
          else v[r] = row && live ? ld_v4_stream(p) : uint4{};
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if constexpr (BYTES == 32) { acc_row(acc[0], v[r].lo); acc_row(acc[1], v[r].hi); }
          else acc_row(acc[0], v[r]);
        }
      }
    }
    if (!live) continue;
    uint8_t* dst = out + (long long)(begin + t - offset) * row_bytes + at;
    auto packed = [](const float (&s)[8]) {
      return make_uint4(pack_bf16x2(s[0], s[1]), pack_bf16x2(s[2], s[3]), pack_bf16x2(s[4], s[5]), pack_bf16x2(s[6], s[7]));
    };
    if constexpr (BYTES == 32) st_v8(dst, Pack32{packed(acc[0]), packed(acc[1])});
    else st_v4(dst, packed(acc[0]));
  }
}

template <bool ALONE>
__device__ __forceinline__ void combine_body(const McbCtx& c, const McbCombineArgs& a, uint32_t parity = 0u, int warp = threadIdx.x >> 5,
                                             int nwarps = blockDim.x >> 5) {
  CombineShape s;
  s.T = a.step_meta[0];
  s.offset = a.step_meta[1];
  s.n = *a.n_local;
  if (s.n < 0) s.n = 0;
  if (s.n > a.cap) s.n = a.cap;
  if (s.T <= 0) return;
  s.packs = a.hidden / 8;
  s.row_bytes = (uint64_t)a.hidden * 2;
  s.partial_off = a.partial_off + (uint64_t)(parity & 1u) * a.partial_par_stride;
  // Packs per lane from sizes that are the same on every rank.
  const long long warps = (long long)gridDim.x * nwarps;
  int pl = 4;
  while (pl > 1 && (long long)s.T * ((s.packs + 32 * pl - 1) / (32 * pl)) < warps) pl >>= 1;
  s.slices = (s.packs + 32 * pl - 1) / (32 * pl);
  const long long items = (long long)s.T * s.slices;
  s.nact = items < (long long)gridDim.x ? (int)items : (int)gridDim.x;
  if ((int)blockIdx.x >= s.nact) return;
  const uint32_t ep = *epoch_ptr(c, a.site, blockIdx.x);
  if (pl == 4) combine_items<4, ALONE>(c, a, s, ep, warp, nwarps);
  else if (pl == 2) combine_items<2, ALONE>(c, a, s, ep, warp, nwarps);
  else combine_items<1, ALONE>(c, a, s, ep, warp, nwarps);
}

}  // namespace mcb
