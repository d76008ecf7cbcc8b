// One whole decode step of the dense dispatcher as ONE persistent kernel for sm_100a.
//
// The reference issues a step as 1 + 2 * 88 kernels (bench_nvls.py:114-121: metadata once, then
// per layer an all-gather-V with a trailing cross-GPU barrier and a reduce-scatter-V with a leading
// one, variable_collectives.py:142-150, 209-219).  Here the whole step is one launch:
//
//   count exchange      block 0 publishes this rank's row count to every rank; every block of
//                       every rank waits for all counts.  Because a rank only publishes after its
//                       previous kernel has finished, passing this point also proves that every
//                       rank has left the previous step: nothing written now can race with it.
//   barrier mode        per layer: push my share of the local rows into the gathered buffers of
//                       every rank (multimem.st, or peer stores), ONE block-matched release barrier,
//                       then the switch-side reduction (multimem.ld_reduce, or peer loads) of the
//                       rows this rank owns.  The gathered buffers are double-buffered by layer
//                       parity, so the barrier of layer l is also the write-after-read fence that
//                       protects the readers of layer l - 1.
//   pipeline groups     optionally the blocks are split into G groups, each owning 1/G of every
//                       rank's rows.  A group's chain push -> barrier -> reduce is unchanged, but
//                       the groups take turns on the push, so one group's reduction (which loads
//                       the outbound direction of every link) runs while the next group's push
//                       fills the inbound direction.  Dependencies are per row: a row is reduced
//                       only after it was gathered everywhere, and pushed for the next layer only
//                       after it was reduced.
//   packet mode         small steps: rows travel as 16-byte {data, flag, data, flag} packets that
//                       the receiver polls, so a layer needs no barrier and no fence.  A packet is
//                       written and read by the same block index on every rank, and after each
//                       layer a block publishes "I have finished reading layer l" in a word of its
//                       own on every rank (one word per (block, source rank): a sum over ranks
//                       could not tell a slow rank from fast ones that ran ahead); a block re-uses
//                       a staging area (two parities) only when every rank's word has reached the
//                       layer that used it last.
//
// All per-step sizes are read from device memory, so one captured launch serves every batch.
// Every wait is bounded and reports through the status words.
//
// FP8 = true dispatches the hidden rows as 1 x 128 block-scaled e4m3 (BASELINE configuration of the
// DeepSeek-V3 shape): tensor 0's source is bf16 [cap, hidden], its gathered form is one byte per value,
// and tensor 3 is the gathered fp32 scales [rows, hidden / 128], produced here; quantisation happens
// inside the push (barrier mode: 16 neighbouring threads share a block and agree on its largest
// magnitude with shuffles; packet mode: every thread scans the 256 bytes of its block itself).
//
// CHECK = true is the self-checking build used by the race tests: the pushed payload is not the
// input rows but a hash of (layer sequence number, position), every receiver verifies the words
// it is entitled to read right after its barrier (or packet poll) and counts mismatches, and a
// rank can be slowed down by a bounded sleep per layer chosen on the host.  A write that
// arrives too early (a broken write-after-read fence) or too late then shows up as a mismatch
// instead of being invisible because consecutive layers carry identical bytes.
#include <cuda_runtime.h>

#include <climits>
#include <type_traits>

#include "mcb_barrier.cuh"
#include "mcb_dense.cuh"
#include "mcb_fp8.cuh"
#include "mcb_launch.h"
#include "mcb_launchers.h"
#include "mcb_step.cuh"

namespace mcb {

struct StepShape {
  int w[MCB_MAX_TENSORS];   // 8-byte words per row of each gathered tensor
  int wpr;                  // their sum
};

// Which tensor and which word of its row is word `jj` of a gathered row.
__device__ __forceinline__ void split_word(const StepShape& s, int jj, int& t, int& j) {
  t = 0;
  j = jj;
#pragma unroll
  for (int k = 0; k < MCB_MAX_TENSORS - 1; ++k)
    if (t == k && j >= s.w[k]) { j -= s.w[k]; t = k + 1; }
}

__device__ __forceinline__ uint32_t check_word(uint32_t seq, uint32_t tensor, uint32_t index) {
  uint32_t h = (seq + 1u) * 0x9E3779B1u ^ (index + 0x7F4A7C15u) * 0x85EBCA77u ^ (tensor + 1u) * 0xC2B2AE3Du;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  return h ^ (h >> 13);
}

__device__ __forceinline__ void check_fail(const McbDenseStepArgs& a) {
  if (a.check_errors) atomicAdd(a.check_errors, 1u);
}

// Packet all-gather of one layer.  Slot i = (global row) * wpr + word is sent by thread
// (i mod nthreads) of the row's owner and read by the same thread index on every rank.
// The 8 payload bytes of word j of gathered tensor t of local row `row` when the hidden rows are
// quantised on the way out: 8 e4m3 values (t == 0) or two fp32 scales (t == 3).
__device__ __forceinline__ uint2 fp8_word(const McbDenseStepArgs& a, int row, int t, int j) {
  const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src[0]) + (uint64_t)row * a.fp8_hidden * 2;
  if (t == 0) {
    const float scale = e4m3_scale(block_absmax_serial(src + (uint64_t)(j >> 4) * 256));
    return quant_pack_e4m3(ld_v4(src + (uint64_t)j * 16), scale);
  }
  return make_uint2(__float_as_uint(e4m3_scale(block_absmax_serial(src + (uint64_t)(2 * j) * 256))),
                    __float_as_uint(e4m3_scale(block_absmax_serial(src + (uint64_t)(2 * j + 1) * 256))));
}

template <bool CHECK, bool FP8>
__device__ __forceinline__ void step_agv_ll(const McbCtx& c, const McbDenseStepArgs& a, const StepShape& s,
                                            int n, int offset, int valid, uint32_t flag, uint32_t par,
                                            uint32_t seq, long long gtid, long long nthreads) {
  const uint64_t stage = a.agv_ll_off + (uint64_t)(flag & 1u) * a.ll_rows * s.wpr * 16;
  const long long lo = (long long)offset * s.wpr, hi = (long long)(offset + n) * s.wpr;
  long long first = lo + ((gtid - lo) % nthreads + nthreads) % nthreads;
  for (long long i0 = first; i0 < hi; i0 += nthreads * 4) {
    uint2 d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * nthreads;
      if (i < hi) {
        const int row = (int)(i / s.wpr);
        int t, j;
        split_word(s, (int)(i - (long long)row * s.wpr), t, j);
        if (FP8 && (t == 0 || t == 3)) d[u] = fp8_word(a, row - offset, t, j);
        else
        d[u] = CHECK ? make_uint2(check_word(seq, 0u, (uint32_t)i * 2u), check_word(seq, 0u, (uint32_t)i * 2u + 1u))
                     : ld_v2(reinterpret_cast<const uint8_t*>(a.src[t]) + (uint64_t)(row - offset) * a.row_bytes[t] +
                             (uint64_t)j * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * nthreads;
      if (i >= hi) break;
      const uint4 pkt = ll_pack(d[u], flag);
      const uint64_t off = stage + (uint64_t)i * 16;
      if (c.transport == MCB_TRANSPORT_MULTIMEM) {
        mm_st_v4(c.heap_mc + off, pkt);
      } else {
        for (int k = 0; k < c.world; ++k) {
          int p = c.rank + 1 + k;
          if (p >= c.world) p -= c.world;
          st_v4(c.heap_peer[p] + off, pkt);
        }
      }
    }
  }
  const long long nrecv = (long long)valid * s.wpr;
  for (long long i0 = gtid; i0 < nrecv; i0 += nthreads * 4) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * nthreads;
      if (i < nrecv) v[u] = ld_v4_volatile(c.heap_local + stage + (uint64_t)i * 16);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * nthreads;
      if (i >= nrecv) break;
      uint2 d = make_uint2(v[u].x, v[u].z);
      if (v[u].y != flag || v[u].w != flag)
        d = ll_wait(c, c.heap_local + stage + (uint64_t)i * 16, flag, MCB_SITE_STEP);
      if (CHECK && (d.x != check_word(seq, 0u, (uint32_t)i * 2u) || d.y != check_word(seq, 0u, (uint32_t)i * 2u + 1u)))
        check_fail(a);
      const int row = (int)(i / s.wpr);
      int t, j;
      split_word(s, (int)(i - (long long)row * s.wpr), t, j);
      st_v2(c.heap_local + a.dst_off[t] + (uint64_t)par * a.dst_par_stride[t] + (uint64_t)row * a.row_bytes[t] +
                (uint64_t)j * 8, d);
    }
  }
}

// Packet reduce-scatter of one layer (bf16).  Word i of owner o's rows is sent by thread
// (i mod nthreads) of every rank and summed, in rank order in fp32, by the same thread index of o.
__device__ __forceinline__ void step_rsv_ll(const McbCtx& c, const McbDenseStepArgs& a, const int* s_prefix,
                                            int n, int ep_max, uint32_t flag, long long gtid, long long nthreads) {
  const int wpr = (int)(a.rsv_row_bytes >> 3);
  const uint64_t per_src = (uint64_t)a.ll_src_rows * wpr * 16;
  const uint64_t stage = a.rsv_ll_off + (uint64_t)(flag & 1u) * c.world * per_src;
  const uint8_t* mine = c.heap_local + a.rsv_off;
  const uint64_t my_region = stage + (uint64_t)c.rank * per_src;
  for (long long i = gtid; i < (long long)ep_max * wpr; i += nthreads) {
    for (int o0 = 0; o0 < c.world; o0 += 4) {
      uint2 d[4];
      bool live[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int o = o0 + u;
        live[u] = o < c.world && i < (long long)(s_prefix[o + 1] - s_prefix[o]) * wpr;
        if (live[u]) d[u] = ld_v2(mine + ((uint64_t)s_prefix[o] * wpr + (uint64_t)i) * 8);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (live[u]) st_v4(c.heap_peer[o0 + u] + my_region + (uint64_t)i * 16, ll_pack(d[u], flag));
    }
  }
  uint8_t* out = reinterpret_cast<uint8_t*>(a.out);
  for (long long i = gtid; i < (long long)n * wpr; i += nthreads) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const uint8_t* slot0 = c.heap_local + stage + (uint64_t)i * 16;
    for (int s0 = 0; s0 < c.world; s0 += 4) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (s0 + u < c.world) v[u] = ld_v4_volatile(slot0 + (uint64_t)(s0 + u) * per_src);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (s0 + u >= c.world) break;
        uint2 d = make_uint2(v[u].x, v[u].z);
        if (v[u].y != flag || v[u].w != flag)
          d = ll_wait(c, slot0 + (uint64_t)(s0 + u) * per_src, flag, MCB_SITE_STEP);
        acc[0] += bf16_lo(d.x); acc[1] += bf16_hi(d.x);
        acc[2] += bf16_lo(d.y); acc[3] += bf16_hi(d.y);
      }
    }
    st_v2(out + (uint64_t)i * 8, make_uint2(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3])));
  }
}

// Self-checking push of one tensor's share (4-byte words) and its verification after the barrier.
__device__ __forceinline__ void check_push(const McbCtx& c, uint64_t dst_off, uint32_t tensor, uint32_t seq,
                                           long long first_word, long long nwords, long long start, long long stride) {
  for (long long i = start; i < nwords; i += stride) {
    const uint32_t v = check_word(seq, tensor, (uint32_t)(first_word + i));
    const uint64_t off = dst_off + (uint64_t)(first_word + i) * 4;
    if (c.transport == MCB_TRANSPORT_MULTIMEM) {
      mm_st_b32(c.heap_mc + off, v);
    } else {
      for (int k = 0; k < c.world; ++k) {
        int p = c.rank + 1 + k;
        if (p >= c.world) p -= c.world;
        st_b32(c.heap_peer[p] + off, v);
      }
    }
  }
}
__device__ __forceinline__ void check_verify(const McbCtx& c, const McbDenseStepArgs& a, uint64_t dst_off,
                                             uint32_t tensor, uint32_t seq, long long first_word, long long nwords,
                                             long long start, long long stride) {
  for (long long i = start; i < nwords; i += stride)
    if (ld_relaxed_sys(c.heap_local + dst_off + (uint64_t)(first_word + i) * 4) !=
        check_word(seq, tensor, (uint32_t)(first_word + i)))
      check_fail(a);
}

// Barrier-mode push of the quantised hidden rows [r0, r1) of this rank and of their scales.  Packs
// (16 bytes of bf16 = 8 values) are dealt to threads in order, so the 16 lanes of a half warp hold one
// 128-value block.  Call from all threads of the block (whole warps take part in the shuffles).
template <bool ALONE = false>
__device__ __forceinline__ void fp8_push(const McbCtx& c, const McbDenseStepArgs& a, uint32_t par, int offset, int r0,
                                         int r1, long long start, long long stride) {
  const int H = (int)a.fp8_hidden, ppr = H / 8, nblk = H / 128;
  const long long total = (long long)(r1 - r0) * ppr;              // a multiple of 16
  const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src[0]) + (uint64_t)r0 * H * 2;
  const uint64_t q_off = a.dst_off[0] + (uint64_t)par * a.dst_par_stride[0] + (uint64_t)(offset + r0) * H;
  const uint64_t s_off = a.dst_off[3] + (uint64_t)par * a.dst_par_stride[3] + (uint64_t)(offset + r0) * nblk * 4;
  const long long warp_start = start - (threadIdx.x & 31);
  constexpr int U = 4;                                             // packs in flight per thread
  for (long long base = warp_start; base < total; base += stride * U) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = base + u * stride + (threadIdx.x & 31);
      v[u] = i < total ? ld_v4_stream(src + i * 16) : make_uint4(0, 0, 0, 0);
    }
    float amax[U];
#pragma unroll
    for (int u = 0; u < U; u += 2) block_absmax_pair(v[u], v[u + 1], amax[u], amax[u + 1]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = base + u * stride + (threadIdx.x & 31);
      if (i >= total) continue;
      const float scale = e4m3_scale(amax[u]);
      const uint2 q = quant_pack_e4m3(v[u], scale);
      const long long row = total >> 32 ? i / ppr : (long long)((uint32_t)i / (uint32_t)ppr);
      const int pk = (int)(i - row * ppr);
      const uint64_t qo = q_off + (uint64_t)row * H + (uint64_t)pk * 8;
      const uint64_t so = s_off + ((uint64_t)row * nblk + (pk >> 4)) * 4;
      if (ALONE) {
        st_v2(c.heap_local + qo, q);
        if ((pk & 15) == 0) st_b32(c.heap_local + so, __float_as_uint(scale));
      } else if (c.transport == MCB_TRANSPORT_MULTIMEM) {
        mm_st_v2(c.heap_mc + qo, q);
        if ((pk & 15) == 0) mm_st_b32(c.heap_mc + so, __float_as_uint(scale));
      } else {
        for (int k = 0; k < c.world; ++k) {
          int p = c.rank + 1 + k;
          if (p >= c.world) p -= c.world;
          st_v2(c.heap_peer[p] + qo, q);
          if ((pk & 15) == 0) st_b32(c.heap_peer[p] + so, __float_as_uint(scale));
        }
      }
    }
  }
}

// ---- a world of one: the layers of a step are local copies ------------------------------------------------------
// What a layer copies; quantised values and scales are pushed on their own.  All threads of the block.
template <bool FP8>
__device__ __forceinline__ void local_ranges(LocalRanges& r, const McbCtx& c, const McbDenseStepArgs& a, int n) {
  constexpr int R = LocalRanges::R;
  if (threadIdx.x == 0) {
    for (int t = 0; t < R - 1; ++t) {
      const bool used = t < a.num_tensors && !(FP8 && (t == 0 || t == 3));
      r.set(t, a.src[t], c.heap_local + a.dst_off[t], a.dst_par_stride[t], used ? (long long)n * a.row_bytes[t] : 0);
    }
    r.set(R - 1, c.heap_local + a.rsv_off, reinterpret_cast<uint8_t*>(a.out), 0, (long long)n * a.rsv_row_bytes);
  }
  __syncthreads();
}

// Layers [first, last) of one pack per lane, the loads of eight of them in flight together, and the stores of one parity before those of the other: they
// go to the same place, and more of them merge in L1 than in the order of the layers.  One B200, us a step: 88 layers of 1000 / 6000 rows of 1024 42.8 / 212 ->
// 38.6 / 180, 58 layers of 333 / 1000 rows of 7168 57.0 / 144 -> 51.2 / 133, 60 rows or fewer up to 5 % faster or the same.  (One parity of a whole run
// before the other: large steps another 0 to 3 % faster, those of up to 60 rows 2 to 10 % slower.  e4m3 rows, which alternate, and all-to-all pieces did not
// gain.)
template <class Load, class Store>
__device__ __forceinline__ void local_layers_of(int first, int last, Load load, Store store) {
  constexpr int D = 8;
  for (int l0 = first; l0 < last; l0 += D) {
    uint4 v[D];
#pragma unroll
    for (int d = 0; d < D; ++d) v[d] = l0 + d < last ? load() : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int d = p; d < D; d += 2) store(v[d], l0 + d < last, l0 + p);
  }
}

// Nothing that a layer reads is written in the step (else: a.in_order), and all layers of a parity deliver the same rows, so the layers
// need no order: a warp takes all layers of a few packs, and every warp gets the same number of (pack, layer) whatever the batch.  The
// chip works on a few MB at a time; layer after layer over all rows, large steps went through up to 90 MB of L2 in every layer, small ones
// left most of the chip idle, and sizes just above a whole number of packs per thread paid for the next one.
// The loads may stay in L1, where 95 % of their sectors hit (24 layers of 2048 rows): large steps are bound by the stores that L1 has to
// take and pass on, and loads with the hint that keeps them out of L1 made 88 layers of 1000 to 8192 rows of 1024 20 to 25 % slower.
// One B200, 58 layers, layer after layer (local_in_order) -> dealt, 1 / 37 / 333 / 2048 rows, us a step:
//   1024 values  bf16 92 -> 4.2 / 109 -> 5.4 / 110 -> 20 / 131 -> 47     e4m3 114 -> 5.3 / 128 -> 7.3 / 130 -> 17.6 / 199 -> 61
//   7168 values  bf16 98 -> 4.3 / 100 -> 11.5 / 128 -> 51 / 956 -> 274   e4m3 120 -> 5.6 / 121 -> 12.2 / 197 -> 67 / 1085 -> 373
// Sixteen layers in flight, or the loads of the next eight ahead of the stores, were 6 to 15 % slower.
// Copies of many layers with enough for every warp go by half of the warps: a layer's stores merge in L1 with earlier ones to the same rows, if these are still
// there (of 26.8 million sectors stored by 24 layers of 8192 rows in the order of the layers 14.2 million went on to L2 with 16 warps per block and 10.8 million
// with 8).  With fewer items a warp the time until a run's first load is there counts for more, and with many groups and fewer layers the rate of the warps.
// One B200, all warps -> half of them, us a step (in brackets: (group, layer) items, groups for each of all warps):
//   88 layers  1024 values, 60 rows (19) 6.0 -> 7.0, 150 (48) 10.7 -> 13.6, 1000 (317) 40.9 -> 38.9, 8192 (2593) 243 -> 238;  7168 values, 60 (125) 20.2 -> 19.7,
//              2048 (4276) 393 -> 388
//   58 layers  1024 values, 150 (31) 7.8 -> 9.8, 1000 (209) 28.0 -> 27.2, 8192 (1709, 29) 163 -> 166;  7168 values, 60 (83) 15.0 -> 14.6, 400 (551, 9) 58.6 -> 56.9,
//              1000 (1376, 24) 133.8 -> 133.6, 2048 (2819, 49) 264 -> 275
//   40 layers  7168 values, 60 (57) 10.5 -> 10.3, 400 (380, 9) 40.7 -> 39.9, 1000 (949, 24) 92.1 -> 94.8;  2048 values, 2048 rows (560, 14) 56.4 -> 56.3, 8192 (56) 211 -> 228
//   32 layers  1024 values, 1000 rows (115) 16.2 -> 16.0, 2048 (236) 26.6 -> 27.0;  26 layers 23.3 -> 24.5
constexpr int kHalfLayers = 40, kHalfItems = 64, kHalfAlways = 64, kHalfGroups = 20;

template <bool FP8>
__device__ __forceinline__ void local_dealt(const McbCtx& c, const McbDenseStepArgs& a, const LocalRanges& r, int n, uint32_t layer_base) {
  const long long packs = r.end[LocalRanges::R - 1], groups = (packs + 31) >> 5;
  int used = (int)(blockDim.x >> 5);                                            // warps of a block that take part
  const int most = a.num_layers >= kHalfAlways ? INT_MAX : kHalfGroups * used * (int)gridDim.x;
  if (!FP8 && a.num_layers >= kHalfLayers && (groups + 1) * a.num_layers >= (long long)kHalfItems * used * gridDim.x && groups <= most) used = (used + 1) / 2;
  if ((int)(threadIdx.x >> 5) >= used) return;
  const int lane = threadIdx.x & 31, warps = (int)gridDim.x * used;
  const int warp = (int)(blockIdx.x + (threadIdx.x >> 5) * gridDim.x);         // the smallest steps spread over the chip
  auto quantise = [&] {
    // Two packs (16 values) per lane, so eight lanes hold a block of 128 values and a lane stores 16 bytes: 13 to 18 % faster than one.
    const int H = (int)a.fp8_hidden, ppr = H / 16, nblk = H / 128;
    const long long total = (long long)n * ppr;                // a multiple of 8
    local_share((total + 31) >> 5, a.num_layers, warp, warps, [&](long long g, int first, int last) {
      const long long i = g * 32 + lane;
      const bool live = i < total;
      const int row = (int)(i / ppr), pk = (int)(i - (long long)row * ppr);
      const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src[0]) + i * 32;
      uint8_t* q_dst = c.heap_local + a.dst_off[0] + (uint64_t)row * H + (uint64_t)pk * 16;
      uint8_t* s_dst = c.heap_local + a.dst_off[3] + ((uint64_t)row * nblk + (pk >> 3)) * 4;
      constexpr int D = 4;
      for (int l0 = first; l0 < last; l0 += D) {
        uint4 v[D][2];
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
          for (int k = 0; k < 2; ++k) v[d][k] = live && l0 + d < last ? ld_v4(src + k * 16) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int d = 0; d < D; d += 2)
          quant_wide_pair(v[d], v[d + 1], [&](int k) { return live && l0 + d + k < last; }, [&](int k, uint4 q, float scale) {
            const uint32_t par = (layer_base + (uint32_t)(l0 + d + k)) & 1u;
            st_v4(q_dst + (par ? a.dst_par_stride[0] : 0), q);
            if ((lane & 7) == 0) st_b32(s_dst + (par ? a.dst_par_stride[3] : 0), __float_as_uint(scale));
          });
      }
    });
  };
  auto copy = [&] {
    const int from = FP8 ? (warp + warps / 2) % warps : warp;       // small steps: not the warps that quantise
    // The group behind the last one: the words behind the last whole pack of each range.
    local_share(groups + 1, a.num_layers, from, warps, [&](long long g, int first, int last) {
      if (g == groups) {
        for (int l0 = first; l0 < last; l0 += 8) {
          uint32_t w[8];
#pragma unroll
          for (int d = 0; d < 8; ++d) w[d] = l0 + d < last ? r.load_word(lane, 0) : 0u;
#pragma unroll
          for (int d = 0; d < 8; ++d)
            if (l0 + d < last) r.store_word((layer_base + (uint32_t)(l0 + d)) & 1u, w[d], lane, 0);
        }
        return;
      }
      const long long i = g * 32 + lane;
      const bool live = i < packs;
      long long off = 0;
      const int t = live ? r.find(i, off) : 0;
      const uint8_t* src = r.src[t] + off;
      uint8_t* dst = r.dst[t] + off;
      const uint64_t par_off = r.par[t];
      local_layers_of(first, last, [&] { return live ? ld_v4(src) : make_uint4(0, 0, 0, 0); },
                      [&](uint4 v, bool on, int l) {
        const uint32_t par = (layer_base + (uint32_t)l) & 1u;
        if (live && on) st_v4(dst + (par ? par_off : 0), v);
      });
    });
  };
  if (!FP8) { copy(); return; }
  // Half of the warps of an SM quantise while the others copy: 5 to 10 % faster than all of them in step.
  const int odd = (int)(threadIdx.x >> 5) & 1;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    if (k == odd) quantise();
    else copy();
  }
}

// A step of up to this many layers has too few of one group of packs to keep loads in flight: there a warp takes all layers of 8 / D groups
// at a time, D = 1, 2, 4 or 8 the layers that it may have.  The groups go round the warps, so no warp divides.  Kernels of their own:
// with both ways in one, the large steps of many layers were 3 to 7 % slower and every step 0.5 to 1 us.
// One B200, a step of 1 / 2 / 4 / 8 layers in a row of steps, dealt in runs -> this way:
//   hidden 1024 and top-22, 64 rows     bf16 4.0 / 4.0 / 3.9 / 4.6 -> 3.8 / 3.6 / 3.3 / 3.6          e4m3 5.6 / 5.8 / 6.0 / 6.1 -> 4.2 / 4.3 / 4.6 / 5.7 us
//                          512 rows     bf16 4.8 / 5.3 / 5.3 / 5.6 -> 4.1 / 4.0 / 4.1 / 4.8          e4m3 5.9 / 6.9 / 7.8 / 8.2 -> 4.6 / 4.9 / 5.3 / 6.4
//                          8192 rows    bf16 29.9 / 33.2 / 33.2 / 35.2 -> 11.8 / 16.1 / 19.5 / 28.5  e4m3 23.6 / 26.4 / 30.5 / 41.9 -> 11.0 / 14.6 / 22.5 / 38.3
//   hidden 7168 and top-8, 2048 rows    bf16 54 / 57 / 57 / 59 -> 20.3 / 29.5 / 35.2 / 49.7          e4m3 41.5 / 46.3 / 52.7 / 70.7 -> 17.6 / 28.6 / 42.0 / 68.4
// Nine to sixteen layers by rounds of eight were up to 25 % slower than runs with bf16 rows and 10 % either way with e4m3 rows, so the line is at one round.
// Stores to one place one after the other instead of layer by layer: 2 / 4 / 8 layers of 333 rows of 7168 6.7 / 8.8 / 10.4 -> 6.1 / 7.3 / 9.4.
constexpr int kFewLayers = 8;

template <bool FP8, int D>
__device__ __forceinline__ void local_few(const McbCtx& c, const McbDenseStepArgs& a, const LocalRanges& r, int n, uint32_t layer_base) {
  constexpr int S = 8 / D, Q = D < 4 ? 4 : D, SQ = Q / D;
  if (a.num_layers < 1) return;
  const int lane = threadIdx.x & 31, warps = (int)(gridDim.x * (blockDim.x >> 5)), L = a.num_layers;
  const long long packs = r.end[LocalRanges::R - 1], groups = (packs + 31) >> 5;
  const int warp = (int)(blockIdx.x + (threadIdx.x >> 5) * gridDim.x);         // the smallest steps spread over the chip
  auto parity = [&](int l) { return (layer_base + (uint32_t)l) & 1u; };
  int from = warp;
  if (FP8) {
    // Rows to quantise: two packs (16 values) per lane, eight lanes a block of 128 values.  Rows follow one another in the input and where
    // they go: lane i of all reads at 32 i and stores at 16 i.
    const long long halves = (long long)n * (a.fp8_hidden / 16), quants = (halves + 31) >> 5;
    const uint8_t* rows = reinterpret_cast<const uint8_t*>(a.src[0]);
    uint8_t *q_dst = c.heap_local + a.dst_off[0], *s_dst = c.heap_local + a.dst_off[3];
    for (long long g = warp; g < quants; g += (long long)warps * SQ) {
      uint4 v[Q][2];
      long long i[Q];
#pragma unroll
      for (int d = 0; d < Q; ++d) {
        i[d] = (g + d / D * warps) * 32 + lane;
        const bool on = i[d] < halves && d % D < L;
#pragma unroll
        for (int k = 0; k < 2; ++k) v[d][k] = on ? ld_v4(rows + i[d] * 32 + k * 16) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int d = 0; d < Q; d += 2) {
        if (g + d / D * warps >= quants || d % D >= L) break;
        quant_wide_pair(v[d], v[d + 1], [&](int k) { return i[d + k] < halves && (d + k) % D < L; }, [&](int k, uint4 q, float scale) {
          const int at = d + k, l = at % D;
          st_v4(q_dst + i[at] * 16 + (parity(l) ? a.dst_par_stride[0] : 0), q);
          if ((lane & 7) == 0) st_b32(s_dst + (i[at] >> 3) * 4 + (parity(l) ? a.dst_par_stride[3] : 0), __float_as_uint(scale));
        });
      }
    }
    from = (warp + warps - (int)(quants % warps)) % warps;      // those that quantise one group more come last
  }
  if constexpr (D == 1) {
    copy_ranges(r, parity(0), (long long)from * 32 + lane, (long long)warps * 32);
    return;
  }
  for (long long g = from; g < groups; g += (long long)warps * S) {
    uint4 v[S][D];
    uint8_t* dst[S];
    uint64_t par_off[S];
#pragma unroll
    for (int u = 0; u < S; ++u) {
      const long long i = (g + u * warps) * 32 + lane;
      dst[u] = nullptr;
      if (i < packs) {
        long long off;
        const int t = r.find(i, off);
        dst[u] = r.dst[t] + off;
        par_off[u] = r.par[t];
#pragma unroll
        for (int d = 0; d < D; ++d)
          if (d < L) v[u][d] = ld_v4(r.src[t] + off);
      }
    }
    // Stores to one place one after the other, where they merge in L1.
#pragma unroll
    for (int u = 0; u < S; ++u)
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int d = p; d < D; d += 2)
          if (d < L && dst[u]) st_v4(dst[u] + (parity(p) ? par_off[u] : 0), v[u][d]);
  }
  // The words behind the last whole pack of each range.
  if (warp == warps - 1) {
    uint32_t w[D];
#pragma unroll
    for (int d = 0; d < D; ++d) w[d] = d < L ? r.load_word(lane, 0) : 0u;
#pragma unroll
    for (int d = 0; d < D; ++d)
      if (d < L) r.store_word(parity(d), w[d], lane, 0);
  }
}

// Layer after layer: steps that read what they write.  `nact`: blocks that a layer fills.  FEW: as in copy_ranges_in_order.  In a kernel of its own a layer
// of few rows is a chain of a load and a store for each range, and what stands between them counts: 58 layers of 1 / 37 / 333 rows of 1024 in the kernel of
// dealt steps 97 / 115 / 120 us, on their own 95 / 121 / 127, with FEW 92 / 109 / 110; e4m3 130 / 155 / 161, 126 / 147 / 152, 114 / 128 / 130.  2048 rows of
// 7168 952, 955, 956 (with FEW there too 976).  The line: three packs of the expert outputs for a thread.
template <bool FP8, bool FEW = false>
__device__ __forceinline__ void local_in_order(const McbCtx& c, const McbDenseStepArgs& a, const LocalRanges& r, int n, int nact, uint32_t layer_base) {
  if ((int)blockIdx.x >= nact) return;
  const long long start = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)nact * blockDim.x;
  for (int l = 0; l < a.num_layers; ++l) {
    const uint32_t par = (layer_base + (uint32_t)l) & 1u;
    if (FP8) fp8_push<true>(c, a, par, 0, 0, n, start, stride);
    copy_ranges_in_order<FEW>(r, par, start, stride);
  }
}

template <bool EMU, bool CHECK, bool FP8>
__global__ void __launch_bounds__(512) dense_step_kernel(const __grid_constant__ McbCtx ctx_p,
                                                         const __grid_constant__ McbDenseStepArgs args_p,
                                                         const McbCtx* ectx, const McbDenseStepArgs* eargs) {
  const McbCtx& c = EMU ? ectx[blockIdx.y] : ctx_p;
  const McbDenseStepArgs& a = EMU ? eargs[blockIdx.y] : args_p;
  __shared__ int s_prefix[MCB_MAX_RANKS + 1];
  __shared__ int s_cnt[MCB_MAX_RANKS];
  __shared__ int s_max;
  const int tid = threadIdx.x, bid = blockIdx.x;
  const int W = c.world, L = a.num_layers;
  pdl_wait();                 // the previous kernel of this rank (the previous step) has finished
  pdl_launch_dependents();
  volatile uint32_t* state = a.state;
  const uint32_t step_seq = state[MCB_STATE_STEP_SEQ], layer_base = state[MCB_STATE_LAYER_BASE],
                 ll_base = state[MCB_STATE_LL_BASE];

  // ---- count exchange -------------------------------------------------------------------------
  const int n = step_count_exchange(c, MCB_SITE_STEP_META, a.counts_off, step_seq, *a.n_local, a.cap, s_cnt, s_prefix,
                                    &s_max);
  const int valid = s_prefix[W], offset = s_prefix[c.rank], ep_max = s_max;

  StepShape shp;
  long long bytes_per_row = 0;
  bool words_ok = (a.rsv_row_bytes & 7u) == 0;
  shp.wpr = 0;
#pragma unroll
  for (int t = 0; t < MCB_MAX_TENSORS; ++t) {
    const uint32_t rb = t < a.num_tensors ? a.row_bytes[t] : 0u;
    shp.w[t] = (int)(rb >> 3);
    shp.wpr += shp.w[t];
    bytes_per_row += rb;
    if (rb & 7u) words_ok = false;
  }
  const bool ll = W > 1 && a.ll_rows > 0 && valid > 0 && valid <= a.ll_rows && a.rsv_dtype == 0 && words_ok;

  // ---- pipeline groups of the barrier mode (identical decision on every rank) ---------------------
  int G = a.groups < 1 ? 1 : (a.groups > MCB_MAX_GROUPS ? MCB_MAX_GROUPS : a.groups);
  if (W == 1 || ll) G = 1;
  while (G > 1 && ((long long)ep_max * bytes_per_row < (long long)G * (long long)a.group_min_bytes ||
                   (int)gridDim.x < 2 * G))
    --G;
  const int bpg = (int)gridDim.x / G;                   // blocks per group (left-over blocks idle)
  const int grp = bid / bpg < G ? bid / bpg : -1;
  const int lb = bid - (grp < 0 ? 0 : grp) * bpg;       // block index inside its group
  const int ep_max_g = (ep_max + G - 1) / G;
  const int nact = active_blocks(bpg, ep_max_g, bytes_per_row, (int)blockDim.x);

  if (bid == 0 && tid == 0) {
    a.step_meta[0] = valid;
    a.step_meta[1] = offset;
    a.step_meta[2] = ep_max;
    a.step_meta[4] = (int)(step_seq + 1u);
    a.step_meta[5] = L > 0 ? (int)((layer_base + (uint32_t)L - 1u) & 1u) : 0;
    a.step_meta[6] = ll ? 1 : 0;
    a.step_meta[7] = G;
  }

  if (ll) {
    // ---- packet mode ---------------------------------------------------------------------------
    int nb = ceil_div_i((long long)valid * shp.wpr, blockDim.x);
    if (nb > (int)gridDim.x) nb = (int)gridDim.x;
    if (bid < nb) {
      const long long gtid = (long long)bid * blockDim.x + tid;
      const long long nthreads = (long long)nb * blockDim.x;
      const uint32_t cb = *epoch_ptr(c, MCB_SITE_STEP_CREDIT, bid);
      for (int l = 0; l < L; ++l) {
        const uint32_t flag = ll_base + (uint32_t)l + 1u;
        const uint32_t par = (layer_base + (uint32_t)l) & 1u;
        // The staging area of this parity was read last in layer l - 2 (every rank has left the
        // previous step: nothing to wait for in the first two layers).
        if (l >= 2) credit_wait(c, a.credit_off, cb + (uint32_t)l - 1u, MCB_SITE_STEP_CREDIT);
        if (CHECK && a.delay_ns && (l + c.rank) % (a.delay_every < 1 ? 1 : a.delay_every) == 0)
          __nanosleep(a.delay_ns > 1000000u ? 1000000u : a.delay_ns);
        step_agv_ll<CHECK, FP8>(c, a, shp, n, offset, valid, flag, par, layer_base + (uint32_t)l, gtid, nthreads);
        __syncthreads();      // the block holds all its gathered words before it starts the combine
        step_rsv_ll(c, a, s_prefix, n, ep_max, flag, gtid, nthreads);
        __syncthreads();
        credit_publish(c, a.credit_off, cb + (uint32_t)l + 1u);
      }
      if (tid == 0) *epoch_ptr(c, MCB_SITE_STEP_CREDIT, bid) = cb + (uint32_t)L;
    }
  } else if (EMU && W == 1 && !CHECK) {      // else dense_alone_kernel
    __shared__ LocalRanges r;
    local_ranges<FP8>(r, c, a, n);
    const int nloc = active_blocks((int)gridDim.x, n, bytes_per_row + a.rsv_row_bytes, (int)blockDim.x);
    if (n > 0 && a.in_order) local_in_order<FP8>(c, a, r, n, nloc, layer_base);
    else if (n > 0) local_dealt<FP8>(c, a, r, n, layer_base);
  } else if (grp >= 0 && lb < nact) {
    // ---- barrier mode ----------------------------------------------------------------------------
    uint32_t ep = *epoch_ptr(c, MCB_SITE_STEP, bid);
    // Rows of this group: an equal share of this rank's rows, and of the rows it owns.
    const int r0 = (int)((long long)n * grp / G), r1 = (int)((long long)n * (grp + 1) / G);
    const long long start = (long long)lb * blockDim.x + tid;
    const long long stride = (long long)nact * blockDim.x;
    const int prev = (grp + G - 1) % G;
    uint8_t* out = reinterpret_cast<uint8_t*>(a.out);
    for (int l = 0; l < L; ++l) {
      const uint32_t par = (layer_base + (uint32_t)l) & 1u;
      if (CHECK && a.delay_ns && (l + c.rank + grp) % (a.delay_every < 1 ? 1 : a.delay_every) == 0)
        __nanosleep(a.delay_ns > 1000000u ? 1000000u : a.delay_ns);
      if (G > 1) {
        // Pushes take turns: group g of layer l goes after group g - 1 of layer l, group 0 after
        // the last group of layer l - 1.
        const uint32_t need = (uint32_t)nact * (uint32_t)(grp == 0 ? l : l + 1);
        if (tid == 0 && need) wait_local(c, a.state + MCB_STATE_GATE0 + prev, need, MCB_SITE_STEP);
        __syncthreads();
      }
      if (FP8) fp8_push(c, a, par, offset, r0, r1, start, stride);
#pragma unroll
      for (int t = 0; t < MCB_MAX_TENSORS; ++t) {
        if (t >= a.num_tensors) break;
        if (FP8 && (t == 0 || t == 3)) continue;      // quantised values and scales: pushed above
        const uint32_t rb = a.row_bytes[t];
        const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src[t]) + (uint64_t)r0 * rb;
        const uint64_t dst_off = a.dst_off[t] + (uint64_t)par * a.dst_par_stride[t] + (uint64_t)(offset + r0) * rb;
        const long long nbytes = (long long)(r1 - r0) * rb;
        if (CHECK) {
          check_push(c, a.dst_off[t] + (uint64_t)par * a.dst_par_stride[t], (uint32_t)t, layer_base + (uint32_t)l,
                     (long long)(offset + r0) * (rb >> 2), nbytes >> 2, start, stride);
          continue;
        }
        if ((rb & 15u) == 0) broadcast_flat<16>(c, src, dst_off, nbytes, start, stride);
        else if ((rb & 7u) == 0) broadcast_flat<8>(c, src, dst_off, nbytes, start, stride);
        else broadcast_flat<4>(c, src, dst_off, nbytes, start, stride);
      }
      if (W > 1) {
        __syncthreads();
        signal_all<true>(c, MCB_SITE_STEP, bid);
        if (tid == 0) {
          // The release above returns once this block's stores have left: the next group may push.
          if (G > 1) atomicAdd(a.state + MCB_STATE_GATE0 + grp, 1u);
          wait_flag(c, MCB_SITE_STEP, bid, (ep + 1u) * (uint32_t)W);
        }
        ++ep;
        __syncthreads();
      }
      if (CHECK) {
        // Words pushed by the matching block of every rank (this group's share of that rank's rows).
        for (int p = 0; p < W; ++p) {
          const int cnt = s_prefix[p + 1] - s_prefix[p];
          const int q0 = (int)((long long)cnt * grp / G), q1 = (int)((long long)cnt * (grp + 1) / G);
#pragma unroll
          for (int t = 0; t < MCB_MAX_TENSORS; ++t) {
            if (t >= a.num_tensors) break;
            const uint32_t rb = a.row_bytes[t];
            check_verify(c, a, a.dst_off[t] + (uint64_t)par * a.dst_par_stride[t], (uint32_t)t,
                         layer_base + (uint32_t)l, (long long)(s_prefix[p] + q0) * (rb >> 2),
                         (long long)(q1 - q0) * (rb >> 2), start, stride);
          }
        }
      }
      const long long nvec = (long long)(r1 - r0) * a.rsv_row_bytes / 16;
      reduce_flat(c, out + (uint64_t)r0 * a.rsv_row_bytes, a.rsv_off + (uint64_t)(offset + r0) * a.rsv_row_bytes,
                  nvec, start, stride, a.rsv_dtype);
    }
    if (tid == 0) *epoch_ptr(c, MCB_SITE_STEP, bid) = ep;
  }

  // ---- the last block out advances the sequence words ---------------------------------------------
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(a.state + MCB_STATE_FINISHED, 1u) == gridDim.x - 1u) {
      state[MCB_STATE_STEP_SEQ] = step_seq + 1u;
      state[MCB_STATE_LAYER_BASE] = layer_base + (uint32_t)L;
      state[MCB_STATE_LL_BASE] = ll_base + (ll ? (uint32_t)L : 0u);
      for (int g = 0; g < MCB_MAX_GROUPS; ++g) state[MCB_STATE_GATE0 + g] = 0u;
      state[MCB_STATE_FINISHED] = 0u;
      __threadfence();
    }
  }
}

// The step of a world of one, a kernel of its own for each way: everything is inline, so the arguments are read from the constant bank and not
// through pointers after every store.  D: as in local_few; kDealt: more layers; kInOrder: steps that read what they write.  With the last way in
// each of the kernels, dealt steps were slower and so was one layer of e4m3 rows: 8192 rows of 1024, 88 layers 336 -> 298 us, 100 rows 9.5 -> 8.5; e4m3
// 365 -> 344, one layer of 37 rows 4.8 -> 3.8.  Few layers of bf16 rows keep it, and are compiled for no number of blocks per SM (93 to 95 registers instead of
// 121 to 128): without either, steps of 3.5 us took 0.1 to 0.5 us more.  2 / 3 / 4 layers of 20 rows of 1024 3.79 / 3.68 / 3.62 -> 3.56 / 3.48 / 3.38 us, of
// 150 rows 3.79 / 3.87 / 3.84 -> 3.58 / 3.52 / 3.46; large steps of two layers would be faster with more (1000 rows of 7168 11.5 and 12.4). Dealt e4m3 steps
// have 20 warps per block where others have 16: the quantisation waits for its own instructions, 344 -> 333 us, 58 layers of 2048 rows of 7168 394 -> 375,
// small ones the same.  Copies do not gain from more warps: 640 threads 342 us where 512 took 331, 768 383.
constexpr int kInOrder = 0, kDealt = -1;
template <bool FP8, int D>
__global__ void __launch_bounds__(FP8 && D == kDealt ? 640 : 512, FP8 || D <= 0 ? 1 : 0)
dense_alone_kernel(const __grid_constant__ McbCtx c, const __grid_constant__ McbDenseStepArgs a) {
  __shared__ int s_prefix[2], s_cnt[1], s_max;
  pdl_wait();                 // the previous kernel of this rank (the previous step) has finished
  pdl_launch_dependents();
  volatile uint32_t* state = a.state;
  const int L = a.num_layers;
  const uint32_t step_seq = state[MCB_STATE_STEP_SEQ], layer_base = state[MCB_STATE_LAYER_BASE];
  const int n = step_count_exchange(c, MCB_SITE_STEP_META, a.counts_off, step_seq, *a.n_local, a.cap, s_cnt, s_prefix, &s_max);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.step_meta[0] = n;
    a.step_meta[1] = 0;
    a.step_meta[2] = n;
    a.step_meta[4] = (int)(step_seq + 1u);
    a.step_meta[5] = L > 0 ? (int)((layer_base + (uint32_t)L - 1u) & 1u) : 0;
    a.step_meta[6] = 0;
    a.step_meta[7] = 1;
  }
  long long bytes_per_row = a.rsv_row_bytes;
#pragma unroll
  for (int t = 0; t < MCB_MAX_TENSORS; ++t)
    if (t < a.num_tensors) bytes_per_row += a.row_bytes[t];
  const int nact = active_blocks((int)gridDim.x, n, bytes_per_row, (int)blockDim.x);
  if (n > 0) {
    __shared__ LocalRanges r;
    local_ranges<FP8>(r, c, a, n);
    if constexpr (D == kDealt) {
      local_dealt<FP8>(c, a, r, n, layer_base);
    } else if constexpr (D == kInOrder) {
      if ((long long)n * a.rsv_row_bytes < 48ll * nact * blockDim.x) local_in_order<FP8, true>(c, a, r, n, nact, layer_base);
      else local_in_order<FP8>(c, a, r, n, nact, layer_base);
    } else {
      if (FP8 || !a.in_order) local_few<FP8, D>(c, a, r, n, layer_base);
      else local_in_order<FP8>(c, a, r, n, nact, layer_base);
    }
  }
  step_close(a.state, step_seq, layer_base + (uint32_t)L);
}

}  // namespace mcb

using namespace mcb;

extern "C" {

int mcb_sizeof_dense_step_args() { return (int)sizeof(McbDenseStepArgs); }

static int check_step_args(const McbDenseStepArgs* a, int grid, int threads) {
  if (!a || grid < 1 || grid > MCB_MAX_BLOCKS || threads < 32 || threads > 512 || (threads & 31)) return 1;
  if (a->num_tensors < 1 || a->num_tensors > MCB_MAX_TENSORS || a->num_layers < 0 || a->cap < 1) return 1;
  if ((a->rsv_row_bytes & 15u) || !a->state || !a->step_meta || !a->n_local || !a->out) return 1;
  if (a->ll_rows > 0 && (a->credit_off == 0 || (a->credit_off & 3u))) return 1;
  for (int t = 0; t < a->num_tensors; ++t)
    if ((a->row_bytes[t] & 3u) || (!a->src[t] && !(a->fp8_hidden && t == 3))) return 1;
  if (a->fp8_hidden) {
    // quantised dispatch: tensor 0 = one byte per value, tensor 3 = one fp32 scale per 128 values
    if (a->check || a->num_tensors != 4 || a->fp8_hidden % 128u || a->row_bytes[0] != a->fp8_hidden ||
        a->row_bytes[3] != a->fp8_hidden / 128u * 4u)
      return 1;
  }
  return 0;
}

// Whether a step in a world of one writes rows that it reads, or writes rows twice: an output on a source (a step in
// place), partial sums that are gathered rows (the identity expert), tensors gathered to one place.  Its copies then keep the order of the
// layers, and within a layer that of the tensors.
int mcb_dense_step_in_order(const McbCtx* ctx, const McbDenseStepArgs* a) {
  if (ctx->world != 1) return 0;
  struct Range { uint64_t at, bytes; };
  auto meet = [](Range x, Range y) { return x.at && y.at && x.at < y.at + y.bytes && y.at < x.at + x.bytes; };
  const uint64_t heap = reinterpret_cast<uint64_t>(ctx->heap_local), cap = (uint64_t)a->cap;
  const Range out{reinterpret_cast<uint64_t>(a->out), cap * a->rsv_row_bytes}, sums{heap + a->rsv_off, cap * a->rsv_row_bytes};
  bool hit = meet(out, sums);
  for (int t = 0; t < a->num_tensors; ++t) {
    const Range rows{heap + a->dst_off[t], a->dst_par_stride[t] + cap * a->row_bytes[t]};
    hit = hit || meet(rows, sums) || meet(rows, out);
    for (int u = 0; u < a->num_tensors; ++u) {
      const Range src{reinterpret_cast<uint64_t>(a->src[u]), cap * (a->fp8_hidden && u == 0 ? 2u * a->fp8_hidden : a->row_bytes[u])};
      hit = hit || meet(src, rows) || meet(src, out);
      for (int k = 0; k < 4 && u < t; ++k) {             // gathered rows of either parity of two tensors
        const Range one{heap + a->dst_off[t] + (k & 1) * a->dst_par_stride[t], cap * a->row_bytes[t]};
        const Range two{heap + a->dst_off[u] + (k >> 1) * a->dst_par_stride[u], cap * a->row_bytes[u]};
        hit = hit || meet(one, two);
      }
    }
  }
  return hit;
}

// The pipeline groups wait on one another inside the launch, so with groups > 1 all blocks must be
// resident at once: the launch is cooperative.
int mcb_launch_dense_step(const McbCtx* ctx, const McbDenseStepArgs* args, int grid, int threads, int pdl,
                          cudaStream_t stream) {
  if (!ctx || check_step_args(args, grid, threads)) return cudaErrorInvalidValue;
  const bool coop = args->groups > 1;
  McbDenseStepArgs a = *args;
  a.in_order = mcb_dense_step_in_order(ctx, args);
  if (ctx->world == 1 && !args->check) {
    auto alone = [&](auto layers) {
      constexpr int D = decltype(layers)::value;
      const int block = D == kDealt && a.fp8_hidden ? threads / 32 * 20 / 16 * 32 : threads;
      return launch_kernel(a.fp8_hidden ? dense_alone_kernel<true, D> : dense_alone_kernel<false, D>, dim3(grid), dim3(block), 0, stream, pdl, false,
                           *ctx, a);
    };
    if (a.in_order && (a.fp8_hidden || a.num_layers > kFewLayers)) return alone(std::integral_constant<int, kInOrder>{});
    if (a.num_layers > kFewLayers) return alone(std::integral_constant<int, kDealt>{});
    if (a.num_layers > 4) return alone(std::integral_constant<int, kFewLayers>{});
    if (a.num_layers > 2) return alone(std::integral_constant<int, 4>{});
    return a.num_layers > 1 ? alone(std::integral_constant<int, 2>{}) : alone(std::integral_constant<int, 1>{});
  }
  if (args->check)
    return launch_kernel(dense_step_kernel<false, true, false>, dim3(grid), dim3(threads), 0, stream, pdl, coop, *ctx,
                         a, (const McbCtx*)nullptr, (const McbDenseStepArgs*)nullptr);
  if (args->fp8_hidden)
    return launch_kernel(dense_step_kernel<false, false, true>, dim3(grid), dim3(threads), 0, stream, pdl, coop, *ctx,
                         a, (const McbCtx*)nullptr, (const McbDenseStepArgs*)nullptr);
  return launch_kernel(dense_step_kernel<false, false, false>, dim3(grid), dim3(threads), 0, stream, pdl, coop, *ctx,
                       a, (const McbCtx*)nullptr, (const McbDenseStepArgs*)nullptr);
}

int mcb_emu_dense_step(const McbCtx* d_ctx, const McbDenseStepArgs* d_args, const McbDenseStepArgs* h_args0,
                       int world, int grid, int threads, cudaStream_t stream) {
  if (!d_ctx || !d_args || world < 1 || check_step_args(h_args0, grid, threads)) return cudaErrorInvalidValue;
  McbCtx dummy{};
  McbDenseStepArgs dargs{};
  if (h_args0->check)
    return launch_kernel(dense_step_kernel<true, true, false>, dim3(grid, world), dim3(threads), 0, stream, 0, true,
                         dummy, dargs, d_ctx, d_args);
  if (h_args0->fp8_hidden)
    return launch_kernel(dense_step_kernel<true, false, true>, dim3(grid, world), dim3(threads), 0, stream, 0, true,
                         dummy, dargs, d_ctx, d_args);
  return launch_kernel(dense_step_kernel<true, false, false>, dim3(grid, world), dim3(threads), 0, stream, 0, true,
                       dummy, dargs, d_ctx, d_args);
}

}  // extern "C"
