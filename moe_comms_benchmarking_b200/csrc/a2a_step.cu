// One whole decode step of the all-to-all dispatcher as ONE persistent kernel for sm_100a.
//
// Contract of the path the reference wraps (bench_deepep.py:68-115): a token travels once to every
// DISTINCT destination rank, routing travels with it, nothing synchronises with the host, and the
// combine returns, per source token, the sum of one row per destination rank.  The two-kernel form
// (a2a.cu) hands out compacted receive slots with atomic counters and publishes row counts; that
// costs two launches, a "last block" hand-over and a pull through a slot map per layer.  Here
//   * a token's slot on every destination is its own index (receive layout [parity][source][cap]):
//     no counters, no slot map, no hand-over; a destination tells valid rows by the stamp in the
//     row's metadata (the layer's sequence number), so stale rows of earlier layers never match;
//   * routing ids, weights, stamp and source index are one packed metadata row written with
//     16-byte stores ({stamp, token, (id, weight) x topk});
//   * a layer is: push -> ONE block-matched release barrier -> pull + fp32 sum, with the receive
//     buffers double buffered by layer parity (the barrier of layer l is the write-after-read fence
//     for the readers of layer l - 1), and the 88 layers run inside one launch after one count
//     exchange that also proves every rank has left the previous step;
//   * optional 1 x 128 block-scaled e4m3 dispatch, quantised on the way out;
//   * packet mode for small steps: rows travel as 16-byte flagged packets, so a layer needs no fence
//     and no barrier.  Every rank receives a one-packet header per token (routed to you or not), so a
//     destination knows which rows to wait for; the destination's warp for that token unpacks the row
//     into the ordinary receive buffers and sends the expert output straight back as packets, and the
//     source sums them as they arrive.  A token is served by a whole block (one 8-byte word per thread), all
//     traffic of a token runs between the same block index on the ranks involved, and the staging areas
//     (two parities) are recycled on per-source credit words.
// Every wait is bounded and reports through the status words.
#include <cuda_runtime.h>

#include <type_traits>

#include "mcb_barrier.cuh"
#include "mcb_dense.cuh"
#include "mcb_fp8.cuh"
#include "mcb_launch.h"
#include "mcb_launchers.h"
#include "mcb_step.cuh"

namespace mcb {

struct DestMask { uint32_t w[3]; };    // 96 bits cover MCB_MAX_RANKS = 72

// Destination ranks of one token (all lanes of the warp get the same mask).
__device__ __forceinline__ DestMask dest_mask(const McbCtx& c, const McbA2AStepArgs& a, int t, int epr, int lane) {
  DestMask m = {{0u, 0u, 0u}};
  for (int k = lane; k < a.topk; k += 32) {
    const long long e = a.topk_idx[(long long)t * a.topk + k];
    if (e < 0 || e >= a.num_experts) {
      report_error(c, MCB_ERR_ROUTING, MCB_SITE_A2A_STEP, blockIdx.x, (uint32_t)t, (uint32_t)e);
      continue;
    }
    const uint32_t d = (uint32_t)e / (uint32_t)epr;
    m.w[d >> 5] |= 1u << (d & 31);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i * 32 < c.world) m.w[i] = __reduce_or_sync(0xffffffffu, m.w[i]);
  return m;
}

// ---- packet mode ------------------------------------------------------------------------------------
struct LLShape {
  int xdata;      // 8-byte words of a dispatched row (bf16: hidden / 4, e4m3: hidden / 8)
  int scales;     // words of fp32 scales (e4m3 only: hidden / 256)
  int meta;       // words of the packed metadata row
  int xw;         // 1 header + xdata + scales + meta
  int yw;         // words of an expert-output row (hidden / 4)
};

__device__ __forceinline__ uint64_t ll_x_slot(const McbA2AStepArgs& a, const LLShape& s, int world, uint32_t par, int src,
                                              int t, int word) {
  return a.ll_x_off + ((((uint64_t)par * world + src) * a.ll_src_rows + t) * s.xw + word) * 16;
}
__device__ __forceinline__ uint64_t ll_y_slot(const McbA2AStepArgs& a, const LLShape& s, int world, uint32_t par, int dst,
                                              int t, int word) {
  return a.ll_y_off + ((((uint64_t)par * world + dst) * a.ll_src_rows + t) * s.yw + word) * 16;
}

// Send one 8-byte word of token t's row to every destination in the mask.
__device__ __forceinline__ void ll_send_x(const McbCtx& c, const McbA2AStepArgs& a, const LLShape& s, const DestMask& m,
                                          uint32_t par, int t, int word, uint2 d, uint32_t flag) {
  const uint4 pkt = ll_pack(d, flag);
#pragma unroll 1
  for (int wi = 0; wi < 3; ++wi) {
    uint32_t bits = m.w[wi];
    while (bits) {
      const int dst = wi * 32 + __ffs(bits) - 1;
      bits &= bits - 1;
      st_v4(c.heap_peer[dst] + ll_x_slot(a, s, c.world, par, c.rank, t, word), pkt);
    }
  }
}

// In packet mode a token is served by a whole BLOCK (steps are small, so blocks are plentiful, and a layer's
// latency is a chain of dependent loads: with one 8-byte word per thread the chain is one load deep).

// Source side of a layer: header to every rank, row / scales / metadata to the routed destinations.
__device__ __forceinline__ void ll_dispatch_token(const McbCtx& c, const McbA2AStepArgs& a, const LLShape& s, int t,
                                                  int epr, uint32_t par, uint32_t flag) {
  const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31;
  const DestMask m = dest_mask(c, a, t, epr, lane);
  for (int p = tid; p < c.world; p += nthreads) {
    const uint32_t routed = (m.w[p >> 5] >> (p & 31)) & 1u;
    st_v4(c.heap_peer[p] + ll_x_slot(a, s, c.world, par, c.rank, t, 0), ll_pack(make_uint2(routed, (uint32_t)t), flag));
  }
  const uint8_t* xrow = reinterpret_cast<const uint8_t*>(a.x) + (uint64_t)t * a.hidden * 2;
  if (!a.fp8) {
    for (int j = tid; j < s.xdata; j += nthreads) ll_send_x(c, a, s, m, par, t, 1 + j, ld_v2(xrow + (uint64_t)j * 8), flag);
  } else {
    const int row_packs = a.hidden / 8;               // a multiple of 32 (hidden % 256 == 0): warps are all in or all out
    for (int p = tid; p < row_packs; p += nthreads) {
      const uint4 v = ld_v4(xrow + (uint64_t)p * 16);
      float amax = pack_absmax(v);                     // 16 lanes hold one 128-value block
#pragma unroll
      for (int sh = 8; sh >= 1; sh >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, sh));
      const float scale = e4m3_scale(amax);
      ll_send_x(c, a, s, m, par, t, 1 + p, quant_pack_e4m3(v, scale), flag);
      // lanes 0-15 hold one block, lanes 16-31 the next one: one word carries both scales
      const float other = __shfl_sync(0xffffffffu, scale, 16);
      if (lane == 0)
        ll_send_x(c, a, s, m, par, t, 1 + s.xdata + (p >> 5), make_uint2(__float_as_uint(scale), __float_as_uint(other)), flag);
    }
  }
  // metadata row: chunk 0 = {stamp, token, id 0, weight 0}, chunk j = {id 2j-1, weight 2j-1, id 2j, weight 2j};
  // taken from the top of the block so that it does not queue behind the row words of the low threads
  for (int j = nthreads - 1 - tid; j < s.meta / 2; j += nthreads) {
    const int k0 = j == 0 ? 0 : 2 * j - 1, k1 = 2 * j;
    const long long tb = (long long)t * a.topk;
    const uint32_t id0 = k0 < a.topk ? (uint32_t)a.topk_idx[tb + k0] : 0xffffffffu;
    const uint32_t w0 = k0 < a.topk ? __float_as_uint(a.topk_w ? a.topk_w[tb + k0] : 1.0f) : 0u;
    uint2 lo, hi;
    if (j == 0) {
      lo = make_uint2(flag, (uint32_t)t);
      hi = make_uint2(id0, w0);
    } else {
      const uint32_t id1 = k1 < a.topk ? (uint32_t)a.topk_idx[tb + k1] : 0xffffffffu;
      const uint32_t w1 = k1 < a.topk ? __float_as_uint(a.topk_w ? a.topk_w[tb + k1] : 1.0f) : 0u;
      lo = make_uint2(id0, w0);
      hi = make_uint2(id1, w1);
    }
    ll_send_x(c, a, s, m, par, t, 1 + s.xdata + s.scales + 2 * j, lo, flag);
    ll_send_x(c, a, s, m, par, t, 1 + s.xdata + s.scales + 2 * j + 1, hi, flag);
  }
}

// Destination side: wait for the header of (source, token); if the token is routed here, unpack its row
// into the ordinary receive buffers and send the expert output (the row itself for the identity expert
// in bf16, the y buffer otherwise) back to the source.
__device__ __forceinline__ void ll_serve_token(const McbCtx& c, const McbA2AStepArgs& a, const LLShape& s, int src, int t,
                                               uint32_t par, uint32_t flag) {
  const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31;
  uint32_t routed = 0;
  if (lane == 0) routed = ll_wait(c, c.heap_local + ll_x_slot(a, s, c.world, par, src, t, 0), flag, MCB_SITE_A2A_STEP).x;
  routed = __shfl_sync(0xffffffffu, routed, 0);
  if (!routed) return;
  const uint64_t row = (uint64_t)src * a.cap + t;
  const uint64_t xrow_bytes = a.fp8 ? (uint64_t)a.hidden : (uint64_t)a.hidden * 2;
  uint8_t* rx = c.heap_local + a.recv_x_off + (uint64_t)par * a.x_par_stride + row * xrow_bytes;
  uint8_t* rs = c.heap_local + a.recv_scale_off + (uint64_t)par * a.scale_par_stride + row * (uint64_t)(a.hidden / 128) * 4;
  uint8_t* rm = c.heap_local + a.recv_meta_off + (uint64_t)par * a.meta_par_stride + row * a.meta_row_bytes;
  const uint8_t* yrow = c.heap_local + a.y_off + (uint64_t)par * a.y_par_stride + row * (uint64_t)a.hidden * 2;
  const int body = s.xdata + s.scales + s.meta;
  const bool echo = !a.fp8 && a.y_off == a.recv_x_off;     // identity expert on bf16 rows: the row is its own output
  if (!echo)     // the expert output is a bf16 row of its own: it can leave before the row has arrived
    for (int j = tid; j < s.yw; j += nthreads)
      st_v4(c.heap_peer[src] + ll_y_slot(a, s, c.world, par, c.rank, t, j), ll_pack(ld_v2(yrow + (uint64_t)j * 8), flag));
  for (int j = tid; j < body; j += nthreads) {
    const uint2 d = ll_wait(c, c.heap_local + ll_x_slot(a, s, c.world, par, src, t, 1 + j), flag, MCB_SITE_A2A_STEP);
    if (j < s.xdata) {
      if (echo) st_v4(c.heap_peer[src] + ll_y_slot(a, s, c.world, par, c.rank, t, j), ll_pack(d, flag));
      st_v2(rx + (uint64_t)j * 8, d);
    } else if (j < s.xdata + s.scales) {
      st_v2(rs + (uint64_t)(j - s.xdata) * 8, d);
    } else {
      st_v2(rm + (uint64_t)(j - s.xdata - s.scales) * 8, d);
    }
  }
}

__device__ __forceinline__ int pop_dest(DestMask& m) {
#pragma unroll
  for (int wi = 0; wi < 3; ++wi)
    if (m.w[wi]) {
      const int b = __ffs(m.w[wi]) - 1;
      m.w[wi] &= m.w[wi] - 1;
      return wi * 32 + b;
    }
  return -1;
}

// Source side again: sum the expert outputs of every destination as their packets arrive (four
// destinations' packets in flight per thread).
__device__ __forceinline__ void ll_combine_token(const McbCtx& c, const McbA2AStepArgs& a, const LLShape& s, int t,
                                                 int epr, uint32_t par, uint32_t flag) {
  const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31;
  const DestMask m = dest_mask(c, a, t, epr, lane);
  uint8_t* orow = reinterpret_cast<uint8_t*>(a.out) + (uint64_t)t * a.hidden * 2;
  for (int j = tid; j < s.yw; j += nthreads) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    DestMask rest = m;
    for (;;) {
      int d[4];
      d[0] = pop_dest(rest);
      if (d[0] < 0) break;
#pragma unroll
      for (int u = 1; u < 4; ++u) d[u] = pop_dest(rest);
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (d[u] >= 0) v[u] = ld_v4_volatile(c.heap_local + ll_y_slot(a, s, c.world, par, d[u], t, j));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (d[u] < 0) continue;
        uint2 w = make_uint2(v[u].x, v[u].z);
        if (v[u].y != flag || v[u].w != flag)
          w = ll_wait(c, c.heap_local + ll_y_slot(a, s, c.world, par, d[u], t, j), flag, MCB_SITE_A2A_STEP);
        acc[0] += bf16_lo(w.x); acc[1] += bf16_hi(w.x);
        acc[2] += bf16_lo(w.y); acc[3] += bf16_hi(w.y);
      }
    }
    st_v2(orow + (uint64_t)j * 8, make_uint2(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3])));
  }
}

// Packet-mode layers of a step: global token g belongs to block g % blocks on every rank.  Kept out of line
// so that the two modes do not share one register allocation.
__device__ __noinline__ void packet_layers(const McbCtx& c, const McbA2AStepArgs& a, const LLShape& shp, const int* s_prefix,
                                           int n, int valid, uint32_t layer_base) {
  const int tid = threadIdx.x, bid = blockIdx.x;
  const int W = c.world, L = a.num_layers;
  const int nb = valid < (int)gridDim.x ? valid : (int)gridDim.x;
  if (bid >= nb) return;
  const int epr_ll = a.num_experts / W;
  const int offset = s_prefix[c.rank];
  const uint32_t cb = *epoch_ptr(c, MCB_SITE_A2A_STEP_CREDIT, bid);
  const int t0 = ((bid - offset) % nb + nb) % nb;      // first own token with (offset + t) % nb == bid
  for (int l = 0; l < L; ++l) {
    const uint32_t par = (layer_base + (uint32_t)l) & 1u;
    const uint32_t flag = layer_base + (uint32_t)l + 1u;
    // the staging areas of this parity were read last in layer l - 2
    if (l >= 2) credit_wait(c, a.credit_off, cb + (uint32_t)l - 1u, MCB_SITE_A2A_STEP_CREDIT);
    for (int t = t0; t < n; t += nb) ll_dispatch_token(c, a, shp, t, epr_ll, par, flag);
    for (int g = bid; g < valid; g += nb) {
      int src = 0;
      while (src + 1 < W && s_prefix[src + 1] <= g) ++src;
      ll_serve_token(c, a, shp, src, g - s_prefix[src], par, flag);
    }
    for (int t = t0; t < n; t += nb) ll_combine_token(c, a, shp, t, epr_ll, par, flag);
    __syncthreads();
    credit_publish(c, a.credit_off, cb + (uint32_t)l + 1u);
  }
  if (tid == 0) *epoch_ptr(c, MCB_SITE_A2A_STEP_CREDIT, bid) = cb + (uint32_t)L;
}

// ---- barrier mode -----------------------------------------------------------------------------------
// A warp serves one slice of a token's row: kSlicePacks 16-byte packs, four per lane, so a wide row (hidden 7168: seven
// slices) has as many loads in flight as seven narrow ones and a step of a few hundred wide tokens fills the chip.  Alone
// on one B200, 58 layers of 333 rows of 7168 values with e4m3 dispatch: 204 us (254 with divisions in the
// quantisation), against 1767 with one warp per token packed into as few blocks as possible and the pull as a pass of its own.
constexpr int kSlicePacks = 128;

struct RowSlice {
  int t, p0;            // token, first pack
  uint64_t row;         // row of the token in the receive layout
};

struct BarrierShape {
  int slices, row_packs, nblk, meta_chunks, epr;
  uint64_t row_bytes, xrow_bytes;
};

__device__ __forceinline__ void load_packs(uint4 (&v)[4], const uint8_t* row, int p0, int row_packs, int lane) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int p = p0 + u * 32 + lane;
    v[u] = p < row_packs ? ld_v4_stream(row + (uint64_t)p * 16) : make_uint4(0, 0, 0, 0);
  }
}

// Chunk j of the metadata row: 0 = {stamp, token, id 0, weight 0}, j = {id 2j-1, weight 2j-1, id 2j, weight 2j}; behind the last id
// {-1, 0}.  Its first id is that of slot meta_slot(j), its second, of a chunk behind the first, the next one.
__device__ __forceinline__ int meta_slot(int j) { return j == 0 ? 0 : 2 * j - 1; }
__device__ __forceinline__ uint4 meta_chunk_of(int j, uint32_t stamp, int t, uint2 first, uint2 second) {
  return j == 0 ? make_uint4(stamp, (uint32_t)t, first.x, first.y) : make_uint4(first.x, first.y, second.x, second.y);
}
__device__ __forceinline__ uint4 meta_chunk(const McbA2AStepArgs& a, int t, int j, uint32_t stamp) {
  const long long tb = (long long)t * a.topk;
  auto slot = [&](int k) {
    if (k >= a.topk) return make_uint2(0xffffffffu, 0u);
    return make_uint2((uint32_t)a.topk_idx[tb + k], __float_as_uint(a.topk_w ? a.topk_w[tb + k] : 1.0f));
  };
  return meta_chunk_of(j, stamp, t, slot(meta_slot(j)), j == 0 ? make_uint2(0u, 0u) : slot(2 * j));
}

// Slice of a row (and, with the first slice, the metadata row) to every destination in the mask.
__device__ __forceinline__ void push_slice(const McbCtx& c, const McbA2AStepArgs& a, const BarrierShape& s, const RowSlice& r,
                                           const DestMask& m, const uint4 (&v)[4], uint4 meta, uint32_t par, uint32_t stamp,
                                           int lane) {
  uint2 q[4];
  float scale[4];
  if (a.fp8) {
#pragma unroll
    for (int u = 0; u < 4; u += 2) {
      block_absmax_pair(v[u], v[u + 1], scale[u], scale[u + 1]);
#pragma unroll
      for (int k = u; k < u + 2; ++k) {
        scale[k] = e4m3_scale(scale[k]);
        q[k] = quant_pack_e4m3(v[k], scale[k]);
      }
    }
  }
#pragma unroll 1
  for (int wi = 0; wi < 3; ++wi) {
    uint32_t bits = m.w[wi];
    while (bits) {
      const int d = wi * 32 + __ffs(bits) - 1;
      bits &= bits - 1;
      uint8_t* peer = c.heap_peer[d];
      uint8_t* dst = peer + a.recv_x_off + (uint64_t)par * a.x_par_stride + r.row * s.xrow_bytes;
      uint8_t* sc = peer + a.recv_scale_off + (uint64_t)par * a.scale_par_stride + r.row * s.nblk * 4;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int p = r.p0 + u * 32 + lane;
        if (p >= s.row_packs) continue;
        if (a.fp8) {
          st_v2(dst + (uint64_t)p * 8, q[u]);
          if ((lane & 15) == 0) st_b32(sc + (p >> 4) * 4, __float_as_uint(scale[u]));
        } else {
          st_v4(dst + (uint64_t)p * 16, v[u]);
        }
      }
      if (r.p0 == 0) {
        uint8_t* md = peer + a.recv_meta_off + (uint64_t)par * a.meta_par_stride + r.row * a.meta_row_bytes;
        if (lane < s.meta_chunks) st_v4(md + lane * 16, meta);
        for (int j = lane + 32; j < s.meta_chunks; j += 32) st_v4(md + (uint64_t)j * 16, meta_chunk(a, r.t, j, stamp));
      }
    }
  }
}

__device__ __forceinline__ void add_packs(float (&acc)[4][8], const uint4 (&v)[4]) {
#pragma unroll
  for (int u = 0; u < 4; ++u) acc_bf16x8(acc[u], v[u]);
}

__device__ __forceinline__ void store_out(const McbA2AStepArgs& a, const BarrierShape& s, const RowSlice& r,
                                          const float (&acc)[4][8], int lane) {
  uint8_t* out = reinterpret_cast<uint8_t*>(a.out) + (uint64_t)r.t * s.row_bytes;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int p = r.p0 + u * 32 + lane;
    if (p < s.row_packs)
      st_v4(out + (uint64_t)p * 16, make_uint4(pack_bf16x2(acc[u][0], acc[u][1]), pack_bf16x2(acc[u][2], acc[u][3]),
                                               pack_bf16x2(acc[u][4], acc[u][5]), pack_bf16x2(acc[u][6], acc[u][7])));
  }
}

__device__ __forceinline__ BarrierShape barrier_shape(const McbCtx& c, const McbA2AStepArgs& a) {
  BarrierShape s;
  s.row_packs = a.hidden / 8;
  s.slices = (s.row_packs + kSlicePacks - 1) / kSlicePacks;
  s.nblk = a.hidden / 128;
  s.meta_chunks = (int)(a.meta_row_bytes >> 4);
  s.epr = a.num_experts / c.world;
  s.row_bytes = (uint64_t)a.hidden * 2;
  s.xrow_bytes = a.fp8 ? (uint64_t)a.hidden : s.row_bytes;     // bytes of a dispatched row
  return s;
}

// Layer after layer in a world of one, any number of ids: a slice is delivered and combined in one go, with every load of it in flight
// at once.
__device__ __forceinline__ void barrier_alone(const McbCtx& c, const McbA2AStepArgs& a, int n, uint32_t layer_base) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const BarrierShape s = barrier_shape(c, a);
  const uint8_t* x = reinterpret_cast<const uint8_t*>(a.x);
  const long long mine = (long long)n * s.slices;
  // one warp per block first, so that the smallest steps spread over the chip
  const long long nact = mine < (long long)gridDim.x ? mine : (long long)gridDim.x;
  if ((long long)blockIdx.x >= nact) return;
  const long long first = blockIdx.x + (long long)warp * nact, step = nact * (blockDim.x >> 5);
  const bool echo = !a.fp8 && a.y_off == a.recv_x_off;
  for (int l = 0; l < a.num_layers; ++l) {
    const uint32_t par = (layer_base + (uint32_t)l) & 1u;
    const uint32_t stamp = layer_base + (uint32_t)l + 1u;
    for (long long i = first; i < mine; i += step) {
      RowSlice r;
      r.t = (int)(i / s.slices);
      r.p0 = (int)(i - (long long)r.t * s.slices) * kSlicePacks;
      r.row = (uint64_t)c.rank * a.cap + r.t;
      uint4 v[4], y[4], meta = make_uint4(0, 0, 0, 0);
      load_packs(v, x + (uint64_t)r.t * s.row_bytes, r.p0, s.row_packs, lane);
      if (!echo) load_packs(y, c.heap_local + a.y_off + (uint64_t)par * a.y_par_stride + r.row * s.row_bytes, r.p0, s.row_packs, lane);
      if (r.p0 == 0 && lane < s.meta_chunks) meta = meta_chunk(a, r.t, lane, stamp);
      const DestMask m = dest_mask(c, a, r.t, s.epr, lane);
      push_slice(c, a, s, r, m, v, meta, par, stamp, lane);
      float acc[4][8] = {};
      if (m.w[0]) {
        if (echo) add_packs(acc, v);
        else add_packs(acc, y);
      }
      store_out(a, s, r, acc, lane);
    }
  }
}

// Barrier-mode layers of a step: push -> one block-matched barrier -> pull + fp32 sum.  Out of line, as above.
__device__ __noinline__ void barrier_layers(const McbCtx& c, const McbA2AStepArgs& a, int n, int ep_max, uint32_t layer_base) {
  const int tid = threadIdx.x, bid = blockIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  const int W = c.world, L = a.num_layers;
  const BarrierShape s = barrier_shape(c, a);
  const uint8_t* x = reinterpret_cast<const uint8_t*>(a.x);
  const uint64_t slot0 = (uint64_t)c.rank * a.cap;             // first row of this source on a destination
  // As many full blocks as the largest rank needs (each costs a flag per rank and layer), the same on every rank.
  const long long want = ((long long)ep_max * s.slices + nwarps - 1) / nwarps;
  const int nact = (int)(want > (long long)gridDim.x ? (long long)gridDim.x : want);
  if (bid >= nact) return;
  const long long mine = (long long)n * s.slices;
  const long long first = (long long)bid * nwarps + warp;
  const long long step = (long long)nact * nwarps;
  auto slice_of = [&](long long i) {
    RowSlice r;
    r.t = (int)(i / s.slices);
    r.p0 = (int)(i - (long long)r.t * s.slices) * kSlicePacks;
    r.row = slot0 + r.t;
    return r;
  };

  uint32_t ep = *epoch_ptr(c, MCB_SITE_A2A_STEP, bid);
  for (int l = 0; l < L; ++l) {
    const uint32_t par = (layer_base + (uint32_t)l) & 1u;
    const uint32_t stamp = layer_base + (uint32_t)l + 1u;
    // ---- push: row (+ scales) and metadata to every distinct destination rank ----
    DestMask m = {{0u, 0u, 0u}};
    for (long long i = first; i < mine; i += step) {
      const RowSlice r = slice_of(i);
      uint4 v[4], meta = make_uint4(0, 0, 0, 0);
      load_packs(v, x + (uint64_t)r.t * s.row_bytes, r.p0, s.row_packs, lane);
      if (r.p0 == 0 && lane < s.meta_chunks) meta = meta_chunk(a, r.t, lane, stamp);
      m = dest_mask(c, a, r.t, s.epr, lane);
      push_slice(c, a, s, r, m, v, meta, par, stamp, lane);
    }
    // ---- one barrier: the matching block of every rank has pushed its tokens of this layer ----
    __syncthreads();
    signal_all<true>(c, MCB_SITE_A2A_STEP, bid);
    if (tid == 0) wait_flag(c, MCB_SITE_A2A_STEP, bid, (ep + 1u) * (uint32_t)W);
    ++ep;
    __syncthreads();
    // ---- pull: one expert-output row per destination rank, summed in fp32 ----
    for (long long i = first; i < mine; i += step) {
      const RowSlice r = slice_of(i);
      if (mine > step) m = dest_mask(c, a, r.t, s.epr, lane);      // else the warp's only slice: the mask of its push
      const uint64_t yoff = a.y_off + (uint64_t)par * a.y_par_stride + r.row * s.row_bytes;
      float acc[4][8] = {};
#pragma unroll 1
      for (int wi = 0; wi < 3; ++wi) {
        uint32_t bits = m.w[wi];
        while (bits) {
          // two destinations per round: 8 independent 16-byte peer loads in flight per lane
          const int d0 = wi * 32 + __ffs(bits) - 1;
          bits &= bits - 1;
          int d1 = -1;
          if (bits) { d1 = wi * 32 + __ffs(bits) - 1; bits &= bits - 1; }
          uint4 v0[4], v1[4];
          load_packs(v0, c.heap_peer[d0] + yoff, r.p0, s.row_packs, lane);
          if (d1 >= 0) load_packs(v1, c.heap_peer[d1] + yoff, r.p0, s.row_packs, lane);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (d1 < 0) v1[u] = make_uint4(0, 0, 0, 0);
            acc[u][0] += bf16_lo(v0[u].x) + bf16_lo(v1[u].x); acc[u][1] += bf16_hi(v0[u].x) + bf16_hi(v1[u].x);
            acc[u][2] += bf16_lo(v0[u].y) + bf16_lo(v1[u].y); acc[u][3] += bf16_hi(v0[u].y) + bf16_hi(v1[u].y);
            acc[u][4] += bf16_lo(v0[u].z) + bf16_lo(v1[u].z); acc[u][5] += bf16_hi(v0[u].z) + bf16_hi(v1[u].z);
            acc[u][6] += bf16_lo(v0[u].w) + bf16_lo(v1[u].w); acc[u][7] += bf16_hi(v0[u].w) + bf16_hi(v1[u].w);
          }
        }
      }
      store_out(a, s, r, acc, lane);
    }
  }
  if (tid == 0) *epoch_ptr(c, MCB_SITE_A2A_STEP, bid) = ep;
}

// Opening of a step, for all threads of every block.
struct A2AStep {
  int n, ep_max;
  uint32_t step_seq, layer_base;
};
__device__ __forceinline__ A2AStep a2a_step_open(const McbCtx& c, const McbA2AStepArgs& a, int* s_cnt, int* s_prefix, int* s_max) {
  volatile uint32_t* state = a.state;
  A2AStep st;
  st.step_seq = state[MCB_STATE_STEP_SEQ];
  st.layer_base = state[MCB_STATE_LAYER_BASE];
  const int L = a.num_layers;
  st.n = step_count_exchange(c, MCB_SITE_A2A_STEP_META, a.counts_off, st.step_seq, *a.n_local, a.cap, s_cnt, s_prefix, s_max);
  st.ep_max = *s_max;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.step_meta[0] = s_prefix[c.world];
    a.step_meta[1] = s_prefix[c.rank];
    a.step_meta[2] = st.ep_max;
    a.step_meta[4] = (int)(st.step_seq + 1u);
    a.step_meta[5] = L > 0 ? (int)((st.layer_base + (uint32_t)L - 1u) & 1u) : 0;
    a.step_meta[7] = (int)(st.layer_base + (uint32_t)L);     // stamp of the last layer's rows
  }
  return st;
}

template <bool EMU>
__global__ void __launch_bounds__(512) a2a_step_kernel(const __grid_constant__ McbCtx ctx_p,
                                                       const __grid_constant__ McbA2AStepArgs args_p,
                                                       const McbCtx* ectx, const McbA2AStepArgs* eargs) {
  const McbCtx& c = EMU ? ectx[blockIdx.y] : ctx_p;
  const McbA2AStepArgs& a = EMU ? eargs[blockIdx.y] : args_p;
  __shared__ int s_prefix[MCB_MAX_RANKS + 1];
  __shared__ int s_cnt[MCB_MAX_RANKS];
  __shared__ int s_max;
  const int W = c.world;
  pdl_wait();
  pdl_launch_dependents();
  const A2AStep st = a2a_step_open(c, a, s_cnt, s_prefix, &s_max);
  const int valid = s_prefix[W];
  LLShape shp;
  shp.xdata = a.fp8 ? a.hidden / 8 : a.hidden / 4;
  shp.scales = a.fp8 ? a.hidden / 256 : 0;
  shp.meta = (int)(a.meta_row_bytes >> 3);
  shp.xw = 1 + shp.xdata + shp.scales + shp.meta;
  shp.yw = a.hidden / 4;
  const bool ll = W > 1 && a.ll_rows > 0 && valid > 0 && valid <= a.ll_rows && (!a.fp8 || a.hidden % 256 == 0);
  if (blockIdx.x == 0 && threadIdx.x == 0) a.step_meta[6] = ll ? 1 : 0;
  if (ll) {
    packet_layers(c, a, shp, s_prefix, st.n, valid, st.layer_base);
  } else if (EMU && W == 1) {      // else a2a_alone_kernel
    barrier_alone(c, a, st.n, st.layer_base);
  } else {
    barrier_layers(c, a, st.n, st.ep_max, st.layer_base);
  }
  step_close(a.state, st.step_seq, st.layer_base + (uint32_t)a.num_layers);
}

// ---- a world of one -----------------------------------------------------------------------------------
// Nobody to wait for: a slice is delivered and combined in one go, with every load of it in flight at once.  The identity expert on
// bf16 rows returns the row just delivered, which is still in registers.  PL = packs per lane; a lane holds one expert id (topk at most 32, others take
// barrier_alone).  KEEP: loads may stay in L1 for the next layer of the slice (steps that write nothing that they read).
template <bool FP8, int PL, bool KEEP = false>
struct AloneSlice {
  const McbA2AStepArgs& a;
  const int lane, row_packs;
  const bool echo, has_id;
  int t, p0;
  bool head;                 // the row's first slice: its warp writes the metadata row
  const uint8_t *x, *y;
  uint8_t *out, *recv, *scales, *meta;
  const int64_t* ids;
  const float* ws;

  __device__ __forceinline__ AloneSlice(const McbA2AStepArgs& args)
      : a(args), lane(threadIdx.x & 31), row_packs(args.hidden / 8), echo(!FP8 && args.y_off == args.recv_x_off), has_id(lane < args.topk) {}
  __device__ __forceinline__ int slices() const { return (row_packs + 32 * PL - 1) / (32 * PL); }
  __device__ __forceinline__ void at(const McbCtx& c, long long item) {
    const int per_row = slices();
    t = (int)(item / per_row);
    p0 = (int)(item - (long long)t * per_row) * 32 * PL + lane;
    head = p0 == lane;
    const uint64_t row = (uint64_t)c.rank * a.cap + t, row_bytes = (uint64_t)a.hidden * 2;
    x = reinterpret_cast<const uint8_t*>(a.x) + t * row_bytes + p0 * 16;
    y = c.heap_local + a.y_off + row * row_bytes + p0 * 16;
    out = reinterpret_cast<uint8_t*>(a.out) + t * row_bytes + p0 * 16;
    recv = c.heap_local + a.recv_x_off + (FP8 ? row * a.hidden + p0 * 8 : row * row_bytes + p0 * 16);
    scales = c.heap_local + a.recv_scale_off + row * (uint64_t)(a.hidden / 128) * 4 + (p0 >> 4) * 4;
    meta = c.heap_local + a.recv_meta_off + row * a.meta_row_bytes + lane * 16;
    ids = a.topk_idx + (int64_t)t * a.topk + lane;
    ws = a.topk_w ? a.topk_w + (int64_t)t * a.topk + lane : nullptr;
  }
  __device__ __forceinline__ long long load_id(bool on) const { return on && has_id ? *reinterpret_cast<const volatile int64_t*>(ids) : 0; }
  __device__ __forceinline__ float load_weight(bool on) const {
    return on && has_id ? (ws ? *reinterpret_cast<const volatile float*>(ws) : 1.0f) : 0.0f;
  }
  // Whether the row goes anywhere.
  __device__ __forceinline__ bool sends(const McbCtx& c, long long id) const {
    const bool good = has_id && id >= 0 && id < a.num_experts;
    if (has_id && !good) report_error(c, MCB_ERR_ROUTING, MCB_SITE_A2A_STEP, blockIdx.x, (uint32_t)t, (uint32_t)id);
    return __any_sync(0xffffffffu, good);
  }
  // The metadata row, chunk by chunk from the lanes that hold its ids and weights.
  __device__ __forceinline__ void deliver_meta(uint64_t par, uint32_t stamp, long long id, float wt) const {
    const uint32_t my_id = has_id ? (uint32_t)id : 0xffffffffu, my_w = has_id ? __float_as_uint(wt) : 0u;
    auto slot = [&](int k) {                 // k up to 63: lanes wrap around
      const uint2 v = make_uint2(__shfl_sync(0xffffffffu, my_id, k), __shfl_sync(0xffffffffu, my_w, k));
      return k < a.topk ? v : make_uint2(0xffffffffu, 0u);
    };
    const uint2 first = slot(meta_slot(lane)), second = slot(2 * lane);
    if (lane < (int)(a.meta_row_bytes >> 4)) st_v4(meta + par * a.meta_par_stride, meta_chunk_of(lane, stamp, t, first, second));
  }
  __device__ __forceinline__ void load(bool on, uint64_t par, uint4 (&v)[PL], uint4 (&w)[PL], long long& id, float& wt) const {
#pragma unroll
    for (int u = 0; u < PL; ++u) {
      const bool live = on && p0 + u * 32 < row_packs;
      auto ld = [](const uint8_t* p) { return KEEP ? ld_v4(p) : ld_v4_stream(p); };
      v[u] = live ? ld(x + u * 512) : make_uint4(0, 0, 0, 0);
      if (!echo) w[u] = live ? ld(y + par * a.y_par_stride + u * 512) : make_uint4(0, 0, 0, 0);
    }
    id = load_id(on);
    wt = load_weight(on && head);
  }
  __device__ __forceinline__ void deliver(const McbCtx& c, uint64_t par, uint32_t stamp, const uint4 (&v)[PL], const uint4 (&w)[PL], long long id,
                                          float wt) const {
    const bool sent = sends(c, id);
    if (sent) {
      uint8_t* dst = recv + par * a.x_par_stride;
      if (FP8) {
        float scale[PL + 1];
#pragma unroll
        for (int u = 0; u < PL; u += 2) block_absmax_pair(v[u], v[u + 1 < PL ? u + 1 : u], scale[u], scale[u + 1]);
#pragma unroll
        for (int u = 0; u < PL; ++u) {
          scale[u] = e4m3_scale(scale[u]);
          const uint2 q = quant_pack_e4m3(v[u], scale[u]);
          if (p0 + u * 32 >= row_packs) continue;
          st_v2(dst + u * 256, q);
          if ((lane & 15) == 0) st_b32(scales + par * a.scale_par_stride + u * 8, __float_as_uint(scale[u]));
        }
      } else {
#pragma unroll
        for (int u = 0; u < PL; ++u)
          if (p0 + u * 32 < row_packs) st_v4(dst + u * 512, v[u]);
      }
      if (head) deliver_meta(par, stamp, id, wt);
    }
    // the sum over one destination's row
#pragma unroll
    for (int u = 0; u < PL; ++u) {
      if (p0 + u * 32 >= row_packs) continue;
      float acc[8] = {};
      if (sent) acc_bf16x8(acc, echo ? v[u] : w[u]);
      st_v4(out + u * 512, make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                                      pack_bf16x2(acc[6], acc[7])));
    }
  }
};

// The sum over one destination's row, as the fp32 accumulation from zero rounds it: 0 + v, which drops the sign of a zero.  bf16 adds two
// values exactly where one of them is zero, so it takes one instruction for two values.
__device__ __forceinline__ uint4 alone_sum(bool sent, uint4 v) {
  const uint4 zero = make_uint4(0, 0, 0, 0);
  return sent ? add_bf16x8(v, zero) : zero;
}

// The layers of a step that writes nothing that it reads (a.apart), dealt to the warps; topk at most 32.
//   pieces   32 packs of a row (64 to quantise, two per lane) and their layers.  All layers of a parity deliver the same rows, so these
//            need no order: every warp takes a run of (piece, layer), a piece's layers one after the other.
//   chains   what a layer leaves behind of its own, layer after layer by one warp: the metadata row of a token and parity, which
//            carries the number of its layer, and 32 packs of a row of sums over expert outputs, which alternate between two buffers.  (The identity
//            expert on bf16 rows returns the row: its sums are the pieces' own.)
// A warp with one chain more than others takes fewer pieces.  Large steps are bound by the stores that leave L1 (below) or, with e4m3 rows, by the
// instructions of the quantisation; the loads may stay in L1, where 95 % of their sectors hit (24 layers of 333 e4m3 rows of 7168).  With the hint that
// keeps them out, e4m3 steps of 333 to 2048 rows of 7168 were 15 to 20 % slower.
// One B200, 58 layers, layer after layer (alone_many) -> dealt, 1 / 37 / 333 / 2048 rows, us a step:
//   1024 values  bf16 55 -> 5.5 / 57 -> 6.8 / 58 -> 12.1 / 87 -> 48     e4m3 84 -> 6.2 / 86 -> 7.2 / 87 -> 15.6 / 132 -> 73
//   7168 values  bf16 54 -> 5.5 / 57 -> 9.2 / 93 -> 46 / 752 -> 245     e4m3 84 -> 6.2 / 86 -> 12.7 / 125 -> 75 / 911 -> 427
// With one chain for both parities of a metadata row, its chunks put together by shuffles, the smallest steps took 16.7 and 14.6 us.
// The ids asked for in every layer again, or more layers in flight than here, were 10 to 25 % slower with e4m3 rows.  Slower than slices
// remain e4m3 steps of five layers, by up to 14 % at some sizes.
// Steps of bf16 rows are bound by the stores that leave L1, where stores to the same rows merge.  So of eight layers of a piece in flight those to the
// received rows of one parity come first, then those of the other, then the sums; and from kHalfLayers layers on half of the warps take part, whose rows are
// still in L1 more often.  All warps -> half of them, us a step (in brackets: (piece, layer) items for each of all warps):
//   58 layers   1024 values, 1 / 150 (15) / 333 (33) / 2048 rows 6.3 -> 6.1, 8.6 -> 9.1, 13.2 -> 12.1, 56.6 -> 47.8;  7168 values, 20 (14) / 2048 7.5 -> 7.2, 331 -> 246
//   48 layers   1024 values, the same rows 5.5 -> 5.2, 7.5 -> 7.9, 11.5 -> 10.8, 47.2 -> 40.8;  2048 values, 20 / 150 (24) / 2048 6.4 -> 6.0, 9.9 -> 9.9, 83.6 -> 66.7
//               768 values, 333 (20) / 2048 9.6 -> 9.8, 34.1 -> 32.1;  7168 values, 20 / 2048 6.8 -> 6.5, 270 -> 206
//   40 layers   768 values, 333 (17) / 1000 (51) / 2048 (104) 8.4 -> 8.9, 15.9 -> 16.3, 28.8 -> 28.3;  1024 values, 150 (10) / 1000 (68) 6.8 -> 7.2, 21.0 -> 20.0
//               7168 values, 20 (9) / 150 (71) / 2048 6.4 -> 6.2, 20.3 -> 17.8, 221 -> 177
//   26 layers   768 values, 333 / 2048 6.9 -> 7.6, 20.2 -> 22.0;  1024 values, 150 / 2048 6.3 -> 7.3, 26.2 -> 26.4;  7168 values, 333 / 2048 27.9 -> 24.3, 139 -> 133
// From 48 layers on half is better but for some 10 to 25 items a warp, by up to 6 %.  Below, large steps of long rows would gain too, but a line that depends
// on the number of rows costs every small step 0.1 us.  With expert outputs of their own, whose sums are chains, half is up to 17 % slower at 10 to 35 items
// a warp (48 layers of 150 rows of 1024 8.2 -> 9.6) and up to 25 % faster beyond (88 layers of 333 rows of 7168 108 -> 80). (e4m3 rows, bound by their
// instructions, take their layers as they come.)
constexpr int kHalfLayers = 48;
template <bool FP8>
__device__ __forceinline__ void alone_dealt(const McbCtx& c, const McbA2AStepArgs& a, int n, uint32_t layer_base) {
  constexpr int K = FP8 ? 2 : 1;             // packs per lane of a piece
  // A (piece, layer) against a layer of sums; a layer of metadata, which loads ids and weights and votes, counts as two.  Measured with 1 to 6,
  // 58 layers of 1 to 2048 rows: e4m3 pieces with 2 instead of 5 up to 25 % slower (333 rows of 1024 19.7 against 24.6 us, 150 rows of 7168 46.0
  // against 51.7), 4 and 6 the same within 2 %; bf16 pieces with 1 up to 7 % slower, with 3 and 4 2 % either way.  Metadata counted as one: the
  // smallest steps 0.2 us slower, others 5 % either way.
  constexpr int kCost = FP8 ? 5 : 2;
  AloneSlice<FP8, 1> s(a);
  const int lane = s.lane, L = a.num_layers, per_row = (s.row_packs + 32 * K - 1) / (32 * K);
  unsigned used = blockDim.x >> 5;                       // warps of a block that take part
  if constexpr (!FP8) {
    if (L >= kHalfLayers) used = (used + 1) / 2;
    if (threadIdx.x >> 5 >= used) return;
  }
  const long long warps = (long long)gridDim.x * used, warp = blockIdx.x + (long long)(threadIdx.x >> 5) * gridDim.x;
  const long long sums = s.echo ? 0 : (long long)n * s.slices(), chains = sums + 2ll * n, items = (long long)n * per_row * L;
  const uint64_t row_bytes = (uint64_t)a.hidden * 2;

  auto chain = [&] {
    for (long long k = warp; k < chains; k += warps) {
      const bool sum = k < sums;
      s.at(c, sum ? k : (k - sums >> 1) * s.slices());
      if (sum) {
        constexpr int D = 8;
        const bool live = s.p0 < s.row_packs, sent = s.sends(c, s.load_id(true));
        for (int l0 = 0; l0 < L; l0 += D) {
          uint4 v[D];
#pragma unroll
          for (int d = 0; d < D; ++d)
            v[d] = live && l0 + d < L ? ld_v4(s.y + ((layer_base + (uint32_t)(l0 + d)) & 1u ? a.y_par_stride : 0)) : make_uint4(0, 0, 0, 0);
#pragma unroll
          for (int d = 0; d < D; ++d)
            if (live && l0 + d < L) st_v4(s.out, alone_sum(sent, v[d]));
        }
      } else {
        // A chunk of the row by each lane, which reads the two ids and weights in it itself.
        const uint32_t par = (uint32_t)(k - sums) & 1u;
        const int k0 = meta_slot(lane), k1 = 2 * lane;
        const bool have0 = k0 < a.topk, have1 = k1 < a.topk, mine = lane < (int)(a.meta_row_bytes >> 4);
        const int64_t* ids = a.topk_idx + (int64_t)s.t * a.topk;
        const float* ws = a.topk_w ? a.topk_w + (int64_t)s.t * a.topk : nullptr;
        uint8_t* meta = s.meta + (par ? a.meta_par_stride : 0);
        constexpr int D = 8;
        for (int l0 = (int)((layer_base ^ par) & 1u); l0 < L; l0 += 2 * D) {
          uint2 id[D][2];
          uint32_t wt[D][2];
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const bool on = l0 + 2 * d < L;
            id[d][0] = on && have0 ? ld_v2(ids + k0) : make_uint2(~0u, ~0u);
            id[d][1] = on && have1 ? ld_v2(ids + k1) : make_uint2(~0u, ~0u);
            wt[d][0] = on && have0 ? (ws ? ld_b32(ws + k0) : __float_as_uint(1.0f)) : 0u;
            wt[d][1] = on && have1 ? (ws ? ld_b32(ws + k1) : __float_as_uint(1.0f)) : 0u;
          }
#pragma unroll
          for (int d = 0; d < D; ++d) {
            if (l0 + 2 * d >= L) break;
            const bool good0 = id[d][0].y == 0u && id[d][0].x < (uint32_t)a.num_experts, good1 = id[d][1].y == 0u && id[d][1].x < (uint32_t)a.num_experts;
            if (have0 && !good0) report_error(c, MCB_ERR_ROUTING, MCB_SITE_A2A_STEP, blockIdx.x, (uint32_t)s.t, id[d][0].x);
            if (have1 && !good1) report_error(c, MCB_ERR_ROUTING, MCB_SITE_A2A_STEP, blockIdx.x, (uint32_t)s.t, id[d][1].x);
            if (!__any_sync(0xffffffffu, good0 || good1) || !mine) continue;
            const uint32_t stamp = layer_base + (uint32_t)(l0 + 2 * d) + 1u;
            st_v4(meta, meta_chunk_of(lane, stamp, s.t, make_uint2(id[d][0].x, wt[d][0]), make_uint2(id[d][1].x, wt[d][1])));
          }
        }
      }
    }
  };

  auto pieces = [&] {
    // The first `extra` warps have a chain more and take `fewer` items fewer, or none where there are not enough.  The fewer warps of the two
    // kinds take whole numbers, the others share what remains: where those with a chain more did at any rate, the rest of 2360 warps went to 8,
    // and five layers of 1180 bf16 rows of 1024 took 63.6 us instead of 9.4.
    const long long extra = chains % warps, fewer = (L + kCost / 2) / kCost, virt = items + fewer * extra;
    const long long least = virt >= fewer * warps ? virt / warps - fewer : 0;
    const bool few = 2 * extra <= warps || least == 0;
    const long long whole = few ? least : least + fewer, shared = items - whole * (few ? extra : warps - extra), sharers = few ? warps - extra : extra;
    const long long each = shared / sharers, more = shared - each * sharers, k = few ? warp - extra : warp;
    const bool mine = (warp < extra) == few;               // a whole number of items
    const long long begin = mine ? (few ? whole * warp : shared + whole * (warp - extra)) : (few ? whole * extra : 0) + each * k + (k < more ? k : more);
    local_runs(begin, begin + (mine ? whole : each + (k < more)), L, [&](long long piece, int first, int last) {
      constexpr int D = FP8 ? 2 : 8;
      s.at(c, (piece / per_row) * s.slices());                                       // its row
      const int p = (int)(piece % per_row) * 32 * K + lane * K;
      const bool live = p < s.row_packs;
      const uint64_t row = (uint64_t)c.rank * a.cap + s.t;
      const uint8_t* src = reinterpret_cast<const uint8_t*>(a.x) + s.t * row_bytes + p * 16;
      uint8_t* out = reinterpret_cast<uint8_t*>(a.out) + s.t * row_bytes + p * 16;
      uint8_t* recv = c.heap_local + a.recv_x_off + (FP8 ? row * a.hidden + p * 8 : row * row_bytes + p * 16);
      uint8_t* scales = c.heap_local + a.recv_scale_off + (row * (a.hidden / 128) + (p >> 4)) * 4;
      const bool sent = s.sends(c, s.load_id(true));                                  // its layers have the same ids
      for (int l0 = first; l0 < last; l0 += D) {
        uint4 v[D][K];
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
          for (int k = 0; k < K; ++k) v[d][k] = live && l0 + d < last ? ld_v4(src + k * 16) : make_uint4(0, 0, 0, 0);
        if constexpr (FP8) {
#pragma unroll
          for (int d = 0; d < D; d += 2) {
            auto at = [&](uint8_t* base, uint64_t par_stride, int k) { return base + ((layer_base + (uint32_t)(l0 + d + k)) & 1u ? par_stride : 0); };
            quant_wide_pair(v[d], v[d + 1], [&](int k) { return l0 + d + k < last && sent && live; }, [&](int k, uint4 q, float scale) {
              st_v4(at(recv, a.x_par_stride, k), q);
              if ((lane & 7) == 0) st_b32(at(scales, a.scale_par_stride, k), __float_as_uint(scale));
            });
          }
        } else {
#pragma unroll
          for (int odd_layer = 0; odd_layer < 2; ++odd_layer) {
            uint8_t* dst = recv + ((layer_base + (uint32_t)(l0 + odd_layer)) & 1u ? a.x_par_stride : 0);
#pragma unroll
            for (int d = odd_layer; d < D; d += 2)
              if (l0 + d < last && live && sent) st_v4(dst, v[d][0]);
          }
          // Left at the first that is not there: with eight predicated sums small steps of five layers and more took 0.2 us more (8 layers of
          // 20 / 150 rows of 1024 4.9 / 6.0 -> 4.7 / 5.7 us), 150 rows of 7168 5 % more (7.8 -> 7.4).
#pragma unroll
          for (int d = 0; d < D; ++d) {
            if (l0 + d >= last || !live || !s.echo) break;
            st_v4(out, alone_sum(sent, v[d][0]));
          }
        }
      }
    });
  };
  // Half of the warps of an SM begin with their chains.
  const int odd = (int)(threadIdx.x >> 5) & 1;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    if (k == odd) chain();
    else pieces();
  }
}

// A warp takes a slice of a row and, D at a time, all its layers; steps that write nothing that they read.
template <bool FP8, int PL, int D>
__device__ __forceinline__ void alone_slices(const McbCtx& c, const McbA2AStepArgs& a, int n, uint32_t layer_base) {
  AloneSlice<FP8, PL, !FP8> s(a);       // e4m3 rows kept in L1: one or two layers of 2048 rows of 7168 3 to 6 % slower
  const long long mine = (long long)n * s.slices(), step = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long i = blockIdx.x + (long long)(threadIdx.x >> 5) * gridDim.x; i < mine; i += step) {
    s.at(c, i);
#pragma unroll 1
    for (int l0 = 0; l0 < a.num_layers; l0 += D) {
      uint4 v[D][PL], w[D][PL];
      long long id[D];
      float wt[D];
#pragma unroll
      for (int d = 0; d < D; ++d) s.load(l0 + d < a.num_layers, (layer_base + (uint32_t)(l0 + d)) & 1u, v[d], w[d], id[d], wt[d]);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        if (l0 + d >= a.num_layers) break;
        s.deliver(c, (layer_base + (uint32_t)(l0 + d)) & 1u, layer_base + (uint32_t)(l0 + d) + 1u, v[d], w[d], id[d], wt[d]);
      }
    }
  }
}

// A step of up to this many layers has too few of one piece to keep loads in flight: there the warps take slices, of one pack per lane
// or two where that still gives every slice a warp of its own, else of four (four instead of two: 811 e4m3 rows of 1024 15 to 25 % slower).  Kernels of their
// own, for one layer (D = 1) and for more (D = 2), which are smaller than that of the dealt steps.  One B200, a step of 1 / 2 / 3 / 4 layers in a row of
// steps, dealt -> slices:
//   hidden 1024 and top-22, 64 rows     bf16 4.7 / 4.7 / 4.8 / 4.7 -> 4.2 / 4.3 / 4.7 / 4.6          e4m3 4.9 / 5.0 / 4.9 / 5.0 -> 4.1 / 4.5 / 5.1 / 5.5 us
//                          512 rows     bf16 5.7 / 5.7 / 5.9 / 5.9 -> 4.3 / 4.3 / 4.8 / 5.0          e4m3 6.1 / 6.4 / 7.2 / 7.4 -> 4.3 / 4.8 / 5.5 / 6.0
//                          8192 rows    bf16 23.4 / 25.4 / 27.2 / 28.5 -> 9.9 / 14.7 / 20.0 / 24.9   e4m3 36.2 / 39.9 / 44.0 / 46.4 -> 12.8 / 19.9 / 26.7 / 32.1
//   hidden 7168 and top-8, 2048 rows    bf16 37.0 / 42.5 / 43.8 / 44.6 -> 16.1 / 24.1 / 31.1 / 38.9  e4m3 56.9 / 62.9 / 68.7 / 72.7 -> 20.6 / 32.6 / 44.2 / 53.4
// Four layers at a time, or eight, were 3 to 40 % slower than two.
constexpr int kFewLayers = 4;
template <bool FP8, int D>
__device__ __forceinline__ void alone_few(const McbCtx& c, const McbA2AStepArgs& a, int n, uint32_t layer_base) {
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5), packs = a.hidden / 8;
  if (n * ((packs + 31) / 32) <= warps) alone_slices<FP8, 1, D>(c, a, n, layer_base);
  else if (n * ((packs + 63) / 64) <= warps) alone_slices<FP8, 2, D>(c, a, n, layer_base);
  else alone_slices<FP8, 4, D>(c, a, n, layer_base);
}

// Whether a step of the identity expert on bf16 rows with five or six layers goes by slices of four packs per lane, where a slice is a whole row.  It writes
// its row, its sums and its metadata in one go, which saves a dealt step's addresses, but it is all layers of a row: a last round of warps that is less than
// 5/6 full is waited for, and where rows are longer, or a warp gets more of them, dealt pieces keep more loads in flight and more of their stores merge. One
// B200, us a step, dealt -> slices, one / two / three rounds of warps (0.96 full):
//   five layers   256 values 7.3 -> 5.8 / 10.3 -> 8.6 / 13.6 -> 11.9        512 values 8.9 -> 7.8 / 12.9 -> 11.8 / 16.4 -> 15.7
//                 768 values 10.1 -> 9.2 / 15.2 -> 14.9 / 19.6 -> 20.0      1024 values 11.2 -> 10.7 / 17.3 -> 17.7 / 23.0 -> 24.5
//   six layers    256 values 7.8 -> 6.7 / 10.5 -> 9.2 / 13.5 -> 12.4        512 values 8.6 -> 8.4 / 13.2 -> 13.2 / 17.3 -> 18.1
//                 768 values 9.9 -> 10.0 / 15.5 -> 16.9 / 20.0 -> 23.2      1024 values 11.1 -> 11.7 / 17.6 -> 20.2 / 23.7 -> 29.0
// Two slices to a row and more: 2048 values, five layers 9.8 -> 10.1 / 15.4 -> 17.3; 7168 values, 324 / 974 rows 9.5 -> 10.3 / 18.3 -> 23.3; six layers
// 15 to 45 % slower; only where the rows in and out no longer stay in L2 (93 MB, five layers) 0 to 3 % faster.  Seven layers: dealt everywhere.
// The line is at so many values for a warp; the host takes the rest out (kSliceLayers), so that the kernel's other way stays as it is.
constexpr int kSliceLayers = 6, kSliceValuesFive = 1536, kSliceValuesSix = 512;
__device__ __forceinline__ bool alone_by_slices(const McbA2AStepArgs& a, int n) {
  const unsigned warps = gridDim.x * (blockDim.x >> 5), items = (unsigned)n * (unsigned)((a.hidden / 8 + 127) / 128);
  const bool full = a.y_off == a.recv_x_off && items * 6ull >= (items + warps - 1) / warps * 5ull * warps;
  return full && (unsigned long long)items * (unsigned)a.hidden <=
                     (unsigned long long)warps * (a.num_layers < kSliceLayers || a.hidden <= 256 ? kSliceValuesFive : kSliceValuesSix);
}

// Layer after layer: steps that read what they write.
template <bool FP8>
__device__ __forceinline__ void alone_many(const McbCtx& c, const McbA2AStepArgs& a, int n, uint32_t layer_base) {
  AloneSlice<FP8, 4> s(a);
  const long long mine = (long long)n * s.slices(), step = (long long)gridDim.x * (blockDim.x >> 5);
  for (int l = 0; l < a.num_layers; ++l)
    for (long long i = blockIdx.x + (long long)(threadIdx.x >> 5) * gridDim.x; i < mine; i += step) {
      uint4 v[4], w[4];
      long long id;
      float wt;
      s.at(c, i);
      s.load(true, (layer_base + (uint32_t)l) & 1u, v, w, id, wt);
      s.deliver(c, (layer_base + (uint32_t)l) & 1u, layer_base + (uint32_t)l + 1u, v, w, id, wt);
    }
}

// The step of a world of one, a kernel of its own for each way: everything is inline, so the arguments are read from the constant bank and not
// through pointers after every store.  D: as in alone_few; kDealt: more layers; kDealtOrSlices: alone_by_slices; kInOrder: steps that read what they write,
// more than 32 ids.  With the last in the kernel of dealt steps, these had 24 bytes of stack and e4m3 ones were slower: 58 layers of 333 rows of 7168 82.2 ->
// 78.1 us, 88 layers of one / 37 / 2048 rows of 1024 7.9 / 9.5 / 115 -> 7.2 / 8.7 / 110.  (More or fewer than 16 warps per block: 3 to 10 % slower with e4m3
// rows.)
constexpr int kInOrder = 0, kDealt = -1, kDealtOrSlices = -2;
template <bool FP8, int D>
__global__ void __launch_bounds__(512, 1) a2a_alone_kernel(const __grid_constant__ McbCtx c, const __grid_constant__ McbA2AStepArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ int s_prefix[2], s_cnt[1], s_max;
  const A2AStep st = a2a_step_open(c, a, s_cnt, s_prefix, &s_max);
  if (blockIdx.x == 0 && threadIdx.x == 0) a.step_meta[6] = 0;
  // The order of the ways is that of their code, and small steps feel it: slices behind dealt pieces cost them 0.1 us, before them 0.25.
  if constexpr (D == kInOrder) {
    if (a.topk > 32) barrier_alone(c, a, st.n, st.layer_base);
    else alone_many<FP8>(c, a, st.n, st.layer_base);
  } else if constexpr (D > 0) {
    alone_few<FP8, D>(c, a, st.n, st.layer_base);
  } else {
    if (D == kDealt || !alone_by_slices(a, st.n)) alone_dealt<FP8>(c, a, st.n, st.layer_base);
    else if constexpr (D != kDealt) alone_slices<FP8, 4, 2>(c, a, st.n, st.layer_base);
  }
  step_close(a.state, st.step_seq, st.layer_base + (uint32_t)a.num_layers);
}

}  // namespace mcb

using namespace mcb;

extern "C" {

int mcb_sizeof_a2a_step_args() { return (int)sizeof(McbA2AStepArgs); }

static int check_a2a_step(const McbCtx* ctx, const McbA2AStepArgs* a, int grid, int threads) {
  if (!ctx || !a || grid < 1 || grid > MCB_MAX_BLOCKS || threads < 32 || threads > 512 || (threads & 31)) return 1;
  if (!a->x || !a->topk_idx || !a->out || !a->n_local || !a->state || !a->step_meta) return 1;
  if (a->hidden < 8 || a->hidden % 8 || (a->fp8 && a->hidden % 128) || a->topk < 1 || a->cap < 1 || a->num_layers < 0) return 1;
  if (ctx->world < 1 || a->num_experts % ctx->world) return 1;
  if ((a->meta_row_bytes & 15u) || a->meta_row_bytes < 8u + 8u * (uint32_t)a->topk) return 1;
  if (a->ll_rows > 0 && (!a->ll_x_off || !a->ll_y_off || !a->credit_off || a->ll_src_rows < 1 || a->hidden % 4)) return 1;
  return 0;
}

// Whether a step in a world of one writes nothing that it reads (an output on its input, expert outputs among received rows),
// and no row by two ways: its layers may then run into each other.
int mcb_a2a_step_apart(const McbCtx* ctx, const McbA2AStepArgs* a) {
  if (ctx->world != 1) return 0;
  struct Range { uint64_t at, bytes; };
  auto meet = [](Range x, Range y) { return x.at && y.at && x.bytes && y.bytes && x.at < y.at + y.bytes && y.at < x.at + x.bytes; };
  auto at = [](const void* p) { return reinterpret_cast<uint64_t>(p); };
  const uint64_t heap = at(ctx->heap_local), cap = (uint64_t)a->cap, row = (uint64_t)a->hidden * 2;
  const bool echo = !a->fp8 && a->y_off == a->recv_x_off;
  const Range reads[] = {{at(a->x), cap * row}, {at(a->topk_idx), cap * a->topk * 8}, {at(a->topk_w), cap * a->topk * 4},
                         {heap + a->y_off, echo ? 0 : a->y_par_stride + cap * row}};
  const Range writes[] = {{at(a->out), cap * row}, {heap + a->recv_x_off, a->x_par_stride + cap * (a->fp8 ? row / 2 : row)},
                          {heap + a->recv_scale_off, a->fp8 ? a->scale_par_stride + cap * (a->hidden / 128) * 4 : 0},
                          {heap + a->recv_meta_off, a->meta_par_stride + cap * a->meta_row_bytes}};
  for (int w = 0; w < 4; ++w) {
    for (const Range& r : reads)
      if (meet(r, writes[w])) return 0;
    for (int v = 0; v < w; ++v)
      if (meet(writes[v], writes[w])) return 0;
  }
  return 1;
}

int mcb_launch_a2a_step(const McbCtx* ctx, const McbA2AStepArgs* args, int grid, int threads, int pdl,
                        cudaStream_t stream) {
  if (check_a2a_step(ctx, args, grid, threads)) return cudaErrorInvalidValue;
  McbA2AStepArgs a = *args;
  a.apart = mcb_a2a_step_apart(ctx, args);
  if (ctx->world == 1) {
    auto alone = [&](auto layers) {
      constexpr int D = decltype(layers)::value;
      auto kernel = a2a_alone_kernel<false, D>;
      if constexpr (D != kDealtOrSlices)
        if (a.fp8) kernel = a2a_alone_kernel<true, D>;
      return launch_kernel(kernel, dim3(grid), dim3(threads), 0, stream, pdl, false, *ctx, a);
    };
    if (!a.apart || a.topk > 32) return alone(std::integral_constant<int, kInOrder>{});
    if (a.num_layers > kFewLayers && a.num_layers <= kSliceLayers && !a.fp8 && a.hidden <= (a.num_layers < kSliceLayers ? 1024 : 512))
      return alone(std::integral_constant<int, kDealtOrSlices>{});
    if (a.num_layers > kFewLayers) return alone(std::integral_constant<int, kDealt>{});
    return a.num_layers > 1 ? alone(std::integral_constant<int, 2>{}) : alone(std::integral_constant<int, 1>{});
  }
  return launch_kernel(a2a_step_kernel<false>, dim3(grid), dim3(threads), 0, stream, pdl, false, *ctx, a,
                       (const McbCtx*)nullptr, (const McbA2AStepArgs*)nullptr);
}

int mcb_emu_a2a_step(const McbCtx* d_ctx, const McbA2AStepArgs* d_args, const McbCtx* h_ctx0,
                     const McbA2AStepArgs* h_args0, int world, int grid, int threads, cudaStream_t stream) {
  if (!d_ctx || !d_args || world < 1 || check_a2a_step(h_ctx0, h_args0, grid, threads)) return cudaErrorInvalidValue;
  McbCtx dummy{};
  McbA2AStepArgs dargs{};
  return launch_kernel(a2a_step_kernel<true>, dim3(grid, world), dim3(threads), 0, stream, 0, true, dummy, dargs,
                       d_ctx, d_args);
}

}  // extern "C"
