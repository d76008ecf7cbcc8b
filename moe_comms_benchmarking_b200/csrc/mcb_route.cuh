// Routing of the gathered tokens to this rank's experts as device functions (histogram -> offsets -> pair lists ->
// row-tile table), shared by the stand-alone routing kernel, the fused dispatch + routing + FC1 kernel and the
// whole-layer kernel.
//
// The (token, k) entries are shared out over the blocks in order.  A block needs two things beyond its own entries: how
// many entries each expert has in all (the offsets follow from these) and where its own entries of an expert begin.
//   few entries   every block counts ALL entries itself, and those before its share once more: no block waits for
//                 another, and every block has the offsets in shared memory at once;
//   many entries  a block counts its share and adds it to a counter per expert, which returns where its entries
//                 begin; after a barrier over the blocks everybody reads the counters.
// Either way every block then works out the offsets for itself (a block-wide scan over the experts) and places its own
// entries with cursors in shared memory.  Against counters handed over through one last block that scanned alone and one
// global atomic per entry: 28 -> 10 us inside the layer kernel at 90112 entries and 512 experts, and with one token the
// experts' weights start 8 us earlier.
#pragma once
#include "mcb_barrier.cuh"
#include "mcb_gemm.h"
#include "mcb_group.cuh"

namespace mcb {

constexpr int kMaxLocalExperts = 1024;
// Shared memory of a routing block: counts, own begins (later cursors), offsets, scan scratch.
constexpr int kRouteSmemWords = 3 * kMaxLocalExperts + 1 + 3 * 32;
// Entries per thread up to which every block counts all of them.  Either way forced, one B200, us a layer with 64 experts of
// 512 x 256 and top-8, all counted by every block (counts shared through global counters):
//   layer kernel, 512 threads      4096 entries 30.8 (34.6), 8192 35.9 (38.2), 12288 41.7 (42.3), 16384 47.4 (47.3), 24576 58.6 (56.4)
//   step, 64 threads of a block    1024 entries 14.5 (15.0), 2048 14.8 (15.3), 3072 15.9 (15.4), 4096 18.1 (16.2), 8192 25.8 (20.0)
// The line lies on the safe side of both crossings (about 32 and 40 entries per thread): beyond them counting all costs ever more.
constexpr int kRouteAllPerThread = 16;

struct RouteSmem {
  int *cnt, *begin, *off, *scan;
  __device__ __forceinline__ explicit RouteSmem(int* base)
      : cnt(base), begin(base + kMaxLocalExperts), off(base + 2 * kMaxLocalExperts), scan(base + 3 * kMaxLocalExperts + 1) {}
  __device__ __forceinline__ RouteSmem(int* cnt_, int* begin_, int* off_, int* scan_) : cnt(cnt_), begin(begin_), off(off_), scan(scan_) {}
};

// This block's share of the entries.
struct RouteShare {
  long long entries, lo, hi;
};
__device__ __forceinline__ RouteShare route_share(const McbRouteArgs& a, int block, int blocks) {
  int T = *a.num_tokens;
  if (T < 0) T = 0;
  if (T > a.max_tokens) T = a.max_tokens;
  RouteShare s;
  s.entries = (long long)T * a.topk;
  const long long per = (s.entries + blocks - 1) / blocks;
  s.lo = per * block < s.entries ? per * block : s.entries;
  s.hi = s.lo + per < s.entries ? s.lo + per : s.entries;
  return s;
}
template <class Group>
__device__ __forceinline__ bool route_counts_all(const Group& g, const RouteShare& s, int per_thread = kRouteAllPerThread) {
  return s.entries <= (long long)per_thread * g.size();
}

// Counts the entries [lo, hi) into m.cnt and, with SPLIT, those before `split` into m.begin too.  All threads of the group.
template <bool SPLIT, class Group>
__device__ __forceinline__ void route_count(const Group& g, const McbRouteArgs& a, const int64_t* topk_idx, const RouteSmem& m, long long lo,
                                            long long hi, long long split) {
  const int tid = g.tid(), E = a.num_local_experts;
  const unsigned threads = g.size();
  for (int e = tid; e < E; e += threads) { m.cnt[e] = 0; m.begin[e] = 0; }
  g.sync();
  for (long long i0 = lo + tid; i0 < hi; i0 += threads * 4) {
    long long e[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * threads;
      e[u] = i < hi ? topk_idx[i] - a.expert_begin : -1;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (e[u] >= 0 && e[u] < E) {
        atomicAdd(&m.cnt[(int)e[u]], 1);
        if (SPLIT && i0 + u * threads < split) atomicAdd(&m.begin[(int)e[u]], 1);
      }
  }
  g.sync();
}

// Many entries, before the barrier: this block's counts into the counters; m.begin = where its entries begin.
template <class Group>
__device__ __forceinline__ void route_publish(const Group& g, int E, int* expert_count, const RouteSmem& m) {
  for (int e = g.tid(); e < E; e += g.size())
    m.begin[e] = m.cnt[e] ? atomicAdd(&expert_count[e], m.cnt[e]) : 0;
}
// ... and after it: the counts of all blocks.
template <class Group>
__device__ __forceinline__ void route_collect(const Group& g, int E, const int* expert_count, const RouteSmem& m) {
  for (int e = g.tid(); e < E; e += g.size())
    m.cnt[e] = *reinterpret_cast<const volatile int*>(&expert_count[e]);
  g.sync();
}

// Offsets of the experts (exclusive prefix of m.cnt) into m.off[0 .. E] by a block-wide scan; the block that `writes` puts
// them, the 128-row tile table of the tokens-as-rows GEMMs, the largest count and the zeroed "gate/up done" counters of
// the fused FFN into global memory.  Returns the largest count in every thread.  All threads of the group.
template <class Group>
__device__ __forceinline__ int route_offsets(const Group& g, const McbRouteArgs& a, const RouteSmem& m, bool writes) {
  const int tid = g.tid(), E = a.num_local_experts, warp = tid >> 5, lane = tid & 31, nw = (int)(g.size() >> 5);
  const int per = (E + (int)g.size() - 1) / (int)g.size();
  const int e0 = tid * per, e1 = e0 + per < E ? e0 + per : E;
  int rows = 0, tiles = 0, mx = 0;
  for (int e = e0; e < e1; ++e) {
    const int c = m.cnt[e];
    rows += c;
    tiles += (c + 127) >> 7;
    mx = c > mx ? c : mx;
  }
  int r_inc = rows, t_inc = tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int r = __shfl_up_sync(0xffffffffu, r_inc, o), t = __shfl_up_sync(0xffffffffu, t_inc, o);
    if (lane >= o) { r_inc += r; t_inc += t; }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 31) { m.scan[warp] = r_inc; m.scan[32 + warp] = t_inc; m.scan[64 + warp] = mx; }
  g.sync();
  // Every warp scans the warps' sums for itself, lane w holding those of warp w.
  int run = r_inc - rows, tile = t_inc - tiles;
  r_inc = lane < nw ? m.scan[lane] : 0;
  t_inc = lane < nw ? m.scan[32 + lane] : 0;
  mx = __reduce_max_sync(0xffffffffu, lane < nw ? m.scan[64 + lane] : 0);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int r = __shfl_up_sync(0xffffffffu, r_inc, o), t = __shfl_up_sync(0xffffffffu, t_inc, o);
    if (lane >= o) { r_inc += r; t_inc += t; }
  }
  const int total = __shfl_sync(0xffffffffu, r_inc, 31), total_tiles = __shfl_sync(0xffffffffu, t_inc, 31);
  const int r_before = __shfl_sync(0xffffffffu, r_inc, warp ? warp - 1 : 0), t_before = __shfl_sync(0xffffffffu, t_inc, warp ? warp - 1 : 0);
  if (warp) { run += r_before; tile += t_before; }
  for (int e = e0; e < e1; ++e) {
    const int c = m.cnt[e];
    m.off[e] = run;
    if (writes) {
      a.expert_offset[e] = run;
      if (a.ffn_done) a.ffn_done[e] = 0;
      for (int r0 = 0; r0 < c; r0 += 128, ++tile) {
        if (tile < a.max_tiles) {
          a.tile_expert[tile] = e;
          a.tile_row0[tile] = run + r0;
          a.tile_rows[tile] = c - r0 < 128 ? c - r0 : 128;
        }
      }
    }
    run += c;
  }
  if (tid == 0) {
    m.off[E] = total;
    if (writes) {
      a.expert_offset[E] = total;
      if (a.max_rows) *a.max_rows = mx;
      if (total_tiles > a.max_tiles || total > a.max_pairs) {
        if (a.status && atomicCAS(a.status, 0u, (uint32_t)MCB_ERR_CAPACITY) == 0u) {
          a.status[1] = 100; a.status[2] = (uint32_t)total_tiles; a.status[3] = (uint32_t)total;
        }
      }
      *a.num_m_tiles = total_tiles < a.max_tiles ? total_tiles : a.max_tiles;
    }
  }
  g.sync();
  return mx;
}

// Places this block's entries: pair row = offset of the expert + where the block's entries of it begin + a cursor (m.begin
// is used up).  All threads of the group.
template <class Group>
__device__ __forceinline__ void route_place(const Group& g, const McbRouteArgs& a, const int64_t* topk_idx, const float* topk_w,
                                            const RouteSmem& m, const RouteShare& s) {
  const int E = a.num_local_experts;
  const unsigned threads = g.size();
  for (long long i0 = s.lo + g.tid(); i0 < s.hi; i0 += threads * 4) {
    long long e[4];
    float w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * threads;
      e[u] = i < s.hi ? topk_idx[i] - a.expert_begin : -1;
      w[u] = i < s.hi && topk_w ? topk_w[i] : 1.0f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * threads;
      if (i >= s.hi) break;
      int pos = -1;
      if (e[u] >= 0 && e[u] < E) {
        pos = m.off[(int)e[u]] + atomicAdd(&m.begin[(int)e[u]], 1);
        if (pos < a.max_pairs) {
          a.pair_token[pos] = (int)(i / a.topk);
          a.pair_prob[pos] = w[u];
        } else {
          pos = -1;
        }
      }
      a.pair_pos[i] = pos;
    }
  }
}

// The whole routing by the blocks of a launch: one of its own, or the fused dispatch + FC1 kernel's.  With few entries nobody waits
// for another block: all count all entries and place their own (one block alone: 21.9 us a launch at 11264 entries of 512
// experts, now 5.8; 8.5 and 4.2 at 1408; 3.0 and 3.8 at 128 of 32, where the wider scan shows); with many the blocks wait for one
// another on a counter that only grows (the grid must be co-resident).  There a thread keeps its first kRouteKept entries from the
// counting to the placing, and the last block to have read the counters is found while the others place: 22528 / 45056 / 90112
// entries, 64 of 512 experts local, 10.4 -> 8.5 / 10.5 -> 8.5 / 10.6 -> 9.3 us (32 blocks of 1024 threads).
// Shares are runs of entries: with entries dealt to the blocks in turn, an expert's rows come in another order, and FFN and
// combine of 8191 tokens with Zipf routing were 2 % slower; asked for before the number of tokens is known, few entries took
// 8.4 us (7.2).  Call from all threads of every block; `smem` is kRouteSmemWords words of shared memory.
constexpr int kRouteKept = 4;
// Blocks of a launch of its own (ROUTE_GRID of the plan).  Blocks of 512 threads cost less to start and at each of their barriers than as many threads in
// blocks of 1024, and 96 of them read and place large batches sooner than 32.  One B200, us a launch in a row of them, 64 of 512 experts local:
//   entries                       352   1408   5632   8800   11264   15400   45056   90112   180202
//   32 blocks of 1024 threads     4.0    4.2    4.9    5.5     5.7     6.3     6.9     7.7      9.7
//   96 of 512                     3.3    3.5    4.6    5.4     5.9     5.9     6.0     6.7      6.5
//   64 of 512                     3.5    3.5    4.5    5.4     5.9     5.7     6.0     6.8      8.1
//   128 of 256 / of 512    3.2 / 3.3  3.7 / 3.6  5.3 / 4.6  5.5 / 5.8  5.7 / 6.1  5.7 / 6.0  6.0 / 6.2  6.7 / 6.8  7.8 / 6.5
// Blocks of 512 threads count all of up to 24 entries per thread, of up to 32 with more than 512 local experts, whose counters cost more.  All counted by
// every block (through the counters), us: 64 local experts 8800 entries 5.4 (5.7), 11264 5.9 (6.0), 15400 6.8 (5.9); 512 of them 11264 5.7 (6.2), 12200 5.8
// (6.7), 15400 6.5 (6.5); 1024 of them 12200 6.1 (7.1), 15400 6.8 (7.3).  (32 blocks of 1024 threads took 5.6 to 6.0 with 11264; asking for eight entries at
// a time instead of four brings these to 5.6 and everything below 9000 entries 5 to 8 % up, as a second loop for more than 10240 entries 0 to 2 %.) Callers
// that ask for fewer than 96 blocks get blocks of 1024 threads where the buffers hold more entries than 512 threads keep: 32 blocks of 512 / 1024 with 45056,
// 90112, 180202 entries 6.4 / 7.0, 8.2 / 7.5, 11.1 / 9.8 us; 8 blocks with 11264, 22528, 90112 6.1 / 6.8, 8.1 / 7.4, 16.1 / 12.9. The fused dispatch + FC1
// kernel (blocks of 320 threads) counts all of as many: a layer of 512 / 64 / 16 experts of 512 x 256 with 5632 entries 102.0 -> 98.7, 40.9 -> 40.4, 40.2 ->
// 39.8 us (16 per thread -> 24), with 7168 entries 102.7 -> 99.6, 43.3 -> 43.0, 41.9 -> 42.1.
constexpr int kRouteThreads = 512, kRouteWideThreads = 1024, kRouteBlocks = 96, kRouteAllAlone = 24, kRouteAllMany = 32;
__device__ __forceinline__ void route_device(const McbRouteArgs& a, int* smem, int all_per_thread = kRouteAllAlone) {
  const RouteSmem m(smem);
  const int tid = threadIdx.x, E = a.num_local_experts;
  const RouteShare s = route_share(a, (int)blockIdx.x, (int)gridDim.x);
  const BlockGroup g;
  if (route_counts_all(g, s, all_per_thread)) {
    if (s.lo >= s.hi && blockIdx.x != 0) return;
    route_count<true>(g, a, a.topk_idx, m, 0, s.entries, s.lo);
    route_offsets(g, a, m, blockIdx.x == 0);
    route_place(g, a, a.topk_idx, a.topk_w, m, s);
    return;
  }
  const int threads = (int)blockDim.x;
  const long long mine = s.lo + tid;                         // entries mine, mine + threads, ... of the block's share
  long long id[kRouteKept];
#pragma unroll
  for (int u = 0; u < kRouteKept; ++u) id[u] = mine + u * threads < s.hi ? a.topk_idx[mine + u * threads] : -1;
  for (int e = tid; e < E; e += blockDim.x) m.cnt[e] = 0;
  __syncthreads();
  int ex[kRouteKept];                                        // local expert, -1 of another rank, -2 no entry
  float w[kRouteKept];
#pragma unroll
  for (int u = 0; u < kRouteKept; ++u) {
    const long long i = mine + u * threads, e = id[u] - a.expert_begin;
    ex[u] = i >= s.hi ? -2 : e >= 0 && e < E ? (int)e : -1;
    if (ex[u] >= 0) atomicAdd(&m.cnt[ex[u]], 1);
    if (ex[u] == -1) a.pair_pos[i] = -1;
    w[u] = ex[u] >= 0 && a.topk_w ? a.topk_w[i] : 1.0f;
  }
  for (long long i = mine + kRouteKept * threads; i < s.hi; i += threads) {
    const long long e = a.topk_idx[i] - a.expert_begin;
    if (e >= 0 && e < E) atomicAdd(&m.cnt[(int)e], 1);
  }
  __syncthreads();
  route_publish(g, E, a.expert_count, m);
  __syncthreads();
  volatile int* arrived = a.sync;                            // back at zero when every block has read the counters
  if (tid == 0) {
    __threadfence();
    atomicAdd(&a.sync[0], 1);
    uint64_t t0 = 0;
    for (uint32_t i = 0; *arrived < (int)gridDim.x; ++i) {
      if ((i & 63u) != 63u) continue;
      if (t0 == 0) t0 = globaltimer_ns();
      if (globaltimer_ns() - t0 > a.timeout_ns) {
        if (a.status && atomicCAS(a.status, 0u, (uint32_t)MCB_ERR_TIMEOUT) == 0u) { a.status[1] = 101; a.status[2] = blockIdx.x; }
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  route_collect(g, E, a.expert_count, m);
  route_offsets(g, a, m, blockIdx.x == 0);
  int left = 0;                                              // blocks that have read the counters before this one
  if (tid == (int)blockDim.x - 32) left = atomicAdd(&a.sync[1], 1);
  auto place = [&](long long i, int e, float weight) {
    int pos = m.off[e] + atomicAdd(&m.begin[e], 1);
    if (pos < a.max_pairs) {
      a.pair_token[pos] = (int)(i / a.topk);
      a.pair_prob[pos] = weight;
    } else {
      pos = -1;
    }
    a.pair_pos[i] = pos;
  };
#pragma unroll
  for (int u = 0; u < kRouteKept; ++u)
    if (ex[u] >= 0) place(mine + u * threads, ex[u], w[u]);
  for (long long i = mine + kRouteKept * threads; i < s.hi; i += threads) {
    const long long e = a.topk_idx[i] - a.expert_begin;
    if (e >= 0 && e < E) place(i, (int)e, a.topk_w ? a.topk_w[i] : 1.0f);
    else a.pair_pos[i] = -1;
  }
  if (tid >= (int)blockDim.x - 32 && __shfl_sync(0xffffffffu, left, 0) == (int)gridDim.x - 1) {
    for (int e = tid - ((int)blockDim.x - 32); e < E; e += 32) a.expert_count[e] = 0;
    if (tid == (int)blockDim.x - 32) { a.sync[0] = 0; a.sync[1] = 0; }
  }
}

}  // namespace mcb
