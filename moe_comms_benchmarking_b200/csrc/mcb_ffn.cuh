// Grouped SwiGLU expert FFN on the 5th-generation tensor cores, from decode to prefill sizes, with the
// WEIGHTS as the M operand and the tokens of one expert as N.
//
// The reference has no expert computation at all (identity expert, bench_nvls.py:109-112).  A layer is
// bound by streaming 6 MB of weights per expert while experts see a handful of tokens, and by the tensor
// pipe once they see a few hundred; in between the limit is what the SMs can take from L2, because every
// weight block needs the rows of all tokens of its expert.  Hence:
//   * a CTA PAIR (cluster of two, cta_group::2) works on one M = 256 tile: each CTA streams 128 weight rows
//     and HALF of the token rows, so a token row enters the SMs once per 256 weight rows, and one thread of
//     the pair issues the MMAs of both SMs.  A work unit is 256 weight rows x the whole reduction length x
//     one chunk of up to 256 tokens of one expert; an expert's tokens are cut into equal chunks, rounded up
//     to 32, and the accumulators are double buffered in TMEM;
//   * every operand arrives by TMA: weights as 16 or 32 KB tiles (pre-packed once into the swizzled K-major
//     image of their shared-memory tile, so a tile is contiguous in memory), activations as boxes of rows.
//     Token rows come four at a time through the pair -> token list (tile::gather4, the routing permute fused
//     into the load) while an expert has at most kFfnGatherN tokens.  One gather costs its issuing thread about
//     100 cycles whatever it moves, which at many tokens is slower than the MMAs it feeds, so there the
//     rows are first copied into pair order (into the memory of the expert outputs, which an expert's down
//     units overwrite only after all its gate/up units have read it) and come as boxes too;
//   * work units are listed per CTA pair in shared memory before the roles start: experts without tokens are
//     left out of the numbering, so the pairs get equally many units whatever the routing, and a
//     popular expert's chunks spread over the chip;
//   * both projections run in one persistent stream.  While the activations of all experts fit in L2 the gate/up
//     units of every expert come first, then the down units; above that a down unit follows its gate/up
//     units at a distance of three rounds of the grid, while its activations are still in L2.  A down
//     unit waits for a counter of its expert's finished gate/up units; units are taken in list order, so the
//     wait cannot deadlock;
//   * the gate/up matrix is stored interleaved (row 2i = gate row i, row 2i + 1 = up row i): the two values
//     of an activation meet in neighbouring TMEM lanes and are exchanged with one shuffle;
//   * weights are loaded with an evict-first policy: a layer reads each of its weights once (the chunks of a weight block
//     are neighbours in time), and without it 138 MB of them threw the kernel's own code, its inputs, the pair lists and the
//     activations out of L2, so that every phase of the next layer began with trips to HBM.  88 layers of one token
//     4595 -> 3757 us (dispatch 6.8 -> 3.8, experts 30.0 -> 27.2, combine 5.8 -> 3.1 us a layer), a layer of 37 tokens
//     406 -> 384 us, of 190 wide tokens 454 -> 435 us, no difference at 4096.  Also with 8 sets of only 50 or 75 MB in use a
//     layer is faster with it (30.5 -> 28.1, 36.6 -> 33.4 us), and an expert of several chunks (16 experts at 375 tokens
//     47.6 -> 44.7); it costs only where ONE set of less than L2 is run again and again (75 MB 12.6 -> 17.3, 100 MB
//     18.3 -> 21.2), which no launch can know;
//   * weights and tokens have producer warps of their own, so the weight stream runs on while a down unit
//     waits; eight epilogue warps read the accumulators with tcgen05.ld (a lane holds one output feature),
//     turn them through a small shared-memory tile and store 16 bytes per lane, feature-contiguous;
//   * every mbarrier wait is bounded and reports through the status words.
// Measured on one B200 with 64 experts of 1024 x 1024 (402.7 MB of weights), against one CTA per unit of 128 weight rows
// with token rows copied by cp.async and units numbered over all experts: 64 us (66 before) at 3 tokens per expert,
// where the weight stream is the limit; 89 (113) at 173 and 157 (204) at 350 tokens per expert; with skewed routing
// (8191 tokens, Zipf 1.2) 222 (536).  With 22 of 512 experts in use 36 (52).  Launches of a few microseconds lose what a CTA
// pair costs to set up and take down, and to gather: 8 experts of 512 x 256 at 1 / 32 / 128 tokens per expert 8.3 / 9.6 /
// 12.9 us (7.2 / 7.7 / 10.4).
#pragma once
#include "mcb_tc.cuh"

namespace mcb {

constexpr int kFfnEpiWarps = 8;
constexpr int kFfnTokWarps = 2;
constexpr int kFfnThreads = 32 * (2 + kFfnEpiWarps + kFfnTokWarps);      // weight TMA, MMA, epilogue, token TMA
constexpr int kFfnRowsM = 256;              // weight rows per unit (128 in each CTA of the pair)
constexpr int kFfnBlockK = 64;              // 128 bytes of bf16
constexpr int kFfnMaxN = 256;               // tokens per chunk
// Largest chunk whose token rows are gathered by TMA.  64 experts of 1024 x 1024, largest 90 / 110 / 128 tokens: 66 / 67 / 70 us
// (70 / 71 / 75 with the copy into pair order from 65 on), 32 of 1024 x 512 at 64 tokens 24.3 (27.2), 8 of 7168 x 2048 at
// 110: 111 (117); no difference with one popular expert, whose size decides for all.
constexpr int kFfnGatherN = 128;
constexpr int kFfnDoubleN = 128;            // up to this many tokens per chunk a stage holds two 64-column blocks
constexpr int kFfnMaxStages = 10;
constexpr int kFfnABytes = 128 * kFfnBlockK * 2;                 // 16 KiB of weights per CTA and 64-column block
constexpr int kFfnPipeBytes = 192 * 1024;   // 6 stages at 256 tokens, 5 of two blocks at 32
constexpr int kFfnMaxExperts = 1024;        // local experts
constexpr int kFfnListUnits = 256;          // units listed at a time
// Shared memory behind the pipeline: barriers, unit list, epilogue tiles, expert offsets, chunk prefix, active experts.
constexpr int kFfnBarBytes = 512;
constexpr int kFfnListBytes = kFfnListUnits * 16;
constexpr int kFfnTileBytes = 2048;         // one 32 column x 32 feature bf16 tile per epilogue warp
constexpr int kFfnEpiBytes = kFfnEpiWarps * kFfnTileBytes;
constexpr int kFfnOffBytes = (kFfnMaxExperts + 1) * 4 + 28;      // rounded to 32
constexpr int kFfnCumBytes = kFfnOffBytes;
constexpr int kFfnIdBytes = kFfnMaxExperts * 2;
constexpr int kFfnSmemBytes = kFfnPipeBytes + 1024 /*align*/ + kFfnBarBytes + kFfnListBytes + kFfnEpiBytes + kFfnOffBytes +
                              kFfnCumBytes + kFfnIdBytes;

__device__ __forceinline__ int ld_acquire_gpu_i32(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Shared memory by its 32-bit address (the generic pointers of the carved-up buffer hide the address space).
__device__ __forceinline__ void sts_bf16(uint32_t addr, float v) {
  asm volatile("st.shared.b16 [%0], %1;" :: "r"(addr), "h"(__bfloat16_as_ushort(__float2bfloat16_rn(v))) : "memory");
}
__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// Equal chunks of an expert's `rows` tokens, at most kFfnMaxN each; all but the last are a multiple of 32.
__device__ __forceinline__ int ffn_chunks(int rows) { return (rows + kFfnMaxN - 1) / kFfnMaxN; }
__device__ __forceinline__ int ffn_chunk_rows(int rows, int chunks) { return ((rows + chunks - 1) / chunks + 31) & ~31; }

// One entry of the unit list.
struct FfnUnit {
  uint32_t e_fc;       // local expert | 1 << 31 for a down unit
  uint32_t j_ch;       // 256-row block of the expert's matrix | chunks of the expert << 12
  int row0;            // first pair row of the chunk
  int n;               // pair rows of the chunk
  __device__ __forceinline__ int fc() const { return (int)(e_fc >> 31); }
  __device__ __forceinline__ int e() const { return (int)(e_fc & 0x7fffffffu); }
  __device__ __forceinline__ int j() const { return (int)(j_ch & 0xfffu); }
  __device__ __forceinline__ int chunks() const { return (int)(j_ch >> 12); }
  __device__ __forceinline__ int half() const { return ((n + 31) & ~31) >> 1; }      // token rows per CTA
};
// What the unit numbering needs, the same in every CTA.  Slots are the experts that have tokens, in order;
// slot s contributes its gate/up units and the down units of slot s - lag.
struct FfnPlanS {
  const int* off;            // [E + 1] first pair row of each expert
  const int* cum;            // [active + 1] chunks of the slots before
  const uint16_t* ids;       // [active] expert of a slot
  int active, lag;
  int n1, n2;                // 256-row blocks of the gate/up and of the down matrix
  __device__ __forceinline__ int total() const { return (n1 + n2) * cum[active]; }
  // units before slot s
  __device__ __forceinline__ int before(int s) const {
    return n1 * cum[s < active ? s : active] + n2 * cum[s > lag ? s - lag : 0];
  }
  __device__ __forceinline__ FfnUnit unit(int u) const {
    int lo = 0, hi = active + lag;                 // before(lo) <= u < before(hi)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (before(mid) <= u) lo = mid; else hi = mid;
    }
    int o = u - before(lo), slot = lo, fc = 0;
    const int u1 = lo < active ? n1 * (cum[lo + 1] - cum[lo]) : 0;
    if (o >= u1) { o -= u1; slot = lo - lag; fc = 1; }
    const int e = ids[slot], ch = cum[slot + 1] - cum[slot];
    const int j = o / ch, c = o - j * ch;          // the chunks of a weight block are neighbours: they share it in L2
    const int rows = off[e + 1] - off[e], cr = ffn_chunk_rows(rows, ch);
    FfnUnit r;
    r.e_fc = (uint32_t)e | ((uint32_t)fc << 31);
    r.j_ch = (uint32_t)j | ((uint32_t)ch << 12);
    r.row0 = off[e] + c * cr;
    r.n = rows - c * cr < cr ? rows - c * cr : cr;
    return r;
  }
};

// Fills cum / ids from the expert offsets; returns the number of experts with tokens.  All threads of the CTA.
__device__ __forceinline__ int ffn_slots(const int* off, int E, int* cum, uint16_t* ids, int* scratch) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = (E + (int)blockDim.x - 1) / (int)blockDim.x;
  const int e0 = threadIdx.x * per, e1 = e0 + per < E ? e0 + per : E;
  int act = 0, chunks = 0;
  for (int e = e0; e < e1; ++e) {
    const int rows = off[e + 1] - off[e];
    act += rows > 0;
    chunks += ffn_chunks(rows);
  }
  int a_inc = act, c_inc = chunks;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, a_inc, o), c = __shfl_up_sync(0xffffffffu, c_inc, o);
    if (lane >= o) { a_inc += a; c_inc += c; }
  }
  if (lane == 31) { scratch[warp] = a_inc; scratch[32 + warp] = c_inc; }
  __syncthreads();
  int a_base = a_inc - act, c_base = c_inc - chunks, total = 0, total_c = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    if (w < warp) { a_base += scratch[w]; c_base += scratch[32 + w]; }
    total += scratch[w];
    total_c += scratch[32 + w];
  }
  for (int e = e0; e < e1; ++e) {
    const int rows = off[e + 1] - off[e];
    if (rows <= 0) continue;
    ids[a_base] = (uint16_t)e;
    cum[a_base] = c_base;
    ++a_base;
    c_base += ffn_chunks(rows);
  }
  if (threadIdx.x == 0) cum[total] = total_c;
  __syncthreads();
  return total;
}

// Bytes of activations up to which all gate/up units come before all down units.  64 experts of 1024 x 1024 with 12 to 65 MB
// of activations ran equally fast in either order (within the 6 % by which two runs differ); the line keeps the
// activations well inside L2 (126 MB, shared with the weight stream, the tokens and the expert outputs).
constexpr long long kFfnActL2Bytes = 24ll << 20;


// Shared memory of the FFN, carved out of the dynamic buffer.
struct FfnSmem {
  uint8_t* pipe;             // [stages][weights x NSUB][token half x NSUB]
  uint64_t* full;            // [kFfnMaxStages], used in the leading CTA
  uint64_t* empty;           // [kFfnMaxStages]
  uint64_t* tfull;           // [2]
  uint64_t* tempty;          // [2], used in the leading CTA
  uint32_t* tmem_slot;
  volatile int* abort_flag;
  uint4* list;
  uint8_t* epi;
  int* off;
  int* cum;
  uint16_t* ids;
  __device__ __forceinline__ FfnSmem() {
    extern __shared__ uint8_t smem_raw[];
    pipe = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    full = reinterpret_cast<uint64_t*>(pipe + kFfnPipeBytes);
    empty = full + kFfnMaxStages;
    tfull = empty + kFfnMaxStages;
    tempty = tfull + 2;
    tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint8_t* p = pipe + kFfnPipeBytes + kFfnBarBytes;
    list = reinterpret_cast<uint4*>(p);
    epi = p + kFfnListBytes;
    off = reinterpret_cast<int*>(epi + kFfnEpiBytes);
    cum = off + kFfnOffBytes / 4;
    ids = reinterpret_cast<uint16_t*>(cum + kFfnCumBytes / 4);
  }
};

// The tensor maps of a launch, as a kernel parameter.
struct FfnMaps {
  CUtensorMap map[MCB_FFN_TMAPS];
};

// Before the FFN, once per kernel: barriers, TMEM, tensor maps (GLOBAL: in global memory).  All threads of both CTAs of the pair; touches nothing
// that another kernel writes, so a kernel with other work to do first calls it at its very start.
template <bool GLOBAL>
__device__ __forceinline__ void ffn_setup(const CUtensorMap* maps) {
  const FfnSmem sm;
  if (threadIdx.x == 0) {
    // full: the weight producer and the first token producer of the leading CTA announce the bytes of both CTAs
    for (int s = 0; s < kFfnMaxStages; ++s) { mbar_init(&sm.full[s], 2); mbar_init(&sm.empty[s], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&sm.tfull[i], 1); mbar_init(&sm.tempty[i], 2 * kFfnEpiWarps); }
    *sm.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x >= 32 && threadIdx.x < 64) tmem_alloc_pair(sm.tmem_slot, 512);
  if (threadIdx.x >= 64 && threadIdx.x < 64 + MCB_FFN_TMAPS) {
    if (GLOBAL) tma_acquire_map(maps + (threadIdx.x - 64));
    tma_prefetch_map(maps + (threadIdx.x - 64));
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                    // barriers initialised and TMEM allocated in both CTAs
  tc_fence_after();
}

// After it: TMEM back.  Nobody leaves before the other CTA of the pair is done with this one's shared memory.  `copied` is
// what ffn_run returned: the last CTA out leaves the counters of the row copy at zero for the next launch.  A CTA counts
// itself out behind the barrier: all its warps have added to the first counter and are done waiting for it.
__device__ __forceinline__ void ffn_teardown(const McbFfnArgs& a, bool copied) {
  const FfnSmem sm;
  tc_fence_before();
  __syncthreads();
  if (copied && threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.sync[1], 1) == (int)gridDim.x - 1) {
      a.sync[0] = 0;
      a.sync[1] = 0;
      __threadfence();
    }
  }
  if (*sm.abort_flag) __nanosleep(50000);            // let any copy still in flight land before the CTA goes away
  cluster_sync();
  if (threadIdx.x >= 32 && threadIdx.x < 64) {
    tc_fence_after();
    tmem_dealloc_pair(*sm.tmem_slot, 512);
  }
}

// Bounded wait for a counter in global memory to reach `want` (acquire); gives up like mbar_wait.
__device__ __forceinline__ void ffn_wait_count(const int* word, int want, const Abort& ab, uint32_t where, uint32_t what) {
  uint64_t t0 = 0;
  for (uint32_t i = 0; ld_acquire_gpu_i32(word) < want; ++i) {
    if (*ab.flag) return;
    if ((i & 31u) != 31u) continue;
    if (t0 == 0) t0 = now_ns();
    if (ab.status && *reinterpret_cast<volatile uint32_t*>(ab.status) != 0u) { *ab.flag = 1; return; }
    if (now_ns() - t0 > ab.timeout_ns) {
      *ab.flag = 1;
      if (ab.status && atomicCAS(ab.status, 0u, (uint32_t)MCB_GEMM_ERR_TIMEOUT) == 0u) {
        ab.status[1] = where; ab.status[2] = blockIdx.x; ab.status[3] = what;
      }
      return;
    }
  }
}

// Token rows into pair order: row p of y = row pair_token[p] of x, for all `pairs` rows, over the warps that call it.
// Eight 512-byte pieces per warp in flight; a.hidden is a multiple of 256, so a piece lies inside one row.
__device__ __forceinline__ void ffn_permute_rows(const McbFfnArgs& a, int pairs, int wid, int nwarps) {
  const int lane = threadIdx.x & 31, per_row = a.hidden / 256;
  const long long pieces = (long long)pairs * per_row;
  const uint8_t* x = reinterpret_cast<const uint8_t*>(a.x) + lane * 16;
  uint8_t* xp = reinterpret_cast<uint8_t*>(a.y) + lane * 16;
  for (long long i0 = (long long)wid * 8; i0 < pieces; i0 += (long long)nwarps * 8) {
    long long src[8];
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const long long i = i0 + k < pieces ? i0 + k : pieces - 1;
      const int row = (int)(i / per_row);
      src[k] = (long long)a.pair_token[row] * a.hidden * 2 + (i - (long long)row * per_row) * 512;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = ld_v4(x + src[k]);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (i0 + k < pieces) st_v4(xp + (i0 + k) * 512, v[k]);
  }
}

// a.w1 is the packed interleaved gate/up matrix (E * 2I rows, H columns), a.w2 the packed down matrix (E * H rows,
// I columns): tile (128-row block v, column block kb) of a matrix with KB column blocks is the 16 KB at byte
// (v * KB + kb) * 16384.
// What the token rows and pair lists still have to wait for: a counter that other CTAs of this launch raise (null:
// nothing).  The weight stream does not wait for it.
struct FfnReady {
  const uint32_t* word;
  int want;
};

template <int NSUB>
__device__ __forceinline__ void ffn_roles(const McbFfnArgs& a, const CUtensorMap* maps, const FfnPlanS& plan, const int n_slot, const FfnReady ready) {
  const FfnSmem sm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();           // 0 = the CTA that issues the MMAs of the pair
  const int H = a.hidden, I = a.intermediate;
  const int npairs = (int)gridDim.x >> 1, pair = (int)blockIdx.x >> 1;
  const int total = plan.total();
  const uint32_t tmem_base = *sm.tmem_slot;
  const Abort ab{sm.abort_flag, a.status, a.timeout_ns};
  const bool gather = n_slot <= kFfnGatherN;

  const int b_sub_bytes = (n_slot >> 1) * 128;                    // token half of one 64-column block
  const int stage_bytes = NSUB * (kFfnABytes + b_sub_bytes);
  int stages = kFfnPipeBytes / stage_bytes;
  if (stages > kFfnMaxStages) stages = kFfnMaxStages;

  // Pipeline position of this warp's role, kept from one batch of the list to the next.
  int s = 0; uint32_t ph = 0;
  int acc = 0; uint32_t acc_ph = 0;
  bool ok = true;

  auto fill = [&](int first) {             // the units first, first + npairs, ... of this pair
    for (int i = threadIdx.x; i < kFfnListUnits; i += blockDim.x) {
      const long long u = first + (long long)i * npairs;
      if (u < total) {
        const FfnUnit un = plan.unit((int)u);
        sm.list[i] = make_uint4(un.e_fc, un.j_ch, (uint32_t)un.row0, (uint32_t)un.n);
      }
    }
    __syncthreads();
  };
  auto listed = [&](int i) {
    const uint4 v = sm.list[i];
    return FfnUnit{v.x, v.y, (int)v.z, (int)v.w};
  };
  fill(pair);
  if (ready.word && warp >= 2) {
    if (lane == 0) ffn_wait_count(reinterpret_cast<const int*>(ready.word), ready.want, ab, 19, 0);
    __syncwarp();
  }
  if (!gather && warp >= 2) {
    // every warp but the weight producer and the MMA issuer takes a share of the copy into pair order
    ffn_permute_rows(a, plan.off[a.num_local_experts], (int)blockIdx.x + (warp - 2) * (int)gridDim.x,
                     (kFfnEpiWarps + kFfnTokWarps) * (int)gridDim.x);
    fence_proxy_async_global();
    __threadfence();
    asm volatile("bar.sync 1, %0;" :: "n"(32 * (kFfnEpiWarps + kFfnTokWarps)) : "memory");
    if (warp == 2 && lane == 0) atomicAdd(&a.sync[0], 1);
  }

  for (int first = pair; first < total; first += kFfnListUnits * npairs) {
    int count = (total - first + npairs - 1) / npairs;
    if (count > kFfnListUnits) count = kFfnListUnits;
    if (warp == 0) {
      // ---------------- weights: 128 rows x 64 NSUB columns per CTA and stage ----------------
      if (elect_one()) {
        const uint64_t stream = l2_evict_first();
        for (int i = 0; i < count && ok; ++i) {
          const FfnUnit un = listed(i);
          const int k_blocks = (un.fc() ? I : H) / kFfnBlockK;
          const CUtensorMap* map = maps + (un.fc() ? MCB_FFN_MAP_W2 : MCB_FFN_MAP_W1) + (NSUB - 1) * 2;
          const int v = (un.e() * (un.fc() ? plan.n2 : plan.n1) + un.j()) * 2 + rank;     // 128-row block of the matrix
          int row = v * k_blocks * (kFfnABytes / 2048);
          for (int kb = 0; kb < k_blocks; kb += NSUB, row += NSUB * kFfnABytes / 2048) {
            if (!(ok = mbar_wait(&sm.empty[s], ph ^ 1u, ab, 11))) break;
            if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * NSUB * kFfnABytes);
            tma_load_2d_pair_hint(sm.pipe + s * stage_bytes, map, cluster_map(&sm.full[s], 0), 0, row, stream);
            if (++s == stages) { s = 0; ph ^= 1u; }
          }
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA: one thread of the leading CTA drives the tensor cores of both ----------------
      if (rank == 0 && elect_one()) {
        for (int i = 0; i < count && ok; ++i) {
          const FfnUnit un = listed(i);
          const int k_blocks = (un.fc() ? I : H) / kFfnBlockK;
          const uint32_t idesc = umma_idesc_bf16(kFfnRowsM, (uint32_t)(un.half() * 2));
          if (!(ok = mbar_wait(&sm.tempty[acc], acc_ph ^ 1u, ab, 12))) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(acc * kFfnMaxN);
          for (int kb = 0; kb < k_blocks; kb += NSUB) {
            if (!(ok = mbar_wait(&sm.full[s], ph, ab, 13))) break;
            tc_fence_after();
            const uint32_t sa = smem_u32(sm.pipe + s * stage_bytes);
#pragma unroll
            for (int sub = 0; sub < NSUB; ++sub) {
              const uint64_t da = make_sw128_desc(sa + sub * kFfnABytes);
              const uint64_t db = make_sw128_desc(sa + NSUB * kFfnABytes + sub * b_sub_bytes);
#pragma unroll
              for (int kk = 0; kk < kFfnBlockK / 16; ++kk)
                umma_bf16_pair(d_tmem, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), idesc, (kb | sub | kk) != 0);
            }
            umma_commit_pair(&sm.empty[s]);
            if (++s == stages) { s = 0; ph ^= 1u; }
          }
          if (!ok) break;
          umma_commit_pair(&sm.tfull[acc]);
          if (++acc == 2) { acc = 0; acc_ph ^= 1u; }
        }
      }
    } else if (warp < 2 + kFfnEpiWarps) {
      // ---------------- epilogue: TMEM (lane = weight row, column = token) -> global ----------------
      const int q = warp & 3;                  // TMEM lane quarter this warp may read
      const int hw = (warp - 2) >> 2;          // it takes the even or the odd 32-column groups
      // A lane holds ONE feature of 32 tokens, memory wants the features of a token side by side: the values
      // cross a small tile in shared memory ([column][feature], 64 or 32 bytes per row) and leave as 16-byte stores.
      const uint32_t tile = smem_u32(sm.epi + (warp - 2) * kFfnTileBytes);
      const uint32_t tempty_addr = cluster_map(sm.tempty, 0);
      for (int i = 0; i < count && ok; ++i) {
        const FfnUnit un = listed(i);
        const int n = un.n;
        if (!(ok = mbar_wait(&sm.tfull[acc], acc_ph, ab, 14))) break;
        tc_fence_after();
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * kFfnMaxN);
        const int wrow = un.j() * kFfnRowsM + rank * 128 + q * 32;       // first weight row of the warp
        auto release = [&] {                   // the accumulator has been read: hand it back before the stores
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(tempty_addr + acc * 8);
        };
        if (hw * 32 >= n) release();
        if (!un.fc()) {
          // rows alternate gate / up: lane pairs (2i, 2i + 1) hold the two halves of activation i; the even lane
          // finishes the even columns, the odd lane the odd ones
          const bool odd = lane & 1;
          uint8_t* obase = reinterpret_cast<uint8_t*>(a.act) + (long long)un.row0 * I * 2 + wrow + (lane & 1) * 16;
#pragma unroll 1
          for (int cc = hw * 32; cc < n; cc += 64) {
            uint32_t v[32];
            tmem_ld32(t_row + cc, v);
            tmem_ld_wait();
            if (cc + 64 >= n) release();
            // Each step over all columns before the next one: the stores keep their order with everything
            // volatile, so a loop over columns would run one column's whole chain after the other.
            uint32_t recv[16];
            float r[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) recv[k] = __shfl_xor_sync(0xffffffffu, odd ? v[2 * k] : v[2 * k + 1], 1);
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const float g = __uint_as_float(odd ? recv[k] : v[2 * k]);
              const float up = __uint_as_float(odd ? v[2 * k + 1] : recv[k]);
              r[k] = silu(g) * up;
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) sts_bf16(tile + (2 * k + (lane & 1)) * 32 + (lane >> 1) * 2, r[k]);
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) {      // 32 columns x 16 features: lane l stores half (l & 1) of column 16h + (l >> 1)
              const int cl = 16 * h + (lane >> 1);
              const uint4 w = lds_v4(tile + cl * 32 + (lane & 1) * 16);
              if (cc + cl < n) st_v4(obase + (long long)(cc + cl) * I * 2, w);
            }
            __syncwarp();
          }
          // This warp's share of the gate/up unit is stored: make it visible to TMA loads of other CTAs and count
          // it for the expert's down units (no barrier between the warps, so nothing can wait for a warp that
          // has given up).
          fence_proxy_async_global();
          __threadfence();
          __syncwarp();
          if (lane == 0) atomicAdd(&a.ffn_done[un.e()], 1);
        } else {
          uint8_t* obase = reinterpret_cast<uint8_t*>(a.y) + ((long long)un.row0 * H + wrow) * 2 + (lane & 3) * 16;
#pragma unroll 1
          for (int cc = hw * 32; cc < n; cc += 64) {
            const float mine = (a.pair_prob && cc + lane < n) ? a.pair_prob[un.row0 + cc + lane] : 1.0f;
            uint32_t v[32];
            tmem_ld32(t_row + cc, v);
            tmem_ld_wait();
            if (cc + 64 >= n) release();
            float r[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) r[k] = __uint_as_float(v[k]) * __shfl_sync(0xffffffffu, mine, k);
#pragma unroll
            for (int k = 0; k < 32; ++k) sts_bf16(tile + k * 64 + lane * 2, r[k]);
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 4; ++h) {      // 32 columns x 32 features: lane l stores quarter (l & 3) of column 8h + (l >> 2)
              const int cl = 8 * h + (lane >> 2);
              const uint4 w = lds_v4(tile + cl * 64 + (lane & 3) * 16);
              if (cc + cl < n) st_v4(obase + (long long)(cc + cl) * H * 2, w);
            }
            __syncwarp();
          }
        }
        if (++acc == 2) { acc = 0; acc_ph ^= 1u; }
      }
    } else {
      // ---------------- tokens: this CTA's half of the chunk into the swizzled K-major B tile ----------------
      // Each of the two warps fetches half of the half, from one thread: four rows per gather, or one box.  Rows past
      // the end of the chunk (they feed columns nobody reads) are fetched too, so that BOTH warps of both CTAs
      // contribute bytes to every stage: one that the stage did not wait for could fall a whole ring behind and
      // misread the parity of `empty`.  The gather indices of the next unit are requested while the current
      // one is still being copied.
      if (elect_one()) {
        const int t = warp - 2 - kFfnEpiWarps;
        constexpr int kOps = kFfnGatherN / 8 / kFfnTokWarps;
        int nxt[kOps][4];
        auto fetch_idx = [&](const FfnUnit& un) {
          if (un.fc() || !gather) return;
          const int rows = un.half() / kFfnTokWarps, base = rank * un.half() + t * rows;
#pragma unroll
          for (int k = 0; k < kOps; ++k) {
            if (k * 4 >= rows) break;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              int r = base + k * 4 + m;
              if (r >= un.n) r %= un.n;              // spread over the chunk's rows, not all on one
              nxt[k][m] = a.pair_token[un.row0 + r];
            }
          }
        };
        fence_proxy_async_global();          // token rows written by ordinary stores before this point
        fetch_idx(listed(0));
        if (!gather && first == pair) {
          ffn_wait_count(&a.sync[0], (int)gridDim.x, ab, 18, 0);
          fence_proxy_async_global();
        }
        for (int i = 0; i < count && ok; ++i) {
          const FfnUnit un = listed(i);
          const int k_blocks = (un.fc() ? I : H) / kFfnBlockK;
          const int rows = un.half() / kFfnTokWarps;           // 8, 16, ... 64
          const uint32_t bytes = (uint32_t)un.half() * 256u * NSUB;
          const int row = un.row0 + rank * un.half() + t * rows;
          const CUtensorMap* map = maps + (un.fc() ? MCB_FFN_MAP_ACT : MCB_FFN_MAP_XP) + (rows >> 3) - 1;
          int cur[kOps][4];
#pragma unroll
          for (int k = 0; k < kOps; ++k)
#pragma unroll
            for (int m = 0; m < 4; ++m) cur[k][m] = nxt[k][m];
          if (i + 1 < count) fetch_idx(listed(i + 1));
          if (un.fc()) {
            // the activations of this expert are complete once every epilogue warp of every gate/up unit has been counted
            ffn_wait_count(&a.ffn_done[un.e()], 2 * kFfnEpiWarps * plan.n1 * un.chunks(), ab, 15, (uint32_t)un.e());
            fence_proxy_async_global();
          }
          const bool box = un.fc() || !gather;
          for (int kb = 0; kb < k_blocks; kb += NSUB) {
            if (!(ok = mbar_wait(&sm.empty[s], ph ^ 1u, ab, 16))) break;
            uint8_t* dst = sm.pipe + s * stage_bytes + NSUB * kFfnABytes + t * rows * 128;
            const uint32_t bar = cluster_map(&sm.full[s], 0);
            if (rank == 0 && t == 0) mbar_arrive_expect_tx(&sm.full[s], bytes);
            if (box) {
#pragma unroll
              for (int sub = 0; sub < NSUB; ++sub)
                tma_load_2d_pair(dst + sub * b_sub_bytes, map, bar, (kb + sub) * kFfnBlockK, row);
            } else {
#pragma unroll
              for (int k = 0; k < kOps; ++k) {
                if (k * 4 >= rows) break;
#pragma unroll
                for (int sub = 0; sub < NSUB; ++sub)
                  tma_gather4_pair(dst + sub * b_sub_bytes + k * 512, maps + MCB_FFN_MAP_X, bar,
                                   (kb + sub) * kFfnBlockK, cur[k][0], cur[k][1], cur[k][2], cur[k][3]);
              }
            }
            if (++s == stages) { s = 0; ph ^= 1u; }
          }
        }
      }
    }
    if (count == kFfnListUnits) {
      __syncthreads();                     // the list is free for the next batch
      fill(first + kFfnListUnits * npairs);
    }
  }
  if (warp == 0 && elect_one()) {
    // The last commits still arrive on both CTAs' `empty` barriers: nobody leaves before they have.
    for (int i = 0; i < stages && ok; ++i) {
      ok = mbar_wait(&sm.empty[s], ph ^ 1u, ab, 17);
      if (++s == stages) { s = 0; ph ^= 1u; }
    }
  }
}

// Call from all kFfnThreads threads of every CTA of the grid (clusters of two CTAs along x), between ffn_setup and
// ffn_teardown, with the experts' offsets in the shared memory of FfnSmem::off (visible to all threads) and the largest
// number of tokens of one expert; dynamic shared memory of at least kFfnSmemBytes.  Returns whether the token rows were copied
// into pair order, for ffn_teardown.
__device__ __forceinline__ bool ffn_run(const McbFfnArgs& a, const CUtensorMap* maps, int max_rows, const FfnReady ready) {
  const FfnSmem sm;
  const int E = a.num_local_experts;
  if (max_rows < 1) max_rows = 1;
  fence_proxy_async_smem();                // the pipeline's memory may have been in ordinary use until here
  __syncthreads();
  FfnPlanS plan;
  plan.off = sm.off; plan.cum = sm.cum; plan.ids = sm.ids;
  plan.n1 = 2 * a.intermediate / kFfnRowsM; plan.n2 = a.hidden / kFfnRowsM;
  plan.active = ffn_slots(sm.off, E, sm.cum, sm.ids, reinterpret_cast<int*>(sm.epi));
  plan.lag = plan.active;
  if ((long long)sm.off[E] * a.intermediate * 2 > kFfnActL2Bytes) {      // three rounds of the grid, in slots of average size
    const int lag = (int)((long long)gridDim.x * 3 / 2 * plan.active / plan.total()) + 2;
    if (lag < plan.lag) plan.lag = lag;
  }
  // Token tile of this launch: the largest expert, rounded up to 32, at most kFfnMaxN per chunk.
  const int n_slot = max_rows > kFfnMaxN ? kFfnMaxN : ((max_rows + 31) & ~31);
  if (n_slot <= kFfnDoubleN) ffn_roles<2>(a, maps, plan, n_slot, ready);
  else ffn_roles<1>(a, maps, plan, n_slot, ready);
  return n_slot > kFfnGatherN;
}

// The same after a routing of its own launch, whose results are in global memory.
__device__ __forceinline__ bool ffn_device(const McbFfnArgs& a, const CUtensorMap* maps) {
  const FfnSmem sm;
  for (int e = threadIdx.x; e <= a.num_local_experts; e += blockDim.x) sm.off[e] = a.expert_offset[e];
  return ffn_run(a, maps, *a.max_rows, FfnReady{nullptr, 0});
}

}  // namespace mcb
