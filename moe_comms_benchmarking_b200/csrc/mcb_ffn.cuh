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
//     to 16, and the accumulators are double buffered in TMEM;
//   * every operand arrives by TMA: weights as 16 or 32 KB tiles (pre-packed once into the swizzled K-major
//     image of their shared-memory tile, so a tile is contiguous in memory), activations as boxes of rows.
//     Token rows come four at a time through the pair -> token list (tile::gather4): the routing permute is
//     fused into the load and no row is copied.  The TMA unit takes a gather every 12 cycles (128 rows in 390 cycles, a box
//     of as many 330, an MMA step over 256 tokens 512), one thread issues one in 35 to 55: four warps share a
//     chunk of up to 128 tokens, six a larger one.  With two warps that also fetched the token numbers, alone, the gathers
//     were the limit, and above 128 tokens the rows were copied into pair order by all CTAs before the first unit
//     (184 MB at 4096 tokens of top-22: 730 -> 672 us a layer without the copy from a cool chip, 896 -> 830 in runs long enough
//     for the power cap; 64 experts at 173 tokens 91 -> 84, at 350 tokens 154 -> 147, with Zipf routing 162 -> 152 us);
//   * work units are listed per CTA pair in shared memory before the roles start: experts without tokens are
//     left out of the numbering, so the pairs get equally many units whatever the routing, and a
//     popular expert's chunks spread over the chip;
//   * both projections run in one persistent stream.  While the activations of all experts fit in L2 the gate/up
//     units of every expert come first, then the down units; above that a down unit follows its gate/up
//     units at a distance of several rounds of the grid (ffn_plan), while its activations are still in L2.  A down
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
// where the weight stream is the limit; 84 (113) at 173 and 147 (204) at 350 tokens per expert.  From about 170 tokens per
// expert on the power cap decides: the clock falls to 1.2-1.4 GHz, and the same launches on rows of zeros take 76 and 122 us.  With
// 22 of 512 experts in use 36 (52).  Launches of a few microseconds lose what a CTA pair costs to set up and take down, and to
// gather: 8 experts of 512 x 256 at 1 / 32 / 128 tokens per expert 8.3 / 9.6 / 12.9 us (7.2 / 7.7 / 10.4).
#pragma once
#include "mcb_group.cuh"
#include "mcb_tc.cuh"

namespace mcb {

constexpr int kFfnEpiWarps = 8;
constexpr int kFfnTokWarps = 6;             // four of them load chunks of up to kFfnDoubleN tokens: one token 41.2 us a layer, 43.6 with six
constexpr int kFfnThreads = 32 * (2 + kFfnEpiWarps + kFfnTokWarps);      // weight TMA, MMA, epilogue, token TMA
constexpr int kFfnRowsM = 256;              // weight rows per unit (128 in each CTA of the pair)
constexpr int kFfnBlockK = 64;              // 128 bytes of bf16
constexpr int kFfnMaxN = 256;               // tokens per chunk
constexpr int kFfnMaxGroups = kFfnMaxN / 8 / 4;      // groups of four rows per token warp and step, of at least four warps
constexpr int kFfnDoubleN = 128;            // up to this many tokens per chunk a stage holds two 64-column blocks
constexpr int kFfnMaxStages = 10;
// Stages of two blocks: four.  A fifth, where it fits, puts 24 MB of weights in flight on the chip instead of 19, and the CTAs then
// share HBM less evenly: 512 experts of 1024 x 1024 at 16 / 37 / 64 / 128 / 512 tokens 235 / 379 / 428 / 462 / 496 us a layer (241 / 389 /
// 443 / 477 / 513 with five); with three, 237 / 381 / 428 / 457 / 488, but 64 experts at 64 tokens 75.6 (73.4; 74.5 with five) and
// 1024 / 4096 tokens 522 / 689 (519 / 680).  Only one token has a use for the fifth (42.0 against 41.6 us).
constexpr int kFfnDoubleStages = 4;
constexpr int kFfnABytes = 128 * kFfnBlockK * 2;                 // 16 KiB of weights per CTA and 64-column block
constexpr int kFfnPipeBytes = 192 * 1024;   // 6 stages at 256 tokens, 4 of two blocks at 128
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
constexpr int kFfnTokIdxBytes = kFfnTokWarps * 128;              // token numbers of a unit's rows, at most 32 per token warp
constexpr int kFfnSmemBytes = kFfnPipeBytes + 1024 /*align*/ + kFfnBarBytes + kFfnListBytes + kFfnEpiBytes + kFfnTokIdxBytes +
                              kFfnOffBytes + kFfnCumBytes + kFfnIdBytes;

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

// Equal chunks of an expert's `rows` tokens, at most kFfnMaxN each; all but the last are a multiple of 16 (the step of N of a CTA
// pair's MMA).
__device__ __forceinline__ int ffn_chunks(int rows) { return (rows + kFfnMaxN - 1) / kFfnMaxN; }
__device__ __forceinline__ int ffn_chunk_rows(int rows, int chunks) { return ((rows + chunks - 1) / chunks + 15) & ~15; }

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
  __device__ __forceinline__ int half() const { return ((n + 15) & ~15) >> 1; }      // token rows per CTA
  // Groups of four rows of that half that one of `warps` token warps fetches, and the first one of warp t.  Every warp has some at
  // every size: where the groups do not divide by the warps, neighbours fetch the same rows to the same place.
  __device__ __forceinline__ int groups(int warps) const { return ((half() >> 2) + warps - 1) / warps; }
  __device__ __forceinline__ int first_group(int t, int warps) const {
    const int g = groups(warps), last = (half() >> 2) - g;
    return t * g < last ? t * g : last;
  }
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
    int slot, o, fc, ch = 1;
    if (lag == active) {                           // all gate/up units first: the slot follows from the chunk at hand
      const int chunks = cum[active];
      fc = u >= n1 * chunks;
      const int v = fc ? u - n1 * chunks : u, nb = fc ? n2 : n1;
      slot = v / nb;
      if (chunks != active) {                      // else every expert is one chunk
        const int x = slot;
        int lo = 0, hi = active;                   // cum[lo] <= x < cum[hi]
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (cum[mid] <= x) lo = mid; else hi = mid;
        }
        slot = lo;
        ch = cum[slot + 1] - cum[slot];
      }
      o = v - nb * cum[slot];
    } else {
      int lo = 0, hi = active + lag;               // before(lo) <= u < before(hi)
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (before(mid) <= u) lo = mid; else hi = mid;
      }
      o = u - before(lo);
      slot = lo;
      fc = 0;
      const int u1 = lo < active ? n1 * (cum[lo + 1] - cum[lo]) : 0;
      if (o >= u1) { o -= u1; slot = lo - lag; fc = 1; }
      ch = cum[slot + 1] - cum[slot];
    }
    const int e = ids[slot];
    const int j = o / ch, c = o - j * ch;          // the chunks of a weight block are neighbours: they share it in L2
    const int rows = off[e + 1] - off[e], cr = ffn_chunk_rows(rows, ch);
    FfnUnit r;
    r.e_fc = (uint32_t)e | ((uint32_t)fc << 31);
    r.j_ch = (uint32_t)j | ((uint32_t)ch << 12);
    r.row0 = off[e] + c * cr;
    r.n = rows - c * cr < cr ? rows - c * cr : cr;
    return r;
  }
  // Units first, first + step, ... into `out`, up to `most` of them; by `threads` threads, of which this is `tid`.
  __device__ __forceinline__ void list(uint4* out, int most, int first, int step, int total, int tid, int threads) const {
    for (int i = tid; i < most; i += threads) {
      const long long u = first + (long long)i * step;
      if (u < total) {
        const FfnUnit un = unit((int)u);
        out[i] = make_uint4(un.e_fc, un.j_ch, (uint32_t)un.row0, (uint32_t)un.n);
      }
    }
  }
};

constexpr int kFfnSlotBits = 11;           // up to 1024 experts with tokens; 2^21 chunks beside them
// Fills cum / ids from the expert offsets; returns the number of experts with tokens.  All threads of the group.
template <class Group>
__device__ __forceinline__ int ffn_slots(const Group& g, const int* off, int E, int* cum, uint16_t* ids, int* scratch) {
  const int tid = g.tid(), warp = tid >> 5, lane = tid & 31;
  const int per = (E + (int)g.size() - 1) / (int)g.size();
  const int e0 = tid * per, e1 = e0 + per < E ? e0 + per : E;
  // Experts with tokens in the low kFfnSlotBits, chunks above: one scan for both, and one of the warps' sums by every warp for itself.  Nothing streams
  // before the units are listed: with a scan each, the warps' sums added up one by one and every unit searched for through both of its bounds (unit), the
  // smallest launches took 14.5 us (14.0 so; 8 tokens of 16 experts of 512 x 256), 64 experts of 1024 x 1024 with 174 / 2800 / 11000 pairs 61.9 / 70.3 / 86.4
  // (61.2 / 69.6 / 85.2).
  uint32_t mine = 0;
  for (int e = e0; e < e1; ++e) {
    const int rows = off[e + 1] - off[e];
    mine += ((uint32_t)ffn_chunks(rows) << kFfnSlotBits) + (rows > 0);
  }
  auto scan = [&](uint32_t v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += x;
    }
    return v;
  };
  const uint32_t inc = scan(mine);
  if (lane == 31) scratch[warp] = (int)inc;
  g.sync();
  const uint32_t warps = scan(lane < (int)(g.size() >> 5) ? (uint32_t)scratch[lane] : 0u);
  const uint32_t all = __shfl_sync(0xffffffffu, warps, 31), before = __shfl_sync(0xffffffffu, warps, warp ? warp - 1 : 0);
  const uint32_t base = inc - mine + (warp ? before : 0u);
  const int total = (int)(all & ((1u << kFfnSlotBits) - 1)), total_c = (int)(all >> kFfnSlotBits);
  int a_base = (int)(base & ((1u << kFfnSlotBits) - 1)), c_base = (int)(base >> kFfnSlotBits);
  for (int e = e0; e < e1; ++e) {
    const int rows = off[e + 1] - off[e];
    if (rows <= 0) continue;
    ids[a_base] = (uint16_t)e;
    cum[a_base] = c_base;
    ++a_base;
    c_base += ffn_chunks(rows);
  }
  if (tid == 0) cum[total] = total_c;
  g.sync();
  return total;
}

// Bytes of activations up to which all gate/up units come before all down units.  64 experts of 1024 x 1024 with 12 to 65 MB
// of activations ran equally fast in either order (within the 6 % by which two runs differ); the line keeps the
// activations well inside L2 (126 MB, shared with the weight stream, the tokens and the expert outputs).
constexpr long long kFfnActL2Bytes = 24ll << 20;


// Token tile of a launch: the largest expert, rounded up to 16, at most kFfnMaxN per chunk.
__device__ __forceinline__ int ffn_token_tile(int max_rows) {
  return max_rows < 1 ? 16 : max_rows > kFfnMaxN ? kFfnMaxN : ((max_rows + 15) & ~15);
}
// The rest of the plan, once its offsets and slots are there.
__device__ __forceinline__ void ffn_plan(FfnPlanS& plan, const McbFfnArgs& a, int active) {
  plan.n1 = 2 * a.intermediate / kFfnRowsM; plan.n2 = a.hidden / kFfnRowsM;
  plan.active = plan.lag = active;
  if ((long long)plan.off[a.num_local_experts] * a.intermediate * 2 > kFfnActL2Bytes) {
    // So many slots, of average size, that their down units alone make two rounds of the grid: that is how far the last slot's are from
    // its gate/up units.  With three rounds of all units (which are one of down units where n1 = 2 n2) they waited there: 8191 tokens with
    // Zipf routing, an eighth of 512 experts of 1024 x 1024, 129.6 -> 127.2 us (three rounds of down units 126.5, all gate/up units first
    // 126.9); 4096 tokens of all experts the same (three rounds of down units 0.3 % slower).  Where down units are more than twice as many as gate/up
    // units three rounds of all units are the longer distance and stay: 48 experts of 3072 x 256 with 1100 tokens 394 us by two rounds of
    // down units, 377 so, 64 of 7168 x 512 with 700 1180 and 1152, 32 of 4096 x 512 with 1100 508 and 520.
    // In slots the distance grows with n1 / n2.  Three rounds of all units -> this, warm clocks, us a launch, with the activations between the two:
    //   n1 = 8 n2   200 experts of 512 x 2048 with 250 tokens 464 -> 460 (14 -> 78 MB), 64 with 256 168.0 -> 165.6 (all first, 67 MB), 48 with 512
    //               218.8 -> 216.5, 16 with 1500 188.5 -> 185.7, 24 of 1024 x 4096 with 400 313.8 -> 314.2
    //   n1 = 6 n2   64 of 512 x 1536 with 256, Zipf 130.8 -> 125.4, with 180 103.5 -> 100.5
    //   n1 = 4 n2   128 of 1024 x 2048 with 200 413.5 -> 424.5 (431 -> 432 on another), Zipf 458 -> 461, 100 of 512 x 1024 with 300 157.6 -> 155.7
    //   n1 = 3 n2   64 of 1536 x 2048 with 300 488 -> 494, 32 of 1024 x 1536 with 300 127 -> 124
    //   n1 = n2     32 of 3072 x 1536 with 700 649 -> 658, 32 of 7168 x 1024 (0.6 n2) with 700 1036 -> 1015
    // so nothing asks for a bound in bytes: one of 24 MB gave between -4 and +2.5 % over shapes up to n1 = 8 n2, with no trend in the shape.
    const long long chunks = plan.cum[active];
    const int down = (int)((long long)gridDim.x * active / (plan.n2 * chunks)) + 2;
    const int all = (int)((long long)gridDim.x * 3 / 2 * active / ((plan.n1 + plan.n2) * chunks)) + 2;
    const int lag = down > all ? down : all;
    if (lag < plan.lag) plan.lag = lag;
  }
}

// Shared memory of the FFN, carved out of the dynamic buffer.
struct FfnSmem {
  uint8_t* pipe;             // [stages][weights x NSUB][token half x NSUB]
  uint64_t* full;            // [kFfnMaxStages], used in the leading CTA
  uint64_t* empty;           // [kFfnMaxStages]
  uint64_t* tfull;           // [2]
  uint64_t* tempty;          // [2], used in the leading CTA
  uint32_t* tmem_slot;
  volatile int* abort_flag;
  int* acts_there;           // down units whose activations are complete, counted by the first token warp
  uint4* list;
  uint8_t* epi;
  int* tok_idx;
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
    acts_there = reinterpret_cast<int*>(tmem_slot + 2);
    uint8_t* p = pipe + kFfnPipeBytes + kFfnBarBytes;
    list = reinterpret_cast<uint4*>(p);
    epi = p + kFfnListBytes;
    tok_idx = reinterpret_cast<int*>(epi + kFfnEpiBytes);
    off = tok_idx + kFfnTokIdxBytes / 4;
    cum = off + kFfnOffBytes / 4;
    ids = reinterpret_cast<uint16_t*>(cum + kFfnCumBytes / 4);
  }
};

// What a step of several layers in one launch (moe_step.cu) keeps behind the token numbers instead: offsets, chunk prefix and
// active experts of the layer being listed, the counters of its routing, and the barriers of the two halves of the unit list.
constexpr int kStepMaxExperts = 768;
constexpr int kStepListUnits = kFfnListUnits / 2;
struct StepSmem {
  int* off;                  // [kStepMaxExperts + 1]
  int* cum;                  // [kStepMaxExperts + 1]; the counts of the routing before the chunks are numbered
  uint16_t* ids;             // [kStepMaxExperts]
  int* begin;                // [kStepMaxExperts]
  int* scan;                 // [96]
  uint64_t* lfull;           // [2]
  uint64_t* lempty;          // [2]
  int* head;                 // [2][2] units of a half, whether it is the last one of its layer
  int* word;                 // [4] hand-over among the epilogue warps (0, 2) and among the routing warps (1, 3)
  static constexpr int kOff = kStepMaxExperts * 4 + 16;
  static constexpr int kBytes = 2 * kOff + kStepMaxExperts * 2 + kStepMaxExperts * 4 + 96 * 4 + 64;
  __device__ __forceinline__ explicit StepSmem(const FfnSmem& sm) {
    off = sm.off;
    cum = off + kOff / 4;
    ids = reinterpret_cast<uint16_t*>(cum + kOff / 4);
    begin = reinterpret_cast<int*>(ids + kStepMaxExperts);
    scan = begin + kStepMaxExperts;
    lfull = reinterpret_cast<uint64_t*>(scan + 96);
    lempty = lfull + 2;
    head = reinterpret_cast<int*>(lempty + 2);
    word = head + 4;
  }
};
constexpr int kStepSmemBytes = kFfnSmemBytes - kFfnOffBytes - kFfnCumBytes - kFfnIdBytes + StepSmem::kBytes;
static_assert(kStepSmemBytes + 256 <= 227 * 1024, "fits beside the static shared memory");

// The tensor maps of a launch, as a kernel parameter.
struct FfnMaps {
  CUtensorMap map[MCB_FFN_TMAPS];
};

// Before the FFN, once per kernel: barriers, TMEM, tensor maps (GLOBAL: in global memory; null: none).  All threads of both CTAs of the pair; touches nothing
// that another kernel writes, so a kernel with other work to do first calls it at its very start.
template <bool GLOBAL>
__device__ __forceinline__ void ffn_setup(const CUtensorMap* maps) {
  const FfnSmem sm;
  if (threadIdx.x == 0) {
    // full: the weight producer and the first token producer of the leading CTA announce the bytes of both CTAs
    for (int s = 0; s < kFfnMaxStages; ++s) { mbar_init(&sm.full[s], 2); mbar_init(&sm.empty[s], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&sm.tfull[i], 1); mbar_init(&sm.tempty[i], 2 * kFfnEpiWarps); }
    *sm.abort_flag = 0;
    *sm.acts_there = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x >= 32 && threadIdx.x < 64) tmem_alloc_pair(sm.tmem_slot, 512);
  if (maps && threadIdx.x >= 64 && threadIdx.x < 64 + MCB_FFN_TMAPS) {
    if (GLOBAL) tma_acquire_map(maps + (threadIdx.x - 64));
    tma_prefetch_map(maps + (threadIdx.x - 64));
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                    // barriers initialised and TMEM allocated in both CTAs
  tc_fence_after();
}

// After it: TMEM back.  Nobody leaves before the other CTA of the pair is done with this one's shared memory.
__device__ __forceinline__ void ffn_teardown() {
  const FfnSmem sm;
  tc_fence_before();
  __syncthreads();
  if (*sm.abort_flag) settle();
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

// The same for a count in this CTA's shared memory.
__device__ __forceinline__ void ffn_wait_told(const int* word, int want, const Abort& ab, uint32_t what) {
  uint64_t t0 = 0;
  for (uint32_t i = 0;; ++i) {
    int v;
    asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(smem_u32(word)) : "memory");
    if (v >= want || *ab.flag) return;
    if ((i & 1023u) != 1023u) continue;
    if (t0 == 0) t0 = now_ns();
    if (now_ns() - t0 > ab.timeout_ns) {
      *ab.flag = 1;
      if (ab.status && atomicCAS(ab.status, 0u, (uint32_t)MCB_GEMM_ERR_TIMEOUT) == 0u) {
        ab.status[1] = 26; ab.status[2] = blockIdx.x; ab.status[3] = what;
      }
      return;
    }
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

// The warps' roles over lists of units.  A role keeps its position in the pipeline from one list to the next; every warp of
// a role sees the same lists in the same order.  TOK: token warps.
template <int NSUB, int TOK>
struct FfnRoles {
  const McbFfnArgs& a;
  const CUtensorMap* xmap;           // token rows
  // Activations by box, where the gate/up units write them, and expert outputs (of the layer at hand).
  const CUtensorMap* actmap;
  uint8_t* act_rows;
  uint8_t* y_rows;
  const FfnSmem sm;
  const int warp, lane, rank;        // rank 0 = the CTA that issues the MMAs of the pair
  const int H, I, n1, n2;
  const uint32_t tmem_base;
  const Abort ab;
  const int b_sub_bytes, stage_bytes, stages;      // token half of one 64-column block, a stage, their number
  // Position of this warp's role (each role uses its own of these).
  int s = 0; uint32_t ph = 0;
  int acc = 0; uint32_t acc_ph = 0;
  int downs = 0;                     // down units so far
  bool ok = true;
  // A count that a down unit waits for before it writes its first row (null: nothing).
  const int* y_free = nullptr;
  int y_free_want = 0;

  __device__ __forceinline__ FfnRoles(const McbFfnArgs& args, const CUtensorMap* x, const CUtensorMap* act, int n_slot)
      : a(args), xmap(x), actmap(act), act_rows(reinterpret_cast<uint8_t*>(args.act)), y_rows(reinterpret_cast<uint8_t*>(args.y)),
        warp(threadIdx.x >> 5), lane(threadIdx.x & 31), rank((int)cluster_ctarank()), H(args.hidden), I(args.intermediate),
        n1(2 * args.intermediate / kFfnRowsM), n2(args.hidden / kFfnRowsM), tmem_base(*sm.tmem_slot), ab{sm.abort_flag, args.status, args.timeout_ns},
        b_sub_bytes((n_slot >> 1) * 128), stage_bytes(NSUB * (kFfnABytes + b_sub_bytes)), stages(stage_count(stage_bytes)) {}
  static __device__ __forceinline__ int stage_count(int bytes) {
    const int fit = kFfnPipeBytes / bytes, most = NSUB == 2 ? kFfnDoubleStages : kFfnMaxStages;
    return fit < most ? fit : most;
  }
  static __device__ __forceinline__ FfnUnit listed(const uint4* list, int i) {
    const uint4 v = list[i];
    return FfnUnit{v.x, v.y, (int)v.z, (int)v.w};
  }

  // One warp: 128 rows x 64 NSUB columns per CTA and stage.  wmaps: MCB_FFN_MAP_W1 ... of the weight set.
  __device__ __forceinline__ void weights(const uint4* list, int count, const CUtensorMap* wmaps) {
    if (elect_one()) {
      const uint64_t stream = l2_evict_first();
      for (int i = 0; i < count && ok; ++i) {
        const FfnUnit un = listed(list, i);
        const int k_blocks = (un.fc() ? I : H) / kFfnBlockK;
        const CUtensorMap* map = wmaps + un.fc() + (NSUB - 1) * 2;
        const int v = (un.e() * (un.fc() ? n2 : n1) + un.j()) * 2 + rank;     // 128-row block of the matrix
        int row = v * k_blocks * (kFfnABytes / 2048);
        for (int kb = 0; kb < k_blocks; kb += NSUB, row += NSUB * kFfnABytes / 2048) {
          if (!(ok = mbar_wait(&sm.empty[s], ph ^ 1u, ab, 11))) break;
          if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * NSUB * kFfnABytes);
          tma_load_2d_pair_hint(smem_u32(sm.pipe) + s * stage_bytes, map, cluster_map(&sm.full[s], 0), 0, row, stream);
          if (++s == stages) { s = 0; ph ^= 1u; }
        }
      }
    }
  }

  // One warp of the leading CTA: one thread drives the tensor cores of both.
  __device__ __forceinline__ void mma(const uint4* list, int count) {
    if (elect_one()) {
      for (int i = 0; i < count && ok; ++i) {
        const FfnUnit un = listed(list, i);
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
  }

  // kFfnEpiWarps warps, `ew` counts them from 0: TMEM (lane = weight row, column = token) -> global.
  __device__ __forceinline__ void epilogue(const uint4* list, int begin, int count, int ew, const float* pair_prob, int* ffn_done) {
    const int q = warp & 3;                  // TMEM lane quarter this warp may read
    const int hw = ew >> 2;          // it takes the even or the odd 32-column groups
    // A lane holds ONE feature of 32 tokens, memory wants the features of a token side by side: the values
    // cross a small tile in shared memory ([column][feature], 64 or 32 bytes per row) and leave as 16-byte stores.
    const uint32_t tile = smem_u32(sm.epi + ew * kFfnTileBytes);
    const uint32_t tempty_addr = cluster_map(sm.tempty, 0);
    for (int i = begin; i < count && ok; ++i) {
      const FfnUnit un = listed(list, i);
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
        uint8_t* obase = act_rows + (long long)un.row0 * I * 2 + wrow + (lane & 1) * 16;
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
        if (lane == 0) atomicAdd(&ffn_done[un.e()], 1);
      } else {
        if (y_free) {
          if (lane == 0) ffn_wait_count(y_free, y_free_want, ab, 20, (uint32_t)un.e());
          __syncwarp();
          y_free = nullptr;
        }
        uint8_t* obase = y_rows + ((long long)un.row0 * H + wrow) * 2 + (lane & 3) * 16;
#pragma unroll 1
        for (int cc = hw * 32; cc < n; cc += 64) {
          const float mine = (pair_prob && cc + lane < n) ? pair_prob[un.row0 + cc + lane] : 1.0f;
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
  }

  // TOK warps, `t` counts them from 0: this CTA's half of the chunk into the swizzled K-major B tile.
  __device__ __forceinline__ void tokens(const uint4* list, int count, int t, const int* pair_token, const int* ffn_done) {
    // Each of the TOK warps fetches its groups of four rows, from one thread: a gather each, or one box.  Rows past
    // the end of the chunk (they feed columns nobody reads) are fetched too, so that ALL warps of both CTAs
    // contribute bytes to every stage: one that the stage did not wait for could fall a whole ring behind and
    // misread the parity of `empty`.  The lanes fetch the token numbers of the next unit, one each, while the current one
    // is still being copied, and hand them to the issuing thread through shared memory.
    constexpr int kOps = (kFfnMaxN / NSUB / 8 + TOK - 1) / TOK;
    static_assert(kOps <= kFfnMaxGroups && kOps * 4 <= 32, "a map per box, a lane per row");
    const uint32_t idx_slot = smem_u32(sm.tok_idx + t * 32);
    const uint32_t pipe0 = smem_u32(sm.pipe) + NSUB * kFfnABytes, full0 = cluster_map(sm.full, 0);
    auto fetch_idx = [&](const FfnUnit& un) {
      const int rows = un.groups(TOK) * 4;
      int r = rank * un.half() + un.first_group(t, TOK) * 4 + lane;
      if (un.fc() || lane >= rows) return 0;
      if (r >= un.n) r %= un.n;                  // spread over the chunk's rows, not all on one
      return pair_token[un.row0 + r];
    };
    fence_proxy_async_global();          // token rows written by ordinary stores before this point
    int nxt = fetch_idx(listed(list, 0));
    for (int i = 0; i < count && ok; ++i) {
      const FfnUnit un = listed(list, i);
      const int steps = (un.fc() ? I : H) / (kFfnBlockK * NSUB);
      const int groups = un.groups(TOK), row_h = un.first_group(t, TOK) * 4;
      if (!un.fc()) asm volatile("st.shared.b32 [%0], %1;" :: "r"(idx_slot + lane * 4), "r"(nxt) : "memory");
      __syncwarp();
      if (i + 1 < count) nxt = fetch_idx(listed(list, i + 1));
      if (elect_one()) {
        const uint32_t bytes = (uint32_t)(groups * TOK) * 1024u * NSUB;
        int su = s; uint32_t pu = ph;
        if (un.fc()) {
          const int row = un.row0 + rank * un.half() + row_h;
          const CUtensorMap* map = actmap + groups - 1;
          // The activations of this expert are complete once every epilogue warp of every gate/up unit has been counted.  One
          // warp asks for the count and tells the others: the answers come from one or two lines that the counting goes through too.
          ++downs;
          if (t == 0) {
            ffn_wait_count(&ffn_done[un.e()], 2 * kFfnEpiWarps * n1 * un.chunks(), ab, 15, (uint32_t)un.e());
            asm volatile("st.release.cta.shared.b32 [%0], %1;" :: "r"(smem_u32(sm.acts_there)), "r"(downs) : "memory");
          } else {
            ffn_wait_told(sm.acts_there, downs, ab, (uint32_t)un.e());
          }
          fence_proxy_async_global();
          for (int k = 0; k < steps; ++k) {
            if (!(ok = mbar_wait(&sm.empty[su], pu ^ 1u, ab, 16))) break;
            if (rank == 0 && t == 0) mbar_arrive_expect_tx(&sm.full[su], bytes);
            const uint32_t dst = pipe0 + su * stage_bytes + row_h * 128;
#pragma unroll
            for (int sub = 0; sub < NSUB; ++sub)
              tma_load_2d_pair(dst + sub * b_sub_bytes, map, full0 + su * 8, (k * NSUB + sub) * kFfnBlockK, row);
            if (++su == stages) { su = 0; pu ^= 1u; }
          }
        } else {
          uint4 idx[kOps];
#pragma unroll
          for (int k = 0; k < kOps; ++k) idx[k] = lds_v4(idx_slot + k * 16);
          for (int k = 0; k < steps; ++k) {
            if (!(ok = mbar_wait(&sm.empty[su], pu ^ 1u, ab, 16))) break;
            if (rank == 0 && t == 0) mbar_arrive_expect_tx(&sm.full[su], bytes);
            const uint32_t dst = pipe0 + su * stage_bytes + row_h * 128;
#pragma unroll
            for (int g = 0; g < kOps; ++g) {
              if (g >= groups) break;
#pragma unroll
              for (int sub = 0; sub < NSUB; ++sub)
                tma_gather4_pair(dst + sub * b_sub_bytes + g * 512, xmap, full0 + su * 8,
                                 (k * NSUB + sub) * kFfnBlockK, idx[g].x, idx[g].y, idx[g].z, idx[g].w);
            }
            if (++su == stages) { su = 0; pu ^= 1u; }
          }
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      s += steps % stages;
      ph ^= (uint32_t)(steps / stages) & 1u;
      if (s >= stages) { s -= stages; ph ^= 1u; }
      __syncwarp();
    }
  }

  // The weight warp, after its last unit: the last commits still arrive on both CTAs' `empty` barriers, and nobody leaves
  // before they have.
  __device__ __forceinline__ void drain() {
    if (!elect_one()) return;
    for (int i = 0; i < stages && ok; ++i) {
      ok = mbar_wait(&sm.empty[s], ph ^ 1u, ab, 17);
      if (++s == stages) { s = 0; ph ^= 1u; }
    }
  }
};

template <int NSUB>
__device__ __forceinline__ void ffn_roles(const McbFfnArgs& a, const CUtensorMap* maps, const FfnPlanS& plan, const int n_slot, const FfnReady ready) {
  constexpr int kTok = NSUB == 2 ? 4 : kFfnTokWarps;      // token warps of this launch
  FfnRoles<NSUB, kTok> r(a, maps + MCB_FFN_MAP_X, maps + MCB_FFN_MAP_ACT, n_slot);
  const int npairs = (int)gridDim.x >> 1, pair = (int)blockIdx.x >> 1, total = plan.total();
  auto fill = [&](int first) {             // the units first, first + npairs, ... of this pair
    plan.list(r.sm.list, kFfnListUnits, first, npairs, total, (int)threadIdx.x, (int)blockDim.x);
    __syncthreads();
  };
  fill(pair);
  if (ready.word && r.warp >= 2) {
    if (r.lane == 0) ffn_wait_count(reinterpret_cast<const int*>(ready.word), ready.want, r.ab, 19, 0);
    __syncwarp();
  }
  for (int first = pair; first < total; first += kFfnListUnits * npairs) {
    int count = (total - first + npairs - 1) / npairs;
    if (count > kFfnListUnits) count = kFfnListUnits;
    if (r.warp == 0) r.weights(r.sm.list, count, maps + MCB_FFN_MAP_W1);
    else if (r.warp == 1) { if (r.rank == 0) r.mma(r.sm.list, count); }
    else if (r.warp < 2 + kFfnEpiWarps) r.epilogue(r.sm.list, 0, count, r.warp - 2, a.pair_prob, a.ffn_done);
    else if (r.warp < 2 + kFfnEpiWarps + kTok) r.tokens(r.sm.list, count, r.warp - 2 - kFfnEpiWarps, a.pair_token, a.ffn_done);
    if (count == kFfnListUnits) {
      __syncthreads();                     // the list is free for the next batch
      fill(first + kFfnListUnits * npairs);
    }
  }
  if (r.warp == 0) r.drain();
}

// Call from all kFfnThreads threads of every CTA of the grid (clusters of two CTAs along x), between ffn_setup and
// ffn_teardown, with the experts' offsets in the shared memory of FfnSmem::off (visible to all threads) and the largest
// number of tokens of one expert; dynamic shared memory of at least kFfnSmemBytes.
__device__ __forceinline__ void ffn_run(const McbFfnArgs& a, const CUtensorMap* maps, int max_rows, const FfnReady ready) {
  const FfnSmem sm;
  const int E = a.num_local_experts;
  fence_proxy_async_smem();                // the pipeline's memory may have been in ordinary use until here
  __syncthreads();
  const int n_slot = ffn_token_tile(max_rows);
  FfnPlanS plan;
  plan.off = sm.off; plan.cum = sm.cum; plan.ids = sm.ids;
  ffn_plan(plan, a, ffn_slots(BlockGroup{}, sm.off, E, sm.cum, sm.ids, reinterpret_cast<int*>(sm.epi)));
  if (n_slot <= kFfnDoubleN) ffn_roles<2>(a, maps, plan, n_slot, ready);
  else ffn_roles<1>(a, maps, plan, n_slot, ready);
}

// The same after a routing of its own launch, whose results are in global memory.
__device__ __forceinline__ void ffn_device(const McbFfnArgs& a, const CUtensorMap* maps) {
  const FfnSmem sm;
  for (int e = threadIdx.x; e <= a.num_local_experts; e += blockDim.x) sm.off[e] = a.expert_offset[e];
  ffn_run(a, maps, *a.max_rows, FfnReady{nullptr, 0});
}

}  // namespace mcb
