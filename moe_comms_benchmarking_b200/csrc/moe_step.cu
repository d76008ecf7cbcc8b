// A decode step with real experts in a world of one as ONE launch for all its layers.
//
// A layer kernel of its own (ffn.cu) spends 20 of 41 us at one token on what is not the weight stream: the launch and its
// set-up, the copy of the rows, the routing, the grid barrier behind the experts, the combine, and the ramp and the tail of the
// stream.  Here every CTA keeps its roles over all layers and the stream does not stop between them:
//
//   weight warp     goes from the last unit of a layer to the first one of the next as soon as that is listed
//   token warps     the same, once all CTAs have published the pair lists of the layer
//   MMA warp        up to two units (the accumulators) ahead of the epilogue
//   epilogue warps  store the units of a layer and, once all CTAs have finished the layer before, their share of its sums over
//                   the experts (mcb_combine.cuh): with two buffers of activations and expert outputs ahead of their first down
//                   unit, so that nobody waits for the slowest CTA; with one buffer ahead of the first unit of the layer
//   routing warps   two of them: while a layer runs they copy the rows of the next one, route it and list its units
//
// The pair lists and counters of a layer alternate between three sets of buffers, so that routing layer l + 1 waits for the
// sums of layer l - 2 only.  With two sets (and the sums right behind a layer's last unit) the stream stood still for 5 of
// 26 us a layer at one token, waiting for the routing that waited for the sums.  Measured on one B200 against a launch per layer, both
// kept running for a second (nvidia-smi beside them), 8 layers of 512 experts of 1024 x 1024, top-22, us a layer:
//   tokens              1       4      16      37     128     512    1024    4096
//   one launch       23.6    72.6     226     339     455     492     520     800     1.9 GHz at one token, 1.6-1.5 up to 512, 1.4, 1.05
//   a launch each    41.7    89.5     244     353     474     503     541     792     1.97, 1.96, 1.67-1.6, 1.43, 1.1 GHz
// From 4 tokens on the power cap is active in both (1000 W); runs of a few milliseconds on a cool chip are up to 15 % shorter at 4096.
// 88 layers of one token 1980 us (3630), whose weights alone are 1860 at the speed of a copy; 64 experts of 768 x 512, one token of
// top-6, 9.3 us a layer (22.5); 4 wide layers (7168 x 2048, 32 experts) of 190 tokens 422 (441).  Four accumulators instead of two
// changed nothing.  The units are numbered through all layers (the first unit of a layer goes to the pair behind the one that has the
// last unit of the layer before), so a layer whose units do not fill its last round costs no round.
// All layers read the same rows, ids and weights, which nothing in the step writes (the host checks that, mcb_moe_step_joins), so
// the experts gather the rows at their source and nobody waits for the copy.
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>

#define MCB_WITH_LAYER_ARGS
#include "mcb_combine.cuh"
#include "mcb_dense.cuh"
#include "mcb_ffn.cuh"
#include "mcb_gemm.h"
#include "mcb_launch.h"
#include "mcb_route.cuh"
#include "mcb_tmap.h"

namespace mcb {

struct StepWeights {
  CUtensorMap map[MCB_STEP_SETS][4];
};

constexpr int kStepRouteWarps = 2;
constexpr int kStepTokWarps = kFfnTokWarps - kStepRouteWarps;
constexpr int kStepRouteWarp = 2 + kFfnEpiWarps + kStepTokWarps;           // first of the routing warps
using RouteGroup = WarpGroup<kStepRouteWarp, kStepRouteWarps, 2>;
using EpilogueGroup = WarpGroup<2, kFfnEpiWarps, 1>;

// Counters of a step (McbMoeStepArgs::sync), a line each.  All but the last only grow during a launch.
enum { kStepRouted = 0, kStepCounted = 32, kStepExperts = 64, kStepCombined = 96, kStepLeft = 128 };

// The copy and the routing of a layer, by a group of threads of every CTA.
struct StepRoute {
  const McbMoeStepArgs& p;
  const LocalRanges& rows;
  const StepSmem& st;
  const Abort& ab;
  McbRouteArgs r;
  int T;
  int counted = 0;             // layers whose counts went through the counters

  __device__ __forceinline__ StepRoute(const McbMoeStepArgs& args, const LocalRanges& ranges, const StepSmem& smem, const Abort& abort, int tokens)
      : p(args), rows(ranges), st(smem), ab(abort), r(args.layer.route), T(tokens) {
    if (two() && p.two_rows < r.max_pairs) r.max_pairs = (int)p.two_rows;
  }
  // Whether the layers alternate between two buffers of activations and expert outputs.
  __device__ __forceinline__ bool two() const { return (long long)T * p.layer.route.topk <= p.two_rows; }

  // Returns the largest number of rows of an expert, -1 once this CTA has given up: counts that are not complete would place rows
  // beyond the buffers.
  template <class Group>
  __device__ __forceinline__ int layer(const Group& g, int set) {
    const int grid = (int)gridDim.x, bid = (int)blockIdx.x, E = r.num_local_experts;
    copy_ranges(rows, 0, (long long)bid * g.size() + g.tid(), (long long)grid * g.size(), g.tid());
    r.pair_token = p.pair_token[set]; r.pair_prob = p.pair_prob[set]; r.pair_pos = p.pair_pos[set]; r.ffn_done = p.ffn_done[set];
    const RouteSmem m(st.cum, st.begin, st.off, st.scan);
    RouteShare share;
    share.entries = (long long)T * r.topk;
    const long long per = (share.entries + grid - 1) / grid;
    share.lo = per * bid < share.entries ? per * bid : share.entries;
    share.hi = share.lo + per < share.entries ? share.lo + per : share.entries;
    if (route_counts_all(g, share)) {
      route_count<true>(g, r, p.ids, m, 0, share.entries, share.lo);
    } else {
      // Three counters per expert, used in turn: those of the next layer are zeroed before the barrier of this one.  By then
      // everybody has read what they held, two layers ago: the barrier of the last layer came after that.
      route_count<false>(g, r, p.ids, m, share.lo, share.hi, 0);
      int* count = p.expert_count + (counted % 3) * E;
      route_publish(g, E, count, m);
      if (bid == 0)
        for (int e = g.tid(); e < E; e += g.size()) p.expert_count[((counted + 1) % 3) * E + e] = 0;
      ++counted;
      g.sync();
      if (g.tid() == 0) {
        __threadfence();
        atomicAdd(&p.sync[kStepCounted], 1);
        ffn_wait_count(&p.sync[kStepCounted], counted * grid, ab, 21, (uint32_t)counted);
        st.word[3] = *ab.flag;
      }
      g.sync();
      if (st.word[3]) return -1;
      route_collect(g, E, count, m);
    }
    const int mx = route_offsets(g, r, m, bid == 0);
    route_place(g, r, p.ids, p.probs, m, share);
    g.sync();
    if (g.tid() == 0) {
      __threadfence();
      atomicAdd(&p.sync[kStepRouted], 1);
    }
    return mx;
  }
};

// All layers of a launch for one token tile.
template <int NSUB>
__device__ __forceinline__ void step_roles(const McbMoeStepArgs& p, const StepWeights& w, StepRoute& route, int layers, int first_set, int sets,
                                           int n_slot) {
  const McbFfnArgs& a = p.layer.ffn;
  FfnRoles<NSUB, kStepTokWarps> r(a, reinterpret_cast<const CUtensorMap*>(p.map_x), nullptr, n_slot);
  const StepSmem st(r.sm);
  const int grid = (int)gridDim.x, npairs = grid >> 1, pair = (int)blockIdx.x >> 1;

  if (r.warp >= kStepRouteWarp) {
    // ---------------- copy and routing of the next layer, lists of units ----------------
    const RouteGroup g;
    int base = 0;              // pair of the layer's first unit
    int half = 0; uint32_t half_ph = 0;
    for (int l = 0; l < layers; ++l) {
      if (l > 0) {
        // the buffers are those of layer l - 3
        if (g.tid() == 0) {
          if (l > 2) ffn_wait_count(&p.sync[kStepCombined], (l - 2) * grid, r.ab, 22, (uint32_t)l);
          st.word[1] = *r.ab.flag;
        }
        g.sync();
        if (st.word[1]) return;
        if (g.tid() < 4) tma_prefetch_map(&w.map[(first_set + l) % sets][g.tid()]);
        if (route.layer(g, (layers - 1 - l) % 3) < 0) return;
      }
      FfnPlanS plan;
      plan.off = st.off; plan.cum = st.cum; plan.ids = st.ids;
      ffn_plan(plan, a, ffn_slots(g, st.off, a.num_local_experts, st.cum, st.ids, st.scan));
      const int total = plan.total();
      int first = pair - base;
      if (first < 0) first += npairs;
      base = (base + total) % npairs;
      for (bool last = false; !last; first += kStepListUnits * npairs) {
        int count = first < total ? (total - first + npairs - 1) / npairs : 0;
        last = count <= kStepListUnits;
        if (!last) count = kStepListUnits;
        if (g.tid() == 0) st.word[1] = mbar_wait(&st.lempty[half], half_ph ^ 1u, r.ab, 23);
        g.sync();
        if (!st.word[1]) return;             // the half may still be read
        plan.list(r.sm.list + half * kStepListUnits, count, first, npairs, total, g.tid(), g.size());
        if (g.tid() == 0) { st.head[half * 2] = count; st.head[half * 2 + 1] = last; }
        g.sync();
        if (g.tid() == 0) mbar_arrive(&st.lfull[half]);
        if (++half == 2) { half = 0; half_ph ^= 1u; }
      }
    }
    return;
  }
  if (r.warp == 1 && r.rank != 0) return;

  int half = 0; uint32_t half_ph = 0;
  const bool epilogue = r.warp >= 2 && r.warp < 2 + kFfnEpiWarps, tokens = r.warp >= 2 + kFfnEpiWarps;
  const bool two = route.two();
  const EpilogueGroup g;
  bool go = true;
  // One round more than there are layers: the sums of a layer are taken in the next one.
  for (int l = 0; l <= layers && go; ++l) {
    if (l == layers && !epilogue) break;
    const int set = (layers + 2 - l) % 3, par = two ? (layers + 1 - l) & 1 : 0;
    if (l < layers) {
      r.actmap = reinterpret_cast<const CUtensorMap*>(p.map_act[par]);
      r.act_rows = reinterpret_cast<uint8_t*>(p.act[par]);
      r.y_rows = reinterpret_cast<uint8_t*>(p.y[par]);
      // rows that a CTA may still be summing: those of the layer before, or of the one before that
      const int summed = two ? l - 1 : l;
      if (summed > 0) { r.y_free = &p.sync[kStepCombined]; r.y_free_want = summed * grid; }
      if (epilogue || tokens) {
        if (r.lane == 0) ffn_wait_count(&p.sync[kStepRouted], (l + 1) * grid, r.ab, 19, (uint32_t)l);
        __syncwarp();
      }
    }
    bool pending = l > 0;              // sums of the layer before
    for (bool last = false; !last;) {
      const uint4* list = r.sm.list + half * kStepListUnits;
      int got = 0, count = 0;
      last = true;
      if (l < layers) {
        if (r.lane == 0) got = mbar_wait(&st.lfull[half], half_ph, r.ab, 24);
        got = __shfl_sync(0xffffffffu, got, 0);
        if (got) {
          count = *reinterpret_cast<volatile int*>(&st.head[half * 2]);
          last = *reinterpret_cast<volatile int*>(&st.head[half * 2 + 1]) != 0;
        } else {
          go = false;                  // an epilogue warp goes on to the end of the layer, where all of them meet
        }
      }
      if (r.warp == 0) r.weights(list, count, w.map[(first_set + l) % sets]);
      else if (r.warp == 1) r.mma(list, count);
      else if (tokens) { if (count > 0) r.tokens(list, count, r.warp - 2 - kFfnEpiWarps, p.pair_token[set], p.ffn_done[set]); }
      else {
        int begin = 0;
#pragma unroll 1
        do {
          int end = count;             // units ahead of the pending sums
          if (pending) {
            if (!two) end = 0;
            else
              for (int i = 0; i < count; i += 32) {
                const uint32_t down = __ballot_sync(0xffffffffu, i + r.lane < count && r.listed(list, i + r.lane).fc());
                if (down) { end = i + __ffs(down) - 1; break; }
              }
          }
          r.epilogue(list, begin, end, r.warp - 2, a.pair_prob ? p.pair_prob[set] : nullptr, p.ffn_done[set]);
          begin = end;
          if (pending && (begin < count || last)) {
            // This CTA's share of the sums, behind the experts of all CTAs.
            pending = false;
            if (g.tid() == 0) {
              ffn_wait_count(&p.sync[kStepExperts], l * grid, r.ab, 25, (uint32_t)l);
              // No rows to sum (the sums are zero) where nothing was routed or this CTA has given up: the list may still hold
              // positions of an earlier, larger step.
              st.word[2] = *r.sm.abort_flag || route.T == 0 ? 0 : p.layer.cmb.topk;
            }
            g.sync();
            McbCombineArgs cmb = p.layer.cmb;
            cmb.pair_pos = p.pair_pos[(layers - l) % 3];

            cmb.topk = st.word[2];
            cmb.y = p.y[two ? (layers - l) & 1 : 0];
            combine_body<false>(p.layer.ctx, cmb, 0u, r.warp - 2, kFfnEpiWarps);
            g.sync();
            if (g.tid() == 0) {
              __threadfence();
              atomicAdd(&p.sync[kStepCombined], 1);
            }
          }
        } while (begin < count);
      }
      __syncwarp();
      if (got && r.lane == 0) mbar_arrive(&st.lempty[half]);
      if (++half == 2) { half = 0; half_ph ^= 1u; }
    }
    if (epilogue && l < layers) {
      g.sync();
      if (g.tid() == 0) {
        __threadfence();
        atomicAdd(&p.sync[kStepExperts], 1);
        st.word[0] = *r.sm.abort_flag;
      }
      g.sync();
      go = st.word[0] == 0;
    }
  }
  if (r.warp == 0) r.drain();
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFfnThreads, 1)
moe_step_kernel(const __grid_constant__ McbMoeStepArgs p, const __grid_constant__ StepWeights w, int layers, int first_set, int sets) {
  const McbCtx& c = p.layer.ctx;
  const FfnSmem sm;
  const StepSmem st(sm);
  __shared__ LocalRanges rows;
  if (threadIdx.x == 0) {
    const uint32_t readers = (cluster_ctarank() == 0 ? 2 : 1) + kFfnEpiWarps + kStepTokWarps;
    for (int i = 0; i < 2; ++i) { mbar_init(&st.lfull[i], 1); mbar_init(&st.lempty[i], readers); }
  }
  if (threadIdx.x >= 128 && threadIdx.x < 129 + kFfnMaxGroups)
    tma_prefetch_map(threadIdx.x == 128 ? (const void*)p.map_x : (const void*)p.map_act[0][threadIdx.x - 129]);
  if (threadIdx.x >= 160 && threadIdx.x < 164) tma_prefetch_map(&w.map[first_set % sets][threadIdx.x - 160]);
  ffn_setup<false>(nullptr);
  pdl_wait();
  pdl_launch_dependents();
  // The rows of this rank, which are all rows.  Counts that the all-gather would refuse are refused.
  const McbAgvArgs& agv = p.layer.agv;
  int n = *agv.n_local;
  const int valid = agv.step_meta[0], offset = agv.step_meta[1];
  const bool bad = n < 0 || n > agv.cap || offset != 0 || valid > n;
  if (bad) {
    if (threadIdx.x == 0 && agv.step_meta[2] > 0)
      report_error(c, n > agv.cap ? MCB_ERR_CAPACITY : MCB_ERR_BOUNDS, (uint32_t)agv.site, blockIdx.x, (uint32_t)n, (uint32_t)offset);
    n = 0;
  }
  if (threadIdx.x == 0)
    for (int t = 0; t < LocalRanges::R; ++t) {
      const bool used = t < agv.num_tensors;
      rows.set(t, used ? agv.src[t] : nullptr, used ? c.heap_local + agv.dst_off[t] : nullptr, 0, used ? (long long)n * agv.row_bytes[t] : 0);
    }
  int T = bad ? 0 : valid;
  if (T < 0) T = 0;
  if (T > p.layer.route.max_tokens) T = p.layer.route.max_tokens;
  const Abort ab{sm.abort_flag, p.layer.ffn.status, p.layer.ffn.timeout_ns};
  StepRoute route(p, rows, st, ab, T);
  __syncthreads();
  const int mx = route.layer(BlockGroup{}, (layers - 1) % 3);      // the first layer's by all warps
  const int n_slot = ffn_token_tile(mx);
  __syncthreads();
  if (mx >= 0) {
    if (n_slot <= kFfnDoubleN) step_roles<2>(p, w, route, layers, first_set, sets, n_slot);
    else step_roles<1>(p, w, route, layers, first_set, sets, n_slot);
  }
  ffn_teardown();
  if (threadIdx.x == 0) {
    __threadfence();
    st.word[0] = atomicAdd(&p.sync[kStepLeft], 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (st.word[0]) {                                                    // last CTA out: the counters back to zero
    for (int i = threadIdx.x; i < 3 * p.layer.route.num_local_experts; i += blockDim.x) p.expert_count[i] = 0;
    if (threadIdx.x <= kStepLeft / 32) p.sync[threadIdx.x * 32] = 0;
  }
}

}  // namespace mcb

using namespace mcb;

extern "C" {

int mcb_sizeof_step_args() { return (int)sizeof(McbMoeStepArgs); }
int mcb_step_smem_bytes() { return kStepSmemBytes; }

namespace {

struct Range { uintptr_t at; uint64_t bytes; };
bool overlap(const Range& a, const Range& b) { return a.bytes && b.bytes && a.at < b.at + b.bytes && b.at < a.at + a.bytes; }
Range range(const void* p, uint64_t bytes) { return Range{reinterpret_cast<uintptr_t>(p), bytes}; }

// Whether set s of the plan differs from set 0 in its weights alone.
bool same_but_weights(const McbLayerArgs& a, const McbLayerArgs& b) {
  McbFfnArgs f = b.ffn;
  f.w1 = a.ffn.w1; f.w2 = a.ffn.w2; f.tmaps = a.ffn.tmaps;
  return !memcmp(&f, &a.ffn, sizeof f) && !memcmp(&a.ctx, &b.ctx, sizeof a.ctx) && !memcmp(&a.agv, &b.agv, sizeof a.agv) &&
         !memcmp(&a.route, &b.route, sizeof a.route) && !memcmp(&a.cmb, &b.cmb, sizeof a.cmb) && a.local_ids == b.local_ids &&
         a.local_probs == b.local_probs;
}

// The rows of this rank's tokens where its all-gather reads them, if the layers can go into one launch.  Null where they cannot: more
// ranks than one, rows or routing that are not read there, plans that do not fit together or differ in more than their weights, too
// many experts, a phase trace, or a layer that writes what the next one reads (rows taken from the output of the layer before, say)
// or writes memory by two ways (an output in the activations, which a layer of its own is done with by then).
const void* joined_rows(const McbLayerArgs* sets, int num_sets, const McbMetaArgs* meta) {
  if (!sets || num_sets < 1 || !meta) return nullptr;
  const McbLayerArgs& p = sets[0];
  const McbRouteArgs& r = p.route;
  const McbFfnArgs& f = p.ffn;
  const McbAgvArgs& g = p.agv;
  const McbCombineArgs& cmb = p.cmb;
  if (p.ctx.world != 1 || p.trace || !p.local_ids || r.num_local_experts > kStepMaxExperts) return nullptr;
  for (int s = 1; s < num_sets; ++s)
    if (!same_but_weights(p, sets[s]) || sets[s].trace) return nullptr;
  if (f.pair_token != r.pair_token || (f.pair_prob && f.pair_prob != r.pair_prob) || f.expert_offset != r.expert_offset ||
      f.ffn_done != r.ffn_done || f.num_local_experts != r.num_local_experts)
    return nullptr;
  if (cmb.y != f.y || cmb.pair_pos != r.pair_pos || cmb.topk != r.topk || cmb.hidden != f.hidden || cmb.n_local != g.n_local ||
      cmb.step_meta != g.step_meta || r.num_tokens != g.step_meta || meta->n_local != g.n_local || meta->step_meta != g.step_meta ||
      meta->cap > g.cap || meta->cap > r.max_tokens || meta->cap > cmb.cap)
    return nullptr;
  const void* x = nullptr;
  for (int t = 0; t < g.num_tensors; ++t)
    if (p.ctx.heap_local + g.dst_off[t] == f.x && g.row_bytes[t] == 2u * (uint32_t)f.hidden) x = g.src[t];
  const uint64_t rows = (uint64_t)g.cap, pairs = (uint64_t)r.max_pairs;
  const Range written[] = {range(f.act, pairs * f.intermediate * 2), range(f.y, pairs * f.hidden * 2),
                           range(cmb.out, (uint64_t)cmb.cap * f.hidden * 2)};
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < i; ++j)
      if (overlap(written[i], written[j])) return nullptr;
  for (int t = 0; t < g.num_tensors; ++t) {
    for (const Range& w : written)      // a row written by two ways has the order of its layers
      if (overlap(w, range(p.ctx.heap_local + g.dst_off[t], rows * g.row_bytes[t]))) return nullptr;
    const Range src = range(g.src[t], rows * g.row_bytes[t]);
    for (const Range& w : written)
      if (overlap(src, w)) return nullptr;
    for (int u = 0; u < g.num_tensors; ++u)
      if (overlap(src, range(p.ctx.heap_local + g.dst_off[u], rows * g.row_bytes[u]))) return nullptr;
  }
  return x;
}

bool configure_step_kernel() {
  static const bool ok = cudaFuncSetAttribute(moe_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmemBytes) == cudaSuccess;
  return ok;
}

}  // namespace

// Whether several layers of a step can go into one launch.
int mcb_moe_step_joins(const McbLayerArgs* sets, int num_sets, const McbMetaArgs* meta) { return joined_rows(sets, num_sets, meta) != nullptr; }

// Fills `out` (64-byte aligned host memory) for steps of several layers in one launch and returns 0, or 1 where the layers cannot
// go into one (mcb_moe_step_joins).  The further buffers come from the caller: two times pair_token and
// pair_prob (route.max_pairs each), pair_pos (max_tokens x topk, -1) and ffn_done (num_local_experts), expert_count (3 x
// num_local_experts) and sync (MCB_STEP_SYNC_WORDS), all zero but for pair_pos; act and y of two_rows rows, or null.
int mcb_prepare_moe_step(McbMoeStepArgs* out, const McbLayerArgs* sets, int num_sets, const McbMetaArgs* meta, int32_t* pair_token,
                         float* pair_prob, int32_t* pair_pos, int32_t* ffn_done, int32_t* expert_count, int32_t* sync, void* act,
                         void* y, int two_rows) {
  const void* x = joined_rows(sets, num_sets, meta);
  if (!x || !out || !pair_token || !pair_prob || !pair_pos || !ffn_done || !expert_count || !sync) return 1;
  const McbLayerArgs& p = sets[0];
  const McbRouteArgs& r = p.route;
  const McbFfnArgs& f = p.ffn;
  const uint64_t rows = (uint64_t)p.agv.cap, pairs = (uint64_t)r.max_pairs;
  memset(out, 0, sizeof *out);
  out->layer = p;
  out->ids = p.local_ids;
  out->probs = p.local_probs;
  out->x = x;
  for (int i = 0; i < 3; ++i) {
    out->pair_token[i] = i ? pair_token + (i - 1) * pairs : r.pair_token;
    out->pair_prob[i] = i ? pair_prob + (i - 1) * pairs : r.pair_prob;
    out->pair_pos[i] = i ? pair_pos + (uint64_t)(i - 1) * r.max_tokens * r.topk : r.pair_pos;
    out->ffn_done[i] = i ? ffn_done + (i - 1) * r.num_local_experts : r.ffn_done;
  }
  out->two_rows = act && y ? two_rows : 0;
  out->act[0] = f.act; out->act[1] = out->two_rows ? act : f.act;
  out->y[0] = f.y;     out->y[1] = out->two_rows ? y : f.y;
  out->expert_count = expert_count;
  out->sync = sync;
  if (make_tmap_bf16(out->map_x, x, rows, (uint64_t)f.hidden, 1)) return 1;
  static_assert(sizeof out->map_act[0] == kFfnMaxGroups * sizeof(CUtensorMap), "a map per box");
  for (int i = 0; i < 2; ++i)
    for (int b = 0; b < kFfnMaxGroups; ++b)
      if (make_tmap_bf16(out->map_act[i][b], out->act[i], i && out->two_rows ? (uint64_t)out->two_rows : pairs, (uint64_t)f.intermediate,
                         4 * (b + 1)))
        return 1;
  return 0;
}

// `num_layers` layers of a step prepared as above, from layer `first` of the step on (layer l uses weight set l % num_sets).
int mcb_launch_moe_step(const McbMoeStepArgs* p, const McbLayerArgs* sets, int num_sets, int first, int num_layers, int grid, int pdl,
                        cudaStream_t stream) {
  if (!p || !sets || num_sets < 1 || first < 0 || num_layers < 1 || grid < 1 || grid > MCB_MAX_BLOCKS) return cudaErrorInvalidValue;
  if (num_sets > MCB_STEP_SETS && num_layers > MCB_STEP_SETS) return cudaErrorInvalidValue;
  if (!configure_step_kernel()) return cudaErrorUnknown;
  StepWeights w;
  memset(&w, 0, sizeof w);
  const bool all = num_sets <= MCB_STEP_SETS;
  const int n = all ? num_sets : num_layers;
  for (int i = 0; i < n; ++i) {
    const McbFfnArgs& f = sets[all ? i : (first + i) % num_sets].ffn;
    memcpy(w.map[i], reinterpret_cast<const uint8_t*>(f.tmaps) + MCB_FFN_MAP_W1 * sizeof(CUtensorMap), sizeof w.map[i]);
  }
  // Waits of CTAs for one another: all must be resident.  The kernel runs in CTA pairs: an odd grid is rounded down.
  return launch_kernel(moe_step_kernel, dim3(grid < 2 ? 2 : grid & ~1), dim3(kFfnThreads), kStepSmemBytes, stream, pdl, true, *p, w, num_layers,
                       all ? first % num_sets : 0, n);
}

}  // extern "C"
