"""Expert path on one GPU: routing kernel, tcgen05 grouped GEMMs (FC1 with fused token gather and
SwiGLU, FC2 with routing-weight epilogue) and the combine, each against the fp32 CPU oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(T, E, K, H, I, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(T, H, device=DEV, generator=g).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(T)])
    w = torch.rand(T, K, device=DEV, generator=g) + 0.1
    return x, idx, w


@pytest.mark.parametrize("T,E,K,H,I", [(200, 8, 4, 256, 128), (37, 4, 2, 1024, 1024), (300, 2, 2, 512, 256),
                                       (4500, 8, 4, 256, 128)])
def test_route_fc1_fc2_combine_against_oracle(world1, T, E, K, H, I):
    from moe_comms_benchmarking_b200.ops import _ext, oracle
    from moe_comms_benchmarking_b200.ops.experts import (ExpertCombinePlan, ExpertWeights, GroupedGemmPlan, RouteBuffers,
                                                         RoutePlan)
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    x, idx, w = _case(T, E, K, H, I, 3)
    cap = T + 5
    heap = SymmetricHeap(world1, cap * H * 2 + (1 << 20), DEV)
    partial = heap.alloc("partial", [cap, H], torch.bfloat16)
    status = heap.status
    xs = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV); xs[:T] = x
    idxs = torch.zeros(cap, K, dtype=torch.int64, device=DEV); idxs[:T] = idx
    ws = torch.zeros(cap, K, device=DEV); ws[:T] = w
    ntok = torch.tensor([T], dtype=torch.int32, device=DEV)
    meta = torch.tensor([T, 0, T, 1], dtype=torch.int32, device=DEV)
    route = RouteBuffers(cap, K, E, DEV)
    weights = ExpertWeights(E, H, I, DEV, seed=5, std=0.05, layout="split")
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(route.max_pairs, H, dtype=torch.bfloat16, device=DEV)
    out = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV)
    rp = RoutePlan(route, idxs, ws, ntok, expert_begin=0, status=status, grid=7)
    fc1 = GroupedGemmPlan(_ext.GEMM_FC1, weights.map_gate_up, route, xs, act, 2 * I, H, status, grid=5)
    fc2 = GroupedGemmPlan(_ext.GEMM_FC2, weights.map_down, route, act, y, H, I, status, grid=148)
    comb = ExpertCombinePlan(heap, y, route, partial, out, ntok, meta, cap, grid=16, threads=256)
    for rep in range(2):        # twice: scratch counters must come back clean
        rp.launch(); fc1.launch(); fc2.launch(); comb.launch()
        torch.cuda.synchronize()
        heap.check_status()
        # routing: per-expert segments hold exactly the tokens routed to that expert
        off = route.expert_offset.cpu().tolist()
        ptok, pprob, ppos = route.pair_token.cpu(), route.pair_prob.cpu(), route.pair_pos.cpu()
        assert off[E] == T * K
        ntiles = int(route.num_m_tiles)
        assert ntiles == sum((off[e + 1] - off[e] + 127) // 128 for e in range(E))
        for e in range(E):
            want = (idx.cpu() == e).any(dim=1).nonzero().flatten().tolist()
            assert sorted(ptok[off[e]:off[e + 1]].tolist()) == want
        tt, kk = torch.arange(T).repeat_interleave(K), torch.arange(K).repeat(T)
        pos = ppos[:T].flatten().long()
        assert (pos >= 0).all() and torch.equal(ptok[pos].long(), tt)
        assert torch.equal(pprob[pos], w.cpu().flatten())
        pair_expert = torch.bucketize(pos, torch.tensor(off[1:]), right=True)
        assert torch.equal(pair_expert, idx.cpu().flatten())
        # FC1: act rows against silu(x Wg^T) * (x Wu^T)
        P = off[E]
        pe = torch.bucketize(torch.arange(P), torch.tensor(off[1:]), right=True)
        xg = x.cpu().float()[ptok[:P].long()]
        wgu = weights.w_gate_up.cpu().float()
        gu = torch.cat([xg[off[e]:off[e + 1]] @ wgu[e].t() for e in range(E)])
        want_act = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
        got_act = act[:P].float().cpu()
        s = float(want_act.abs().max())
        assert float((got_act - want_act).abs().max()) < 0.02 * s + 1e-3, "FC1"
        # FC2 on the kernel's own bf16 activations
        wd = weights.w_down.cpu().float()
        want_y = torch.cat([got_act[off[e]:off[e + 1]] @ wd[e].t() for e in range(E)]) * pprob[:P].unsqueeze(1)
        got_y = y[:P].float().cpu()
        s = float(want_y.abs().max())
        assert float((got_y - want_y).abs().max()) < 0.02 * s + 1e-3, "FC2"
        # whole layer against the oracle
        ref = oracle.moe_layer(x.cpu(), idx.cpu(), w.cpu(), weights.w_gate_up.cpu(), weights.w_down.cpu())
        s = float(ref.abs().max())
        assert float((out[:T].float().cpu() - ref).abs().max()) < 0.03 * s + 1e-3, "layer"


@pytest.mark.parametrize("T,E,K,H,I,grid", [(64, 16, 4, 256, 128, 148), (37, 4, 2, 1024, 1024, 24), (700, 2, 2, 512, 256, 5),
                                            (3, 8, 2, 256, 128, 148), (4500, 8, 4, 256, 128, 148),
                                            (400, 8, 2, 256, 256, 3), (400, 8, 2, 256, 256, 5)])
def test_expert_ffn_weights_as_m_against_oracle(world1, T, E, K, H, I, grid):
    """The grouped FFN with the weights as the M operand of a CTA pair (gate/up + SwiGLU + down in one
    persistent launch): experts with no token, with a few, with more than 128 (one column block per pipeline
    stage) and more than 256 (several chunks), more units than CTA pairs, an odd grid, interleaved
    gate/up rows."""
    from moe_comms_benchmarking_b200.ops import oracle
    from moe_comms_benchmarking_b200.ops.experts import ExpertFfnPlan, ExpertWeights, RouteBuffers, RoutePlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    x, idx, w = _case(T, E, K, H, I, 9)
    if T == 3:
        idx = idx % 3                       # most experts stay empty
        idx[:, 1] = (idx[:, 0] + 1) % 3
    cap = T + 5
    heap = SymmetricHeap(world1, 1 << 20, DEV)
    xs = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV); xs[:T] = x
    idxs = torch.zeros(cap, K, dtype=torch.int64, device=DEV); idxs[:T] = idx
    ws = torch.zeros(cap, K, device=DEV); ws[:T] = w
    ntok = torch.tensor([T], dtype=torch.int32, device=DEV)
    route = RouteBuffers(cap, K, E, DEV)
    weights = ExpertWeights(E, H, I, DEV, seed=5, std=0.05)
    from moe_comms_benchmarking_b200.ops.experts import pack_weight_tiles
    assert torch.equal(pack_weight_tiles(ExpertWeights.interleave(weights.w_gate_up)), weights.w1)
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(route.max_pairs, H, dtype=torch.bfloat16, device=DEV)
    rp = RoutePlan(route, idxs, ws, ntok, expert_begin=0, status=heap.status, grid=7)
    ffn = ExpertFfnPlan(weights, route, xs, act, y, heap.status, grid=grid)
    for rep in range(2):
        act.fill_(float("nan")); y.fill_(float("nan"))
        rp.launch(); ffn.launch()
        torch.cuda.synchronize()
        heap.check_status()
        off = route.expert_offset.cpu().tolist()
        P = off[E]
        assert P == T * K and int(route.max_rows) == max(off[e + 1] - off[e] for e in range(E))
        ptok, pprob = route.pair_token.cpu(), route.pair_prob.cpu()
        xg = x.cpu().float()[ptok[:P].long()]
        wgu = weights.w_gate_up.cpu().float()
        gu = torch.cat([xg[off[e]:off[e + 1]] @ wgu[e].t() for e in range(E)])
        want_act = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
        got_act = act[:P].float().cpu()
        s = float(want_act.abs().max())
        assert float((got_act - want_act).abs().max()) < 0.02 * s + 1e-3, "gate/up + SwiGLU"
        wd = weights.w_down.cpu().float()
        want_y = torch.cat([got_act[off[e]:off[e + 1]] @ wd[e].t() for e in range(E)]) * pprob[:P].unsqueeze(1)
        got_y = y[:P].float().cpu()
        s = float(want_y.abs().max())
        assert float((got_y - want_y).abs().max()) < 0.02 * s + 1e-3, "down"
        # per-token sum of the pair rows against the full-layer oracle
        pos = route.pair_pos[:T].cpu().long()
        out = got_y[pos.flatten()].view(T, K, H).sum(1)
        ref = oracle.moe_layer(x.cpu(), idx.cpu(), w.cpu(), weights.w_gate_up.cpu(), weights.w_down.cpu())
        assert float((out - ref).abs().max()) < 0.03 * float(ref.abs().max()) + 1e-3, "layer"


@pytest.mark.parametrize("E,used", [(1024, 1024), (1024, 1023), (700, 640)])
def test_expert_ffn_many_experts(world1, E, used):
    """Up to as many experts as there may be, most with a token or two, some with two and three chunks, the last one empty or not: every pair's output against
    fp32 with the same weights."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertFfnPlan, ExpertWeights, RouteBuffers, RoutePlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    T, K, H, I = 1900, 2, 256, 128
    x, _, w = _case(T, 8, K, H, I, 47)
    t = torch.arange(T, device=DEV)
    large = torch.tensor([3, 300, used - 1], device=DEV)                       # 600, 300 and 257 tokens, and one to three more
    second = torch.cat([large[0].expand(600), large[1].expand(300), large[2].expand(257), t[1157:] * 7 % used])
    idx = torch.stack([t % used, second], dim=1)
    idx[:, 1] = torch.where(idx[:, 0] == idx[:, 1], (idx[:, 1] + 1) % used, idx[:, 1])
    counts = torch.bincount(idx.flatten(), minlength=E)
    assert bool((counts[:used] > 0).all()) and int(counts.max()) > 512 and int((counts > 256).sum()) == 3
    heap = SymmetricHeap(world1, 1 << 20, DEV)
    route = RouteBuffers(T, K, E, DEV)
    weights = ExpertWeights(E, H, I, DEV, seed=5, std=0.05)
    act = torch.full((route.max_pairs, I), float("nan"), dtype=torch.bfloat16, device=DEV)
    y = torch.full((route.max_pairs, H), float("nan"), dtype=torch.bfloat16, device=DEV)
    RoutePlan(route, idx, w, torch.tensor([T], dtype=torch.int32, device=DEV), 0, heap.status).launch()
    ExpertFfnPlan(weights, route, x, act, y, heap.status).launch()
    torch.cuda.synchronize()
    heap.check_status()
    off, token = route.expert_offset.tolist(), route.pair_token.long()
    w1, w2 = weights.w_gate_up, weights.w_down
    # Rounded to bf16 once (2^-9, and as much again where that falls on the other side) from fp32 sums: 256 products whose magnitudes add up to about 10,
    # each partial sum within 2^-23, 3e-4.
    close = lambda got, want: bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 3e-4).all())
    assert off[E] == T * K and torch.equal(route.expert_offset[1:].long() - route.expert_offset[:-1].long(), counts)
    for e in range(E):
        lo, hi = off[e], off[e + 1]
        if lo == hi:
            continue
        gu = x[token[lo:hi]].double() @ w1[e].double().t()
        assert close(act[lo:hi], torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]), f"activations of expert {e}"
        down = act[lo:hi].double() @ w2[e].double().t()                         # of the kernel's own activations
        assert close(y[lo:hi], down * route.pair_prob[lo:hi].double().unsqueeze(1)), f"outputs of expert {e}"


@pytest.mark.parametrize("W,B,ll_rows", [(2, 96, 0), (4, 40, 0), (2, 7, 16), (4, 1, 16)])
def test_moe_layer_kernel_emulated_ranks(lib, W, B, ll_rows):
    """The whole-layer kernel (dispatch, routing, experts, combine in one cooperative launch) with W
    ranks emulated on one GPU: the cross-rank protocol of the product kernel against the oracle,
    twice in a row (every counter must come back clean), with an uneven split and packet mode."""
    from moe_comms_benchmarking_b200.ops import _ext, oracle
    from moe_comms_benchmarking_b200.ops.dense import agv_ll_stage_bytes
    from moe_comms_benchmarking_b200.ops.experts import ExpertWeights, RouteBuffers
    from moe_comms_benchmarking_b200.parallel.emulation import EmuWorld
    E_loc, K, H, I = 4, 3, 256, 128
    E = E_loc * W
    counts = [B // W + (1 if r < B % W else 0) for r in range(W)]
    counts[0], counts[-1] = counts[0] + counts[-1] // 2, counts[-1] - counts[-1] // 2     # uneven
    cap, g = max(counts), max(counts) * W
    w = EmuWorld(W, 8 << 20, DEV)
    dst = [w.alloc([g, H], torch.bfloat16), w.alloc([g, K], torch.int64), w.alloc([g, K], torch.float32)]
    partial = w.alloc([2, g, H], torch.bfloat16)
    ll = w.alloc([max(16, agv_ll_stage_bytes(ll_rows, [H * 2, K * 8, K * 4]))], torch.uint8)
    gen = torch.Generator(device=DEV).manual_seed(41)
    ranks = []
    for r in range(W):
        route = RouteBuffers(g, K, E_loc, DEV)
        ranks.append(dict(
            weights=ExpertWeights(E_loc, H, I, DEV, seed=100 + r, std=0.05), route=route, expert_begin=r * E_loc,
            src=(torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV), torch.zeros(cap, K, dtype=torch.int64, device=DEV),
                 torch.zeros(cap, K, device=DEV)),
            dst=tuple(t[r] for t in dst), partial=partial[r], ll_stage=ll[r],
            n_local=torch.tensor([counts[r]], dtype=torch.int32, device=DEV),
            step_meta=torch.zeros(4, dtype=torch.int32, device=DEV),
            act=torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV),
            y=torch.zeros(route.max_pairs, H, dtype=torch.bfloat16, device=DEV),
            out=torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV)))
    wgu = torch.cat([d["weights"].w_gate_up.cpu() for d in ranks])
    wd = torch.cat([d["weights"].w_down.cpu() for d in ranks])
    for rep in range(2):
        xs, idxs, ps = [], [], []
        for r, d in enumerate(ranks):
            n = counts[r]
            x = torch.randn(n, H, device=DEV, generator=gen).to(torch.bfloat16)
            idx = torch.stack([torch.randperm(E, device=DEV, generator=gen)[:K] for _ in range(n)]) if n else \
                torch.zeros(0, K, dtype=torch.int64, device=DEV)
            p = torch.rand(n, K, device=DEV, generator=gen) + 0.1
            d["src"][0][:n], d["src"][1][:n], d["src"][2][:n] = x, idx, p
            d["out"].zero_()
            xs.append(x.cpu()); idxs.append(idx.cpu()); ps.append(p.cpu())
        w.metadata([d["n_local"] for d in ranks], [d["step_meta"] for d in ranks], cap)
        w.moe_layer(ranks, grid=148 // W, topk=K, cap=cap, ll_rows=ll_rows)
        w.check_status()
        for r, d in enumerate(ranks):
            ref = oracle.moe_layer(xs[r], idxs[r], ps[r], wgu, wd)
            if counts[r]:
                s = float(ref.abs().max())
                assert float((d["out"][:counts[r]].float().cpu() - ref).abs().max()) < 0.03 * s + 1e-3, f"rank {r} rep {rep}"


def test_fused_dispatcher_routes_more_than_one_block_of_entries(world1):
    """More (token, expert) entries than every block counts by itself, so the routing that shares counts through global
    counters and a grid-wide barrier runs INSIDE the cooperative layer kernel; a sample of tokens is checked against
    the oracle."""
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    from moe_comms_benchmarking_b200.utils.inputs import make_inputs
    cfg = Config(num_experts=16, topk=8, hidden=256, intermediate=128, ep_size=1, per_rank_cap=2304)
    d = FusedExpertDispatcher(cfg, world1, num_layers=1, weight_budget_gb=0.5)
    d.build()
    h, i, w = make_inputs(cfg, 2304, DEV)          # 18432 entries, 16 per thread are 6144
    d.setup_batch(h, i, w)
    for _ in range(2):
        d.decode_step(1)
        torch.cuda.synchronize()
        d.check_health()
    sample = torch.arange(0, 2304, 37)
    ref = d.reference_output(h[sample], i[sample], w[sample])
    s = float(ref.abs().max())
    assert float((d.out[sample].float().cpu() - ref).abs().max()) < 0.05 * s
    d.destroy()


@pytest.mark.parametrize("fuse,fuse_d", [(True, True), (False, False), (True, False), (False, True)])
def test_two_kernel_fused_dispatcher_world1(world1, fuse, fuse_d):
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    from moe_comms_benchmarking_b200.utils.inputs import make_inputs
    from moe_comms_benchmarking_b200.utils.timing import capture_graph
    cfg = Config(num_experts=16, topk=4, hidden=512, intermediate=256, ep_size=1, per_rank_cap=160)
    d = FusedExpertDispatcher(cfg, world1, num_layers=3, weight_budget_gb=1.0, fuse_combine=fuse, fuse_dispatch=fuse_d,
                              layer_kernel=False)
    d.build()
    for name, ok, detail in d.validate():
        assert ok, f"{name}: {detail}"
    h, i, w = make_inputs(cfg, 150, DEV)
    d.setup_batch(h, i, w)
    g = capture_graph(lambda: d.decode_step(3))
    g.replay()
    torch.cuda.synchronize()
    d.check_health()
    ref = d.reference_output(h, i, w, layer=2)
    s = float(ref.abs().max())
    assert float((d.out.float().cpu() - ref).abs().max()) < 0.05 * s
    d.destroy()


def test_layer_kernel_fused_dispatcher_world1(world1):
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    from moe_comms_benchmarking_b200.utils.inputs import make_inputs
    from moe_comms_benchmarking_b200.utils.timing import capture_graph
    cfg = Config(num_experts=16, topk=4, hidden=512, intermediate=256, ep_size=1, per_rank_cap=160)
    d = FusedExpertDispatcher(cfg, world1, num_layers=3, weight_budget_gb=1.0)
    d.build()
    for name, ok, detail in d.validate():
        assert ok, f"{name}: {detail}"
    h, i, w = make_inputs(cfg, 150, DEV)
    d.setup_batch(h, i, w)
    g = capture_graph(lambda: d.decode_step(3))
    g.replay()
    torch.cuda.synchronize()
    d.check_health()
    ref = d.reference_output(h, i, w, layer=2)
    s = float(ref.abs().max())
    assert float((d.out.float().cpu() - ref).abs().max()) < 0.05 * s
    d.destroy()


def test_layer_kernel_phase_trace_world1(world1):
    """The optional device trace of the layer kernel: seven phases in order, none negative, together no
    longer than the step they belong to; and the traced layer still computes the right rows."""
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    from moe_comms_benchmarking_b200.utils.inputs import make_inputs
    cfg = Config(num_experts=16, topk=4, hidden=512, intermediate=256, ep_size=1, per_rank_cap=96)
    d = FusedExpertDispatcher(cfg, world1, num_layers=1, weight_budget_gb=1.0, phase_trace=True)
    d.build()
    h, i, w = make_inputs(cfg, 80, DEV)
    d.setup_batch(h, i, w)
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    d.decode_step(1)                       # warm-up
    torch.cuda.synchronize()
    t0.record(); d.decode_step(1); t1.record()
    torch.cuda.synchronize()
    d.check_health()
    phases = d.layer_plan.phase_times()
    assert [n for n, _ in phases] == ["dispatch", "grid barrier", "routing", "grid barrier", "experts", "grid barrier", "combine"]
    assert all(us >= 0 for _, us in phases)
    total = sum(us for _, us in phases)
    assert 0 < total <= t0.elapsed_time(t1) * 1e3 + 50.0
    ref = d.reference_output(h, i, w, layer=0)
    assert float((d.out.float().cpu() - ref).abs().max()) < 0.05 * float(ref.abs().max())
    d.destroy()


@pytest.mark.parametrize("rows,H,I,grid", [
    ([1, 31, 32, 33, 0, 64], 256, 128, 148),             # gathered token rows: below, at and above a multiple of 32, an idle expert
    ([65, 0, 3], 512, 256, 6),                           # rows gathered past 64, fewer CTA pairs than units
    ([128, 97, 96, 127, 33, 0], 256, 128, 148),          # up to 32 gathered rows per producer, two column blocks per stage
    ([129, 1], 256, 128, 148),                           # one column block per stage; more CTAs than units
    ([256, 257, 0, 513, 5], 256, 384, 148),              # one, two and three chunks of an expert
    ([40] * 200, 512, 256, 2),                           # more units than one list holds
    ([2600, 300, 1, 900, 2400, 700], 256, 2048, 148),    # activations beyond the L2 bound, but too few experts for a distance
])
def test_expert_ffn_chunk_edges(world1, rows, H, I, grid):
    """expert_ffn_kernel where the token count of an expert meets the edges of its chunks, its token path and
    its unit list.  Tokens are routed to one expert each, so `rows` sets the counts exactly.  bf16 inputs with fp32
    sums: the error of an activation is its rounding to bf16 (2^-9 relative) plus that of its inputs' sum order."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertFfnPlan, ExpertWeights, RouteBuffers, RoutePlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    E, T = len(rows), sum(rows)
    g = torch.Generator(device=DEV).manual_seed(29)
    x = torch.randn(T, H, device=DEV, generator=g).to(torch.bfloat16)
    idx = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(rows, device=DEV))
    idx = idx[torch.randperm(T, device=DEV, generator=g)].view(T, 1).contiguous()
    w = torch.rand(T, 1, device=DEV, generator=g) + 0.1
    heap = SymmetricHeap(world1, 1 << 20, DEV)
    ntok = torch.tensor([T], dtype=torch.int32, device=DEV)
    route = RouteBuffers(T, 1, E, DEV)
    weights = ExpertWeights(E, H, I, DEV, seed=6, std=0.05)
    act = torch.zeros(T, I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)
    rp = RoutePlan(route, idx, w, ntok, expert_begin=0, status=heap.status)
    ffn = ExpertFfnPlan(weights, route, x, act, y, heap.status, grid=grid)
    for rep in range(2):
        act.fill_(float("nan")); y.fill_(float("nan"))
        rp.launch(); ffn.launch()
        torch.cuda.synchronize()
        heap.check_status()
        off, tok = route.expert_offset.tolist(), route.pair_token[:T].long()
        wgu, wd = weights.w_gate_up.float(), weights.w_down.float()
        for e in range(E):
            if not rows[e]:
                continue
            sl = slice(off[e], off[e + 1])
            gu = x.float()[tok[sl]] @ wgu[e].t()
            want = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
            assert float((act[sl].float() - want).abs().max()) < 2 ** -7 * float(want.abs().max()), f"expert {e} gate/up"
            want = act[sl].float() @ wd[e].t() * route.pair_prob[sl].unsqueeze(1)
            assert float((y[sl].float() - want).abs().max()) < 2 ** -7 * float(want.abs().max()), f"expert {e} down"


def _down_distance(rows, H, I, grid):
    """The numbering of the kernels (ffn_plan in mcb_ffn.cuh): experts with tokens, and how many of them the down units of one
    come behind its gate/up units."""
    active, chunks, grid = sum(r > 0 for r in rows), sum((r + 255) // 256 for r in rows), max(grid & ~1, 2)
    beyond = sum(rows) * I * 2 > 24 << 20                # bytes of activations that stay within L2
    down, both = H // 256 * chunks, (H + 2 * I) // 256 * chunks
    return active, min(active, max(grid * active // down, grid * 3 // 2 * active // both) + 2) if beyond else active


@pytest.mark.parametrize("rows,H,I,grid", [
    ([700, 300, 1, 900, 0, 600, 256, 257, 500, 1200], 1024, 2816, 14),     # seven CTA pairs, chunked, tiny and idle experts
    ([700, 300, 1, 900, 0, 600, 256, 257, 500, 1200], 1024, 2816, 15),
    ([96 + 5 * i for i in range(20)] + [0] + [110] * 40, 1024, 2048, 148), # one chunk each; the whole chip
    ([300, 40, 700] * 16, 4096, 896, 148),                                 # more down units than twice the gate/up units
    ([257] * 30, 2560, 1664, 6),                                           # a second chunk of one row, long distance in units
])
def test_expert_ffn_down_units_at_a_distance(world1, rows, H, I, grid):
    """Beyond the activations that stay within L2, down units follow the gate/up units of their expert at a distance of fewer
    experts than there are.  Tolerance as in the test of the chunks."""
    active, distance = _down_distance(rows, H, I, grid)
    assert 2 <= distance < active
    test_expert_ffn_chunk_edges(world1, rows, H, I, grid)


@pytest.mark.parametrize("rows", [
    [1, 15, 16, 17, 48, 49, 80, 81, 112, 113, 128],                                     # four token warps, every number of row groups
    [129, 144, 145, 160, 161, 176, 177, 192, 193, 208, 209, 224, 225, 240, 241, 256],   # six, dividing and not
    [272, 273, 289, 350, 512, 513, 529, 16],                                            # equal chunks on either side of a multiple of 16
])
def test_expert_ffn_row_groups(world1, rows):
    """Token rows in groups of four that the token warps share: where the groups do not divide by the warps, two of them fetch
    the same rows.  Tolerance as in the test of the chunks."""
    test_expert_ffn_chunk_edges(world1, rows, 512, 256, 148)


@pytest.mark.parametrize("W,B", [(2, 900), (2, 2200), (1, 1), (1, 2100)])
def test_moe_layer_kernel_routing_and_combine_branches(lib, W, B):
    """The whole-layer kernel where its routing and combine change form: four packs per lane in the combine (900 tokens),
    counts shared through global counters instead of taken by every block (from about 2050 tokens of top-3), with a
    peer and alone (ids read from the inputs, sums written straight to the output)."""
    test_moe_layer_kernel_emulated_ranks(lib, W, B, 0)


@pytest.mark.parametrize("T,K,H", [(1, 22, 1024), (3, 40, 264), (500, 5, 1032), (40, 8, 7168), (2600, 3, 256)])
def test_expert_combine_slices(world1, T, K, H):
    """One, two and four packs per lane, a ragged last slice, more than 32 routing slots, entries of other ranks (-1)."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertCombinePlan, RouteBuffers
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    g = torch.Generator(device=DEV).manual_seed(T + K)
    heap = SymmetricHeap(world1, T * H * 2 + (1 << 20), DEV)
    partial = heap.alloc("partial", [T, H], torch.bfloat16)
    route = RouteBuffers(T, K, K, DEV)
    y = torch.randn(route.max_pairs, H, device=DEV, generator=g).to(torch.bfloat16)
    pos = torch.randint(0, route.max_pairs, (T, K), device=DEV, generator=g, dtype=torch.int32)
    pos[torch.rand(T, K, device=DEV, generator=g) < 0.4] = -1
    route.pair_pos.copy_(pos)
    out = torch.full((T, H), float("nan"), dtype=torch.bfloat16, device=DEV)
    n = torch.tensor([T], dtype=torch.int32, device=DEV)
    meta = torch.tensor([T, 0, T, 1], dtype=torch.int32, device=DEV)
    ExpertCombinePlan(heap, y, route, partial, out, n, meta, T).launch()
    torch.cuda.synchronize()
    heap.check_status()
    live = (pos >= 0).unsqueeze(-1)
    ref = torch.stack([(y[pos[t].clamp(min=0).long()].float() * live[t]).sum(0) for t in range(T)])
    assert torch.allclose(out.float(), ref, rtol=2 ** -8, atol=1e-5)      # fp32 sums in another order, rounded once


@pytest.mark.parametrize("T,K,H,shift,own", [
    (4, 5, 512, 0, None), (148, 5, 512, 0, None), (149, 5, 512, 0, None),      # 296 warps: a slice of 512 bytes each, more of them: slices of 1024 bytes
    (150, 33, 528, 0, None), (3, 2, 16, 0, None),        # a ragged last slice of either, more ids than lanes, half a pack
    (9, 5, 520, 0, None), (9, 5, 512, 8, None),          # no packs of 32 bytes: by the length of a row, by where the rows lie
    (400, 4, 768, 0, (7, 210)), (400, 4, 768, 0, (300, 250)), (400, 4, 768, 0, (3, 0)),      # own rows inside, past the end, none
    (9, 5, 512, -1, None), (40, 4, 768, -1, (7, 21)),    # two blocks: the kernel of any world
])
def test_expert_combine_alone(world1, T, K, H, shift, own):
    """The sums of a world of one add a token's rows in the order of its ids, in fp32 from zero, and round once, whichever way they go;
    rows of others keep what they held."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertCombinePlan, RouteBuffers
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    grid, shift = (2, 0) if shift < 0 else (None, shift)
    g = torch.Generator(device=DEV).manual_seed(T * K + H)
    heap = SymmetricHeap(world1, T * H * 2 + (1 << 20), DEV)
    route = RouteBuffers(T, K, K, DEV)
    y = torch.randn(route.max_pairs * H + shift, device=DEV, generator=g).to(torch.bfloat16)[shift:].view(-1, H)
    pos = torch.randint(0, route.max_pairs, (T, K), device=DEV, generator=g, dtype=torch.int32)
    pos[torch.rand(T, K, device=DEV, generator=g) < 0.4] = -1
    pos[0] = -1
    route.pair_pos.copy_(pos)
    first, rows = own or (0, T)
    out = torch.full((T, H), 7.0, dtype=torch.bfloat16, device=DEV)
    n, meta = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([rows], [T, first, rows, 1]))
    plan = ExpertCombinePlan(heap, y, route, heap.alloc("partial", [T, H], torch.bfloat16), out, n, meta, T, grid=grid, threads=32)
    assert plan.grid == (2 if grid else 148 if H % 16 or shift else 296)
    plan.launch()
    torch.cuda.synchronize()
    heap.check_status()
    ref = torch.zeros(T, H, device=DEV)
    for k in range(K):
        ref += torch.where((pos[:, k] >= 0).unsqueeze(1), y[pos[:, k].clamp(min=0).long()].float(), torch.zeros(1, device=DEV))
    want = torch.full_like(out, 7.0)
    mine = ref[first:first + rows].to(torch.bfloat16)
    want[:mine.shape[0]] = mine
    assert torch.equal(out, want)


@pytest.mark.parametrize("form", ["gathered", "no_weights", "own", "own_weights", "hidden_only", "order"])
def test_layer_plan_follows_its_routing_plan(world1, form):
    """The layer kernel of a world of one routes by the ids and weights of its RoutePlan: the gathered ones, tensors of
    the caller's own, or weight 1, whatever tensors the all-gather carries and in whatever order."""
    from moe_comms_benchmarking_b200.ops import oracle
    from moe_comms_benchmarking_b200.ops.dense import AllGatherVPlan, MetadataPlan
    from moe_comms_benchmarking_b200.ops.experts import (ExpertCombinePlan, ExpertFfnPlan, ExpertWeights, MoeLayerPlan,
                                                         RouteBuffers, RoutePlan)
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    T, cap, E, K, H, I = 40, 44, 6, 3, 256, 128
    pad = lambda t: torch.cat([t, t[:cap - T]]).contiguous()
    x, idx, w = (pad(t) for t in _case(T, E, K, H, I, 17))
    _, own_idx, own_w = (pad(t) for t in _case(T, E, K, H, I, 18))
    heap = SymmetricHeap(world1, 2 << 20, DEV)
    gx, gi, gw = heap.alloc("gx", [cap, H], torch.bfloat16), heap.alloc("gi", [cap, K], torch.int64), heap.alloc("gw", [cap, K], torch.float32)
    pairs = {"hidden_only": [(gx, x)], "order": [(gw, w), (gx, x), (gi, idx)]}.get(form, [(gx, x), (gi, idx), (gw, w)])
    r_idx = own_idx if form in ("own", "hidden_only") else gi.tensor
    r_w = {"no_weights": None, "own": own_w, "own_weights": own_w, "hidden_only": own_w}.get(form, gw.tensor)
    n = torch.tensor([T], dtype=torch.int32, device=DEV)
    meta = torch.zeros(4, dtype=torch.int32, device=DEV)
    route = RouteBuffers(cap, K, E, DEV)
    weights = ExpertWeights(E, H, I, DEV, seed=19, std=0.05)
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(route.max_pairs, H, dtype=torch.bfloat16, device=DEV)
    out = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV)
    partial = heap.alloc("partial", [2, cap, H], torch.bfloat16)
    plan = MoeLayerPlan(heap, AllGatherVPlan(heap, [d for d, _ in pairs], [s for _, s in pairs], n, meta, cap),
                        RoutePlan(route, r_idx, r_w, meta[0:1], expert_begin=0, status=heap.status),
                        [ExpertFfnPlan(weights, route, gx.tensor, act, y, heap.status)],
                        ExpertCombinePlan(heap, y, route, partial, out, n, meta, cap), MetadataPlan(heap, n, meta, cap))
    used_idx = own_idx if form in ("own", "hidden_only") else idx
    used_w = {"no_weights": torch.ones_like(w), "own": own_w, "own_weights": own_w, "hidden_only": own_w}.get(form, w)
    ref = oracle.moe_layer(x[:T].cpu(), used_idx[:T].cpu(), used_w[:T].cpu(), weights.w_gate_up.cpu(), weights.w_down.cpu())
    for rep in range(2):        # twice: counters must come back clean
        out.fill_(float("nan"))
        plan.decode_step(1)
        torch.cuda.synchronize()
        heap.check_status()
        s = float(ref.abs().max())
        assert float((out[:T].float().cpu() - ref).abs().max()) < 0.03 * s + 1e-3, f"rep {rep}"


@pytest.mark.parametrize("rows", [[40, 10], [140, 3]])       # two column blocks per pipeline stage, and one
def test_expert_ffn_plan_at_once_on_another_stream(world1, rows):
    """A plan is ready when its constructor returns: plans over changing inputs, one after the other and each launched
    on a stream of its own while the stream that it was built on is still busy.  The reference rounds the activations by
    itself: one unit in the last place of bf16 (2^-8) apart for some, that and the rounding of y (2^-9) within 2^-6."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertFfnPlan, ExpertWeights, RouteBuffers, RoutePlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    E, T, H, I = len(rows), sum(rows), 256, 128
    idx = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(rows, device=DEV)).view(T, 1)
    w = torch.ones(T, 1, device=DEV)
    heap = SymmetricHeap(world1, 1 << 20, DEV)
    route = RouteBuffers(T, 1, E, DEV)
    rp = RoutePlan(route, idx, w, torch.tensor([T], dtype=torch.int32, device=DEV), expert_begin=0, status=heap.status)
    weights = ExpertWeights(E, H, I, DEV, seed=8, std=0.05)
    wgu, wd = weights.w_gate_up.float(), weights.w_down.float()
    bufs = [(torch.randn(T, H, device=DEV).to(torch.bfloat16), torch.zeros(T, I, dtype=torch.bfloat16, device=DEV),
             torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)) for _ in range(3)]
    side = torch.cuda.Stream()
    for i in range(9):
        x, act, y = bufs[i % 3]
        act.zero_(); y.zero_()
        rp.launch()
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)            # about 10 ms
        plan = ExpertFfnPlan(weights, route, x, act, y, heap.status)
        plan.launch(stream=side)
        side.synchronize()
        got, tok = y.float(), route.pair_token[:T].long()
        torch.cuda.synchronize()
        heap.check_status()
        for e, lo in ((0, 0), (1, rows[0])):
            gu = x.float()[tok[lo:lo + rows[e]]] @ wgu[e].t()
            want = (torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]).to(torch.bfloat16).float() @ wd[e].t()
            assert float((got[lo:lo + rows[e]] - want).abs().max()) < 2 ** -6 * float(want.abs().max()), f"plan {i} expert {e}"
        del plan


@pytest.mark.parametrize("grid", [2, 6, 148])
def test_expert_ffn_row_copy_counters_return(world1, grid):
    """Launches back to back with fewer and with more CTA pairs than units: the counters of the routing are back at zero, and the
    last launch is as right as the first."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertFfnPlan, ExpertWeights, RouteBuffers, RoutePlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    T, H, I = 290, 256, 128
    heap = SymmetricHeap(world1, 1 << 20, DEV)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    idx = (torch.arange(T, device=DEV) >= 150).long().view(T, 1)
    route = RouteBuffers(T, 1, 2, DEV)
    weights = ExpertWeights(2, H, I, DEV, seed=9, std=0.05)
    act, y = torch.zeros(T, I, dtype=torch.bfloat16, device=DEV), torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)
    rp = RoutePlan(route, idx, torch.ones(T, 1, device=DEV), torch.tensor([T], dtype=torch.int32, device=DEV), 0, heap.status)
    plan = ExpertFfnPlan(weights, route, x, act, y, heap.status, grid=grid)
    rows = []
    for n in (1, 60):
        for _ in range(n):
            rp.launch(); plan.launch()
        torch.cuda.synchronize()
        heap.check_status()
        assert route.sync.tolist() == [0] * 4
        rows.append(y[route.pair_pos.flatten().long()].clone())
    assert torch.equal(rows[0], rows[1])            # a token's row does not depend on its place among its expert's rows


@pytest.mark.parametrize("shape", [(3, 20), (1, 1, 60)])
def test_expert_ffn_token_rows_of_any_shape(world1, shape):
    """Token rows as a tensor of more than two dimensions (a parity of gathered rows, say): the pair lists count its rows."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertFfnPlan, ExpertWeights, RouteBuffers, RoutePlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    T, K, E, H, I = 60, 2, 4, 256, 128
    x, idx, w = _case(T, E, K, H, I, 23)
    heap = SymmetricHeap(world1, 1 << 20, DEV)
    route = RouteBuffers(T, K, E, DEV)
    weights = ExpertWeights(E, H, I, DEV, seed=9, std=0.05)
    RoutePlan(route, idx, w, torch.tensor([T], dtype=torch.int32, device=DEV), 0, heap.status).launch()
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV)
    got = []
    for rows in (x, x.view(*shape, H)):
        y = torch.full((route.max_pairs, H), float("nan"), dtype=torch.bfloat16, device=DEV)
        route.ffn_done.zero_()
        ExpertFfnPlan(weights, route, rows, act, y, heap.status).launch()
        torch.cuda.synchronize()
        heap.check_status()
        got.append(y)
    assert torch.equal(got[0], got[1]) and bool(got[0].count_nonzero() > got[0].numel() // 2)


@pytest.mark.parametrize("T,grid", [(4097, 1), (4097, 3), (3277, 1), (5000, 128), (12300, 3)])
def test_route_many_entries(world1, T, grid, E=24):
    """Routing whose entries are shared out over waiting blocks: all of a thread's kept until they are placed, more than that,
    and blocks without any; every entry of a local expert in its expert's rows once, the others marked, twice."""
    from moe_comms_benchmarking_b200.ops.experts import RouteBuffers, RoutePlan
    K, first = 5, 7
    _, idx, w = _case(T, E + 16, K, 8, 8, 41)
    route = RouteBuffers(T + 3, K, E, DEV)
    pad = lambda t: torch.cat([t, t[:3]]).contiguous()
    status = torch.zeros(8, dtype=torch.int32, device=DEV)
    ids, ws = pad(idx), pad(w)
    plan = RoutePlan(route, ids, ws, torch.tensor([T], dtype=torch.int32, device=DEV), expert_begin=first, status=status, grid=grid)
    local = (idx >= first) & (idx < first + E)
    counts = torch.bincount((idx[local] - first).flatten(), minlength=E)
    for rep in range(2):
        for t in (route.pair_token, route.pair_pos, route.pair_prob):
            t.fill_(-7)
        plan.launch()
        torch.cuda.synchronize()
        assert not status.any() and not route.sync.any() and not route.expert_count.any()
        assert torch.equal(route.expert_offset.long(), torch.cat([counts.new_zeros(1), counts.cumsum(0)]))
        pos = route.pair_pos[:T]
        assert bool((pos[~local] == -1).all()) and torch.equal(pos[local].sort().values.long(), torch.arange(int(counts.sum()), device=DEV))
        t, k = local.nonzero(as_tuple=True)
        at = pos[t, k].long()
        assert torch.equal(route.pair_token[at].long(), t) and torch.equal(route.pair_prob[at], w[t, k])
        assert torch.equal(torch.bucketize(at, route.expert_offset.long(), right=True) - 1, idx[t, k] - first)
        assert bool((route.pair_pos[T:] == -7).all()) and int(route.max_rows) == int(counts.max())


@pytest.mark.parametrize("T,grid", [(2457, 96), (2458, 96), (2458, 128), (3, 96), (3, 1),      # blocks of 512 threads
                                    (816, 2), (817, 2), (3276, 3), (3277, 3)])                 # two wider ones and not, three of 1024
def test_route_around_the_line(world1, T, grid):
    """The last size whose entries every block counts, the first that is shared out; the last buffers that fewer blocks take with 512 threads, the first
    with 1024."""
    test_route_many_entries(world1, T, grid)


@pytest.mark.parametrize("T,E", [(2458, 512), (2457, 513), (3276, 1024), (3277, 1024)])
def test_route_around_the_line_many_experts(world1, T, E):
    """From 513 local experts on every block counts more entries before they are shared out."""
    test_route_many_entries(world1, T, 96, E)


@pytest.mark.parametrize("E,K,H,I,T,layers,sets,grid", [
    (8, 2, 256, 128, 3, 2, 1, 148),          # two layers; fewer units than CTA pairs
    (8, 2, 256, 128, 90, 40, 20, 148),       # more weight sets than one launch takes, buffers used many times over
    (64, 6, 768, 512, 700, 5, 2, 148),       # counts of the later layers through the shared counters
    (6, 3, 512, 384, 1500, 4, 3, 148),       # several chunks per expert, one block per stage
    (40, 4, 256, 128, 200, 7, 2, 2),         # one pair of CTAs: more units than half a list holds
    (768, 22, 256, 128, 65, 3, 1, 30),       # as many experts as fit
    (769, 5, 256, 128, 40, 3, 1, 148),       # one more: layer by layer
    (4, 2, 2048, 256, 1600, 3, 2, 148),      # one buffer of expert outputs for all layers
])
def test_step_of_several_layers(world1, E, K, H, I, T, layers, sets, grid):
    """decode_step with its layers in one launch against the same layers launched one by one, bit for bit (both add the same
    products in the same order), and the rows that it gathers; smaller batches and none through the same plan; twice, so counters
    come back clean."""
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.ops.experts import MoeLayerPlan
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    cfg = Config(num_experts=E, topk=K, hidden=H, intermediate=I, ep_size=1, per_rank_cap=T + 3, probs="softmax")
    d = FusedExpertDispatcher(cfg, world1, num_layers=layers, weight_budget_gb=(sets * 6 * E * H * I + 1) / 2**30)
    d.build()
    plan = MoeLayerPlan(d.heap, d.agv_plan, d.route_plan, d.ffn, d.combine_plan, d.meta_plan, grid=grid)
    assert len(d.ffn) == sets and (plan._step is None) == (E > 768)
    for n in (T, T // 3 + 1, 0, T):
        x, idx, w = _case(max(n, 1), E, K, H, I, n + 31)
        d.setup_batch(x[:n], idx[:n], w[:n])
        d.metadata()
        for l in range(layers):
            plan.launch(l % sets)
        torch.cuda.synchronize()
        want = d.out.clone()
        for rep in range(2):
            for t in (d.out_buf, d.y, d.act, d.agv_h.tensor):
                t.fill_(float("nan"))
            plan.decode_step(layers)
            torch.cuda.synchronize()
            d.check_health()
            assert torch.equal(d.out, want), f"{n} tokens, rep {rep}"
            assert torch.equal(d.agv_h.tensor[:n], x[:n]) and torch.equal(d.agv_r.tensor[:n], idx[:n]) and torch.equal(d.agv_p.tensor[:n], w[:n])
    d.destroy()


@pytest.mark.parametrize("E,K,H,I,T,grid", [(24, 4, 1024, 512, 7000, 148), (24, 4, 1024, 512, 7000, 11)])
def test_step_with_down_units_at_a_distance(world1, E, K, H, I, T, grid):
    """A step of several layers whose down units follow at a distance of fewer experts than there are, against its layers."""
    rows = torch.bincount(_case(T, E, K, H, I, T + 31)[1].flatten(), minlength=E).tolist()
    active, distance = _down_distance(rows, H, I, grid)
    assert 2 <= distance < active
    test_step_of_several_layers(world1, E, K, H, I, T, 4, 2, grid)


def test_step_on_its_own_output_goes_layer_by_layer(world1):
    """Layers that read what the layer before has written keep their order: rows gathered from the combined output."""
    from moe_comms_benchmarking_b200.ops.dense import AllGatherVPlan, MetadataPlan
    from moe_comms_benchmarking_b200.ops.experts import (ExpertCombinePlan, ExpertFfnPlan, ExpertWeights, MoeLayerPlan,
                                                         RouteBuffers, RoutePlan)
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    T, E, K, H, I = 40, 6, 3, 256, 128
    x, idx, w = _case(T, E, K, H, I, 27)
    heap = SymmetricHeap(world1, 2 << 20, DEV)
    gx, gi, gw = heap.alloc("gx", [T, H], torch.bfloat16), heap.alloc("gi", [T, K], torch.int64), heap.alloc("gw", [T, K], torch.float32)
    n, meta = torch.tensor([T], dtype=torch.int32, device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
    route = RouteBuffers(T, K, E, DEV)
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(route.max_pairs, H, dtype=torch.bfloat16, device=DEV)
    rows = x.clone()
    partial = heap.alloc("partial", [2, T, H], torch.bfloat16)
    ffn = [ExpertFfnPlan(ExpertWeights(E, H, I, DEV, seed=s, std=0.05), route, gx.tensor, act, y, heap.status) for s in (3, 4)]
    plan = MoeLayerPlan(heap, AllGatherVPlan(heap, [gx, gi, gw], [rows, idx, w], n, meta, T),
                        RoutePlan(route, gi.tensor, gw.tensor, meta[0:1], expert_begin=0, status=heap.status), ffn,
                        ExpertCombinePlan(heap, y, route, partial, rows, n, meta, T), MetadataPlan(heap, n, meta, T))
    assert plan._step is None and plan.launches(3) == 4
    for out in (gx.tensor, torch.zeros_like(rows)):         # an output on the gathered rows, and one of its own
        p = MoeLayerPlan(heap, AllGatherVPlan(heap, [gx, gi, gw], [rows, idx, w], n, meta, T),
                         RoutePlan(route, gi.tensor, gw.tensor, meta[0:1], expert_begin=0, status=heap.status), ffn,
                         ExpertCombinePlan(heap, y, route, partial, out, n, meta, T), MetadataPlan(heap, n, meta, T))
        assert (p._step is None) == (out is gx.tensor)
    plan.meta.launch()
    for l in range(3):
        plan.launch(l % 2)
    torch.cuda.synchronize()
    want = rows.clone()
    rows.copy_(x)
    plan.decode_step(3)
    torch.cuda.synchronize()
    heap.check_status()
    assert torch.equal(rows, want) and not torch.equal(rows, x)


@pytest.mark.parametrize("rows,grid", [([40, 10], 148), ([140, 3], 148), ([300] * 12, 6)])
def test_expert_ffn_whose_wait_runs_out(world1, rows, grid):
    """Down units whose activations are never complete (the counters held back): the launch ends by itself and says so in the
    status words, with copies and MMAs landed; the next one is right."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertFfnPlan, ExpertWeights, RouteBuffers, RoutePlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import DeviceStatusError, SymmetricHeap
    E, T, H, I = len(rows), sum(rows), 512, 256
    heap = SymmetricHeap(world1, 1 << 20, DEV)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    idx = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(rows, device=DEV)).view(T, 1)
    route = RouteBuffers(T, 1, E, DEV)
    act, y = torch.zeros(T, I, dtype=torch.bfloat16, device=DEV), torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)
    rp = RoutePlan(route, idx, torch.ones(T, 1, device=DEV), torch.tensor([T], dtype=torch.int32, device=DEV), 0, heap.status)
    ffn = ExpertFfnPlan(ExpertWeights(E, H, I, DEV, seed=9, std=0.05), route, x, act, y, heap.status, grid=grid, timeout_s=0.05)
    out = []
    for held in (False, True, False):
        rp.launch()
        if held:
            route.ffn_done.fill_(-(1 << 20))
        ffn.launch()
        torch.cuda.synchronize()
        if held:
            with pytest.raises(DeviceStatusError) as e:
                heap.check_status()
            assert e.value.code == 5 and 11 <= e.value.words[1] <= 26
        else:
            heap.check_status()
            out.append(y[route.pair_pos.flatten().long()].clone())
    assert torch.equal(*out)


def _step_behind_a_larger_one(world1, small, layers=4, K=6):
    """A plan whose three sets of pair lists hold the positions of a step that fills one buffer of expert outputs, with a batch
    of `small` tokens loaded that alternates between two; its waits end after 50 ms.  (dispatcher, plan, output of the batch)"""
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.ops.experts import STEP_TWO_BUFFERS_BYTES, MoeLayerPlan
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    E, H, I, T = 8, 256, 128, 2100
    assert small * K * 2 * H <= STEP_TWO_BUFFERS_BYTES < T * K * 2 * H
    cfg = Config(num_experts=E, topk=K, hidden=H, intermediate=I, ep_size=1, per_rank_cap=T, probs="softmax")
    d = FusedExpertDispatcher(cfg, world1, num_layers=2, weight_budget_gb=1.0)
    d.build()
    for f in d.ffn:
        f.args.timeout_ns = 50_000_000
    plan = MoeLayerPlan(d.heap, d.agv_plan, d.route_plan, d.ffn, d.combine_plan, d.meta_plan)
    assert plan._step is not None
    for n in (T, small):
        d.setup_batch(*_case(n, E, K, H, I, n + 43))
        plan.decode_step(layers)
    torch.cuda.synchronize()
    d.check_health()
    return d, plan, d.out.clone()


def test_step_with_a_refused_count(world1):
    """More tokens than the capacity: reported, nothing is routed, and no position of an earlier, larger step is summed (the
    second buffer of expert outputs does not hold its rows).  The next step is right."""
    from moe_comms_benchmarking_b200.parallel.symm_heap import DeviceStatusError
    d, plan, want = _step_behind_a_larger_one(world1, 300)
    n = int(d.n_local)
    for bad in (d.cap + 1, 1 << 30):
        d.n_local.fill_(bad)
        for y in (d.y, plan._step_bufs[0][2]):
            y.fill_(float("nan"))
        plan.decode_step(4)
        torch.cuda.synchronize()
        with pytest.raises(DeviceStatusError) as e:
            d.check_health()
        assert e.value.code == 2 and not d.out_buf.isnan().any()
        d.n_local.fill_(n)
        plan.decode_step(4)
        torch.cuda.synchronize()
        d.check_health()
        assert torch.equal(d.out, want)
    d.destroy()


@pytest.mark.parametrize("word,small", [("routed", 300), ("counted", 300), ("counted", 2000), ("experts", 300), ("combined", 300)])
def test_step_whose_waits_run_out(world1, word, small):
    """Each counter that CTAs of a step wait for, held back so that it is never reached: the launch ends by itself, says so in
    the status words, and leaves its counters clean for the next one.  With 2000 tokens the first layer's counts are shared too."""
    from moe_comms_benchmarking_b200.parallel.symm_heap import DeviceStatusError
    d, plan, want = _step_behind_a_larger_one(world1, small)
    mem, b = plan._step_bufs[0][0], d.route
    sync = mem[mem.numel() - 160:]
    assert not sync.any()
    sync[{"routed": 0, "counted": 32, "experts": 64, "combined": 96}[word]] = -(1 << 20)
    plan.decode_step(4)
    torch.cuda.synchronize()
    with pytest.raises(DeviceStatusError) as e:
        d.check_health()
    assert e.value.code == 5 and 11 <= e.value.words[1] <= 26
    assert not sync.any()
    plan.decode_step(4)
    torch.cuda.synchronize()
    d.check_health()
    assert torch.equal(d.out, want)
    d.destroy()


def test_step_with_its_output_in_the_activations_goes_layer_by_layer(world1):
    """A combined output in the memory of the activations: a layer of its own is done with them before it writes the first row."""
    from moe_comms_benchmarking_b200.ops.dense import AllGatherVPlan, MetadataPlan
    from moe_comms_benchmarking_b200.ops.experts import (ExpertCombinePlan, ExpertFfnPlan, ExpertWeights, MoeLayerPlan,
                                                         RouteBuffers, RoutePlan)
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    T, E, K, H, I = 600, 6, 3, 256, 128
    x, idx, w = _case(T, E, K, H, I, 29)
    heap = SymmetricHeap(world1, 8 << 20, DEV)
    gx, gi, gw = heap.alloc("gx", [T, H], torch.bfloat16), heap.alloc("gi", [T, K], torch.int64), heap.alloc("gw", [T, K], torch.float32)
    n, meta = torch.tensor([T], dtype=torch.int32, device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
    route = RouteBuffers(T, K, E, DEV)
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(route.max_pairs, H, dtype=torch.bfloat16, device=DEV)
    partial = heap.alloc("partial", [2, T, H], torch.bfloat16)
    ffn = [ExpertFfnPlan(ExpertWeights(E, H, I, DEV, seed=s, std=0.05), route, gx.tensor, act, y, heap.status) for s in (3, 4)]
    got = []
    for out in (act.view(-1)[:T * H].view(T, H), torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)):
        plan = MoeLayerPlan(heap, AllGatherVPlan(heap, [gx, gi, gw], [x, idx, w], n, meta, T),
                            RoutePlan(route, gi.tensor, gw.tensor, meta[0:1], expert_begin=0, status=heap.status), ffn,
                            ExpertCombinePlan(heap, y, route, partial, out, n, meta, T), MetadataPlan(heap, n, meta, T))
        assert (plan._step is None) == (not got)
        plan.decode_step(5)
        torch.cuda.synchronize()
        heap.check_status()
        got.append(out.clone())
    assert torch.equal(*got) and bool(got[0].any())


@pytest.mark.parametrize("E,trace", [(768, False), (769, False), (8, True)])
def test_plan_that_goes_layer_by_layer_keeps_no_step_buffers(world1, E, trace):
    """Pair lists and buffers of further layers in flight are there only where layers share a launch."""
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    cfg = Config(num_experts=E, topk=4, hidden=256, intermediate=128, ep_size=1, per_rank_cap=8)
    d = FusedExpertDispatcher(cfg, world1, num_layers=1, weight_budget_gb=1.0, phase_trace=trace)
    d.build()
    joins = E <= 768 and not trace
    assert (d.layer_plan._step is not None) == joins and (d.layer_plan._step_bufs is not None) == joins
    assert d.layer_plan.launches(4) == (2 if joins else 5)
    d.destroy()


def test_validate_sees_the_kernels_of_a_step(world1, monkeypatch):
    """The self-check runs decode steps through every weight set, and finds a step that delivers nothing."""
    from moe_comms_benchmarking_b200.config import Config
    from moe_comms_benchmarking_b200.parallel.fused import FusedExpertDispatcher
    cfg = Config(num_experts=16, topk=4, hidden=256, intermediate=128, ep_size=1, per_rank_cap=48)
    d = FusedExpertDispatcher(cfg, world1, num_layers=3, weight_budget_gb=1.0)
    d.build()
    results = d.validate()
    assert all(ok for _, ok, _ in results), results
    steps = []
    with monkeypatch.context() as m:
        m.setattr(d.layer_plan, "decode_step", lambda layers, *a, **kw: steps.append(layers))
        broken = d.validate()
    assert steps and set(steps) == {len(d.weights) + 1}
    assert {name for name, ok, _ in broken if not ok} == {name for name, _, _ in results if "step" in name} != set()
    d.destroy()


@pytest.mark.parametrize("form", ["plain", "no_weights", "two_tensors", "order", "odd_ids", "own_weights"])
def test_step_forms_like_single_layers(world1, form):
    """What a joined step accepts against the same layers launched one by one, bit for bit: no routing weights, fewer tensors or another
    order of them in the all-gather, ids of no expert and an expert twice in a row.  Weights that the all-gather does not bring are
    the caller's own, and the layers go one by one."""
    from moe_comms_benchmarking_b200.ops.dense import AllGatherVPlan, MetadataPlan
    from moe_comms_benchmarking_b200.ops.experts import (ExpertCombinePlan, ExpertFfnPlan, ExpertWeights, MoeLayerPlan,
                                                         RouteBuffers, RoutePlan)
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    T, cap, E, K, H, I = 310, 333, 6, 5, 256, 128
    pad = lambda t: torch.cat([t, t[:cap - T]]).contiguous()
    x, idx, w = (pad(t) for t in _case(T, E, K, H, I, 61))
    if form == "odd_ids":
        idx[::3, 0], idx[1::3, 1], idx[2::3, 2], idx[::2, 3], idx[7] = -1, E, 1 << 40, idx[::2, 4], -5
    heap = SymmetricHeap(world1, 8 << 20, DEV)
    gx, gi, gw = heap.alloc("gx", [cap, H], torch.bfloat16), heap.alloc("gi", [cap, K], torch.int64), heap.alloc("gw", [cap, K], torch.float32)
    pairs = {"two_tensors": [(gx, x), (gi, idx)], "order": [(gw, w), (gi, idx), (gx, x)]}.get(form, [(gx, x), (gi, idx), (gw, w)])
    r_w = {"no_weights": None, "two_tensors": None, "own_weights": w.clone()}.get(form, gw.tensor)
    n, meta = torch.tensor([T], dtype=torch.int32, device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
    route = RouteBuffers(cap, K, E, DEV)
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(route.max_pairs, H, dtype=torch.bfloat16, device=DEV)
    out, partial = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV), heap.alloc("partial", [2, cap, H], torch.bfloat16)
    ffn = [ExpertFfnPlan(ExpertWeights(E, H, I, DEV, seed=s, std=0.05), route, gx.tensor, act, y, heap.status) for s in (3, 4, 5)]
    plan = MoeLayerPlan(heap, AllGatherVPlan(heap, [d for d, _ in pairs], [s for _, s in pairs], n, meta, cap),
                        RoutePlan(route, gi.tensor, r_w, meta[0:1], expert_begin=0, status=heap.status), ffn,
                        ExpertCombinePlan(heap, y, route, partial, out, n, meta, cap), MetadataPlan(heap, n, meta, cap))
    assert (plan._step is None) == (form == "own_weights")
    plan.meta.launch()
    for l in range(5):
        plan.launch(l % 3)
    torch.cuda.synchronize()
    want, rows = out.clone(), [d.tensor[:T].clone() for d, _ in pairs]
    for rep in range(2):
        for t in [out, y, act] + [d.tensor for d, _ in pairs]:
            t.zero_()
        plan.decode_step(5)
        torch.cuda.synchronize()
        heap.check_status()
        assert torch.equal(out, want) and bool(out[:T].any()) and all(torch.equal(d.tensor[:T], r) for (d, _), r in zip(pairs, rows))
