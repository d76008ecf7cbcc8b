"""The work a user of this framework has it do on one GPU, as cases that can be timed and compared.

Every case goes through public entry points: the decode engine (``MoEDecodeEngine``), a dispatcher's own
per-layer calls, or the launch plans of ``ops/experts.py``.  A case is a dict of plain values:

``path``      moe      a decode step with real SwiGLU experts through the engine (one rank that holds every expert)
              experts  routing, expert FFN and combine through their plans, with the share of the experts that one
                       rank of an ``ep``-rank job holds
              dense    a decode step of the dense dispatcher (all-gather / reduce-scatter) through the engine
              a2a      a decode step of the all-to-all dispatcher through the engine
              layer    one layer of a dispatcher called operation by operation, as a program with experts of its own does
              host     an end-to-end step from pinned host tensors to a pinned host result
``impl``      the dispatcher of a ``layer`` or ``host`` case (dense, a2a)
``experts``, ``topk``, ``hidden``, ``intermediate``, ``tokens``, ``layers``, ``ep``, ``fp8``, ``routing``
"""
from __future__ import annotations

import math

import torch

from moe_comms_benchmarking_b200.config import Config
from moe_comms_benchmarking_b200.models.engine import MoEDecodeEngine
from moe_comms_benchmarking_b200.ops.experts import (ExpertCombinePlan, ExpertFfnPlan, ExpertWeights, RouteBuffers,
                                                     RoutePlan)
from moe_comms_benchmarking_b200.parallel.a2a import A2ADispatcher
from moe_comms_benchmarking_b200.parallel.dense import DenseDispatcher
from moe_comms_benchmarking_b200.parallel.dist import init_distributed
from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
from moe_comms_benchmarking_b200.utils.inputs import expert_log_popularity, make_inputs

DEV = "cuda:0"
SET_BYTES_MAX = 3.3e9           # weights of one layer: 512 experts x 3 x 1024^2 bf16 is the largest the repository runs
MOE_FLOPS_MAX = 8 * 6.0 * 4096 * 22 * 1024 * 1024


def _case(name=None, path="moe", experts=512, topk=22, hidden=1024, intermediate=1024, tokens=1, layers=1, ep=1, fp8=False,
          routing="uniform", impl="dense"):
    c = dict(path=path, experts=experts, topk=topk, hidden=hidden, intermediate=intermediate, tokens=tokens, layers=layers,
             ep=ep, fp8=fp8, routing=routing, impl=impl)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # Decode of a single sequence with real experts, all 88 layers: 22 experts' weights per layer, latency counts.
        _case("moe_one_token", tokens=1, layers=88),
        # A small ragged decode batch: most experts have tokens, two or three each; a stream of weights.
        _case("moe_b37", tokens=37, layers=8),
        # The largest batch the repository's configurations run with real experts.
        _case("moe_b4096", tokens=4096, layers=8),
        # The wide shape (hidden 7168, intermediate 2048) with an eighth of its 256 experts: long reductions, few experts.
        _case("moe_wide_b190", experts=32, topk=8, hidden=7168, intermediate=2048, tokens=190, layers=4),
        # What one rank of an 8-rank job does per layer: a small decode batch, ...
        _case("experts_ep8_t64", path="experts", tokens=64, ep=8),
        # ... the largest decode batch, ...
        _case("experts_ep8_t4096", path="experts", tokens=4096, ep=8),
        # ... and a prefill-size batch with skewed expert popularity and an odd token count.
        _case("experts_ep8_t8191_zipf", path="experts", tokens=8191, ep=8, routing="zipf"),
        # The headline benchmark's step at its smallest and its largest batch.
        _case("dense_one_token", path="dense", tokens=1, layers=88),
        _case("dense_b8192", path="dense", tokens=8192, layers=88),
        # The wide shape's step on the all-to-all path with e4m3 dispatch, at an ordinary ragged batch.
        _case("a2a_fp8_wide_b333", path="a2a", experts=256, topk=8, hidden=7168, intermediate=2048, tokens=333, layers=58,
              fp8=True),
        # One layer called operation by operation, at an ordinary decode batch.
        _case("layer_dense_b100", path="layer", tokens=100),
        # An end-to-end step from pinned host memory, at an ordinary batch.
        _case("host_dense_b512", path="host", tokens=512, layers=88),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _moe_shape(rng, ep):
    """A MoE shape whose weights of one rank and layer stay within SET_BYTES_MAX."""
    while True:
        if rng.random() < 0.4:
            experts, topk, hidden, inter = 512, 22, 1024, 1024
        else:
            hidden = 256 * rng.choice([2, 4, 6, 8, 12, 16, 20, 28])
            inter = 128 * rng.choice([2, 4, 6, 8, 11, 12, 16])
            experts = 8 * _log_int(rng, ep, 64)
            topk = rng.randint(1, min(22, experts))
        if experts % ep == 0 and 6.0 * experts // ep * hidden * inter <= SET_BYTES_MAX:
            return experts, topk, hidden, inter


def draw(rng):
    path = rng.choice(["moe"] * 4 + ["experts"] * 3 + ["dense"] * 2 + ["a2a"] * 2 + ["layer", "host"])
    routing = "zipf" if rng.random() < 0.25 else "uniform"
    if path in ("moe", "experts"):
        ep = 1 if path == "moe" else rng.choice([2, 4, 8])
        experts, topk, hidden, inter = _moe_shape(rng, ep)
        layers = rng.choice([4, 8]) if path == "moe" else 1
        per_token = 6.0 * layers * topk / ep * hidden * inter
        most = min(4096 if path == "moe" else 8192, int(MOE_FLOPS_MAX / per_token))
        least = 1 if path == "moe" else 16 * ep // topk + 1      # a rank of a job sees some of its experts chosen
        return _case(path=path, experts=experts, topk=topk, hidden=hidden, intermediate=inter,
                     tokens=_log_int(rng, least, max(least, most)), layers=layers, ep=ep, routing=routing)
    experts, topk, hidden, layers = rng.choice([(512, 22, 1024, 88), (256, 8, 7168, 58), (128, 8, 2048, 48), (64, 6, 768, 26)])
    fp8 = path in ("dense", "a2a") and rng.random() < 0.4
    tokens = _log_int(rng, 1, 2048 if hidden > 2048 else 8192)
    return _case(path=path, experts=experts, topk=topk, hidden=hidden, tokens=tokens, layers=1 if path == "layer" else layers,
                 fp8=fp8, routing=routing, impl=rng.choice(["dense", "a2a"]))


def _impl(case):
    return case["impl"] if case["path"] in ("layer", "host") else case["path"]


def _config(case, seed):
    # an engine is built once for a capacity and then serves every batch up to it
    return Config(num_experts=case["experts"], topk=case["topk"], hidden=case["hidden"], intermediate=case["intermediate"],
                  ep_size=1, per_rank_cap=(case["tokens"] + 63) // 64 * 64, seed=int(seed) % (1 << 40) + 1, routing=case["routing"],
                  probs="sigmoid" if case["topk"] <= 8 else "softmax")


def _moe(case, seed, cfg, group):
    set_bytes = 6 * case["experts"] * case["hidden"] * case["intermediate"]
    eng = MoEDecodeEngine(cfg, group, impl="fused", num_layers=case["layers"], weight_budget_gb=(2 * set_bytes + 1) / 2**30,
                          weight_seed=int(seed) % 9973 + 1)
    eng.build()
    return {"engine": eng, "inputs": make_inputs(cfg, case["tokens"], DEV)}


def _experts(case, seed, cfg):
    T, K, H, I = case["tokens"], case["topk"], case["hidden"], case["intermediate"]
    E = case["experts"] // case["ep"]
    heap = SymmetricHeap(None, T * H * 2 + (1 << 20), DEV)
    partial = heap.alloc("partial", [T, H], torch.bfloat16)
    weights = ExpertWeights(E, H, I, DEV, seed=int(seed) % 9973 + 1)
    route = RouteBuffers(T, K, E, DEV)
    x, idx, w = make_inputs(cfg, T, DEV)
    act = torch.zeros(max(route.max_pairs, 1), I, dtype=torch.bfloat16, device=DEV)
    y = torch.zeros(max(route.max_pairs, 1), H, dtype=torch.bfloat16, device=DEV)
    out = torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)
    ntok = torch.tensor([T], dtype=torch.int32, device=DEV)
    meta = torch.tensor([T, 0, T, 1], dtype=torch.int32, device=DEV)
    begin = E * (int(seed) % case["ep"])            # any rank of the job
    status = heap.status
    return {"plans": (RoutePlan(route, idx, w, ntok, expert_begin=begin, status=status),
                      ExpertFfnPlan(weights, route, x, act, y, status),
                      ExpertCombinePlan(heap, y, route, partial, out, ntok, meta, T)), "out": out}


def prepare(case, seed):
    group, *_ = init_distributed()
    torch.manual_seed(int(seed))
    cfg = _config(case, seed)
    T, H, path = case["tokens"], case["hidden"], case["path"]
    if path == "experts":
        return dict(_experts(case, seed, cfg), path=path)
    if path == "moe":
        s = _moe(case, seed, cfg, group)
    else:
        impl = _impl(case)
        kw = {"fp8_dispatch": True} if case["fp8"] else {}
        s = {"inputs": make_inputs(cfg, T, DEV), "impl": impl, "tokens": T}
        if path == "layer":
            s["dispatcher"] = {"dense": DenseDispatcher, "a2a": A2ADispatcher}[impl](cfg, group)
            s["dispatcher"].build()
        else:
            s["engine"] = MoEDecodeEngine(cfg, group, impl=impl, num_layers=case["layers"], **kw)
            s["engine"].build()
            s["dispatcher"] = s["engine"].dispatcher
        # The expert outputs that the combine reduces (the identity expert of the bf16 all-to-all path has none of its own).
        d = s["dispatcher"]
        experts_out = torch.randn(T, H, device=DEV).to(torch.bfloat16)
        if impl == "dense":
            d.rsv.tensor[:T] = experts_out
        elif case["fp8"]:
            d.step_bufs.y.tensor[:, 0, :T] = experts_out
    if "engine" in s:
        s["engine"].load_batch(*s["inputs"])
        s["engine"].capture()
    if path == "host":
        s["inputs"] = tuple(t.cpu().pin_memory() for t in s["inputs"])
    return dict(s, path=path)


def _gathered(s):
    """What the dispatch of a step delivers: rows, routing and weights as received (both layer parities)."""
    d, n = s["dispatcher"], s["tokens"]
    if s["impl"] == "dense":
        got = [t.tensor[:, :n] for t in (d.agv2_h, d.agv2_r, d.agv2_p)]
        return got + ([d.agv2_s.tensor[:, :n]] if d.fp8 else [])
    b = d.step_bufs
    got = [b.recv_x.tensor[:, 0, :n]] + ([b.recv_scale.tensor[:, 0, :n]] if d.fp8 else [])
    for par in (0, 1):
        got += b.meta_fields(par, 0, n)[1:]         # token, expert ids, weights (the stamp counts layers)
    return got


def run(state):
    path = state["path"]
    if path == "experts":
        for plan in state["plans"]:
            plan.launch()
        return state["out"]
    if path == "host":
        return state["engine"].step_host(*state["inputs"])
    if path == "layer":
        d, n = state["dispatcher"], state["tokens"]
        d.setup_batch(*state["inputs"])
        if state["impl"] == "dense":
            d.metadata()
        d.dispatch()
        d.combine()
        if state["impl"] == "dense":
            return [d.out, d.agv_h.tensor[:n], d.agv_r.tensor[:n], d.agv_p.tensor[:n]]
        b = d.bufs      # slots of one source are handed out in any order: the combined rows are in token order
        return [d.out, b.recv_count.tensor[:1]]
    eng = state["engine"]
    eng.load_batch(*state["inputs"])
    eng.run()
    if path == "moe":
        return eng.dispatcher.out
    return [eng.dispatcher.out] + _gathered(state)


def _active_experts(case):
    """Expected number of this rank's experts that have a token."""
    E, K, T = case["experts"], case["topk"], case["tokens"]
    if case["routing"] == "uniform":
        return E / case["ep"] * (1.0 - (1.0 - K / E) ** T)
    logp = expert_log_popularity(Config(num_experts=E, topk=K, routing="zipf"), "cpu")
    hit = (logp.exp().double() * K).clamp(max=1.0)
    return float((1.0 - (1.0 - hit) ** T).sum()) / case["ep"]


def work(case):
    T, K, H, I, L = case["tokens"], case["topk"], case["hidden"], case["intermediate"], case["layers"]
    row, routing = 2 * H, 12 * K            # bf16 hidden row; int64 expert ids and fp32 weights
    if case["path"] in ("moe", "experts"):
        # weights of the experts in use, tokens and routing in, combined rows out
        return {"bytes": L * (_active_experts(case) * 6.0 * H * I + T * (row + routing) + T * row),
                "flops": L * 6.0 * T * K / case["ep"] * H * I}
    sent = H + H // 128 * 4 if case["fp8"] else row
    meta = routing if _impl(case) == "dense" else 8 * K
    # a layer reads rows and routing and delivers them, then reads the expert outputs and writes the combined rows
    layer = T * (row + routing + sent + meta + row + row)
    return {"bytes": float(L * layer + (T * (2 * row + routing) if case["path"] == "host" else 0)), "flops": 0.0}


def tolerance(case):
    # Real experts: bf16 activations and expert outputs, fp32 accumulation.  Everything else moves bytes, and the sum
    # over one rank's rows is the row.
    return {"rel": 1e-2} if case["path"] in ("moe", "experts") else "exact"
