"""All-to-all-V dispatcher on our own peer-load/store kernels.

Fills the slot of the reference's ``DeepEPBencher`` (bench_deepep.py:26-168), whose
``deep_ep`` dependency cannot be built offline: one copy of a token per distinct destination
rank, count exchange inside dispatch, device-resident (no CPU sync, graph-capturable),
rank-layout combine that returns ``m * x`` for the identity expert, a CTA-count knob
(``set_num_sms``), plus 1x128 block-scaled e4m3 dispatch.
"""
from __future__ import annotations

import torch
import torch.distributed as dist

from ..config import Config
from ..ops import _ext
from ..ops.a2a import (A2ABuffers, A2ACombinePlan, A2ADispatchPlan, A2AStepBuffers, A2AStepPlan, a2a_decode_step,
                       dequant_e4m3_1x128)
from ..ops.dense import DEFAULT_GRID, DEFAULT_THREADS
from .base import Dispatcher
from .symm_heap import SymmetricHeap, required_bytes


def resolve_a2a_ll_rows(cfg: Config, ll_rows: int) -> int:
    """Largest step (tokens over all ranks) the packet mode of the persistent kernel serves; 0 = off, -1 = the
    measured default of 1024.  On 8 GPUs a step takes 0.61 / 0.66 / 0.85 / 1.20 / 2.48 ms in packets at 1 / 256 /
    512 / 1024 / 2048 tokens against 1.31 / 1.73 / 1.77 / 1.83 / 2.3 ms on the barrier path (0.42-0.47 against
    1.06-1.23 ms up to 256 tokens on 2 GPUs); packets double the bytes on the wire, so large steps stay on the
    barrier path."""
    if cfg.ep_size == 1:
        return 0
    if ll_rows < 0:
        ll_rows = 1024
    return min(int(ll_rows), max(cfg.global_cap, 1))


class A2ADispatcher(Dispatcher):
    name = "a2a"

    def __init__(self, cfg: Config, group, heap: SymmetricHeap | None = None, num_sms: int = DEFAULT_GRID,
                 threads: int = DEFAULT_THREADS, pdl: bool = True, fp8_dispatch: bool = False,
                 transport: str = "auto", persistent: bool = True, ll_rows: int = -1, device=None):
        super().__init__(cfg, group, device)
        self.heap = heap
        self._own_heap = heap is None
        self.num_sms, self.threads, self.pdl = int(num_sms), int(threads), bool(pdl)
        self.fp8 = bool(fp8_dispatch)
        self.transport = transport
        if self.fp8:
            self.name = "a2a-fp8"
        # persistent: a whole decode step is ONE kernel (token-indexed slots, one barrier per layer);
        # otherwise 2 x layers launches of the dispatch / combine kernels with compacted slots and counts.
        self.persistent = bool(persistent)
        # packet mode of the persistent kernel serves steps of at most ll_rows tokens over all ranks
        self.ll_rows = resolve_a2a_ll_rows(cfg, ll_rows) if self.persistent else 0
        self.kernel_launches_per_step = lambda nl: 1 if self.persistent else 2 * nl
        self._step_plans = {}

    @staticmethod
    def heap_specs(cfg: Config, fp8: bool = False, ll_rows: int = -1):
        cap = max(cfg.per_rank_cap, 1)
        return (A2ABuffers.specs(cfg.ep_size, cap, cfg.hidden, cfg.topk, fp8)
                + A2AStepBuffers.specs(cfg.ep_size, cap, cfg.hidden, cfg.topk, fp8, resolve_a2a_ll_rows(cfg, ll_rows)))

    def build(self):
        cfg, dev = self.cfg, self.device
        cap, H, K = max(cfg.per_rank_cap, 1), cfg.hidden, cfg.topk
        self.cap = cap
        if self.heap is None:
            self.heap = SymmetricHeap(self.group, required_bytes(self.heap_specs(cfg, self.fp8, self.ll_rows)), dev,
                                      transport=self.transport)
        self.bufs = A2ABuffers(self.heap, cap, H, K, self.fp8, prefix="a2a8" if self.fp8 else "a2a")
        self.step_bufs = A2AStepBuffers(self.heap, cap, H, K, self.fp8, prefix="a2as8" if self.fp8 else "a2as",
                                        ll_rows=self.ll_rows)
        if self.step_bufs.credits is not None:        # the per-block credit counts restart with the epochs
            self.heap.register_reset_hook(self.step_bufs.credits.tensor.zero_)
        self.step_metadata = torch.zeros(8, dtype=torch.int32, device=dev)
        self.step_state = torch.zeros(_ext.STEP_STATE_WORDS, dtype=torch.int32, device=dev)
        self.heap.register_reset_hook(self.step_state.zero_)
        self.in_hidden = torch.zeros(cap, H, dtype=torch.bfloat16, device=dev)
        self.in_routing = torch.zeros(cap, K, dtype=torch.int64, device=dev)
        self.in_probs = torch.zeros(cap, K, dtype=torch.float32, device=dev)
        self.out_buf = torch.zeros(cap, H, dtype=torch.bfloat16, device=dev)
        self.n_local = torch.zeros(1, dtype=torch.int32, device=dev)
        self.local_tokens = 0
        if self.fp8:
            self.bufs.y.tensor.normal_()    # timed combine reduces valid data
            self.step_bufs.y.tensor.normal_()
        self._make_plans()
        torch.cuda.synchronize()
        dist.barrier(self.group)
        self._built = True

    def _make_plans(self):
        self.dispatch_plan = A2ADispatchPlan(self.heap, self.bufs, self.in_hidden, self.in_routing, self.in_probs,
                                             self.n_local, self.cfg.num_experts, grid=self.num_sms,
                                             threads=self.threads)
        self.combine_plan = A2ACombinePlan(self.heap, self.bufs, self.out_buf, self.n_local, grid=self.num_sms,
                                           threads=self.threads)
        self._step_plans = {}

    def _step_plan(self, num_layers: int) -> A2AStepPlan:
        plan = self._step_plans.get(num_layers)
        if plan is None:
            plan = A2AStepPlan(self.heap, self.step_bufs, self.in_hidden, self.in_routing, self.in_probs, self.out_buf,
                               self.n_local, self.step_metadata, self.cfg.num_experts, num_layers, grid=self.num_sms,
                               threads=self.threads, state=self.step_state)
            self._step_plans[num_layers] = plan
        return plan

    def set_num_sms(self, num_sms: int):
        self.num_sms = int(num_sms)
        if self._built:
            self._make_plans()

    def setup_batch(self, hidden, topk_idx, topk_weights):
        self._load_rows(hidden, topk_idx, topk_weights)

    @property
    def out(self):
        return self.out_buf[:self.local_tokens]

    def dispatch(self):
        self.dispatch_plan.launch(self.pdl)

    def combine(self):
        self.combine_plan.launch(self.pdl)

    def decode_step(self, num_layers: int):
        if self.persistent:
            self._step_plan(num_layers).launch(self.pdl)
        else:
            a2a_decode_step(self.heap, self.dispatch_plan, self.combine_plan, num_layers, self.pdl)

    def check_health(self):
        self.heap.check_status()

    # -- received data accessors (valid after dispatch) -------------------------------------------------
    def recv_counts(self) -> torch.Tensor:
        return self.bufs.recv_count.tensor[:self.cfg.ep_size]

    def received_rows(self, src: int) -> torch.Tensor:
        """bf16 rows received from ``src`` (dequantised when the dispatch was e4m3)."""
        c = int(self.recv_counts()[src].item())
        if self.fp8:
            return dequant_e4m3_1x128(self.bufs.recv_x.tensor[src, :c], self.bufs.recv_scale.tensor[src, :c])
        return self.bufs.recv_x.tensor[src, :c]

    def _sync_all(self):
        torch.cuda.synchronize()
        dist.barrier(self.group)

    def functional_roundtrip(self, hidden, topk_idx):
        """dispatch -> identity expert -> combine = m * x (bench_deepep.py:104-147)."""
        n = hidden.shape[0]
        self.setup_batch(hidden, topk_idx, torch.ones(n, self.cfg.topk, device=self.device))
        self.dispatch()
        self._sync_all()
        if self.fp8:
            for s in range(self.cfg.ep_size):
                rows = self.received_rows(s)
                self.bufs.y.tensor[s, :rows.shape[0]] = rows
        self._sync_all()
        self.combine()
        self._sync_all()
        return self.out

    def _validate_step_kernel(self, B: int):
        """The persistent step kernel on tokens every rank can regenerate: what each source sent here
        (rows, packed routing, stamps) and the combined output m * x."""
        w, rank, dev = self.cfg.ep_size, self.cfg.rank, self.device
        H, K, E, sb = self.cfg.hidden, self.cfg.topk, self.cfg.num_experts, self.step_bufs
        epr = E // w
        counts = self._validation_counts(B)
        offs = [sum(counts[:r]) for r in range(w)]
        gen = torch.Generator(device=dev).manual_seed(880801 + B)          # same on all ranks
        full_x = torch.randn(B, H, generator=gen, device=dev).to(torch.bfloat16)
        full_i = torch.stack([torch.randperm(E, generator=gen, device=dev)[:K] for _ in range(B)])
        full_w = torch.rand(B, K, generator=gen, device=dev)
        n, off = counts[rank], offs[rank]
        self.setup_batch(full_x[off:off + n], full_i[off:off + n], full_w[off:off + n])
        ok, why = True, []
        for nl in (3, 2):
            sb.recv_meta.tensor.zero_()
            self._sync_all()
            self.decode_step(nl)
            self._sync_all()
            par, stamp = int(self.step_metadata[5]), int(self.step_metadata[7])
            for s in range(w):
                c = counts[s]
                if not c:
                    continue
                st, tok, ids, wts = sb.meta_fields(par, s, c)
                here = ((full_i[offs[s]:offs[s] + c] // epr) == rank).any(dim=1)
                if not torch.equal(st == stamp, here):
                    ok = False; why.append(f"stamps of source {s}")
                    continue
                sel = here.nonzero().flatten()
                if sel.numel() == 0:
                    continue
                good = (torch.equal(tok[sel].long(), sel) and torch.equal(ids[sel].long(), full_i[offs[s] + sel])
                        and torch.equal(wts[sel], full_w[offs[s] + sel]))
                want = full_x[offs[s] + sel]
                if self.fp8:
                    got = dequant_e4m3_1x128(sb.recv_x.tensor[par, s][sel], sb.recv_scale.tensor[par, s][sel]).float()
                    good = good and bool(((got - want.float()).abs() <= 0.07 * want.float().abs() + 0.02).all())
                else:
                    good = good and torch.equal(sb.recv_x.tensor[par, s][sel], want)
                if not good:
                    ok = False; why.append(f"rows of source {s}")
            if self.fp8:
                # identity expert on the host: expert outputs = the dequantised received rows; one more step
                for s in range(w):
                    if counts[s]:
                        sb.y.tensor[:, s, :counts[s]] = dequant_e4m3_1x128(sb.recv_x.tensor[par, s, :counts[s]],
                                                                          sb.recv_scale.tensor[par, s, :counts[s]])
                self._sync_all()
                self.decode_step(2)
                self._sync_all()
            if n:
                m = torch.tensor([torch.unique(full_i[off + t] // epr).numel() for t in range(n)], device=dev,
                                 dtype=torch.float32).view(n, 1)
                ref = m * full_x[off:off + n].float()
                err = float((self.out.float() - ref).abs().max()) / (float(ref.abs().max()) + 1e-6)
                if err >= (0.08 if self.fp8 else 0.02):
                    ok = False; why.append(f"combine off by {100 * err:.2f}%")
        return ok, ("received rows, packed routing and stamps match every source; combine == m*x (steps of 3 and 2 layers)"
                    if ok else "; ".join(why))

    def validate(self):
        w, rank, dev = self.cfg.ep_size, self.cfg.rank, self.device
        H, K, E = self.cfg.hidden, self.cfg.topk, self.cfg.num_experts
        epr = E // w
        tol = 0.08 if self.fp8 else 0.05
        results = []
        if self.persistent:
            # small steps run the packet mode (when enabled), the last one the barrier path
            for B in (w * 2, 1, self.ll_rows + w):
                if max(self._validation_counts(B)) <= self.cap:
                    ok, detail = self._validate_step_kernel(B)
                    mode = "packets" if int(self.step_metadata[6]) else "barrier"
                    results.append((f"{self.name} step kernel       B={B:<4d}", bool(ok), f"[{mode}] {detail}"))
        for B in (w * 2, 1):
            counts = self._validation_counts(B)
            if max(counts) > self.cap:
                results.append((f"{self.name} dispatch->combine B={B:<4d}", True, "skipped: batch exceeds capacity"))
                continue
            n = counts[rank]
            gen = torch.Generator(device=dev).manual_seed(770701 + B + rank * 211)
            x = torch.randn(n, H, generator=gen, device=dev).to(torch.bfloat16)
            idx = (torch.stack([torch.randperm(E, generator=gen, device=dev)[:K] for _ in range(n)])
                   if n else torch.empty(0, K, dtype=torch.int64, device=dev))
            got = self.functional_roundtrip(x, idx).float()
            if n:
                m = torch.tensor([torch.unique(idx[t] // epr).numel() for t in range(n)], device=dev,
                                 dtype=torch.float32).view(n, 1)
                ref = m * x.float()
                scale = float(ref.abs().max()) + 1e-6
                err = float((got - ref).abs().max())
                ok = err / scale < tol
                detail = f"n={n} max|got-m*x|={err:.4f} ({100 * err / scale:.2f}% of {scale:.2f})"
            else:
                ok, detail = True, "n=0 (idle rank still takes part in dispatch and combine)"
            results.append((f"{self.name} dispatch->combine B={B:<4d}", bool(ok), detail))
        try:
            self.check_health()
        except Exception as e:
            results.append((f"{self.name} device status", False, str(e)))
        return results

    def destroy(self):
        if self._own_heap and self.heap is not None:
            self.heap.destroy()
        self.heap = None
        self._built = False
