"""Dense dispatcher on our own sm_100a kernels: AllGather-V -> local experts -> ReduceScatter-V.

Capabilities of the reference's ``NVLSBencher`` (bench_nvls.py:37-223): symmetric buffers for
hidden / routing / probabilities / combine input, once-per-step token-count metadata, the
per-layer dispatch and combine, ``validate`` with its bit-exact gather check and its
``world * rsv`` reduce check, and ``functional_roundtrip`` (masked identity expert, m * x).

Differences: all inputs live in capacity-sized persistent buffers and the local token count
is a device scalar, so ONE captured graph serves every batch up to the capacity (the
reference bakes ``local_tokens`` into the launch and re-captures per batch,
variable_collectives.py:749,785); a whole decode step (count exchange + every layer) is ONE
persistent kernel launch with one cross-GPU barrier per layer (``persistent=True``, the default;
``persistent=False`` issues the 1 + 2 * layers separate kernels from one native call, with
programmatic dependent launch between them); and the transport is NVSwitch multicast when
available, plain peer access otherwise (EP=1 included).
"""
from __future__ import annotations

import torch
import torch.distributed as dist

from ..config import Config
from ..ops import _ext
from ..ops.dense import (AllGatherVPlan, DenseStepPlan, MetadataPlan, ReduceScatterVPlan, dense_decode_step,
                         DEFAULT_GRID, DEFAULT_THREADS, agv_ll_stage_bytes, rsv_ll_stage_bytes, step_credit_bytes)
from .base import Dispatcher
from .symm_heap import HeapTensor, SymmetricHeap, required_bytes


def resolve_ll_rows(cfg: Config, ll_rows: int) -> int:
    """Row limit of the packet mode.  ``-1`` picks 512 rows: inside the persistent step kernel packets
    beat barrier + multicast up to about that many rows in total (measured on B200: 0.57 against 1.00 ms per
    88-layer step at 512 rows and EP=2; packets double the bytes, so the barrier mode wins from ~1000 rows)."""
    if cfg.ep_size <= 1:
        return 0
    if ll_rows < 0:
        ll_rows = 512
    return min(int(ll_rows), max(cfg.global_cap, 1))


class DenseDispatcher(Dispatcher):
    name = "dense"

    def __init__(self, cfg: Config, group, heap: SymmetricHeap | None = None, num_sms: int = DEFAULT_GRID,
                 threads: int = DEFAULT_THREADS, pdl: bool = True, transport: str = "auto",
                 combine_dtype=torch.bfloat16, ll_rows: int = -1, persistent: bool = True, groups: int = 1,
                 group_min_bytes: int = 256 << 10, fp8_dispatch: bool = False, device=None):
        super().__init__(cfg, group, device)
        self.heap = heap
        self._own_heap = heap is None
        self.persistent = bool(persistent)
        # 1 x 128 block-scaled e4m3 dispatch of the hidden rows (quantised inside the step kernel's
        # push, scales gathered as a fourth tensor); the combine stays bf16.
        self.fp8 = bool(fp8_dispatch)
        if self.fp8:
            if not self.persistent:
                raise ValueError("fp8 dispatch is part of the persistent step kernel")
            if cfg.hidden % 256:
                raise ValueError("fp8 dispatch needs a hidden size that is a multiple of 256")
            self.name = "dense-fp8"
        self.num_sms = self._grid_for(cfg, num_sms)
        self.threads = int(threads)
        self.pdl = bool(pdl)
        self.transport = transport
        self.combine_dtype = combine_dtype
        # Low-latency packet mode serves steps that hold at most ll_rows tokens over all ranks.
        self.ll_rows = resolve_ll_rows(cfg, ll_rows)
        self.persistent = bool(persistent)
        # Pipeline groups of the persistent kernel wait on one another: they need one block per SM.
        self.groups = int(groups) if cfg.ep_size > 1 else 1
        self.group_min_bytes = int(group_min_bytes)
        self.kernel_launches_per_step = lambda nl: 1 if self.persistent else 1 + 2 * nl
        self._step_plans = {}

    @staticmethod
    def _ll_bytes(cfg: Config, ll_rows: int, fp8: bool = False):
        H, K = cfg.hidden, cfg.topk
        ll_rows = resolve_ll_rows(cfg, ll_rows)
        rows = [H, K * 8, K * 4, H // 128 * 4] if fp8 else [H * 2, K * 8, K * 4]
        return (agv_ll_stage_bytes(ll_rows, rows),
                rsv_ll_stage_bytes(cfg.ep_size, ll_rows, max(cfg.per_rank_cap, 1), H * 2))

    @staticmethod
    def heap_specs(cfg: Config, combine_dtype=torch.bfloat16, ll_rows: int = -1, fp8: bool = False):
        g, H, K = max(cfg.global_cap, 1), cfg.hidden, cfg.topk
        a, r = DenseDispatcher._ll_bytes(cfg, ll_rows, fp8)
        hidden = [([2, g, H], torch.uint8), ([2, g, H // 128], torch.float32)] if fp8 else [([2, g, H], torch.bfloat16)]
        return hidden + [([2, g, K], torch.int64), ([2, g, K], torch.float32),
                         ([g, H], combine_dtype), ([max(a, 16)], torch.uint8), ([max(r, 16)], torch.uint8),
                         ([step_credit_bytes()], torch.uint8)]

    def build(self):
        cfg, dev = self.cfg, self.device
        cap, g, H, K = max(cfg.per_rank_cap, 1), max(cfg.global_cap, 1), cfg.hidden, cfg.topk
        self.cap = cap
        if self.heap is None:
            self.heap = SymmetricHeap(self.group,
                                      required_bytes(self.heap_specs(cfg, self.combine_dtype, self.ll_rows, self.fp8)), dev,
                                      transport=self.transport)
        h = self.heap
        # Gathered rows, double buffered by layer parity for the persistent step kernel; the
        # stand-alone dispatch and the validation use parity 0.
        self.agv2_h = h.alloc("ep_agv_h", [2, g, H], torch.uint8 if self.fp8 else torch.bfloat16)
        self.agv2_s = h.alloc("ep_agv_s", [2, g, H // 128], torch.float32) if self.fp8 else None
        self.agv2_r = h.alloc("ep_agv_r", [2, g, K], torch.int64)
        self.agv2_p = h.alloc("ep_agv_p", [2, g, K], torch.float32)
        self.agv_h, self.agv_r, self.agv_p = (HeapTensor(t.tensor[0], t.offset, t.nbytes // 2)
                                              for t in (self.agv2_h, self.agv2_r, self.agv2_p))
        self.rsv = h.alloc("ep_rsv", [g, H], self.combine_dtype)
        a_bytes, r_bytes = self._ll_bytes(cfg, self.ll_rows, self.fp8)
        self.ll_agv = h.alloc("ep_ll_agv", [max(a_bytes, 16)], torch.uint8)
        self.ll_rsv = h.alloc("ep_ll_rsv", [max(r_bytes, 16)], torch.uint8)
        self.step_credits = h.alloc("ep_step_credit", [step_credit_bytes()], torch.uint8)
        # Persistent local buffers (stable addresses for graph replay).
        self.in_hidden = torch.zeros(cap, H, dtype=torch.bfloat16, device=dev)
        self.in_routing = torch.zeros(cap, K, dtype=torch.int64, device=dev)
        self.in_probs = torch.zeros(cap, K, dtype=torch.float32, device=dev)
        self.out_buf = torch.zeros(cap, H, dtype=self.combine_dtype, device=dev)
        self.n_local = torch.zeros(1, dtype=torch.int32, device=dev)
        self.step_metadata = torch.zeros(8, dtype=torch.int32, device=dev)
        self.step_state = torch.zeros(_ext.STEP_STATE_WORDS, dtype=torch.int32, device=dev)
        self.local_tokens = 0
        self._make_plans()
        h.register_reset_hook(self._reset_step_state)
        # Combine timing reduces valid data (bench_nvls.py:81).
        self.rsv.tensor.normal_()
        torch.cuda.synchronize()
        dist.barrier(self.group)
        self._built = True

    def _make_plans(self):
        h = self.heap
        self._step_plans = {}
        if self.fp8:        # the quantised dispatch exists only inside the step kernel
            self.meta_plan = self.agv_plan = self.rsv_plan = None
            return
        self.meta_plan = MetadataPlan(h, self.n_local, self.step_metadata, self.cap)
        self.agv_plan = AllGatherVPlan(h, [self.agv_h, self.agv_r, self.agv_p],
                                       [self.in_hidden, self.in_routing, self.in_probs], self.n_local,
                                       self.step_metadata, self.cap, grid=self.num_sms, threads=self.threads,
                                       ll_stage=self.ll_agv, ll_rows=self.ll_rows)
        self.rsv_plan = ReduceScatterVPlan(h, self.out_buf, self.rsv, self.n_local, self.step_metadata, self.cap,
                                           grid=self.num_sms, threads=self.threads,
                                           ll_stage=self.ll_rsv, ll_rows=self.ll_rows)
        self._step_plans = {}

    def _step_plan(self, num_layers: int, **check) -> DenseStepPlan:
        cached = not check            # plans of the self-checking build are made per use
        plan = self._step_plans.get(num_layers) if cached else None
        if plan is None:
            dsts, srcs = [self.agv2_h, self.agv2_r, self.agv2_p], [self.in_hidden, self.in_routing, self.in_probs]
            if self.fp8:
                dsts, srcs, check = dsts + [self.agv2_s], srcs + [None], dict(check, fp8_hidden=self.cfg.hidden)
            plan = DenseStepPlan(self.heap, dsts, srcs, self.out_buf, self.rsv,
                                 self.n_local, self.step_metadata, self.cap, num_layers, grid=self.num_sms,
                                 threads=self.threads, agv_ll_stage=self.ll_agv, rsv_ll_stage=self.ll_rsv,
                                 ll_rows=self.ll_rows, credits=self.step_credits,
                                 groups=self.groups if self.num_sms <= DEFAULT_GRID else 1,
                                 group_min_bytes=self.group_min_bytes, state=self.step_state, **check)
            if cached:
                self._step_plans[num_layers] = plan
        return plan

    def race_check(self, total_layers: int = 200):
        """Write-after-read stress of the step kernel on the real transport: steps of 5-8 layers that
        alternate between packet mode and barrier mode, run with the self-checking payload (a hash of
        layer number and position that every receiver verifies right after its barrier or poll) while
        a different rank is slowed down in every step by a bounded sleep per layer.  Returns
        ``(ok, detail)``; collective."""
        w, rank = self.cfg.ep_size, self.cfg.rank
        errs = torch.zeros(1, dtype=torch.int32, device=self.device)
        small = max(1, min(w + 1, self.ll_rows)) if self.ll_rows > 0 else 0
        big = min(self.cap * w, max(self.ll_rows + w, 6 * w))
        done, step, modes = 0, 0, set()
        saved = int(self.n_local.item())
        while done < total_layers:
            B = small if (step % 2 == 0 and small) else big
            layers = 5 + step % 4
            self.n_local.fill_(self._validation_counts(B)[rank])
            delay = 20000 + 3000 * (step % 5) if step % w == rank else (7000 if (step + 2) % w == rank else 0)
            self._step_plan(layers, check_errors=errs, delay_ns=delay, delay_every=1 + step % 3).launch(self.pdl)
            modes.add(int(self.step_metadata[6].item()))
            done += layers
            step += 1
        self._sync_all()
        self.n_local.fill_(saved)
        bad = int(errs.item())
        return bad == 0, (f"{done} layers in {step} steps (modes seen: "
                          f"{'+'.join('packets' if m else 'barrier' for m in sorted(modes))}, groups={self.groups}), "
                          f"per-rank delays up to 32 us per layer: {bad} payload mismatches")


    def _reset_step_state(self):
        """After the heap's flags were cleared: restart the sequence words of the step kernel.  The
        packet flag base keeps growing (staging areas may hold packets with earlier flags) and is
        made equal on all ranks."""
        base = self.step_state[_ext.STATE_LL_BASE:_ext.STATE_LL_BASE + 1].to(torch.int64) + 4 * 1024
        if self.cfg.ep_size > 1:
            dist.all_reduce(base, op=dist.ReduceOp.MAX, group=self.group)
        self.step_state.zero_()
        self.step_state[_ext.STATE_LL_BASE] = int(base.item()) & 0x7FFFFFFF
        self.step_credits.tensor.zero_()          # the per-block credit counts restart with the epochs

    def _grid_for(self, cfg: Config, num_sms: int) -> int:
        # A world of one is a local copy: with one kernel per operation two blocks per SM keep more
        # bytes in flight (measured); the persistent kernel holds one block per SM and unrolls deeper.
        if self.persistent:
            return int(num_sms)
        return int(num_sms) * (2 if cfg.ep_size == 1 and int(num_sms) == DEFAULT_GRID else 1)

    def set_num_sms(self, num_sms: int):
        self.num_sms = self._grid_for(self.cfg, num_sms)
        if self._built:
            self._make_plans()

    # -- per-batch ---------------------------------------------------------------------------------
    def setup_batch(self, hidden, topk_idx, topk_weights):
        assert self._built
        self._load_rows(hidden, topk_idx, topk_weights)

    @property
    def out(self):
        return self.out_buf[:self.local_tokens]

    # -- timed ops -----------------------------------------------------------------------------------
    def _standalone(self, plan):
        if plan is None:
            raise RuntimeError("with fp8 dispatch the dense path runs as whole decode steps only (decode_step)")
        return plan

    def metadata(self):
        self._standalone(self.meta_plan).launch(self.pdl)

    def dispatch(self):
        self._standalone(self.agv_plan).launch(self.pdl)

    def combine(self):
        self._standalone(self.rsv_plan).launch(self.pdl)

    def decode_step(self, num_layers: int):
        if self.persistent:
            self._step_plan(num_layers).launch(self.pdl)
        else:
            dense_decode_step(self.heap, self.meta_plan, self.agv_plan, self.rsv_plan, num_layers, self.pdl)

    def gathered(self):
        """(hidden, routing, probs) views of the rows gathered by the LAST decode step
        (host-synchronising: reads the parity word the step kernel wrote).  With fp8 dispatch the first
        entry is the pair (e4m3 bytes, fp32 scales)."""
        par = int(self.step_metadata[5].item()) if self.persistent else 0
        hid = (self.agv2_h.tensor[par], self.agv2_s.tensor[par]) if self.fp8 else self.agv2_h.tensor[par]
        return hid, self.agv2_r.tensor[par], self.agv2_p.tensor[par]

    def gathered_hidden_bf16(self, rows: int):
        """The first ``rows`` gathered hidden rows as bf16 (dequantised when the dispatch was fp8)."""
        hid = self.gathered()[0]
        if not self.fp8:
            return hid[:rows]
        from ..ops.a2a import dequant_e4m3_1x128
        return dequant_e4m3_1x128(hid[0][:rows], hid[1][:rows])

    def check_health(self):
        self.heap.check_status()

    # -- correctness ------------------------------------------------------------------------------------
    def _sync_all(self):
        torch.cuda.synchronize()
        dist.barrier(self.group)

    def validate(self):
        """Known-value checks with random per-element data at B = 2*ep and B = 1 (idle ranks):
        gather bit-exact, reduce == world * rsv (bench_nvls.py:124-172)."""
        w, rank, dev = self.cfg.ep_size, self.cfg.rank, self.device
        H, K, E, g = self.cfg.hidden, self.cfg.topk, self.cfg.num_experts, max(self.cfg.global_cap, 1)
        results = []
        if self.fp8:
            return self._validate_fp8()
        for B in (w * 2, 1):
            counts = self._validation_counts(B)
            if max(counts) > self.cap:
                results.append((f"dense AGV-V gather   B={B:<4d}", True, "skipped: batch exceeds capacity"))
                continue
            n, off, valid = counts[rank], sum(counts[:rank]), sum(counts)
            gen = torch.Generator(device=dev).manual_seed(20260701 + B)      # same on all ranks
            full_h = torch.randn(valid, H, generator=gen, device=dev).to(torch.bfloat16)
            full_r = torch.stack([torch.randperm(E, generator=gen, device=dev)[:K] for _ in range(valid)])
            full_p = torch.rand(valid, K, generator=gen, device=dev)
            self.setup_batch(full_h[off:off + n], full_r[off:off + n], full_p[off:off + n])
            self.metadata()
            self.dispatch()
            self._sync_all()
            meta = self.step_metadata[:3].tolist()
            ok = (meta == [valid, off, max(counts)]
                  and torch.equal(self.agv_h.tensor[:valid], full_h)
                  and torch.equal(self.agv_r.tensor[:valid], full_r)
                  and torch.equal(self.agv_p.tensor[:valid], full_p))
            results.append((f"dense AGV-V gather   B={B:<4d}", bool(ok),
                            f"metadata={meta}; gathered hidden+routing+probs == full tensors bit-exact"))
            rsv_full = torch.randn(valid, H, generator=gen, device=dev).to(self.combine_dtype)
            self.rsv.tensor[:valid] = rsv_full
            self._sync_all()
            self.combine()
            self._sync_all()
            ok = n == 0 or torch.allclose(self.out.float(), w * rsv_full[off:off + n].float(), rtol=2e-2, atol=2e-2)
            results.append((f"dense RSV-V reduce   B={B:<4d}", bool(ok),
                            f"output == world*rsv[global_id] element-wise; local_tokens={n}"))
            if self.persistent:
                # the whole step as one persistent kernel: 3 layers, then 2 (both parities end a step)
                for nl in (3, 2):
                    for t in (self.agv2_h, self.agv2_r, self.agv2_p):
                        t.tensor.zero_()
                    self.out_buf.zero_()
                    self._sync_all()
                    self.decode_step(nl)
                    self._sync_all()
                    meta = self.step_metadata.tolist()
                    gh, gr, gp = self.gathered()
                    ok = (meta[:3] == [valid, off, max(counts)]
                          and torch.equal(gh[:valid], full_h) and torch.equal(gr[:valid], full_r)
                          and torch.equal(gp[:valid], full_p)
                          and (n == 0 or torch.allclose(self.out.float(), w * rsv_full[off:off + n].float(),
                                                        rtol=2e-2, atol=2e-2)))
                    results.append((f"dense step kernel    B={B:<4d}", bool(ok),
                                    f"{nl} layers in one launch: gathered rows bit-exact in parity {meta[5]}, "
                                    f"output == world*rsv; mode={'packets' if meta[6] else 'barrier'} groups={meta[7]}"))
        if self.persistent:
            ok, detail = self.race_check()
            results.append(("dense step kernel race check", ok, detail))
        try:
            self.check_health()
        except Exception as e:
            results.append(("dense device status", False, str(e)))
        return results

    def _validate_fp8(self):
        """Quantised dispatch: gathered routing/probs bit-exact, scales == amax / 448 per 128 values,
        dequantised rows within e4m3 rounding of the inputs, combine == world * rsv; B = 2*ep (and a step
        of 3 layers, then 2) and B = 1."""
        from ..ops import oracle
        w, rank, dev = self.cfg.ep_size, self.cfg.rank, self.device
        H, K, E = self.cfg.hidden, self.cfg.topk, self.cfg.num_experts
        results = []
        for B in (w * 2, 1):
            counts = self._validation_counts(B)
            if max(counts) > self.cap:
                continue
            n, off, valid = counts[rank], sum(counts[:rank]), sum(counts)
            gen = torch.Generator(device=dev).manual_seed(20260701 + B)
            full_h = torch.randn(valid, H, generator=gen, device=dev).to(torch.bfloat16)
            full_h[0, :128] = 0                      # an all-zero block: scale 1, values 0
            full_r = torch.stack([torch.randperm(E, generator=gen, device=dev)[:K] for _ in range(valid)])
            full_p = torch.rand(valid, K, generator=gen, device=dev)
            rsv_full = torch.randn(valid, H, generator=gen, device=dev).to(self.combine_dtype)
            self.setup_batch(full_h[off:off + n], full_r[off:off + n], full_p[off:off + n])
            self.rsv.tensor[:valid] = rsv_full
            for nl in (3, 2):
                for t in (self.agv2_h, self.agv2_r, self.agv2_p, self.agv2_s):
                    t.tensor.zero_()
                self.out_buf.zero_()
                self._sync_all()
                self.decode_step(nl)
                self._sync_all()
                meta = self.step_metadata.tolist()
                (q, sc), gr, gp = self.gathered()
                _, s_ref = oracle.quant_e4m3_1x128(full_h.float().cpu())
                back = oracle.dequant_e4m3_1x128(q[:valid].cpu().view(torch.float8_e4m3fn), sc[:valid].cpu())
                want = full_h.float().cpu()
                ok = (meta[:3] == [valid, off, max(counts)] and torch.equal(gr[:valid], full_r)
                      and torch.equal(gp[:valid], full_p)
                      and torch.allclose(sc[:valid].cpu(), s_ref, rtol=1e-6, atol=0)
                      and bool(((back - want).abs() <= 0.0625 * want.abs()
                                + 2e-3 * sc[:valid].cpu().repeat_interleave(128, dim=1)).all())
                      and (n == 0 or torch.allclose(self.out.float(), w * rsv_full[off:off + n].float(),
                                                    rtol=2e-2, atol=2e-2)))
                results.append((f"dense-fp8 step kernel B={B:<4d}", bool(ok),
                                f"{nl} layers: e4m3 rows + fp32 scales match the 1x128 quantisation of the inputs, "
                                f"routing/probs bit-exact, output == world*rsv; mode={'packets' if meta[6] else 'barrier'}"))
        try:
            self.check_health()
        except Exception as e:
            results.append(("dense-fp8 device status", False, str(e)))
        return results

    def functional_roundtrip(self, hidden, topk_idx):
        """dispatch -> masked identity expert -> combine; returns ``[n, H]`` = m * x
        (bench_nvls.py:174-199)."""
        w, rank = self.cfg.ep_size, self.cfg.rank
        epr = self.cfg.num_experts // w
        n = hidden.shape[0]
        if self.fp8:
            # The quantised dispatch lives in the step kernel: one layer to gather, the masked identity
            # expert on the host, one more layer whose combine then reduces the masked rows.
            self.setup_batch(hidden, topk_idx, torch.ones(n, self.cfg.topk, device=self.device))
            self.rsv.tensor.zero_()
            self._sync_all()
            self.decode_step(1)
            self._sync_all()
            valid = int(self.step_metadata[0].item())
            gh, gr = self.gathered_hidden_bf16(valid), self.gathered()[1][:valid]
            local = ((gr >= rank * epr) & (gr < (rank + 1) * epr)).any(dim=1, keepdim=True)
            self.rsv.tensor[:valid] = torch.where(local, gh.float(), torch.zeros((), device=self.device)).to(self.combine_dtype)
            self._sync_all()
            self.decode_step(1)
            self._sync_all()
            return self.out
        self.setup_batch(hidden, topk_idx, torch.ones(n, self.cfg.topk, device=self.device))
        self.metadata()
        self.dispatch()
        self._sync_all()
        valid = int(self.step_metadata[0].item())
        gh, gr = self.agv_h.tensor[:valid], self.agv_r.tensor[:valid]
        local = ((gr >= rank * epr) & (gr < (rank + 1) * epr)).any(dim=1, keepdim=True)
        self.rsv.tensor[:valid] = torch.where(local, gh.float(), torch.zeros((), device=self.device)).to(self.combine_dtype)
        self._sync_all()
        self.combine()
        self._sync_all()
        return self.out

    def destroy(self):
        if self._own_heap and self.heap is not None:
            self.heap.destroy()
        self.heap = None
        self._built = False
