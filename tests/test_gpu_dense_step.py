"""The persistent decode-step kernel (count exchange + every layer in one launch), emulated as W
ranks inside one cooperative launch on ONE GPU, against the CPU oracle; plus its race test: the
self-checking build with per-rank delays chosen on the host, alternating packet and barrier steps."""
import pytest
import torch

from moe_comms_benchmarking_b200.ops import _ext, oracle
from moe_comms_benchmarking_b200.ops.dense import agv_ll_stage_bytes, rsv_ll_stage_bytes
from moe_comms_benchmarking_b200.parallel.emulation import EmuWorld
from moe_comms_benchmarking_b200.parallel.symm_heap import DeviceStatusError

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scalars(vals):
    return [torch.tensor([v], dtype=torch.int32, device=DEV) for v in vals]


class _Rig:
    """Buffers of an emulated dense dispatcher: [2, cap*W, cols] gathered tensors per rank."""

    def __init__(self, W, cap, H, K, LL, dtype=torch.bfloat16):
        self.W, self.cap, self.H, self.K, self.LL = W, cap, H, K, LL
        self.w = EmuWorld(W, 16 << 20, DEV)
        self.dst_h = self.w.alloc([2, cap * W, H], torch.bfloat16)
        self.dst_r = self.w.alloc([2, cap * W, K], torch.int64)
        self.dst_p = self.w.alloc([2, cap * W, K], torch.float32)
        self.rsv = self.w.alloc([cap * W, H], dtype)
        self.st_a = self.w.alloc([max(16, agv_ll_stage_bytes(LL, [H * 2, K * 8, K * 4]))], torch.uint8)
        self.st_r = self.w.alloc([max(16, rsv_ll_stage_bytes(W, LL, cap, H * 2))], torch.uint8)
        self.metas = [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(W)]
        self.outs = [torch.zeros(cap, H, dtype=dtype, device=DEV) for _ in range(W)]
        self.g = torch.Generator(device=DEV).manual_seed(77)
        self.dtype = dtype

    def new_inputs(self):
        W, cap, H, K, g = self.W, self.cap, self.H, self.K, self.g
        self.src_h = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
        self.src_r = [torch.randint(0, 512, (cap, K), device=DEV, generator=g) for _ in range(W)]
        self.src_p = [torch.rand(cap, K, device=DEV, generator=g) for _ in range(W)]
        for r in range(W):
            self.rsv[r].tensor.copy_(torch.randn(cap * W, H, device=DEV, generator=g).to(self.dtype))

    def step(self, counts, layers, grid, threads, groups=1, **kw):
        self.w.dense_step([self.dst_h, self.dst_r, self.dst_p], [self.src_h, self.src_r, self.src_p], self.outs,
                          self.rsv, _scalars(counts), self.metas, self.cap, layers, grid=grid, threads=threads,
                          agv_ll_stage=self.st_a, rsv_ll_stage=self.st_r, ll_rows=self.LL, groups=groups,
                          group_min_bytes=0, **kw)

    def check(self, counts, expect_mode=None, tol=2e-2):
        W = self.W
        valid = sum(counts)
        want_meta = oracle.metadata(counts)
        full = [oracle.all_gather_v([s[r][:counts[r]] for r in range(W)]) for s in (self.src_h, self.src_r, self.src_p)]
        want = oracle.reduce_scatter_v([self.rsv[r].tensor[:valid].cpu() for r in range(W)], counts)
        for r in range(W):
            m = self.metas[r].tolist()
            assert m[:3] == want_meta[r]
            if expect_mode is not None:
                assert m[6] == expect_mode
            par = m[5]
            assert torch.equal(self.dst_h[r].tensor[par, :valid], full[0])
            assert torch.equal(self.dst_r[r].tensor[par, :valid], full[1])
            assert torch.equal(self.dst_p[r].tensor[par, :valid], full[2])
            assert torch.allclose(self.outs[r][:counts[r]].float().cpu(), want[r], rtol=tol, atol=tol)


@pytest.mark.parametrize("grid,threads,groups", [(1, 128, 1), (8, 256, 1), (8, 256, 2), (12, 128, 3)])
def test_step_kernel_barrier_and_packet_modes(lib, grid, threads, groups):
    """Steps of 1-3 layers on the same buffers, switching between packet mode (<= 8 rows in total)
    and barrier mode, with idle ranks and an empty step; every step against the oracle."""
    rig = _Rig(W=4, cap=16, H=256, K=22, LL=8)
    plan = [([5, 0, 16, 3], 3, 0), ([1, 2, 3, 2], 2, 1), ([1, 0, 0, 0], 3, 1), ([16, 16, 16, 16], 1, 0),
            ([0, 0, 0, 0], 2, None), ([0, 8, 0, 0], 5, 1), ([4, 4, 4, 4], 2, 0), ([2, 2, 2, 2], 4, 1)]
    for counts, layers, mode in plan:
        rig.new_inputs()
        rig.step(counts, layers, grid, threads, groups)
        rig.check(counts, expect_mode=mode)
        if mode == 0 and groups > 1 and grid >= 2 * groups:
            assert rig.metas[0][7].item() == groups
    rig.w.check_status()


def test_step_kernel_grid_may_change_between_steps(lib):
    """The sequence words live outside the per-block counters, so a step may use another grid size
    than the one before (packet flags and barrier targets stay in agreement)."""
    rig = _Rig(W=2, cap=32, H=256, K=22, LL=8)
    for counts, layers, grid in (([3, 2], 3, 4), ([3, 2], 3, 16), ([20, 32], 2, 2), ([20, 32], 2, 24), ([4, 4], 3, 8)):
        rig.new_inputs()
        rig.step(counts, layers, grid, 256)
        rig.check(counts)
    rig.w.check_status()


def test_step_kernel_fp32_combine(lib):
    rig = _Rig(W=2, cap=8, H=128, K=4, LL=0, dtype=torch.float32)
    rig.new_inputs()
    rig.step([3, 8], 2, 4, 128)
    rig.check([3, 8], expect_mode=0, tol=1e-5)
    rig.w.check_status()


@pytest.mark.parametrize("grid,threads", [(2, 128), (8, 256)])
def test_step_kernel_fp8_dispatch(lib, grid, threads):
    """1 x 128 block-scaled e4m3 dispatch inside the step kernel, in barrier mode and in packet mode:
    scales == amax / 448, values within e4m3 rounding of the inputs (against the CPU oracle's
    quantiser), routing / probs bit-exact, combine unaffected."""
    W, cap, H, K, LL = 4, 16, 512, 6, 8
    w = EmuWorld(W, 16 << 20, DEV)
    dst_q = w.alloc([2, cap * W, H], torch.uint8)
    dst_r = w.alloc([2, cap * W, K], torch.int64)
    dst_p = w.alloc([2, cap * W, K], torch.float32)
    dst_s = w.alloc([2, cap * W, H // 128], torch.float32)
    rsv = w.alloc([cap * W, H], torch.bfloat16)
    st_a = w.alloc([agv_ll_stage_bytes(LL, [H, K * 8, K * 4, H // 128 * 4])], torch.uint8)
    st_r = w.alloc([rsv_ll_stage_bytes(W, LL, cap, H * 2)], torch.uint8)
    metas = [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(W)]
    outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
    g = torch.Generator(device=DEV).manual_seed(5)
    for counts, layers, mode in (([5, 0, 16, 3], 2, 0), ([1, 2, 3, 2], 3, 1), ([16, 16, 16, 16], 1, 0), ([0, 1, 0, 0], 2, 1)):
        src_h = [(torch.randn(cap, H, device=DEV, generator=g) * (1 + r)).to(torch.bfloat16) for r in range(W)]
        src_h[1][0, :128] = 0                      # an all-zero block
        src_r = [torch.randint(0, 512, (cap, K), device=DEV, generator=g) for _ in range(W)]
        src_p = [torch.rand(cap, K, device=DEV, generator=g) for _ in range(W)]
        for r in range(W):
            rsv[r].tensor.copy_(torch.randn(cap * W, H, device=DEV, generator=g).to(torch.bfloat16))
        w.dense_step([dst_q, dst_r, dst_p, dst_s], [src_h, src_r, src_p, None], outs, rsv, _scalars(counts), metas, cap,
                     layers, grid=grid, threads=threads, agv_ll_stage=st_a, rsv_ll_stage=st_r, ll_rows=LL, fp8_hidden=H)
        valid = sum(counts)
        full_h = oracle.all_gather_v([src_h[r][:counts[r]] for r in range(W)]).float().cpu()
        full_r = oracle.all_gather_v([src_r[r][:counts[r]] for r in range(W)])
        full_p = oracle.all_gather_v([src_p[r][:counts[r]] for r in range(W)])
        q_ref, s_ref = oracle.quant_e4m3_1x128(full_h)
        want = oracle.reduce_scatter_v([rsv[r].tensor[:valid].cpu() for r in range(W)], counts)
        for r in range(W):
            m = metas[r].tolist()
            assert m[6] == mode
            par = m[5]
            sc = dst_s[r].tensor[par, :valid].cpu()
            q = dst_q[r].tensor[par, :valid].cpu().view(torch.float8_e4m3fn)
            assert torch.allclose(sc, s_ref, rtol=1e-6, atol=0)
            back = oracle.dequant_e4m3_1x128(q, sc)
            assert ((back - full_h).abs() <= 0.0625 * full_h.abs() + 2e-3 * sc.repeat_interleave(128, dim=1)).all()
            assert (q.float() == q_ref.float()).float().mean() > 0.999
            assert torch.equal(dst_r[r].tensor[par, :valid], full_r) and torch.equal(dst_p[r].tensor[par, :valid], full_p)
            assert torch.allclose(outs[r][:counts[r]].float().cpu(), want[r], rtol=2e-2, atol=2e-2)
    w.check_status()


def test_step_kernel_bounded_wait_with_a_phantom_rank(lib):
    """A world that counts a rank which never runs: the count exchange cannot complete, the
    bounded wait runs out, the status words say so and the GPU context stays usable."""
    W, cap, H, K = 2, 4, 128, 4
    w = EmuWorld(W, 1 << 20, DEV, timeout_s=0.2, phantom_ranks=1)
    T = W + 1
    dst = [w.alloc([2, cap * T, c], dt) for c, dt in ((H, torch.bfloat16), (K, torch.int64), (K, torch.float32))]
    rsv = w.alloc([cap * T, H], torch.bfloat16)
    srcs = [[torch.zeros(cap, c, dtype=dt, device=DEV) for _ in range(W)]
            for c, dt in ((H, torch.bfloat16), (K, torch.int64), (K, torch.float32))]
    outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
    metas = [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(W)]
    w.dense_step(dst, srcs, outs, rsv, _scalars([1, 1]), metas, cap, 2, grid=2, threads=128)
    with pytest.raises(DeviceStatusError) as e:
        w.check_status()
    assert e.value.code == 1 and e.value.words[1] == _ext.SITE_STEP_META
    assert torch.ones(4, device=DEV).sum().item() == 4.0     # the context still works


@pytest.mark.parametrize("groups", [1, 2])
def test_step_kernel_race_check_with_delays(lib, groups):
    """Write-after-read stress: >= 200 layers in steps that alternate between packet mode and
    barrier mode, self-checking payload (a hash of the layer number and the position, verified by
    every receiver right after its barrier or poll), and a different rank slowed down in every step
    by a bounded sleep per layer.  A push that overtakes a reader, or a stale packet, is a mismatch."""
    W, cap, LL = 4, 16, 8
    rig = _Rig(W, cap, H=256, K=22, LL=LL)
    rig.new_inputs()
    errs = [torch.zeros(1, dtype=torch.int32, device=DEV) for _ in range(W)]
    layers_done = 0
    step = 0
    while layers_done < 220:
        packet = step % 2 == 0
        counts = [[2, 1, 0, 3], [1, 1, 1, 1], [0, 0, 5, 0]][step % 3] if packet else \
                 [[16, 9, 0, 12], [7, 16, 16, 1]][(step // 2) % 2]
        layers = 5 + step % 4
        delays = [0] * W
        delays[step % W] = 20000 + 3000 * (step % 5)
        delays[(step + 2) % W] = 7000
        rig.step(counts, layers, 8, 256, groups, check_errors=errs, delays_ns=delays, delay_every=1 + step % 3)
        for r in range(W):
            assert rig.metas[r][6].item() == (1 if packet else 0)
        layers_done += layers
        step += 1
    rig.w.check_status()
    assert [int(e.item()) for e in errs] == [0] * W
    # the combine of the last step is the real one (only the gathered payload is synthetic)
    want = oracle.reduce_scatter_v([rig.rsv[r].tensor[:sum(counts)].cpu() for r in range(W)], counts)
    for r in range(W):
        assert torch.allclose(rig.outs[r][:counts[r]].float().cpu(), want[r], rtol=2e-2, atol=2e-2)


def test_step_kernel_check_payload_depends_on_the_layer(lib):
    """The self-checking payload is a function of the layer number: two consecutive one-layer steps
    leave different words in the two parities of the gathered buffer, identical on all ranks."""
    rig = _Rig(W=2, cap=8, H=128, K=4, LL=0)
    rig.new_inputs()
    errs = [torch.zeros(1, dtype=torch.int32, device=DEV) for _ in range(2)]
    rig.step([4, 4], 1, 2, 128, check_errors=errs)
    par = rig.metas[1][5].item()
    first = rig.dst_h[1].tensor[par, :8].view(torch.int16).clone()      # raw words (the hash may spell NaNs)
    assert torch.equal(first, rig.dst_h[0].tensor[par, :8].view(torch.int16)) and first.count_nonzero().item() > 0
    rig.step([4, 4], 1, 2, 128, check_errors=errs)
    par2 = rig.metas[1][5].item()
    assert par2 != par and not torch.equal(rig.dst_h[1].tensor[par2, :8].view(torch.int16), first)
    assert [int(e.item()) for e in errs] == [0, 0]
    rig.w.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("K,grid,threads", [(22, 148, 512), (5, 2, 64), (3, 1, 32)])
def test_world_of_one_copies(lib, dtype, K, grid, threads):
    """A world of one: the layers of a step are flat copies of all ranges of a layer at once.  Rows of 8, 12, 20,
    24 or 40 bytes leave words behind the last whole 16-byte pack, and the small grids take several rounds of packs."""
    cap, H = 132, 264
    rig = _Rig(1, cap, H, K, 0, dtype)
    for step, (n, layers) in enumerate([(1, 3), (3, 2), (132, 2), (0, 1), (7, 4)]):
        rig.new_inputs()
        rig.step([n], layers, grid, threads)
        rig.check([n], expect_mode=0)
        assert torch.equal(rig.outs[0][:n], rig.rsv[0].tensor[:n])
    rig.w.check_status()


@pytest.mark.parametrize("n", [1, 2, 4, 5, 9, 16])          # 17.5 packs a row on two warps: a ragged group of packs, words behind the last one
@pytest.mark.parametrize("layers", [1, 2, 7, 8, 9, 17])     # every number of groups at a time, one less, and steps dealt in runs
def test_world_of_one_layers_in_flight(lib, n, layers):
    rig = _Rig(1, 16, 64, 2, 0)
    rig.new_inputs()
    rig.step([n], layers, 1, 64)
    rig.check([n], expect_mode=0)
    par = int(rig.metas[0][5])
    for p in {par, (par + layers - 1) % 2}:                 # the last two layers, where there are two
        for dst, src in ((rig.dst_h, rig.src_h), (rig.dst_r, rig.src_r), (rig.dst_p, rig.src_p)):
            assert torch.equal(dst[0].tensor[p, :n], src[0][:n])
    rig.w.check_status()


@pytest.mark.parametrize("form", ["in_place", "in_place_fp8", "identity"])
@pytest.mark.parametrize("n,layers", [(1, 1), (1, 9), (5, 2), (5, 3), (40, 4), (130, 3)])      # 1 to 140 packs a thread and more on 2 x 64 threads
def test_world_of_one_step_on_its_own_rows(lib, form, n, layers):
    """A step whose output is its source (each layer dispatches what the layer before combined), and one whose partial
    sums are the gathered rows of parity 0 (the identity expert): layer by layer, as with peers."""
    from moe_comms_benchmarking_b200.ops.a2a import dequant_e4m3_1x128
    from moe_comms_benchmarking_b200.ops.dense import DenseStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    cap, H, K, fp8 = 132, 256, 4, form == "in_place_fp8"
    g = torch.Generator(device=DEV).manual_seed(n + layers)
    heap = SymmetricHeap(None, 4 << 20, DEV)
    x = torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16)
    ids, w = torch.randint(0, 64, (cap, K), device=DEV, generator=g), torch.rand(cap, K, device=DEV, generator=g)
    gh = heap.alloc("gh", [2, cap, H], torch.uint8 if fp8 else torch.bfloat16)
    gi, gw = heap.alloc("gi", [2, cap, K], torch.int64), heap.alloc("gw", [2, cap, K], torch.float32)
    gs = heap.alloc("gs", [2, cap, H // 128], torch.float32)
    rsv = heap.alloc("rsv", [cap, H], torch.bfloat16)
    rsv.tensor.normal_()
    if form == "identity":
        gh.tensor.normal_()
        rsv, out = gh, torch.zeros_like(x)
    else:
        out = x
    meta = torch.zeros(8, dtype=torch.int32, device=DEV)
    plan = DenseStepPlan(heap, [gh, gi, gw] + [gs] * fp8, [x, ids, w] + [None] * fp8, out, rsv,
                         torch.tensor([n], dtype=torch.int32, device=DEV), meta, cap, layers, grid=2, threads=64,
                         fp8_hidden=H if fp8 else 0)
    for step in range(2):
        src, rows = x[:n].clone(), [gh.tensor[p, :n].clone() for p in (0, 1)]
        first = 0 if step == 0 else layers % 2
        for l in range(layers):                     # the step, one layer after the other
            par = (first + l) % 2
            rows[par] = src
            res = (rows[0] if form == "identity" else rsv.tensor[:n]).clone()
            if form != "identity":
                src = res
        plan.launch()
        torch.cuda.synchronize()
        heap.check_status()
        assert int(meta[5]) == par
        assert torch.equal(out[:n], res)
        for p in {par, (par + layers - 1) % 2}:
            if fp8:     # e4m3 has three bits behind the leading one: half a unit of the last is 2^-4 of the value, 2^-10 of the scale
                got, want = dequant_e4m3_1x128(gh.tensor[p, :n], gs.tensor[p, :n]).float(), rows[p].float()
                lim = want.abs() * (2 ** -4 + 2 ** -8) + gs.tensor[p, :n].repeat_interleave(128, 1) * 2 ** -9
                assert bool(((got - want).abs() <= lim).all())
            else:
                assert torch.equal(gh.tensor[p, :n], rows[p])
            assert torch.equal(gi.tensor[p, :n], ids[:n]) and torch.equal(gw.tensor[p, :n], w[:n])


@pytest.mark.parametrize("form", ["in_place", "in_place_fp8", "identity"])
@pytest.mark.parametrize("n,layers", [(11, 9), (12, 9), (130, 10)])      # fewer than three packs of the outputs for each of 128 threads, three, 33
def test_world_of_one_step_on_its_own_rows_many_layers(lib, form, n, layers):
    test_world_of_one_step_on_its_own_rows(lib, form, n, layers)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 17])          # 32 packs to quantise a row on three warps: fewer groups of 64 than warps, and more
@pytest.mark.parametrize("layers", [1, 3, 8, 9])
@pytest.mark.parametrize("out_cols", [256, 64])             # as many packs of expert outputs, and fewer than are quantised
def test_world_of_one_quantised_layers_in_flight(lib, n, layers, out_cols):
    """e4m3 dispatch of a world of one: the bytes, scales and copies of the last two layers, whatever number of layers is in flight."""
    from moe_comms_benchmarking_b200.ops.dense import DenseStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    cap, H, K = 20, 256, 3
    g = torch.Generator(device=DEV).manual_seed(n)
    heap = SymmetricHeap(None, 1 << 20, DEV)
    x = torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16)
    ids, w = torch.randint(0, 64, (cap, K), device=DEV, generator=g), torch.rand(cap, K, device=DEV, generator=g)
    gh, gs = heap.alloc("gh", [2, cap, H], torch.uint8), heap.alloc("gs", [2, cap, H // 128], torch.float32)
    gi, gw = heap.alloc("gi", [2, cap, K], torch.int64), heap.alloc("gw", [2, cap, K], torch.float32)
    rsv = heap.alloc("rsv", [cap, out_cols], torch.bfloat16)
    rsv.tensor.normal_()
    out, meta = torch.zeros(cap, out_cols, dtype=torch.bfloat16, device=DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
    plan = DenseStepPlan(heap, [gh, gi, gw, gs], [x, ids, w, None], out, rsv, torch.tensor([n], dtype=torch.int32, device=DEV), meta, cap,
                         layers, grid=1, threads=96, fp8_hidden=H)
    q, scale = oracle.quant_e4m3_1x128(x[:n].float().cpu())
    for step in range(2):
        for t in (gh, gs, gi, gw):
            t.tensor.zero_()
        plan.launch()
        torch.cuda.synchronize()
        heap.check_status()
        par = int(meta[5])
        assert torch.equal(out[:n], rsv.tensor[:n])
        for p in {par, (par + layers - 1) % 2}:
            assert torch.equal(gh.tensor[p, :n].cpu(), q.view(torch.uint8)) and torch.equal(gs.tensor[p, :n].cpu(), scale)
            assert torch.equal(gi.tensor[p, :n], ids[:n]) and torch.equal(gw.tensor[p, :n], w[:n])
        assert not gh.tensor[:, n:].any() and not gs.tensor[:, n:].any()


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("n,layers,grid,threads", [
    (1, 88, 148, 512),           # more warps than groups of packs times layers
    (1, 3, 148, 512),
    (5, 17, 7, 96),              # runs that begin and end inside a group's layers
    (5, 9, 2, 160),
    (7, 19, 1, 32),              # all by one warp
    (4, 0, 148, 512),
])
def test_world_of_one_layers_dealt(lib, fp8, n, layers, grid, threads):
    """The layers of a step, dealt to the warps in runs of a group of packs after the other.  What the last two layers deliver, and
    nothing besides."""
    from moe_comms_benchmarking_b200.ops.dense import DenseStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    cap, H, K = 8, 256, 3
    g = torch.Generator(device=DEV).manual_seed(n + layers)
    heap = SymmetricHeap(None, 1 << 20, DEV)
    x = torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16)
    ids, w = torch.randint(0, 64, (cap, K), device=DEV, generator=g), torch.rand(cap, K, device=DEV, generator=g)
    gh, gs = heap.alloc("gh", [2, cap, H], torch.uint8 if fp8 else torch.bfloat16), heap.alloc("gs", [2, cap, H // 128], torch.float32)
    gi, gw = heap.alloc("gi", [2, cap, K], torch.int64), heap.alloc("gw", [2, cap, K], torch.float32)
    rsv = heap.alloc("rsv", [cap, H], torch.bfloat16)
    rsv.tensor.normal_()
    out, meta = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
    plan = DenseStepPlan(heap, [gh, gi, gw] + [gs] * fp8, [x, ids, w] + [None] * fp8, out, rsv, torch.tensor([n], dtype=torch.int32, device=DEV),
                         meta, cap, layers, grid=grid, threads=threads, fp8_hidden=H if fp8 else 0)
    q, scale = oracle.quant_e4m3_1x128(x[:n].float().cpu())
    for step in range(3):
        for t in (gh, gs, gi, gw):
            t.tensor.zero_()
        plan.launch()
        torch.cuda.synchronize()
        heap.check_status()
        par = int(meta[5])
        assert not layers or par == (step * layers + layers - 1) % 2
        assert torch.equal(out[:n], rsv.tensor[:n] if layers else torch.zeros_like(out[:n])) and not out[n:].any()
        for p in (0, 1):
            there = p in [(par + l) % 2 for l in range(min(layers, 2))]
            want = [(q.view(torch.uint8) if fp8 else x[:n]).to(DEV), ids[:n], w[:n]] + [scale.to(DEV)] * fp8
            for t, v in zip((gh, gi, gw, gs), want):
                assert torch.equal(t.tensor[p, :n], v if there else torch.zeros_like(v)) and not t.tensor[p, n:].any()


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("n,layers,grid,threads", [
    (1, 1, 148, 512), (8, 1, 1, 64),      # one layer: a group per warp, several rounds of eight groups
    (5, 2, 2, 32), (7, 2, 148, 512),      # four groups at a time
    (7, 3, 1, 32), (8, 4, 3, 96),         # two, with and without a layer that is not there
    (3, 5, 1, 64), (8, 8, 5, 32),         # one
    (7, 9, 2, 64),                        # the first that is dealt in runs
])
def test_world_of_one_few_layers(lib, fp8, n, layers, grid, threads):
    """Steps of up to eight layers, whose warps take all layers of one group of packs or more at a time."""
    test_world_of_one_layers_dealt(lib, fp8, n, layers, grid, threads)


@pytest.mark.parametrize("n,layers,grid,threads", [
    (8, 40, 1, 96), (8, 41, 2, 64), (7, 88, 1, 32),       # half of three warps, of two, one
    (8, 39, 1, 96), (1, 40, 2, 96),                       # too few layers, too few items per warp
    (8, 63, 1, 32), (5, 63, 1, 32), (8, 64, 1, 32),       # one warp: more groups than go by half with 63 layers, as many; more with 64
])
def test_world_of_one_half_of_the_warps(lib, n, layers, grid, threads):
    """Large bf16 copies of many layers go by half of the warps of a block."""
    test_world_of_one_layers_dealt(lib, False, n, layers, grid, threads)


@pytest.mark.parametrize("n,layers,grid,threads", [
    (8, 88, 1, 512), (8, 41, 2, 384), (7, 17, 1, 128),    # 20 warps for 16, 15 for 12, five for four: several runs a warp, which begin inside a group's layers
    (3, 60, 1, 96), (8, 39, 1, 32),                       # none more for three and for one
    (5, 9, 148, 512),                                     # fewer items than warps
])
def test_world_of_one_more_warps(lib, n, layers, grid, threads):
    """Dealt e4m3 steps have five warps for every four that the caller asked for."""
    test_world_of_one_layers_dealt(lib, True, n, layers, grid, threads)
