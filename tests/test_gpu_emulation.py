"""Multi-rank protocol of every kernel, emulated on ONE GPU (all ranks inside one cooperative
launch), against the CPU oracle."""
import pytest
import torch

from moe_comms_benchmarking_b200.ops import _ext, oracle
from moe_comms_benchmarking_b200.parallel.emulation import EmuWorld
from moe_comms_benchmarking_b200.parallel.symm_heap import DeviceStatusError

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scalars(vals):
    return [torch.tensor([v], dtype=torch.int32, device=DEV) for v in vals]


def _metas(world):
    return [torch.zeros(4, dtype=torch.int32, device=DEV) for _ in range(world)]


def test_metadata_two_steps(lib):
    w = EmuWorld(4, 1 << 16, DEV)
    metas = _metas(4)
    for step, counts in enumerate(([3, 0, 5, 2], [1, 1, 0, 7], [0, 0, 0, 0])):
        w.metadata(_scalars(counts), metas, cap=8)
        want = oracle.metadata(counts)
        for r in range(4):
            assert metas[r][:3].tolist() == want[r] and int(metas[r][3]) == step + 1
    w.check_status()


def test_metadata_capacity_error_is_reported(lib):
    w = EmuWorld(2, 1 << 16, DEV)
    w.metadata(_scalars([9, 1]), _metas(2), cap=4)
    with pytest.raises(DeviceStatusError) as e:
        w.check_status()
    assert e.value.code == 2


@pytest.mark.parametrize("grid,threads", [(1, 64), (4, 256), (16, 512)])
def test_all_gather_v_and_reduce_scatter_v(lib, grid, threads):
    W, cap, H, K = 4, 16, 256, 22
    w = EmuWorld(W, 4 << 20, DEV)
    g = torch.Generator(device=DEV).manual_seed(5)
    dst_h = w.alloc([cap * W, H], torch.bfloat16)
    dst_r = w.alloc([cap * W, K], torch.int64)
    dst_p = w.alloc([cap * W, K], torch.float32)       # 88-byte rows: the 8-byte access path
    rsv = w.alloc([cap * W, H], torch.bfloat16)
    rsv32 = w.alloc([cap * W, H], torch.float32)
    metas = _metas(W)
    for counts in ([5, 0, 16, 3], [1, 2, 3, 4]):
        n_locals = _scalars(counts)
        src_h = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
        src_r = [torch.randint(0, 512, (cap, K), device=DEV, generator=g) for _ in range(W)]
        src_p = [torch.rand(cap, K, device=DEV, generator=g) for _ in range(W)]
        w.metadata(n_locals, metas, cap)
        w.all_gather_v([dst_h, dst_r, dst_p], [src_h, src_r, src_p], n_locals, metas, cap, grid, threads)
        valid = sum(counts)
        full_h = oracle.all_gather_v([src_h[r][:counts[r]] for r in range(W)])
        full_r = oracle.all_gather_v([src_r[r][:counts[r]] for r in range(W)])
        full_p = oracle.all_gather_v([src_p[r][:counts[r]] for r in range(W)])
        for r in range(W):
            assert torch.equal(dst_h[r].tensor[:valid], full_h)
            assert torch.equal(dst_r[r].tensor[:valid], full_r)
            assert torch.equal(dst_p[r].tensor[:valid], full_p)
        # reduce-scatter: every rank contributes its own random partial sums
        for buf, dt, tol in ((rsv, torch.bfloat16, 2e-2), (rsv32, torch.float32, 1e-5)):
            for r in range(W):
                buf[r].tensor.copy_(torch.randn(cap * W, H, device=DEV, generator=g).to(dt))
            outs = [torch.zeros(cap, H, dtype=dt, device=DEV) for _ in range(W)]
            w.reduce_scatter_v(outs, buf, n_locals, metas, cap, grid, threads)
            want = oracle.reduce_scatter_v([buf[r].tensor[:valid].cpu() for r in range(W)], counts)
            for r in range(W):
                assert torch.allclose(outs[r][:counts[r]].float().cpu(), want[r], rtol=tol, atol=tol)
    w.check_status()


@pytest.mark.parametrize("grid,threads", [(1, 128), (6, 512)])
def test_low_latency_packet_mode(lib, grid, threads):
    """Small steps travel as flagged packets (no barrier).  Steps alternate between packet mode
    and the ordinary mode (more rows than the limit) on the same buffers."""
    from moe_comms_benchmarking_b200.ops.dense import agv_ll_stage_bytes, rsv_ll_stage_bytes
    W, cap, H, K, LL = 4, 16, 256, 22, 8
    w = EmuWorld(W, 8 << 20, DEV)
    g = torch.Generator(device=DEV).manual_seed(31)
    dst_h = w.alloc([cap * W, H], torch.bfloat16)
    dst_r = w.alloc([cap * W, K], torch.int64)
    dst_p = w.alloc([cap * W, K], torch.float32)
    rsv = w.alloc([cap * W, H], torch.bfloat16)
    st_a = w.alloc([agv_ll_stage_bytes(LL, [H * 2, K * 8, K * 4])], torch.uint8)
    st_r = w.alloc([rsv_ll_stage_bytes(W, LL, cap, H * 2)], torch.uint8)
    metas = _metas(W)
    for counts in ([4, 0, 2, 1], [1, 0, 0, 0], [3, 9, 1, 0], [2, 2, 2, 2], [0, 0, 0, 0], [0, 8, 0, 0], [4, 4, 4, 4]):
        n_locals = _scalars(counts)
        src_h = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
        src_r = [torch.randint(0, 512, (cap, K), device=DEV, generator=g) for _ in range(W)]
        src_p = [torch.rand(cap, K, device=DEV, generator=g) for _ in range(W)]
        for d in (dst_h, dst_r, dst_p):
            for r in range(W):
                d[r].tensor.zero_()
        w.metadata(n_locals, metas, cap)
        w.all_gather_v([dst_h, dst_r, dst_p], [src_h, src_r, src_p], n_locals, metas, cap, grid, threads,
                       ll_stage=st_a, ll_rows=LL)
        valid = sum(counts)
        full = [oracle.all_gather_v([s[r][:counts[r]] for r in range(W)]) for s in (src_h, src_r, src_p)]
        for r in range(W):
            assert torch.equal(dst_h[r].tensor[:valid], full[0])
            assert torch.equal(dst_r[r].tensor[:valid], full[1])
            assert torch.equal(dst_p[r].tensor[:valid], full[2])
        for r in range(W):
            rsv[r].tensor.copy_(torch.randn(cap * W, H, device=DEV, generator=g).to(torch.bfloat16))
        outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
        w.reduce_scatter_v(outs, rsv, n_locals, metas, cap, grid, threads, ll_stage=st_r, ll_rows=LL)
        want = oracle.reduce_scatter_v([rsv[r].tensor[:valid].cpu() for r in range(W)], counts)
        for r in range(W):
            assert torch.allclose(outs[r][:counts[r]].float().cpu(), want[r], rtol=2e-2, atol=2e-2)
    w.check_status()


def _a2a_case(W, E, K, H, counts, fp8, seed):
    cap = max(max(counts), 1)
    w = EmuWorld(W, 16 << 20, DEV)
    g = torch.Generator(device=DEV).manual_seed(seed)
    b = w.a2a_buffers(cap, H, K, fp8)
    xs = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
    idxs = [torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(cap)]) for _ in range(W)]
    ws = [torch.rand(cap, K, device=DEV, generator=g) for _ in range(W)]
    return w, b, xs, idxs, ws, _scalars(counts), cap


@pytest.mark.parametrize("counts", [[5, 0, 8, 3], [1, 0, 0, 0], [0, 0, 0, 0]])
def test_a2a_dispatch_and_combine_bf16(lib, counts):
    W, E, K, H = 4, 32, 6, 256
    w, b, xs, idxs, ws, n_locals, cap = _a2a_case(W, E, K, H, counts, False, 11)
    outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
    for _ in range(2):      # twice: counters and epochs must return to a clean state
        w.a2a_dispatch(b, xs, idxs, ws, n_locals, E)
        recv = oracle.a2a_dispatch([xs[r][:counts[r]].cpu() for r in range(W)],
                                   [idxs[r][:counts[r]].cpu() for r in range(W)], E, W)
        for d in range(W):
            got_counts = b["recv_count"][d].tensor[:W].tolist()
            assert got_counts == [recv[d][s][0].numel() for s in range(W)]
            for s in range(W):
                c = got_counts[s]
                if not c:
                    continue
                src_tok = b["recv_src"][d].tensor[s, :c].cpu().long()
                order = torch.argsort(src_tok)
                assert torch.equal(src_tok[order], recv[d][s][0])
                assert torch.equal(b["recv_x"][d].tensor[s, :c].cpu()[order], recv[d][s][1])
                assert torch.equal(b["recv_idx"][d].tensor[s, :c].cpu()[order], idxs[s][:counts[s]].cpu()[recv[d][s][0]])
                assert torch.equal(b["recv_w"][d].tensor[s, :c].cpu()[order], ws[s][:counts[s]].cpu()[recv[d][s][0]])
        w.a2a_combine(b, outs, n_locals)
        for r in range(W):
            ref = oracle.roundtrip_identity(xs[r][:counts[r]], idxs[r][:counts[r]].cpu(), E, W)
            assert torch.allclose(outs[r][:counts[r]].float().cpu(), ref, rtol=2e-2, atol=2e-2)
    w.check_status()


def test_launch_numbers_do_not_depend_on_the_grid(lib):
    """The launch number that the all-to-all combine hands from block 0 to the other blocks, and the
    packet flag of the low-latency collectives, are per-block counters that the host levels when the
    grid of a site changes: a launch with more blocks than any earlier one must neither skip the
    combine's leading cross-rank barrier nor disagree about the flag.  Every launch uses new data,
    so a block that ran ahead of the barrier or matched a stale packet produces a wrong result."""
    W, E, K, H, counts = 4, 32, 6, 256, [5, 2, 8, 3]
    w, b, xs, idxs, ws, n_locals, cap = _a2a_case(W, E, K, H, counts, False, 19)
    outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
    g = torch.Generator(device=DEV).manual_seed(3)
    for grid in (2, 8, 16, 3, 16):
        xs = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
        w.a2a_dispatch(b, xs, idxs, ws, n_locals, E, grid=grid)
        w.a2a_combine(b, outs, n_locals, grid=grid)
        for r in range(W):
            ref = oracle.roundtrip_identity(xs[r][:counts[r]], idxs[r][:counts[r]].cpu(), E, W)
            assert torch.allclose(outs[r][:counts[r]].float().cpu(), ref, rtol=2e-2, atol=2e-2)
    w.check_status()
    # packet mode of the stand-alone all-gather / reduce-scatter with a changing grid
    from moe_comms_benchmarking_b200.ops.dense import agv_ll_stage_bytes, rsv_ll_stage_bytes
    cap, LL = 8, 8
    w = EmuWorld(W, 8 << 20, DEV)
    dst = w.alloc([cap * W, H], torch.bfloat16)
    rsv = w.alloc([cap * W, H], torch.bfloat16)
    st_a = w.alloc([agv_ll_stage_bytes(LL, [H * 2])], torch.uint8)
    st_r = w.alloc([rsv_ll_stage_bytes(W, LL, cap, H * 2)], torch.uint8)
    metas, counts = _metas(W), [2, 1, 0, 3]
    n_locals = _scalars(counts)
    for grid in (1, 6, 2, 12):
        src = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
        w.metadata(n_locals, metas, cap)
        w.all_gather_v([dst], [src], n_locals, metas, cap, grid, 128, ll_stage=st_a, ll_rows=LL)
        full = oracle.all_gather_v([src[r][:counts[r]] for r in range(W)])
        for r in range(W):
            assert torch.equal(dst[r].tensor[:sum(counts)], full)
            rsv[r].tensor.copy_(torch.randn(cap * W, H, device=DEV, generator=g).to(torch.bfloat16))
        outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
        w.reduce_scatter_v(outs, rsv, n_locals, metas, cap, grid, 128, ll_stage=st_r, ll_rows=LL)
        want = oracle.reduce_scatter_v([rsv[r].tensor[:sum(counts)].cpu() for r in range(W)], counts)
        for r in range(W):
            assert torch.allclose(outs[r][:counts[r]].float().cpu(), want[r], rtol=2e-2, atol=2e-2)
    w.check_status()


@pytest.mark.parametrize("ll_rows", [0, 20])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("grid,threads", [(1, 64), (6, 256)])
def test_a2a_step_kernel(lib, fp8, grid, threads, ll_rows):
    """The persistent all-to-all step (count exchange + every layer in one launch): token-indexed
    slots, packed metadata rows with the layer's stamp, one barrier per layer; steps of 1-5 layers with
    idle ranks; received rows / routing / stamps and the combined rows against the oracle.  With
    ``ll_rows`` the small steps run in packet mode (flagged packets, credits, no barrier) and the step of 48
    tokens on the barrier path, in the same sequence of launches."""
    W, E, K, H, cap = 4, 32, 6, 512, 12
    w = EmuWorld(W, 16 << 20, DEV)
    b = w.a2a_step_buffers(cap, H, K, fp8, ll_rows=ll_rows)
    g = torch.Generator(device=DEV).manual_seed(29)
    metas = [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(W)]
    outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
    epr = E // W
    if fp8:
        for r in range(W):
            b["y"][r].tensor.copy_(torch.randn(2, W, cap, H, device=DEV, generator=g))
    for counts, layers in (([5, 0, 12, 3], 5), ([1, 0, 0, 0], 2), ([0, 0, 0, 0], 1), ([12, 12, 12, 12], 2), ([2, 7, 1, 4], 1),
                           ([3, 3, 3, 3], 4)):
        xs = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
        idxs = [torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(cap)]) for _ in range(W)]
        ws = [torch.rand(cap, K, device=DEV, generator=g) for _ in range(W)]
        if fp8:
            xs[0][0, :128] = 0
        for o in outs:
            o.fill_(-7.0)
        w.a2a_step(b, xs, idxs, ws, outs, _scalars(counts), metas, E, layers, grid=grid, threads=threads)
        par, stamp = int(metas[0][5]), int(metas[0][7])
        assert metas[0][:3].tolist() == oracle.metadata(counts)[0]
        assert int(metas[0][6]) == int(0 < sum(counts) <= ll_rows)
        for d in range(W):
            for s in range(W):
                c = counts[s]
                if not c:
                    continue
                words = b["recv_meta"][d].tensor[par, s, :c].view(torch.int32).view(c, -1)
                here = ((idxs[s][:c] // epr) == d).any(dim=1)
                assert torch.equal(words[:, 0] == stamp, here)
                sel = here.nonzero().flatten()
                if not sel.numel():
                    continue
                assert torch.equal(words[sel, 1].long(), sel)
                assert torch.equal(words[sel][:, 2:2 + 2 * K:2].long(), idxs[s][sel])
                assert torch.equal(words[sel][:, 3:3 + 2 * K:2].contiguous().view(torch.float32), ws[s][sel])
                if fp8:
                    q = b["recv_x"][d].tensor[par, s][sel].cpu().view(torch.float8_e4m3fn)
                    sc = b["recv_scale"][d].tensor[par, s][sel].cpu()
                    want = xs[s][sel].float().cpu()
                    _, s_ref = oracle.quant_e4m3_1x128(want)
                    assert torch.allclose(sc, s_ref, rtol=1e-6, atol=0)
                    back = oracle.dequant_e4m3_1x128(q, sc)
                    assert ((back - want).abs() <= 0.0625 * want.abs() + 2e-3 * sc.repeat_interleave(128, dim=1)).all()
                else:
                    assert torch.equal(b["recv_x"][d].tensor[par, s][sel], xs[s][sel])
        for r in range(W):
            c = counts[r]
            if not c:
                continue
            if not fp8:         # identity expert: the combine reads the received rows
                ref = oracle.roundtrip_identity(xs[r][:c], idxs[r][:c].cpu(), E, W)
            else:               # the sum of one expert-output row per distinct destination rank
                ref = torch.zeros(c, H)
                for d in range(W):
                    here = ((idxs[r][:c] // epr) == d).any(dim=1).cpu()
                    ref += b["y"][d].tensor[par, r, :c].float().cpu() * here[:, None]
            assert torch.allclose(outs[r][:c].float().cpu(), ref, rtol=2e-2, atol=2e-2)
    w.check_status()


@pytest.mark.parametrize("W", [1, 2])
@pytest.mark.parametrize("fp8,H", [(False, 2056), (True, 1152), (False, 1024)])
@pytest.mark.parametrize("grid,threads", [(2, 64), (37, 512)])
def test_a2a_step_kernel_row_slices(lib, W, fp8, H, grid, threads):
    """Rows served slice by slice (128 packs of 16 bytes per warp): one pack and 16 packs in the last slice, more slices
    than warps and fewer, alone and with a peer."""
    E, K, cap = 16, 5, 9
    w = EmuWorld(W, 16 << 20, DEV)
    b = w.a2a_step_buffers(cap, H, K, fp8)
    g = torch.Generator(device=DEV).manual_seed(31)
    metas = [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(W)]
    outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(W)]
    if fp8:
        for r in range(W):
            b["y"][r].tensor.copy_(torch.randn(2, W, cap, H, device=DEV, generator=g))
    for counts, layers in (([9, 4], 3), ([1, 2], 2)):
        counts = counts[:W]
        xs = [torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
        idxs = [torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(cap)]) for _ in range(W)]
        ws = [torch.rand(cap, K, device=DEV, generator=g) for _ in range(W)]
        w.a2a_step(b, xs, idxs, ws, outs, _scalars(counts), metas, E, layers, grid=grid, threads=threads)
        par, stamp = int(metas[0][5]), int(metas[0][7])
        for s in range(W):
            c = counts[s]
            ref = torch.zeros(c, H)
            for d in range(W):
                here = ((idxs[s][:c] // (E // W)) == d).any(dim=1)
                words = b["recv_meta"][d].tensor[par, s, :c].view(torch.int32).view(c, -1)
                assert torch.equal(words[:, 0] == stamp, here)
                sel = here.nonzero().flatten()
                assert torch.equal(words[sel][:, 2:2 + 2 * K:2].long(), idxs[s][sel])
                if fp8:
                    q, s_ref = oracle.quant_e4m3_1x128(xs[s][sel].float().cpu())
                    assert torch.equal(b["recv_scale"][d].tensor[par, s][sel].cpu(), s_ref)
                    assert torch.equal(b["recv_x"][d].tensor[par, s][sel].cpu(), q.view(torch.uint8))
                    ref += b["y"][d].tensor[par, s, :c].float().cpu() * here.cpu()[:, None]
                else:
                    assert torch.equal(b["recv_x"][d].tensor[par, s][sel], xs[s][sel])
                    ref += xs[s][:c].float().cpu() * here.cpu()[:, None]
            # at most two bf16 rows are summed in fp32 and rounded once
            assert torch.allclose(outs[s][:c].float().cpu(), ref, rtol=2 ** -8, atol=1e-6)
    w.check_status()


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,K,n,layers,grid,threads", [
    (128, 1, 1, 1, 148, 512),            # half a slice of one pack per lane, one id
    (1024, 32, 5, 17, 148, 512),         # 17 metadata chunks; a remainder of layers
    (1152, 5, 8, 9, 2, 320),             # 20 warps: pieces of 16 packs at the end of a row, a chain each for 16 warps
    (1152, 5, 9, 3, 2, 320),             # three layers: slices of four packs per lane, a ragged one a row
    (2048, 8, 5, 2, 10, 64),             # two: more slices of one pack per lane than warps, so of four
    (2048, 8, 6, 4, 5, 64),              # four: more slices of four than warps
    (7168, 33, 3, 4, 148, 512),          # more ids than lanes
    (1152, 5, 3, 9, 6, 256),             # 48 warps: a chain each for some, runs that begin and end inside a piece's layers
    (256, 2, 2, 33, 8, 64),              # more layers than a chain has in flight
    (1152, 5, 7, 5, 1, 64),              # two warps: many chains each, one of them one more
    (256, 3, 7, 6, 3, 160), (256, 3, 9, 33, 3, 160),      # 15 warps, 14 with a chain more: runs that the others alone take, and all
    (128, 2, 8, 7, 1, 96), (2048, 4, 4, 5, 16, 512),      # most warps with a chain more; fewer items than warps without
])
def test_a2a_step_alone_like_the_ranks(lib, world1, fp8, H, K, n, layers, grid, threads):
    """A step in a world of one whose layers run into each other, against the kernel of the emulated ranks, which takes
    layer after layer: every received byte of both parities and the combined rows.  An id outside the experts is reported by
    both and the rest delivered."""
    from moe_comms_benchmarking_b200.ops.a2a import A2AStepBuffers, A2AStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    E, cap = 40, n + 2
    w, heap = EmuWorld(1, 8 << 20, DEV), SymmetricHeap(world1, 8 << 20, DEV)
    b, bufs = w.a2a_step_buffers(cap, H, K, fp8), A2AStepBuffers(heap, cap, H, K, fp8)
    g = torch.Generator(device=DEV).manual_seed(37)
    x, y = (torch.randn(s, device=DEV, generator=g).to(torch.bfloat16) for s in ((cap, H), (2, 1, cap, H)))
    x[0, :9] = torch.tensor([0.0, -0.0, float("inf"), -float("inf"), float("nan"), 1e-40, -1e-40, 3e38, 448.0])
    y[:, 0, 0, :9] = x[0, :9]
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(cap)])
    wt = torch.rand(cap, K, device=DEV, generator=g)
    count = torch.tensor([n], dtype=torch.int32, device=DEV)
    metas = [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(2)]
    outs = [torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    for buf in [b[k][0].tensor for k in ("recv_x", "recv_meta")] + [bufs.recv_x.tensor, bufs.recv_meta.tensor]:
        buf.zero_()
    if fp8:
        b["recv_scale"][0].tensor.zero_(); bufs.recv_scale.tensor.zero_()
        b["y"][0].tensor.copy_(y); bufs.y.tensor.copy_(y)
    plan = A2AStepPlan(heap, bufs, x, idx, wt, outs[1], count, metas[1], E, layers, grid=grid, threads=threads)
    assert lib.mcb_a2a_step_apart(heap.ctx_ref(), plan._ref) == 1
    same = lambda s, t: torch.equal(s.contiguous().view(torch.uint8), t.contiguous().view(torch.uint8))
    for step in range(3):
        if step == 2:
            idx[n - 1, 0] = -1
            idx[0] = E
        w.a2a_step(b, [x], [idx], [wt], [outs[0]], [count], [metas[0]], E, layers, grid=grid, threads=threads)
        plan.launch()
        torch.cuda.synchronize()
        assert same(outs[0], outs[1]) and same(metas[0], metas[1]), f"step {step}"
        for name in ("recv_x", "recv_meta") + (("recv_scale",) if fp8 else ()):
            assert same(b[name][0].tensor, getattr(bufs, name).tensor), f"{name} in step {step}"
        assert int(w.status[0][0]) == int(heap.status.view(torch.int32)[0]) == (4 if step == 2 else 0)        # MCB_ERR_ROUTING


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,K,n,layers,grid,threads", [
    (1152, 5, 6, 1, 148, 512), (2048, 32, 5, 2, 148, 512),      # a warp for every slice of one pack per lane
    (1152, 5, 9, 1, 2, 512), (1152, 5, 10, 3, 2, 512),          # for every slice of two, the third of a row of 16 packs
    (1152, 5, 9, 1, 1, 64), (1152, 5, 9, 2, 2, 64),             # slices of four, the second of a row ragged, in several rounds
    (256, 8, 7, 3, 3, 32), (1024, 6, 8, 4, 2, 96),              # an odd layer at the end, and none
    (1024, 6, 8, 5, 2, 96),                                     # the first that is dealt
    (1152, 5, 3, 7, 1, 192), (1152, 5, 5, 8, 2, 192),           # more layers, dealt: three and five rows of two slices each for six and twelve warps
    (1152, 5, 4, 9, 1, 192), (128, 1, 29, 6, 3, 320),           # four rows; bf16: 29 slices for 30 warps
])
def test_a2a_step_alone_few_layers(lib, world1, fp8, H, K, n, layers, grid, threads):
    """Steps of up to four layers, whose warps take slices of rows, and somewhat more."""
    test_a2a_step_alone_like_the_ranks(lib, world1, fp8, H, K, n, layers, grid, threads)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,K,n,layers,grid,threads", [
    (1152, 5, 3, 5, 1, 192), (1152, 5, 5, 6, 2, 192), (1152, 5, 4, 6, 1, 192),      # bf16 rows of two slices: dealt
    (1024, 5, 6, 5, 1, 192), (1024, 5, 5, 5, 1, 192), (1024, 5, 4, 5, 1, 192),      # of one: a full round of six warps, five of six; four, dealt
    (1024, 5, 12, 5, 1, 192), (512, 5, 18, 5, 1, 192), (512, 5, 23, 5, 1, 192),     # two rounds, dealt; three of half the length; four, dealt
    (512, 5, 6, 6, 1, 192), (512, 5, 12, 6, 1, 192), (896, 5, 6, 6, 1, 192),        # six layers: slices; two rounds and longer rows, dealt
    (256, 3, 29, 5, 1, 192), (256, 3, 30, 6, 1, 192), (128, 1, 11, 6, 1, 192),      # short rows, any number of rounds
    (256, 3, 7, 47, 3, 160), (256, 3, 7, 48, 3, 160), (1152, 5, 3, 49, 2, 64),      # bf16 rows: all warps, half of them
    (128, 1, 2, 60, 1, 32), (1024, 6, 5, 51, 1, 96),                                # one warp, two of three
])
def test_a2a_step_alone_ways_of_bf16_rows(lib, world1, fp8, H, K, n, layers, grid, threads):
    """Where bf16 steps go by slices or half of the warps."""
    test_a2a_step_alone_like_the_ranks(lib, world1, fp8, H, K, n, layers, grid, threads)


@pytest.mark.parametrize("form", ["out_on_x", "out_on_ids", "echo"])
def test_a2a_step_that_reads_what_it_writes(lib, world1, form):
    """The host tells steps whose layers may run into each other from those that write what they read."""
    from moe_comms_benchmarking_b200.ops.a2a import A2AStepBuffers, A2AStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    heap = SymmetricHeap(world1, 4 << 20, DEV)
    bufs = A2AStepBuffers(heap, 8, 256, 8, False)
    mem = torch.zeros(8 * 256 * 4, dtype=torch.bfloat16, device=DEV)
    x, out = mem[:2048].view(8, 256), mem[4096:6144].view(8, 256)
    idx = torch.zeros(8, 8, dtype=torch.int64, device=DEV)
    if form == "out_on_x":
        out = mem[1024:3072].view(8, 256)
    if form == "out_on_ids":
        idx = mem[6016:6272].view(torch.int64).view(8, 8)
    count, meta = torch.tensor([8], dtype=torch.int32, device=DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
    plan = A2AStepPlan(heap, bufs, x, idx, None, out, count, meta, 4, 3)
    assert lib.mcb_a2a_step_apart(heap.ctx_ref(), plan._ref) == int(form == "echo")


def _all_quotients(exponent):
    """Blocks of 128 values whose largest has each of the 128 bf16 significands, the others every significand at
    distances of 0 .. 23 binades with alternating signs, and both zeros: every quotient the quantisation can meet."""
    sig = 1 + torch.arange(128, dtype=torch.float64) / 128
    d = torch.arange(24, dtype=torch.float64)
    v = sig.view(1, 1, 128) * 2.0 ** -d.view(1, 24, 1)
    v = torch.minimum(v, sig.view(128, 1, 1)) * (1 - 2 * (torch.arange(128) % 2))
    v[..., 0] = sig.view(128, 1)
    v[..., 1], v[..., 2] = -0.0, 0.0
    return (v * 2.0 ** exponent).to(torch.bfloat16).view(-1, 1024)


@pytest.mark.parametrize("exponent", [0, -70, -73, -126, 85, 90, 127])     # scales on both sides of the short division's range
def test_fp8_quantisation_bytes(lib, exponent):
    x = _all_quotients(exponent)
    cap, H = x.shape
    w = EmuWorld(1, 32 << 20, DEV)
    b = w.a2a_step_buffers(cap, H, 1, True)
    meta, out = torch.zeros(8, dtype=torch.int32, device=DEV), torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV)
    idx, wt = torch.zeros(cap, 1, dtype=torch.int64, device=DEV), torch.ones(cap, 1, device=DEV)
    w.a2a_step(b, [x.to(DEV)], [idx], [wt], [out], _scalars([cap]), [meta], 4, 1)
    q, scale = oracle.quant_e4m3_1x128(x.float())
    par = int(meta[5])
    assert torch.equal(b["recv_scale"][0].tensor[par, 0].cpu(), scale)
    assert torch.equal(b["recv_x"][0].tensor[par, 0].cpu(), q.view(torch.uint8))
    w.check_status()


def test_fp8_scale_passes_over_nan(lib):
    """A block's scale comes from the largest magnitude of its values that are numbers, wherever that stands and whatever its sign; from
    infinities too; and is 1 where there are none."""
    nan, inf = float("nan"), float("inf")
    x = torch.ones(128 * 4, 128)
    for i in range(128):
        x[i, i] = -3.0                                                    # the largest in every place of a block, negative
        x[128 + i, i], x[128 + i, (i + 1) % 128] = nan, -5.0              # behind a NaN
        x[256 + i] = -nan if i % 2 else nan                               # only NaNs, but for one number in half of the blocks
        if i % 4 > 1:
            x[256 + i, i] = -0.25
        x[384 + i, i], x[384 + i, i ^ 1] = (inf if i % 2 else -inf), nan
    x = x.view(-1, 1024).to(torch.bfloat16)
    w = EmuWorld(1, 32 << 20, DEV)
    cap, H = x.shape
    b = w.a2a_step_buffers(cap, H, 1, True)
    meta, out = torch.zeros(8, dtype=torch.int32, device=DEV), torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV)
    idx, wt = torch.zeros(cap, 1, dtype=torch.int64, device=DEV), torch.ones(cap, 1, device=DEV)
    w.a2a_step(b, [x.to(DEV)], [idx], [wt], [out], _scalars([cap]), [meta], 4, 1)
    xb = x.float().view(-1, 128)
    amax = torch.where(xb.isnan(), torch.zeros_like(xb), xb.abs()).amax(dim=1, keepdim=True)
    scale = torch.where(amax > 0, amax / 448.0, torch.ones_like(amax))
    q = (xb / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
    par = int(meta[5])
    assert torch.equal(b["recv_scale"][0].tensor[par, 0].cpu().view(-1, 1), scale)
    got, undefined = b["recv_x"][0].tensor[par, 0].cpu().view(-1, 128), (xb / scale).isnan()
    assert torch.equal(got[~undefined], q[~undefined]) and (got[undefined] & 0x7f == 0x7f).all()
    w.check_status()


def test_a2a_fp8_dispatch(lib):
    W, E, K, H, counts = 2, 16, 4, 512, [6, 3]
    w, b, xs, idxs, ws, n_locals, cap = _a2a_case(W, E, K, H, counts, True, 13)
    xs[0][0, :128] = 0      # an all-zero block must get scale 1 and zero values
    w.a2a_dispatch(b, xs, idxs, ws, n_locals, E)
    recv = oracle.a2a_dispatch([xs[r][:counts[r]].cpu() for r in range(W)],
                               [idxs[r][:counts[r]].cpu() for r in range(W)], E, W)
    for d in range(W):
        for s in range(W):
            c = int(b["recv_count"][d].tensor[s])
            assert c == recv[d][s][0].numel()
            if not c:
                continue
            order = torch.argsort(b["recv_src"][d].tensor[s, :c].cpu().long())
            q = b["recv_x"][d].tensor[s, :c].cpu()[order].view(torch.float8_e4m3fn)
            sc = b["recv_scale"][d].tensor[s, :c].cpu()[order]
            want = recv[d][s][1].float()
            q_ref, s_ref = oracle.quant_e4m3_1x128(want)
            assert torch.allclose(sc, s_ref, rtol=1e-6, atol=0)
            back = oracle.dequant_e4m3_1x128(q, sc)
            assert ((back - want).abs() <= 0.0625 * want.abs() + 2e-3 * sc.repeat_interleave(128, dim=1)).all()
            assert (q.float() == q_ref.float()).float().mean() > 0.999
    w.check_status()


def test_a2a_bad_expert_id_is_reported(lib):
    W, E, K, H = 2, 16, 4, 256
    w, b, xs, idxs, ws, n_locals, cap = _a2a_case(W, E, K, H, [2, 2], False, 17)
    idxs[1][0, 0] = 99
    w.a2a_dispatch(b, xs, idxs, ws, n_locals, E)
    with pytest.raises(DeviceStatusError) as e:
        w.check_status()
    assert e.value.code == 4


@pytest.mark.parametrize("hidden", [256, 1024, 4096])
def test_rs_add_norm_ag(lib, hidden):
    W, tokens = 2, 8
    w = EmuWorld(W, 1 << 20, DEV)
    g = torch.Generator(device=DEV).manual_seed(23)
    buf = w.alloc([tokens, hidden], torch.bfloat16)
    parts = [torch.randn(tokens, hidden, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
    res = [torch.randn(tokens // W, hidden, device=DEV, generator=g).to(torch.bfloat16) for _ in range(W)]
    weight = (1 + 0.1 * torch.randn(hidden, device=DEV, generator=g)).to(torch.bfloat16)
    for r in range(W):
        buf[r].tensor.copy_(parts[r])
    want, want_res = oracle.rs_add_norm_ag([p.cpu() for p in parts], [r_.cpu() for r_ in res], weight.cpu(), 1e-5)
    w.rs_add_norm_ag(buf, res, weight, 1e-5, grid=3)
    for r in range(W):
        assert torch.allclose(buf[r].tensor.float().cpu(), want, rtol=2e-2, atol=2e-2)
        assert torch.allclose(res[r].float().cpu(), want_res[r].float(), rtol=2e-2, atol=2e-2)
    w.check_status()


def test_barrier_rounds_and_bounded_wait(lib):
    """A healthy barrier passes many rounds.  With a rank that never arrives the wait runs out:
    the kernel returns, the status word says timeout, and the context keeps working."""
    w = EmuWorld(4, 1 << 16, DEV)
    w.barrier_test(grid=8, rounds=50)
    w.check_status()
    assert int(w.epochs[0][_ext.SITE_TEST * _ext.MAX_BLOCKS]) == 50
    lonely = EmuWorld(2, 1 << 16, DEV, timeout_s=0.05, phantom_ranks=1)
    lonely.barrier_test(grid=2, rounds=1)
    with pytest.raises(DeviceStatusError) as e:
        lonely.check_status()
    assert e.value.code == 1 and e.value.words[1] == _ext.SITE_TEST and e.value.words[4] == 3
    x = torch.ones(8, device=DEV)
    assert float((x * 2).sum()) == 16.0          # the context is still usable
    w.barrier_test(grid=8, rounds=1)
    w.check_status()


@pytest.mark.parametrize("H,n,layers,grid,threads", [(1024, 5, 9, 148, 512), (7168, 3, 6, 148, 512), (1152, 40, 4, 2, 320)])
def test_a2a_step_in_place(world1, H, n, layers, grid, threads):
    """A step whose output is its input, e4m3 rows: each layer sends what the layer before has put out, so the received rows of
    either parity are the expert outputs of the other one.  Fewer slices than warps and more."""
    from moe_comms_benchmarking_b200.ops.a2a import A2AStepBuffers, A2AStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    E, K, cap = 16, 4, n + 1
    heap = SymmetricHeap(world1, 16 << 20, DEV)
    bufs = A2AStepBuffers(heap, cap, H, K, True)
    g = torch.Generator(device=DEV).manual_seed(53)
    x, y = (torch.randn(s, device=DEV, generator=g).to(torch.bfloat16) for s in ((cap, H), (2, 1, cap, H)))
    bufs.y.tensor.copy_(y)
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(cap)])
    idx[n - 1] = -1 if n > 4 else idx[n - 1]            # a row for no expert: zero from the first layer on
    wt = torch.rand(cap, K, device=DEV, generator=g)
    meta = torch.zeros(8, dtype=torch.int32, device=DEV)
    before = x.clone()
    A2AStepPlan(heap, bufs, x, idx, wt, x, torch.tensor([n], dtype=torch.int32, device=DEV), meta, E, layers, grid=grid, threads=threads).launch()
    torch.cuda.synchronize()
    if n > 4:
        with pytest.raises(DeviceStatusError):
            heap.check_status()
    last = int(meta[5])                                 # parity of the last layer
    sent = n - 1 if n > 4 else n
    assert torch.equal(x[:sent], y[last, 0, :sent]) and torch.equal(x[n:], before[n:]) and not x[sent:n].any()
    for par in (0, 1):                                  # sent in a layer of parity `par`: what the layer before has put out
        q, scale = oracle.quant_e4m3_1x128(y[1 - par, 0, :sent].float().cpu())
        assert torch.equal(bufs.recv_x.tensor[par, 0, :sent].cpu(), q.view(torch.uint8))
        assert torch.equal(bufs.recv_scale.tensor[par, 0, :sent].cpu(), scale)
        words = bufs.recv_meta.tensor[par, 0, :sent].view(torch.int32).view(sent, -1)
        assert bool((words[:, 0] == int(meta[7]) - (par != last)).all())


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("K", [1, 2, 31, 32, 33, 64, 65])
def test_a2a_step_alone_metadata(world1, fp8, K):
    """Received rows and metadata of a step in a world of one against values made in torch, up to and beyond one id per lane."""
    from moe_comms_benchmarking_b200.ops.a2a import A2AStepBuffers, A2AStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    E, H, n, layers = 80, 1152, 6, 5
    heap = SymmetricHeap(world1, 16 << 20, DEV)
    bufs = A2AStepBuffers(heap, n, H, K, fp8)
    g = torch.Generator(device=DEV).manual_seed(K)
    x, y = (torch.randn(s, device=DEV, generator=g).to(torch.bfloat16) for s in ((n, H), (2, 1, n, H)))
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(n)])
    wt = torch.rand(n, K, device=DEV, generator=g)
    out, meta = torch.zeros(n, H, dtype=torch.bfloat16, device=DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
    if fp8:
        bufs.y.tensor.copy_(y)
    bufs.recv_meta.tensor.zero_()
    A2AStepPlan(heap, bufs, x, idx, wt, out, torch.tensor([n], dtype=torch.int32, device=DEV), meta, E, layers).launch()
    torch.cuda.synchronize()
    heap.check_status()
    last = int(meta[5])
    assert torch.equal(out, y[last, 0] if fp8 else x)
    for par in (0, 1):
        words = bufs.recv_meta.tensor[par, 0].contiguous().view(torch.int32).view(n, -1)
        want = torch.zeros_like(words)
        want[:, 2::2] = -1                              # no id
        want[:, 0], want[:, 1] = int(meta[7]) - (par != last), torch.arange(n, device=DEV)
        want[:, 2:2 + 2 * K:2], want[:, 3:3 + 2 * K:2] = idx.int(), wt.view(torch.int32)
        assert torch.equal(words, want)
        if fp8:
            q, scale = oracle.quant_e4m3_1x128(x.float().cpu())
            assert torch.equal(bufs.recv_x.tensor[par, 0].cpu(), q.view(torch.uint8)) and torch.equal(bufs.recv_scale.tensor[par, 0].cpu(), scale)
        else:
            assert torch.equal(bufs.recv_x.tensor[par, 0], x)


@pytest.mark.parametrize("n,layers,grid,threads", [(3, 1, 148, 512), (5, 8, 148, 512), (40, 3, 2, 320)])
def test_a2a_step_in_place_bf16(world1, n, layers, grid, threads):
    """A step whose output is its input, identity expert on bf16 rows: the rows stay as they are but for the sign of zeros, which the
    first layer's sum drops, and the row for no expert, which is zero."""
    from moe_comms_benchmarking_b200.ops.a2a import A2AStepBuffers, A2AStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    E, K, H, cap = 16, 4, 1152, n + 1
    heap = SymmetricHeap(world1, 16 << 20, DEV)
    bufs = A2AStepBuffers(heap, cap, H, K, False)
    g = torch.Generator(device=DEV).manual_seed(59)
    x = torch.randn(cap, H, device=DEV, generator=g).to(torch.bfloat16)
    x[0, :2] = torch.tensor([0.0, -0.0])
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(cap)])
    idx[n - 1] = -1
    meta = torch.zeros(8, dtype=torch.int32, device=DEV)
    bufs.recv_x.tensor.zero_()
    before = x.clone()
    A2AStepPlan(heap, bufs, x, idx, torch.rand(cap, K, device=DEV), x, torch.tensor([n], dtype=torch.int32, device=DEV), meta, E, layers,
                grid=grid, threads=threads).launch()
    torch.cuda.synchronize()
    with pytest.raises(DeviceStatusError):
        heap.check_status()
    bits = lambda t: t.contiguous().view(torch.int16)
    plain = before + 0.0                                # -0 + 0 = +0
    assert torch.equal(bits(x[:n - 1]), bits(plain[:n - 1])) and not bits(x[n - 1]).any() and torch.equal(bits(x[n:]), bits(before[n:]))
    last = int(meta[5])
    for age, par in enumerate((last, 1 - last)[:layers]):
        sent = before if layers - 1 - age == 0 else plain
        assert torch.equal(bits(bufs.recv_x.tensor[par, 0, :n - 1]), bits(sent[:n - 1])) and not bits(bufs.recv_x.tensor[par, 0, n - 1:]).any()
        words = bufs.recv_meta.tensor[par, 0, :n - 1].view(torch.int32).view(n - 1, -1)
        assert bool((words[:, 0] == int(meta[7]) - age).all())


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("K,layers", [(5, 1), (5, 3), (5, 9), (32, 9), (33, 9)])
def test_a2a_step_alone_without_weights(world1, fp8, K, layers):
    """Without weights a step delivers weight 1: every received byte as with a tensor of ones, by slices, pieces and beyond one id per lane."""
    from moe_comms_benchmarking_b200.ops.a2a import A2AStepBuffers, A2AStepPlan
    from moe_comms_benchmarking_b200.parallel.symm_heap import SymmetricHeap
    E, H, n = 40, 1152, 7
    g = torch.Generator(device=DEV).manual_seed(K + layers)
    x, y = (torch.randn(s, device=DEV, generator=g).to(torch.bfloat16) for s in ((n, H), (2, 1, n, H)))
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:K] for _ in range(n)])
    got = []
    for wt in (None, torch.ones(n, K, device=DEV)):
        heap = SymmetricHeap(world1, 16 << 20, DEV)
        bufs = A2AStepBuffers(heap, n, H, K, fp8)
        if fp8:
            bufs.y.tensor.copy_(y)
        out, meta = torch.zeros(n, H, dtype=torch.bfloat16, device=DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
        for t in (bufs.recv_x, bufs.recv_meta):
            t.tensor.zero_()
        A2AStepPlan(heap, bufs, x, idx, wt, out, torch.tensor([n], dtype=torch.int32, device=DEV), meta, E, layers).launch()
        torch.cuda.synchronize()
        heap.check_status()
        got.append([t.contiguous().view(torch.uint8).clone() for t in (out, meta, bufs.recv_x.tensor, bufs.recv_meta.tensor)])
        words = bufs.recv_meta.tensor[int(meta[5]), 0].view(torch.int32).view(n, -1)
        assert torch.equal(words[:, 2:2 + 2 * K:2].long(), idx) and bool((words[:, 3:3 + 2 * K:2].contiguous().view(torch.float32) == 1).all())
    assert all(torch.equal(a, b) for a, b in zip(*got))
