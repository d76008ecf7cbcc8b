"""Library build, struct layouts and host-side argument validation (CPU: nothing is launched)."""
import ctypes as C

import pytest
import torch

from moe_comms_benchmarking_b200.ops import _ext
from moe_comms_benchmarking_b200.ops.a2a import A2ABuffers, A2ACombinePlan, A2ADispatchPlan
from moe_comms_benchmarking_b200.ops.dense import AllGatherVPlan, MetadataPlan, ReduceScatterVPlan
from moe_comms_benchmarking_b200.ops.norm import RsAddNormAgPlan
from moe_comms_benchmarking_b200.parallel.symm_heap import (RESERVED_BYTES, DeviceStatusError, SymmetricHeap,
                                                            SymmetricHeapManager, required_bytes)


def test_library_builds_and_layouts_match(lib):
    assert lib.mcb_max_ranks() == _ext.MAX_RANKS
    assert lib.mcb_max_blocks() == _ext.MAX_BLOCKS
    assert lib.mcb_num_sites() == _ext.NUM_SITES
    assert lib.mcb_sizeof_ctx() == C.sizeof(_ext.McbCtx)


def _heap(nbytes=1 << 20):
    return SymmetricHeap(None, nbytes, "cpu")


def test_heap_bump_allocator_and_registry():
    h = _heap()
    a = h.alloc("a", [10, 3], torch.float32)
    b = h.alloc("b", [7], torch.int64)
    assert a.offset == RESERVED_BYTES and a.offset % 256 == 0 and b.offset % 256 == 0
    assert b.offset >= a.offset + a.nbytes
    assert h.alloc("a", [10, 3], torch.float32) is a
    with pytest.raises(ValueError):
        h.alloc("a", [11, 3], torch.float32)
    with pytest.raises(MemoryError):
        h.alloc("huge", [1 << 22], torch.float32)
    a.tensor.fill_(3.0)
    assert h.buffer[a.offset:a.offset + 4].view(torch.float32).item() == 3.0
    assert required_bytes([([10, 3], torch.float32), ([7], torch.int64)]) == RESERVED_BYTES + 256 + 256
    c = h.ctx()
    assert c.world == 1 and c.rank == 0 and c.transport == _ext.TRANSPORT_P2P
    assert c.heap_peer[0] == c.heap_local == h.buffer.data_ptr()


def test_heap_manager_registry():
    SymmetricHeapManager.destroy()
    assert not SymmetricHeapManager.is_initialized("k")
    h = SymmetricHeapManager.get_heap("k", None, 1 << 16, device="cpu")
    assert SymmetricHeapManager.get_heap("k") is h and SymmetricHeapManager.is_initialized("k")
    SymmetricHeapManager.destroy("k")
    assert not SymmetricHeapManager.is_initialized("k")


def test_multimem_transport_needs_multicast():
    with pytest.raises(RuntimeError):
        SymmetricHeap(None, 1 << 16, "cpu", transport="multimem")


def test_heap_allocator_choice(monkeypatch):
    """The allocator is a named choice (argument first, then the environment); a CPU heap or a world of one
    needs none of them, whatever is asked for."""
    with pytest.raises(ValueError):
        SymmetricHeap(None, 1 << 16, "cpu", allocator="cudamalloc")
    h = SymmetricHeap(None, 1 << 16, "cpu", allocator="native")
    assert h.allocator == "native" and h.buffer.device.type == "cpu" and h.mc_ptr == 0
    monkeypatch.setenv("MCB_HEAP_ALLOCATOR", "native")
    assert SymmetricHeap(None, 1 << 16, "cpu").allocator == "native"
    monkeypatch.delenv("MCB_HEAP_ALLOCATOR")
    assert SymmetricHeap(None, 1 << 16, "cpu").allocator == "torch"


def test_status_error_decoding():
    e = DeviceStatusError([1, 2, 7, 5, 8, 3, 0, 0])
    assert e.code == 1 and "timeout" in str(e) and "site 2 block 7 on rank 3" in str(e)


def test_dense_plans_validate_arguments():
    h = _heap(4 << 20)
    cap, H, K = 8, 64, 6
    n_local = torch.zeros(1, dtype=torch.int32)
    meta = torch.zeros(4, dtype=torch.int32)
    gh = h.alloc("gh", [cap, H], torch.bfloat16)
    gr = h.alloc("gr", [cap, K], torch.int64)
    src_h = torch.zeros(cap, H, dtype=torch.bfloat16)
    src_r = torch.zeros(cap, K, dtype=torch.int64)
    MetadataPlan(h, n_local, meta, cap)
    with pytest.raises(ValueError):
        MetadataPlan(h, torch.zeros(1, dtype=torch.int64), meta, cap)
    AllGatherVPlan(h, [gh, gr], [src_h, src_r], n_local, meta, cap)
    with pytest.raises(ValueError):      # source smaller than capacity
        AllGatherVPlan(h, [gh], [src_h[:4]], n_local, meta, cap)
    with pytest.raises(ValueError):      # gathered buffer too small
        AllGatherVPlan(h, [gh], [src_h], n_local, meta, cap * 2)
    with pytest.raises(ValueError):      # dtype mismatch
        AllGatherVPlan(h, [gh], [src_h.float()], n_local, meta, cap)
    with pytest.raises(ValueError):      # row not a multiple of 4 bytes
        odd = h.alloc("odd", [cap, 3], torch.uint8)
        AllGatherVPlan(h, [odd], [torch.zeros(cap, 3, dtype=torch.uint8)], n_local, meta, cap)
    with pytest.raises(ValueError):      # grid beyond the flag slots
        AllGatherVPlan(h, [gh], [src_h], n_local, meta, cap, grid=_ext.MAX_BLOCKS + 1)
    out = torch.zeros(cap, H, dtype=torch.bfloat16)
    ReduceScatterVPlan(h, out, gh, n_local, meta, cap)
    with pytest.raises(ValueError):      # rows must be multiples of 16 bytes
        g6 = h.alloc("g6", [cap, 6], torch.bfloat16)
        ReduceScatterVPlan(h, torch.zeros(cap, 6, dtype=torch.bfloat16), g6, n_local, meta, cap)
    with pytest.raises(ValueError):
        ReduceScatterVPlan(h, out.float(), gh, n_local, meta, cap)


def test_a2a_and_norm_plans_validate_arguments():
    h = _heap(8 << 20)
    cap, H, K = 4, 256, 4
    bufs = A2ABuffers(h, cap, H, K, fp8=False)
    assert bufs.y is bufs.recv_x
    n_local = torch.zeros(1, dtype=torch.int32)
    x = torch.zeros(cap, H, dtype=torch.bfloat16)
    idx = torch.zeros(cap, K, dtype=torch.int64)
    w = torch.ones(cap, K)
    A2ADispatchPlan(h, bufs, x, idx, w, n_local, 16)
    with pytest.raises(ValueError):
        A2ADispatchPlan(h, bufs, x.float(), idx, w, n_local, 16)
    with pytest.raises(ValueError):
        A2ADispatchPlan(h, bufs, x, idx.int(), w, n_local, 16)
    A2ACombinePlan(h, bufs, torch.zeros(cap, H, dtype=torch.bfloat16), n_local)
    with pytest.raises(ValueError):
        A2ABuffers(h, cap, 200, K, fp8=True, prefix="bad")
    b8 = A2ABuffers(h, cap, H, K, fp8=True, prefix="f8")
    assert b8.recv_scale.tensor.shape == (1, cap, 2) and b8.y is not b8.recv_x
    buf = h.alloc("norm", [8, 64], torch.bfloat16)
    RsAddNormAgPlan(h, buf, torch.zeros(8, 64, dtype=torch.bfloat16), torch.ones(64, dtype=torch.bfloat16))
    with pytest.raises(ValueError):
        RsAddNormAgPlan(h, buf, torch.zeros(4, 64, dtype=torch.bfloat16), torch.ones(64, dtype=torch.bfloat16))


def test_expert_plans_validate_arguments(lib):
    from moe_comms_benchmarking_b200.ops.experts import (DispatchRouteFc1Plan, ExpertCombinePlan, Fc2CombinePlan,
                                                         GroupedGemmPlan, RouteBuffers, RoutePlan)
    h = _heap(8 << 20)
    T, K, E, H, I = 16, 4, 8, 256, 128
    route = RouteBuffers(T, K, E, "cpu")
    assert route.max_pairs == T * 4 and route.max_tiles == E + route.max_pairs // 128 + 1
    idx = torch.zeros(T, K, dtype=torch.int64)
    ntok = torch.zeros(1, dtype=torch.int32)
    rp = RoutePlan(route, idx, None, ntok, expert_begin=0)
    with pytest.raises(ValueError):
        RoutePlan(route, idx.int(), None, ntok, expert_begin=0)
    with pytest.raises(ValueError):
        RoutePlan(route, idx, None, ntok, expert_begin=0, grid=500)
    x = torch.zeros(T, H, dtype=torch.bfloat16)
    act = torch.zeros(route.max_pairs, I, dtype=torch.bfloat16)
    y = torch.zeros(route.max_pairs, H, dtype=torch.bfloat16)
    tmap = (None, 0)            # plans only store the tensor-map handle
    fc1 = GroupedGemmPlan(_ext.GEMM_FC1, tmap, route, x, act, 2 * I, H)
    fc2 = GroupedGemmPlan(_ext.GEMM_FC2, tmap, route, act, y, H, I)
    with pytest.raises(ValueError):      # A rows do not match k_total
        GroupedGemmPlan(_ext.GEMM_FC1, tmap, route, x, act, 2 * I, H * 2)
    with pytest.raises(ValueError):      # out has the wrong width
        GroupedGemmPlan(_ext.GEMM_FC2, tmap, route, act, act, H, I)
    with pytest.raises(ValueError):      # k_total not a multiple of 64
        GroupedGemmPlan(_ext.GEMM_FC2, tmap, route, torch.zeros(route.max_pairs, 96, dtype=torch.bfloat16), y, H, 96)
    partial = h.alloc("partial", [T, H], torch.bfloat16)
    meta = torch.zeros(4, dtype=torch.int32)
    out = torch.zeros(T, H, dtype=torch.bfloat16)
    comb = ExpertCombinePlan(h, y, route, partial, out, ntok, meta, T)
    with pytest.raises(ValueError):      # partial buffer smaller than the capacity
        ExpertCombinePlan(h, y, route, partial, out, ntok, meta, T * 2)
    Fc2CombinePlan(h, fc2, comb)
    with pytest.raises(ValueError):
        Fc2CombinePlan(h, fc1, comb)
    with pytest.raises(ValueError):      # all blocks must be resident at once
        Fc2CombinePlan(h, fc2, comb, grid=149)
    gh = h.alloc("gh2", [T, H], torch.bfloat16)
    agv = AllGatherVPlan(h, [gh], [x], ntok, meta, T)
    DispatchRouteFc1Plan(h, agv, rp, fc1)
    with pytest.raises(ValueError):
        DispatchRouteFc1Plan(h, agv, rp, fc2)


def test_layer_reads_ids_at_their_source_only_if_gathered():
    """The short cut of the layer kernel in a world of one: taken for the rows that the all-gather copies and counts, by
    address and row size, in any order of the tensors; refused for everything else."""
    from moe_comms_benchmarking_b200.ops.experts import RouteBuffers, RoutePlan, local_routing
    h = _heap(2 << 20)
    T, K, H = 8, 4, 256
    x, idx, w = torch.zeros(T, H, dtype=torch.bfloat16), torch.zeros(T, K, dtype=torch.int64), torch.zeros(T, K)
    gx, gi, gw = h.alloc("gx", [T, H], torch.bfloat16), h.alloc("gi", [T, K], torch.int64), h.alloc("gw", [T, K], torch.float32)
    n, meta = torch.zeros(1, dtype=torch.int32), torch.zeros(4, dtype=torch.int32)
    route = RouteBuffers(T, K, 8, "cpu")

    def found(dsts, srcs, ids, weights, count=meta):
        agv = AllGatherVPlan(h, dsts, srcs, n, meta, T)
        return local_routing(h, agv.args, RoutePlan(route, ids, weights, count, expert_begin=0).args)

    here = (idx.data_ptr(), w.data_ptr())
    assert found([gx, gi, gw], [x, idx, w], gi.tensor, gw.tensor, meta[0:1]) == here
    assert found([gw, gx, gi], [w, x, idx], gi.tensor, gw.tensor) == here
    assert found([gx, gi], [x, idx], gi.tensor, None) == (idx.data_ptr(), None)
    for ids, weights, count in ((idx.clone(), gw.tensor, meta), (gi.tensor, w.clone(), meta), (gi.tensor, gw.tensor, n)):
        assert found([gx, gi, gw], [x, idx, w], ids, weights, count) == (None, None)
    assert found([gx], [x], idx, w) == (None, None) and found([gx, gi], [x, idx], gi.tensor, gw.tensor) == (None, None)


def test_capability_checks():
    from moe_comms_benchmarking_b200 import ops
    assert not ops.is_device_multimem_capable("cpu") and not ops.is_device_tcgen05_capable("cpu")
    h = _heap(1 << 16)
    assert not ops.heap_has_multicast(h)
    assert ops.row_access_bytes(torch.zeros(4, 1024, dtype=torch.bfloat16)) == 16
    assert ops.row_access_bytes(torch.zeros(4, 22, dtype=torch.float32)) == 8      # 88-byte rows
    assert ops.row_access_bytes(torch.zeros(4, 3, dtype=torch.float32)) == 4
    assert ops.row_access_bytes(torch.zeros(4, 3, dtype=torch.uint8)) == 0
    assert ops.row_access_bytes(torch.zeros(4, 8, dtype=torch.float32).t()) == 0   # not contiguous
    assert ops.are_tensors_gather_eligible(torch.zeros(2, 22, dtype=torch.int64), torch.zeros(2, 22))
    assert not ops.are_tensors_gather_eligible()
    assert ops.are_tensors_reduce_eligible(torch.zeros(2, 1024, dtype=torch.bfloat16))
    assert not ops.are_tensors_reduce_eligible(torch.zeros(2, 22))                 # 88-byte rows
    assert not ops.are_tensors_reduce_eligible(torch.zeros(2, 8, dtype=torch.int32))


def test_step_plans_validate_arguments():
    """Host-side checks of the persistent step plans (dense and all-to-all): shapes, capacities,
    parity buffers, packet staging, fp8 tensor layout.  Nothing is launched."""
    from moe_comms_benchmarking_b200.ops.a2a import A2AStepBuffers, A2AStepPlan, a2a_meta_row_bytes
    from moe_comms_benchmarking_b200.ops.dense import (DenseStepPlan, agv_ll_stage_bytes, rsv_ll_stage_bytes,
                                                       step_credit_bytes)
    h = _heap(16 << 20)
    cap, H, K = 8, 256, 6
    n_local = torch.zeros(1, dtype=torch.int32)
    meta8 = torch.zeros(8, dtype=torch.int32)
    g2h = h.alloc("g2h", [2, cap, H], torch.bfloat16)
    g2r = h.alloc("g2r", [2, cap, K], torch.int64)
    rsv = h.alloc("rsv2", [cap, H], torch.bfloat16)
    src_h = torch.zeros(cap, H, dtype=torch.bfloat16)
    src_r = torch.zeros(cap, K, dtype=torch.int64)
    out = torch.zeros(cap, H, dtype=torch.bfloat16)
    p = DenseStepPlan(h, [g2h, g2r], [src_h, src_r], out, rsv, n_local, meta8, cap, 88)
    assert p.args.num_layers == 88 and p.args.dst_par_stride[0] == cap * H * 2 and p.args.ll_rows == 0
    with pytest.raises(ValueError):      # step_meta too short
        DenseStepPlan(h, [g2h], [src_h], out, rsv, n_local, torch.zeros(4, dtype=torch.int32), cap, 2)
    with pytest.raises(ValueError):      # gathered buffer without the parity dimension
        DenseStepPlan(h, [h.alloc("flat", [cap, H], torch.bfloat16)], [src_h], out, rsv, n_local, meta8, cap, 2)
    with pytest.raises(ValueError):      # pipeline groups need one block per SM
        DenseStepPlan(h, [g2h], [src_h], out, rsv, n_local, meta8, cap, 2, grid=296, groups=2)
    st_a = h.alloc("st_a", [agv_ll_stage_bytes(4, [H * 2, K * 8])], torch.uint8)
    st_r = h.alloc("st_r", [rsv_ll_stage_bytes(1, 4, cap, H * 2)], torch.uint8)
    with pytest.raises(ValueError):      # packet mode without its credit region
        DenseStepPlan(h, [g2h, g2r], [src_h, src_r], out, rsv, n_local, meta8, cap, 2, agv_ll_stage=st_a,
                      rsv_ll_stage=st_r, ll_rows=4)
    cr = h.alloc("cr", [step_credit_bytes(148)], torch.uint8)
    p = DenseStepPlan(h, [g2h, g2r], [src_h, src_r], out, rsv, n_local, meta8, cap, 2, agv_ll_stage=st_a,
                      rsv_ll_stage=st_r, ll_rows=4, credits=cr)
    assert p.args.ll_rows == 4 and p.args.credit_off == cr.offset
    # fp8 dispatch: uint8 rows + fp32 scales as a fourth tensor without a source
    q = h.alloc("q8", [2, cap, H], torch.uint8)
    sc = h.alloc("sc8", [2, cap, H // 128], torch.float32)
    g2p = h.alloc("g2p", [2, cap, K], torch.float32)
    src_p = torch.zeros(cap, K, dtype=torch.float32)
    p = DenseStepPlan(h, [q, g2r, g2p, sc], [src_h, src_r, src_p, None], out, rsv, n_local, meta8, cap, 2, fp8_hidden=H)
    assert p.args.fp8_hidden == H and p.args.row_bytes[0] == H and p.args.row_bytes[3] == H // 128 * 4 and p.args.src[3] is None
    with pytest.raises(ValueError):
        DenseStepPlan(h, [g2h, g2r, g2p, sc], [src_h, src_r, src_p, None], out, rsv, n_local, meta8, cap, 2, fp8_hidden=H)
    # all-to-all step
    assert a2a_meta_row_bytes(22) == 192 and a2a_meta_row_bytes(8) == 80
    for fp8 in (False, True):
        b = A2AStepBuffers(h, cap, H, K, fp8, prefix=f"t{int(fp8)}")
        assert b.recv_meta.tensor.shape == (2, 1, cap, a2a_meta_row_bytes(K))
        p = A2AStepPlan(h, b, src_h, src_r, src_p, out, n_local, meta8, 16, 88)
        assert p.args.x_par_stride == b.recv_x.nbytes // 2 and p.args.fp8 == int(fp8) and p.args.meta_row_bytes == 64
        assert (p.args.y_off == p.args.recv_x_off) == (not fp8)
        with pytest.raises(ValueError):
            A2AStepPlan(h, b, src_h[:4], src_r, src_p, out, n_local, meta8, 16, 88)
    st, tok, ids, wts = b.meta_fields(0, 0, 3)
    assert st.shape == (3,) and ids.shape == (3, K) and wts.dtype == torch.float32


def test_step_on_its_own_rows_keeps_its_order(lib):
    """A step of a world of one whose output lies on a source, or whose partial sums lie on gathered rows, is marked to keep
    the order of its layers; one on buffers of its own, next to one another even, is not."""
    from moe_comms_benchmarking_b200.ops.dense import DenseStepPlan
    h = _heap(4 << 20)
    cap, H, K = 8, 256, 6
    n_local, meta = torch.zeros(1, dtype=torch.int32), torch.zeros(8, dtype=torch.int32)
    gh, gr = h.alloc("gh", [2, cap, H], torch.bfloat16), h.alloc("gr", [2, cap, K], torch.int64)
    q, gp, sc = h.alloc("q", [2, cap, H], torch.uint8), h.alloc("gp", [2, cap, K], torch.float32), h.alloc("sc", [2, cap, 2], torch.float32)
    rsv = h.alloc("rsv", [cap, H], torch.bfloat16)
    both = torch.zeros(2 * cap, H, dtype=torch.bfloat16)
    x, ids, p = both[:cap], torch.zeros(cap, K, dtype=torch.int64), torch.zeros(cap, K)

    def marked(out, sums=rsv, fp8=False):
        dsts, srcs = ([q, gr, gp, sc], [x, ids, p, None]) if fp8 else ([gh, gr], [x, ids])
        plan = DenseStepPlan(h, dsts, srcs, out, sums, n_local, meta, cap, 4, fp8_hidden=H if fp8 else 0)
        return lib.mcb_dense_step_in_order(C.byref(h.ctx()), C.byref(plan.args))

    assert marked(both[cap:]) == 0 and marked(both[cap:], fp8=True) == 0
    assert marked(x) == 1 and marked(both[1:cap + 1]) == 1 and marked(x, fp8=True) == 1      # all rows, all but one, fp8
    assert marked(both[cap - 1:2 * cap - 1], fp8=True) == 1                                  # the last bf16 row of an fp8 source
    assert marked(both[cap:], gh) == 1 and marked(gh.tensor[1]) == 1 and marked(rsv.tensor) == 1


def test_step_that_gathers_twice_to_one_place_keeps_its_order(lib):
    """Gathered tensors that share rows, in either parity, are written in turn; ones whose parities lie between one another's are apart."""
    from moe_comms_benchmarking_b200.ops.dense import DenseStepPlan
    h = _heap(4 << 20)
    cap, H = 8, 256
    rows = cap * H * 2
    n_local, meta = torch.zeros(1, dtype=torch.int32), torch.zeros(8, dtype=torch.int32)
    a, b, rsv = h.alloc("a", [2, cap, H], torch.bfloat16), h.alloc("b", [2, cap, H], torch.bfloat16), h.alloc("r", [cap, H], torch.bfloat16)
    x, out = torch.zeros(cap, H, dtype=torch.bfloat16), torch.zeros(cap, H, dtype=torch.bfloat16)
    plan = DenseStepPlan(h, [a, b], [x, torch.zeros_like(x)], out, rsv, n_local, meta, cap, 4)

    def marked(off_a, stride_a, off_b, stride_b):
        for t, (off, stride) in enumerate(((off_a, stride_a), (off_b, stride_b))):
            plan.args.dst_off[t], plan.args.dst_par_stride[t] = a.offset + off, stride
        return lib.mcb_dense_step_in_order(C.byref(h.ctx()), C.byref(plan.args))

    assert marked(0, rows, 2 * rows, rows) == 0 and marked(0, 2 * rows, rows, 2 * rows) == 0
    assert marked(0, rows, 0, rows) == 1 and marked(0, rows, rows, rows) == 1 and marked(rows, rows, 0, rows) == 1
    assert marked(0, rows, 2 * rows - 16, rows) == 1


def test_weight_tile_packing_round_trip():
    """The pre-packed weight layout: tile (row block, column block) is 16 KB of contiguous memory in the
    swizzled K-major shared-memory image; packing and unpacking are inverse, and chunk c of row r of a
    tile sits at chunk position c ^ (r % 8)."""
    from moe_comms_benchmarking_b200.ops.experts import ExpertWeights, pack_weight_tiles, unpack_weight_tiles
    w = torch.randn(3, 256, 192).to(torch.bfloat16)
    p = pack_weight_tiles(w)
    assert p.shape == (3, 2, 3, 128, 64) and p.is_contiguous()
    assert torch.equal(unpack_weight_tiles(p), w)
    for (e, rb, kb, r, c) in ((0, 0, 0, 0, 0), (1, 1, 2, 5, 3), (2, 0, 1, 127, 7), (2, 1, 0, 9, 6)):
        pos = c ^ (r % 8)
        assert torch.equal(p[e, rb, kb, r, pos * 8:pos * 8 + 8], w[e, rb * 128 + r, kb * 64 + c * 8:kb * 64 + c * 8 + 8])
    split = torch.arange(2 * 8 * 4, dtype=torch.float32).view(2, 8, 4)
    il = ExpertWeights.interleave(split)
    assert torch.equal(il[:, 0::2], split[:, :4]) and torch.equal(il[:, 1::2], split[:, 4:])
    with pytest.raises(ValueError):
        pack_weight_tiles(torch.zeros(1, 100, 64, dtype=torch.bfloat16))


def _step_args(act=1 << 32, y=2 << 32, out=3 << 32):
    """Argument blocks of two layers over buffers at made-up addresses: 16 rows of 256 values, 2 experts per token, 128 activations."""
    from moe_comms_benchmarking_b200.ops.experts import _aligned_layer_args
    cap, K, H = 16, 2, 256
    raw, addr, stride = _aligned_layer_args(2)
    meta = _ext.McbMetaArgs()
    meta.n_local, meta.step_meta, meta.cap = 0x1000, 0x1100, cap
    for s in range(2):
        p = _ext.McbLayerArgs.from_address(addr + s * stride)
        p.ctx.world, p.ctx.heap_local = 1, 4 << 32
        g, r, f, c = p.agv, p.route, p.ffn, p.cmb
        g.num_tensors, g.cap, g.n_local, g.step_meta = 3, cap, 0x1000, 0x1100
        for t, nbytes in enumerate((2 * H, 8 * K, 4 * K)):
            g.src[t], g.dst_off[t], g.row_bytes[t] = (5 + t) << 32, t << 20, nbytes
        r.num_local_experts, r.topk, r.max_tokens, r.max_pairs, r.num_tokens = 4, K, cap, cap * K, 0x1100
        r.pair_token, r.pair_prob, r.pair_pos, r.expert_offset, r.ffn_done = 0x2000, 0x3000, 0x4000, 0x5000, 0x6000
        f.x, f.pair_token, f.pair_prob, f.expert_offset, f.ffn_done = 4 << 32, 0x2000, 0x3000, 0x5000, 0x6000
        f.act, f.y, f.num_local_experts, f.hidden, f.intermediate, f.w1 = act, y, 4, H, 128, 0x7000 + s
        c.y, c.pair_pos, c.topk, c.hidden, c.cap, c.out, c.n_local, c.step_meta = y, 0x4000, K, H, cap, out, 0x1000, 0x1100
        p.local_ids, p.local_probs = g.src[1], g.src[2]
    return raw, addr, meta


def test_step_joins_only_layers_that_keep_apart(lib):
    """Layers share a launch where none writes what another one reads or writes: activations (8 KB), expert outputs (16 KB) and combined
    rows (8 KB) apart from one another, from the gathered rows and from their sources."""
    def joins(**at):
        raw, addr, meta = _step_args(**at)
        return lib.mcb_moe_step_joins(addr, 2, C.addressof(meta))
    act, y, rows, src = 1 << 32, 2 << 32, 4 << 32, 5 << 32
    assert joins() == 1 and joins(out=act + 8192) == 1 and joins(y=act + 8192, out=act + 8192 + 16384) == 1
    for out in (act, act + 8176, act - 8176, y, y + 16368, rows, rows + 8176, rows + (1 << 20), src, src + 8176, 6 << 32):
        assert joins(out=out) == 0, hex(out)
    for at in (act, act + 8176, act - 16368, rows, src):
        assert joins(y=at) == 0, hex(at)
    raw, addr, meta = _step_args()
    meta.cap = 17
    assert lib.mcb_moe_step_joins(addr, 2, C.addressof(meta)) == 0


def test_launcher_follows_context_grid_and_stream(monkeypatch):
    """The kept block of a plan's launches names the heap's present context, grid, threads and PDL, and errors are raised."""
    import types
    from moe_comms_benchmarking_b200.ops import _ext
    seen, err = [], 0

    def launch(addr, stream):
        b = _ext.McbLaunch.from_address(addr)
        seen.append((b.ctx, b.args, b.op, b.grid, b.threads, b.pdl, stream))
        return err

    monkeypatch.setattr(_ext, "_lib", types.SimpleNamespace(mcb_launch=launch, mcb_error_string=lambda e: b"refused"))
    monkeypatch.setattr(_ext, "_current_raw_stream", lambda: 7)
    one, two, args = _ext.McbCtx(), _ext.McbCtx(), _ext.McbAgvArgs()
    heap = types.SimpleNamespace(ctx=lambda: one)
    go = _ext.Launcher(_ext.OP_AGV, args, "all_gather_v")
    at = lambda c: C.addressof(c)
    go(heap, 148, 512, False)
    go(heap, 148, 512, True, types.SimpleNamespace(cuda_stream=9))
    go(heap, 16, 512, True)
    heap.ctx = lambda: two
    go(heap, 16, 64, True)
    assert seen == [(at(one), at(args), _ext.OP_AGV, 148, 512, 0, 7), (at(one), at(args), _ext.OP_AGV, 148, 512, 1, 9),
                    (at(one), at(args), _ext.OP_AGV, 16, 512, 1, 7), (at(two), at(args), _ext.OP_AGV, 16, 64, 1, 7)]
    err = 1
    with pytest.raises(_ext.CudaLaunchError, match="all_gather_v"):
        go(heap, 16, 64, True)


def test_operation_numbers_are_the_librarys(lib, monkeypatch):
    """Loading refuses a library that numbers the operations otherwise, and a launch of none of them is an error."""
    from moe_comms_benchmarking_b200.ops import _ext
    assert [lib.mcb_op_name(op).decode() for op in range(len(_ext.OPS))] == list(_ext.OPS)
    for op in (-1, len(_ext.OPS)):
        assert lib.mcb_op_name(op) is None
        assert lib.mcb_launch(C.addressof(_ext.McbLaunch(op=op, grid=1, threads=32)), 0) != 0
    for ops in (_ext.OPS[:-1], _ext.OPS[1::-1] + _ext.OPS[2:]):         # one less than in the library; two the other way round
        with monkeypatch.context() as m:
            m.setattr(_ext, "_lib", None)
            m.setattr(_ext, "OPS", ops)
            with pytest.raises(_ext.ExtensionMissing, match="operation drift"):
                _ext.load()
    assert _ext.load() is lib


def test_route_grid_is_the_most_blocks():
    """A routing launch takes as many blocks as the caller asks for, fewer only where the device holds fewer at once; wider blocks where few have many entries."""
    lib = _ext.load()
    assert [lib.mcb_route_blocks(g, 592) for g in (1, 2, 32, 96, 128)] == [1, 2, 32, 96, 128]
    assert [lib.mcb_route_blocks(g, 72) for g in (1, 72, 73, 128)] == [1, 72, 72, 72]
    assert [lib.mcb_route_blocks(g, 592) for g in (-1, 0, 129)] == [0, 0, 0]
    threads = lambda entries, g: lib.mcb_route_threads(C.byref(_ext.McbRouteArgs(max_tokens=entries, topk=1)), g)
    assert [threads(n, 2) for n in (1, 4096, 4097)] == [512, 512, 1024]
    assert threads(1 << 20, 95) == 1024 and threads(1 << 20, 96) == threads(1 << 20, 128) == 512
