"""Expert layers at counts, types and routes where routing and the expert shares can go wrong."""
import pytest
import torch


def _plan(**kw):
    from maco_b200.models.moe_layer import MoEEPLayer
    from maco_b200.parallel.symm_heap import PlanningHeap
    return MoEEPLayer(device=torch.device("cpu"), heap=PlanningHeap(0, 1, 1 << 26), **kw)


@pytest.mark.parametrize("experts", [1, 2, 3, 5, 7, 8, 9, 12, 20, 64, 255])
def test_router_rows_are_whole_vectors(experts):
    """The router's tail stores 16-byte vectors of 8 logits and routing reads two logits at a time, up to the last odd one: all of
    them aligned, inside the allocation, and the kernel told the row length that the tensor has."""
    import struct
    layer = _plan(hidden=256, experts=experts, top_k=1, inter=128, tokens=128, capacity_factor=1.0)
    ld = layer.logits.stride(0)
    assert layer.logits.shape == (128, experts) and ld % 8 == 0 and layer.logits.data_ptr() % 16 == 0
    assert layer.logits.storage_offset() == 0
    last = layer.logits.untyped_storage().nbytes() // 2
    for t in range(128):
        for e in range(0, experts, 2):
            assert (t * ld + e) % 2 == 0 and t * ld + e + 1 < last
    words = struct.unpack("<QQQQQQQQQiiiiiiii", layer.d_params.numpy().tobytes())
    assert words[0] == layer.logits.data_ptr() and words[-1] == ld


@pytest.mark.parametrize("world", [1, 2])
def test_rows_for_other_ranks_leave_through_the_bulk_engine(world):
    """Expert shares store their rows from registers, which is for this GPU's memory alone: with more ranks the down projection is tiles
    with a destination rank, whose epilogue stages its rows, and each of them signals that rank."""
    from maco_b200.models.moe_layer import MoEEPLayer
    from maco_b200.ops import megakernel as mk
    from maco_b200.parallel.symm_heap import PlanningHeap
    layer = MoEEPLayer(hidden=256, experts=8, top_k=2, inter=128, tokens=256, rank=0, world=world, heap=PlanningHeap(0, world, 1 << 26),
                       device=torch.device("cpu"), capacity_factor=4.0)
    shares = [t for t in layer.builder.tasks if t["type"] == mk.T_MOE_EXPERTS]
    assert (len(shares) > 0) == (world == 1)
    if world > 1:
        to = {t["signal_peer"] for t in layer.builder.tasks if t["type"] in (100, 101, 102) and t["signal_peer_event"] >= 0}
        assert to == set(range(world))


def test_makespan_of_an_expert_layer_follows_its_tiles():
    """Twice the experts' width is about twice the tiles: the estimate of the launch grows by as much as a share does."""
    from maco_b200.ops import megakernel as mk
    spans, shares = [], []
    for inter in (256, 512):
        b = _plan(hidden=256, experts=8, top_k=2, inter=inter, tokens=1024, capacity_factor=2.0).builder
        costs = {mk.default_task_cost(t) for t in b.tasks if t["type"] == mk.T_MOE_EXPERTS}
        assert len(costs) == 1
        # 8 slabs of 256 rows: 16 row blocks; inter / 128 gate tiles of 4 k-blocks and one down tile of inter / 64 each
        want = 16 * (inter // 128 * (2 + 0.45 * 4) + 1 * (2 + 0.45 * (inter // 64))) / b.num_workers
        assert costs.pop() == pytest.approx(want)
        shares.append(want)
        r = mk.estimate_makespan([(b.tasks, mk.assign_static_queues(b.tasks, b.num_workers, b.num_comm_workers))])
        spans.append(r["span_us"][0])
    assert spans[1] - spans[0] == pytest.approx(shares[1] - shares[0])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["static", "dynamic"])
@pytest.mark.parametrize("experts,top_k", [(1, 1), (3, 2), (5, 5), (12, 4), (31, 8)])
def test_any_number_of_experts(experts, top_k, mode):
    from maco_b200 import _native
    from maco_b200.models.moe_layer import MoEEPLayer
    layer = MoEEPLayer(hidden=256, experts=experts, top_k=top_k, inter=128, tokens=256, capacity_factor=float(experts), seed=3, mode=mode,
                       weight_std=0.05, router_std=0.5)
    x = torch.randn(256, 256, device="cuda", dtype=torch.bfloat16)
    ref = layer.reference(x)
    for _ in range(2):
        out = layer(x)
        torch.cuda.synchronize()
        assert layer.dropped() == 0
        # the bound of the single-GPU layer test: bf16 activations, and a token whose logits tie may take another expert
        assert (out.float() - ref).abs().max().item() < 4e-2 * max(1.0, ref.abs().max().item())
    # the router's rows, the ragged last vector among them: fp32 sums of 256 terms, rounded once
    logits = x.float() @ layer.w_router.float().t()
    assert ((layer.logits.float() - logits).abs() <= 2.0 ** -8 * logits.abs() * 1.01 + 1e-3).all()
    assert _native.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode,fused_return", [("static", True), ("static", False), ("dynamic", True)])
def test_routed_and_received_counts_of_a_step(mode, fused_return):
    """What a step routed to each expert, beyond a slab's capacity too, and what the slabs received, by a recount of the logits."""
    from maco_b200.models.moe_layer import MoEEPLayer
    layer = MoEEPLayer(hidden=256, experts=12, top_k=3, inter=128, tokens=1024, capacity_factor=0.5, seed=11, weight_std=0.05, router_std=2.0,
                       mode=mode, fused_return=fused_return, on_drop="ignore")
    for seed in (1, 2):
        layer(torch.randn(1024, 256, generator=torch.Generator("cuda").manual_seed(seed), device="cuda", dtype=torch.bfloat16))
        idx = torch.sort(layer.logits.float(), dim=-1, descending=True, stable=True)[1][:, :3]
        load = torch.bincount(idx.flatten(), minlength=12)
        assert (load > layer.capacity).any()
        assert torch.equal(layer.routed.long(), load)
        assert torch.equal(layer.cnt.view(-1).long(), load.clamp(max=layer.capacity))
        assert layer.dropped() == int((load - layer.capacity).clamp(min=0).sum())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mode,fused_return", [("static", True), ("static", False), ("dynamic", True)])
def test_expert_layer_in_both_types_against_its_own_logits(dtype, mode, fused_return):
    """fp16 and bf16 on all three routes, positive, negative, tied and zero logits among them, against routing and experts in plain torch
    from the logits that the router wrote: no token may take another expert."""
    from maco_b200 import _native
    from maco_b200.models.moe_layer import MoEEPLayer
    E, K, H, I, T = 16, 4, 256, 128, 256
    layer = MoEEPLayer(hidden=H, experts=E, top_k=K, inter=I, tokens=T, capacity_factor=4.0, seed=3, mode=mode, dtype=dtype, weight_std=0.05,
                       router_std=0.3, fused_return=fused_return)
    layer.w_router[5].copy_(layer.w_router[2])       # equal logits: the lower expert goes first
    layer.w_router[7].zero_()
    x = torch.randn(T, H, device="cuda", dtype=dtype)
    out = layer(x)
    assert layer.dropped() == 0
    val, idx = torch.sort(layer.logits.float(), dim=-1, descending=True, stable=True)
    weight, idx = torch.softmax(val[:, :K].double(), dim=-1), idx[:, :K]
    rnd = lambda t: t.to(dtype).double()
    ref = torch.zeros(T, H, device="cuda", dtype=torch.float64)
    for e in range(E):
        tok, k = (idx == e).nonzero(as_tuple=True)
        wg, wu, wd = (w.double() for w in layer.expert_weights(e))
        xe = x[tok].double()
        h = rnd(torch.nn.functional.silu(xe @ wg.t()) * (xe @ wu.t()))
        ref.index_add_(0, tok, rnd(rnd(h @ wd.t()) * weight[tok, k].unsqueeze(1)))
    # what is rounded, activations, expert outputs, weighted rows and the sum, is rounded alike on both sides but for fp32 sums near a
    # tie: a few units of the type's half ulp in norm, where another expert would show as a difference of the size of the output
    half = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert (out.double() - ref).norm() <= 2 * half * ref.norm()
    assert ((out.double() - ref).norm(dim=1) <= 8 * half * ref.norm(dim=1) + half).all()
    assert _native.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_slabs_around_a_row_block(dtype):
    """Slabs of a few rows store from registers, of a whole row block through shared memory, warps without rows not at all: no row, one, a
    warp's 32 less and more one, a row block's 128 less and more one. The router sends token t where it is told to."""
    from maco_b200 import _native
    from maco_b200.models.moe_layer import MoEEPLayer
    counts = [0, 1, 31, 33, 127, 128, 129, 63]
    E, H, I, T = len(counts), 256, 128, sum(counts)
    layer = MoEEPLayer(hidden=H, experts=E, top_k=1, inter=I, tokens=T, capacity_factor=4.0, seed=3, dtype=dtype, weight_std=0.05)
    layer.w_router.copy_(4.0 * torch.eye(E, H, device="cuda"))
    g = torch.Generator("cuda").manual_seed(5)
    to = torch.cat([torch.full((n,), e, device="cuda") for e, n in enumerate(counts)])[torch.randperm(T, generator=g, device="cuda")]
    x = torch.randn(T, H, device="cuda", generator=g)
    x[:, :E] = torch.nn.functional.one_hot(to, E).float()
    x = x.to(dtype)
    rnd = lambda t: t.to(dtype).double()
    half = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for _ in range(2):
        out = layer(x)
        assert layer.cnt.view(-1).tolist() == counts and layer.dropped() == 0
        for e in range(E):
            wg, wu, wd = (w.double() for w in layer.expert_weights(e))
            xe = x[to == e].double()
            ref = rnd(rnd(torch.nn.functional.silu(xe @ wg.t()) * (xe @ wu.t())) @ wd.t())
            # rounded alike on both sides but for fp32 sums near a tie, in the activations and in the result (routing weight 1)
            assert ((out[to == e].double() - ref).norm(dim=1) <= 4 * half * ref.norm(dim=1)).all()
    assert _native.status() == 0
