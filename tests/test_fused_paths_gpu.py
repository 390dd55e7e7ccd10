"""Fused epilogues, the expert shares of the MoE layer and the fp32 chain, at the sizes where they can go wrong."""
import pytest
import torch

import maco_b200 as maco
from maco_b200 import _native, ops

pytestmark = pytest.mark.gpu
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}      # half a unit in the last place, relative


def _gelu(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,pair", [(1, 128, 64, False), (130, 264, 128, False), (257, 520, 192, True), (128, 256, 64, True), (300, 136, 64, False)])
def test_gelu_dual_writes_the_product_and_the_gelu_of_what_it_wrote(dtype, m, n, k, pair):
    torch.manual_seed(m * n)
    a, b = torch.randn(m, k, device="cuda", dtype=dtype), torch.randn(n, k, device="cuda", dtype=dtype)
    z, act = torch.empty(m, n, device="cuda", dtype=dtype), torch.empty(m, n, device="cuda", dtype=dtype)
    ops.gemm(a, b, out=z, aux=act, epilogue="gelu_dual", cta_pair=pair)
    plain = ops.gemm(a, b, cta_pair=pair)
    assert torch.equal(z, plain)
    ref = _gelu(z.double())
    # one rounding to 16 bits, and fp32 arithmetic whose cancellation in the left tail stays far below |z| ulp
    assert ((act.double() - ref).abs() <= EPS[dtype] * ref.abs() * 1.01 + 1e-6 * z.double().abs() + 1e-7).all()
    with pytest.raises(ValueError):
        ops.gemm(a, b, out=z, epilogue="gelu_dual")
    with pytest.raises(ValueError):
        ops.gemm(a.float(), b.float(), aux=act, epilogue="gelu_dual")


@pytest.mark.parametrize("n", [264, 512])            # a ragged last tile, whole tiles
@pytest.mark.parametrize("pair", [False, True])
def test_gelu_backward_epilogue_takes_whole_and_ragged_tiles(n, pair):
    dt = torch.bfloat16
    a, b = torch.randn(200, 128, device="cuda", dtype=dt), torch.randn(n, 128, device="cuda", dtype=dt)
    z = (torch.randn(200, n, device="cuda") * 3).to(dt)
    z[0, :4] = torch.tensor([12.0, -12.0, 300.0, -300.0])
    out = ops.gemm(a, b, aux=z, epilogue="gelu_bwd", cta_pair=pair)
    zd = z.double().requires_grad_(True)
    _gelu(zd).sum().backward()
    prod = a.double() @ b.double().t()
    ref = prod * zd.grad
    # a product of 128 terms in fp32 (relative to the sum of magnitudes), a derivative of about 1e-6 absolute error, one rounding
    mag = a.double().abs() @ b.double().abs().t()
    assert ((out.double() - ref).abs() <= EPS[dt] * ref.abs() * 1.01 + 1e-5 * mag).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [8, 1000, 8 * 1031])   # less than one vector per thread, a ragged last block
def test_mse_gelu_bwd(dtype, n):
    a, t, z = (torch.randn(n, device="cuda", dtype=dtype) * 2 for _ in range(3))
    out = ops.mse_gelu_bwd(a, t, z, torch.empty_like(a), 0.125)
    zd = z.double().requires_grad_(True)
    _gelu(zd).sum().backward()
    ref = 0.125 * (a.double() - t.double()) * zd.grad
    assert ((out.double() - ref).abs() <= EPS[dtype] * ref.abs() * 1.01 + 2e-6 * (a.double() - t.double()).abs() + 6e-8).all()
    with pytest.raises(ValueError):
        ops.mse_gelu_bwd(a, t, z.float(), torch.empty_like(a), 1.0)
    if n == 1000:
        with pytest.raises(RuntimeError):            # not a whole number of vectors
            ops.mse_gelu_bwd(a[:9], t[:9], z[:9], torch.empty_like(a[:9]), 1.0)


@pytest.mark.parametrize("rows,hidden,ffn", [(130, 256, 256), (1003, 512, 384), (300, 2048, 1536), (513, 264, 256)])
def test_residual_add_in_the_epilogue_is_the_add(rows, hidden, ffn):
    """Both outputs as if the add were a node of its own: the sum is exactly the rounded product plus x, rounded."""
    dt = torch.float16
    x, w = torch.randn(rows, hidden, device="cuda", dtype=dt), torch.randn(ffn, hidden, device="cuda", dtype=dt) * 0.05
    w2 = torch.randn(hidden, ffn, device="cuda", dtype=dt) * 0.05
    g = maco.TaskGraph()
    y = g.linear(g.linear(x, w).output, w2)
    s = g.add(y.output, x)
    t = g.add(x, s.output)                            # its other operand is written by the graph: stays a node of its own
    g.compile()
    for _ in range(2):
        g.execute()
    torch.cuda.synchronize()
    # one add in the product's epilogue and one as tasks of its own: as many as a graph with that add alone has
    alone = maco.TaskGraph()
    alone.add(x, torch.empty_like(x))
    alone.compile()
    assert g.runtime_kind == alone.runtime_kind == "persistent"
    kinds = g._runtime._program.task_types
    assert (kinds == 113).sum() == (alone._runtime._program.task_types == 113).sum() > 0
    h = (x.float() @ w.float().t()).to(dt).float()
    assert (y.output.float() - h @ w2.float().t()).abs().max() < 2e-2 * h.abs().max()
    assert torch.equal(s.output, (y.output.float() + x.float()).to(dt))
    assert torch.equal(t.output, (x.float() + s.output.float()).to(dt))
    assert _native.status() == 0


@pytest.mark.parametrize("experts,top_k,tokens,hidden,inter,factor,std", [
    (8, 8, 128, 256, 128, 1.0, 0.5),                  # every expert takes every token: exactly full slabs
    (64, 1, 128, 256, 128, 64.0, 3.0),                # most experts without a token
    (16, 4, 640, 768, 384, 4.0, 0.3),                 # ragged row blocks
    (256, 2, 256, 256, 128, 64.0, 0.5),               # the largest table of slabs
    (8, 2, 4736, 256, 128, 3.0, 0.3),                 # more tokens per task than one batch of 32
])
def test_expert_shares_over_counts(experts, top_k, tokens, hidden, inter, factor, std):
    from maco_b200.models.moe_layer import MoEEPLayer
    kw = dict(hidden=hidden, experts=experts, top_k=top_k, inter=inter, tokens=tokens, capacity_factor=factor, seed=5, weight_std=0.05, router_std=std)
    layer = MoEEPLayer(**kw)
    x = torch.randn(tokens, hidden, device="cuda", dtype=torch.bfloat16)
    outs = []
    for _ in range(3):
        outs.append(layer(x).clone())
        assert layer.dropped() == 0
    tiles = MoEEPLayer(**kw, fused_return=False)      # a task per tile of every slab
    ref = tiles(x)
    assert tiles.dropped() == 0
    torch.cuda.synchronize()
    # same operands, same roundings; SwiGLU's division may round an activation differently once in a while
    assert (outs[0].float() - ref.float()).norm() <= 2e-3 * ref.float().norm()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert not layer.counts.any() and not layer.ready.any()
    assert _native.status() == 0


def test_routing_takes_the_lower_expert_on_equal_logits_and_zero_is_zero():
    from maco_b200.models.moe_layer import MoEEPLayer
    layer = MoEEPLayer(hidden=256, experts=16, top_k=4, inter=128, tokens=128, capacity_factor=16.0, seed=1)
    layer.w_router.zero_()
    layer.w_router[3] = -0.0
    x = torch.randn(128, 256, device="cuda", dtype=torch.bfloat16)
    out = layer(x)
    torch.cuda.synchronize()
    ref = layer.reference(x)                          # all logits are 0 or -0: experts 0 to 3, weight 1/4 each
    assert (out.float() - ref).abs().max() < 4e-2 * max(1.0, ref.abs().max().item())


def test_fp32_chain_follows_its_tensors():
    g = maco.TaskGraph()
    x, w1 = torch.randn(7, 96, device="cuda"), torch.randn(130, 200, device="cuda")[:, 3:99]        # strided, not 16-byte aligned
    b1, w2 = torch.randn(130, device="cuda"), torch.randn(130, 40, device="cuda")
    a = g.linear(x, w1, b1, activation="silu")
    c = g.matmul(a.output, w2)
    g.compile()
    assert g.runtime_kind == "stream"

    def check():
        h = torch.nn.functional.silu(x.double() @ w1.double().t() + b1.double())
        # fp32 sums of 130 terms
        assert (c.output.double() - h @ w2.double()).abs().max() <= 1e-5 * (h.abs() @ w2.double().abs()).max()

    g.execute()
    check()
    assert g._runtime._chain is not None
    x.copy_(torch.randn_like(x))
    w2.data = torch.randn(130, 40, device="cuda")     # moves: the graph reads the new weight at once, then in a chain again
    for _ in range(2):
        g.execute()
        check()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g.execute(stream=s)
    s.synchronize()
    check()
    maco.config.allow_tf32, old = True, maco.config.allow_tf32
    try:
        assert g._runtime._f32_chain(g._schedule) is None
    finally:
        maco.config.allow_tf32 = old
