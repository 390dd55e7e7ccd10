"""GEMM epilogues that walk over a tile in steps of 16 columns: ragged last rows, both tile widths and forms, every operator, stand-alone and
in a graph, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F = torch.nn.functional


def _operands(M, N, K, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    return x, w, g, x.double() @ w.double().t()


def _close(got, want, dtype, slack=0.0):
    # one rounding to the output type, and a fast exponential or sums of K products in fp32 (a few 2^-20) in front of it
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10, torch.float32: 2.0 ** -18}[dtype]
    assert ((got.double() - want).abs() <= eps * want.abs() + 2.0 ** -16 + slack).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 32, 97, 129, 300])
@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("pair", [False, True])
def test_standalone(dtype, M, bn, pair):
    from maco_b200 import ops
    N, K = 512, 192
    x, w, g, z = _operands(M, N, K, dtype, M)
    bias = torch.randn(N, device="cuda", generator=g)
    kw = dict(bn=bn, cta_pair=pair)
    _close(ops.gemm(x, w, bias=bias, **kw), z + bias.double(), dtype)
    _close(ops.gemm(x, w, bias=bias.to(dtype), epilogue="gelu", **kw), F.gelu(z + bias.to(dtype).double(), approximate="tanh"), dtype)
    _close(ops.gemm(x, w, epilogue="silu", **kw), F.silu(z), dtype)
    _close(ops.gemm(x, w, epilogue="f32", **kw), z, torch.float32)
    _close(ops.gemm(x, w, bias=bias, epilogue="f32", alpha=0.5, **kw), 0.5 * z + bias.double(), torch.float32)
    aux = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    a = aux.double().requires_grad_(True)
    F.gelu(a, approximate="tanh").sum().backward()
    _close(ops.gemm(x, w, epilogue="gelu_bwd", aux=aux, **kw), z * a.grad, dtype, slack=2.0 ** -14)
    act = torch.empty(M, N, device="cuda", dtype=dtype)
    out = ops.gemm(x, w, epilogue="gelu_dual", aux=act, **kw)
    _close(out, z, dtype)
    _close(act, F.gelu(out.double(), approximate="tanh"), dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N", [(97, 1024), (300, 512), (1000, 4096), (2049, 2048)])
def test_graph(dtype, M, N):
    import maco_b200 as maco
    x, w, g, z = _operands(M, N, 320, dtype, N)
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    r = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    for bias_, act in ((bias, None), (None, "gelu"), (bias, "silu")):
        graph = maco.TaskGraph()
        y = graph.linear(x, w, bias=bias_, activation=act) if act else graph.linear(x, w, bias=bias_)
        graph.compile()
        graph.execute()
        v = z if bias_ is None else z + bias_.double()
        _close(y.output, F.gelu(v, approximate="tanh") if act == "gelu" else F.silu(v) if act == "silu" else v, dtype)
    graph = maco.TaskGraph()
    y = graph.linear(x, w)
    s = graph.add(y.output, r)
    graph.compile()
    for _ in range(2):
        graph.execute()
    _close(y.output, z, dtype)
    _close(s.output, y.output.double() + r.double(), dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N", [32, 64, 96, 160, 288, 40, 264])       # whole steps of 32 columns, and not
@pytest.mark.parametrize("M", [129, 640])
def test_graph_tiles_that_end_early(dtype, N, M):
    import maco_b200 as maco
    x, w, _, z = _operands(M, N, 320, dtype, N)
    graph = maco.TaskGraph()
    y = graph.linear(x, w)
    graph.compile()
    y.output.fill_(7.0)
    graph.execute()
    _close(y.output, z, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N", [16, 32, 144, 272, 40, 264])           # whole steps of 16 columns, and not
@pytest.mark.parametrize("M", [1, 129, 640])
def test_bias_on_tiles_that_end_early(dtype, N, M):
    import maco_b200 as maco
    from maco_b200 import ops
    x, w, g, z = _operands(M, N, 320, dtype, N)
    bias = torch.randn(N, device="cuda", generator=g)
    for b in (bias, bias.to(dtype)):
        _close(ops.gemm(x, w, bias=b), z + b.double(), dtype)
    graph = maco.TaskGraph()
    y = graph.linear(x, w, bias=bias.to(dtype))
    graph.compile()
    y.output.fill_(7.0)
    graph.execute()
    _close(y.output, z + bias.to(dtype).double(), dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N", [264, 520, 1032])
@pytest.mark.parametrize("act", [None, "gelu", "silu"])
def test_both_epilogues_of_one_product_agree(dtype, N, act):
    """The last 8 columns, a tile of their own, go through the general epilogue, the others through the one in steps: equal weight rows, biases
    and scales of 1 to 100 give equal bits."""
    import maco_b200 as maco
    from maco_b200 import ops
    x, w, g, _ = _operands(300, 8, 320, dtype, N)
    w, x = w.repeat(N // 8, 1), (x * torch.logspace(0, 2, 300, device="cuda")[:, None]).to(dtype)
    bias = torch.randn(8, device="cuda", generator=g).to(dtype).repeat(N // 8)
    graph = maco.TaskGraph()
    y = graph.linear(x, w, bias=bias, activation=act) if act else graph.linear(x, w, bias=bias)
    graph.compile()
    graph.execute()
    for out in (y.output, ops.gemm(x, w, bias=bias, epilogue=act)):
        cols = out.view(300, N // 8, 8)
        assert torch.equal(cols, cols[:, -1:].expand_as(cols))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N", [8, 200, 264, 640])                    # last column chunks of 8 columns and whole ones
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("offset", [0, 1])                           # rows beside the product aligned to 16 bytes, and not
def test_residual_beside_ragged_tiles(dtype, N, pair, offset):
    from maco_b200.ops import megakernel as mk
    M = 300
    x, w, g, z = _operands(M, N, 320, dtype, N)
    aux = torch.randn(M, N + 8, device="cuda", generator=g).to(dtype)[:, offset:offset + N]
    out, both = (torch.full((M + 1, N), 7.0, device="cuda", dtype=dtype) for _ in range(2))
    b = mk.ProgramBuilder(torch.device("cuda"), cta_pair=pair)
    b.gemm(x, w, out[:M], epilogue="residual_dual", aux=aux, second=both[:M])
    b.build().run()
    torch.cuda.synchronize()
    _close(out[:M], z, dtype)
    assert torch.equal(both[:M], (out[:M].float() + aux.float()).to(dtype))      # the sum of two rounded values, rounded once
    assert (out[M:] == 7).all() and (both[M:] == 7).all()
