"""The load and MMA loops (whole warps, one elected lane issuing) at the numbers of k-blocks where their ring of stages can go wrong."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rings of four (one-CTA, 256 columns) and six stages: one block, a ring less one, a whole ring, one more, two rings and a bit
@pytest.mark.parametrize("k_blocks", [1, 3, 4, 5, 6, 7, 13])
@pytest.mark.parametrize("trans", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("bn", [128, 256])
def test_gemm_by_k_blocks(k_blocks, trans, pair, bn):
    from maco_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(k_blocks)
    M, N, K = 300, 520, 64 * k_blocks - 8                  # the last block is ragged too
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    want = (a.double() @ b.double().t())
    A = a.t().contiguous() if trans[0] else a
    B = b.t().contiguous() if trans[1] else b
    if trans[0]:                                           # rows of whole 16-byte vectors for the loads
        A = torch.nn.functional.pad(A, (0, 4))[:, :M]
    got = ops.gemm(A, B, trans_a=trans[0], trans_b=trans[1], cta_pair=pair, bn=bn, epilogue="f32")
    # exact products, fp32 sums of at most 832 of them: K * 2^-24 of the sum of magnitudes
    bound = K * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t()) + 1e-6
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("rows", [1, 64])
@pytest.mark.parametrize("steps", [1, 3, 4, 5, 9])
def test_few_row_graph_by_k_steps(rows, steps):
    import maco_b200 as maco
    g = torch.Generator(device="cuda").manual_seed(steps)
    K = 128 * steps
    x = torch.randn(rows, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2560, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    graph = maco.TaskGraph()
    y = graph.linear(x, w)
    graph.compile()
    for _ in range(3):
        graph.execute()
    want = x.double() @ w.double().t()
    # one rounding to bf16 and fp32 sums of K products
    bound = 2.0 ** -8 * want.abs() + K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    assert ((y.output.double() - want).abs() <= bound).all()
