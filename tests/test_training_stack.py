"""The training stack on one-CTA and two-CTA tiles: an odd number of 128-token blocks, more layers than gradient buffers."""
import pytest
import torch

from maco_b200.ops import megakernel as mk


@pytest.mark.parametrize("hidden,tokens,asked,got", [
    (512, 896, None, False), (512, 896, True, True), (512, 896, False, False),
    (3072, 3072, None, True), (3072, 3072, False, False),                       # 144 tiles of 256 x 256: two-CTA unless told otherwise
    (2816, 8192, None, False),
])
def test_stack_takes_the_tiles_that_were_asked_for(hidden, tokens, asked, got):
    from maco_b200.models.dp_mlp_stack import DPMLPStackBackward
    m = DPMLPStackBackward(layers=1 if hidden > 512 else 5, hidden=hidden, tokens=tokens, device=torch.device("cpu"), cta_pair=asked)
    assert m.cta_pair == got and m.builder.cta_pair == got
    mk.simulate_static_queues([(m.builder.tasks, mk.assign_static_queues(m.builder.tasks, m.builder.num_workers, m.builder.num_comm_workers))])


@pytest.mark.gpu
@pytest.mark.parametrize("cta_pair", [True, False])
@pytest.mark.parametrize("layers,hidden,tokens", [(1, 256, 128), (4, 512, 896), (6, 768, 384)])
def test_gradients_on_both_kinds_of_tiles(layers, hidden, tokens, cta_pair):
    from maco_b200 import _native
    from maco_b200.models.dp_mlp_stack import DPMLPStackBackward
    m = DPMLPStackBackward(layers=layers, hidden=hidden, tokens=tokens, seed=2, weight_std=0.05, cta_pair=cta_pair)
    assert m.program.cta_pair == cta_pair
    ref = m.reference_grads()
    outs = []
    for _ in range(3):
        m.forward()
        outs.append(m.backward().clone())
    torch.cuda.synchronize()
    # bf16 activations and gradients between the layers: the bound of the one-CTA test, of every layer's own largest gradient
    for g, r in zip(outs[0], ref):
        assert (g - r).abs().max().item() < 3e-2 * r.abs().max().item() + 1e-7
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert _native.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layers,hidden,tokens", [(2, 256, 128), (3, 768, 384), (2, 2048, 2048), (2, 2048, 2176)])     # 2^22 activations, and more
def test_forward_in_one_launch_a_layer_or_two(layers, hidden, tokens, dtype):
    """Pre-activations and activations of both forms of the forward are those of the product and its GELU one behind the other, bit by bit."""
    from maco_b200 import ops
    from maco_b200.models.dp_mlp_stack import DPMLPStackBackward
    m = DPMLPStackBackward(layers=layers, hidden=hidden, tokens=tokens, seed=2, weight_std=0.05, dtype=dtype)
    for t in m.z + m.a:
        t.fill_(float("nan"))
    last, cur = m.forward(), m.x
    for l in range(layers):
        z = ops.gemm(cur, m.weights[l])
        cur = ops.gelu(z)
        assert torch.equal(m.z[l], z) and torch.equal(m.a[l], cur)
    assert last is m.a[-1]
