"""Waits of the load, MMA and epilogue warps that run out: plain GEMM tiles, two-CTA tiles with both halves or one of them blocked, expert
shares whose condition nothing signals, and one whose row blocks another share never finishes. The launch ends by itself within its
budget, reports a timeout, writes nothing, and what runs behind it works."""
import pytest
import torch

from maco_b200 import _native

pytestmark = pytest.mark.gpu
DT = torch.bfloat16


def _ends_in_time(prog):
    _native.status(clear=True)
    prog.run()
    torch.cuda.synchronize()                # returns: every wait is bounded
    # (the combine pass of an expert layer counts its conditions among those that other ranks fulfil)
    assert _native.status(clear=True) & (_native.STATUS_TIMEOUT | _native.STATUS_PEER_TIMEOUT)
    prog.reset_after_failure()


@pytest.mark.parametrize("form", ["static", "dynamic", "pair", "pair_half_0", "pair_half_1"])
@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("k_blocks", [2, 12])                     # fewer k-blocks than the ring has stages, and more
def test_gemm_tiles(form, bn, k_blocks):
    from maco_b200.ops import megakernel as mk
    x = torch.randn(512, 64 * k_blocks, device="cuda", dtype=DT)
    w = torch.randn(512, 64 * k_blocks, device="cuda", dtype=DT) * (64 * k_blocks) ** -0.5
    out = torch.zeros(512, 512, device="cuda", dtype=DT)

    def program(blocked):
        b = mk.ProgramBuilder(torch.device("cuda"), mode="dynamic" if form == "dynamic" else "static", cta_pair=form.startswith("pair"),
                              wait_budget_ms=20.0 if blocked else None)
        orphan = (b.new_event(), 1, False, False)
        half = {"pair_half_0": 0, "pair_half_1": 1}.get(form)
        kw = {}
        if blocked and half is None:
            kw["extra_waits"] = [orphan]
        elif blocked:
            kw["row_wait"] = lambda mb: orphan if mb % 2 == half else None
        b.gemm(x, w, out, bn=bn, **kw)
        return b.build()

    _ends_in_time(program(True))
    assert torch.all(out == 0)
    program(False).run()
    torch.cuda.synchronize()
    assert _native.status() == 0
    want = x.double() @ w.double().t()
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16).all()


@pytest.mark.parametrize("what", ["condition", "row_block"])
def test_expert_shares(what):
    from maco_b200.models.moe_layer import MoEEPLayer
    from maco_b200.ops import megakernel as mk
    from maco_b200.task_graph.nodes import TaskType

    class Blocked(MoEEPLayer):
        def _expert_shares(self, b, arrived, e_ret):
            b.wait_budget_ms = 20.0
            if what == "condition":
                return super()._expert_shares(b, (b.new_event(), 1, False, False), e_ret)
            n = super()._expert_shares(b, arrived, e_ret)
            first = next(t for t in b.tasks if t["type"] == mk.T_MOE_EXPERTS)
            first["type"] = int(TaskType.NOP)                     # its gate / up tiles are nobody's: down tiles of their row blocks wait
            return n

    sizes = dict(hidden=256, experts=8, top_k=2, inter=256, tokens=256, capacity_factor=4.0, seed=3, weight_std=0.05, router_std=0.5)
    layer = Blocked(**sizes)
    layer.x.copy_(torch.randn(256, 256, device="cuda"))
    layer.out.zero_()
    _ends_in_time(layer.program)
    assert torch.all(layer.out == 0)
    good = MoEEPLayer(**sizes)
    out = good(layer.x.clone())
    torch.cuda.synchronize()
    assert _native.status() == 0
    ref = good.reference(layer.x)
    # the bound of the single-GPU layer test: bf16 activations, and a token whose logits tie may take another expert
    assert (out.float() - ref).abs().max().item() < 4e-2 * max(1.0, ref.abs().max().item())
