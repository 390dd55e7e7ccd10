"""SwiGLU epilogues against SiLU in 64 bits, far into the tail where the result is still a bf16 number."""
import pytest
import torch

import maco_b200 as maco
from maco_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [8, 64, 300])       # few-row tiles (whole, and cut along K where there are enough weights), plain tiles
@pytest.mark.parametrize("hidden,ffn", [(1024, 512), (1024, 2560)])
def test_swiglu_epilogue_in_the_tails(rows, hidden, ffn):
    """One non-zero per row of x and 1 as its weight: the accumulators are exactly the gates and ups that are put in."""
    dt = torch.bfloat16
    gates = torch.cat([torch.linspace(-88.5, -80.0, 96), torch.linspace(-12.0, 12.0, 384), torch.tensor([0.0, -0.0, -100.0, -300.0, 300.0, 1e30, -1e30, 87.0])])
    gate = gates[torch.randint(len(gates), (rows, ffn))].to(dt).cuda()
    gate[0, : len(gates)] = gates[:ffn].to(dt).cuda()
    x = torch.zeros(rows, hidden, device="cuda", dtype=dt)
    wg, wu = torch.zeros(ffn, hidden, device="cuda", dtype=dt), torch.zeros(ffn, hidden, device="cuda", dtype=dt)
    x[:, 0], x[:, 1] = 1.0, 1.0
    wu[:, 1] = 1.0
    out = []
    graph = maco.TaskGraph()
    w = ops.interleave_gate_up(wg, wu)
    y = graph.linear(x, w, activation="swiglu")
    graph.compile()
    for r in range(min(rows, 4)):                    # gates of row r as the weights of the first input feature: every row of x sees them
        wg[:, 0] = gate[r]
        w.copy_(ops.interleave_gate_up(wg, wu))
        graph.execute()
        out.append(y.output.clone())
    g = gate[: len(out)].double()
    ref = g * torch.sigmoid(g)
    for r, o in enumerate(out):
        e = (o.double() - ref[r]).abs()
        # fp32: 2 ulp of the exponential and half of one for each rounding of its argument (|x| 2^-24) and of the quotient; then bf16, whose
        # 8 significant bits are a half unit of at most 2^-8 of the value. Beyond exp(88.7) the quotient is 0 (the value below 1e-40).
        assert (e <= ref[r].abs() * (2.0 ** -8 + g[r].abs().clamp(max=90) * 2.0 ** -23 + 2.0 ** -21) + 1e-40).all()
        assert (o[:, (g[r] > -88.0) & (g[r] < -80.0)] < 0).all()
