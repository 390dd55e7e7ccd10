"""Graphs whose later nodes overwrite what an earlier product still reads."""
import types

import pytest
import torch

import maco_b200 as maco
from maco_b200.ops import megakernel as mk

ADD = 113


def _lower(graph, monkeypatch):
    """The task list of a CPU graph, planned for 148 workers."""
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d=None: types.SimpleNamespace(multi_processor_count=148))
    monkeypatch.setattr(mk.ProgramBuilder, "build", lambda self: self)
    graph._infer_dependencies()
    return mk.lower_graph(graph, mode="static", trace=False)


def _graph(device, form, rows, n, dtype=torch.bfloat16):
    """``y`` = a product, ``z`` = ``y + r`` written over the product's rows ("x"), over its weight ("w"), over the right-hand operand of a
    matmul ("b"), or into a tensor of its own ("free")."""
    g = maco.TaskGraph(num_workers=148, device=device)
    x, r = torch.randn(rows, n, device=device).to(dtype), torch.randn(rows, n, device=device).to(dtype)
    w = (torch.randn(n, n, device=device) * n ** -0.5).to(dtype)
    if form == "b":
        a = (torch.randn(rows, rows, device=device) * rows ** -0.5).to(dtype)
        y, args = g.matmul(a, x), (a, x)
    else:
        y, args = g.linear(x, w), (x, w)
    z = g.add(y.output, r, output={"x": x, "w": w, "b": x, "free": None}[form])
    return g, y, z, args, r


@pytest.mark.parametrize("form,folded", [("free", True), ("x", False), ("w", False), ("b", False)])
def test_an_add_over_an_operand_of_its_product_is_a_task_of_its_own(form, folded, monkeypatch):
    g, *_ = _graph("cpu", form, 512, 512)
    kinds = [t["type"] for t in _lower(g, monkeypatch).tasks]
    assert (ADD not in kinds) == folded


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [130, 512, 1300])
def test_residual_add_over_the_rows_of_its_product(rows):
    """Several column tiles read the rows that the add overwrites."""
    g, y, z, (x, w), r = _graph("cuda", "x", rows, 1024)
    x0, w0 = x.clone(), w.clone()
    want = maco.ops.gemm(x0, w0)
    g.compile()
    assert g.runtime_kind == "persistent" and z.output.data_ptr() == x.data_ptr()
    for _ in range(20):
        x.copy_(x0)
        g.execute()
        # fp32 sums of 1024 terms in the tensor cores' order either way; one rounding each
        assert torch.allclose(y.output.float(), want.float(), rtol=2 ** -7, atol=1e-3)
        assert torch.equal(z.output, (y.output.float() + r.float()).to(x.dtype)) and torch.equal(w, w0)
