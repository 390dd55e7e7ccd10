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


def _ran_without(tasks, withheld):
    """Indices of the tasks that run when those in ``withheld`` never do: wait conditions alone, in any order of workers."""
    done, events, again = set(), {}, True
    while again:
        again = False
        for i, t in enumerate(tasks):
            if i in done or i in withheld or any(e >= 0 and events.get(e, 0) < c for e, c in zip(t["wait_event"], t["wait_count"])):
                continue
            done.add(i)
            again = True
            for e in t["signal_event"]:
                events[e] = events.get(e, 0) + 1
    return done


@pytest.mark.parametrize("form,whole", [("b", True), ("w", True), ("x", False)])
def test_an_add_over_what_every_row_of_the_product_reads_waits_for_all_of_it(form, whole, monkeypatch):
    """Over the weight or the right-hand side: behind every tile. Over the product's rows: behind the tiles of these rows."""
    tasks = _lower(_graph("cpu", form, 512, 512)[0], monkeypatch).tasks
    gemm, adds = [i for i, t in enumerate(tasks) if t["type"] in (100, 101)], [i for i, t in enumerate(tasks) if t["type"] == ADD]
    assert len(gemm) >= 4 and adds
    ran = [len(_ran_without(tasks, {g}) & set(adds)) for g in gemm]
    assert all(n == 0 if whole else 0 < n < len(adds) for n in ran)


def test_a_product_with_one_tensor_on_both_sides_waits_for_all_of_it(monkeypatch):
    """``h @ h``: a tile reads every row of the right-hand side."""
    g = maco.TaskGraph(num_workers=148, device="cpu")
    h = g.gelu(torch.randn(512, 512).bfloat16())
    g.matmul(h.output, h.output)
    tasks = _lower(g, monkeypatch).tasks
    gelu, gemm = [i for i, t in enumerate(tasks) if t["type"] not in (0, 100, 101)], {i for i, t in enumerate(tasks) if t["type"] in (100, 101)}
    assert len(gelu) > 1 and all(not _ran_without(tasks, {i}) & gemm for i in gelu)


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


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["b", "w"])
def test_add_over_what_every_row_of_the_product_reads(form):
    g, y, z, args, r = _graph("cuda", form, 1024, 1024)
    kept = [t.clone() for t in args]
    want = kept[0].float() @ (kept[1].float() if form == "b" else kept[1].float().t())
    g.compile()
    assert g.runtime_kind == "persistent"
    for _ in range(20):
        for t, k in zip(args, kept):
            t.copy_(k)
        g.execute()
        assert torch.allclose(y.output.float(), want, rtol=2 ** -7, atol=1e-3)      # fp32 sums in another order, one rounding
        assert torch.equal(z.output, (y.output.float() + r.float()).to(r.dtype))
