"""Which form a graph's products take, from the sizes alone: lowered on the CPU for 148 workers."""
import types

import pytest
import torch

import maco_b200 as maco
from maco_b200.ops import megakernel as mk


def _lower(graph, monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d=None: types.SimpleNamespace(multi_processor_count=148))
    monkeypatch.setattr(mk.ProgramBuilder, "build", lambda self: self)
    graph._infer_dependencies()
    return mk.lower_graph(graph, mode="static", trace=False)


def _bf(*shape):
    return torch.empty(*shape, dtype=torch.bfloat16)


@pytest.mark.parametrize("rows,n,k,bias,act,pair", [
    (200, 8192, 2048, False, None, False), (640, 4096, 2048, False, None, False), (2000, 1024, 4096, False, None, False),      # 128 columns
    (1000, 4096, 4096, True, None, False), (200, 4096, 4096, False, "silu", False),                                            # long epilogues
    (4000, 4096, 4096, False, None, True), (4000, 4096, 4096, True, "gelu", True), (2048, 4608, 1024, False, None, True),       # every pair has a tile
])
def test_single_products_take_two_cta_tiles_only_where_they_cover_every_pair(rows, n, k, bias, act, pair, monkeypatch):
    g = maco.TaskGraph(num_workers=148, device="cpu")
    g.linear(_bf(rows, k), _bf(n, k), _bf(n) if bias else None, activation=act)
    assert _lower(g, monkeypatch).cta_pair == pair


@pytest.mark.parametrize("rows,hidden,ffn,pair", [(1003, 2048, 5504, True), (640, 2048, 4096, True), (300, 4096, 8192, True), (8192, 4096, 14336, True),
                                                  (2048, 1024, 2816, False), (128, 4096, 8192, False), (64, 4096, 14336, False)])
def test_mlp_blocks_take_two_cta_tiles_where_their_products_are_long(rows, hidden, ffn, pair, monkeypatch):
    g = maco.TaskGraph(num_workers=148, device="cpu")
    y = g.linear(_bf(rows, hidden), _bf(2 * ffn, hidden), activation="swiglu")
    g.linear(y.output, _bf(hidden, ffn))
    assert _lower(g, monkeypatch).cta_pair == pair


@pytest.mark.parametrize("n_tiles,steps,rows,parts", [(100, 32, 1, False), (100, 32, 8, False), (100, 32, 16, True), (100, 32, 64, True), (100, 8, 1, True),
                                                      (96, 16, 3, True), (24, 16, 1, True), (124, 32, 1, True), (76, 32, 64, False)])
def test_few_rows_keep_long_parts_in_one_line(n_tiles, steps, rows, parts):
    """Whole tiles or equal parts of them, against one line that every worker has a piece of."""
    pieces = mk.stream_pieces(n_tiles, steps, 148, rows)
    per_tile = {t: sum(1 for p in pieces if p[0] == t) for t in range(n_tiles)}
    assert (len(set(per_tile.values())) == 1 and len({w for *_, w in pieces}) == len(pieces)) == parts
    assert sorted((t, s) for t, s0, n, _ in pieces for s in range(s0, s0 + n)) == [(t, s) for t in range(n_tiles) for s in range(steps)]
