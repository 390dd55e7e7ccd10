"""Host-side planning helpers of the program builder (no GPU): the K-slice choice of few-row GEMMs
and the per-worker key shares of decode attention."""
import collections

import pytest

from maco_b200.ops.megakernel import attention_pieces, pick_split_k, stream_pieces


@pytest.mark.parametrize("groups,kv_len,workers", [(256, 4097, 148), (512, 4097, 148), (64, 4097, 148),
                                                   (6, 1037, 148), (16, 1400, 148), (3, 301, 5), (1, 1, 148)])
def test_attention_pieces_cover_every_key_once_and_balance(groups, kv_len, workers):
    pieces = attention_pieces(groups, kv_len, workers)
    covered = collections.defaultdict(list)
    load = collections.Counter()
    for g, s0, keys, w in pieces:
        assert keys > 0 and 0 <= w < workers
        assert s0 % 128 == 0                              # cuts inside a group sit on chunk boundaries
        covered[g].append((s0, keys))
        load[w] += keys
    assert sorted(covered) == list(range(groups))
    for g, spans in covered.items():                      # contiguous, in order, whole range
        pos = 0
        for s0, keys in spans:
            assert s0 == pos
            pos += keys
        assert pos == kv_len
    target = -(-(groups * kv_len) // workers)
    assert max(load.values()) <= -(-target // 128) * 128 + 128
    # a worker's pieces are consecutive in emission order (its queue reads memory front to back)
    seen, last = set(), None
    for _, _, _, w in pieces:
        if w != last:
            assert w not in seen
            seen.add(w)
            last = w


def test_split_k_fills_the_machine_without_extra_waves():
    W = 148
    for n_tiles, k_blocks in [(20, 80), (20, 64), (100, 80), (20, 200), (5, 80), (25, 80)]:
        sp = pick_split_k(n_tiles, k_blocks, W)
        assert 1 <= sp <= max(1, k_blocks // 2)
        waves = -(-n_tiles * sp // W)
        # never worse than the unsplit GEMM under the same cost model
        assert waves * (-(-k_blocks // sp) + 8) <= -(-n_tiles // W) * (k_blocks + 8)
    assert pick_split_k(20, 80, W) * 20 <= W            # one wave when the tiles fit
    assert pick_split_k(400, 16, W) == 1 or pick_split_k(400, 16, W) <= 8


def test_block_weight_round_trip_and_tile_contiguity():
    import torch
    from maco_b200.ops.gemm import block_weight, unblock_weight
    w = torch.arange(512 * 192, dtype=torch.float32).view(512, 192).to(torch.bfloat16)
    wb = block_weight(w)
    assert wb.shape == (2, 3, 256, 64) and wb.is_contiguous()
    assert torch.equal(wb[1, 2], w[256:512, 128:192])           # one tile's k-block is one contiguous 32 KB block
    assert torch.equal(unblock_weight(wb), w)
    with pytest.raises(ValueError):
        block_weight(w[:100])


def test_trace_records_come_back_in_the_builders_order():
    """Static programs upload their tasks queue after queue; record i of a trace still belongs to the builder's task i."""
    import numpy as np
    import torch
    from maco_b200.ops import megakernel as mk
    b = mk.ProgramBuilder(torch.device("cpu"), num_workers=3)
    for ty in (105, 106, 112, 113, 300, 105, 0):
        b.add_task(ty, b"")
    queues = mk.assign_static_queues(b.tasks, 3, 0)
    order = np.array([i for q in queues for i in q])
    assert order.tolist() != sorted(order.tolist())
    rec = np.zeros(len(order), dtype=mk.TRACE_DTYPE)
    for pos, i in enumerate(order):
        if i != 3:                                       # one task did not run
            rec[pos]["task"], rec[pos]["type"], rec[pos]["t_end_ns"] = pos, b.tasks[i]["type"], 100 + i
    out = mk.records_in_builder_order(rec, order)
    for i, t in enumerate(b.tasks):
        assert (out[i]["task"], out[i]["type"], out[i]["t_end_ns"]) == ((i, t["type"], 100 + i) if i != 3 else (0, 0, 0))


def test_switch_of_the_fused_finishing_pass_holds_for_few_rows(monkeypatch):
    """MACO_SPLITK_FUSED=0 selects split-K tiles with finishing tasks, also up to 64 rows; shapes that only the few-row form
    takes, and the QKV projection whose finishing is always fused, keep it."""
    import torch
    from maco_b200.ops import megakernel as mk

    def types(N, K=512, M=8, **kw):
        b = mk.ProgramBuilder(torch.device("cpu"), num_workers=16)
        z = lambda *s: torch.empty(*s, dtype=torch.bfloat16)
        b.gemm_splitk(z(M, K), z(N, K), z(M, N), **kw)
        return [t["type"] for t in b.tasks], [t["raw"][7] & 4 for t in b.tasks if t["type"] == 101]

    monkeypatch.delenv("MACO_SPLITK_FUSED", raising=False)
    kinds, few = types(1024)
    assert mk.T_SPLITK_FIN not in kinds and all(few)
    monkeypatch.setenv("MACO_SPLITK_FUSED", "0")
    kinds, few = types(1024)
    assert mk.T_SPLITK_FIN in kinds and not any(few)
    assert all(types(1152)[1]) and all(types(1024, K=520)[1])
    assert all(types(1024, fused_finish=True)[1])                        # the argument goes before the switch


@pytest.mark.parametrize("n_tiles,steps", [(1, 1), (1, 3), (16, 16), (20, 40), (24, 16), (40, 16), (96, 16), (100, 40), (148, 7), (149, 7), (224, 32), (60, 2)])
def test_stream_pieces_cover_every_step_once(n_tiles, steps):
    """A few-row GEMM's (tile, k-step) pairs: each in one part, and one part per worker where the tiles divide well over them."""
    pieces = stream_pieces(n_tiles, steps, 148)
    seen = sorted((t, s) for t, s0, n, _ in pieces for s in range(s0, s0 + n))
    assert seen == [(t, s) for t in range(n_tiles) for s in range(steps)]
    assert all(0 <= w < 148 and n > 0 for _, _, n, w in pieces)
    if 90 <= n_tiles * (148 // n_tiles if n_tiles <= 148 else 0) and steps // 2 >= 148 // n_tiles:
        workers = [w for _, _, _, w in pieces]
        assert len(set(workers)) == len(workers)
        assert max(n for _, _, n, _ in pieces) - min(n for _, _, n, _ in pieces) <= 1
