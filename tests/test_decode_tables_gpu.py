"""Captured decode steps of a design without a position limit, whose block tables are copied entry by entry: what a step reads
when requests change rows, end, grow, are cut back and lose pages to a window."""
import numpy as np
import pytest
import torch

from tests import replay
from tests.test_sarizen import TINY, _engine, tiny_tensors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["P", "R"])             # windows of 9 and 32 tokens, pages smaller than both
def test_captured_steps_equal_eager_ones_as_the_batch_changes(which):
    vocab = TINY[which]["vocab"]
    toks = {f"r{i}": replay.random_tokens(vocab, 200, 40 + i) for i in range(4)}
    engines = [_engine(which, tiny_tensors(which), "float32", "cuda:0", max_tokens=900) for _ in range(2)]
    at = {}

    def both(rids, captured):
        fed = [toks[r][at[r]] for r in rids]
        want = engines[1].step([(r, [t], [0]) for r, t in zip(rids, fed)])
        got = engines[0].decode_logits(rids, fed) if captured else engines[0].step([(r, [t], [0]) for r, t in zip(rids, fed)])
        for r in rids:
            at[r] += 1
        if captured:
            # a row holds its request's pages and -1 behind them, whoever was in it before
            graph = engines[0]._decode_graphs[len(rids)]
            for group, (o, shape) in zip(engines[0].cache.groups, graph.bt_offsets):
                rows = graph.meta[o:o + shape[0] * shape[1]].view(shape)
                for row, r in zip(rows, rids):
                    n = group.tables.length(r)
                    held = [(a, int(b)) for a, b in zip(row[:n].tolist(), group.tables.tail(r, 0)) if b >= 0]   # (a window lets pages go)
                    assert held and all(a == b for a, b in held) and int(row[n:].max()) == -1
        assert torch.allclose(got, want, rtol=0, atol=2e-5 * float(want.abs().max()))

    def begin(rid, n):
        at[rid] = n
        for e in engines:
            e.step([(rid, toks[rid][:n], [])])
    assert max(-(-e.spec.max_positions // e.page_tokens) for e in engines) > 16384
    for rid, n in (("r0", 5), ("r1", 61), ("r2", 30)):
        begin(rid, n)
    for rids, steps in ((["r0", "r1"], 40), (["r1", "r0"], 3), (["r2", "r0"], 20), (["r0", "r1"], 2)):
        for _ in range(steps):
            both(rids, True)
    both(["r0", "r1"], False)                              # a step outside the graph moves the tables on
    both(["r0", "r1"], True)
    for e in engines:
        e.close("r1")
    begin("r3", 44)                                        # on pages that r1 gave back
    for _ in range(30):
        both(["r0", "r3"], True)
