"""The order in which a decode attention's sequences start: what a step hands the kernel, and that it changes no bits."""
import math

import numpy as np
import pytest
import torch

from leone_b200.engine.batch import ORDER_FROM, StepEntry, longest_first
from leone_b200.engine.engine import Engine
from tests.emulated_ops import EmulatedOps
from tests.tiny import make_folder


def test_longest_first_is_a_stable_order():
    rng = np.random.default_rng(0)
    for n in (1, 9, 64, 1024):
        lens = rng.integers(1, 20, n)
        order = longest_first(lens)
        assert order.dtype == np.int32 and sorted(order.tolist()) == list(range(n))
        assert order.tolist() == sorted(range(n), key=lambda i: (-lens[i], i))


def test_a_step_orders_the_decode_rows_in_front_of_its_portions(tmp_path):
    eng = Engine.from_folder(make_folder(tmp_path, "A"), dtype="float32", device="cpu", ops=EmulatedOps(), page_tokens=4,
                             num_pages=200, max_requests=16, max_batch_tokens=128)
    lens = [3, 8, 5, 8, 1, 2, 9, 4, 7, 6, 2]
    for i, n in enumerate(lens):
        eng.step([(i, list(range(1, n + 1)), [])])
    rows = [StepEntry(i, [1], [0]) for i in range(len(lens))]
    for entries, single in ((rows, 11), (rows[:9], 9), (rows[:8], None), (rows[:9] + [StepEntry(9, [1, 2]), rows[10]], 9),
                            ([StepEntry(0, [1, 2])] + rows[1:], None)):
        ctx = eng.build_context(entries)
        if single is None:
            assert ctx.seq_order is None
        else:
            assert single >= ORDER_FROM and ctx.seq_order.tolist() == longest_first(np.array(lens[:single])).tolist()
        assert ctx.ctx_len.tolist() == [lens[e.rid] + len(e.tokens) for e in entries]
        tables = eng.cache.block_table(0, [e.rid for e in entries])
        assert torch.equal(ctx.block_tables[0], torch.from_numpy(np.ascontiguousarray(tables)))


# more blocks than start at once, in one wave of kernels with and without prepared queries; equal lengths too
@pytest.mark.gpu
@pytest.mark.parametrize("n_seqs,n_q,n_kv,d", [(300, 2, 1, 64), (41, 16, 8, 128), (40, 8, 8, 128)])
@pytest.mark.parametrize("equal", [False, True])
def test_the_order_changes_no_bits(n_seqs, n_q, n_kv, d, equal):
    from leone_b200.ops.cuda import CudaOps
    from tests.test_kernels_gpu import DEV, _ctx, _paged_setup, _randn
    import types
    ops = CudaOps(DEV, torch.bfloat16)
    lens = [70] * n_seqs if equal else [int(n) for n in np.random.default_rng(1).integers(1, 200, n_seqs)]
    table, k_pool, v_pool = _paged_setup(lens, 16, n_kv, d, torch.bfloat16, 3)
    k_pool.copy_(_randn(k_pool.shape, 1))
    v_pool.copy_(_randn(v_pool.shape, 2))
    i32 = dict(dtype=torch.int32, device=DEV)
    ctx = _ctx([n - 1 for n in lens], list(range(n_seqs)))
    ctx.q_start, ctx.ctx_len = torch.arange(n_seqs + 1, **i32), torch.tensor(lens, **i32)
    ctx.n_seqs, ctx.max_q_len, ctx.max_ctx_len, ctx.decode_only = n_seqs, 1, max(lens), True
    qkv = _randn((n_seqs, (n_q + 2 * n_kv) * d), 4).to(torch.bfloat16)
    ops.fast.force_decode_splits = 1
    outs = []
    for order in (None, longest_first(np.array(lens)), np.random.default_rng(2).permutation(n_seqs).astype(np.int32)):
        for fuse in (None, dict(q_w=None, k_w=None, eps=1e-6, rope=None, write_cache=False)):
            ctx.seq_order = None if order is None else torch.from_numpy(order).to(DEV)
            cache = types.SimpleNamespace(k_pool=k_pool, v_pool=v_pool, block_table=table, page_tokens=16)
            out = torch.full((n_seqs, n_q * d), 7.0, device=DEV, dtype=torch.bfloat16)
            ops.attention(ctx, qkv, out, n_q, n_kv, d, 1 / math.sqrt(d), None, cache, fuse=fuse)
            outs.append(out)
    assert ctx.status.tolist() == [0, 0, 0, 0]
    assert all(torch.equal(o, outs[i % 2]) for i, o in enumerate(outs)) and torch.isfinite(outs[0]).all()
