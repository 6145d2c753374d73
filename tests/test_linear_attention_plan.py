"""How the linear attention of a step is cut into launches: the method on stand-in libraries, which record what they are given."""
import signal
import types

import numpy as np
import pytest
import torch

from leone_b200.ops.cuda import CudaOps


class _Library:
    """Any entry returns 0; the calls of the recurrence's entries are kept."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append((name, args))
            return 1 if name.endswith("_supported") else 0
        return entry


def _plan(q_lens, heads, dim, vdim, dtype=torch.bfloat16, chunk=64):
    """The scratch sizes that the call takes and its launches."""
    ops = object.__new__(CudaOps)
    lib, scratch = _Library(), {}
    ops.__dict__.update(_mixers=lib, fast=types.SimpleNamespace(sm_count=148), launches=0, device=torch.device("cpu"))

    def take(name, rows, cols, dt):
        scratch[name] = (rows, cols)
        return torch.empty((1, 1), dtype=dt)
    ops._scratch = take
    ops._stream = lambda: 0
    n = sum(q_lens)
    ctx = types.SimpleNamespace(q_lens=np.array(q_lens), max_q_len=max(q_lens), n_seqs=len(q_lens), decode_only=max(q_lens) == 1,
                                q_start=torch.zeros(len(q_lens) + 1, dtype=torch.int32),
                                slot_ids=torch.zeros(len(q_lens), dtype=torch.int32), status=torch.zeros(4, dtype=torch.int32))
    cols = heads * (2 * dim + vdim)
    # (nothing reads them, and clearing gigabytes would take the caller's time limit on a slow host)
    ops.linear_attention(ctx, torch.empty((n, cols), dtype=dtype), torch.empty((n, heads * vdim)),
                         torch.zeros((1, heads, dim, vdim)), torch.ones(heads), heads, dim, vdim, 0, heads * dim, 2 * heads * dim,
                         chunk=chunk)
    return scratch, [c for c in lib.calls if not c[0].endswith("_supported")]


# one sequence, as many as fit two rounds of blocks and one more, a server's worth; short, equal and ragged portions
@pytest.mark.parametrize("heads,vdim", [(4, 64), (16, 128), (32, 128), (64, 256)])
@pytest.mark.parametrize("q_lens", [[2048], [77] * 9, [77] * 10, [16] * 19, [1] * 18 + [300], [1] * 63 + [16], [40] * 300,
                                    [16, 900] * 40, [1] * 999 + [4000]])
def test_the_choice_of_a_chunk_ends(q_lens, heads, vdim):
    def give_up(*_):
        raise TimeoutError("the choice of a chunk length does not end")
    before = signal.signal(signal.SIGALRM, give_up)
    signal.alarm(5)
    try:
        scratch, calls = _plan(q_lens, heads, 64, vdim)
    finally:
        signal.alarm(0)
        signal.signal(signal.SIGALRM, before)
    assert calls
    # every sequence has at least one chunk, and a chunk holds at least 64 tokens of one
    if "linattn_chunks" in scratch:
        assert scratch["linattn_chunks"][0] <= sum(-(-q // 64) for q in q_lens)


# decode rows lead a mixed step: they are walked, and only what follows goes through tiles of 64 tokens; a row of one token
# between portions stays with them
@pytest.mark.parametrize("q_lens,walked", [([1] * 24 + [100], 24), ([1, 16], 1), ([100], 0), ([100, 1, 1], 0), ([1, 1, 70, 1, 16], 2)])
def test_decode_rows_of_a_mixed_step_are_walked(q_lens, walked):
    _, calls = _plan(q_lens, 4, 64, 64)
    walks = [args for name, args in calls if name == "leone_linear_attention"]
    assert [args[12] for args in walks] == ([walked] if walked else [])        # (its sequences)
    assert len(calls) == len(walks) + 1


def test_steps_of_one_kind_are_one_launch():
    for q_lens, dtype in (([1] * 8, torch.bfloat16), ([15, 1, 2], torch.bfloat16), ([1, 100], torch.float32)):
        _, calls = _plan(q_lens, 4, 64, 64, dtype)
        assert [(name, args[12]) for name, args in calls] == [("leone_linear_attention", len(q_lens))]
