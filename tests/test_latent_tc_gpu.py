"""Latent attention of prompt portions on tcgen05 (csrc/attention_latent_tc.cu): against float64 and beside the mma.sync kernel."""
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DK, DV = 576, 512


@pytest.fixture(scope="module")
def ops():
    from leone_b200.ops.cuda import CudaOps
    o = CudaOps(DEV, torch.bfloat16)
    o.bind_status(torch.zeros(4, dtype=torch.int32, device=DEV))
    o.use_latent_tc = True              # also where the rule takes the other kernel
    return o


def _case(q_lens, before, heads, page_tokens, seed, stale=float("nan")):
    """A step's queries and cache: sequence i brings q_lens[i] tokens after before[i].  What pages hold behind a sequence's last row
    is ``stale``."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    ctx_lens = [a + b for a, b in zip(q_lens, before)]
    blocks = [-(-c // page_tokens) for c in ctx_lens]
    pages = sum(blocks) + 2
    order = np.random.RandomState(seed).permutation(pages).tolist()
    pool = torch.full((pages, 1, page_tokens, DK), stale, device=DEV, dtype=torch.bfloat16)
    table = torch.full((len(q_lens), max(blocks) + 1), -1, dtype=torch.int32)
    rows = []
    for i, c in enumerate(ctx_lens):
        mine = [order.pop() for _ in range(blocks[i])]
        table[i, :len(mine)] = torch.tensor(mine, dtype=torch.int32)
        r = torch.randn((c, DK), device=DEV, generator=g).to(torch.bfloat16)
        rows.append(r)
        for b, page in enumerate(mine):
            part = r[b * page_tokens:(b + 1) * page_tokens]
            pool[page, 0, :len(part)] = part
    n = sum(q_lens)
    q = torch.randn((n, heads * DK), device=DEV, generator=g).to(torch.bfloat16)
    to = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)        # noqa: E731
    ctx = types.SimpleNamespace(
        q_start=to([0] + np.cumsum(q_lens).tolist()), ctx_len=to(ctx_lens), n_seqs=len(q_lens), max_q_len=max(q_lens),
        max_ctx_len=max(ctx_lens), decode_only=max(q_lens) == 1, q_lens=np.array(q_lens), ctx_lens=np.array(ctx_lens),
        positions=to([b + t for a, b in zip(q_lens, before) for t in range(a)]),
        seq_of_token=to([i for i, a in enumerate(q_lens) for _ in range(a)]), status=torch.zeros(4, dtype=torch.int32, device=DEV))
    cache = types.SimpleNamespace(k_pool=pool, v_pool=None, block_table=table.to(DEV), page_tokens=page_tokens, writes=True)
    return ctx, cache, q, rows


def _exact(q_lens, before, heads, q, rows, scale, window, sink, gate):
    out, at = [], 0
    for a, b, r in zip(q_lens, before, rows):
        qs = q[at:at + a].double().view(a, heads, DK)
        k = r.double()
        s = torch.einsum("thd,jd->htj", qs, k) * scale
        p = b + torch.arange(a, device=DEV)[:, None]
        j = torch.arange(len(k), device=DEV)[None, :]
        hidden = (j > p) | ((p - j >= window) if window else (j < 0))
        s = s.masked_fill(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None, None].expand(heads, a, 1)], 2)
        w = torch.softmax(s, -1)[:, :, :len(k)]
        o = torch.einsum("htj,jd->thd", w, k[:, :DV])
        if gate is not None:
            o = o * torch.sigmoid(gate[at:at + a, :heads].double())[:, :, None]
        out.append(o.reshape(a, heads * DV))
        at += a
    return torch.cat(out)


# one tile of queries and one token more, keys that end on a tile's edge and one past it, portions after a context, windows that start
# inside a tile and release pages, decode rows in front, heads that fill a group in part and two groups; pages of 8 to 128 tokens
@pytest.mark.parametrize("q_lens,before,heads,window,page_tokens", [
    ([8], [0], 16, None, 16), ([9], [56], 16, None, 16), ([64], [0], 16, 20, 8), ([65, 3, 130], [0, 70, 5], 16, 64, 16),
    ([200], [700], 18, 100, 32), ([1, 1, 40], [300, 0, 11], 16, 33, 16), ([333], [0], 5, None, 64), ([70, 17], [1, 127], 32, 90, 128)])
def test_against_float64(ops, q_lens, before, heads, window, page_tokens):
    ctx, cache, q, rows = _case(q_lens, before, heads, page_tokens, 3 + len(q_lens) + sum(q_lens))
    if window:                                     # pages that no query reads any more are gone
        for i, b in enumerate(before):
            cache.block_table[i, :max(0, b - window + 1) // page_tokens] = -1
    g = torch.Generator(device=DEV).manual_seed(9)
    sink, gate = torch.randn(heads, device=DEV, generator=g), torch.randn((len(q), heads + 3), device=DEV, generator=g).to(torch.bfloat16)
    for s_, g_ in ((None, None), (sink, gate)):
        out = torch.full((len(q), heads * DV), 5.0, device=DEV, dtype=torch.bfloat16)
        ops.attention_latent(ctx, q, out, cache, heads, DK, DV, DK ** -0.5, window, s_, g_)
        want = _exact(q_lens, before, heads, q, rows, DK ** -0.5, window, s_, g_)
        # probabilities and outputs are rounded to bfloat16: 2^-9 of values of order one
        assert float((out.double() - want).norm() / want.norm()) < 4e-3
        assert bool(((out.double() - want).abs() <= 2e-2 * want.abs().max()).all())
    assert int(ctx.status.abs().sum()) == 0


def test_no_further_from_float64_than_the_other_kernel(ops, monkeypatch):
    """Both round weights and outputs to bfloat16.  One input's rounding errors differ by a percent or two either way between two
    sums of the same weights, so eight inputs' are taken together (about half a percent)."""
    err = {"0": 0.0, "1": 0.0}
    for seed in range(8):
        ctx, cache, q, rows = _case([300], [0], 16, 16, 5 + seed, stale=0.0)
        want = _exact([300], [0], 16, q, rows, DK ** -0.5, 128, None, None)
        for form in err:
            monkeypatch.setenv("LEONE_NO_LATENT_TC", form)
            out = torch.empty((300, 16 * DV), device=DEV, dtype=torch.bfloat16)
            ops.attention_latent(ctx, q, out, cache, 16, DK, DV, DK ** -0.5, 128)
            err[form] += float((out.double() - want).square().sum() / want.square().sum())
    assert err["0"] <= 1.01 * err["1"], err


def test_a_missing_page_is_reported(ops):
    ctx, cache, q, _ = _case([100], [0], 16, 16, 6)
    cache.block_table[0, 2] = 9999
    out = torch.empty((100, 16 * DV), device=DEV, dtype=torch.bfloat16)
    ops.attention_latent(ctx, q, out, cache, 16, DK, DV, DK ** -0.5, None)
    assert int(ctx.status[0]) == 2 and int(ctx.status[3]) in range(32, 48)


def test_sinks_without_weight_and_rows_that_are_nan(ops, monkeypatch):
    """A sink of -inf, or of the type's lowest value, adds nothing to the denominator; a query that is NaN gives NaN in its token's rows
    and in no other's.  As in the other kernel."""
    ctx, cache, q, rows = _case([40, 30], [0, 100], 16, 16, 21, stale=0.0)
    sink = torch.randn(16, device=DEV, generator=torch.Generator(device=DEV).manual_seed(8))
    sink[3], sink[7], sink[9] = float("-inf"), torch.finfo(torch.float32).min, torch.finfo(torch.bfloat16).min
    want = _exact([40, 30], [0, 100], 16, q, rows, DK ** -0.5, 50, sink, None)
    for form in ("0", "1"):
        monkeypatch.setenv("LEONE_NO_LATENT_TC", form)
        for s_ in (sink, sink.to(torch.bfloat16)):
            out = torch.empty((70, 16 * DV), device=DEV, dtype=torch.bfloat16)
            ops.attention_latent(ctx, q, out, cache, 16, DK, DV, DK ** -0.5, 50, s_)
            heads = (out.double() - want).view(70, 16, DV)[:, [3, 7, 9]]
            assert float(heads.norm() / want.view(70, 16, DV)[:, [3, 7, 9]].norm()) < 4e-3        # as in test_against_float64
        poisoned = q.clone()
        poisoned[13, 5] = float("nan")                      # head 0 of token 13
        out = torch.empty((70, 16 * DV), device=DEV, dtype=torch.bfloat16)
        ops.attention_latent(ctx, poisoned, out, cache, 16, DK, DV, DK ** -0.5, 50, sink)
        nan = out.view(70, 16, DV).isnan()
        assert bool(nan[13, 0].all()) and int(nan.sum()) == DV
    assert int(ctx.status.abs().sum()) == 0
