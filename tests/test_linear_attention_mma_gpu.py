"""Linear attention with a decaying state in prompt portions, and the row kernels beside it, against float64."""
import types

import numpy as np
import pytest
import torch

from tests.test_kernels_gpu import DEV, _randn, ops16  # noqa: F401

pytestmark = pytest.mark.gpu


def _walk(q, k, v, decay, state):
    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=torch.float64, device=q.device)
    for t in range(q.shape[0]):
        state = decay[:, None, None] * state + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", state, q[t])
    return out, state


def _step(heads, dim, vdim, q_lens):
    n, slots = sum(q_lens), [4, 1, 3][:len(q_lens)] if len(q_lens) <= 3 else [6 + i for i in range(len(q_lens))]
    cols = 2 * heads * dim + heads * vdim
    proj = _randn((n, cols + 8), 3, torch.bfloat16, 1.5)[:, :cols]
    state = _randn((6 + len(q_lens), heads, dim, vdim), 4)
    decay = torch.tensor([0.97, 0.0, 1.0, 1.01][:heads], device=DEV)
    i32 = dict(dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(q_start=torch.tensor(np.concatenate([[0], np.cumsum(q_lens)]), **i32),
                                slot_ids=torch.tensor(slots, **i32), n_seqs=len(q_lens), q_lens=np.array(q_lens),
                                max_q_len=max(q_lens), decode_only=False, status=torch.zeros(4, **i32))
    return proj, state, decay, ctx, slots


# dim: below, at and above the widths of the kernels' forms; vdim: a part of a block's 64 or 128 columns, one block, a block and a part.
# Lengths: one token, around a tile of 64, several tiles; decode rows in front
# of a portion and more sequences than two rounds of blocks hold; decays of 0, weak, 1 and above 1.
@pytest.mark.parametrize("heads,dim,vdim", [(2, 8, 8), (3, 40, 72), (2, 64, 64), (4, 128, 128), (1, 88, 24), (2, 72, 136)])
@pytest.mark.parametrize("q_lens", [[16], [63, 1, 65], [200, 64, 130], [700],
                                    [1] * 24 + [100], [17, 1] * 160])
def test_prompt_portions_against_the_recurrence(ops16, heads, dim, vdim, q_lens):  # noqa: F811
    proj, state, decay, ctx, slots = _step(heads, dim, vdim, q_lens)
    n, before, starts = sum(q_lens), state.clone(), ctx.q_start.tolist()
    out = torch.full((n, heads * vdim), 9.0, device=DEV)
    ops16.linear_attention(ctx, proj, out, state, decay, heads, dim, vdim, 0, heads * dim, 2 * heads * dim, chunk=64)
    assert ctx.status.tolist() == [0, 0, 0, 0]
    act = torch.nn.functional.silu(proj.double())
    q, k = (act[:, i * heads * dim:(i + 1) * heads * dim].view(n, heads, dim) for i in (0, 1))
    v = act[:, 2 * heads * dim:].view(n, heads, vdim)
    for s, (a, b, slot) in enumerate(zip(starts[:-1], starts[1:], slots)):
        want, end = _walk(q[a:b], k[a:b], v[a:b], decay.double(), before[slot].double())
        size, end_size = _walk(q[a:b].abs(), k[a:b].abs(), v[a:b].abs(), decay.double(), before[slot].double().abs())
        # a silu is within 2^-21 (an exponential of two units of the last place, a sum, a division), an output has three; sums
        # of n terms in fp32 add n 2^-24, the weights a rounding each
        rel = 3 * 2.0 ** -21 + (b - a + dim + 8) * 2.0 ** -24
        got = out[a:b].view(b - a, heads, vdim).double()
        assert ((got - want).abs() <= rel * size + 1e-30).all(), s
        assert ((state[slot].double() - end).abs() <= rel * end_size + 1e-30).all(), s
        # roundings of either sign grow with the root of their number; operands short of 32 bits show (two bfloat16 terms: 1.5e-6 to 5e-6)
        assert (got - want).norm() <= 8e-7 * want.norm() and (state[slot].double() - end).norm() <= 8e-7 * end.norm()
    others = [i for i in range(6 + len(q_lens)) if i not in slots]
    assert torch.equal(state[others], before[others])


# in the first tile, at its end, and in the last of several; an infinity or a NaN in a key, a query or a value
@pytest.mark.parametrize("at", [5, 63, 130])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_token_that_is_not_finite_reaches_no_earlier_one(ops16, at, bad):  # noqa: F811
    heads, dim, vdim = 2, 64, 72
    hd, c = heads * dim, 9                             # channel or column 9 of head 0
    runs = []
    for column in (None, c, hd + c, 2 * hd + c):
        proj, state, decay, ctx, slots = _step(heads, dim, vdim, [150])
        decay.fill_(0.9)
        proj = proj.clone()
        if column is not None:
            proj[at, column] = bad
        out = torch.full((150, heads * vdim), 9.0, device=DEV)
        ops16.linear_attention(ctx, proj, out, state, decay, heads, dim, vdim, 0, hd, 2 * hd, chunk=64)
        assert ctx.status.tolist() == [0, 0, 0, 0]
        runs.append((out.view(150, heads, vdim), state[slots[0]]))
    (clean, end), (q, q_end), (k, k_end), (v, v_end) = runs
    for out, state in runs[1:]:
        assert torch.equal(out[:at], clean[:at]) and torch.equal(out[:, 1], clean[:, 1]) and torch.equal(state[1], end[1])
    # a query is its own token's; a key's channel is a row of the state and reaches every later output; a value's column stays one
    others = [i for i in range(vdim) if i != c]
    assert torch.equal(q[at + 1:], clean[at + 1:]) and not torch.isfinite(q[at, 0]).any() and torch.equal(q_end, end)
    rows = [i for i in range(dim) if i != c]
    assert torch.equal(k_end[0, rows], end[0, rows]) and not torch.isfinite(k_end[0, c]).any()
    assert not torch.isfinite(k[at:, 0]).any()
    assert torch.equal(v[:, 0, others], clean[:, 0, others]) and torch.equal(v_end[0][:, others], end[0][:, others])
    assert not torch.isfinite(v[at:, 0, c]).any() and not torch.isfinite(v_end[0, :, c]).any()


def test_silu_of_every_bfloat16(ops16):  # noqa: F811
    """A state that is forgotten at once (decay 0), keys and values of 128, whose silu is 128: outputs are 2^14 silu(q)."""
    words = torch.arange(1 << 16, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    z = words[(words.float().abs() < 2.0 ** 80)]
    n = z.numel()
    proj = torch.zeros((n, 24), device=DEV, dtype=torch.bfloat16)
    proj[:, 0], proj[:, 8], proj[:, 16:] = z, 128.0, 128.0
    i32 = dict(dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(q_start=torch.tensor([0, n], **i32), slot_ids=torch.zeros(1, **i32), n_seqs=1, q_lens=np.array([n]),
                                max_q_len=n, decode_only=False, status=torch.zeros(4, **i32))
    out = torch.empty((n, 8), device=DEV)
    ops16.linear_attention(ctx, proj, out, torch.zeros((1, 1, 8, 8), device=DEV), torch.zeros(1, device=DEV), 1, 8, 8, 0, 8, 16)
    want = torch.nn.functional.silu(z.double())[:, None]
    # the exponential's two units of the last place, its product, the divisor's sum and the quotient: four; an exponential below
    # 2^-126 is held to 2^-149, and |z| times it
    bound = 2.0 ** -21 * want.abs() + (z.double().abs()[:, None] + 2) * 2.0 ** -149
    wrong = ((out.double() * 2.0 ** -14 - want).abs() > bound).any(1)
    assert not wrong.any(), (z[wrong][:8], out[wrong][:8, 0] * 2.0 ** -14, want[wrong][:8])


# the smallest vector row, one that fills no round of 256 threads, the widest in registers, and the first that is not
@pytest.mark.parametrize("width", [4, 1028, 4096, 4100])
@pytest.mark.parametrize("wdtype", [torch.float32, torch.bfloat16])
def test_gate_norm(ops16, width, wdtype):  # noqa: F811
    n, eps = 5, 1e-6
    o, w = _randn((n, width), 1, scale=3.0), _randn((width,), 2).to(wdtype)
    gate = _randn((n, width + 12), 3, torch.bfloat16)[:, 8:8 + width]
    out = torch.empty((n, width), device=DEV, dtype=torch.bfloat16)
    ops16.gate_norm(o, w, gate, out, eps)
    x = o.double()
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double() * torch.sigmoid(gate.double())
    # the result's own rounding, and a few units of fp32 before it
    assert ((out.double() - want).abs() <= (2.0 ** -8 + 1e-5) * want.abs() + 1e-30).all()


@pytest.mark.parametrize("width", [4, 1028, 4096, 4100])
@pytest.mark.parametrize("wdtype", [torch.float32, torch.bfloat16])
def test_two_norms_of_the_same_rows(ops16, width, wdtype):  # noqa: F811
    n, eps = 5, 1e-6
    x, a, b = _randn((n, width), 1, scale=3.0), _randn((width,), 2).to(wdtype), _randn((width,), 3).to(wdtype)
    out = [torch.empty((n, width), device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    ops16.rms_norm_pair(x, a, b, *out, eps)
    y = x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + eps)
    for got, w in zip(out, (a, b)):
        assert ((got.double() - y * w.double()).abs() <= (2.0 ** -8 + 1e-5) * (y * w.double()).abs() + 1e-30).all()
