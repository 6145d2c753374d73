"""The 32-bit path's matrix product and attention at the sizes where their forms change, against float64."""
import math
import types

import numpy as np
import pytest
import torch

from tests.test_kernels_gpu import DEV, _paged_setup, _randn, _ref_attention, ops32  # noqa: F401

pytestmark = pytest.mark.gpu


# m: the last and first size of every form (1, 2, 4, 8 tokens a block | 128 a tile) and ragged ones; n: fewer than a
# block's four rows, a tile's edge, ragged; k: one piece, the
# last of the any-size kernel and the first of the tensor cores', a ragged stage, several rounds of 256 threads, enough for eight splits
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 24, 25, 64, 128, 129, 257])
@pytest.mark.parametrize("n,k", [(3, 4), (129, 252), (129, 256), (256, 2052), (1030, 4096)])
def test_product_in_32_bits(ops32, m, n, k):  # noqa: F811
    x, w = _randn((m, k + 4), 1)[:, :k], _randn((n, k), 2)
    bias, res = _randn((n,), 3), _randn((m, n + 5), 4)[:, :n]
    want = x.double() @ w.double().t()
    # a sum of k products in any order is within k 2^-24 of the sum of their magnitudes, to first order
    bound = (k + 4) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t() + bias.double().abs() + res.double().abs())
    out = torch.full((m, n), 9.0, device=DEV)
    ops32._gemm_simt(x, w, out, 0, None)
    assert ((out.double() - want).abs() <= bound).all()
    ops32._gemm_simt(x, w, out, 1, None, bias)
    assert ((out.double() - want - bias.double()).abs() <= bound).all()
    got = _randn((m, n + 5), 4)[:, :n]
    ops32._gemm_simt(x, w, got, 2, got, bias)
    assert ((got.double() - want - bias.double() - res.double()).abs() <= bound).all()


# 1, 2, 4 and 8 blocks over K, the last three with an odd number of steps of 32; a whole stage ring and a ragged last step
@pytest.mark.parametrize("k", [256, 544, 1056, 2080, 2052, 6116])
def test_product_on_tensor_cores_keeps_the_small_terms(ops32, k):  # noqa: F811
    x, w = _randn((40, k), 11), _randn((256, k), 12)
    out = torch.empty((40, 256), device=DEV)
    ops32._gemm_simt(x, w, out, 0, None)
    want = x.double() @ w.double().t()
    # 2.0e-7 to 2.7e-7 measured at any K; one term of 11 bits alone, or a lost product of the small terms in one of the
    # blocks, is 1e-4 and more
    assert (out.double() - want).norm() <= 5e-7 * want.norm()
    half = out[:, ::2].double() - want[:, ::2]
    assert half.norm() <= 5e-7 * want[:, ::2].norm() and (out.double() - want).abs().max() <= 3e-6 * want.norm() / want.numel() ** 0.5


def test_rows_of_any_magnitude_keep_their_bits(ops32):  # noqa: F811
    """Token rows and weight rows of every magnitude in one tile: where the second terms would be lost or products leave the range
    the result is a chain of FMA's."""
    k = 288
    ex = torch.tensor([0, -60, -99, -101, -110, -120, -126, 60, 100, 125, 0, 0], device=DEV)
    ew = torch.tensor([0, -60, -99, -101, -115, -126, 50, 90, 124], device=DEV)
    x = (_randn((48, k), 13).clamp(-2, 2).double() * 2.0 ** ex.repeat(4).double()[:, None]).float()
    w = (_randn((180, k), 14).clamp(-2, 2).double() * 2.0 ** ew.repeat(20).double()[:, None]).float()
    x[10::12] = 0
    w[5] = 0
    out = torch.empty((48, 180), device=DEV)
    ops32._gemm_simt(x, w, out, 0, None)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    inside = size < 2.0 ** 126
    assert inside.sum() > 4000 and (~inside).sum() > 500
    # a sum of k products within k 2^-24 of their magnitudes; what falls below the least number is lost, 2^-149 a product
    bound = (k + 4) * 2.0 ** -24 * size + 2 * k * 2.0 ** -149
    assert ((out.double() - want).abs() <= bound)[inside].all()
    small = inside & (size < 2.0 ** -90) & (size > 2.0 ** -110)
    assert small.sum() > 100 and (out.double() - want)[small].norm() <= 1e-6 * want[small].norm()
    x, w = torch.full((40, k), 1e30, device=DEV), torch.full((130, k), 1e30, device=DEV)
    x[3], w[7] = 1.0 + 2.0 ** -11, -1e30
    out = torch.empty((40, 130), device=DEV)
    ops32._gemm_simt(x, w, out, 0, None)
    inf = float("inf")
    assert (out[:3, :7] == inf).all() and (out[:3, 7] == -inf).all()
    assert ((out[3].double() - x[3].double() @ w.double().t()).abs() <= (k + 4) * 2.0 ** -24 * k * 1.001e30).all()


def test_values_at_the_edge_of_the_range_pass_through_the_product(ops32):  # noqa: F811
    """The largest number, one that rounds past it at 11 bits, and NaNs of any payload, alone in their row and column."""
    m, n, k = 40, 300, 256
    for word in (0x7f7fffff, 0x7f7ff000, 0x7f7fefff, 0xff7fffff, 0x7fffffff, 0x7f800001, 0x7fc00000):
        x, w = torch.zeros((m, k), device=DEV), torch.eye(n, k, device=DEV)
        x.view(torch.int32)[7, 3] = word - (1 << 32) if word >> 31 else word
        x[8, 5] = 1.5
        out = torch.empty((m, n), device=DEV)
        ops32._gemm_simt(x, w, out, 0, None)
        if word & 0x7fffffff > 0x7f800000:
            assert torch.isnan(out[7]).any()
        else:                                          # (such a row is summed by FMA; two terms would hold a word to 2^-23 of it)
            assert ((out[7, :k].double() - x[7].double()).abs() <= 2.0 ** -23 * x[7].double().abs()).all()
        assert torch.equal(out[8, :k], x[8]) and torch.isfinite(out[:7]).all() and torch.isfinite(out[9:]).all()


def test_a_row_of_the_product_with_an_infinity_stays_its_own(ops32):  # noqa: F811
    for m in (4, 40):
        x, w = _randn((m, 260), 5), _randn((130, 260), 6)
        x[1, 3] = float("inf")
        out = torch.empty((m, 130), device=DEV)
        ops32._gemm_simt(x, w, out, 0, None)
        keep = [i for i in range(m) if i != 1]
        assert torch.isfinite(out[keep]).all() and torch.equal(out[1], torch.copysign(torch.tensor(float("inf"), device=DEV), w[:, 3]))


# groups of 1, 2, 3 (padded to 4) and 9 (two runs of 8) heads; pages that no tile of 64 divides; windows inside and across tiles
@pytest.mark.parametrize("n_q,n_kv,d,pt,window", [(4, 4, 64, 16, None), (16, 8, 128, 16, None), (6, 2, 128, 5, 70),
                                                  (9, 1, 64, 3, 1), (32, 4, 128, 16, 300)])
@pytest.mark.parametrize("seq_lens,starts", [([1, 65, 700, 33], [0, 64, 699, 32]),          # one token each: the decode form
                                             ([150, 3, 131, 64], [0, 0, 100, 0]),           # prompts
                                             ([640, 9, 200], [639, 8, 71])])                # decode rows, then a portion
def test_attention_in_32_bits(ops32, n_q, n_kv, d, pt, window, seq_lens, starts):  # noqa: F811
    table, k_pool, v_pool = _paged_setup(seq_lens, pt, n_kv, d, torch.float32, 9)
    k_pool.fill_(float("inf"))                          # rows that no sequence holds must not be read into a sum
    v_pool.fill_(float("inf"))
    keys = [_randn((l, n_kv, d), 30 + s) for s, l in enumerate(seq_lens)]
    vals = [_randn((l, n_kv, d), 40 + s) for s, l in enumerate(seq_lens)]
    positions, q_start = [], [0]
    for s, (l, st) in enumerate(zip(seq_lens, starts)):
        pos = torch.arange(l)
        pages = table[s, (pos // pt).to(DEV)].long()
        k_pool[pages, :, (pos % pt).to(DEV)] = keys[s]
        v_pool[pages, :, (pos % pt).to(DEV)] = vals[s]
        if window:
            table[s, :max(0, st - window + 1) // pt] = -1          # pages the window has passed are gone
        positions += [(s, p) for p in range(st, l)]
        q_start.append(len(positions))
    n = len(positions)
    qkv = _randn((n, (n_q + 2 * n_kv) * d), 50)
    for s in range(len(seq_lens)):                      # a far key that dominates: a wrong page would show
        qkv.view(n, -1, d)[q_start[s], 0] = keys[s][min(3, starts[s]), 0] * 3
    out = torch.full((n, n_q * d), 7.0, device=DEV)
    q_lens = np.diff(q_start)
    i32 = dict(dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(q_start=torch.tensor(q_start, **i32), ctx_len=torch.tensor(seq_lens, **i32), n_seqs=len(seq_lens),
                                max_q_len=int(q_lens.max()), max_ctx_len=max(seq_lens), decode_only=int(q_lens.max()) == 1,
                                fixed_shapes=False, q_lens=q_lens, ctx_lens=np.array(seq_lens), status=torch.zeros(4, **i32))
    cache = types.SimpleNamespace(k_pool=k_pool, v_pool=v_pool, block_table=table, page_tokens=pt)
    scale = 1 / math.sqrt(d)
    assert ops32._attention_f32(ctx, qkv, out, n_q, n_kv, d, scale, window, cache)
    assert ctx.status.tolist() == [0, 0, 0, 0]
    for i, (s, p) in enumerate(positions):
        q = qkv[i].double().view(-1, d)[:n_q]
        want = _ref_attention(q, keys[s][:p + 1].double(), vals[s][:p + 1].double(), n_q, n_kv, scale,
                              max(0, p - window + 1) if window else 0)
        # a score is a sum of d products (|s| <= |q| |k| scale, error d 2^-24 of it), a weight moves by as much relatively;
        # the weighted mean of values moves by twice that of the largest value, plus its own sum's rounding
        s_err = d * 2.0 ** -24 * scale * q.norm(dim=1).max() * keys[s][:p + 1].double().norm(dim=2).max()
        bound = (2 * s_err + (p + 8) * 2.0 ** -23) * vals[s][:p + 1].abs().max().double()
        assert ((out[i].view(n_q, d).double() - want).abs() <= bound).all(), (s, p)


# a position at the start, inside and at the end of a tile of 64 keys; windows that leave it inside the tile and across tiles
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("n_q,n_kv,d", [(4, 2, 128), (3, 1, 64)])
@pytest.mark.parametrize("at,window", [(40, None), (64, None), (127, None), (40, 9), (64, 70), (127, 33)])
def test_a_position_that_is_not_finite_reaches_only_the_rows_that_see_it(ops32, n_q, n_kv, d, at, window, bad):  # noqa: F811
    length, pt = 200, 16
    i32 = dict(dtype=torch.int32, device=DEV)
    qkv = _randn((length, (n_q + 2 * n_kv) * d), 3)
    runs = []
    for pool in (None, 0, 1):
        table, *pools = _paged_setup([length], pt, n_kv, d, torch.float32, 9)
        for i, p in enumerate(pools):
            p.copy_(_randn(p.shape, 10 + i))
        if pool is not None:
            pools[pool][table[0, at // pt], :, at % pt, d // 2] = bad
        ctx = types.SimpleNamespace(q_start=torch.tensor([0, length], **i32), ctx_len=torch.tensor([length], **i32), n_seqs=1,
                                    max_q_len=length, max_ctx_len=length, decode_only=False, fixed_shapes=False,
                                    q_lens=np.array([length]), ctx_lens=np.array([length]), status=torch.zeros(4, **i32))
        cache = types.SimpleNamespace(k_pool=pools[0], v_pool=pools[1], block_table=table, page_tokens=pt)
        out = torch.full((length, n_q * d), 7.0, device=DEV)
        assert ops32._attention_f32(ctx, qkv, out, n_q, n_kv, d, 0.1, window, cache)
        runs.append(out)
    sees = [p for p in range(length) if at <= p and (window is None or at > p - window)]
    others = [p for p in range(length) if p not in sees]
    clean, key, value = runs
    assert torch.isfinite(clean).all()
    assert torch.equal(key[others], clean[others]) and torch.equal(value[others], clean[others])
    column = [h * d + d // 2 for h in range(n_q)]
    assert not torch.isfinite(value[sees][:, column]).any()
    value[:, column] = clean[:, column]
    assert torch.equal(value, clean)


def test_attention_on_pools_of_any_alignment(ops32):  # noqa: F811
    """Pools that do not start on 16 bytes are the any-size kernel's."""
    length, n_q, n_kv, d, pt = 21, 2, 1, 64, 4
    table, k_pool, v_pool = _paged_setup([length], pt, n_kv, d, torch.float32, 9)
    k_pool.copy_(_randn(k_pool.shape, 1))
    v_pool.copy_(_randn(v_pool.shape, 2))
    shifted = [torch.empty(p.numel() + 1, device=DEV)[1:].view(p.shape).copy_(p) for p in (k_pool, v_pool)]
    i32 = dict(dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(q_start=torch.tensor([0, length], **i32), ctx_len=torch.tensor([length], **i32), n_seqs=1,
                                max_q_len=length, max_ctx_len=length, decode_only=False, fixed_shapes=False,
                                q_lens=np.array([length]), ctx_lens=np.array([length]), status=torch.zeros(4, **i32),
                                positions=torch.arange(length, **i32), seq_of_token=torch.zeros(length, **i32))
    qkv, outs = _randn((length, (n_q + 2 * n_kv) * d), 3), []
    for k, v in ((k_pool, v_pool), shifted):
        cache = types.SimpleNamespace(k_pool=k, v_pool=v, block_table=table, page_tokens=pt)
        outs.append(torch.empty((length, n_q * d), device=DEV))
        ops32.attention(ctx, qkv, outs[-1], n_q, n_kv, d, 0.125, None, cache)
    # both within (2 d 2^-24 |q| |k| scale + length 2^-23) of the largest value; |q| |k| scale is below 20 for these
    assert (outs[0] - outs[1]).abs().max() <= 2 * (2 * d * 2.0 ** -24 * 20 + length * 2.0 ** -23) * v_pool.abs().max()


def test_attention_in_32_bits_reports_a_missing_page(ops32):  # noqa: F811
    i32 = dict(dtype=torch.int32, device=DEV)
    for q_len in (1, 2):
        table, k_pool, v_pool = _paged_setup([20], 16, 1, 64, torch.float32, 1)
        table[0, 1] = -1
        ctx = types.SimpleNamespace(q_start=torch.tensor([0, q_len], **i32), ctx_len=torch.tensor([20], **i32), n_seqs=1,
                                    max_q_len=q_len, max_ctx_len=20, decode_only=q_len == 1, fixed_shapes=True,
                                    status=torch.zeros(4, **i32))
        cache = types.SimpleNamespace(k_pool=k_pool, v_pool=v_pool, block_table=table, page_tokens=16)
        out = torch.empty((q_len, 64), device=DEV)
        assert ops32._attention_f32(ctx, _randn((q_len, 192), 1), out, 1, 1, 64, 0.1, None, cache)
        assert ctx.status[0].item() == 2
