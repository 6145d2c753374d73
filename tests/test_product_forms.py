"""Which form a product without a norm around it takes, on the CPU: narrow tiles on single SMs (33 to 128 tokens), tiles of a fitted
width on pairs (from 129), and everything that stays where it was."""
import pytest

from leone_b200.ops.fast import FastKernels


class _Sizes:
    """Stand-in for the library's host-side size queries on 148 SMs."""

    @staticmethod
    def leone_gemm_tc_tiles_token_major(m, n):
        return -(-m // 128) * -(-n // 256)

    @staticmethod
    def leone_gemm_tc_cluster_capacity_token_major(splits):
        return {2: 74, 3: 44, 4: 33, 5: 26, 6: 22, 7: 18, 8: 15}.get(splits, 0)

    @staticmethod
    def leone_gemm_pair_capacity(width, splits):
        return {2: 33, 4: 15}.get(splits, 0)

    @staticmethod
    def leone_gemm_tc_tile(m):
        return min(256, max(16, 1 << (m - 1).bit_length()))

    @staticmethod
    def leone_gemm_tc_cluster_capacity(m, splits):
        return 148 // splits

    @staticmethod
    def leone_gemm_tc_norm_parts(m, n):
        return -(-n // 32)

    @staticmethod
    def leone_gemm_pair_workspace_floats(m, n, width, splits):
        return splits * m * n

    @staticmethod
    def leone_gemm_tc_tiles(m, n):
        return -(-n // 128)

    @staticmethod
    def leone_gemm_tc_scratch(m, tiles, splits, floats, counters):
        pass


@pytest.fixture()
def fast():
    f = FastKernels.__new__(FastKernels)
    f.sm_count = 148
    f.lib = _Sizes()
    f._configure()
    for name in ("use_clusters", "use_token_major", "use_pairs", "use_pair_splits", "use_narrow"):
        setattr(f, name, True)
    return f


def _plan(f, m, n, k, epilogue=0, splits=None, cluster=False, token_major=None, norm_in=False, norm_out=False):
    return f._plan_gemm(m, n, k, epilogue, splits, 0, cluster, token_major, norm_in, norm_out)


SHAPES = [(4096, 2048), (2048, 2048), (12288, 2048), (2048, 6144), (6144, 4096), (4096, 4096), (24576, 4096), (4096, 12288), (1000, 520),
          (16, 64), (45, 128), (151936, 4096), (32, 8)]


@pytest.mark.parametrize("n,k", SHAPES)
def test_widths_are_what_the_kernels_take(fast, n, k):
    for m in (1, 32, 33, 64, 65, 77, 128, 129, 256, 257, 300, 384, 385, 1027, 8193):
        for gated in (False, True) if n % 32 == 0 else (False,):
            step = 32 if gated else 16
            w = fast.narrow_width(m, n, k, gated)
            assert w == 0 or (33 <= m <= 128 and 16 <= w <= 256 and w % step == 0)
            if m > 128:
                w = fast.pair_tile(m, n, k, gated)
                assert 64 <= w <= 256 and w % step == 0
            plan = _plan(fast, m, n, k, 3 if gated else 0)
            assert (plan[0] == 2) == (fast.narrow_width(m, n, k, gated) > 0)
            if m > 128 and fast.pairs_unsplit(m):
                assert plan[:3] == (True, True, 1) and plan[8] == fast.pair_tile(m, n, k, gated)


def test_measured_choices(fast):
    assert 16 <= fast.narrow_width(77, 2048, 2048, False) <= 32 and fast.narrow_width(77, 12288, 2048, True) == 96
    assert fast.narrow_width(77, 2048, 6144, False) == 0            # a long K stays split
    assert fast.narrow_width(77, 151936, 4096, False) == 0 and fast.narrow_width(64, 24576, 4096, True) == 192
    assert fast.pair_tile(256, 2048, 2048, False) == 64 and fast.pair_tile(2048, 24576, 4096, True) >= 224
    assert not fast.pairs_unsplit(128) and fast.pairs_unsplit(129) and fast.pairs_unsplit(300)


def test_norms_are_folded_where_pairs_fit(fast):
    for n, k in ((2048, 2048), (4096, 12288), (6144, 4096)):
        for m in (385, 512, 600, 1027, 2048):
            assert fast.fuses_norm(m, n, k)
            for kw in (dict(norm_in=True), dict(norm_out=True, epilogue=2)):
                plan = _plan(fast, m, n, k, **kw)
                width = fast.pair_width(m, n, False)
                assert plan[:3] == (True, True, 1) and plan[5] == 0 and plan[7] == -(-n // width) == fast.norm_parts(m, n) and plan[8] == width
    # elsewhere as it was: not where tiles of 256 tokens would be half empty and K is split, nor from 33 to 256 tokens
    assert not fast.fuses_norm(300, 4096, 4096) and fast.fuses_norm(300, 640, 64) and not fast.fuses_norm(100, 2048, 2048)
    fast.use_pairs = False
    assert not fast.fuses_norm(400, 4096, 4096)


def test_what_a_caller_asks_for_stays(fast):
    """Forced forms, norms around the product and every switch give the plan they gave without the narrow forms."""
    cases = [dict(splits=1), dict(splits=4, cluster=True), dict(token_major=True), dict(token_major=False), dict(norm_in=True), dict(norm_out=True)]
    for m in (1, 8, 32, 40, 77, 128, 200, 300, 512, 2048):
        for n, k in ((2048, 2048), (4096, 12288), (24576, 4096)):
            for kw in cases:
                fast.use_narrow = True
                got = _plan(fast, m, n, k, **kw)
                fast.use_narrow = False
                assert got == _plan(fast, m, n, k, **kw)
            fast.use_narrow = True
            if m <= 32:
                got = _plan(fast, m, n, k)
                fast.use_narrow = False
                assert got == _plan(fast, m, n, k)
    fast.use_narrow = True
    fast.pair_width_override = 96
    assert _plan(fast, 512, 2048, 2048)[8] == 96
    fast.pair_width_override, fast.pair_split_override = 0, 2
    assert _plan(fast, 512, 2048, 2048)[2] == 2
    fast.pair_split_override, fast.use_pairs = 0, False
    assert _plan(fast, 512, 2048, 2048)[0] is False


@pytest.mark.parametrize("max_tokens,size", [(24, 2048), (200, 2048), (512, 2048), (512, 4096), (1100, 4096), (2048, 2048), (2048, 5120), (3000, 1024)])
def test_a_norms_sums_are_allocated_once(fast, monkeypatch, max_tokens, size):
    """A decode step first, then steps of every size up to the largest: the buffer of the sums of squares stays where it is."""
    import types

    import torch
    from leone_b200.parts.base import DeferredNorm, Runtime
    # as the library has it: 32 weight rows a part for few tokens, tiles of at least 240 for prompts on single SMs
    monkeypatch.setattr(_Sizes, "leone_gemm_tc_norm_parts", staticmethod(lambda m, n: -(-n // (32 if m <= 256 else 240))))
    rt = Runtime("cpu", torch.bfloat16, types.SimpleNamespace(norm_sums_floats=fast.norm_sums_floats), max_tokens)
    at, most = set(), 0
    for m in [*range(1, 33, 5), 32, *range(257, max_tokens, 37), *range(384, max_tokens, 128), *range(385, max_tokens, 128), max_tokens]:
        if m > max_tokens or not fast.fuses_norm(m):
            continue
        d = DeferredNorm(None, None, torch.empty((m, size)), None, 1e-6)
        d.prepare(rt, fast.norm_parts(m, size))
        at.add(d.ss.data_ptr())
        most = max(most, d.ss.numel())
    assert len(at) == 1
    assert fast.norm_sums_floats(max_tokens, size) >= most
