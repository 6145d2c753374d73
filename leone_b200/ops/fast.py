"""The bfloat16 serving kernels: tensor-core products (and tiled attention).

Each call returns ``True`` if it ran and ``False`` if the kernel refuses the
sizes (the caller then uses the any-size kernel).  Refusal is decided on the
host from the kernel's stated limits, never by trying.
"""
from __future__ import annotations

import ctypes
import os
from ctypes import addressof, byref, c_float, c_int, c_longlong

import torch

from ..csrc.build import ensure_built
from .entry_points import EntryPoints


def leading_ones(ctx, q_lens) -> int:
    """How many of a step's first sequences bring one token; counted once a step (a context is made for one step)."""
    n = getattr(ctx, "leading_ones", None)
    if n is None:
        n = 0
        while n < len(q_lens) and q_lens[n] == 1:
            n += 1
        ctx.leading_ones = n
    return n


class FastKernels:
    def __init__(self, device):
        self.device = torch.device(device)
        self.lib = ctypes.CDLL(ensure_built("bf16"))
        self.calls = EntryPoints(self.lib)
        self.sm_count = torch.cuda.get_device_properties(self.device).multi_processor_count
        self._configure()
        self.lib.leone_attention_decode_scratch.restype = ctypes.c_longlong
        self.lib.leone_gemm_pair_workspace_floats.restype = ctypes.c_longlong

    def _configure(self) -> None:
        """The switches and rules of the dispatchers (everything but the device and the library)."""
        self._workspace = None
        self._retired = []
        self.min_scratch_floats = 1 << 20
        self._counters = None
        # LEONE_NO_TENSOR_CORES=1 routes every product to the CUDA-core kernel (for fault finding)
        self.use_tensor_cores = os.environ.get("LEONE_NO_TENSOR_CORES", "0") != "1"
        # LEONE_NO_CLUSTERS=1 sums split-K partial tiles through a workspace instead of inside clusters
        self.use_clusters = os.environ.get("LEONE_NO_CLUSTERS", "0") != "1"
        self._cluster_capacity = {}
        # LEONE_NO_FUSED_NORM=1 keeps every RMSNorm a kernel of its own
        self.fuse_norm = os.environ.get("LEONE_NO_FUSED_NORM", "0") != "1"
        self.fuse_norm_tokens = 32
        # LEONE_NO_TOKEN_MAJOR=1 keeps every product of up to 256 tokens in the swapped form
        # LEONE_NO_DIVIDED_STEPS=1 sends a mixed step's decode rows through the prompt attention kernel too
        self.divide_mixed_steps = os.environ.get("LEONE_NO_DIVIDED_STEPS", "0") != "1"
        self.mixed_decode_rows_from = 1
        self.use_token_major = os.environ.get("LEONE_NO_TOKEN_MAJOR", "0") != "1"
        self.token_major_from = 64         # tokens above which the token-major form is considered
        self.token_major_split_from = 128  # .. and its split along K (up to 128 tokens the swapped form's split measured the same or better)
        self.token_major_fill = 0.6        # of the SMs that its tiles must fill
        self.force_decode_splits = 0       # > 0: every decode attention splits its keys this many ways (kernel_bench sets it)
        # LEONE_NO_FUSED_DECODE=1 keeps q/k norm, rotation and cache write in their own kernel
        self.fuse_decode = os.environ.get("LEONE_NO_FUSED_DECODE", "0") != "1"
        self.max_cluster = 8               # the portable cluster size
        # LEONE_NO_PAIRS=1 keeps prompt-sized products on single SMs (cta_group::1)
        self.use_pairs = os.environ.get("LEONE_NO_PAIRS", "0") != "1"
        self.pairs_from = 129              # tokens from which unsplit products run on pairs
        # LEONE_NO_PAIR_SPLITS=1 leaves the narrow products' split along K to the single-block kernel (only where pairs_unsplit is off)
        self.use_pair_splits = os.environ.get("LEONE_NO_PAIR_SPLITS", "0") != "1"
        self.pair_padding = 0.8            # a pair's half tile against a single block's tile, at most (see in_pairs)
        self.pair_width_override = 0       # > 0: the tile width of every product on pairs (kernel_bench sets it)
        self.pair_split_override = 0       # > 0: pairs per tile of every product on pairs (tests set it)
        # LEONE_NO_NARROW=1 leaves products without a norm around them to the rules from before the unsplit forms: those of 33 to 128
        # tokens (narrow_width) and those from 129 on (pairs_unsplit) to plan_product, which splits K where tiles are few
        self.use_narrow = os.environ.get("LEONE_NO_NARROW", "0") != "1"
        self._pair_widths = {}
        self._plans = {}                   # _gemm's decisions per (sizes, arguments)
        self.decode_cluster_rounds = 1     # rounds of blocks a clustered decode attention may take (kernel_bench sets it)
        # (n, k) -> (splits, cluster): a forced split of an [n x k] product at decode sizes; empty
        # in the product, filled by kernel_bench's sweeps
        self.split_override = {}
        self.status = None
        self._attn_ws = None
        self._pinned_stream = None
        self.use_tiled_attention = os.environ.get("LEONE_NO_TILED_ATTENTION", "0") != "1"
        # LEONE_NO_TC_ATTENTION=1 keeps prompt attention on the mma.sync kernel
        self.use_tc_attention = os.environ.get("LEONE_NO_TC_ATTENTION", "0") != "1"

    def __setattr__(self, name, value):
        # a switch changed (a test, the kernel bench): the remembered decisions may no longer hold
        if not name.startswith("_") and "_plans" in self.__dict__:
            self._plans.clear()
            self._pair_widths.clear()
        object.__setattr__(self, name, value)

    def _stream(self):
        if self._pinned_stream is not None:        # (a handle of 0, the default stream, is a valid pin)
            return self._pinned_stream
        return torch.cuda.current_stream(self.device).cuda_stream

    def pin_stream(self, handle) -> None:
        """The stream every launch goes to until ``pin_stream(None)``: a step looks its stream up
        once, not once per launch (the lookup costs microseconds, a step has hundreds of launches)."""
        object.__setattr__(self, "_pinned_stream", handle)

    # -- split-K scratch ----------------------------------------------------------------
    def _retire(self, tensor) -> None:
        """A scratch buffer that is outgrown is kept, not freed: a captured CUDA graph may have
        its address baked in and will go on using it."""
        if tensor is not None:
            self._retired.append(tensor)

    def token_major_workspace_floats(self) -> int:
        """One 128 x 256 fp32 partial tile per block of a round."""
        return self.sm_count * 128 * 256

    def scratch_bytes(self) -> int:
        """What these ops allocate for themselves at most: the split products' workspace and the
        split decode attention's partial results."""
        return 4 * (max(self.min_scratch_floats, self.token_major_workspace_floats()) + self.min_scratch_floats)

    def _scratch(self, floats: int, counters: int):
        if self._workspace is None or self._workspace.numel() < floats:
            self._retire(self._workspace)
            self._workspace = torch.empty(max(floats, self.min_scratch_floats), dtype=torch.float32,
                                          device=self.device)
        if self._counters is None or self._counters.numel() < counters:
            self._retire(self._counters)
            self._counters = torch.zeros(max(counters, 4096), dtype=torch.int32, device=self.device)
        return self._workspace, self._counters

    def cluster_capacity(self, m: int, splits: int) -> int:
        """Clusters of ``splits`` blocks of the GEMM for ``m`` tokens that fit on the device at once."""
        key = (int(self.lib.leone_gemm_tc_tile(m)) if m <= 256 else 0, splits)
        if key not in self._cluster_capacity:
            self._cluster_capacity[key] = int(self.lib.leone_gemm_tc_cluster_capacity(m, splits))
        return self._cluster_capacity[key]

    def choose_splits(self, m: int, n: int, k: int):
        """How to split K: ``(splits, full_tiles, cluster)``; tiles before ``full_tiles`` are not split.

        Fewer tiles than SMs: every tile is split, and its splits form a thread-block cluster that
        sums the partial tiles through distributed shared memory.  The most splits (up to 8) win
        that keep the blocks within two thirds of the block slots: more blocks keep more bytes in
        flight, but the last third is what lets the next kernels' blocks start early and fetch
        their first weights while this product is still running (measured on the decode step:
        filling every slot was slower than leaving the product unsplit).  More tiles than SMs:
        only a small remainder of tiles (under a quarter of the SMs) is split, through a
        workspace, so that those few tiles do not cost a round of their own; such a unit keeps
        at least 12 k-blocks.  Prompt-sized M is never split."""
        tiles = int(self.lib.leone_gemm_tc_tiles(m, n))
        if m > 256:
            return 1, tiles, False
        k_blocks = -(-k // 64)
        sms = self.sm_count
        if (n, k) in self.split_override:
            s, cluster = self.split_override[(n, k)]
            return (s, 0, cluster) if s > 1 else (1, tiles, False)
        if tiles < sms:
            slots = sms * (2 if m <= 64 else 1)
            if self.use_clusters:
                for s in (8, 7, 6, 5, 4, 3, 2):
                    if tiles * s <= slots * 2 // 3 and k_blocks // s >= 4 and s <= self.max_cluster and self.cluster_capacity(m, s) > 0:
                        return s, 0, True
            s = max(1, min(sms // tiles, k_blocks // 12, 8))
            return (s, 0, False) if s > 1 else (1, tiles, False)
        rem = tiles % sms
        if rem == 0 or rem * 4 > sms:
            return 1, tiles, False
        s = min(sms // rem, k_blocks // 12, 8)
        return (s, tiles - rem, False) if s > 1 else (1, tiles, False)

    def token_major(self, m: int, n: int) -> bool:
        """Which form of the product runs: tokens on the MMA's 128-row side and 256 weight rows
        per tile (True), or weights on that side and the tokens as the tile's width (False).
        Always above 256 tokens.  From 65 to 256 tokens too when the token-major tiles fill
        at least ``token_major_fill`` of the SMs and at most two rounds of them (the gate/up
        product of a wide feed-forward): the swapped form re-reads the whole token operand for
        every 128 weight rows, twice the bytes of the weights at 256 tokens (gate/up of the 8B
        shape: 65 µs against 49 at 128 tokens, 100 against 68 at 256).  With fewer tiles the
        swapped form's split along K keeps more SMs busy; with many more (an output head, whose
        time is the fp32 logits it writes) the swapped form measured a few percent faster."""
        if m > 256:
            return True
        if m <= self.token_major_from or not self.use_token_major:
            return False
        tiles = int(self.lib.leone_gemm_tc_tiles_token_major(m, n))
        return self.token_major_fill * self.sm_count <= tiles <= 2 * self.sm_count

    def in_pairs(self, m: int, n: int = 0, k: int = 0) -> bool:
        """Whether an unsplit product of ``m`` tokens with a norm around it runs on pairs of SMs (tiles of 256 tokens,
        the width chosen by :meth:`pair_width`; one without a norm: :meth:`pairs_unsplit`): from 129 tokens on, except from 257 to 384
        tokens, where the second of two tiles of 256 would be half empty and the single-block
        kernel's three tiles of 128 measured faster (gate/up at 384 tokens 62.3 us against 67.2;
        at 640 tokens three pairs already beat five single tiles, 95.9 against 105.6).  With
        ``n`` and ``k``: whether this ``[n x k]`` product does where :meth:`pairs_unsplit` is
        switched off; the narrow products of a layer are then split along K up to about 600 tokens."""
        if n and k and self.token_major_split(m, n, k) > 1:
            return self.pair_split(m, n, k) > 1
        return self._pairs_fit(m)

    def _pairs_fit(self, m: int) -> bool:
        return self.use_pairs and m >= self.pairs_from and 2 * -(-m // 256) * self.pair_padding <= -(-m // 128)

    def pair_split(self, m: int, n: int, k: int) -> int:
        """Pairs of SMs per tile of a narrow product (one that the single-block kernel would split
        along K), asked only where :meth:`pairs_unsplit` is switched off (the times below are from before its epilogue and are kept as
        the reason of this rule): 4 or 2 pairs share the k-blocks of a tile of 256 tokens x 256 weight rows when
        their clusters of 8 or 4 blocks are all resident at once and a pair keeps at least 8
        k-blocks; 1: not split on pairs.  Only where the pairs can split as many ways as the single
        blocks would: with the same number of splits the pairs' k-loop wins (down at 512 tokens
        50.3 us against 56.6, qkv at 256 tokens 23.4 against 25.3), against four single-block
        splits two pairs lose (o_proj at 256 tokens 25.1 us against 18.8, down 46.5 against 37.4).
        Also from 257 to 384 tokens, where unsplit products stay in single blocks (down at 320
        tokens 48.6 us against 55.4)."""
        if self.pair_split_override:
            return self.pair_split_override
        if not (self.use_pair_splits and self.use_clusters and self.use_pairs and m >= self.pairs_from) or \
                self.token_major_split(m, n, k) == 1:
            return 1
        tiles, k_blocks = -(-n // 256) * -(-m // 256), -(-k // 64)
        single = self.token_major_split(m, n, k)
        for s in (4, 2):
            if tiles * s <= self.sm_count // 2 and k_blocks // s >= 8 and tiles <= self._pair_capacity(s):
                return s if s >= single else 1
        return 1

    def _pair_capacity(self, splits: int) -> int:
        key = ("pairs", splits)
        if key not in self._cluster_capacity:
            self._cluster_capacity[key] = int(self.lib.leone_gemm_pair_capacity(256, splits))
        return self._cluster_capacity[key]

    def pair_width(self, m: int, n: int, swiglu: bool) -> int:
        """Weight rows per tile of a product on pairs of SMs: the width whose tiles cost the
        fewest rounds over the pairs.  A tile's k-block costs what the copy of its operands
        into a block's shared memory takes (128 token rows beside width / 2 weight rows: the
        k-loop runs at the rate of those copies, 32 KB in 0.36 us, at every width that was
        measured); of two widths within 1 percent the wider one stays."""
        if self.pair_width_override:
            return self.pair_width_override
        key = (-(-m // 256), n, bool(swiglu))
        if key not in self._pair_widths:
            pairs, best = self.sm_count // 2, None
            for w in range(256, 31, -32 if swiglu else -16):
                rounds = -(-(-(-n // w) * key[0]) // pairs)
                cost = rounds * (0.18 + 0.0007 * w)
                if best is None or cost < 0.99 * best[0]:
                    best = (cost, w)
            self._pair_widths[key] = best[1]
        return self._pair_widths[key]

    def token_major_split(self, m: int, n: int, k: int) -> int:
        """Splits along K of the token-major form, summed inside thread-block clusters (1: none).
        A product whose token-major tiles fill at most half of the SMs (the narrow products of a
        layer between 65 and about 600 tokens) is split so that tiles x splits blocks fill them;
        a split keeps at least 8 k-blocks.  Such a product takes no folded norm.  Products without one that :meth:`narrow_width` or
        :meth:`pairs_unsplit` takes do not ask; from 257 to 384 tokens, where no pairs fit a norm, the answer decides whether
        the norm is folded (:meth:`fuses_norm`)."""
        if not (self.use_clusters and self.use_token_major) or m <= self.token_major_split_from:
            return 1
        tiles = int(self.lib.leone_gemm_tc_tiles_token_major(m, n))
        if tiles * 2 > self.sm_count:
            return 1
        k_blocks = -(-k // 64)
        # all clusters must be resident at once: a cluster needs its blocks' SMs free in one GPC
        # at the same moment, and a grid that needs a second round of clusters was measured at
        # twice the time (the occupancy query's count of resident clusters is what holds)
        for s in range(min(8, self.sm_count // tiles, self.max_cluster), 1, -1):
            if k_blocks // s >= 8 and tiles <= self._token_major_capacity(s):
                return s
        return 1

    def _token_major_capacity(self, splits: int) -> int:
        key = ("token-major", splits)
        if key not in self._cluster_capacity:
            self._cluster_capacity[key] = int(self.lib.leone_gemm_tc_cluster_capacity_token_major(splits))
        return self._cluster_capacity[key]

    def narrow_width(self, m: int, n: int, k: int, gated: bool) -> int:
        """Weight rows per tile of an unsplit product on single SMs (gemm_narrow.cu) where that is the best form, else 0: from 33
        to 128 tokens, if the estimate below is under that of the swapped form's split along K.  Both in us, fitted to products of
        40, 77 and 128 tokens with 11 matrices of 2048 x 2048 to 24576 x 4096.  Narrow tiles: 3.2, 0.012 for every tile past 64, and
        for every round of tiles over the SMs and k-block 0.12 + 0.0007 a weight row (what the thread that issues the MMAs
        takes); no less than the weights at 6 MB a us (24576 x 4096 at 64 tokens 36.8 us against 40.7 split).  The split: 7.3 + 0.165 a
        MB of weights up to 64 tokens, 9.2 + 0.215 above (partial tiles of 128 columns are exchanged).  So K decides: 2048 x 2048 at 77 tokens 7.5 us against 10.3,
        12288 x 2048 11.6 against 18.5, 2048 x 6144 16.0 against 13.7 (stays split).  Not for an output head, whose time is its
        logits."""
        if not self.use_narrow or not 32 < m <= 128:
            return 0
        k_blocks, mb, best = -(-k // 64), n * k * 2e-6, None
        if n > 256 * self.sm_count:
            return 0
        for w in range(256, 15, -32 if gated else -16):
            tiles = -(-n // w)
            cost = 3.2 + 0.012 * max(0, min(tiles, self.sm_count) - 64) + -(-tiles // self.sm_count) * k_blocks * (0.12 + 0.0007 * w)
            if best is None or cost < 0.99 * best[0]:
                best = (cost, w)
        split = 7.3 + 0.165 * mb if m <= 64 else 9.2 + 0.215 * mb
        return best[1] if max(best[0], 3.2 + mb / 6) < split else 0

    def pairs_unsplit(self, m: int) -> bool:
        """Whether a product that carries no norm runs unsplit on pairs of SMs with tiles of :meth:`pair_tile`'s width: from 129 tokens
        on.  A split along K is faster alone where K is long (4096 x 12288 at 256 tokens 35.1 us against 39.2), but its exchange
        holds up the next kernel's start: a layer's products with their norms take 56.3 us unsplit and 59.3 with only the
        2048 x 6144 one split (129 tokens; 58.5 and 62.0 at 256, 69.3 and 71.1 at 400), and 119.5 and 116.5 in the 8B shape."""
        return self.use_pairs and m >= self.pairs_from and not self.pair_split_override

    def pair_tile(self, m: int, n: int, k: int, gated: bool) -> int:
        """Weight rows per tile of an unsplit product on pairs of SMs that carries no norm around it: the width of the lowest
        estimate, in us: 2.3 + 0.016 a weight row (start, and the epilogue of the last tile), and for every round of tiles over the
        pairs and k-block the MMAs' time (0.0013 a weight row), what the issuing thread takes (0.18), or the operands' way from
        the L2 (18 MB a us), whichever is longest.  Fitted to 56 products of 144 to 2,048 tokens and 2,048 to 24,576 weight rows, measured
        on 7 to 11 widths each: its width is 0.3 percent slower than the best of them on average, 5.4 at most.  Unlike
        :meth:`pair_width` it knows K: short products take narrow tiles for the sake of their epilogue (2048 x 2048 at 256
        tokens: 8.9 us at 64 rows, 17.5 at 256)."""
        if self.pair_width_override:
            return self.pair_width_override
        pairs, m_pairs, k_blocks, best = self.sm_count // 2, -(-m // 256), -(-k // 64), None
        for w in range(256, 63, -32 if gated else -16):
            tiles = -(-n // w) * m_pairs
            block = max(0.18, 0.0013 * w, min(tiles, pairs) * (256 + w) * 128 / 18e6)
            cost = 2.3 + 0.016 * w + -(-tiles // pairs) * k_blocks * block
            if best is None or cost < 0.99 * best[0]:
                best = (cost, w)
        return best[1]

    def plan_product(self, m: int, n: int, k: int):
        """``(token_major, splits, full_tiles, cluster)`` for a product without a folded norm that :meth:`narrow_width` and
        :meth:`pairs_unsplit` leave: decode sizes, the output head up to 128 tokens, everything where those are switched off."""
        if self.in_pairs(m, n, k):
            return True, 1, 0, False                 # on pairs of SMs (_gemm takes them where nothing is forced)
        s = self.token_major_split(m, n, k)
        if s > 1:
            return True, s, 0, True
        if self.token_major(m, n):
            return True, 1, 0, False
        return (False, *self.choose_splits(m, n, k))

    def _gemm(self, x, w, out, epilogue, residual, n_rows, splits=None, full_tiles=0, cluster=False,
              norm_in=None, norm_out=None, token_major=None, gate_shape=None, bias=None) -> bool:
        """``splits=None`` lets :meth:`choose_splits` decide; otherwise tiles from
        ``full_tiles`` on are split ``splits`` ways, summed through a workspace or, with
        ``cluster``, inside a thread-block cluster.

        ``norm_out=(xn, weight, ss)``: the product (fp32 output) also leaves
        ``xn = bf16(out * weight)`` and the partial sums of ``out^2`` in ``ss`` ``[parts, m]``
        for the RMSNorm that follows it; ``norm_in=(ss, parts, eps)``: ``x`` is such an ``xn``
        and every output row is scaled by the norm's ``rsqrt(mean + eps)``."""
        m, k = x.shape
        key = (m, n_rows, k, epilogue, splits, full_tiles, cluster, token_major, norm_in is not None,
               norm_out is not None)
        plan = self._plans.get(key)
        if plan is None:
            plan = self._plans[key] = self._plan_gemm(*key)
        return self._launch_gemm(plan, x, x.stride(0), w, w.stride(0), out, out.stride(0), epilogue, residual, m, n_rows, k, norm_in,
                                 norm_out, gate_shape, bias)

    def _product(self, x, w, out, epilogue, residual, norm_in, norm_out, gate_shape=None) -> bool:
        """A product with a prepared matrix in the form that the rules choose; False if it cannot run on tensor cores."""
        weight = w.weight
        m, k = x.shape
        ldx, ldw = x.stride(0), weight.stride(0)
        if not self.use_tensor_cores or x.dtype != torch.bfloat16 or (k | ldx | ldw) & 7 or (x.data_ptr() | weight.data_ptr()) & 15:
            return False
        n_rows = w.out_features
        key = (m, n_rows, k, epilogue, norm_in is not None, norm_out is not None)
        plan = self._plans.get(key)
        if plan is None:
            plan = self._plans[key] = self._plan_gemm(m, n_rows, k, epilogue, None, 0, False, None, norm_in is not None,
                                                      norm_out is not None)
        return self._launch_gemm(plan, x, ldx, weight, ldw, out, out.stride(0), epilogue, residual, m, n_rows, k, norm_in, norm_out,
                                 gate_shape, w.bias)

    def _launch_gemm(self, plan, x, ldx, w, ldw, out, ldc, epilogue, residual, m, n_rows, k, norm_in, norm_out, gate_shape, bias) -> bool:
        pairs, token_major, splits, full_tiles, cluster, ws_floats, ws_counters, parts, width = plan
        ws = ct = None
        if ws_floats or ws_counters:
            ws, ct = self._scratch(ws_floats, ws_counters)
            if not ws_counters:
                ct = None
        if norm_out is not None and norm_out[2].shape[0] != parts:
            raise ValueError(f"the sums of squares have {norm_out[2].shape[0]} parts, this product leaves {parts}")
        no = (None, None, None, 0) if norm_out is None else \
            (norm_out[0], norm_out[1], norm_out[2], norm_out[0].stride(0))
        ni = (None, 0, 0.0) if norm_in is None else (norm_in[0], int(norm_in[1]), float(norm_in[2]))
        # the gate's shape of the gated epilogue: four host floats, or null for SwiGLU
        shape = None if gate_shape is None else (c_float * 4)(*[float(v) for v in gate_shape])
        gs = None if shape is None else addressof(shape)
        if pairs == 2:
            # unsplit on single SMs, tiles as narrow as fill the chip (gemm_narrow.cu)
            code = self.calls.leone_gemm_narrow(x, w, out, residual, m, n_rows, k, ldx, ldw, ldc, epilogue,
                                                width, self.status, self.sm_count, *ni, gs, bias, self._stream())
            if code != 0:
                raise RuntimeError(f"gemm_narrow refused or failed with code {code} for m={m} n={n_rows} k={k} width={width}")
            return True
        if pairs:
            # pairs of SMs on tiles of 256 tokens (gemm_pair.cu)
            code = self.calls.leone_gemm_pair(x, w, out, residual, m, n_rows, k,
                                            ldx, ldw, ldc, epilogue, width, splits, ws,
                                            self.status, self.sm_count, *no, *ni, gs, bias, self._stream())
            if code != 0:
                raise RuntimeError(f"gemm_pair refused or failed with code {code} for m={m} n={n_rows} k={k}")
            return True
        code = self.calls.leone_gemm_tc(x, w, out, residual, m, n_rows, k,
                                      ldx, ldw, ldc, epilogue, splits,
                                      full_tiles, ws, ct, self.status, self.sm_count,
                                      1 if cluster else 0, 1 if token_major else 0, *no, *ni, gs, bias, self._stream())
        if code != 0:
            raise RuntimeError(f"gemm_tc refused or failed with code {code} for m={m} n={n_rows} k={k} "
                               f"splits={splits} cluster={cluster} token_major={token_major}")
        return True

    def _plan_gemm(self, m, n_rows, k, epilogue, splits, full_tiles, cluster, token_major, has_norm_in, has_norm_out):
        """What :meth:`_gemm` does for one combination of sizes and arguments (kept per combination;
        every change of a switch of this object forgets the plans): ``(pairs, token_major, splits,
        full_tiles, cluster, workspace floats, counters, parts of a folded norm's sums, tile width
        on pairs or of narrow tiles)``.  ``pairs`` is 2 for narrow tiles on single SMs; on pairs, ``splits`` is the number of pairs
        per tile."""
        no_norm = not has_norm_in and not has_norm_out
        if token_major is None and splits is None and no_norm and not cluster:
            width = self.narrow_width(m, n_rows, k, epilogue == 3)
            if width:
                return 2, True, 1, 0, False, 0, 0, 0, width
            if self.use_narrow and self.pairs_unsplit(m):
                return True, True, 1, 0, False, 0, 0, self.norm_parts(m, n_rows, True), self.pair_tile(m, n_rows, k, epilogue == 3)
        # on pairs of SMs unless the caller forces another form
        pairs = token_major is None and splits in (None, 1) and not cluster and \
            (self.in_pairs(m, n_rows, k) or (not no_norm and self._pairs_fit(m)))
        if pairs:
            ps = self.pair_split(m, n_rows, k) if no_norm else 1
            width, floats = self.pair_width(m, n_rows, epilogue == 3), 0
            if ps > 1:
                width = 256
                floats = max(self.token_major_workspace_floats(),
                             int(self.lib.leone_gemm_pair_workspace_floats(m, n_rows, width, ps)))
            return True, True, ps, 0, False, floats, 0, self.norm_parts(m, n_rows, True), width
        if token_major is None and splits is None and no_norm:
            token_major, splits, full_tiles, cluster = self.plan_product(m, n_rows, k)
        token_major = bool(token_major) or m > 256
        if token_major and not cluster:
            splits, full_tiles = 1, 0
        elif splits is None:
            splits, full_tiles, cluster = self.choose_splits(m, n_rows, k)
        floats = counters = 0
        if splits > 1 and not cluster:
            tiles = int(self.lib.leone_gemm_tc_tiles(m, n_rows))
            f, c = c_longlong(0), c_int(0)
            self.lib.leone_gemm_tc_scratch(m, max(tiles - full_tiles, 0), splits, byref(f), byref(c))
            floats, counters = f.value, c.value
        elif splits > 1 and token_major:
            # the token-major form's partial tiles (128 tokens x 256 weight rows, fp32) cross
            # between the blocks of a cluster through the workspace
            # (one round of blocks at most, so the largest request is asked for at once and the
            # buffer never grows with the step's size)
            floats = self.token_major_workspace_floats()
        return False, token_major, splits, full_tiles, bool(cluster), floats, counters, \
            self.norm_parts(m, n_rows, False), 0

    def fuses_norm(self, m: int, n: int = 0, k: int = 0) -> bool:
        """Whether the products of ``m`` tokens carry an RMSNorm between them: decode-sized steps
        (up to 32 tokens; from there to 256 the extra work in the two epilogues was measured to
        cost more than the norm kernel it replaces) and prompt-sized ones (over 256 tokens,
        where a thread owns a token row and the sums are its own).  With ``n`` and ``k``: whether
        this ``[n x k]`` product does; one that is split in the token-major form does not, and where an unsplit one fits pairs of
        SMs (:meth:`in_pairs`) none is split for it (a step of 1,027 tokens on the 1.7B
        shape 5.80 ms with norm kernels, 5.57 without)."""
        if not (self.use_tensor_cores and self.fuse_norm and (0 < m <= self.fuse_norm_tokens or m > 256)):
            return False
        return self._pairs_fit(m) or not (n and k and self.token_major_split(m, n, k) > 1)

    def norm_parts(self, m: int, n: int, pairs=None) -> int:
        """Parts of the sums of squares that a product of ``m`` tokens with ``n`` outputs leaves
        for the norm after it: on pairs of SMs (``pairs=None``: where the dispatcher takes them
        for an unsplit product) one per tile of weight rows, else what the single-block kernel
        leaves."""
        if self.in_pairs(m) if pairs is None else pairs:
            return -(-n // self.pair_width(m, n, False))
        return int(self.lib.leone_gemm_tc_norm_parts(m, n))

    def norm_sums_floats(self, max_tokens: int, n: int) -> int:
        """The most floats that products with ``n`` outputs of up to ``max_tokens`` tokens leave for the norm after them
        (:meth:`norm_parts` times the tokens).  Not the parts of the largest step: one of 512 tokens with 2,048 outputs leaves 32, one
        of 2,048 tokens 9.  The parts are the same for up to 32 tokens and for every 128 from there on."""
        key = ("sums", max_tokens, n)
        if key not in self._pair_widths:
            steps = [min(max_tokens, self.fuse_norm_tokens), *range(384, max_tokens, 128), max_tokens]
            self._pair_widths[key] = max((m * self.norm_parts(m, n) for m in steps if self.fuses_norm(m)), default=0)
        return self._pair_widths[key]

    def linear(self, x, w, out, epilogue, residual, norm_in=None, norm_out=None) -> bool:
        return self._product(x, w, out, epilogue, residual, norm_in, norm_out)

    # -- gate/up --------------------------------------------------------------------------
    def prepare_gate_up(self, gate, up, gate_bias=None, up_bias=None):
        from .cuda import PreparedMatrix
        inter, hidden = gate.shape
        if gate.dtype == torch.bfloat16 and inter % 16 == 0 and hidden % 8 == 0 and self.use_tensor_cores:
            # groups of 32 rows: 16 gate rows, then the 16 up rows of the same columns
            stacked = torch.stack([gate.view(inter // 16, 16, hidden), up.view(inter // 16, 16, hidden)],
                                  dim=1).reshape(2 * inter, hidden).contiguous()
            bias = None
            if gate_bias is not None:
                bias = torch.stack([gate_bias.view(inter // 16, 16), up_bias.view(inter // 16, 16)], dim=1).reshape(2 * inter)
            m = PreparedMatrix(stacked, bias)
            m.gate_up_layout = "interleaved16"
            return m
        m = PreparedMatrix(torch.cat([gate, up], dim=0).contiguous(),
                           None if gate_bias is None else torch.cat([gate_bias, up_bias]))
        m.gate_up_layout = "stacked"
        return m

    def linear_swiglu(self, x, w, out, norm_in=None, gate_shape=None) -> bool:
        if getattr(w, "gate_up_layout", None) != "interleaved16":
            return False
        return self._product(x, w, out, 3, None, norm_in, None, gate_shape)

    # -- attention ------------------------------------------------------------------------
    def decode_splits(self, n_seqs: int, n_kv: int, g: int, max_ctx: int) -> int:
        """Splits of the key range.  Two blocks fit an SM; the cost of a choice is its number of
        rounds over those slots times the share of the keys a block walks, plus a little per
        split for the merge (since the partial results are pushed into the finishing block the
        merge costs next to nothing: batch 1 at 2,048 keys 9.7 / 9.1 / 8.6 us for six / seven /
        eight splits, at 16,384 keys 50 / 39 us for six / eight), plus a fixed charge when the
        splits cannot merge inside clusters
        (scratch, a merge kernel and the q/k preparation in a kernel of its own: a fixed part,
        measured at batch 64: one split 101 us, two to four 109-112, and at batch 20: one fused
        split 50.0 us, seven splits 52.1; and a fifth of the walk, measured at batches 160 to 224:
        one fused split 242 / 289 / 326 us, three to six splits 250 / 309 / 366; at batch 48
        three splits are still the better choice, 91 us against 97).  The fixed parts were
        measured at 2,048 keys and are so many microseconds whatever the context, so in units of
        a walk they shrink as the context grows: at batch 1 sixteen to thirty-two unclustered
        splits beat eight clustered ones from 16,384 keys on (33 against 40 us; at 32,768 keys 46
        against 75), at 8,192 keys they do not (24.5 against 22.4); the share of the walk shrinks
        too, with the root of that factor (a short block's own start and end are what it stands
        for: batch 16 at 32,768 keys, nine unclustered splits 351 us against 378 for two
        clustered ones).  A split keeps at least 128 keys."""
        if self.force_decode_splits:
            return self.force_decode_splits
        blocks = n_seqs * n_kv * (-(-g // 16))
        slots = 2 * self.sm_count
        best, best_cost = 1, None
        fixed = 2048.0 / max(max_ctx, 128)        # the charges that do not grow with the keys, in walks
        for s in range(1, min(32, max(1, max_ctx // 128)) + 1):
            clustered = self.use_clusters and s <= 8 and blocks * s <= self._decode_cluster_slots()
            walk = -(-(blocks * s) // slots) / s
            cost = walk + fixed * (0.01 * s + (0.0 if s == 1 or clustered else 0.3)) + \
                (0.0 if s == 1 or clustered else 0.2 * fixed ** 0.5 * walk)
            if best_cost is None or cost < best_cost - 1e-9:
                best, best_cost = s, cost
        return best

    def attention_supported(self, dtype, n_q, n_kv, d, row_stride) -> bool:
        return (self.use_tiled_attention and dtype == torch.bfloat16 and d % 16 == 0 and d <= 128
                and n_q // n_kv <= 64 and row_stride % 8 == 0)

    def decode_fusable(self, ctx, dtype, n_q, n_kv, d, row_stride) -> bool:
        """True if a decode step's attention runs as clusters that can also do the q/k norm,
        the rotation and the cache write."""
        return (self.attention_supported(dtype, n_q, n_kv, d, row_stride) and self.fuse_decode
                and ctx.decode_only and d in (64, 128)
                and self.decode_in_clusters(ctx.n_seqs, n_kv, n_q // n_kv, ctx.max_ctx_len))

    def decode_in_clusters(self, n_seqs: int, n_kv: int, g: int, max_ctx: int) -> bool:
        """Whether a decode step runs the kernel whose splits merge inside thread-block clusters
        (and which can do the q/k preparation itself): with one split, or when all blocks are
        resident at once.  With several rounds of blocks, clusters (which need all their
        blocks' slots free in one GPC at the same moment) were measured slower than scratch
        and a merge kernel."""
        splits = self.decode_splits(n_seqs, n_kv, g, max_ctx)
        blocks = n_seqs * n_kv * (-(-g // 16)) * splits
        return self.use_clusters and (splits == 1 or (splits <= 8 and blocks <= self._decode_cluster_slots()))

    def _decode_cluster_slots(self) -> int:
        """Blocks of the decode attention that clusters may count on at once: nine tenths of the
        two per SM (a cluster needs its blocks' slots in one GPC, and the GPCs are not all the same
        size: 96 clusters of three, 288 of 296 slots, measured 42.7 us at batch 12 where 96
        clusters of two take 33.9 us; 64 clusters of four, 256 slots, are the best choice at
        batch 8)."""
        return 2 * self.sm_count * 9 // 10 * self.decode_cluster_rounds

    def leading_decode_rows(self, ctx) -> int:
        """In a mixed step, how many sequences at the front of the batch bring a single token
        (the scheduler puts decode rows first).  Their attention runs on the decode kernel
        (which streams a sequence's keys once for all its heads) and the rest on the prompt
        kernel, which would spend a 128-row tile on each of them.  0: do not divide the step."""
        q_lens = getattr(ctx, "q_lens", None)
        if ctx.decode_only or getattr(ctx, "fixed_shapes", False) or q_lens is None or not self.divide_mixed_steps:
            return 0
        n = leading_ones(ctx, q_lens)
        return n if self.mixed_decode_rows_from <= n < len(q_lens) else 0

    def attention(self, ctx, qkv, out, n_q, n_kv, d, scale, window, cache, fuse=None) -> bool:
        if not self.attention_supported(qkv.dtype, n_q, n_kv, d, qkv.stride(0)):
            return False
        bt = cache.block_table
        args = (qkv, out, n_q, n_kv, d, scale, window, cache)
        if ctx.decode_only:
            self._attention_decode(*args, ctx.q_start, ctx.ctx_len, bt, ctx.n_seqs, ctx.max_ctx_len, ctx.status, fuse,
                                   getattr(ctx, "seq_order", None))
            return True
        if fuse is not None:
            raise RuntimeError("fused q/k preparation is a decode-step feature")
        n_dec = self.leading_decode_rows(ctx)
        if n_dec:
            self._attention_decode(*args, ctx.q_start[:n_dec + 1], ctx.ctx_len[:n_dec], bt[:n_dec], n_dec,
                                   int(ctx.ctx_lens[:n_dec].max()), ctx.status, None, getattr(ctx, "seq_order", None))
            self._attention_prompt(*args, ctx.q_start[n_dec:], ctx.ctx_len[n_dec:], bt[n_dec:], ctx.n_seqs - n_dec,
                                   int(ctx.q_lens[n_dec:].max()), ctx.status)
        else:
            self._attention_prompt(*args, ctx.q_start, ctx.ctx_len, bt, ctx.n_seqs, ctx.max_q_len, ctx.status)
        return True

    def _attention_decode(self, qkv, out, n_q, n_kv, d, scale, window, cache, q_start, ctx_len, bt, n_seqs,
                          max_ctx, status, fuse, order=None) -> None:
        """Sequences with one query token each (row ``q_start[s]``); ``order``: these sequences, the longest first."""
        if order is not None and order.numel() != n_seqs:
            raise ValueError(f"an order of {order.numel()} sequences for {n_seqs}")
        g = n_q // n_kv
        kp, vp = cache.k_pool, cache.v_pool
        common = (qkv, qkv.stride(0), out, out.stride(0), kp, vp, bt,
                  bt.stride(0), q_start, ctx_len, n_seqs)
        splits = self.decode_splits(n_seqs, n_kv, g, max_ctx)
        if self.decode_in_clusters(n_seqs, n_kv, g, max_ctx):
            # the splits of a (sequence, KV head) merge inside a cluster; optionally the
            # kernel norms and rotates q and the new k and writes the cache itself
            fz = (0, None, None, 0.0, None, 0, 0, 0)
            if fuse is not None:
                rope = fuse["rope"]
                fz = (1, fuse["q_w"], fuse["k_w"], float(fuse["eps"]), rope,
                      rope.shape[0] if rope is not None else 0, 1 if fuse["write_cache"] else 0,
                      1 if fuse.get("pairing", "half_split") == "adjacent" else 0)
            code = self.calls.leone_attention_decode_cluster_ordered(
                *common, n_q, n_kv, d, float(scale), int(window or 0), cache.page_tokens,
                kp.shape[0], splits, *fz, order, status, self._stream())
        else:
            if fuse is not None:
                raise RuntimeError("fused decode attention asked for where decode_fusable() is false")
            scratch = None
            if splits > 1:
                need = self.lib.leone_attention_decode_scratch(n_seqs, n_q, d, splits)
                scratch = self._attn_scratch(need)
            code = self.calls.leone_attention_decode(
                *common, n_q, n_kv, d, float(scale), int(window or 0), cache.page_tokens,
                kp.shape[0], splits, scratch, status, self._stream())
        if code != 0:
            raise RuntimeError(f"decode attention refused or failed with code {code}")

    def _attention_prompt(self, qkv, out, n_q, n_kv, d, scale, window, cache, q_start, ctx_len, bt, n_seqs,
                          max_q_len, status) -> None:
        """Sequences with any number of query tokens (rows ``q_start[s] .. q_start[s + 1]``)."""
        g = n_q // n_kv
        kp, vp = cache.k_pool, cache.v_pool
        # head sizes 64 and 128 run on tcgen05; the others on the mma.sync kernel
        ldo = out.stride(0)
        tc = self.use_tc_attention and d in (64, 128) and g <= 128 and ldo % 8 == 0
        entry = self.calls.leone_attention_prefill_pingpong if tc else self.calls.leone_attention_prefill
        code = entry(qkv, qkv.stride(0), out, ldo, kp, vp, bt, bt.stride(0), q_start, ctx_len, n_seqs, max_q_len, n_q, n_kv, d,
                     float(scale), int(window or 0), cache.page_tokens, kp.shape[0], status, self._stream())
        if code != 0:
            raise RuntimeError(f"prompt attention refused or failed with code {code}")

    def attention_rules(self, ctx, qkv, out, n_q, n_kv, d, scale, window, chunk, weights, bias, cache) -> bool:
        """Prompt portions and mixed steps of an attention layer with another mask (``chunk``) or
        weight rule (``weights``: 0 softmax, 1 softmax with a silent member of score 0, 2 sigmoid
        with a ``bias`` per head) on the tcgen05 prompt kernel: head sizes 64 and 128 with values
        as wide as keys.  False: not this kernel's case."""
        g = n_q // n_kv
        if not (self.attention_supported(qkv.dtype, n_q, n_kv, d, qkv.stride(0)) and self.use_tc_attention
                and d in (64, 128) and g <= 128 and out.stride(0) % 8 == 0 and not ctx.decode_only):
            return False
        kp, vp, bt = cache.k_pool, cache.v_pool, cache.block_table
        code = self.calls.leone_attention_prefill_pingpong_rules(
            qkv, qkv.stride(0), out, out.stride(0), kp, vp, bt, bt.stride(0),
            ctx.q_start, ctx.ctx_len, ctx.n_seqs, ctx.max_q_len, n_q, n_kv, d, float(scale),
            int(window or 0), int(weights), int(chunk or 0), bias, cache.page_tokens, kp.shape[0],
            ctx.status, self._stream())
        if code != 0:
            raise RuntimeError(f"prompt attention refused or failed with code {code}")
        return True

    def attention_pooled_window(self, ctx, q, out, args, n_q, n_kv, d, scale, window, pool, out_scale) -> bool:
        """Prompt portions and mixed steps of attention over a window and pooled blocks before it on
        the tcgen05 prompt kernel (its form with tiles of block means ahead of the token tiles): head
        sizes 64 and 128 with values as wide as keys.  ``args``: the token pools and the pools of block
        means as ``CudaOps._pooled_args`` lists them.  False: not this kernel's case."""
        g = n_q // n_kv
        if not (self.attention_supported(q.dtype, n_q, n_kv, d, q.stride(0)) and self.use_tc_attention
                and d in (64, 128) and g <= 128 and q.stride(0) % 8 == 0 and out.stride(0) % 8 == 0
                and not ctx.decode_only):
            return False
        kp, vp, bt, bt_width, pages, page_tokens, kb, vb, pt, pt_width, pool_pages, rows = args
        code = self.calls.leone_attention_prefill_pingpong_pooled(
            q, q.stride(0), out, out.stride(0), kp, vp, bt, bt_width, pages, page_tokens, kb, vb, pt, pt_width,
            pool_pages, rows, ctx.q_start, ctx.ctx_len, ctx.n_seqs, int(ctx.max_q_len), n_q, n_kv, d,
            float(scale), int(window), int(pool), float(out_scale), ctx.status, self._stream())
        if code != 0:
            raise RuntimeError(f"prompt attention with pooled blocks refused or failed with code {code}")
        return True

    def _attn_scratch(self, floats: int):
        if self._attn_ws is None or self._attn_ws.numel() < floats:
            self._retire(self._attn_ws)
            self._attn_ws = torch.empty(max(floats, self.min_scratch_floats), dtype=torch.float32,
                                        device=self.device)
        return self._attn_ws
