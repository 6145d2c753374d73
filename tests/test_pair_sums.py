"""The folded norm's sums of squares on pairs of SMs, where a pair walks several tiles with different token rows and the last ones are
ragged: the order of the hand-over on the CPU (``csrc/pair_sums.h`` walked through the kernel's tiles), the sums on the GPU."""
import ctypes
import math
import os
import shutil
import subprocess

import pytest
import torch

from leone_b200.csrc import build
from leone_b200.ops.fast import FastKernels

# Two warps of one quarter walk a block's tiles under every order that is tried: the second writes and arrives, the first waits by
# parity, reads and releases the accumulator; a tile's accumulator is there once its buffer's last tile was released by both.
WALK = r"""
#include <cstdlib>
#include <vector>
#include "pair_sums.h"
using leone::SumsHandover;
struct ByCount { SumsHandover h; int place(int buf, int q) { return SumsHandover::place(buf, q); } unsigned next(int, int buf) { return h.next(buf); } };
struct ByTile { int place(int, int q) { return q; } unsigned next(int it, int) { return it & 1; } };      // a barrier a quarter, the tile's number

// 0 right, 1 sums of another tile were read, 2 a wait that never ends
template <class Rule> int walk(const std::vector<char>& skip, int quarter, int order) {
  Rule rule[2];
  const int n = (int)skip.size();
  int at[2] = {0, 0}, step[2] = {0, 0}, done[8] = {0}, tag[8];
  unsigned parity[2] = {0, 0};
  for (int& t : tag) t = -1;
  auto go = [&](int w) -> int {                       // one step of warp w: 1 made, 0 has to wait, -1 wrong
    if (at[w] == n) return 0;
    const int i = at[w], buf = i & 1, place = rule[w].place(buf, quarter);
    if (step[w] == 0) {
      if (i >= 2 && (at[0] <= i - 2 || at[1] <= i - 2)) return 0;
      if (!skip[i]) parity[w] = rule[w].next(i, buf);
      step[w] = 1;
    } else if (step[w] == 1) {
      if (!skip[i] && w == 1) tag[place] = i, ++done[place];
      if (!skip[i] && w == 0) {
        if ((unsigned)(done[place] & 1) == parity[0]) return 0;
        if (tag[place] != i) return -1;
      }
      step[w] = 2;
    } else {
      ++at[w];
      step[w] = 0;
    }
    return 1;
  };
  while (at[0] < n || at[1] < n) {
    const int first = order == 2 ? std::rand() & 1 : order;
    int r = go(first);
    if (r == 0) r = go(first ^ 1);
    if (r < 0) return 1;
    if (r == 0) return 2;
  }
  return 0;
}
template <class Rule> int all(int m, int n, int width, int pairs) {
  const int m_pairs = ((m + 127) / 128 + 1) / 2, total = (n + width - 1) / width * m_pairs;
  if (pairs > total) pairs = total;
  int worst = 0;
  for (int pair = 0; pair < pairs; ++pair)
    for (int rank = 0; rank < 2; ++rank)
      for (int q = 0; q < 4; ++q) {
        std::vector<char> skip;
        for (int t = pair; t < total; t += pairs) skip.push_back((t % m_pairs * 2 + rank) * 128 + q * 32 >= m);
        for (int order = 0; order < 3; ++order) {
          const int r = walk<Rule>(skip, q, order);
          if (r > worst) worst = r;
        }
      }
  return worst;
}
extern "C" int by_count(int m, int n, int width, int pairs) { return all<ByCount>(m, n, width, pairs); }
extern "C" int by_tile(int m, int n, int width, int pairs) { return all<ByTile>(m, n, width, pairs); }
"""


@pytest.fixture(scope="module")
def walks(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("walks")
    (d / "w.cpp").write_text(WALK)
    here = os.path.dirname(os.path.abspath(build.__file__))
    subprocess.run([cxx, "-O1", "-shared", "-fPIC", "-I", here, str(d / "w.cpp"), "-o", str(d / "w.so")], check=True)
    return ctypes.CDLL(str(d / "w.so"))


def _width(m, n):
    f = FastKernels.__new__(FastKernels)
    f.sm_count = 148
    f._configure()
    return f.pair_width(m, n, False)


@pytest.mark.parametrize("n", [2048, 4096, 5120, 8192])
def test_every_tiles_sums_are_its_own(walks, n):
    for m in [*range(385, 4097, 31), *range(512, 4097, 256), *range(513, 4097, 256)]:
        assert walks.by_count(m, n, _width(m, n), 74) == 0, m


def test_the_walk_sees_a_barrier_that_loses_step(walks):
    """Counting the block's tiles in place of the hand-overs reads another tile's sums, or waits for good."""
    assert walks.by_tile(1100, 4096, 144, 74) > 0
    assert walks.by_tile(2048, 4096, 48, 74) > 0           # no ragged tile, but three rounds and a second warp ahead


DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,width", [(1100, 4096, 256, 0), (1500, 4096, 256, 0), (1800, 4096, 256, 0), (900, 5120, 256, 0),
                                         (2700, 2048, 64, 0), (1100, 4096, 64, 48), (1025, 4096, 128, 0)])
def test_sums_of_squares_over_several_rounds(m, n, k, width):
    """Every part of the sums, over its tile's columns, against float64, and the same bits on every run; the places hold NaN before."""
    from leone_b200.ops.cuda import CudaOps
    from tests.test_kernels_gpu import _close, _randn
    ops = CudaOps(DEV, torch.bfloat16)
    fast = ops.fast
    if not fast.use_pairs:
        pytest.skip("LEONE_NO_PAIRS is set")
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    ops.bind_status(status)
    fast.pair_width_override = width
    assert fast.fuses_norm(m, n, k)
    width = width or fast.pair_width(m, n, False)
    parts = fast.norm_parts(m, n)
    assert parts == -(-n // width) and parts * -(-m // 256) > fast.sm_count // 2          # several rounds
    x = _randn((m, k), 181, torch.bfloat16)
    w = _randn((n, k), 182, torch.bfloat16, scale=0.05)
    res = _randn((m, n), 183)
    g = 1 + 0.2 * _randn((n,), 184)
    want = x.double() @ w.double().t() + res.double()
    first = None
    for _ in range(5):
        hidden = res.clone()
        xn = torch.full((m, n), math.nan, device=DEV, dtype=torch.bfloat16)
        ss = torch.full((parts, m), math.nan, device=DEV)
        fast._gemm(x, w, hidden, 2, hidden, n, norm_out=(xn, g, ss))
        got = (hidden, xn, ss)
        if first is None:
            first = got
            _close(hidden, want, 1e-5, 2e-6 * math.sqrt(k) * 4, f"residual in place m{m} n{n} width {width}")
            h64 = hidden.double()
            _close(xn, h64 * g.double(), 2 ** -8, 1e-6, "bf16(out * weight)")
            # at most 256 terms, none negative, each rounded with every addition after it: 256 roundings bound the error
            for i in range(parts):
                _close(ss[i], (h64[:, i * width:(i + 1) * width] ** 2).sum(1), 256 * 2 ** -24, 0.0, f"sums of squares, part {i}")
        assert all(torch.equal(a, b) for a, b in zip(first, got))
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
