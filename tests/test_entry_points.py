"""Calls of C entry points (ops/entry_points.py): every argument arrives where ctypes would put it."""
import ctypes
import shutil
import subprocess

import pytest
import torch

from leone_b200.ops import entry_points

SOURCE = r"""
#include <cstdio>
extern "C" int few(void* a, float x, int b, long long c) { return (a == 0) * 1000 + (int)(x * 8) + b + (int)(c >> 33); }
// 34 integers around six floats: registers, stack and both kinds of places
extern "C" int many(void* p, int a1, float f1, int a2, int a3, long long a4, void* q, int a5, int a6, float f2, float f3, int a7, int a8,
                    int a9, int a10, int a11, int a12, int a13, int a14, float f4, int a15, int a16, int a17, int a18, int a19, int a20,
                    int a21, int a22, int a23, int a24, float f5, long long a25, int a26, int a27, int a28, int a29, int a30, float f6, void* r, int* out) {
  const long long v[] = {(long long)p, a1, a2, a3, a4, (long long)q, a5, a6, a7, a8, a9, a10, a11, a12, a13, a14, a15, a16, a17, a18, a19, a20,
                         a21, a22, a23, a24, a25, a26, a27, a28, a29, a30, (long long)r};
  const float f[] = {f1, f2, f3, f4, f5, f6};
  long long h = 17;
  for (long long x : v) h = h * 1000003 + x;
  for (float x : f) h = h * 1000003 + (long long)(x * 1024);
  out[0] = (int)(h & 0x7fffffff);
  return -3;
}
// places on the stack that the callee reads as 64 bits
extern "C" int wide(int, int, int, int, int, int, int a, long long b, long long c, void* d, long long e, long long* out) {
  out[0] = a; out[1] = b; out[2] = c; out[3] = (long long)d; out[4] = e;
  return 0;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("entries")
    (d / "e.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-O1", "-shared", "-fPIC", str(d / "e.cpp"), "-o", str(d / "e.so")], check=True)
    return ctypes.CDLL(str(d / "e.so"))


@pytest.mark.parametrize("native", [True, False])
def test_arguments_arrive(lib, native, monkeypatch):
    if native:
        bind = entry_points._bind()
        if bind is entry_points._through_ctypes:
            pytest.skip("the extension is not built here")
    else:
        monkeypatch.setattr(entry_points, "_BIND", entry_points._through_ctypes)
    calls = entry_points.EntryPoints(lib)
    assert calls.few(None, 1.5, -7, 5 << 33) == 1000 + 12 - 7 + 5
    t, out = torch.zeros(4), torch.zeros(1, dtype=torch.int32)
    ints = [3 + 7 * i for i in range(31)]
    ints[3], ints[24] = -(1 << 40), 1 << 50
    f = [0.5, -2.25, 3.0, 1e3, 0.125, -7.5]
    args = [t, ints[0], f[0], ints[1], ints[2], ints[3], None, ints[4], ints[5], f[1], f[2], *ints[6:14], f[3], *ints[14:24], f[4],
            *ints[24:30], f[5], t, out]
    assert calls.many(*args) == -3
    h = 17
    for x in [t.data_ptr(), ints[0], ints[1], ints[2], ints[3], 0, *ints[4:30], t.data_ptr(), *[int(v * 1024) for v in f]]:
        h = (h * 1000003 + x) % (1 << 64)
    assert int(out[0]) == h & 0x7FFFFFFF
    with pytest.raises((AttributeError, TypeError)):
        calls.few("x", 1.0, 1, 1)


def test_the_extension_belongs_to_its_interpreter(monkeypatch):
    """Another interpreter, or another version of it, neither finds this one's file nor takes it for its own."""
    import sys
    import sysconfig
    from leone_b200.csrc import build
    path, digest, others = build.library_path("call"), build._digest("call"), {m: build.library_path(m) for m in build.MODULES if m != "call"}
    real = sysconfig.get_config_var
    monkeypatch.setattr(sysconfig, "get_config_var", lambda name: "cpython-399-test" if name == "SOABI" else real(name))
    assert build.library_path("call") != path and build._digest("call") != digest
    monkeypatch.undo()
    monkeypatch.setattr(sys, "version", sys.version + "+1")
    assert build.library_path("call") == path and build._digest("call") != digest
    assert others == {m: build.library_path(m) for m in others}


@pytest.mark.parametrize("native", [True, False])
def test_small_numbers_in_64_bit_places(lib, native, monkeypatch):
    """Zero, small and negative numbers behind the sixth integer, where the stack held other bits before."""
    if native:
        if entry_points._bind() is entry_points._through_ctypes:
            pytest.skip("the extension is not built here")
    else:
        monkeypatch.setattr(entry_points, "_BIND", entry_points._through_ctypes)
    calls = entry_points.EntryPoints(lib)
    out = torch.zeros(5, dtype=torch.int64)
    full = (1 << 62) + 0x5A5A5A5A5A5A5A5A % (1 << 60)
    for row in ([0, 0, 0, 0, 0], [-1, 5, -5, 0, 7], [3, -1, 1, 1 << 20, -(1 << 31)], [9, 1 << 31, -(1 << 31) - 1, (1 << 64) - 16, 0],
                [2, (1 << 31) - 1, 0, 0, -2]):
        assert calls.wide(*[full] * 11, out) == 0
        assert calls.wide(1, 2, 3, 4, 5, 6, *row, out) == 0
        assert out.tolist() == [*row[:3], row[3] if row[3] < 1 << 63 else row[3] - (1 << 64), row[4]]
    for too_long in (1 << 64, -(1 << 63) - 1):
        with pytest.raises(OverflowError):
            calls.wide(1, 2, 3, 4, 5, 6, 7, too_long, 9, 10, 11, out)


def test_tails_of_block_tables():
    """The rows of a mirror of the tables: new entries, and -1 as far as asked."""
    import numpy as np
    from leone_b200.cache.pages import CacheError, CacheManager, GroupSpec
    c = CacheManager([GroupSpec("full", 1, 8)], 4, 40, 4)
    for rid, n in (("a", 9), ("b", 1), ("c", 30)):
        c.open(rid)
        c.reserve({rid: n})
    rids = ["a", "b", "c"]
    want = c.block_table(0, rids, 10)
    i32 = lambda *v: np.array(v, dtype=np.int32)                       # noqa: E731
    rows = np.full((3, 10), 77, dtype=np.int32)
    c.copy_table_tails(0, rids, i32(0, 0, 0), i32(10, 10, 10), rows)
    assert (rows == want).all()
    rows[:] = 77
    c.copy_table_tails(0, rids, i32(2, 1, 8), i32(3, 4, 8), rows)       # one entry, three that are cleared, none
    assert rows[0].tolist() == [77, 77, want[0, 2]] + [77] * 7 and rows[1].tolist() == [77, -1, -1, -1] + [77] * 6
    assert (rows[2] == 77).all()
    with pytest.raises(CacheError):
        c.copy_table_tails(0, rids, i32(0, 0, 0), i32(2, 1, 8), rows)   # fewer places than entries
