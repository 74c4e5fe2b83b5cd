"""Calls of the C ABI without ctypes: every kind of argument arrives as ctypes would pass it, and what it cannot pass goes to ctypes."""
import ctypes
import shutil
import subprocess
import sysconfig
from pathlib import Path

import pytest

from llm_in_practise_b200 import _build
from llm_in_practise_b200.ops import _native as nv

vp, i32, i64, u64, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_ulonglong, ctypes.c_float

# eight floats, more integers than registers, in every order: a bit per argument that came as it was sent
SRC = """
#include <stdint.h>
extern "C" int probe(const void* a, long long b, float f0, int c, unsigned long long d, const void* e, float f1, float f2, long long g, int h, int i,
                     float f3, long long j, float f4, float f5, const void* k, int l, float f6, float f7, void* m) {
  return (a == (void*)16) | (b == -5) << 1 | (f0 == 1.5f) << 2 | (c == -3) << 3 | (d == 18446744073709551615ull) << 4 | (e == 0) << 5 |
         (f1 == 2.0f) << 6 | (f2 == -0.25f) << 7 | (g == (1ll << 40)) << 8 | (h == -1) << 9 | (i == 2147483647) << 10 | (f3 == 3.f) << 11 |
         (j == -9) << 12 | (f4 == 4.f) << 13 | (f5 == 5.f) << 14 | (k == (void*)0xffff00000000ull) << 15 | (l == 1) << 16 | (f6 == 6.f) << 17 |
         (f7 == 7.f) << 18 | (m == (void*)99) << 19;
}
"""
TYPES = [vp, i64, f32, i32, u64, vp, f32, f32, i64, i32, i32, f32, i64, f32, f32, vp, i32, f32, f32, vp]
ARGS = (16, -5, 1.5, -3, 2 ** 64 - 1, None, 2, -0.25, 1 << 40, -1, 2 ** 31 - 1, 3.0, -9, 4.0, 5.0, 0xffff00000000, True, 6.0, 7.0, 99)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    if nv._make_entry is None or shutil.which("g++") is None:
        pytest.skip("no extension here")
    d = tmp_path_factory.mktemp("fastcall")
    (d / "probe.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", str(d / "probe.cpp"), "-o", str(d / "probe.so")], check=True)
    fn = ctypes.CDLL(str(d / "probe.so")).probe
    fn.argtypes, fn.restype = TYPES, ctypes.c_int
    entry = nv._make_entry(ctypes.cast(fn, vp).value, "".join(nv._KINDS[t] for t in TYPES), fn)
    assert entry is not None
    return fn, entry


def test_arguments_arrive(probe):
    fn, entry = probe
    assert fn(*ARGS) == entry(*ARGS) == 2 ** 20 - 1
    assert entry(vp(16), *ARGS[1:]) == 2 ** 20 - 1                        # a ctypes object: by way of ctypes


@pytest.mark.parametrize("bad", [ARGS[:-1], ARGS[:1] + (1.0,) + ARGS[2:], ARGS[:2] + (None,) + ARGS[3:]])
def test_errors_are_those_of_ctypes(probe, bad):
    for fn in probe:
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            fn(*bad)


def test_what_is_not_made():
    if nv._make_entry is None:
        pytest.skip("no extension here")
    assert nv._make_entry(16, "i" * 33, len) is None and nv._make_entry(16, "f" * 9, len) is None
    assert nv._make_entry(0, "i", len) is None and nv._make_entry(16, "d", len) is None


def test_only_the_file_of_this_python_is_loaded(tmp_path, monkeypatch):
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    assert _build.fastcall_path().name == "_b200_fastcall" + suffix and "cpython" in suffix
    monkeypatch.setattr(nv, "_LIBDIR", tmp_path)
    (tmp_path / ("_b200_fastcall" + suffix)).write_bytes(b"not a module")
    assert nv._fastcall() is None
    if _build.fastcall_path().exists():
        (tmp_path / ("_b200_fastcall" + suffix)).unlink()
        shutil.copy(_build.fastcall_path(), tmp_path / "_b200_fastcall.so")
        shutil.copy(_build.fastcall_path(), tmp_path / "_b200_fastcall.cpython-39-x86_64-linux-gnu.so")
        assert nv._fastcall() is None
        shutil.copy(_build.fastcall_path(), tmp_path / ("_b200_fastcall" + suffix))
        assert nv._fastcall() is not None


def test_no_compiler_leaves_ctypes(tmp_path, monkeypatch):
    monkeypatch.setattr(_build, "LIBDIR", tmp_path)
    monkeypatch.setenv("PATH", str(tmp_path))
    if not Path(sysconfig.get_paths()["include"], "Python.h").exists():
        pytest.skip("no headers here")
    with pytest.warns(UserWarning, match="ctypes"):
        assert _build.build_fastcall() is None
    assert not list(tmp_path.iterdir())


def test_a_fresh_checkout_builds_it(monkeypatch):
    built = []
    monkeypatch.setattr(_build, "build_cuda", lambda **kw: "library")
    monkeypatch.setattr(_build, "build_fastcall", lambda: built.append(1))
    assert _build.ensure_built(["gemv"]) == "library" and built
