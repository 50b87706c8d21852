"""The extension module through which Python calls the kernel library: every kind of argument reaches the function as through
ctypes, in registers and on the stack, and what the module does not take is left to ctypes."""
import ctypes
import platform
import shutil
import subprocess
import sysconfig
from pathlib import Path

import pytest

SOURCE = r"""
int f(int a, const void* p, long long b, float x, int c, float y, int d, long long e, int g, int h, void* q, float z, unsigned long long k, int m) {
  return (a == -1) + (p == 0) * 2 + (b == -(1ll << 40)) * 4 + (x == 1.5f) * 8 + (c == 7) * 16 + (y == -2.f) * 32 + (d == 1) * 64 + (e == (1ll << 50)) * 128
       + (g == 9) * 256 + (h == 10) * 512 + (q == (void*)4096) * 1024 + (z == 3.f) * 2048 + (k == 0xfffffffffffffff0ull) * 4096 + (m == -5) * 8192;
}
"""
ARGS = (-1, None, -(1 << 40), 1.5, 7, -2, True, 1 << 50, 9, 10, 4096, 3.0, 0xfffffffffffffff0, -5)


def needed():
    """The module, wherever it can be built; a machine that cannot build it goes through ctypes."""
    from lucciola_b200 import csrc
    if platform.machine() != "x86_64" or not shutil.which("gcc") or not (Path(sysconfig.get_paths()["include"]) / "Python.h").exists():
        pytest.skip("no Python headers, no compiler, or not x86-64: calls go through ctypes")
    module = csrc.caller()
    assert module is not None
    return module


def test_arguments_arrive(tmp_path):
    module = needed()
    (tmp_path / "f.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-fPIC", "-shared", "-o", str(tmp_path / "f.so"), str(tmp_path / "f.c")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "f.so"))
    f = module.bind(ctypes.cast(lib.f, ctypes.c_void_p).value, "ipififiiiipfii")
    assert f(*ARGS) == 2 ** 14 - 1
    assert f(*ARGS[:10], (ctypes.c_int * 2)(), *ARGS[11:]) is NotImplemented
    with pytest.raises(TypeError):
        f(1)
    with pytest.raises(ValueError):
        module.bind(1, "x")
    with pytest.raises(ValueError):
        module.bind(1, "f" * 9)


def test_same_answers_as_ctypes():
    from lucciola_b200 import ops
    needed()
    for args in ((1, 16, 128, 128, 512), (4, 32, 64, 40, 3), (1, 1, 1000, 7, 64)):
        assert ops._invoke("lb_decay_row_split", *args) == ops._fn("lb_decay_row_split")(*args)


def test_without_the_module(monkeypatch):
    from lucciola_b200 import ops
    monkeypatch.setattr(ops, "_native", {})
    monkeypatch.setattr(ops, "caller", lambda: None)
    assert ops.expert_tile_rows(1) == 16 and ops._native is None


def test_built_when_only_it_is_missing(tmp_path, monkeypatch, capfd):
    """Beside a library of the right stamp that another interpreter has built; and a compiler that fails says so."""
    from lucciola_b200 import csrc
    needed()
    other = tmp_path / "lb_caller-0123456789abcdef.cpython-399-x86_64-linux-gnu.so"
    other.write_bytes(b"of another interpreter")
    stale = csrc._caller_path(tmp_path).with_name(csrc._caller_path(tmp_path).name.replace(csrc._digest([csrc._CALLER]), "0" * 16))
    stale.write_bytes(b"of an earlier source")
    (tmp_path / csrc.LIB_NAME).write_bytes(b"")
    (tmp_path / "stamp").write_text(csrc.source_digest())
    monkeypatch.setattr(csrc, "build_dir", lambda: tmp_path)
    monkeypatch.setattr(csrc, "find_nvcc", lambda: "nvcc")
    assert csrc.build() == tmp_path / csrc.LIB_NAME
    assert csrc._caller_path(tmp_path).exists() and other.exists() and not stale.exists()
    csrc._caller_path(tmp_path).unlink()
    broken = tmp_path / "broken.c"
    broken.write_text("#error broken on purpose\n")
    monkeypatch.setattr(csrc, "_CALLER", broken)
    capfd.readouterr()
    csrc.build()
    assert not csrc._caller_path(tmp_path).exists() and "broken on purpose" in capfd.readouterr().err


def test_looked_for_once(monkeypatch):
    from lucciola_b200 import csrc
    module = needed()
    monkeypatch.setattr(csrc, "_caller_path", None)
    assert csrc.caller() is module


def test_another_thread_finds_no_module(monkeypatch):
    """The table of bound functions goes away between two looks at it."""
    from lucciola_b200 import ops

    class Table(dict):
        def get(self, name):
            monkeypatch.setattr(ops, "_native", None)
            return None

    monkeypatch.setattr(ops, "_native", Table())
    assert ops.expert_tile_rows(1) == 16
