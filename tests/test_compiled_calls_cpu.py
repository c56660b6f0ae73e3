"""The compiled calls of the launchers: arguments arrive as ctypes delivers them, wrong ones raise, and without a compiler ctypes is used."""
import ctypes
import fractions
import os
import subprocess

import numpy as np
import pytest

from arle_b200.ops import build, launchers

P, I, F, L = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_long
SIGNATURES = {"echo_all": [P, I, F, L, P, F, F, F, F, I, I, I, F, F, F, F, P], "echo_none": [P, P]}
C_SOURCE = """
int echo_all(long* out, int i, float f, long l, void* p, float f1, float f2, float f3, float f4, int a, int b, int c, float g1, float g2, float g3,
             float g4, void* q) {
  out[0] = i; out[1] = (long)(f * 1000); out[2] = l; out[3] = (long)p; out[4] = (long)(f1 + 10 * f2 + 100 * f3 + 1000 * f4); out[5] = a + 2 * b + 4 * c;
  out[6] = (long)(g1 + 10 * g2 + 100 * g3 + 1000 * g4); out[7] = (long)q;
  return i < 0 ? -3 : 7;
}
int echo_none(void* a, void* b) { return !a && !b; }
"""


def _library(folder):
    (folder / "e.c").write_text(C_SOURCE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(folder / "e.so"), str(folder / "e.c")], check=True)
    return str(folder / "e.so")


@pytest.fixture(params=[True, False])
def lib(request, tmp_path, monkeypatch):
    if not request.param:
        monkeypatch.setattr(launchers, "_compile", lambda text, path: False)
    loaded = launchers.load(_library(tmp_path), SIGNATURES)
    assert isinstance(loaded, ctypes.CDLL) != request.param
    return loaded


def test_arguments_and_results(lib):
    out = (ctypes.c_long * 8)()
    args = [ctypes.addressof(out), 5, 0.25, -(1 << 40), (1 << 47) + 3, 1.0, 2, 3.0, 4.0, True, 2, 3, 4.0, 3.0, 2.0, 1, None]
    assert lib.echo_all(*args) == 7
    assert list(out) == [5, 250, -(1 << 40), (1 << 47) + 3, 4321, 17, 1234, 0]
    assert lib.echo_all(*args[:1], -2, *args[2:]) == -3 and out[0] == -2
    assert lib.echo_none(None, None) == 1 and lib.echo_none(None, 8) == 0


def _arguments(out):
    return [ctypes.addressof(out), 5, 0.25, 1, 0, 1.0, 2, 3.0, 4.0, 1, 2, 3, 4.0, 3.0, 2.0, 1, None]


@pytest.mark.parametrize("at,value", [(0, 1.5), (0, np.int64(8)), (1, 2.0), (1, None), (1, np.float32(2)), (2, "x"), (3, 1.0), (3, "x")])
def test_wrong_arguments_raise(lib, at, value):
    args = _arguments((ctypes.c_long * 8)())
    args[at] = value
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        lib.echo_all(*args)
    with pytest.raises(TypeError):
        lib.echo_none(None)


@pytest.mark.parametrize("value", ["x", b"x", (ctypes.c_long * 2)()])
def test_compiled_calls_take_no_text_or_arrays_for_pointers(tmp_path, value):
    loaded = launchers.load(_library(tmp_path), SIGNATURES)
    with pytest.raises(TypeError):
        loaded.echo_none(value, None)


def test_numbers_of_other_types(lib):
    out = (ctypes.c_long * 8)()
    args = _arguments(out)
    args[1:4] = np.int32(-5), np.float32(0.5), np.int64(-(1 << 40))
    args[5:8] = fractions.Fraction(1), np.int64(2), np.float64(3)
    assert lib.echo_all(*args) == -3 and list(out)[:5] == [-5, 500, -(1 << 40), 0, 4321]


def _answers(lib):
    assert lib.echo_none(None, None) == 1 and lib.echo_none(None, 8) == 0


@pytest.mark.parametrize("compiler", ["/no/such/compiler", "false"])
def test_a_compiler_that_does_not_run_leaves_ctypes(compiler, tmp_path, monkeypatch):
    monkeypatch.setenv("CC", compiler)
    path = _library(tmp_path)
    before = sorted(os.listdir(tmp_path))
    loaded = launchers.load(path, SIGNATURES)
    assert isinstance(loaded, ctypes.CDLL) and sorted(os.listdir(tmp_path)) == before
    _answers(loaded)


def _no_writing_below(folder, monkeypatch):
    """open(..., "w") below ``folder`` fails, as for a user who may not write there (chmod does not stop root)."""
    real = open

    def guarded(file, mode="r", *args, **kwargs):
        if str(file).startswith(str(folder)) and mode != "r":
            raise PermissionError(13, "Permission denied", str(file))
        return real(file, mode, *args, **kwargs)

    monkeypatch.setattr(launchers, "open", guarded, raising=False)


def test_a_folder_that_cannot_be_written(tmp_path, monkeypatch):
    (tmp_path / "shared").mkdir(), (tmp_path / "own").mkdir()
    path = _library(tmp_path / "shared")
    monkeypatch.setattr(build, "build_dir", lambda: str(tmp_path / "own"))
    _no_writing_below(tmp_path / "shared", monkeypatch)
    loaded = launchers.load(path, SIGNATURES)              # the calls go to the user's folder
    assert not isinstance(loaded, ctypes.CDLL) and len(os.listdir(tmp_path / "own")) == 1
    _answers(loaded)
    monkeypatch.setattr(launchers, "_compile", None)       # and are found there again
    again = launchers.load(path, SIGNATURES)
    assert not isinstance(again, ctypes.CDLL)
    _answers(again)


def test_no_folder_that_can_be_written(tmp_path, monkeypatch):
    path = _library(tmp_path)
    monkeypatch.setattr(build, "build_dir", lambda: str(tmp_path))
    _no_writing_below(tmp_path, monkeypatch)
    loaded = launchers.load(path, SIGNATURES)
    assert isinstance(loaded, ctypes.CDLL)
    _answers(loaded)


def test_calls_that_cannot_be_loaded_are_compiled_anew(tmp_path):
    (tmp_path / "first").mkdir(), (tmp_path / "other").mkdir()
    path = _library(tmp_path / "first")
    before = set(os.listdir(tmp_path / "first"))
    launchers.load(path, SIGNATURES)
    name, = set(os.listdir(tmp_path / "first")) - before
    path = _library(tmp_path / "other")                    # a path that this process has not loaded yet
    (tmp_path / "other" / name).write_text("not a library")
    loaded = launchers.load(path, SIGNATURES)
    assert not isinstance(loaded, ctypes.CDLL)
    _answers(loaded)
