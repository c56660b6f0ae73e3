"""The compiled calls of the launchers: arguments arrive as ctypes delivers them, wrong ones raise, and without a compiler ctypes is used."""
import ctypes
import subprocess

import pytest

from arle_b200.ops import launchers

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


@pytest.fixture(params=[True, False])
def lib(request, tmp_path, monkeypatch):
    (tmp_path / "e.c").write_text(C_SOURCE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "e.so"), str(tmp_path / "e.c")], check=True)
    if not request.param:
        monkeypatch.setattr(launchers, "_compile", lambda text, path: False)
    loaded = launchers.load(str(tmp_path / "e.so"), SIGNATURES)
    assert isinstance(loaded, ctypes.CDLL) != request.param
    return loaded


def test_arguments_and_results(lib):
    out = (ctypes.c_long * 8)()
    args = [ctypes.addressof(out), 5, 0.25, -(1 << 40), (1 << 47) + 3, 1.0, 2, 3.0, 4.0, True, 2, 3, 4.0, 3.0, 2.0, 1, None]
    assert lib.echo_all(*args) == 7
    assert list(out) == [5, 250, -(1 << 40), (1 << 47) + 3, 4321, 17, 1234, 0]
    assert lib.echo_all(*args[:1], -2, *args[2:]) == -3 and out[0] == -2
    assert lib.echo_none(None, None) == 1 and lib.echo_none(None, 8) == 0


@pytest.mark.parametrize("at,value", [(0, 1.5), (0, "x"), (1, 2.0), (1, None), (2, "x"), (3, 1.0)])
def test_wrong_arguments_raise(lib, at, value):
    out = (ctypes.c_long * 8)()
    args = [ctypes.addressof(out), 5, 0.25, 1, 0, 1.0, 2, 3.0, 4.0, 1, 2, 3, 4.0, 3.0, 2.0, 1, None]
    args[at] = value
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        if at == 0 and value == "x" and isinstance(lib, ctypes.CDLL):
            raise TypeError("ctypes takes text for a pointer")
        lib.echo_all(*args)
    with pytest.raises(TypeError):
        lib.echo_none(None)
