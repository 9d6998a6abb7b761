"""The extension module that calls launchers: arguments arrive in their places whatever stands between them."""
import ast
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from railgun_b200 import native, ops

SOURCE = """
extern "C" int probe(void* p, int a, float x, const int* q, long long b, float y, int c, int d, int e, int g, float z, int n8,
                     int n9, void* last) {
    return (p == (void*)0x123456789abcLL) + 2 * (a == -7) + 4 * (x == 1.5f) + 8 * (q == nullptr) + 16 * (b == 1LL << 40) +
           32 * (y == -2.25f) + 64 * (c == 3) + 128 * (d == 4) + 256 * (e == 5) + 512 * (g == 6) + 1024 * (z == 0.1f) +
           2048 * (n8 == 8) + 4096 * (n9 == 1) + 8192 * (last == (void*)0x7fffffffffffLL);
}
"""


@pytest.fixture(scope="module")
def fast():
    try:
        return native.load_module("fastcall")
    except native.NativeBuildError as e:
        pytest.skip(f"no Python headers: {e}")


def test_arguments_in_their_places(fast, tmp_path):
    src, lib = tmp_path / "probe.cpp", tmp_path / "probe.so"
    src.write_text(SOURCE)
    subprocess.run([native._find("g++", ["/usr/bin/g++"]), "-O2", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    so = ctypes.CDLL(str(lib))
    address = ctypes.cast(so.probe, ctypes.c_void_p).value
    args = (0x123456789abc, -7, fast.real(1.5), None, 1 << 40, fast.real(-2.25), 3, 4, 5, 6, fast.real(0.1), 8, True, 0x7fffffffffff)
    assert fast.call(address, *args) == 2 ** 14 - 1


def test_what_it_refuses(fast):
    with pytest.raises(TypeError):
        fast.call("address")
    with pytest.raises(ValueError):
        fast.call(0)
    with pytest.raises(TypeError):
        fast.call(1, *range(49))
    with pytest.raises(TypeError):
        fast.call(1, *[0.5] * 9)
    with pytest.raises(TypeError):
        fast.call(1, "text")
    assert fast.ptr(None) == 0 and fast.pointer(None) == 0


# values that a caller may put in an argument's place by mistake, or as another type of number
VALUES = [3, -2, True, 0, 2.0, float("nan"), None, "1.5", "text", b"7", 1 << 40, [1], 1 + 2j, np.int32(3), np.float32(2.5), np.float64(2.5)]


@pytest.mark.parametrize("kind", ["c_int", "c_longlong", "c_void_p", "c_float"])
def test_each_kind_takes_what_ctypes_takes(kind):
    """A float that reached the call in an integer's place would move every argument behind it by one place."""
    converter, own = getattr(ctypes, kind), getattr(ops, kind)
    for value in VALUES:
        try:
            want = converter(value).value
        except TypeError:
            with pytest.raises(TypeError):
                own(value)
            continue
        got = own(value)
        assert isinstance(got, float if kind == "c_float" else int) or isinstance(got, converter)
        got = (got if isinstance(got, converter) else converter(got)).value
        assert got == want or (got != got and want != want)


def test_every_argument_of_a_launcher_has_a_kind():
    """In ops.py nothing reaches a launcher but through the converters (or one of the named groups of converted arguments)."""
    source = Path(ops.__file__).read_text()
    kinds = {"c_int", "c_longlong", "c_void_p", "c_float", "_ptr", "_at", "_stream"}
    of_kinds = {"_ptr", "_at", "_stream", "_pooled", "none", "who", "at"}           # functions whose results are converted
    groups, seen = {"x", "B", "C"}, 0
    for node in ast.walk(ast.parse(source)):
        if isinstance(node, ast.Call) and isinstance(node.func, ast.Call) and getattr(node.func.func, "id", "") == "_fn":
            for arg in node.args:
                value = arg.value if isinstance(arg, ast.Starred) else arg
                name = value.func.id if isinstance(value, ast.Call) else value.id
                assert name in kinds | of_kinds | groups, ast.unparse(node)
                seen += 1
    assert seen > 1000
