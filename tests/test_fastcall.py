"""The extension module that calls launchers: arguments arrive in their places whatever stands between them."""
import ctypes
import subprocess

import pytest

from railgun_b200 import native

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
    with pytest.raises(ValueError):
        fast.real("text")
    assert fast.ptr(None) == 0 and fast.same(fast) is fast
