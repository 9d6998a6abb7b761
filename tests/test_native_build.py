"""The builder of the native libraries (railgun_b200/native.py), on the CPU with
the host library: names carry a digest of the source and its headers, a missing
source or a failing compiler is one clear error, the build folder can be moved."""
import ctypes
import os
import subprocess
import sys

import pytest

from railgun_b200 import native


def test_library_names_carry_the_digest_of_source_and_flags():
    src, out, flags, compiler = native.library_path("runtime", "host")
    assert src.name == "runtime.cpp" and compiler == "g++"
    digest = native._source_digest(src, flags)
    assert out.name == f"librailgun_runtime.{digest}.so" and len(digest) == 16
    assert native._source_digest(src, flags + ["-DX"]) != digest          # other flags, another library
    ksrc, kout, kflags, kcompiler = native.library_path("norm", "kernel")
    assert kcompiler == "nvcc" and "arch=compute_100a,code=sm_100a" in kflags
    assert "norm" in native.kernel_sources() and "runtime" in native.host_sources()


def test_a_missing_source_is_a_clear_error():
    with pytest.raises(native.NativeBuildError, match="no source file .*no_such_kernel.cu"):
        native.load("no_such_kernel")


def test_the_build_folder_can_be_moved(tmp_path, monkeypatch):
    monkeypatch.setenv("RAILGUN_B200_BUILD_DIR", str(tmp_path / "built"))
    monkeypatch.setattr(native, "_build_dir_cache", [])
    path = native.build("runtime", "host")
    assert path.parent == tmp_path / "built" and path.is_file()
    lib = ctypes.CDLL(str(path))
    assert hasattr(lib, "rg_cache_create") and hasattr(lib, "rg_sched_schedule")
    assert native.build("runtime", "host") == path                       # built once


def _import_ops(tmp_path, before):
    """A process of its own that runs ``before`` (with railgun_b200.native as n), imports ops without anything built and says how
    launchers are called there."""
    code = f"import railgun_b200.native as n\n{before}\nimport railgun_b200.ops as o, ctypes\nprint('ctypes', o.c_int is ctypes.c_int)"
    env = dict(os.environ, RAILGUN_B200_BUILD_DIR=str(tmp_path))
    return subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)


def test_without_pythons_headers_launchers_go_through_ctypes_and_it_is_said(tmp_path):
    done = _import_ops(tmp_path, "n.python_headers = lambda: False")
    assert done.returncode == 0 and done.stdout.strip() == "ctypes True"
    assert "through ctypes" in done.stderr and "Python's headers" in done.stderr


def test_an_extension_module_that_does_not_compile_is_an_error(tmp_path):
    done = _import_ops(tmp_path, "n.GXX_FLAGS.append('-fno-such-option')")
    assert done.returncode != 0 and "NativeBuildError" in done.stderr and "fastcall.cpp" in done.stderr


def test_everything_builds_without_pythons_headers(monkeypatch):
    built = []
    monkeypatch.setattr(native, "build", lambda name, kind: built.append((name, kind)) or name)
    monkeypatch.setattr(native, "python_headers", lambda: False)
    native.build_all()
    assert set(built) == {(n, "kernel") for n in native.kernel_sources()} | {("runtime", "host")}
    monkeypatch.setattr(native, "python_headers", lambda: True)
    native.build_all()
    assert ("fastcall", "host") in built
