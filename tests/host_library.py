"""The library's host code over a stand-in for the CUDA runtime (tests/cuda/fake_runtime.cpp): what it
orders, launches and sets, tested without a GPU."""
import ctypes as C
import glob
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
OBJECTS = os.path.join(HERE, "..", "epic_gb300", "_lib")


@pytest.fixture(scope="session")
def host_library_file(cuda_lib, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("host") / "libepic_host.so")
    objects = sorted(glob.glob(os.path.join(OBJECTS, "*.o")))
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w", "-Wl,-Bsymbolic", "-Wl,--no-undefined", "-I/usr/local/cuda/include",
                    "-o", so, os.path.join(HERE, "cuda", "fake_runtime.cpp"), *objects], check=True)
    return so


@pytest.fixture
def host_library(host_library_file, tmp_path, monkeypatch):
    """The library linked with the stand-in, loaded in place of the real one; a copy of its own per test,
    so that no test finds another's process-wide state."""
    import epic_gb300
    so = shutil.copy(host_library_file, str(tmp_path / "libepic_host.so"))
    monkeypatch.setattr(epic_gb300, "_lib", None)
    lib = epic_gb300.load_library(so)
    lib.fake_unordered_writes.restype, lib.fake_unordered_writes.argtypes = C.c_long, [C.c_void_p]
    for n in ("fake_graph_launches", "fake_direct_launches"):
        getattr(lib, n).restype = C.c_long
    lib.fake_launches.restype = C.c_long
    lib.fake_launches.argtypes = [C.c_char_p] + 4 * [C.POINTER(C.c_uint)]
    yield lib
    monkeypatch.undo()


def launches(lib, part):
    """(count, cluster size, threads, grid x, grid y) of the launches whose kernel's name contains part."""
    out = [C.c_uint() for _ in range(4)]
    n = lib.fake_launches(part.encode(), *[C.byref(o) for o in out])
    return (n, *[o.value for o in out])
