"""The library's host code on a machine without a GPU: the built objects linked against
tests/fake_cudart.c, which records launches instead of running them."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

from bridct_b200 import _lib
from bridct_b200.build import nvcc

ROOT = Path(__file__).resolve().parents[1]


def build(out: Path) -> Path:
    objs = sorted((ROOT / "_build").glob("*.o"))
    cxx = shutil.which("g++")
    if not objs or not cxx:
        pytest.skip("needs the library's objects (python -m bridct_b200.build) and g++")
    include = Path(nvcc()).resolve().parents[1] / "include"
    fake = out / "fake_cudart.o"
    subprocess.run(["gcc", "-O1", "-fPIC", "-I", str(include), "-c", str(ROOT / "tests" / "fake_cudart.c"), "-o",
                    str(fake)], check=True)
    lib = out / "libbridct_fake.so"
    # -Bsymbolic: the CUDA names bind to the stand-in whatever else the process has loaded
    subprocess.run([cxx, "-shared", "-Wl,-Bsymbolic", "-o", str(lib)] + [str(o) for o in objs] +
                   [str(fake), "-lpthread"], check=True)
    return lib


def load(lib: Path, monkeypatch) -> C.CDLL:
    """The stand-in library with the signatures of the real one, in place of it."""
    monkeypatch.setattr(_lib, "LIB_PATH", lib)
    monkeypatch.setattr(_lib, "_lib", None)
    L = _lib.lib()
    L.fake_launch_name.restype = C.c_char_p
    return L


def launched(L) -> list:
    return [(L.fake_launch_name(i).decode(), L.fake_launch_grid(i)) for i in range(L.fake_launches())]
