"""Builds csrc/engine.cpp with the host stand-in of the CUDA runtime
(fake_cuda.cpp) and a test's own C++ driver, once per test process, and runs it."""
import atexit
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
_dir = None
_drivers: dict[str, str] = {}


def _build(source: str) -> str:
    global _dir
    from libfluid_gb300 import build as B
    if shutil.which(B.CXX) is None:
        pytest.skip("needs a C++ compiler")
    cxx = [B.CXX, *B.CXX_FLAGS, "-O1", f"-I{HERE}"]
    if _dir is None:
        d = tempfile.mkdtemp(prefix="host_engine")
        atexit.register(shutil.rmtree, d, ignore_errors=True)
        for src in (os.path.join(HERE, "fake_cuda.cpp"), os.path.join(B.CSRC, "engine.cpp")):
            subprocess.run([*cxx, "-c", src, "-o", os.path.join(d, os.path.basename(src) + ".o")], check=True)
        _dir = d
    exe = os.path.join(_dir, f"driver{len(_drivers)}")
    with open(exe + ".cpp", "w") as f:
        f.write(source)
    subprocess.run([*cxx, exe + ".cpp", os.path.join(_dir, "fake_cuda.cpp.o"), os.path.join(_dir, "engine.cpp.o"),
                    "-o", exe], check=True)
    return exe


def run_driver(source: str, *args) -> str:
    if source not in _drivers:
        _drivers[source] = _build(source)
    return subprocess.run([_drivers[source], *map(str, args)], check=True, capture_output=True, text=True,
                          timeout=120).stdout
