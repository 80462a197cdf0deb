"""Builds csrc/engine.cpp with the host stand-in of the CUDA runtime
(fake_cuda.cpp) and a test's own C++ driver, and runs it."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def run_driver(tmp_path, source: str, *args) -> str:
    from libfluid_gb300 import build as B
    if shutil.which(B.CXX) is None:
        pytest.skip("needs a C++ compiler")
    drv, exe = tmp_path / "driver.cpp", tmp_path / "driver"
    drv.write_text(source)
    subprocess.run([B.CXX, *B.CXX_FLAGS, "-O1", f"-I{HERE}", str(drv), os.path.join(HERE, "fake_cuda.cpp"),
                    os.path.join(B.CSRC, "engine.cpp"), "-o", str(exe)], check=True)
    return subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True, text=True, timeout=120).stdout
