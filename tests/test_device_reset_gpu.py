"""A host program may reset the device between two uses of the library: its memory
pool is made anew in the new context."""
import os
import shutil
import subprocess

import pytest

from cola_b200 import _lib

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_build_after_device_reset(tmp_path):
    exe = str(tmp_path / "device_reset_main")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-I", os.path.join(REPO, "include"), "-I",
                           "/usr/local/cuda/include", os.path.join(REPO, "tests", "device_reset_main.cpp"), "-o", exe,
                           "-L", os.path.dirname(_lib.LIB_PATH), "-lcola_b200", "-L", "/usr/local/cuda/lib64",
                           "-lcudart", "-Wl,-rpath," + os.path.dirname(_lib.LIB_PATH)])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-2000:] + r.stderr[-2000:]
