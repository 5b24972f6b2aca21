"""Device memory of a factorization (host): nothing that only set-up reads is held."""
import os
import shutil
import subprocess

import pytest


def test_maps_of_the_set_up_are_not_held(pkg, tmp_path):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if shutil.which("g++") is None or not os.path.isdir(cuda):
        pytest.skip("no C++ compiler or CUDA headers")
    here = os.path.dirname(os.path.abspath(__file__))
    lib_dir = os.path.dirname(pkg.LIB_PATH)
    exe = str(tmp_path / "held_bytes")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(os.path.dirname(pkg.__file__), "csrc"), "-I", cuda,
                    os.path.join(here, "native", "held_bytes.cpp"), "-L" + lib_dir, "-ltdem_b200",
                    "-Wl,-rpath," + lib_dir, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
