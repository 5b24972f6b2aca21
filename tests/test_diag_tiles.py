"""Update tiles of the diagonal-block kernel (host): every shared-memory access in bounds,
every element of the lower triangle updated once (CPU driver over the kernel's own index
functions)."""
import os
import shutil
import subprocess

import pytest


def test_update_tiles_stay_in_the_shared_block(pkg, tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "diag_tiles")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(os.path.dirname(pkg.__file__), "csrc"),
                    os.path.join(here, "native", "diag_tiles.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
