"""Kernels launched as programmatic dependents (source check): the vectors that the chain's
kernels write are not declared constant in a kernel that may start before its predecessor
has ended."""
import os
import re


def test_dependents_do_not_declare_the_chains_vectors_constant(pkg):
    with open(os.path.join(os.path.dirname(pkg.__file__), "csrc", "gpu_cholesky.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    names = set(re.findall(r"launch_next\((k_\w+)", src)) | set(re.findall(r"\bgo\((k_\w+mrhs)<", src))
    assert {"k_fwd_gather", "k_bwd_init", "k_fwd_stream", "k_bwd_stream", "k_fwd_mrhs", "k_bwd_mrhs",
            "k_fwd_level", "k_bwd_level"} <= names
    for name in names:
        params = re.search(r"__global__[^;{]*?\b%s\(([^)]*)\)" % name, src).group(1)
        for p in params.split(","):
            if re.search(r"\b(W|x|part)\s*$", p):
                assert not ("const" in p and "__restrict__" in p), (name, p.strip())


def test_a_solve_reports_launches_that_fail(pkg, tmp_path):
    """Without a device every CUDA call of a solve fails, which its callers are told (host
    driver over the library)."""
    import shutil
    import subprocess
    import pytest
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if shutil.which("g++") is None or not os.path.isdir(cuda):
        pytest.skip("no C++ compiler or CUDA headers")
    here = os.path.dirname(os.path.abspath(__file__))
    lib_dir = os.path.dirname(pkg.LIB_PATH)
    exe = str(tmp_path / "solve_launch_errors")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(os.path.dirname(pkg.__file__), "csrc"), "-I", cuda,
                    os.path.join(here, "native", "solve_launch_errors.cpp"), "-L" + lib_dir, "-ltdem_b200",
                    "-Wl,-rpath," + lib_dir, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
