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
