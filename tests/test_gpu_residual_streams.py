"""Residual norms from several threads and streams at once (each call takes its scratch from
the context's pool), and in a process whose context was reset between two calls."""
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_threads_and_streams_do_not_share_scratch(pkg):
    jobs = []
    for k in range(4):
        n = 3000 + 700 * k
        rng = np.random.default_rng(k)
        ptr = np.arange(n + 1, dtype=np.int64) * 27
        dev = [torch.from_numpy(v).cuda() for v in (ptr, rng.integers(0, n, 27 * n).astype(np.int32),
                                                   rng.standard_normal(27 * n), *rng.standard_normal((2, 16, n)))]
        jobs.append((n, dev, torch.cuda.Stream()))

    def call(job, out):
        n, dev, stream = job
        pkg.residual_norms(0, n, *[v.data_ptr() for v in dev], n, 16, out.data_ptr(), stream.cuda_stream)

    alone = [torch.zeros(32, dtype=torch.float64, device="cuda") for _ in jobs]
    torch.cuda.synchronize()
    for job, out in zip(jobs, alone):
        call(job, out)
        torch.cuda.synchronize()
    outs = [[torch.zeros(32, dtype=torch.float64, device="cuda") for _ in range(100)] for _ in jobs]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=lambda j=j, o=o: [call(j, v) for v in o]) for j, o in zip(jobs, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for want, got in zip(alone, outs):
        assert all(torch.equal(want, v) for v in got)


RESET = """
import ctypes, glob, importlib, os, sys
import numpy as np
import torch  # (for its CUDA runtime only: no tensor on the device)
sys.path.insert(0, sys.argv[1])
pkg = importlib.import_module(sys.argv[2])
lib = pkg.load_library()
rt = ctypes.CDLL(None)
if not hasattr(rt, "cudaDeviceReset"):
    names = [l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l]
    rt = ctypes.CDLL(names[0])
def dev(v):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(v.nbytes)) == 0
    assert rt.cudaMemcpy(p, v.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(v.nbytes), 1) == 0
    return p
n = 1000
for k in range(3):
    ptr, col = dev(np.arange(n + 1, dtype=np.int64)), dev(np.arange(n, dtype=np.int32))
    val, x, b = dev(np.full(n, 2.0)), dev(np.ones(n)), dev(np.full(n, 3.0))
    out, norms = dev(np.zeros(2)), np.zeros(2)
    pkg.residual_norms(0, n, ptr.value, col.value, val.value, x.value, b.value, n, 1, out.value, None)
    assert rt.cudaMemcpy(norms.ctypes.data_as(ctypes.c_void_p), out, ctypes.c_size_t(16), 2) == 0
    assert np.allclose(norms, [np.sqrt(1000.0), 3 * np.sqrt(1000.0)], rtol=1e-14, atol=0), norms
    assert rt.cudaDeviceReset() == 0
print("ok")
"""


def test_calls_after_a_context_reset(pkg):
    r = subprocess.run([sys.executable, "-c", RESET, ROOT, PKG], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stderr[-2000:]
