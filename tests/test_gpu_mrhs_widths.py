"""Many-column level solves at every width of their kernels (up to 8, 16 and 32 columns a
group, one or more tiles of eight, the last one padded): the number of groups is set, and
once left to the rule on a mesh where it takes one, two and four on different levels.
Against the one-unit-per-CTA schedule, which multiplies the same blocks column tile by tile
but applies the inverted diagonal blocks on the CUDA cores: the same system, so the parity
tolerance of two direct solvers."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import FP64_TOL

pytestmark = pytest.mark.gpu


def _runs(pkg, mg, tmp_path, monkeypatch, cells, wires, schedules):
    spec = mg.small_model(cells=cells, n_dec=1, steps_per_dec=4, n_sources=wires, n_receivers=2)
    d = str(tmp_path / "m")
    mg.write_model(d, spec)
    mg.write_analytic_initial_field(d, spec)
    out = []
    for sched in schedules:
        monkeypatch.setenv("TDEM_SOLVE_SCHEDULE", sched)
        with pkg.Solver(d, "A", 2) as s:
            s.run()
            out.append(s.results())
            assert s.info()["solve_schedule"] == int(sched[0])
    return d, out


def _agree(got, want):
    for a, b in zip(got, want):
        assert np.all(np.isfinite(a)) and np.abs(a - b).max() <= FP64_TOL * np.abs(b).max()


@pytest.mark.parametrize("wires", [9, 15, 16, 17, 25, 31, 32])
def test_every_number_of_groups(pkg, mg, tmp_path, monkeypatch, wires):
    groups = [1, 2] + ([4] if wires > 16 else [])
    _, (want, *got) = _runs(pkg, mg, tmp_path, monkeypatch, 9, wires, ["0,1"] + ["2,1,%d" % g for g in groups])
    for g in got:
        _agree(g, want)


@pytest.mark.parametrize("wires", [9, 17, 32])
def test_groups_by_the_rule(pkg, mg, tmp_path, monkeypatch, wires):
    d, (want, got) = _runs(pkg, mg, tmp_path, monkeypatch, 24, wires, ["0,1", "2,1"])
    _agree(got, want)
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if shutil.which("g++") is None or not os.path.isdir(cuda):
        return
    here, lib_dir, exe = os.path.dirname(os.path.abspath(__file__)), os.path.dirname(pkg.LIB_PATH), str(tmp_path / "groups")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(os.path.dirname(pkg.__file__), "csrc"), "-I", cuda,
                    os.path.join(here, "native", "column_groups.cpp"), "-L" + lib_dir, "-ltdem_b200",
                    "-Wl,-rpath," + lib_dir, "-o", exe], check=True)
    r = subprocess.run([exe, d, str(wires)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
    assert set(r.stdout.split()[1:]) == ({"1", "2"} if wires <= 16 else {"1", "2", "4"})


def test_schedules_that_are_refused(pkg, mg, tmp_path, monkeypatch):
    spec = mg.small_model(cells=6, n_dec=1, steps_per_dec=4, n_sources=3, n_receivers=1)
    mg.write_model(str(tmp_path), spec)
    mg.write_analytic_initial_field(str(tmp_path), spec)
    for sched in ("2,1,3", "2,1,8", "3,1", "2"):
        monkeypatch.setenv("TDEM_SOLVE_SCHEDULE", sched)
        with pytest.raises(pkg.TdemError, match="TDEM_SOLVE_SCHEDULE"):
            pkg.Solver(str(tmp_path), "A", 2)
