"""The history right-hand side of several sources at the edges of its lane groups (2, 4, 8,
16, 32 sources and more than 32) against the numpy oracle, both schemes' histories."""
import os
import shutil

import pytest

import tdem_oracle
from conftest import FP64_TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wires", [2, 3, 4, 5, 8, 9, 17, 32, 33])
@pytest.mark.parametrize("variant", ["A3", "E2"])
def test_transients_of_every_source_match_the_oracle(pkg, mg, outs, tmp_path, wires, variant):
    ref, d = str(tmp_path / "oracle"), str(tmp_path / "gpu")
    spec = mg.small_model(cells=6, n_dec=2, steps_per_dec=5, n_sources=wires, n_receivers=2)
    mg.write_model(ref, spec)
    mg.write_analytic_initial_field(ref, spec)
    shutil.copytree(ref, d)
    tdem_oracle.run(ref, variant[0], int(variant[1]))
    pkg.run_directory(d, variant[0], int(variant[1]))
    for name in ("edsall_anom", "ball_anom", "eall_anom"):
        for w in range(1, wires + 1):
            f = "%s.%d" % (name, w)
            assert outs.compare_files(os.path.join(d, f), os.path.join(ref, f)) <= FP64_TOL, f
