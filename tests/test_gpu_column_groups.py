"""Level solves with many columns where a level's chain splits them into groups: every
group's width and remainder (two groups from 9 columns on, four from 17 on) gives the
solutions of the one-unit-per-CTA schedule, which has no groups, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wires", [3, 8, 9, 10, 15, 16, 17, 18, 25, 31, 32])
def test_groups_of_columns_give_the_same_bits(pkg, mg, tmp_path, monkeypatch, wires):
    spec = mg.small_model(cells=9, n_dec=1, steps_per_dec=4, n_sources=wires, n_receivers=2)
    out = []
    for sched in ("0,1", "2,1"):
        monkeypatch.setenv("TDEM_SOLVE_SCHEDULE", sched)
        d = str(tmp_path / sched.replace(",", "_"))
        mg.write_model(d, spec)
        mg.write_analytic_initial_field(d, spec)
        with pkg.Solver(d, "A", 2) as s:
            s.run()
            out.append(s.results())
            assert s.info()["solve_schedule"] == int(sched[0])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
