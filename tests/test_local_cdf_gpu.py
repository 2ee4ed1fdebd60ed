"""Density-biased recruitment against the oracle (float64) where its kernel's
work divides: feedback grids of 484 cells (not a multiple of the eight the
summing thread holds ahead), 529 (past one tile of 512) and 1,024 (two full
tiles); few recruitment candidates (most steps need no cumulative density) and
many."""
import numpy as np
import pytest

from tests import cases
from tests.harness import Pair, compare_state

F64_TOL = 1e-12  # µm


@pytest.mark.gpu
@pytest.mark.parametrize("box", [22.0, 23.0, 32.0])
@pytest.mark.parametrize("rate", [0.02, 5.0])
def test_local_recruitment_matches_the_oracle(box, rate):
    d = cases.get("adaptive_local")
    d["membrane"]["size"] = [box, box]
    for ex in d["compartment_exchanges"]:
        ex["k_on"] *= rate
    P = Pair(d, precision=64, photons=False)
    ex = next(x for x in P.dp.exch[:P.dp.n_exch] if x.local_recruit)
    grid = P.dp.grid[P.dp.rule[ex.rule_on].grid]
    assert grid.nx == grid.ny == int(box)
    for t in range(60):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        if t % 10 == 9:
            compare_state(P.gpu_state(), P.orc, F64_TOL)
    assert np.array_equal(P.eng.counters()[0][:6], P.orc.counters[:6])
    assert P.orc.counters[3] > 0, "nobody was recruited"
    assert P.eng.status() == 0
