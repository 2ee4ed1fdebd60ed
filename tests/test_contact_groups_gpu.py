"""The grouped neighbour sweep of the contact search at its edges.

Lane groups walk the runs of the 3x3 block's columns laid end to end, with a
second part for the row that wraps in y.  A three-cell periodic box (every
column wraps, every row is some particle's wrapped row, some fifty neighbours
a sweeper: several rounds of 4, 8 and 16 lanes) and a closed box (runs cut at
the walls), each with the tile form (0, 1) and the list form at 8, 4 and 16
lanes per sweeper (2, 3, 4): the float64 path against the oracle, the float32
path against its own tile form bit for bit.
"""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests.harness import Pair, compare_state

F64_TOL = 1e-12  # µm


def _system(walls: bool) -> dict:
    d = W.membrane_pip3_pten(counts={"PIP2": 80, "PIP3": 30, "PI3K": 10, "PTEN_T1": 12, "PTEN_T2": 8},
                             pools={"PI3K": 5, "PTEN_T1": 6}, box=1.1 if walls else 0.5, pixels=8,
                             pixel_size_nm=137.0 if walls else 62.0, seed=23, k_cat_scale=20000.0)
    if walls:
        d["membrane"]["periodic"] = [False, False]
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("shape", [0, 1, 2, 3, 4])
def test_grouped_sweep_matches_the_oracle(walls, shape):
    P = Pair(_system(walls), precision=64, photons=False)
    P.eng.set_launch_shapes([-1, -1, shape])
    for t in range(40):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        if t % 10 == 9:
            compare_state(P.gpu_state(), P.orc, F64_TOL)
    assert np.array_equal(P.eng.counters()[0][:6], P.orc.counters[:6])
    assert P.orc.counters[2] > 0, "no catalytic events"
    assert P.eng.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [False, True])
def test_float32_forms_agree(walls):
    ref = None
    for shape in (0, 2, 3, 4):
        P = Pair(_system(walls), precision=32, photons=False)
        P.eng.set_launch_shapes([-1, -1, shape])
        P.eng.dynamics_step(30)
        run = dict(P.gpu_state(), counters=P.eng.counters())
        ref = ref or run
        for k in ref:
            assert np.array_equal(ref[k], run[k]), (shape, k)
