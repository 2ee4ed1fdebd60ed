"""The grouped sweep of the binding candidates at its edges, against the oracle
(float64): a three-cell periodic box (every row wraps for some particle, several
rounds of lanes per sweeper), closed walls, the binding species swept from
either side (whichever is rarer at the first state), and a homodimer, whose
pairs are seen from both partners.  No catalysis: in a box this small a partner
that dissociates within a step can also meet an enzyme of its stale position."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests.harness import Pair, compare_state

F64_TOL = 1e-12  # µm


def _system(box: float, walls: bool, sensors: int, reactants) -> dict:
    d = W.membrane_pip3_pten(counts={"PIP2": 20, "PIP3": 40, "PI3K": 6, "PTEN_T1": 8, "PTEN_T2": 4},
                             pools={"PI3K": 4, "PTEN_T1": 4}, box=box, pixels=8, pixel_size_nm=box * 125.0, seed=29,
                             k_cat_scale=0.0)
    if walls:
        d["membrane"]["periodic"] = [False, False]
    d["species"].append({"name": "Sensor", "diffusion_coefficient": 0.08, "radius": 3.0})
    d["species"].append({"name": "Complex", "diffusion_coefficient": 0.06, "radius": 3.5})
    d["initial_populations"]["Sensor"] = sensors
    d["reactions"] = [{"name": "bind", "reactants": list(reactants), "products": ["Complex"],
                       "kon": 5.0, "koff": 400.0, "contact_radius": 40.0}]
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("box,walls", [(0.5, False), (1.1, True)])
@pytest.mark.parametrize("sensors,reactants", [(20, ("Sensor", "PIP3")), (60, ("Sensor", "PIP3")),
                                               (60, ("Sensor", "Sensor"))])
def test_binding_matches_the_oracle(box, walls, sensors, reactants):
    P = Pair(_system(box, walls, sensors, reactants), precision=64, photons=False)
    for t in range(40):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        if t % 10 == 9:
            compare_state(P.gpu_state(), P.orc, F64_TOL)
    c = P.orc.counters[:6]
    assert np.array_equal(P.eng.counters()[0][:6], c)
    assert c[0] > 0, "no binding"
    assert P.eng.status() == 0
