"""Binding candidates settled by a block per replica and dissociations by list,
against the oracle (float64): hundreds of candidates in a step, most of them
sharing a particle with another; more dissociations in a step than one block's
threads (several blocks per replica); and a state whose complexes' partners are
alive, which the candidates may take before the dissociation does."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests.harness import Pair, compare_state

F64_TOL = 1e-12  # µm


def _system(name: str) -> dict:
    box = 4.0
    counts = {"contested": (500, 900), "lists": (1600, 1700), "awake": (300, 900)}[name]
    d = W.membrane_pip3_pten(counts={"PIP2": 20, "PIP3": counts[1], "PI3K": 6, "PTEN_T1": 8, "PTEN_T2": 4},
                             pools={"PI3K": 4, "PTEN_T1": 4}, box=box, pixels=8, pixel_size_nm=box * 125.0, seed=41,
                             k_cat_scale=0.0)
    d["species"].append({"name": "Sensor", "diffusion_coefficient": 0.08, "radius": 3.0})
    d["species"].append({"name": "Complex", "diffusion_coefficient": 0.06, "radius": 3.5})
    d["initial_populations"]["Sensor"] = counts[0]
    d["reactions"] = [{"name": "bind", "reactants": ["Sensor", "PIP3"], "products": ["Complex"], "kon": 1.0e6,
                       "koff": 3000.0, "contact_radius": {"contested": 60.0, "lists": 5.0, "awake": 30.0}[name]}]
    return d


def _bind_initially(o, sid, n: int, awake: bool) -> None:
    """The first n sensors of the oracle's state as complexes of the first n lipids."""
    a, b = np.flatnonzero(o.species == sid["Sensor"])[:n], np.flatnonzero(o.species == sid["PIP3"])[:n]
    o.species[a] = sid["Complex"]
    o.bond[a] = b
    if not awake:
        o.bond[b] = a
        o.alive[b] = False


@pytest.mark.gpu
@pytest.mark.parametrize("name,bound", [("contested", 0), ("lists", 1600), ("awake", 200)])
def test_binding_matches_the_oracle(name, bound):
    P = Pair(_system(name), precision=64, photons=False)
    sid = {s.name: k for k, s in enumerate(P.cfg.species)}
    _bind_initially(P.orc, sid, bound, name == "awake")
    P.load_oracle_state_into_gpu()
    # in the sixth step of the last case two complexes that share a partner
    # dissociate, and either may place it last
    for t in range(5 if name == "awake" else 6):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        compare_state(P.gpu_state(), P.orc, F64_TOL)
    assert np.array_equal(P.eng.counters()[0][:6], P.orc.counters[:6])
    assert (P.orc.counters[:2] > 50).all(), P.orc.counters[:2]
    assert P.eng.status() == 0
