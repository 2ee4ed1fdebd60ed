"""Particles woken by a dissociation in the passes behind it, against the oracle
(float64).  The reference's pair list holds every particle, so one that wakes in a
step can meet an enzyme, a substrate, another woken particle or a binding partner
in the same step by the place it slept in; the engine's cells hold the alive ones.

* substrate / enzyme: the woken species is the substrate (the enzyme) of the
  catalytic passes, swept from either side;
* both: two bindings wake substrates and enzymes, and a catalytic pass makes
  substrates that woken enzymes take in the same step;
* rebind: a second binding reaction takes what the first one freed;
* dimer: what the first one freed binds to its own kind.
"""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble
from tests.harness import Pair, compare_state

F64_TOL = 1e-12  # µm
BINDINGS = {"substrate": [("Sensor", "PIP3")], "enzyme": [("Sensor", "PTEN_T1")],
            "both": [("Sensor", "PIP3"), ("Anchor", "PTEN_T1")], "rebind": [("Sensor", "PIP3"), ("Anchor", "PIP3")],
            "dimer": [("Sensor", "PIP3"), ("PIP3", "PIP3")]}


def _system(name: str, walls: bool) -> dict:
    box = 1.1 if walls else 0.5
    k = 3 if walls else 1
    d = W.membrane_pip3_pten(counts={"PIP2": 30 * k, "PIP3": 40 * k, "PI3K": 6 * k, "PTEN_T1": 20 * k, "PTEN_T2": 4 * k},
                             pools={"PI3K": 4, "PTEN_T1": 4}, box=box, pixels=8, pixel_size_nm=box * 125.0, seed=29)
    for c, k_cat in zip(d["catalytic_reactions"], (150.0, 20.0, 20.0)):
        c["k_cat"] = k_cat
    if walls:
        d["membrane"]["periodic"] = [False, False]
    for s in ("Sensor", "Anchor"):
        d["species"].append({"name": s, "diffusion_coefficient": 0.08, "radius": 3.0})
        d["initial_populations"][s] = 15 * k
    d["reactions"] = []
    for i, (a, b) in enumerate(BINDINGS[name]):
        d["species"].append({"name": f"Complex{i}", "diffusion_coefficient": 0.06, "radius": 3.5})
        d["reactions"].append({"name": f"bind{i}", "reactants": [a, b], "products": [f"Complex{i}"], "kon": 300.0,
                               "koff": 3000.0, "contact_radius": 40.0})
    return d


def _compare(P: Pair, steps: int) -> None:
    for t in range(steps):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        if t % 10 == 9:
            compare_state(P.gpu_state(), P.orc, F64_TOL)
    c = P.orc.counters[:6]
    assert np.array_equal(P.eng.counters()[0][:6], c), (P.eng.counters()[0][:6], c)
    assert (c[:3] > 25).all(), c
    assert P.eng.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("name", list(BINDINGS))
@pytest.mark.parametrize("sides", [0, 7])
def test_woken_particles_match_the_oracle(name, walls, sides):
    P = Pair(_system(name, walls), precision=64, photons=False)
    P.eng.contact_sides(sides)
    _compare(P, 60)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [2, 3, 4])
def test_over_the_sweeper_list(shape):
    P = Pair(_system("both", False), precision=64, photons=False)
    P.eng.set_launch_shapes([-1, -1, shape])
    _compare(P, 60)


@pytest.mark.gpu
def test_float32_sides_agree():
    runs = []
    for mask in (0, 7):
        P = Pair(_system("both", True), precision=32, photons=False)
        P.eng.contact_sides(mask)
        P.eng.dynamics_step(60)
        runs.append(dict(P.gpu_state(), counters=P.eng.counters()))
    for key in runs[0]:
        assert np.array_equal(runs[0][key], runs[1][key]), key


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
def test_replicas_in_launches_of_their_own_agree_with_one_alone(precision):
    """Two replicas whose catalytic probabilities reach 0.1 a step: the passes go
    as separate launches there and as one in an engine of one replica."""
    raw = _system("both", True)
    raw["catalytic_reactions"][1]["k_cat"] = 100.0
    ens, one = Ensemble([raw] * 2, precision=precision, photons=False), Ensemble([raw], precision=precision,
                                                                               photons=False)
    assert "catalytic" in [k for k, _, _ in ens.engine.profile_passes(1)]
    assert "react" in [k for k, _, _ in one.engine.profile_passes(1)]
    ens.engine.dynamics_step(40)
    one.engine.dynamics_step(40)
    g, h = ens.engine.get_state(), one.engine.get_state()
    for r in range(2):
        for key in ("positions", "species", "alive", "bond"):
            assert np.array_equal(g[key][ens.replica_slice(r)], h[key]), (r, key)
        assert np.array_equal(ens.engine.counters()[r], one.engine.counters()[0])
