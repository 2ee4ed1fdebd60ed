"""The reaction passes taken by one block per replica (k_react) at their edges,
against the oracle (float64, free running):

* long_walk: conversions, detachments and catalysis of thousands of particles
  per step, so that a replica's list outgrows its shared-memory part (512
  entries), its grid changes outgrow theirs (512), and a block walks its lists
  in several rounds;
* late_draws: a conversion of a species that the catalytic passes produce, so
  that the draw sweep runs after them and only the passes behind it are the
  block's;
* long_lists: more expected entries than a block takes (10^6): the passes run
  as launches of their own.
"""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests.harness import Pair, compare_state

F64_TOL = 1e-12  # µm


def _system(name: str) -> dict:
    counts = {"PIP2": 2000, "PIP3": 700, "PI3K": 300, "PTEN_T1": 900, "PTEN_T2": 700}
    pools, box, seed = {"PI3K": 60, "PTEN_T1": 100}, 3.0, 31
    if name == "late_draws":
        counts, box = {k: v // 4 for k, v in counts.items()}, 1.6
    if name == "long_lists":
        counts, box = W.scaled_counts(200_000), 75.6
    d = W.membrane_pip3_pten(counts=counts, pools=pools, box=box, pixels=8, pixel_size_nm=box * 125.0, seed=seed)
    for c in d["catalytic_reactions"]:
        c["k_cat"] = 8000.0 if name == "long_lists" else 3000.0
        c["contact_radius"] = 60.0 if name == "long_lists" else 30.0
    for ex in d["compartment_exchanges"]:
        ex["k_on"], ex["k_off"], ex["max_recruits_per_step"] = ex["k_on"] * 1000.0, ex["k_off"] * 200.0, 8
    for cv in d["unimolecular_conversions"]:
        cv["rate"] = 12000.0
    if name == "late_draws":
        d["unimolecular_conversions"].append({"name": "PIP3_back", "from_species": "PIP3", "to_species": "PIP2",
                                              "rate": 500.0, "feedback_rule": "pip3_activation"})
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("name,steps", [("long_walk", 10), ("late_draws", 30), ("long_lists", 2)])
def test_passes_match_the_oracle(name, steps):
    P = Pair(_system(name), precision=64, photons=False)
    for t in range(steps):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        if t % 5 == 4 or t == steps - 1:
            compare_state(P.gpu_state(), P.orc, F64_TOL)
    c = P.orc.counters[:6]
    assert np.array_equal(P.eng.counters()[0][:6], c), (P.eng.counters()[0][:6], c)
    assert (c[2:6] > 0).all(), c
    assert P.eng.status() == 0
