"""The reaction passes in crowded systems, whose conversions look at many neighbours:
one replica's go as launches of their own, a block per replica takes those of four
(whose limit is four times as high) and of a sparse one.  Either way the same."""
import math

import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble


def _system(per_um2: float, k_cat: float) -> dict:
    box = math.sqrt(500 / per_um2)
    d = W.membrane_pip3_pten(counts=W.scaled_counts(500), pools=W.scaled_pools(500), box=box, pixels=8,
                             pixel_size_nm=box * 125.0, seed=3)
    d["catalytic_reactions"][0].pop("feedback_rule")
    for c in d["catalytic_reactions"]:
        c["k_cat"] = k_cat
    return d


def _passes(ens: Ensemble) -> list:
    return [kind for kind, _, _ in ens.engine.profile_passes(1)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
def test_crowded_passes_in_launches_and_in_a_block(precision):
    raw = _system(1000.0, 10.0)
    one, four = (Ensemble([raw] * R, precision=precision, photons=False) for R in (1, 4))
    assert "react" not in _passes(one) and "react" in _passes(four)
    for e in (one, four):
        e.engine.dynamics_step(30)
    g, h = four.engine.get_state(), one.engine.get_state()
    for r in range(4):
        for key in ("positions", "species", "alive"):
            assert np.array_equal(g[key][four.replica_slice(r)], h[key]), (r, key)
        assert np.array_equal(four.engine.counters()[r], one.engine.counters()[0])
    assert one.engine.counters()[0][2] > 100 and one.engine.status() == four.engine.status() == 0


@pytest.mark.gpu
def test_a_sparse_system_keeps_its_block():
    assert "react" in _passes(Ensemble([_system(130.0, 10.0)], precision=32, photons=False))
