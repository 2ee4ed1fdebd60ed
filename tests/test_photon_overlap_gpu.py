"""The photon pass's two places in the step.  Up to 2^20 slots it runs after the next
step's sort, beside the move and the contact search; above, beside the next step's
scan and sort, from the copies that the sort does not write.  Replicas of an engine
above that size equal the same replicas in a small one: state, counters and stacks,
through a chunk without a graph, one that is captured and replays."""
import numpy as np
import pytest
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble


def _system(k: int, sensor: bool) -> dict:
    n = 9000 + 37 * k
    box = (n / 130.0) ** 0.5
    d = W.membrane_pip3_pten(counts=W.scaled_counts(n), pools=W.scaled_pools(n), box=box, pixels=16,
                             pixel_size_nm=box * 1000.0 / 16, seed=100 + k, k_cat_scale=20.0)
    d["laser"]["power"] = 4.0e-5
    if sensor:  # binding and bond FRET: flags and bonds that the photon pass reads change in every step
        d["species"] += [{"name": "Sensor", "diffusion_coefficient": 0.08, "radius": 3.0},
                         {"name": "Complex", "diffusion_coefficient": 0.06, "radius": 3.5}]
        d["initial_populations"]["Sensor"] = n // 5
        d["initial_populations"]["PIP2"] -= n // 5
        d["reactions"] = [{"name": "bind", "reactants": ["Sensor", "PIP3"], "products": ["Complex"], "kon": 50.0,
                           "koff": 400.0, "contact_radius": 20.0}]
        d["dye_attachments"] = [{"species": "Sensor", "fluorophore": "mTFP1", "labeling_efficiency": 0.9},
                                {"species": "PIP3", "fluorophore": "Venus", "labeling_efficiency": 0.5}]
        d["fret_pairs"][0]["intramolecular"] = False
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("sensor", [False, True])
def test_both_places_give_the_same(precision, sensor):
    few = 3
    raws = [_system(k % few, sensor) for k in range(84)]
    large = Ensemble(raws, precision=precision, photons=True)
    small = Ensemble(raws[:few], precision=precision, photons=True)
    assert large.engine.N > 1 << 20 and small.engine.N < 1 << 20
    for e in (large, small):
        s = torch.cuda.Stream()
        e.engine.pipeline_steps(40, True, 10, stream=s)
        e.engine.pipeline_steps(3, True, 0, stream=s)
        s.synchronize()
    g, h = large.engine.get_state(), small.engine.get_state()
    gc, hc = large.engine.counters(), small.engine.counters()
    photons = 0
    for r in [0, 1, 2, 81, 82, 83]:
        q = r % few
        for key in g:
            assert np.array_equal(g[key][large.replica_slice(r)], h[key][small.replica_slice(q)]), (r, key)
        assert np.array_equal(gc[r], hc[q]), (r, gc[r], hc[q])
        stack = large.engine.flim(r)
        assert np.array_equal(stack, small.engine.flim(q)), r
        photons += int(stack.sum())
    assert photons > 1000
    assert large.engine.status() == small.engine.status()
