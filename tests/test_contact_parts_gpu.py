"""Dense replicas of an ensemble, whose listed contacts in one step outnumber the
replica's own part of the contact list: each equals itself alone in an engine, bit
for bit, and nothing is reported lost."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble


def _system(n: int, seed: int) -> dict:
    """n particles in a three-cell box: every enzyme is in contact with one substrate in three."""
    d = W.membrane_pip3_pten(counts={"PIP2": int(0.3 * n), "PIP3": int(0.35 * n), "PI3K": int(0.15 * n),
                                     "PTEN_T1": int(0.15 * n), "PTEN_T2": int(0.05 * n)},
                             pools={"PI3K": 10, "PTEN_T1": 10}, box=0.5, pixels=8, pixel_size_nm=62.5, seed=seed)
    d["potentials"] = []  # nobody is pushed out of a contact
    for c in d["catalytic_reactions"]:
        c.pop("feedback_rule", None)
        c["k_cat"] = 40.0
    return d


def _compare(ens: Ensemble, raws: list, set_state, precision: int, steps: int) -> np.ndarray:
    assert "react" in [k for k, _, _ in ens.engine.profile_passes(1)]  # a block per replica
    set_state(ens, range(len(raws)))
    ens.engine.set_step(0)
    before = ens.engine.counters()
    ens.engine.dynamics_step(steps)
    g, c = ens.engine.get_state(), ens.engine.counters() - before
    assert ens.engine.status() == 0
    for r, raw in enumerate(raws):
        one = Ensemble([raw], precision=precision, photons=False)
        set_state(one, [r])
        one.engine.dynamics_step(steps)
        h = one.engine.get_state()
        for key in ("positions", "species", "alive"):
            assert np.array_equal(g[key][ens.replica_slice(r)], h[key]), (r, key)
        assert np.array_equal(c[r], one.engine.counters()[0])
        assert one.engine.status() == 0
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
def test_dense_replicas_equal_themselves_alone(precision):
    """One catalytic reaction: only the contact search files pairs."""
    raws = [_system(n, 11 + n) for n in (7000, 200, 3000)]
    for d in raws:
        d["catalytic_reactions"] = d["catalytic_reactions"][1:2]
    ens = Ensemble(raws, precision=precision, photons=False)
    c = _compare(ens, raws, lambda e, _: e.upload(), precision, 3)
    assert c[0][2] > 0.9 * raws[0]["initial_populations"]["PIP3"], "few conversions: the lists are short"


@pytest.mark.gpu
def test_crowded_corners_equal_themselves_alone():
    """Sparse boxes whose particles all stand in a corner: the conversions of the first
    pass file late contacts behind the search's."""
    raws = []
    for n in (6000, 300, 5000):
        d = _system(n, 5 + n)
        d["membrane"]["size"] = [40.0, 40.0]
        raws.append(d)

    def set_state(e, replicas):
        h = e.host
        h["positions"] = np.ascontiguousarray(h["positions"] * (0.5 / 40.0))
        e.upload()

    ens = Ensemble(raws, precision=64, photons=False)
    c = _compare(ens, raws, set_state, 64, 1)
    assert (c[[0, 2], 2] > 3000).all(), c[:, 2]
