"""The photon pass in tiles of 256 emitters against the oracle (float64): one
emitter below, at and above a tile's edge and several tiles, with hundreds of
photons per tile and step, through eager steps (photon streams) and graph
chunks (TCSPC stacks, photon counters), where the pass runs beside the next
step's scan and sort; proximity FRET, whose pass must not, in graph chunks."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import params as PR
from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests import cases
from tests.harness import Pair, compare_state

F64_TOL = 1e-12  # µm


def _system(emitters: int) -> dict:
    d = W.membrane_pip3_pten(counts={"PIP2": 300, "PIP3": emitters, "PI3K": 30, "PTEN_T1": 60, "PTEN_T2": 30},
                             pools={"PI3K": 20, "PTEN_T1": 20}, box=3.2, pixels=16, pixel_size_nm=200.0, seed=41,
                             k_cat_scale=500.0)
    d["laser"]["power"] = 2.0e-3
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("emitters", [1, 255, 256, 257, 1100])
def test_photon_streams_and_stacks(emitters):
    import torch
    raw = _system(emitters)
    P, Q = Pair(raw, precision=64), Pair(raw, precision=64)
    photons = 0
    for t in range(12):
        P.eng.dynamics_step(1)
        P.eng.photon_step()
        P.eng.scope_process()
        ob = P.orc.bd_step()
        pid, tt, ch, fr = P.eng.photons(0)
        assert np.array_equal(pid, ob[0]), f"photon emitters differ at step {t}"
        assert np.array_equal(ch, ob[2]) and np.array_equal(fr, ob[3])
        np.testing.assert_allclose(tt, ob[1], rtol=1e-14, atol=0)
        photons += pid.size
    assert photons > 0
    assert np.array_equal(P.eng.flim(0), P.orc.flim)
    c = P.eng.counters()[0]
    assert c[PR.C_PHOTONS] == photons and c[PR.C_RECEIVED] == photons
    s = torch.cuda.Stream()
    Q.eng.pipeline_steps(12, True, 6, stream=s)
    s.synchronize()
    assert np.array_equal(Q.eng.flim(0), P.eng.flim(0))
    assert np.array_equal(Q.eng.counters(), P.eng.counters())


@pytest.mark.gpu
def test_proximity_fret_in_graph_chunks():
    import torch
    P = Pair(cases.get("proximity_small"), precision=64)
    s = torch.cuda.Stream()
    P.eng.pipeline_steps(30, True, 10, stream=s)
    s.synchronize()
    for _ in range(30):
        P.orc.bd_step()
    assert np.array_equal(P.eng.flim(0), P.orc.flim)
    compare_state(P.gpu_state(), P.orc, F64_TOL)


@pytest.mark.gpu
def test_host_batch_of_particles_without_dye():
    """A batch from the host may name any particle, the sorts keep the slots of
    dye carriers only: detection after 9 steps equals detection by an engine
    that was given the state at that point."""
    P, Q = Pair(_system(200), precision=64), Pair(_system(200), precision=64)
    P.eng.dynamics_step(9)
    g = P.gpu_state()
    st = P.state
    Q.eng.set_state(g["positions"], g["species"], g["alive"], g["bond"], g["has_dye"], st.dye_type_id, g["ctmc"],
                    g["bleached"])
    pid = np.flatnonzero(~st.has_dye)[:300].astype(np.int32)
    for X in (P, Q):
        X.eng.set_photons(0, pid, np.linspace(0.0, 2.0e-8, pid.size), np.zeros(pid.size, np.int8),
                          np.zeros(pid.size, np.uint8), batch_key=5)
        X.eng.scope_process()
    a, b = P.eng.flim(0), Q.eng.flim(0)
    assert a.sum() > 0 and np.array_equal(a, b)
