"""Photon batches far beyond the photon buffer: 300 emitters of some twelve million
photons each (more than 2^31 in a tile of 256) into a buffer of 1,000.  The first
1,000 of the stream are kept, the rest dropped and reported."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import params as PR
from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from flim_microscopy_simulator_with_causal_inference_b200.config import config_from_dict
from flim_microscopy_simulator_with_causal_inference_b200.engine import Engine
from flim_microscopy_simulator_with_causal_inference_b200.particles import ParticleState

STATUS_PHOTON_CAP = 0x1


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("emitters", [200, 300])
def test_the_buffer_keeps_the_first_photons(precision, emitters):
    cfg = config_from_dict(W.membrane_pip3_pten(
        counts={"PIP2": 30, "PIP3": emitters, "PI3K": 5, "PTEN_T1": 5, "PTEN_T2": 5}, pools={"PI3K": 2, "PTEN_T1": 2},
        box=3.0, pixels=8, pixel_size_nm=375.0, seed=9))
    st = ParticleState(cfg)
    dp, hill, _ = PR.build_dyn_params(cfg, st.N)
    pp, _ = PR.build_phot_params(cfg, st.N, int(st.has_dye.sum()), 1.0)
    sp, _ = PR.build_scope_params(cfg)
    pp.max_photons = pp.est_photons = 1000
    for dye in range(pp.n_fluoro):
        for state in range(2):
            for c in range(len(pp.mean_d[dye][state])):
                pp.mean_d[dye][state][c], pp.exp_neg_d[dye][state][c] = 1.2e7, 0.0
    eng = Engine([dp], hill, [pp], [sp], precision=precision)
    eng.set_state(st.positions, st.species_id, st.is_alive, st.bond_partner, st.has_dye, st.dye_type_id, st.ctmc_state,
                  st.is_bleached)
    eng.dynamics_step(1)
    eng.photon_step()
    assert eng.photon_counts()[0] == 1000
    pid, _, _, fret = eng.photons(0)
    first = np.flatnonzero(st.has_dye)[0]
    assert (pid == first).all() and not fret.any()
    c = eng.counters()[0]
    assert c[PR.C_PHOTONS] == 1000
    assert eng.status() & STATUS_PHOTON_CAP
