"""The PSF projection's two tiles (128 x 64 for few fields of view, 128 x 256 from 32):
a field of view of a large batch equals the same one of a small batch bit for bit (the
same products, summed in the same order), and the float64 projection within the
band test's tolerance."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import flim_acquire as FA
from oracle import flim_oracle as FO

pytestmark = pytest.mark.gpu

SEED = 5


@pytest.mark.parametrize("taps", [0, 15, 64, 127])
def test_large_batches_project_as_small_ones(monkeypatch, taps):
    build = FA.build_flim_params

    def with_taps(*a, **k):
        p, d = build(*a, **k)
        p.half_taps, p.sigma_psf_px = taps, max(0.7, taps / 3.0)
        return p, d

    monkeypatch.setattr(FA, "build_flim_params", with_taps)
    bound = np.linspace(0.0, 1.0, 33)
    maps = {}
    for R in (2, 31, 32, 33):
        a = FA.FlimAcquisition(FA.flim_config(), R, n_emitters=50_000, photon_budget=5.0, seed=SEED,
                               bound_fraction=bound[:R])
        a.project()
        maps[R] = a.read(FA.INTENSITY)
        assert a.error_word() == 0
        sigma = a.params.sigma_psf_px
        a.close()
    for R in (2, 31, 32):
        np.testing.assert_array_equal(maps[R], maps[33][:R])
    G = FO.band(sigma, taps)
    I = FO.intensity(FO.emitter_counts(SEED, 32, 50_000, bound[32]), G)
    assert np.abs(maps[33][32] - I).max() <= (3e-5 + 2 * (2 * taps + 1) * 2.0 ** -23) * I.max()
