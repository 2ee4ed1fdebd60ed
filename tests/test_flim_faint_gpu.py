"""Histograms of faint fields of view, whose writer runs with half the blocks (256 bins,
below 8 photons a pixel): a field's counts do not depend on how many blocks or other
fields there are, and per-bin totals lie within 6 sigma of the float64 means."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import flim_acquire as FA
from oracle import flim_oracle as FO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_bins", [128, 256])
@pytest.mark.parametrize("budget", [0.3, 7.9, 8.1])
def test_counts_are_the_fields_own(n_bins, budget):
    cfg = FA.flim_config()
    cfg["tcspc"]["n_bins"] = n_bins
    bound = np.linspace(0.1, 0.9, 12)
    hist = {}
    for R in (1, 12):
        a = FA.FlimAcquisition(cfg, R, n_emitters=50_000, photon_budget=budget, seed=31, bound_fraction=bound[:R])
        a.acquire()
        hist[R] = a.read(FA.HIST)
        assert a.error_word() == 0
        params = a.params
        a.close()
    np.testing.assert_array_equal(hist[1][0], hist[12][0])
    for r in (0, 11):
        exp = FO.acquire_expected(params, bound, r)["mu"].sum(axis=(0, 1))
        z = (hist[12][r].astype(np.float64).sum(axis=(0, 1)) - exp) / np.sqrt(np.maximum(exp, 1.0))
        assert np.abs(z).max() < 6.0, (r, np.abs(z).max())
