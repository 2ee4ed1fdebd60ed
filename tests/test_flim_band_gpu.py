"""The PSF projection's band for every kind of half-width (the K chunks a tile loads
follow from it: none but its own, one more on either side, all), and the histogram
writer for 128 bins, against the float64 oracle.

Intensity: BF16 hi/lo-split factors keep 16 bits, two of them a product, 3e-5 of the
map's largest value in all; the FP32 sums of 2 taps + 1 terms in either pass add at
most that many roundings of 2^-24, taken twice for the accumulator's truncation."""
import math

import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import flim_acquire as FA
from oracle import flim_oracle as FO

pytestmark = pytest.mark.gpu

SEED = 77
BOUND = np.array([0.3, 1.0])


@pytest.mark.parametrize("taps", [0, 1, 15, 31, 32, 33, 63, 64, 65, 100, 127])
def test_projection_over_band_half_widths(monkeypatch, taps):
    build = FA.build_flim_params

    def with_taps(*a, **k):
        p, d = build(*a, **k)
        p.half_taps, p.sigma_psf_px = taps, max(0.7, taps / 3.0)
        return p, d

    monkeypatch.setattr(FA, "build_flim_params", with_taps)
    a = FA.FlimAcquisition(FA.flim_config(), 2, n_emitters=50_000, photon_budget=50.0, seed=SEED, bound_fraction=BOUND)
    try:
        a.acquire()
        got, counts = a.read(FA.INTENSITY), a.read(FA.COUNTS)
        assert a.error_word() == 0
        for r in range(2):
            G = FO.band(a.params.sigma_psf_px, taps)
            want = FO.emitter_counts(SEED, r, 50_000, BOUND[r])
            np.testing.assert_array_equal(counts[r], want)
            I = FO.intensity(want, G)
            tol = 3e-5 + 2 * (2 * taps + 1) * 2.0 ** -23
            assert np.abs(got[r] - I).max() <= tol * I.max(), (r, np.abs(got[r] - I).max() / I.max())
    finally:
        a.close()


@pytest.mark.parametrize("budget", [30.0, 1000.0])
def test_histograms_of_128_bins(budget):
    """Per-bin totals and per-pixel totals within 6 sigma of the float64 means; the
    expected lifetime map; the same counts when drawn again."""
    cfg = FA.flim_config()
    cfg["tcspc"]["n_bins"] = 128
    a = FA.FlimAcquisition(cfg, 2, n_emitters=50_000, photon_budget=budget, seed=SEED, bound_fraction=BOUND)
    try:
        a.acquire()
        hist, tau = a.read(FA.HIST), a.read(FA.TAU)
        assert hist.shape[-1] == 128 and a.error_word() == 0
        np.testing.assert_allclose(a.read(FA.BINS), FO.acquire_expected(a.params, BOUND, 0)["h"], rtol=1e-12,
                                   atol=1e-300)
        for r in range(2):
            ref = FO.acquire_expected(a.params, BOUND, r)
            exp = ref["mu"].sum(axis=(0, 1))
            z = (hist[r].astype(np.float64).sum(axis=(0, 1)) - exp) / np.sqrt(np.maximum(exp, 1.0))
            assert np.abs(z).max() < 6.0, (r, np.abs(z).max())
            lam, n = ref["mu"].sum(axis=-1), hist[r].astype(np.float64).sum(axis=-1)
            m = lam > 1.0
            assert abs((n[m] - lam[m]).sum()) / math.sqrt(lam[m].sum()) < 6.0
            disp = float((((n[m] - lam[m]) ** 2) / lam[m]).mean())
            assert abs(disp - 1.0) < 6.0 * math.sqrt(3.0 / m.sum()), (r, disp)
            assert np.abs(tau[r][m] - ref["tau"][m]).max() <= 1e-4
        a.acquire()
        np.testing.assert_array_equal(a.read(FA.HIST), hist)
    finally:
        a.close()
