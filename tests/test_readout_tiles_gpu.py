"""Lifetime readouts at the edges of their pixel groups (8 per warp step) and
row lengths (1 to 64 words of four bins, an odd word count among them), counts
up to 2^32 - 1, against the float64 restatement: rtol 1e-12, exact intensity."""
import numpy as np
import pytest
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import readouts as RD
from oracle import flim_oracle as FO


@pytest.mark.gpu
@pytest.mark.parametrize("n_bins", [4, 8, 12, 64, 100, 128, 252, 256])
@pytest.mark.parametrize("n_px", [1, 7, 8, 9, 95, 96, 97, 60_001])
def test_groups_and_rows(n_bins, n_px):
    rng = np.random.default_rng(n_bins * 100_003 + n_px)
    stack = rng.poisson(30.0 * np.exp(-np.arange(n_bins) / (0.2 * n_bins)), (n_px, n_bins)).astype(np.uint32)
    stack[rng.random(n_px) < 0.1] = 0
    if n_px > 1:
        stack[n_px // 2] = np.uint32(2 ** 32 - 1) - rng.integers(0, 9, n_bins).astype(np.uint32)
    dev = torch.from_numpy(stack.view(np.int32)).cuda()
    out = RD.lifetimes_device(dev.data_ptr(), n_px, n_bins, 25e-9).cpu().numpy()
    ref = FO.readouts(stack, 25e-9)
    np.testing.assert_array_equal(out[0], ref["intensity"])
    for i, k in enumerate(RD.FIELDS):
        if k in ("tau_phi_ns", "tau_mod_ns"):  # 1e-14 absolute in g and s, divided by them
            ok = np.hypot(ref["g"], ref["s"]) > 1e-3
            np.testing.assert_allclose(out[i][ok], ref[k][ok], rtol=1e-10, atol=0, equal_nan=True, err_msg=k)
        else:
            np.testing.assert_allclose(out[i], ref[k], rtol=1e-12, atol=1e-14, equal_nan=True, err_msg=k)
