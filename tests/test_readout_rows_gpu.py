"""Lifetime readouts on both sides of the pixel counts where the kernel's form changes
(2^14 up to 96 bins, 2^20 up to 176, 2^17 above), against the float64 restatement:
rtol 1e-12, exact intensity, and the same values from either side of the line."""
import numpy as np
import pytest
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import readouts as RD
from oracle import flim_oracle as FO


@pytest.mark.gpu
@pytest.mark.parametrize("n_bins,line", [(4, 1 << 14), (16, 1 << 14), (60, 1 << 14), (96, 1 << 14), (100, 1 << 20),
                                         (176, 1 << 20), (180, 1 << 17), (252, 1 << 17)])
def test_both_forms_at_the_line(n_bins, line):
    rng = np.random.default_rng(n_bins)
    n_px = line + 3
    gen = torch.Generator(device="cuda").manual_seed(n_bins)
    mean = 30.0 * torch.exp(-torch.arange(n_bins, device="cuda") / (0.2 * n_bins))
    stack = torch.poisson(mean.expand(n_px, n_bins), generator=gen).to(torch.int32)
    stack[torch.rand(n_px, device="cuda", generator=gen) < 0.1] = 0
    stack[5] = -1  # 2^32 - 1 in every bin
    some = np.unique(np.concatenate([np.arange(40), rng.integers(0, n_px, 2000), np.arange(n_px - 40, n_px)]))
    ref = FO.readouts(stack[some].cpu().numpy().view(np.uint32), 25e-9)
    for n in (line - 1, line, n_px):
        out = RD.lifetimes_device(stack.data_ptr(), n, n_bins, 25e-9).cpu().numpy()
        keep = some < n
        got = out[:, some[keep]]
        np.testing.assert_array_equal(got[0], ref["intensity"][keep])
        for i, k in enumerate(RD.FIELDS):
            want = ref[k][keep]
            if k in ("tau_phi_ns", "tau_mod_ns"):  # 1e-14 absolute in g and s, divided by them
                ok = np.hypot(ref["g"], ref["s"])[keep] > 1e-3
                np.testing.assert_allclose(got[i][ok], want[ok], rtol=1e-10, atol=0, equal_nan=True, err_msg=k)
            else:
                np.testing.assert_allclose(got[i], want, rtol=1e-12, atol=1e-14, equal_nan=True, err_msg=k)
