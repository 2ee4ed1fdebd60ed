"""Lifetime readouts from several host threads at once, with bin counts that share
a kernel but not the amount of shared memory (64 and 100 bins; 4 and 252): each
call sets up and launches on its own, whatever another thread does between."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import engine as E
from flim_microscopy_simulator_with_causal_inference_b200 import readouts as RD


@pytest.mark.gpu
@pytest.mark.parametrize("pair", [(64, 100), (4, 252)])
def test_threads_with_different_bin_counts(pair):
    n_px, calls, bins = 16, 20000, pair * 2
    rng = np.random.default_rng(7)
    dev = [torch.from_numpy(rng.integers(1, 9, (n_px, nb), dtype=np.int32)).cuda() for nb in bins]
    out = [torch.empty((6, n_px), dtype=torch.float64, device="cuda") for _ in bins]
    alone = [RD.lifetimes_device(d.data_ptr(), n_px, nb, 25e-9).cpu().numpy() for d, nb in zip(dev, bins)]
    streams = [torch.cuda.Stream() for _ in bins]
    torch.cuda.synchronize()
    call = E.load_library().edm_readout_lifetimes  # as lifetimes_device calls it
    codes = []
    gate = threading.Barrier(len(bins))

    def work(k):
        args = (C.c_void_p(dev[k].data_ptr()), n_px, bins[k], 25e-9, 1, 10, 20, C.c_void_p(out[k].data_ptr()),
                C.c_void_p(streams[k].cuda_stream))
        gate.wait()
        codes.append(sum(call(*args) != 0 for _ in range(calls)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(bins))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [0] * len(bins), f"calls that failed: {codes}"
    for a, b in zip(alone, out):
        np.testing.assert_array_equal(a, b.cpu().numpy())
