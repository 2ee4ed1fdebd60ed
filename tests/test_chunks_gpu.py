"""Pipeline chunks through all their stages (the first without a graph, the second
captured, the rest replays) with several replicas: chained launches and ordinary ones
give the same, whatever the chunk's size and parity."""
import os

import numpy as np
import pytest
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble


def _run(raws, precision: int, chunk: int, chained: bool) -> dict:
    old = os.environ.get("EDM_PDL")
    try:
        os.environ["EDM_PDL"] = "1" if chained else "0"
        ens = Ensemble(raws, precision=precision, photons=True)
    finally:
        if old is None:
            os.environ.pop("EDM_PDL", None)
        else:
            os.environ["EDM_PDL"] = old
    s = torch.cuda.Stream()
    ens.engine.pipeline_steps(100, True, chunk, stream=s)
    s.synchronize()
    out = dict(ens.engine.get_state(stream=s), counters=ens.engine.counters(), status=ens.engine.status())
    out.update({f"stack{r}": ens.engine.flim(r) for r in range(ens.R)})
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
def test_chunks_of_every_stage_agree(precision):
    raws = W.ensemble_replicas(8, seed=5, n_min=600, n_max=2000)
    want = _run(raws, precision, 0, False)  # no graph, no chained launches
    for chunk, chained in ((25, True), (25, False), (20, True), (100, True)):
        got = _run(raws, precision, chunk, chained)
        for key in want:
            assert np.array_equal(want[key], got[key]), (chunk, chained, key)
