"""Detection of a host-set photon batch around graphs that the caller captures.

A batch from the host may name any particle, and the engine rebuilds its map from
particles to slots for it (the sorts keep the slots of dye carriers only).  The
caller's capture runs nothing by itself, and what it recorded runs later on any
batch: neither may leave a batch to a stale map."""
import numpy as np
import pytest
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests.harness import Pair


def _system() -> dict:
    d = W.membrane_pip3_pten(counts={"PIP2": 600, "PIP3": 100, "PI3K": 30, "PTEN_T1": 60, "PTEN_T2": 30},
                             pools={"PI3K": 20, "PTEN_T1": 20}, box=3.2, pixels=16, pixel_size_nm=200.0, seed=41)
    d["laser"]["power"] = 2.0e-3
    return d


def _set_batch(P: Pair) -> None:
    pid = np.flatnonzero(~P.state.has_dye)[:400].astype(np.int32)
    P.eng.set_photons(0, pid, np.linspace(0.0, 2.0e-8, pid.size), np.zeros(pid.size, np.int8),
                      np.zeros(pid.size, np.uint8), batch_key=5)


@pytest.fixture
def pairs():
    """Two equal engines after nine steps and a photon pass; the second's map is complete."""
    P, Q = Pair(_system(), precision=64), Pair(_system(), precision=64)
    for X in (P, Q):
        X.eng.dynamics_step(9)
        X.eng.photon_step()
    torch.cuda.synchronize()
    _set_batch(Q)
    Q.eng.scope_process()
    return P, Q


@pytest.mark.gpu
def test_captured_detection_runs_on_a_host_batch(pairs):
    P, Q = pairs
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        P.eng.scope_process(stream=s)
    _set_batch(P)
    with torch.cuda.stream(s):
        g.replay()
    torch.cuda.synchronize()
    a, b = P.eng.flim(0), Q.eng.flim(0)
    assert b.sum() > 0 and np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["photon_step", "pipeline_steps"])
def test_a_capture_leaves_the_host_batch_as_it_is(pairs, call):
    P, Q = pairs
    _set_batch(P)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):  # recorded, not run
        if call == "photon_step":
            P.eng.photon_step(stream=s)
        else:
            P.eng.pipeline_steps(2, True, 0, stream=s)  # two: the slots' buffers are back where they were
    P.eng.scope_process()
    a, b = P.eng.flim(0), Q.eng.flim(0)
    assert b.sum() > 0 and np.array_equal(a, b)
