"""The one-launch bucket scan (a block per replica) at its edges against the
oracle (float64): the most cells it takes (127 x 127 + 1 buckets, four rounds of
4,096), one more row and column (the tiled scan), a handful of cells, and
replicas whose buckets start at every alignment."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests import cases
from tests.harness import Pair, cell_sets_oracle, compare_state

F64_TOL = 1e-12  # µm


def _system(box: float) -> dict:
    return W.membrane_pip3_pten(counts={"PIP2": 1500, "PIP3": 80, "PI3K": 60, "PTEN_T1": 200, "PTEN_T2": 90},
                                pools={"PI3K": 50, "PTEN_T1": 90}, box=box, pixels=8, pixel_size_nm=box * 125.0,
                                seed=37, k_cat_scale=500.0)


@pytest.mark.gpu
@pytest.mark.parametrize("box,cells", [(20.98, 127), (21.15, 128), (0.9, 5), (2.65, 16)])
def test_scan_gives_the_oracle_cells(box, cells):
    P = Pair(_system(box), precision=64, photons=False)
    assert P.dp.nx == P.dp.ny == cells
    # at 0.9 µm the oracle's bounded pair list is full in the first step, and the
    # two part after it; the first step's cells are still comparable there
    for _ in range(4 if box > 1.0 else 1):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        start, mem = P.eng.cells(0)
        got = [sorted(mem[start[c]:start[c + 1]].tolist()) for c in range(P.dp.nx * P.dp.ny)]
        assert got == cell_sets_oracle(P.orc, P.dp.nx, P.dp.ny)
    if box > 1.0:
        compare_state(P.gpu_state(), P.orc, F64_TOL)


@pytest.mark.gpu
def test_replicas_at_every_alignment_agree_with_themselves_alone():
    from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble
    raws = cases.jittered_ensemble(7, seed=5)
    ens = Ensemble(raws, precision=64, photons=False)
    assert len({p.cell_offset % 4 for p in ens.dyn_params}) == 4
    ens.engine.dynamics_step(12)
    g = ens.engine.get_state()
    for r, raw in enumerate(raws):
        one = Ensemble([raw], precision=64, photons=False)
        one.engine.dynamics_step(12)
        h = one.engine.get_state()
        for k in ("positions", "species", "alive"):
            assert np.array_equal(g[k][ens.replica_slice(r)], h[k]), (r, k)
