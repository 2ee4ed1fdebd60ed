"""edm_get_state at the size up to which a state comes down in one block, and just
above: the same arrays by either way, into pageable arrays, pinned ones and a mix of
both, for particle counts that leave the block's fields unaligned."""
import numpy as np
import pytest
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests.harness import Pair


def _arrays(eng, pinned) -> dict:
    out = {}
    for k, dt, w in eng.STATE_FIELDS:
        a = np.zeros((eng.N, w) if w > 1 else eng.N, dtype=dt)
        out[k] = torch.from_numpy(a).pin_memory().numpy() if k in pinned else a
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [37, 16381, 16384, 16385])
def test_every_way_down_gives_the_same(precision, n):
    pools = {"PI3K": min(30, n // 8), "PTEN_T1": min(30, n // 8)}
    free = n - sum(pools.values())
    counts = {"PIP2": free - 4 * (free // 6), "PIP3": free // 6, "PI3K": free // 6, "PTEN_T1": free // 6,
              "PTEN_T2": free // 6}
    P = Pair(W.membrane_pip3_pten(counts=counts, pools=pools, box=9.0, pixels=8, pixel_size_nm=1125.0, seed=3),
             precision=precision)
    assert P.eng.N == n
    s = torch.cuda.Stream()
    P.eng.pipeline_steps(5, True, 0, stream=s)
    fields = [k for k, _, _ in P.eng.STATE_FIELDS]
    late = P.eng.get_state_async(_arrays(P.eng, fields), stream=s)
    P.eng.transfers_wait()
    for pinned in ([], fields, fields[:1], fields[1:], fields[::2]):
        got = P.eng.get_state(stream=s, out=_arrays(P.eng, pinned))
        for k in fields:
            assert np.array_equal(got[k], late[k]), (pinned, k)
    assert set(np.unique(late["alive"])) == {0, 1}
    assert (np.bincount(late["species"])[:5] > 0).all() and late["has_dye"].sum() == counts["PIP3"]
