"""Dissociations in states that no binding leaves but a caller may set, against
the oracle (float64): complexes whose partner is alive, several complexes with
one partner (dormant or alive), and complexes whose partner is a complex itself.
They dissociate in particle order, each by the state the earlier ones left; two
that share a partner and dissociate in one step must move it between buckets
once each, or the next sort writes past a bucket."""
import numpy as np
import pytest

from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from tests.harness import Pair, cell_sets_oracle, compare_state

F64_TOL = 1e-12  # µm


def _system(box: float, counts: dict) -> dict:
    d = W.membrane_pip3_pten(counts=counts, pools={"PI3K": 40, "PTEN_T1": 40}, box=box, pixels=8,
                             pixel_size_nm=box * 125.0, seed=43, k_cat_scale=0.0)
    d["species"].append({"name": "Sensor", "diffusion_coefficient": 0.08, "radius": 3.0})
    d["species"].append({"name": "Complex", "diffusion_coefficient": 0.06, "radius": 3.5})
    d["initial_populations"]["Sensor"] = 700
    d["reactions"] = [{"name": "bind", "reactants": ["Sensor", "PIP3"], "products": ["Complex"], "kon": 1.0e5,
                       "koff": 3000.0, "contact_radius": 30.0}]
    for ex in d["compartment_exchanges"]:  # recruitment reads the lipid's density grid
        ex["k_on"] *= 200.0
    return d


def _bind(o, sid, name: str) -> None:
    a, b = np.flatnonzero(o.species == sid["Sensor"]), np.flatnonzero(o.species == sid["PIP3"])
    n = 600
    o.species[a[:n]] = sid["Complex"]
    if name == "awake":  # every partner alive
        o.bond[a[:n]] = b[:n]
    elif name == "dormant":  # three complexes to a dormant partner, which names the middle one
        o.bond[a[:n]] = np.repeat(b[:n // 3], 3)
        o.bond[b[:n // 3]] = a[1:n:3]
        o.alive[b[:n // 3]] = False
    elif name == "crowd":  # fifty complexes to an alive partner, beside plain complexes
        o.bond[a[:300]] = np.repeat(b[:6], 50)
        o.bond[a[300:n]] = b[300:n]
        o.bond[b[300:n]] = a[300:n]
        o.alive[b[300:n]] = False
    else:  # chain: each complex bound to the one before it, pairs of complexes, one to itself
        o.bond[a[1:300]] = a[:299]
        o.bond[a[0]] = a[0]
        o.bond[a[300:n]] = a[300:n].reshape(-1, 2)[:, ::-1].ravel()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["awake", "dormant", "crowd", "chain"])
@pytest.mark.parametrize("box", [4.0, 2.0])
def test_odd_bonds_dissociate_in_order(name, box):
    P = Pair(_system(box, {"PIP2": 20, "PIP3": 900, "PI3K": 6, "PTEN_T1": 8, "PTEN_T2": 4}), precision=64,
             photons=False)
    sid = {s.name: k for k, s in enumerate(P.cfg.species)}
    _bind(P.orc, sid, name)
    P.load_oracle_state_into_gpu()
    for t in range(25):
        P.eng.dynamics_step(1)
        P.orc.dynamics_step()
        P.orc.step_index += 1
        compare_state(P.gpu_state(), P.orc, F64_TOL)
    start, mem = P.eng.cells(0)
    nx, ny = P.dp.nx, P.dp.ny
    got = [sorted(mem[start[c]:start[c + 1]].tolist()) for c in range(nx * ny)]
    assert got == cell_sets_oracle(P.orc, nx, ny)
    assert np.array_equal(P.eng.counters()[0][:6], P.orc.counters[:6])
    assert P.orc.counters[1] > 100, P.orc.counters[:6]
    assert P.eng.status() == 0


@pytest.mark.gpu
def test_odd_bonds_in_one_replica_leave_the_others_alone():
    """Three replicas, the middle one with shared partners: each equals itself alone."""
    from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble
    raw = _system(4.0, {"PIP2": 20, "PIP3": 900, "PI3K": 6, "PTEN_T1": 8, "PTEN_T2": 4})
    ens = Ensemble([raw] * 3, precision=32, photons=False)
    one = [Ensemble([raw], precision=32, photons=False) for _ in range(3)]
    sid = {s["name"]: k for k, s in enumerate(raw["species"])}
    P = Pair(raw, precision=64, photons=False)
    states = []
    for k in range(3):
        st = P.state
        s = dict(positions=st.positions.copy(), species=st.species_id.copy(), alive=st.is_alive.copy(),
                 bond=st.bond_partner.copy())
        if k == 1:
            class O:
                species, alive, bond = s["species"], s["alive"], s["bond"]
            _bind(O, sid, "dormant")
        states.append(s)
        one[k].engine.set_state(s["positions"], s["species"], s["alive"], s["bond"], st.has_dye, st.dye_type_id,
                                st.ctmc_state, st.is_bleached)
    st = P.state
    cat = {k: np.concatenate([s[k] for s in states]) for k in states[0]}
    ens.engine.set_state(cat["positions"], cat["species"], cat["alive"], cat["bond"], np.tile(st.has_dye, 3),
                         np.tile(st.dye_type_id, 3), np.tile(st.ctmc_state, 3), np.tile(st.is_bleached, 3))
    ens.engine.dynamics_step(20)
    g = ens.engine.get_state()
    for k in range(3):
        one[k].engine.dynamics_step(20)
        h = one[k].engine.get_state()
        for key in ("positions", "species", "alive", "bond"):
            assert np.array_equal(g[key][ens.replica_slice(k)], h[key]), (k, key)
