"""The work that users of this package have the GPU do, as cases that can be timed.

Five kinds, each through the entry points a program calls:

* drop_in   one Brownian-dynamics step of the reference's own loop, object by
            object: DynamicsEngine.step, PhotonSimulator.evolve_one_bd_step,
            VirtualMicroscope.process_photons (float64, host arrays current
            after every call);
* frame     one FLIM frame of one system: `steps` BD steps with photons and
            detection in a CUDA graph (Engine.pipeline_steps), the frame's
            end (finalize), its stacks read as nonzero bins
            (frame_out_sparse) and the particle state read back (get_state);
* ensemble  the same frame of many jittered replicas in one engine;
* flim      one batched FLIM acquisition: new bound fractions, emitter maps,
            PSF projection, Poisson TCSPC histograms;
* readout   lifetime readouts (mean arrival time, phasor) of TCSPC stacks that
            lie on the device.

`tuned` engines time their launch shapes first, as a long run does; the
others take the shapes an engine starts with.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from flim_microscopy_simulator_with_causal_inference_b200 import api
from flim_microscopy_simulator_with_causal_inference_b200 import flim_acquire as FA
from flim_microscopy_simulator_with_causal_inference_b200 import readouts as RO
from flim_microscopy_simulator_with_causal_inference_b200 import workloads as W
from flim_microscopy_simulator_with_causal_inference_b200.batch import Ensemble
from flim_microscopy_simulator_with_causal_inference_b200.config import config_from_dict
from flim_microscopy_simulator_with_causal_inference_b200.particles import ParticleState

T_RANGE = 25e-9


def listed():
    return [
        # a user of the reference's loop, who reads the state after every object: latency and launches
        dict(name="drop_in_step", kind="drop_in", n=3500, pixels=64),
        # the 10x10 µm² PIP3/PTEN membrane, the package's smallest shipped system, at the default precision
        dict(name="membrane_frame", kind="frame", chem="pip3", n=3500, precision=64, steps=100, pixels=64,
             tuned=False),
        # the dense 13,000-particle membrane with its sine D(x) field, float32
        dict(name="sine_frame", kind="frame", chem="sine", n=13000, precision=32, steps=100, pixels=128,
             tuned=False),
        # a biosensor that binds its lipid reversibly: binding, dissociation, bond FRET, slow-diffusion disc
        dict(name="sensor_frame", kind="frame", chem="sensor", n=9731, precision=64, steps=100, pixels=64,
             tuned=False),
        # the wave script's switches: adaptation field and density-biased recruitment
        dict(name="wave_frame", kind="frame", chem="wave", n=30011, precision=32, steps=100, pixels=64,
             tuned=False),
        # the 100x100 µm² membrane (1.3M particles and 0.56M in the cytosol pools), harmonic repulsion
        dict(name="large_frame", kind="frame", chem="harmonic", n=1300000, precision=32, steps=100, pixels=256,
             tuned=True),
        # a quarter of it in float64 with the shapes an engine starts with
        dict(name="large_frame_f64", kind="frame", chem="harmonic", n=325007, precision=64, steps=100, pixels=256,
             tuned=False),
        # a small parameter scan: few uneven replicas
        dict(name="ensemble_24", kind="ensemble", replicas=24, n_min=1000, n_max=20000, precision=32, steps=100,
             pixels=64, tuned=False),
        # the batched ensemble of the benchmark at half its replicas
        dict(name="ensemble_256", kind="ensemble", replicas=256, n_min=1000, n_max=50000, precision=32, steps=100,
             pixels=64, tuned=True),
        # one field of view
        dict(name="flim_1", kind="flim", replicas=1, emitters=50000, budget=1000.0, n_bins=256),
        # the benchmark's batch of fields of view
        dict(name="flim_256", kind="flim", replicas=256, emitters=50000, budget=1000.0, n_bins=256),
        # lifetime maps of a batch of stacks
        dict(name="readout_stack", kind="readout", px=64 * 65536, n_bins=256, harmonic=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop_in", "frame", "frame", "frame", "ensemble", "ensemble", "flim", "flim", "readout"])
    if kind == "drop_in":
        return dict(kind=kind, n=_log(rng, 700, 14000), pixels=rng.choice([32, 64, 128]))
    if kind == "frame":
        chem = rng.choice(["pip3", "sine", "sensor", "wave", "harmonic"])
        top = {"pip3": 300000, "sine": 100000, "sensor": 20000, "wave": 60000, "harmonic": 1000000}[chem]
        return dict(kind=kind, chem=chem, n=_log(rng, 700, top), precision=rng.choice([32, 64]),
                    steps=rng.choice([20, 50, 100]), pixels=rng.choice([32, 64, 128]), tuned=False)
    if kind == "ensemble":
        return dict(kind=kind, replicas=_log(rng, 3, 200), n_min=1000, n_max=_log(rng, 2000, 50000),
                    precision=rng.choice([32, 32, 64]), steps=rng.choice([20, 50, 100]), pixels=rng.choice([32, 64]),
                    tuned=rng.random() < 0.5)
    if kind == "flim":
        return dict(kind=kind, replicas=_log(rng, 1, 200), emitters=_log(rng, 4000, 60000),
                    budget=round(math.exp(rng.uniform(math.log(50.0), math.log(1500.0))), 1),
                    n_bins=rng.choice([128, 256]))
    return dict(kind=kind, px=_log(rng, 3000, 64 * 65536), n_bins=rng.choice([64, 100, 128, 256]),
                harmonic=rng.choice([1, 2]))


# ---- systems ---------------------------------------------------------------
def _raw(chem, n, pixels, seed, steps=100):
    """A system of n membrane particles as a YAML-equivalent dict."""
    per_um2 = {"pip3": 35.0, "wave": 35.0, "sine": 130.0, "harmonic": 130.0, "sensor": 125.0}[chem]
    box = math.sqrt(n / per_um2)
    d = W.membrane_pip3_pten(counts=W.scaled_counts(n), pools=W.scaled_pools(n), box=box,
                             potential="harmonic" if chem == "harmonic" else "wca", steps_per_frame=steps,
                             pixels=pixels, pixel_size_nm=max(30.0, box * 1000.0 / pixels), sine_d_field=chem == "sine",
                             seed=1 + seed % (2 ** 31 - 2))
    if chem == "wave":
        for fb in d["feedback_rules"]:
            fb["grid_resolution"] = 1.0
        d["_script_attributes"] = {"use_adaptation": True, "adaptation_tau_w": 0.01, "adaptation_K_w": 10.0,
                                   "adaptation_n_w": 2.0, "use_local_pi3k_recruitment": True, "recruit_sigma": 0.5}
    if chem == "sensor":  # a fifth of the membrane is sensor
        d["species"].append({"name": "Sensor", "diffusion_coefficient": 0.08, "radius": 3.0})
        d["species"].append({"name": "Sensor_PIP3", "diffusion_coefficient": 0.06, "radius": 3.5})
        pop = d["initial_populations"]
        pop["Sensor"] = n // 5
        pop["PIP2"] = max(1, pop["PIP2"] - n // 5)
        d["reactions"] = [{"name": "bind", "reactants": ["Sensor", "PIP3"], "products": ["Sensor_PIP3"],
                           "kon": 5.0, "koff": 40.0, "contact_radius": 20.0}]
        d["diffusion_field"] = {"type": "regions", "regions": [
            {"shape": "circle", "center": [box / 2, box / 2], "radius": box / 4, "D_factor": 0.3}]}
        d["dye_attachments"] = [{"species": "Sensor", "fluorophore": "mTFP1", "labeling_efficiency": 0.9},
                                {"species": "PIP3", "fluorophore": "Venus", "labeling_efficiency": 0.5}]
        d["fret_pairs"] = [{"donor_type": "mTFP1", "acceptor_type": "Venus", "R0": 5.4,
                            "intra_complex_distance": 5.0, "fret_mode": "bond", "intramolecular": False}]
    return d


def _pinned(n, dtype):
    return torch.zeros(n, dtype=dtype).pin_memory().numpy()


def _frame_state(raws, precision, steps, tuned):
    ens = Ensemble(raws, precision=precision, photons=True)
    eng = ens.engine
    stream = torch.cuda.Stream()
    if tuned:
        eng.autotune(3, stream=stream)
        ens.upload(stream=stream)  # the tuning stepped the system: back to its initial state
        eng.set_step(0)
    kinds = {np.float64: torch.float64, np.int32: torch.int32, np.uint8: torch.uint8, np.int8: torch.int8}
    out = {k: _pinned((eng.N, w) if w > 1 else (eng.N,), kinds[t]) for k, t, w in eng.STATE_FIELDS}
    cap = min(eng.flim_elems(), 1 << 20)  # nonzero bins of a frame: some hundred thousand at most
    stream.synchronize()
    return dict(ens=ens, eng=eng, stream=stream, steps=steps, frame=0, out=out, idx=_pinned(cap, torch.int64),
                cnt=_pinned(cap, torch.int32).view(np.uint32))


class _Borrowed:
    """A device array of the package for torch (no copy); holds its owner, so the tensor does too."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(acq, what, shape, typestr):
    return torch.as_tensor(_Borrowed(acq, acq.device_ptr(what)[0], shape, typestr), device="cuda")


def _flim_config(case):
    d = FA.flim_config()
    d["tcspc"]["n_bins"] = case["n_bins"]
    return config_from_dict(d)


def _bound(case, seed):
    return np.random.default_rng(seed).random(case["replicas"])


def _decays(case, seed):
    """A stack [px][n_bins] of Poisson counts: mixed 2.8 ns and 1.1 ns decays of 0 to some hundred photons."""
    px, nb = case["px"], case["n_bins"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = (torch.arange(nb, device="cuda", dtype=torch.float32) + 0.5) * (25.0 / nb)
    slow, fast = torch.exp(-t / 2.8), torch.exp(-t / 1.1)
    stack = torch.empty((px, nb), dtype=torch.int32, device="cuda")
    for a in range(0, px, 1 << 18):
        b = min(px, a + (1 << 18))
        amount = 700.0 * torch.rand((b - a, 1), device="cuda", generator=gen) ** 2
        share = torch.rand((b - a, 1), device="cuda", generator=gen)
        mean = amount * (share * slow / slow.sum() + (1.0 - share) * fast / fast.sum())
        stack[a:b] = torch.poisson(mean, generator=gen).to(torch.int32)
    return stack


def prepare(case, seed):
    kind = case["kind"]
    if kind == "drop_in":
        cfg = config_from_dict(_raw("pip3", case["n"], case["pixels"], seed))
        st = ParticleState(cfg)
        duty = min(1.0, cfg.scan.dwell_time / cfg.scan.frame_interval)
        phot = api.PhotonSimulator(cfg, st, scan_duty_fraction=duty)
        return dict(kind=kind, st=st, phot=phot, dyn=api.DynamicsEngine(cfg, st),
                    mic=api.VirtualMicroscope(cfg, st))
    if kind == "frame":
        raws = [_raw(case["chem"], case["n"], case["pixels"], seed, case["steps"])]
        return dict(_frame_state(raws, case["precision"], case["steps"], case["tuned"]), kind=kind)
    if kind == "ensemble":
        # the scan's sizes and rates are the case's, the replicas' positions and draws the seed's
        raws = W.ensemble_replicas(case["replicas"], n_min=case["n_min"], n_max=case["n_max"], pixels=case["pixels"])
        for r, d in enumerate(raws):
            d["random_seed"] = 1 + (seed * 1009 + r) % (2 ** 31 - 2)
        return dict(_frame_state(raws, case["precision"], case["steps"], case["tuned"]), kind=kind)
    if kind == "flim":
        bound = _bound(case, seed)
        acq = FA.FlimAcquisition(_flim_config(case), case["replicas"], n_emitters=case["emitters"],
                                 photon_budget=case["budget"], seed=seed, bound_fraction=bound)
        R, nb, px = case["replicas"], case["n_bins"], FA.NPIX
        view = {"hist": _view(acq, FA.HIST, (R, px, px, nb), "<i4"),
                "intensity": _view(acq, FA.INTENSITY, (R, 2, px, px), "<f4"),
                "counts": _view(acq, FA.COUNTS, (R, 2, px, px), "<i4"),
                "tau": _view(acq, FA.TAU, (R, px, px), "<f8")}
        stream = torch.cuda.Stream()
        return dict(kind=kind, acq=acq, bound=bound, seed=seed, view=view, stream=stream)
    stack = _decays(case, seed)
    out = torch.empty((6, case["px"]), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return dict(kind=kind, stack=stack, out=out, harmonic=case["harmonic"])


def run(state):
    kind = state["kind"]
    if kind == "drop_in":
        st = state["st"]
        state["dyn"].step()
        batch = state["phot"].evolve_one_bd_step()
        detected = state["mic"].process_photons(batch)
        return dict(positions=st.positions, species=st.species_id, alive=st.is_alive, bond=st.bond_partner,
                    ctmc=st.ctmc_state, bleached=st.is_bleached, photons=int(batch.n_photons), detected=detected)
    if kind in ("frame", "ensemble"):
        eng, s = state["eng"], state["stream"]
        eng.pipeline_steps(state["steps"], True, state["steps"], stream=s)
        eng.finalize(state["frame"], stream=s)
        state["frame"] += 1
        n = eng.frame_out_sparse(state["idx"], state["cnt"], stream=s)
        eng.get_state(stream=s, out=state["out"])
        return dict(state["out"], bins=state["idx"], counts=state["cnt"], nonzero=n)
    if kind == "flim":
        acq, s = state["acq"], state["stream"].cuda_stream
        acq.set_inputs(state["bound"], state["seed"], stream=s)
        acq.acquire(stream=s)
        return state["view"]
    return RO.lifetimes_device(state["stack"].data_ptr(), state["stack"].shape[0], state["stack"].shape[1], T_RANGE,
                               harmonic=state["harmonic"], out=state["out"])


def work(case):
    """Bytes and operations of one pass: inputs read once, outputs written once."""
    kind = case["kind"]
    if kind in ("drop_in", "frame"):
        # 64 B per particle and step: position, cell, flags and id read and written, cell list and draws once
        return {"bytes": 64.0 * case["n"] * case.get("steps", 1), "flops": 150.0 * case["n"] * case.get("steps", 1)}
    if kind == "ensemble":
        lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
        mean = (case["n_max"] - case["n_min"]) / (hi - lo) if hi > lo else case["n_min"]
        n = case["replicas"] * mean * case["steps"]
        return {"bytes": 64.0 * n, "flops": 150.0 * n}
    if kind == "flim":
        px = case["replicas"] * 65536.0
        # histogram and expected lifetime out, two intensity maps out, count maps out; the PSF's two 31-tap passes
        # of two maps (float multiply-adds)
        return {"bytes": px * (4.0 * case["n_bins"] + 8.0 + 8.0 + 8.0), "flops": px * 2 * 2 * 31 * 2.0}
    # counts in, six float64 maps out; per bin the intensity, first moment and phasor sums
    return {"bytes": case["px"] * (4.0 * case["n_bins"] + 48.0), "flops": case["px"] * case["n_bins"] * 8.0}


# ---- the same outputs in 64 bits, in plain torch -----------------------------
def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words."""
    mask = 0xFFFFFFFF

    def mul(m, x):
        hi = (m * (x >> 16) + ((m * (x & 0xFFFF)) >> 16)) >> 16
        lo = ((m * (x >> 16) << 16) + m * (x & 0xFFFF)) & mask
        return hi & mask, lo

    k0, k1 = key & mask, key >> 32
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c0)
        h1, l1 = mul(0xCD9E8D57, c2)
        c0, c1, c2, c3 = (h1 ^ c1 ^ k0), l1, (h0 ^ c3 ^ k1), l0
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0, c1, c2, c3


def _exact_counts(case, seed, r, bound):
    """Emitter counts [free, bound][x][y] of replica r: the keyed pixels and states of its emitters."""
    key = (seed ^ ((0x9E3779B97F4A7C15 * (r + 1)) & (2 ** 64 - 1))) & (2 ** 64 - 1)
    e = torch.arange(case["emitters"], device="cuda", dtype=torch.int64)
    zero = torch.zeros_like(e)
    _, u0, _, u1 = _philox(e, zero, zero, zero + (200 << 16), key)
    w0, w1, _, _ = _philox(e, zero, zero, zero + (201 << 16), key)
    part = ((((w1 << 32) | w0) >> 11) & (2 ** 53 - 1)).double() * 2.0 ** -53
    pixel = ((part < bound).long() * 256 + (u0 >> 24)) * 256 + (u1 >> 24)
    return torch.bincount(pixel, minlength=2 * 65536).double().reshape(2, 256, 256)


def _exact_bins(tau, sigma, width, n):
    """Bin probabilities of an exponential decay with a Gaussian instrument response, early times in bin 0."""
    t = torch.arange(n + 1, dtype=torch.float64, device="cuda") * width
    root = math.sqrt(0.5)
    sf = 0.5 * torch.erfc(t / sigma * root) + torch.exp(-t / tau + 0.5 * (sigma / tau) ** 2) * 0.5 * torch.erfc(
        -(t / sigma - sigma / tau) * root)
    sf[0] = 1.0
    return sf[:-1] - sf[1:]


def exact(case, seed):
    kind = case["kind"]
    if kind == "flim":
        # histograms are draws of a generator; the emitter counts are whole numbers
        d = FA.derive_flim(_flim_config(case), case["emitters"], case["budget"])
        i = torch.arange(256, device="cuda", dtype=torch.float64)
        gap = i[:, None] - i[None, :]
        band = torch.exp(-0.5 * (gap / d.sigma_psf_px) ** 2) * (gap.abs() <= d.half_taps)
        band = band / band.sum(0, keepdim=True)
        centre = (torch.arange(case["n_bins"], device="cuda", dtype=torch.float64) + 0.5) * d.bin_width_ns
        hf = _exact_bins(d.tau_free_ns, d.sigma_irf_ns, d.bin_width_ns, case["n_bins"]) * d.yield_free
        hb = _exact_bins(d.tau_bound_ns, d.sigma_irf_ns, d.bin_width_ns, case["n_bins"]) * d.yield_bound
        bound = _bound(case, seed)
        maps, taus = [], []
        for r in range(case["replicas"]):
            m = band @ _exact_counts(case, seed, r, float(bound[r])) @ band.T
            num = m[0] * (hf * centre).sum() + m[1] * (hb * centre).sum()
            den = m[0] * hf.sum() + m[1] * hb.sum()
            maps.append(m)
            taus.append(torch.where(den > 0, num / den, torch.zeros_like(num)))
        return dict(hist=None, intensity=torch.stack(maps), counts=None, tau=torch.stack(taus))
    if kind == "readout":
        stack = _decays(case, seed)
        nb = case["n_bins"]
        k = torch.arange(nb, device="cuda", dtype=torch.float64) + 0.5
        phi = 2.0 * math.pi * case["harmonic"] * k / nb
        weight = torch.stack([torch.ones_like(k), k * (T_RANGE * 1e9 / nb), torch.cos(phi), torch.sin(phi)], 1)
        sums = torch.cat([stack[a:a + (1 << 18)].double() @ weight for a in range(0, case["px"], 1 << 18)])
        n, nt, nc, ns = sums.T
        nan = torch.full_like(n, float("nan"))
        omega = 2.0 * math.pi * case["harmonic"] / (T_RANGE * 1e9)
        mask = n >= 20
        g = torch.where(mask, nc / n, torch.zeros_like(n))
        s = torch.where(mask, ns / n, torch.zeros_like(n))
        valid, m2 = mask & (g > 1e-10), g * g + s * s
        return torch.stack([n, torch.where(n >= 10, nt / n, nan), g, s, torch.where(valid, (s / g) / omega, nan),
                            torch.where(valid & (m2 > 1e-10) & (m2 < 1 - 1e-10), torch.sqrt(1.0 / m2 - 1.0) / omega,
                                        nan)])
    # a trajectory with collisions, thresholded events and keyed draws has no value that more bits converge to
    return None
