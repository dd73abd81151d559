"""What the framework is timed on: the calls that its users' programs make.

A case is a plain dict; `kind` says which of the programs below it stands for.

  step     a host program that keeps the reference's MCS loop: one Metropolis call with its
           acceptance, the total energy and the configuration of every replica, per pass
  mcs      a temperature scan or parallel-tempering run through Sweep.mcs: the whole loop body
           (overrelaxation, sweep, swaps, measurement) for a number of MCS, then the
           accumulators, acceptance counts and slots; with `records` the driver hands every
           replica's ion record over before the loop and takes it back after it
  series   Sweep.record_series, the autocorrelation measurement: plain sweeps with |M| of every
           replica recorded every `stride` sweeps, then energies and magnetisations
  sq       the structure factor of every replica on a grid of wave vectors
  batch    a mixed batch of chains, every member's MCS loop through Batch.mcs
  learned  plain and learned patch sweeps in turn, |M| recorded
  train    Adam steps of the learned proposal's network on collected patches
"""
import ctypes
import functools
import math

import numpy as np
import torch

import ether_gb300 as eg
from ether_gb300 import abi

MEV = 1e-3
KTC = {"ising": 4.511, "xyz": 1.443}   # k_B T_c / J of the simple-cubic lattice
MODEL = {"ising": 0, "xyz": 1}         # ETHER_MODEL_*
SITE = {"ising": 1, "xyz": 16}         # bytes of a spin on the device
BATCH_SIZES = (8, 12, 16, 24, 32, 48)


def listed():
    return [
        # one lattice at one temperature, driven from the host call by call: the smallest use
        {"name": "ising_step_8", "kind": "step", "model": "ising", "l1": 8, "l2": 8, "l3": 8, "replicas": 1},
        # the 16^3 Ising deck: 19 temperatures x 10 REPEATs, records in and out
        {"name": "ising_deck_16", "kind": "mcs", "model": "ising", "lattice": "sc", "l1": 16, "l2": 16, "l3": 16,
         "bc": "ccc", "slots": 19, "groups": 10, "steps": 2000, "ovrr": 0, "pt": 0, "field": 0.0, "aniso": 0.0,
         "angle": False, "records": True},
        # the headline: plain sweeps of 64^3 Ising at T_c, 1024 replicas, the series for tau
        {"name": "ising_series_64", "kind": "series", "model": "ising", "l1": 64, "l2": 64, "l3": 64,
         "replicas": 1024, "sweeps": 100, "stride": 10},
        # an uneven lattice with an open axis and a field: no closed-form neighbours, PT
        {"name": "ising_open_ragged", "kind": "mcs", "model": "ising", "lattice": "sc", "l1": 21, "l2": 18, "l3": 15,
         "bc": "cco", "slots": 16, "groups": 4, "steps": 220, "ovrr": 0, "pt": 11, "field": 1.0, "aniso": 0.0,
         "angle": False, "records": True},
        # the 32^3 Heisenberg deck: 29 temperatures x 10 REPEATs, overrelaxation every 5 MCS
        {"name": "heis_deck_32", "kind": "mcs", "model": "xyz", "lattice": "sc", "l1": 32, "l2": 32, "l3": 32,
         "bc": "ccc", "slots": 29, "groups": 10, "steps": 100, "ovrr": 5, "pt": 0, "field": 0.0, "aniso": 0.0,
         "angle": False, "records": False},
        # plain sweeps of 64^3 Heisenberg at T_c
        {"name": "heis_series_64", "kind": "series", "model": "xyz", "l1": 64, "l2": 64, "l3": 64,
         "replicas": 64, "sweeps": 50, "stride": 10},
        # the frustrated pyrochlore: J1 / J2, local easy axes, a field, 64 temperatures, PT
        {"name": "pyro_pt_12", "kind": "mcs", "model": "xyz", "lattice": "pyro", "l1": 12, "l2": 12, "l3": 12,
         "bc": "ccc", "slots": 64, "groups": 1, "steps": 220, "ovrr": 0, "pt": 11, "field": 1.0, "aniso": -0.2,
         "angle": False, "records": True},
        # its structure factor on a 64^3 grid
        {"name": "pyro_sq_12", "kind": "sq", "model": "xyz", "cells": 12, "replicas": 64, "q1": 64, "q2": 64, "q3": 64},
        # a batch of unlike chains, half Ising and half Heisenberg, each on its own ladder
        {"name": "batch_32", "kind": "batch", "chains": 32, "ladder": 32, "steps": 20, "mix": 7},
        # the learned 4^3-patch proposal interleaved 1:1 with plain sweeps at T_c
        {"name": "learned_ising_64", "kind": "learned", "model": "ising", "l1": 64, "l2": 64, "l3": 64,
         "replicas": 256, "steps": 10, "stride": 10},
        {"name": "learned_heis_64", "kind": "learned", "model": "xyz", "l1": 64, "l2": 64, "l3": 64,
         "replicas": 64, "steps": 10, "stride": 10},
        # its training: forward, backward and Adam on minibatches of collected patches
        {"name": "train_heis", "kind": "train", "model": "xyz", "l1": 16, "l2": 16, "l3": 16, "replicas": 32,
         "batch": 1024, "steps": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "mcs", "mcs", "mcs", "mcs", "series", "series", "sq", "batch", "learned", "train"])
    model = rng.choice(["ising", "xyz"])
    if kind == "step":
        return {"kind": kind, "model": model, "l1": rng.randint(4, 24), "l2": rng.randint(4, 24),
                "l3": rng.randint(4, 24), "replicas": rng.randint(1, 4)}
    if kind == "mcs":
        lattice = rng.choice(["sc", "sc", "pyro"])
        even = rng.random() < 0.6
        if lattice == "pyro":
            ls = [rng.randint(3, 10) for _ in range(3)]
            sites = 16 * ls[0] * ls[1] * ls[2]
        else:
            ls = [2 * _log_int(rng, 4, 20) if even else _log_int(rng, 7, 40) for _ in range(3)]
            sites = ls[0] * ls[1] * ls[2]
        slots = rng.randint(2, 40)
        most = (1.5e6 if model == "xyz" else 3e6) / (sites * slots)
        groups = max(1, min(rng.randint(1, 12), int(most)))
        slots = max(2, min(slots, int((1.5e6 if model == "xyz" else 3e6) / (sites * groups))))
        return {"kind": kind, "model": model, "lattice": lattice, "l1": ls[0], "l2": ls[1], "l3": ls[2],
                "bc": rng.choice(["ccc", "ccc", "cco", "oco"]) if lattice == "sc" else "ccc",
                "slots": slots, "groups": groups, "steps": rng.choice([60, 110, 220]),
                "ovrr": rng.choice([0, 5, 7]), "pt": rng.choice([0, 11]),
                "field": rng.choice([0.0, 0.0, 1.0]), "aniso": rng.choice([0.0, 0.0, -0.2]) if model == "xyz" else 0.0,
                "angle": model == "xyz" and rng.random() < 0.25, "records": rng.random() < 0.5}
    if kind == "series":
        ls = [2 * _log_int(rng, 6, 36) for _ in range(3)]
        sites = ls[0] * ls[1] * ls[2]
        most = max(1, int((2.0e8 if model == "ising" else 1.6e7) / sites))
        return {"kind": kind, "model": model, "l1": ls[0], "l2": ls[1], "l3": ls[2],
                "replicas": min(most, _log_int(rng, 8, 1024)), "sweeps": rng.choice([20, 50, 100]),
                "stride": rng.choice([1, 5, 10])}
    if kind == "sq":
        return {"kind": kind, "model": model, "cells": rng.randint(2, 11), "replicas": rng.randint(1, 60),
                "q1": 64, "q2": rng.randint(3, 64), "q3": rng.randint(3, 64)}
    if kind == "batch":
        return {"kind": kind, "chains": rng.randint(6, 30), "ladder": rng.randint(4, 32),
                "steps": rng.choice([10, 20]), "mix": rng.randint(0, 10 ** 6)}
    if kind == "learned":
        ls = [8 * rng.randint(1, 8) for _ in range(3)]
        sites = ls[0] * ls[1] * ls[2]
        most = max(1, int((6e7 if model == "ising" else 1.5e7) / sites))
        return {"kind": kind, "model": model, "l1": ls[0], "l2": ls[1], "l3": ls[2],
                "replicas": min(most, _log_int(rng, 4, 256)), "steps": rng.choice([4, 10]), "stride": 2}
    return {"kind": "train", "model": model, "l1": 16, "l2": 8, "l3": 24, "replicas": rng.randint(8, 32),
            "batch": rng.choice([256, 500, 1024]), "steps": rng.randint(8, 16)}


# ------------------------------------------------------------------- what a program holds --
@functools.lru_cache(maxsize=None)
def _lattice(lattice, l1, l2, l3, bc):
    if lattice == "pyro":
        return eg.pyrochlore((l1, l2, l3), shells=(2.97243, 5.1484), tol=1e-3)
    return eg.simple_cubic((l1, l2, l3), bc=bc)


@functools.lru_cache(maxsize=None)
def _axes(l1, l2, l3):
    return eg.local_111_axes(_lattice("pyro", l1, l2, l3, "ccc"))


def _spins(n, sites, model, seed):
    """n configurations: (n, sites, 3) unit vectors or +-1 along z, as the records hold them."""
    rng = np.random.default_rng(seed)
    out = np.zeros((n, sites, 3))
    if model == "ising":
        out[:, :, 2] = rng.integers(0, 2, (n, sites)) * 2.0 - 1.0
    else:
        v = rng.standard_normal((n, sites, 3), dtype=np.float32)
        v /= np.linalg.norm(v, axis=2, keepdims=True)
        out[:] = v
    return out


def _sweep(lat, model, replicas, seed, couplings=((-1.0, -1.0, -1.0),), **kw):
    j = eg.couplings(1, [[(1, 1, c)] for c in couplings], [1.0])
    return eg.Sweep.from_lattice(lat, j, np.array([1.0]), MODEL[model], replicas=replicas, seed=seed % (1 << 31), **kw)


def _one_start(sw, lat, model, seed):
    ion = lat.ion.copy()
    ion[:, 1:4] = _spins(1, lat.N, model, seed)[0]
    sw.set_spins(ion)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_step(c, seed):
    lat = _lattice("sc", c["l1"], c["l2"], c["l3"], "ccc")
    sw = _sweep(lat, c["model"], c["replicas"], seed)
    sw.set_beta(1.0 / (KTC[c["model"]] * MEV))
    _one_start(sw, lat, c["model"], seed)
    ions = np.repeat(lat.ion[None], c["replicas"], axis=0)
    return {"run": _run_step, "sw": sw, "ions": ions}


def _run_step(s):
    sw = s["sw"]
    accept = sw.metropolis(1)
    energy = sw.tot_energy()
    sw.get_spins_batch(s["ions"])
    return {"accept": accept, "energy": energy, "spins": s["ions"][:, :, 1:4]}


def _prepare_mcs(c, seed):
    lat = _lattice(c["lattice"], c["l1"], c["l2"], c["l3"], c["bc"])
    R = c["slots"] * c["groups"]
    kw = {}
    if c["field"]:
        kw.update(zeeman=True, h=(0.0, 0.0, c["field"]), g_factor=2.0)
    if c["angle"]:
        kw.update(angle=True, dphi=0.6)
    if c["lattice"] == "pyro":
        if c["model"] == "ising":
            j = ((-1.0,) * 3, (-0.1,) * 3)
        else:
            j = ((1.0,) * 3, (-0.1,) * 3)
            if c["aniso"]:
                axes = _axes(c["l1"], c["l2"], c["l3"])
                kw["sia_local"] = np.concatenate([axes, np.full((lat.N, 1), c["aniso"] * MEV)], axis=1)
        beta = 1.0 / (eg.KB_EV * np.geomspace(1.0, 50.0, c["slots"]))
    else:
        j = ((-1.0,) * 3,)
        if c["aniso"]:
            kw.update(sia=True, sia_vec=np.array([[0.0, 0.0, c["aniso"] * MEV]]))
        top = 100.0 if c["model"] == "ising" else 150.0
        beta = 1.0 / (eg.KB_EV * np.linspace(top, 10.0, c["slots"]))
    sw = _sweep(lat, c["model"], R, seed, j, **kw)
    sw.set_ladder(beta)
    s = {"run": _run_mcs, "sw": sw, "step": 0, "swap": 0, "case": c, "ions": None}
    if c["records"]:
        ions = np.empty((R, lat.N, 9))
        ions[:] = lat.ion
        ions[:, :, 1:4] = _spins(R, lat.N, c["model"], seed)
        s["ions"] = ions
        sw.set_spins_batch(ions)
    else:
        _one_start(sw, lat, c["model"], seed)
    sw.zero_avg()
    return s


def _run_mcs(s):
    c, sw = s["case"], s["sw"]
    if s["ions"] is not None:
        sw.set_spins_batch(s["ions"])
    s["swap"] = sw.mcs(s["step"], c["steps"], 0, 10, ovrr=c["ovrr"] > 0, ovrr_para=1.0, ovrr_mcs=c["ovrr"],
                       pt=c["pt"] > 0, exchange_interval=c["pt"], swap_count=s["swap"])
    s["step"] += c["steps"]
    out = {"sums": sw.sums(), "slots": sw.slots(), "accepted": sw.slot_accept_counts().astype(np.int64),
           "energy": sw.tot_energy(), "magnetisation": sw.tot_magnetisation()}
    if s["ions"] is not None:
        sw.get_spins_batch(s["ions"])
        out["spins"] = s["ions"][:, :, 1:4]
    return out


def _prepare_series(c, seed):
    lat = _lattice("sc", c["l1"], c["l2"], c["l3"], "ccc")
    sw = _sweep(lat, c["model"], c["replicas"], seed)
    sw.set_beta(1.0 / (KTC[c["model"]] * MEV))
    _one_start(sw, lat, c["model"], seed)
    sw.autotune()
    sw.metropolis(100, accept=False)
    return {"run": _run_series, "sw": sw, "case": c}


def _run_series(s):
    c, sw = s["case"], s["sw"]
    m = sw.record_series(c["sweeps"], stride=c["stride"])
    return {"absm": m, "energy": sw.tot_energy(), "magnetisation": sw.tot_magnetisation(),
            "accepted": sw.accept_counts().astype(np.int64)}


def _grid(c):
    q0 = np.array([-1.0, -1.0, -1.0])
    dq = np.array([2.0 / c["q1"], 2.0 / c["q2"], 2.0 / c["q3"]])
    return q0, dq


def _prepare_sq(c, seed):
    lat = _lattice("pyro", c["cells"], c["cells"], c["cells"], "ccc")
    R = c["replicas"]
    sw = _sweep(lat, c["model"], R, seed, ((1.0,) * 3, (-0.1,) * 3))
    ions = np.zeros((R, lat.N, 9))
    ions[:, :, 1:4] = _spins(R, lat.N, c["model"], seed)
    sw.set_spins_batch(ions)
    Q = c["q1"] * c["q2"] * c["q3"]
    q0, dq = _grid(c)
    return {"run": _run_sq, "sw": sw, "abc": np.ascontiguousarray(lat.abc).ravel(),
            "nq": np.array([c["q1"], c["q2"], c["q3"]], dtype=np.int32), "q0": q0, "dq": dq,
            "sq": np.zeros((R, Q), np.float32), "comp": np.zeros((R, Q, 3), np.float32)}


def _run_sq(s):
    pf = ctypes.POINTER(ctypes.c_float)
    abi.check(s["sw"].lib.ether_structure_factor(
        s["sw"].h, abi.dptr(s["abc"]), abi.iptr(s["nq"]), abi.dptr(s["q0"]), abi.dptr(s["dq"]),
        s["sq"].ctypes.data_as(pf), s["comp"].ctypes.data_as(pf)))
    return {"sq": s["sq"], "comp": s["comp"]}


def _members(c):
    """(model, L, J sign) of every chain."""
    rng = np.random.default_rng(c["mix"])
    return [("ising" if k < c["chains"] // 2 else "xyz", int(rng.choice(BATCH_SIZES)), float(rng.choice([-1, 1])))
            for k in range(c["chains"])]


def _prepare_batch(c, seed):
    members = []
    for k, (model, L, sign) in enumerate(_members(c)):
        lat = _lattice("sc", L, L, L, "ccc")
        sw = _sweep(lat, model, c["ladder"], seed + 101 * k, ((sign,) * 3,))
        sw.set_ladder(1.0 / (KTC[model] * MEV * np.geomspace(0.6, 1.6, c["ladder"])))
        _one_start(sw, lat, model, seed + k)
        members.append(sw)
    return {"run": _run_batch, "batch": eg.Batch(members), "members": members, "step": 0,
            "swap": np.zeros(len(members), np.int32), "case": c}


def _run_batch(s):
    c = s["case"]
    s["swap"] = s["batch"].mcs(s["step"], c["steps"], 0, 10, ovrr=True, ovrr_para=1.0, ovrr_mcs=5, pt=True,
                               exchange_interval=5, swap_counts=s["swap"])
    s["step"] += c["steps"]
    m = s["members"]
    return {"sums": np.concatenate([x.sums() for x in m]), "slots": np.concatenate([x.slots() for x in m]),
            "accepted": np.concatenate([x.accept_counts() for x in m]).astype(np.int64), "swaps": s["swap"],
            "energy": np.concatenate([x.tot_energy() for x in m])}


def _learner(c, seed, capacity):
    lat = _lattice("sc", c["l1"], c["l2"], c["l3"], "ccc")
    sw = _sweep(lat, c["model"], c["replicas"], seed)
    sw.set_beta(1.0 / (KTC[c["model"]] * MEV * np.linspace(0.9, 1.1, c["replicas"])))
    _one_start(sw, lat, c["model"], seed)
    sw.metropolis(50, accept=False)
    return sw, eg.Learned(sw, seed=seed % 1000, capacity=capacity)


def _prepare_learned(c, seed):
    sw, lr = _learner(c, seed, 1024)
    return {"run": _run_learned, "sw": sw, "lr": lr, "case": c}


def _run_learned(s):
    c, sw, lr = s["case"], s["sw"], s["lr"]
    m = lr.record_series(c["steps"], 1, 1, stride=c["stride"])
    return {"absm": m, "patches": lr.accepts().astype(np.int64), "energy": sw.tot_energy(),
            "magnetisation": sw.tot_magnetisation(), "accepted": sw.accept_counts().astype(np.int64)}


def _prepare_train(c, seed):
    sw, lr = _learner(c, seed, 8192)
    for _ in range(4):
        sw.metropolis(5, accept=False)
        lr.collect(64)
    return {"run": _run_train, "sw": sw, "lr": lr, "case": c}


def _run_train(s):
    c, lr = s["case"], s["lr"]
    loss = lr.train(c["steps"], batch=c["batch"], lr=1e-3)
    return {"loss": loss, "params": lr.params()}


# -------------------------------------------------------------- what a pass has to do --
def _state_bytes(sites, model, sweeps):
    """A state that no cache holds is read and written once a sweep, a smaller one once a pass."""
    state = sites * SITE[model]
    return 2.0 * state * (sweeps if state > 100e6 else 1)


#: arithmetic of one site update: six neighbours, the random draw, the decision
OPS = {"ising": 20.0, "xyz": 120.0}


def work(c):
    kind = c["kind"]
    if kind == "sq":
        n, q = 16 * c["cells"] ** 3, c["q1"] * c["q2"] * c["q3"]
        comp = 1 if c["model"] == "ising" else 3
        return {"bytes": 16.0 * q * c["replicas"] + SITE[c["model"]] * n * c["replicas"],
                "flops": 4.0 * q * n * comp * c["replicas"]}
    if kind == "batch":
        b = f = 0.0
        for model, L, _ in _members(c):
            sites = float(L ** 3) * c["ladder"]
            b += _state_bytes(sites, model, c["steps"])
            f += OPS[model] * sites * c["steps"]
        return {"bytes": b, "flops": f}
    if kind == "train":
        n_in, n_out = (128, 32) if c["model"] == "ising" else (304, 96)
        p = n_in * 128 + 128 * 128 + 128 * n_out
        return {"bytes": 4.0 * c["steps"] * (c["batch"] * (n_in + n_out) + 6 * p), "flops": 6.0 * c["steps"] * c["batch"] * p}
    cell = 16 if c.get("lattice") == "pyro" else 1
    replicas = c["replicas"] if "replicas" in c else c["slots"] * c["groups"]
    sites = float(cell * c["l1"] * c["l2"] * c["l3"]) * replicas
    if kind == "step":
        return {"bytes": _state_bytes(sites, c["model"], 1) + 32.0 * sites, "flops": OPS[c["model"]] * sites}
    sweeps = c["sweeps"] if kind == "series" else c["steps"]
    b = _state_bytes(sites, c["model"], sweeps)
    f = OPS[c["model"]] * sites * sweeps
    if c.get("records"):
        b += 2 * (8.0 if c["model"] == "ising" else 32.0) * sites
    if kind == "learned":   # plus the network on every patch of 64 sites
        p = 128 * 128 + 128 * 128 + 128 * 32 if c["model"] == "ising" else 304 * 128 + 128 * 128 + 128 * 96
        b, f = 2 * b, f + 2.0 * p * sites / 64 * c["steps"]
    return {"bytes": b, "flops": f}


def exact(c, seed):
    """The structure factor in 64 bits.  The other kinds are chaotic or random chains and the
    training of a network: their outputs have no value that another arithmetic reproduces."""
    if c["kind"] != "sq":
        return None
    lat = _lattice("pyro", c["cells"], c["cells"], c["cells"], "ccc")
    R, N = c["replicas"], lat.N
    dev = torch.device("cuda")
    spins = _spins(R, N, c["model"], seed).astype(np.float32).astype(np.float64)
    comps = [2] if c["model"] == "ising" else [0, 1, 2]
    B = torch.from_numpy(np.ascontiguousarray(spins[:, :, comps].transpose(1, 0, 2).reshape(N, -1))).to(dev)
    frac = torch.from_numpy(lat.ion[:, 6:9] @ np.linalg.inv(np.asarray(lat.abc).T).T).to(dev)
    q0, dq = _grid(c)
    e = [torch.polar(torch.ones((), dtype=torch.float64, device=dev), 2 * math.pi * (
        torch.from_numpy(q0[a] + dq[a] * np.arange(c["q%d" % (a + 1)])).to(dev)[:, None] * frac[None, :, a]))
        for a in range(3)]
    sq = torch.empty(R, c["q3"], c["q2"], c["q1"], dtype=torch.float64, device=dev)
    comp = torch.zeros(R, c["q3"], c["q2"], c["q1"], 3, dtype=torch.float64, device=dev)
    per = max(1, int(4e8 / (N * c["q1"])))
    for h3 in range(c["q3"]):
        for h2 in range(0, c["q2"], per):
            ph = (e[1][h2:h2 + per] * e[2][h3])[:, None, :] * e[0][None]
            rows = ph.reshape(-1, N)
            s2 = (torch.mm(rows.real, B) ** 2 + torch.mm(rows.imag, B) ** 2).reshape(ph.shape[0], c["q1"], R, len(comps))
            s2 = s2.permute(2, 0, 1, 3)
            sq[:, h3, h2:h2 + per] = s2.sum(-1) / N ** 2
            comp[:, h3, h2:h2 + per, :, comps] = s2.sqrt() / N
    return {"sq": sq.reshape(R, -1), "comp": comp.reshape(R, -1, 3)}
