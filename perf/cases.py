"""The work a user has this framework do, as measurable cases.

Every case is a job on one GPU through the public classes of
``espins_gb300.lib`` (``Engine``, ``Batch``): Monte Carlo jobs (the measurement
phase of a run, then what it hands back: the accumulators and the spins), the
direct energies of given spins, and training steps of the learned proposal.
Sizes and Hamiltonians are those of the reference's example inputs and of the
benchmark configurations, and the lattices around them.

A case is a dict of plain values; ``kind`` is one of
  run     one lattice: ``units`` measurement units (a unit is a measurement, or
          a whole swap interval with parallel tempering), collect, read spins
  batch   lattices of several sizes in one handle each, advanced together
  energy  set spins from host memory, direct energies and magnetisations
  train   optimiser steps of the learned proposal's network
"""
from __future__ import annotations

import functools
import math

import numpy as np

from espins_gb300.lib import Batch, Engine
from espins_gb300.mcin import parse_mcin
from espins_gb300.tables import build_hamiltonian, build_shells, sfactor_qpoints, site_positions

SC = (((1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0)), ((0.0, 0.0, 0.0),))
BCC = (SC[0], ((0.0, 0.0, 0.0), (0.5, 0.5, 0.5)))
# four sites on the corners of a tetrahedron in the primitive fcc cell
PYRO = (((5.16, 0.0, 5.16), (0.0, 5.16, 5.16), (5.16, 5.16, 0.0)),
        ((0.0, 0.0, 0.0), (0.0, 0.0, 0.5), (0.0, 0.5, 0.0), (0.5, 0.0, 0.0)))
# two honeycomb layers
HONEY = (((4.97, 0.0, 0.0), (-2.485, 4.3041463, 0.0), (0.0, 0.0, 13.16)),
         ((2 / 3, 1 / 3, 0.0), (2 / 3, 1 / 3, 0.375), (1 / 3, 2 / 3, 0.0), (1 / 3, 2 / 3, 0.375)))

# Hamiltonians: exchange per distance shell, nearest-neighbour biquadratic and
# DM (along the bond), single-ion along z, all in eV
HAMS = {
    "sc_j1": dict(lattice=SC, J=(3e-3,)),
    "sc_j12_afm": dict(lattice=SC, J=(-4e-3, -1.04e-3)),
    "sc_j12_frustrated": dict(lattice=SC, J=(1e-3, -6e-4), bq=5e-5, si=2e-4),
    "sc_j12_dm": dict(lattice=SC, J=(1e-3, 3e-4), dm=1e-4, si=-3e-5),
    "sc_bq_dm": dict(lattice=SC, J=(1e-3,), bq=1e-4, dm=2e-4),
    "bcc_j123": dict(lattice=BCC, J=(2e-3, 5e-4, -1e-4), si=-5e-5),
    "pyro_bq_dm": dict(lattice=PYRO, J=(-2e-3,), bq=1e-4, dm=2e-4),
    "honey_j6": dict(lattice=HONEY, J=(-1.4e-3, -4e-4, -3e-4, 5e-5, -2.5e-4, -1e-4)),
}


def _shells(cell, atoms, n):
    """Per shell of the n shortest distances: (atom a, atom b, cell offset) of every neighbour."""
    A = np.array(cell)
    off = np.array([(x, y, z) for x in range(-2, 3) for y in range(-2, 3) for z in range(-2, 3)], dtype=float)
    rows = []
    for a, pa in enumerate(atoms):
        for b, pb in enumerate(atoms):
            d = np.linalg.norm((off + np.array(pb) - np.array(pa)) @ A, axis=1)
            rows += [(round(float(dd), 3), a, b, tuple(map(float, o))) for dd, o in zip(d, off) if dd > 1e-6]
    dist = sorted({r[0] for r in rows})[:n]
    return [[r[1:] for r in rows if r[0] == d] for d in dist]


def _mcin_text(ham, lx, ly, lz, open_boundary, shells_wanted, mesh):
    h = HAMS[ham]
    cell, atoms = h["lattice"]
    out = ["begin unit_cell_cart"] + [" ".join(map(repr, v)) for v in cell] + ["end unit_cell_cart"]
    out += ["begin atoms_frac"] + ["Fe %r %r %r 1.0" % p for p in atoms] + ["end atoms_frac"]
    out += ["supercell_size = %d %d %d" % (lx, ly, lz), "tems_mode = man", "tems_num = 1", "tems = 10.0",
            "steps_warmup = 10", "steps_mc = 1000", "steps_measure = 1"]
    if open_boundary:
        out.append("boundary = open")
    if shells_wanted:
        out.append("spin_correlation = .true.")
    if mesh:
        out += ["sfactor = .true.", "sfactor_2dqmesh = %d %d" % (mesh, mesh)]
    shells = _shells(cell, atoms, len(h["J"]))

    def pair(a, b, o):
        return "f1=%r,%r,%r:f2=%r,%r,%r" % (*atoms[a], *(p + q for p, q in zip(atoms[b], o)))

    out.append("begin jij_parameters")
    for s, (J, rows) in enumerate(zip(h["J"], shells)):
        out += [pair(*r) + ":jij=%r" % J + (":sh=%d" % (s + 1) if shells_wanted else "") for r in rows]
    out.append("end jij_parameters")
    if "bq" in h:
        out += ["ham_bij = .true.", "begin bij_parameters"]
        out += [pair(*r) + ":bij=%r" % h["bq"] for r in shells[0]] + ["end bij_parameters"]
    if "dm" in h:
        A = np.array(cell)
        out += ["ham_dij = .true.", "begin dij_parameters"]
        out += [pair(*r) + ":dij=%r" % h["dm"] for r in shells[0]] + ["end dij_parameters", "begin dij_vectors_cart"]
        for a, b, o in shells[0]:
            v = (np.array(o) + np.array(atoms[b]) - np.array(atoms[a])) @ A
            out.append("%r %r %r" % tuple(float(x) for x in v / np.linalg.norm(v)))
        out.append("end dij_vectors_cart")
    if "si" in h:
        out += ["ham_singleion = .true.", "begin singleion_axes_cart"]
        out += ["Fe 0 0 1 %r" % h["si"] for _ in atoms] + ["end singleion_axes_cart"]
    return "\n".join(out) + "\n"


@functools.lru_cache(maxsize=12)
def _lattice(ham, lx, ly, lz, open_boundary=False, shells_wanted=False, mesh=0):
    """The parsed input, its tables and (where wanted) its neighbour shells: made once for a lattice."""
    inp = parse_mcin(_mcin_text(ham, lx, ly, lz, open_boundary, shells_wanted, mesh), ham)
    return inp, build_hamiltonian(inp, check=False), build_shells(inp) if shells_wanted else None


def _run(name, ham, L, replicas, t0, t1, units, **more):
    lx, ly, lz = (L, L, L) if isinstance(L, int) else L
    return {"name": name, "kind": "run", "ham": ham, "lx": lx, "ly": ly, "lz": lz, "replicas": replicas,
            "t0": t0, "t1": t1, "units": units, "measure": 1, "pt": False, "swap": 1, "cone": False, "open": False,
            "binning": False, "series": False, "order": False, "corr": False, "mesh": 0, "every": 10,
            "learned": "", **more}


def listed():
    return [
        # the smallest example: 64 spins, independent temperatures; latency alone
        _run("sc4_plain", "sc_j1", 4, 20, 25.0, 75.0, 2000, measure=2),
        # 14^3 antiferromagnet, parallel tempering, cone moves, energy series
        _run("sc14_cone_pt", "sc_j12_afm", 14, 32, 36.0, 39.875, 10, measure=5, pt=True, swap=10, cone=True,
             series=True),
        # four atoms a cell with biquadratic and DM terms, order parameter, binning
        _run("pyro4_order", "pyro_bq_dm", 4, 28, 10.0, 40.0, 600, measure=2, order=True, binning=True),
        # a two-dimensional lattice (one cell along z), long-ranged exchange, spin correlations
        _run("honey24_corr", "honey_j6", (24, 24, 1), 64, 4.0, 70.0, 50, measure=5, corr=True),
        # an odd film with open boundaries, structure factor on a mesh of q-points
        _run("film21_open", "sc_j1", (21, 21, 7), 24, 5.0, 60.0, 100, open=True, mesh=12),
        # the reference-sized parallel-tempering benchmark
        _run("bcc24_pt", "bcc_j123", 24, 48, 10.0, 80.0, 60, pt=True, swap=10),
        # several CTAs to a replica, frustrated
        _run("sc48_frustrated", "sc_j12_frustrated", 48, 32, 2.0, 30.0, 30, pt=True, swap=10),
        # many lattices of several sizes together, replica exchange within each
        {"name": "batch_mixed", "kind": "batch", "l0": 8, "l1": 48, "step": 8, "lattices": 8, "replicas": 16,
         "units": 24, "graph": 4},
        # larger than a cluster's shared memory
        _run("slab96_dm", "sc_j12_dm", (96, 96, 48), 64, 5.0, 40.0, 20, pt=True, swap=10),
        # the learned proposal's sweep
        _run("learned_sc32", "sc_j12_frustrated", 32, 32, 2.0, 30.0, 20, pt=True, swap=10, learned="tcgen05"),
        # the learned proposal's training steps
        {"name": "train_4096", "kind": "train", "l": 16, "replicas": 32, "batch": 4096, "steps": 40,
         "engine": "tcgen05"},
        # energies of configurations a program holds in host memory
        {"name": "energy_bcc24", "kind": "energy", "ham": "bcc_j123", "lx": 24, "ly": 24, "lz": 24, "replicas": 48},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    """One more case: the kinds of the listed ones over their ranges of sizes, odd ones among them."""
    kind = rng.choice(["small", "pt", "large", "open", "layer", "batch", "learned", "train", "energy"])
    if kind == "batch":
        l0 = 2 * rng.randint(2, 8)
        step = 2 * rng.randint(1, 6)
        l1 = l0 + step * rng.randint(1, min(4, (48 - l0) // step))
        return {"kind": "batch", "l0": l0, "l1": l1, "step": step, "lattices": rng.randint(1, 9),
                "replicas": rng.randint(4, 16), "units": rng.randint(4, 12), "graph": rng.choice([1, 2, 4])}
    if kind == "train":
        return {"kind": "train", "l": 2 * rng.randint(4, 10), "replicas": rng.randint(8, 40),
                "batch": _log(rng, 500, 12000), "steps": rng.randint(5, 30), "engine": rng.choice(["mma", "tcgen05"])}
    if kind == "energy":
        ham = rng.choice(sorted(HAMS))
        most = 28 if len(HAMS[ham]["lattice"][1]) == 1 else 18
        return {"kind": "energy", "ham": ham, "lx": rng.randint(5, most), "ly": rng.randint(5, most),
                "lz": rng.randint(5, most), "replicas": _log(rng, 1, 60)}
    t0 = rng.uniform(2.0, 12.0)
    if kind == "learned":
        c = _run("", rng.choice(["sc_j12_frustrated", "bcc_j123"]), 2 * rng.randint(4, 12), rng.randint(6, 40), t0,
                 t0 + rng.uniform(10.0, 60.0), 10, pt=rng.random() < 0.5, learned=rng.choice(["mma", "tcgen05"]))
    elif kind == "small":
        c = _run("", rng.choice(["sc_j1", "sc_j12_afm", "pyro_bq_dm", "bcc_j123", "sc_bq_dm"]), 2 * rng.randint(2, 9),
                 rng.randint(5, 40), t0, t0 + rng.uniform(20.0, 60.0), 100, measure=rng.randint(1, 3),
                 cone=rng.random() < 0.3, binning=rng.random() < 0.5, order=rng.random() < 0.3,
                 corr=rng.random() < 0.2)
    elif kind == "pt":
        c = _run("", rng.choice(["sc_j1", "sc_j12_frustrated", "sc_j12_dm", "bcc_j123"]), 2 * rng.randint(9, 22),
                 rng.randint(8, 48), t0, t0 + rng.uniform(20.0, 60.0), 30, pt=True, swap=rng.choice([5, 10, 20]),
                 cone=rng.random() < 0.3)
    elif kind == "large":
        c = _run("", rng.choice(["sc_j1", "sc_j12_dm"]), rng.choice([66, 72, 75, 80, 88]), rng.choice([8, 12, 16, 24]),
                 t0, t0 + rng.uniform(20.0, 60.0), 10, pt=True, swap=5)
    elif kind == "open":
        L = tuple(rng.randint(5, 30) for _ in range(3))
        c = _run("", rng.choice(["sc_j1", "sc_j12_dm", "bcc_j123"]), L, rng.randint(5, 40), t0,
                 t0 + rng.uniform(20.0, 60.0), 60, open=rng.random() < 0.7, mesh=rng.choice([0, 0, 8, 15]),
                 corr=rng.random() < 0.2, binning=rng.random() < 0.3)
    else:
        c = _run("", rng.choice(["honey_j6", "sc_j12_frustrated"]), (rng.randint(8, 40), rng.randint(8, 40), 1),
                 rng.randint(8, 64), t0, t0 + rng.uniform(20.0, 60.0), 60, measure=rng.randint(1, 5),
                 corr=rng.random() < 0.5, order=rng.random() < 0.3, pt=rng.random() < 0.3, swap=4)
        if c["ham"] == "sc_j12_frustrated":
            c["open"] = True   # one layer has no periodic neighbours along z
    del c["name"]
    # about as many updates as the listed ones of its kind make
    sweeps = c["measure"] * (c["swap"] if c["pt"] else 1)
    per_unit = _sites(c) * c["replicas"] * sweeps
    most = {"open": 1.5e8, "layer": 1.0e8, "learned": 1.0e8, "small": 4e8, "pt": 8e8, "large": 1e9}[kind]
    c["units"] = max(1, min(int(most / per_unit), 400 // sweeps))
    return c


def _sites(case):
    return len(HAMS[case["ham"]]["lattice"][1]) * case["lx"] * case["ly"] * case["lz"]


def _tems(case):
    return np.geomspace(case["t0"], case["t1"], case["replicas"])


def _prepare_run(case, seed):
    inp, ham, shells = _lattice(case["ham"], case["lx"], case["ly"], case["lz"], case["open"], case["corr"],
                                case["mesh"])
    e = Engine(ham.n, ham.num_atoms, ham.supercell, case["replicas"], case["open"])
    e.upload(ham)
    e.set_temperatures(_tems(case))
    if case["order"]:
        ax = np.array([(1.0, 1.0, 1.0), (-1.0, -1.0, 1.0), (1.0, -1.0, -1.0), (-1.0, 1.0, -1.0)]) / math.sqrt(3.0)
        e.set_observables(order_axes=ax[np.arange(ham.num_atoms) % 4],
                          staggered_coeff=[1 if a % 2 == 0 else -1 for a in range(ham.num_atoms)])
    if case["corr"]:
        e.set_spin_correlation(shells)
    if case["mesh"]:
        e.set_structure_factor(sfactor_qpoints(inp), inp.sfactor_polar, case["every"], inp.real_lattice,
                               site_positions(inp))
    if case["learned"]:
        e.lp_init(seed)
        e.lp_set_engine(case["learned"])
        e.set_proposal("learned")
    e.init_spins("rand", seed)
    per_unit = case["swap"] if case["pt"] else 1
    if case["series"]:
        e.set_series(case["units"] * per_unit)
    e.begin(e.schedule(20, 1000000, case["measure"], pt=case["pt"], pt_steps_swap=case["swap"],
                       mode=1 if case["cone"] else 0, tilt=0.25, seed=seed,
                       binning_level=[1, 2, 3, 4, 5] if case["binning"] else None))
    return {"case": case, "engines": [e]}


def _prepare_batch(case, seed):
    engines = []
    for k, L in enumerate(range(case["l0"], case["l1"] + 1, case["step"])):
        _, ham, _ = _lattice("sc_bq_dm", L, L, L)
        n = max(1, case["lattices"] >> k)   # fewer of the large ones
        e = Engine(ham.n, ham.num_atoms, ham.supercell, n * case["replicas"])
        e.upload(ham)
        e.set_temperatures(np.tile(np.geomspace(2.0, 25.0, case["replicas"]), n))
        e.set_pt_groups(case["replicas"])
        e.init_spins("rand", seed + k)
        e.begin(e.schedule(20, 1000000, 1, pt=True, pt_steps_swap=10, seed=seed + k))
        engines.append(e)
    b = Batch(engines)
    b.set_units_per_graph(case["graph"])
    return {"case": case, "engines": engines, "batch": b}


def _prepare_train(case, seed):
    _, ham, _ = _lattice("sc_j12_frustrated", case["l"], case["l"], case["l"])
    e = Engine(ham.n, ham.num_atoms, ham.supercell, case["replicas"])
    e.upload(ham)
    e.set_temperatures(np.geomspace(2.0, 30.0, case["replicas"]))
    e.init_spins("rand", seed)
    e.sweep(20, 0, seed=seed)
    e.lp_set_engine(case["engine"])
    e.lp_init(seed)
    e.lp_reserve(ham.n * case["replicas"])
    for c in range(e.colouring()[1]):
        e.lp_collect(c)
    return {"case": case, "engines": [e], "seed": seed}


def _random_spins(case, seed):
    v = np.random.default_rng(seed).normal(size=(case["replicas"], _sites(case), 3))
    return v / np.linalg.norm(v, axis=2, keepdims=True)


def _prepare_energy(case, seed):
    _, ham, _ = _lattice(case["ham"], case["lx"], case["ly"], case["lz"])
    e = Engine(ham.n, ham.num_atoms, ham.supercell, case["replicas"])
    e.upload(ham)
    e.set_temperatures(np.geomspace(5.0, 50.0, case["replicas"]))
    return {"case": case, "engines": [e], "spins": _random_spins(case, seed)}


def prepare(case, seed):
    return {"run": _prepare_run, "batch": _prepare_batch, "train": _prepare_train,
            "energy": _prepare_energy}[case["kind"]](case, seed)


def run(state):
    case, e = state["case"], state["engines"][0]
    if case["kind"] == "run":
        e.advance(case["units"])
        out = e.collect()
        out["spins"] = e.get_spins()
        if case["series"]:
            out["series"] = e.series()
        return out
    if case["kind"] == "batch":
        state["batch"].advance(case["units"])
        out = []
        for e in state["engines"]:
            r = e.collect()
            out.append({"data": r["data"], "energy": r["energy"], "rejected": r["rejected"], "map": r["map"],
                        "spins": e.get_spins()})
        return out
    if case["kind"] == "train":
        loss = e.lp_train(case["steps"], batch=case["batch"], lr=1e-3, seed=state["seed"])
        return {"loss": loss, "weights": e.lp_weights()}
    e.set_spins(state["spins"])
    return {"energy": e.energy(), "magnetization": e.running_magnetization()}


def _terms(ham):
    """(exchange + biquadratic + DM neighbours per site, flops per update of their fields)"""
    h = HAMS[ham]
    s = _shells(*h["lattice"], len(h["J"]))
    na = len(h["lattice"][1])
    nn, n1 = sum(map(len, s)) / na, len(s[0]) / na
    return nn, 6 * nn + (15 if "bq" in h else 0) * n1 + (12 if "dm" in h else 0) * n1


def work(case):
    if case["kind"] == "train":
        mlp = 12 * 128 + 128 * 128 + 128 * 20
        # forward, input gradients and weight gradients of every row; rows read, parameters read and written
        return {"bytes": case["steps"] * (case["batch"] * 48 + 3 * 8 * 20756),
                "flops": case["steps"] * case["batch"] * 6.0 * mlp}
    if case["kind"] == "energy":
        n = _sites(case) * case["replicas"]
        nn, _ = _terms(case["ham"])
        return {"bytes": 24 * n, "flops": n * (3.5 * nn + 6)}
    if case["kind"] == "batch":
        n = sum(max(1, case["lattices"] >> k) * L ** 3 for k, L in
                enumerate(range(case["l0"], case["l1"] + 1, case["step"]))) * case["replicas"]
        return {"bytes": 36 * n, "flops": 10.0 * case["units"] * n * (_terms("sc_bq_dm")[1] + 60)}
    n = _sites(case) * case["replicas"]
    meas = case["units"] * (case["swap"] if case["pt"] else 1)
    nn, field = _terms(case["ham"])
    flops = meas * case["measure"] * n * (field + 60 + (2 * (12 * 128 + 128 * 128 + 128 * 20) if case["learned"] else 0))
    if case["corr"]:
        flops += meas * n * nn * 8
    if case["mesh"]:
        flops += (meas // case["every"]) * n * (case["mesh"] + 1) ** 2 * 12
    return {"bytes": 36 * n, "flops": float(flops)}   # the FP32 state read, the FP64 spins written


def exact(case, seed):
    """Energies and magnetisations of given spins in 64 bits.  A Monte Carlo job and a training run have no such
    value: one decision or rounding taken otherwise leads to another, equally valid, trajectory."""
    if case["kind"] != "energy":
        return None
    h = HAMS[case["ham"]]
    cell, atoms = h["lattice"]
    lx, ly, lz, na, R = case["lx"], case["ly"], case["lz"], len(atoms), case["replicas"]
    s = _random_spins(case, seed).reshape(R, lz, ly, lx, na, 3)
    k_b = 8.6173303e-5   # eV per kelvin, CODATA 2014
    A = np.array(cell)
    e = np.zeros(R)
    shells = _shells(cell, atoms, len(h["J"]))
    for k, rows in enumerate(shells):
        for a, b, o in rows:
            si = s[..., a, :]
            sj = np.roll(s[..., b, :], tuple(-int(x) for x in o[::-1]), axis=(1, 2, 3))
            d = np.einsum("rzyxc,rzyxc->rzyx", si, sj)
            e -= 0.5 * h["J"][k] / k_b * d.sum(axis=(1, 2, 3))
            if k == 0 and "bq" in h:
                e += 0.5 * h["bq"] / k_b * (d * d).sum(axis=(1, 2, 3))
            if k == 0 and "dm" in h:
                v = (np.array(o) + np.array(atoms[b]) - np.array(atoms[a])) @ A
                e += 0.5 * h["dm"] / k_b * (np.cross(si, sj).sum(axis=(1, 2, 3)) @ (v / np.linalg.norm(v)))
    if "si" in h:
        e += h["si"] / k_b * (s[..., 2] ** 2).sum(axis=(1, 2, 3, 4))
    return {"energy": e, "magnetization": s.sum(axis=(1, 2, 3, 4))}
