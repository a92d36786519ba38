"""The cluster-resident sweep on lattices without parity classes (odd
supercells, open boundaries, one-cell layers), which run it in the ELL
kernel's place, against the ELL kernel called colour by colour
(esp_sweep_colour): the same trajectory bit for bit, and the measurements of a
run equal to those made on the host from the ELL engine's state."""
import numpy as np
import pytest

from espins_gb300.lib import Batch, Engine
from espins_gb300.tables import build_hamiltonian
from espins_gb300.workloads import BCC, BCC1, lattice_mcin
from espins_gb300.mcin import parse_mcin
from helpers import NN, NNN, energy_scale, sc_mcin

pytestmark = pytest.mark.gpu


def _ham(L, kind, open_):
    if kind == "bcc":
        inp = parse_mcin(lattice_mcin(BCC, 4, [(2e-3, BCC1), (5e-4, NN)], tems=[10.0], single_ion=-5e-5), "bcc")
    else:
        inp = sc_mcin(4, [(1e-3, NN)] if kind == "j1" else [(1e-3, NN), (3e-4, NNN)], [5.0],
                      **({"dm": 1e-4, "bq": 5e-5} if kind == "dm" else {}))
    inp.supercell_size = list(L)
    inp.boundary_open = open_
    return build_hamiltonian(inp, check=False)


def _engine(h, tems, open_):
    e = Engine(h.n, h.num_atoms, h.supercell, len(tems), open_)
    e.upload(h)
    e.set_temperatures(tems)
    assert e.sweep_kernel()[0] == "ell"
    return e


def _colour_sweep(e, sweep, seed, mode=0):
    for c in range(e.colouring()[1]):
        e.sweep_colour(c, sweep, seed=seed, mode=mode, tilt=0.3)


# one warp and less, one site per thread, several rounds, several CTAs (19,683
# sites and more do not fit one), rows of edge sites, two atoms a cell
@pytest.mark.parametrize("L,kind,open_,R,mode", [
    ((3, 3, 3), "j1", True, 3, 0), ((5, 4, 7), "dm", True, 5, 1), ((9, 11, 1), "j1", True, 4, 0),
    ((7, 6, 5), "j12", False, 2, 0), ((13, 12, 11), "dm", True, 3, 0), ((27, 27, 27), "j1", True, 2, 0),
    ((25, 17, 23), "bcc", False, 2, 0), ((35, 34, 33), "j12", True, 1, 1)])
def test_sweeps_follow_the_ell_kernel(L, kind, open_, R, mode):
    h = _ham(L, kind, open_)
    tems = np.geomspace(4.0, 60.0, R)
    v = np.random.default_rng(3).normal(size=(R, h.n, 3))
    s0 = v / np.linalg.norm(v, axis=2, keepdims=True)
    out = []
    for resident in (True, False):
        with _engine(h, tems, open_) as e:
            e.set_spins(s0)
            if resident:
                n0 = e.launch_count()
                e.sweep(6, 2, seed=11, mode=mode, tilt=0.3)
                one_launch = e.launch_count() - n0 <= 2   # one launch of all sweeps (and a transpose)
            else:
                for k in range(6):
                    _colour_sweep(e, 2 + k, 11, mode)
            out.append((e.get_spins(), e.rejected(), e.running_energy(), e.energy()))
    assert one_launch
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    # FP64 against float-pair sums of the same FP32 terms
    assert np.max(np.abs(out[0][2] - out[1][2])) <= 1e-12 * energy_scale(h)
    assert np.array_equal(out[0][3], out[1][3])


@pytest.mark.parametrize("L,kind", [((5, 3, 5), "bcc"), ((9, 7, 1), "j1")])
def test_measurements_of_a_run_match_the_ell_state(L, kind):
    h = _ham(L, kind, True)
    R, units, na, n = 3, 12, h.num_atoms, h.n
    tems = np.array([6.0, 20.0, 50.0])
    axes = np.array([[0.0, 0.6, 0.8], [1.0, 0.0, 0.0]])[:na]
    coeff = np.array([1, -1])[:na]
    with _engine(h, tems, True) as e, _engine(h, tems, True) as f:
        for x in (e, f):
            x.init_spins("rand", seed=4)
        e.set_observables(order_axes=axes, staggered_coeff=coeff)
        e.set_series(units)
        e.begin(e.schedule(0, units, 2, seed=9, binning_level=[1, 2]))
        e.advance(units)
        res, ser = e.collect(), e.series()
        f.energy()
        data, obs = np.zeros((R, 6)), np.zeros((R, 6))
        for k in range(units):
            for s in (2 * k, 2 * k + 1):
                _colour_sweep(f, s, 9)
            en, m = f.running_energy(), f.running_magnetization() / n
            am = np.linalg.norm(m, axis=1)
            sp = f.get_spins().reshape(R, n // na, na, 3)
            op = np.abs((sp * axes).sum(axis=(1, 2, 3)) / n)
            sm = np.linalg.norm((sp * coeff[:, None]).sum(axis=(1, 2)) / n, axis=1)
            data += np.stack([en, en ** 2, en ** 4, am, am ** 2, am ** 4], axis=1) / units
            obs += np.stack([op, op ** 2, op ** 4, sm, sm ** 2, sm ** 4], axis=1) / units
            assert np.allclose(ser[k, :, 0], en, rtol=1e-12, atol=1e-9)
        assert np.array_equal(e.get_spins(), f.get_spins())
    assert np.allclose(res["data"], data, rtol=1e-11)
    # FP32 products of the order parameter: 2^-24 of terms of size one
    assert np.allclose(res["obs_data"], obs, rtol=1e-5, atol=1e-7)
    # every cell is counted once per measurement (density 100 per hit and unit of m)
    for p in (res["pm"], res["pm_op"], res["pm_sm"]):
        assert np.allclose(p.sum(axis=1), 100.0, rtol=1e-12)


def test_graph_replays_of_a_general_lattice_equal_advances():
    h = _ham((9, 8, 7), "dm", True)
    out = []
    for graph in (False, True):
        with _engine(h, np.geomspace(4.0, 40.0, 6), True) as e:
            e.init_spins("rand", seed=2)
            e.begin(e.schedule(4, 100, 1, pt=True, pt_steps_swap=3, seed=8, binning_level=[1, 2]))
            if graph:
                with Batch([e]) as b:
                    b.set_units_per_graph(2)
                    b.advance(5)
            else:
                e.advance(5)
            r = e.collect()
            out.append((e.get_spins(), r))
    assert np.array_equal(out[0][0], out[1][0])
    for k in ("rejected", "data", "binning", "num_swaps", "map", "energy", "pm"):
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
