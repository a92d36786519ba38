"""Running sums of lattices without parity classes: the cluster-resident sweep's
general form against the ELL kernel, which adds the same FP32 terms (the
accepted energy and spin changes, the sites' parts of the order parameter and
staggered magnetisation) in FP64.  A sum of either passes at most 64 roundings
of 2^-53 on its way from the terms (slots and trees of a launch, launches,
measurements), each of no more than the terms' sum."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, NNN, energy_scale, sc_mcin

pytestmark = pytest.mark.gpu

TOL = 64 * 2.0 ** -53


def _engine(h, tems, kind):
    e = Engine(h.n, h.num_atoms, h.supercell, len(tems), True)
    e.upload(h)
    e.set_temperatures(tems)
    e.set_sweep_kernel(kind)
    assert (e.sweep_kernel()[1] > 0) == (kind == "auto")
    return e


# one warp with a warp of its own for the fold, several, one site a thread
# without helpers, two sites a thread, several CTAs
@pytest.mark.parametrize("L,kind,mode", [((3, 3, 3), "j1", 0), ((9, 8, 7), "dm", 1), ((13, 9, 8), "j1", 0),
                                         ((19, 12, 7), "dm", 0), ((27, 27, 27), "j1", 0)])
def test_running_sums_are_those_of_fp64(L, kind, mode):
    inp = sc_mcin(4, [(1e-3, NN), (3e-4, NNN)] if kind == "dm" else [(1e-3, NN)], [5.0],
                  **({"dm": 1e-4, "bq": 5e-5} if kind == "dm" else {}))
    inp.supercell_size, inp.boundary_open = list(L), True
    h = build_hamiltonian(inp, check=False)
    tems = [4.0, 60.0, 5000.0]
    out = []
    for choice in ("auto", "ell"):
        with _engine(h, tems, choice) as e:
            e.init_spins("rand", seed=2)
            e.set_observables(order_axes=np.array([[0.0, 0.6, 0.8]]), staggered_coeff=[-1])
            e.sweep(40, 0, seed=5, mode=mode, tilt=0.3)
            sums = [(e.running_energy(), e.running_magnetization())]
            e.begin(e.schedule(0, 1000, 2, mode=mode, tilt=0.3, seed=6, binning_level=[1, 2]))
            e.advance(7)
            sums.append((e.running_energy(), e.running_magnetization()))
            out.append((e.get_spins(), e.collect(), sums))
    (sa, ra, suma), (sb, rb, sumb) = out
    assert np.array_equal(sa, sb)
    for (ea, ma), (eb, mb) in zip(suma, sumb):
        assert np.max(np.abs(ea - eb)) <= TOL * energy_scale(h)
        assert np.max(np.abs(ma - mb)) <= TOL * h.n
    # |order parameter| and |staggered magnetisation| per site, of terms of at
    # most 1; squares and fourth powers double and quadruple an error
    assert np.max(np.abs(ra["obs_data"] - rb["obs_data"])) <= 4 * TOL


def test_an_infinite_energy_change_stays_infinite():
    """A field of 2e38 K: sites far from it gain more than the largest FP32 number."""
    extra = "ham_field = .true.\nbegin field_axes_cart\nFe 0 0 1 1.0\nend field_axes_cart\n"
    inp = sc_mcin(4, [(1e-12, NN)], [5.0], extra=extra)
    inp.supercell_size, inp.boundary_open = [5, 5, 5], True
    h = build_hamiltonian(inp, check=False)
    h.field_val[:] = 2e38
    s0 = np.zeros((2, h.n, 3))
    s0[0, :, 2], s0[1, :, 2] = 1.0, -1.0
    out = []
    for choice in ("auto", "ell"):
        with _engine(h, [5.0, 5.0], choice) as e:
            e.set_spins(s0)
            e.sweep(1, 0, seed=3)
            out.append((e.get_spins(), e.running_energy()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.isneginf(out[1][1]).any()
    assert np.array_equal(out[0][1], out[1][1])
