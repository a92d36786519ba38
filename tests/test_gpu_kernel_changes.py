"""The state follows the lattice through changes of the kernel that sweeps it:
an even lattice that fits one CTA of the cluster-resident sweep without the
optional measurements' histograms and not with them (86 x 108 x 2 sites; its
edges take no tiles), which then runs that sweep's general form, and back."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, sc_mcin

pytestmark = pytest.mark.gpu

TEMS = [5.0, 20.0]


def _ham():
    inp = sc_mcin(4, [(1e-3, NN)], TEMS)
    inp.supercell_size = [86, 108, 2]
    return build_hamiltonian(inp, check=False)


def _engine(h):
    e = Engine(h.n, h.num_atoms, h.supercell, len(TEMS))
    e.upload(h)
    e.set_temperatures(TEMS)
    e.init_spins("rand", seed=3)
    return e


def _observe(e, on):
    e.set_observables(**({"order_axes": np.array([[0.0, 0.0, 1.0]]), "staggered_coeff": [1]} if on else {}))


def _sweeps(e, first):
    n0 = e.launch_count()
    e.sweep(2, first, seed=9)
    return e.launch_count() - n0


def test_spins_survive_changes_between_the_cluster_and_the_general_form():
    h = _ham()
    with _engine(h) as e, _engine(h) as f:
        assert e.cluster_geometry()[0] == 1
        _sweeps(e, 0)
        _observe(e, True)                            # no cluster geometry is left
        assert e.cluster_geometry()[0] == 0
        assert _sweeps(e, 2) <= 3                    # one resident launch, at most a transpose each way
        _observe(e, False)
        _sweeps(e, 4)
        e.set_cluster_geometry(1, 512, 1)            # possible again
        _sweeps(e, 6)
        for s in range(8):
            for c in range(f.colouring()[1]):
                f.sweep_colour(c, s, seed=9)
        assert np.array_equal(e.get_spins(), f.get_spins())
        assert np.array_equal(e.rejected(), f.rejected())


def test_spins_survive_new_tables_after_the_cluster_was_given_up():
    h = _ham()
    with _engine(h) as e, _engine(h) as f:
        for x in (e, f):
            _sweeps(x, 0)
        _observe(e, True)
        e.upload(h)
        e.set_temperatures(TEMS)
        assert np.array_equal(e.get_spins(), f.get_spins())
