"""A batch whose handles change between its calls: the recorded graph belongs to
the tables, kernels, measurements and schedules it was recorded with, so it is
recorded again, and the results are those of advancing every handle by itself."""
import numpy as np
import pytest

from espins_gb300.lib import Batch, Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, NNN, sc_mcin

pytestmark = pytest.mark.gpu

TEMS = list(np.geomspace(4.0, 40.0, 4))
AXES = np.array([[0.0, 0.6, 0.8]])


def _engine(L, open_):
    inp = sc_mcin(4, [(1e-3, NN), (3e-4, NNN)], TEMS)
    inp.supercell_size, inp.boundary_open = list(L), open_
    h = build_hamiltonian(inp, check=False)
    e = Engine(h.n, h.num_atoms, h.supercell, len(TEMS), open_)
    e.upload(h)
    e.set_temperatures(TEMS)
    e.init_spins("rand", seed=2)
    return e, h


# (what changes, whether the run begins anew)
CHANGES = {
    "observables": lambda e, h: e.set_observables(order_axes=AXES, staggered_coeff=[-1]),
    "kernel": lambda e, h: e.set_sweep_kernel("ell"),
    "series": lambda e, h: e.set_series(20),
    "tables": lambda e, h: (e.upload(h), e.set_temperatures(TEMS)),
    "nothing": lambda e, h: None,
}


@pytest.mark.parametrize("what", sorted(CHANGES))
@pytest.mark.parametrize("L,open_", [((9, 8, 7), True), ((8, 8, 8), False)])
def test_a_changed_handle_is_recorded_again(L, open_, what):
    out = []
    for batch in (True, False):
        e, h = _engine(L, open_)
        f, _ = _engine((6, 6, 6), False)
        engines = [e, f]
        b = Batch(engines) if batch else None

        def advance(n):
            if b:
                b.advance(n)
            else:
                for x in engines:
                    x.advance(n)

        if b:
            b.set_units_per_graph(2)
        for x in engines:
            x.begin(x.schedule(2, 1000, 2, pt=True, pt_steps_swap=2, seed=8, binning_level=[1]))
        advance(4)
        CHANGES[what](e, h)
        for seed, levels in ((8, [1]), (9, [1, 2, 3])):
            e.begin(e.schedule(2, 1000, 2, pt=True, pt_steps_swap=2, seed=seed, binning_level=levels))
            advance(4)
        out.append([(x.get_spins(), x.collect(), x.rejected()) for x in engines])
        if b:
            b.close()
        for x in engines:
            x.close()
    for (sa, ra, na), (sb, rb, nb) in zip(*out):
        assert np.array_equal(sa, sb)
        assert np.array_equal(na, nb)
        for k in ra:
            if isinstance(ra[k], np.ndarray):
                # (a level with one block has no variance: 0 / 0 in both)
                assert np.array_equal(ra[k], rb[k], equal_nan=True), k
