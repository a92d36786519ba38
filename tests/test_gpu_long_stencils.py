"""Long-ranged exchange on even periodic lattices in the cluster-resident
sweep, against the ELL kernel called colour by colour: sites with more than 128
neighbours, and stencil rows that do not fit in shared memory and are read from
global memory (those variants take one site per thread and read their own CTA's
spins through the cluster's window too)."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from helpers import energy_scale
from test_resident_long_stencils import fcc_ham, lib  # noqa: F401  (a fixture)
from test_resident_tables import _check

pytestmark = pytest.mark.gpu


def _compare(h, tems, mode, geometry=None):
    R = len(tems)
    v = np.random.default_rng(5).normal(size=(R, h.n, 3))
    s0 = v / np.linalg.norm(v, axis=2, keepdims=True)
    out = []
    for resident in (True, False):
        with Engine(h.n, h.num_atoms, h.supercell, R) as e:
            e.upload(h)
            e.set_temperatures(tems)
            assert e.sweep_kernel()[0] == "cluster"
            if geometry:
                e.set_cluster_geometry(*geometry)
            e.set_spins(s0)
            if resident:
                e.sweep(4, 1, seed=7, mode=mode, tilt=0.3)
            else:
                for k in range(4):
                    for c in range(e.colouring()[1]):
                        e.sweep_colour(c, 1 + k, seed=7, mode=mode, tilt=0.3)
            out.append((e.get_spins(), e.rejected(), e.running_energy(), e.energy()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    # FP32 sums of a sweep's energy changes, grouped by thread in both
    assert np.max(np.abs(out[0][2] - out[1][2])) <= 1e-6 * energy_scale(h)
    assert np.array_equal(out[0][3], out[1][3])


# 134 neighbours; 6^3 cells are 864 sites with a row each
@pytest.mark.parametrize("L,shells,R,mode", [(6, 7, 3, 0), (8, 7, 2, 1)])
def test_more_than_128_neighbours_follow_the_ell_kernel(L, shells, R, mode):
    tems = np.geomspace(5.0, 60.0, R)
    _compare(fcc_ham(L, shells, tems), tems, mode)


# one site a thread and two, one CTA and two (peers' spins in the rows), the
# longest list, and biquadratic and DM terms on the nearest neighbours
@pytest.mark.parametrize("L,shells,rich,geometry,mode", [
    (12, 5, False, (1, 512, 1), 0), (12, 5, False, (1, 512, 2), 1), (12, 7, False, (2, 512, 1), 0),
    (16, 2, False, (1, 512, 2), 0), (16, 2, True, (1, 512, 2), 0), (12, 5, True, (1, 256, 1), 1),
    (12, 7, True, (2, 512, 2), 0)])
def test_rows_in_global_memory_follow_the_ell_kernel(lib, L, shells, rich, geometry, mode):
    tems = [5.0, 40.0]
    h = fcc_ham(L, shells, tems, rich)
    rc, (row_words, _, sites) = _check(lib, h, (L,) * 3, geometry[0], False)
    # rows, spins, the histogram of four moments, reduction scratch, header
    assert rc == 0 and 4 * row_words + 12 * sites + 4 * 801 + 8 * (152 + 284) + 576 > 227 * 1024
    _compare(h, tems, mode, geometry)
