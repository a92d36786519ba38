"""Long-ranged exchange on even periodic lattices in the cluster-resident
sweep, against the ELL kernel called colour by colour: sites with more than 128
neighbours, and stencil rows that do not fit in shared memory and are read from
global memory (those variants take one site per thread and read their own CTA's
spins through the cluster's window too)."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from helpers import energy_scale
from test_resident_long_stencils import fcc_ham

pytestmark = pytest.mark.gpu


# 134 neighbours; 6^3 cells are 864 sites with a row each
@pytest.mark.parametrize("L,shells,R,mode", [(6, 7, 3, 0), (8, 7, 2, 1)])
def test_more_than_128_neighbours_follow_the_ell_kernel(L, shells, R, mode):
    tems = np.geomspace(5.0, 60.0, R)
    h = fcc_ham(L, shells, tems)
    v = np.random.default_rng(5).normal(size=(R, h.n, 3))
    s0 = v / np.linalg.norm(v, axis=2, keepdims=True)
    out = []
    for resident in (True, False):
        with Engine(h.n, h.num_atoms, h.supercell, R) as e:
            e.upload(h)
            e.set_temperatures(tems)
            assert e.sweep_kernel()[0] == "cluster"
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
