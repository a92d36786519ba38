"""Structure factor of meshes whose phases exceed the table (64 MB: sites x
q-points of 8 bytes): every block makes its own phases, from the same
arithmetic, so a mesh gives the bits that its pieces give from tables, in both
block shapes."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian, site_positions
from helpers import NN, sc_mcin

pytestmark = pytest.mark.gpu


# 13,824 sites x 612 or 643 q-points: 67.7 and 71.1 million bytes; 10 or 11 x 1
# and x 16 blocks of 64 q x 16 replicas (which are taken from 152 blocks on)
@pytest.mark.parametrize("nq,R", [(612, 3), (643, 250)])
def test_phases_made_in_the_kernel_are_those_of_the_table(nq, R):
    L = 24
    inp = sc_mcin(L, [(1e-3, NN)], list(np.geomspace(4.0, 40.0, R)))
    h = build_hamiltonian(inp, check=False)
    q = 2 * np.pi * np.random.default_rng(nq).uniform(-1.0, 1.0, size=(nq, 3))
    pos = site_positions(inp)
    assert h.n * nq * 8 > 64 << 20 and h.n * 300 * 8 < 64 << 20

    def run(qs):
        with Engine(h.n, h.num_atoms, h.supercell, R) as e:
            e.upload(h)
            e.set_temperatures(inp.tems)
            e.set_structure_factor(qs, [0.0, 0.0, 1.0], 2, inp.real_lattice, pos)
            e.init_spins("rand", seed=2)
            e.begin(e.schedule(2, 100, 1, seed=5))
            e.advance(4)
            r = e.collect()
        assert r["sfactor_count"] == 2
        return r["sfactor"]

    whole = run(q)
    for lo, hi in ((0, 300), (300, nq - 1), (nq - 1, nq)):
        if hi - lo <= 300 or h.n * (hi - lo) * 8 <= 64 << 20:
            assert np.array_equal(whole[:, lo:hi], run(q[lo:hi])), (lo, hi)
