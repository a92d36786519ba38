"""The structure factor's two block shapes (many q-points: 64 q x 16 replicas
a block, few: 8 x 8) give the same bits: a mesh that fills the GPU against
pieces of it, with replicas and sites that fill no block or tile."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian, site_positions
from helpers import NN, sc_mcin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,R", [(3, 1), (5, 17)])
def test_block_shapes_agree(L, R):
    inp = sc_mcin(L, [(1e-3, NN)], list(np.geomspace(4.0, 40.0, R)))
    h = build_hamiltonian(inp, check=False)
    rng = np.random.default_rng(L)
    q = 2 * np.pi * rng.uniform(-1.0, 1.0, size=(64 * 152 + 5, 3))
    pos = site_positions(inp)

    def run(qs):
        with Engine(h.n, h.num_atoms, h.supercell, R) as e:
            e.upload(h)
            e.set_temperatures(inp.tems)
            e.set_structure_factor(qs, [0.0, 0.0, 1.0], 3, inp.real_lattice, pos)
            e.init_spins("rand", seed=2)
            e.begin(e.schedule(2, 100, 1, seed=5))
            e.advance(7)
            r = e.collect()
        assert r["sfactor_count"] == 2
        return r["sfactor"]

    whole = run(q)
    for lo, hi in ((0, 1), (1, 10), (9000, 9150), (9725, len(q))):
        assert np.array_equal(whole[:, lo:hi], run(q[lo:hi]))
