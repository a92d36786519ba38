"""Learned-proposal sweeps over block edges: fewer trials than threads, ragged
last trials spread over the blocks, more replicas than a block has threads,
neighbour lists with and without a biquadratic coupling in a part of eight
(first shell only, of one and two shells).  The running energy, summed from the
trials' changes, must be that of the spins; both engines' sweeps are
reproducible."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, NNN, energy_scale, sc_mcin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["mma", "tcgen05"])
@pytest.mark.parametrize("L,R,shells,bq", [(4, 3, 1, 5e-5), (10, 7, 2, 5e-5), (18, 37, 2, None), (16, 150, 2, 5e-5)])
def test_learned_sweeps_over_block_edges(L, R, shells, bq, engine):
    sh = [(1e-3, NN), (-4e-4, NNN)][:shells]
    inp = sc_mcin(L, sh, list(np.linspace(3.0, 40.0, R)), bq=bq, si=1e-4)
    h = build_hamiltonian(inp)
    rng = np.random.default_rng(8)
    s0 = rng.normal(size=(R, h.n, 3))
    s0 /= np.linalg.norm(s0, axis=2, keepdims=True)
    out = []
    for _ in range(2):
        with Engine(h.n, h.num_atoms, h.supercell, R) as e:
            e.upload(h)
            e.set_temperatures(inp.tems)
            e.lp_init(3)
            e.lp_set_engine(engine)
            e.set_proposal("learned")
            e.set_spins(s0)
            e.sweep(6, 1, seed=17)
            s = e.get_spins()
            assert np.max(np.abs(e.running_energy() - e.energy())) <= 1e-5 * energy_scale(h)
            assert np.allclose(np.linalg.norm(s, axis=2), 1.0, atol=2e-6)
            assert np.all(np.sum(e.rejected(), axis=1) < 6 * h.n)
            out.append(s)
    assert np.array_equal(out[0], out[1])
