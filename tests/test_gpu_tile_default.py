"""The tiled sweep's default geometry: of the replica groups and variants of
the model's tile edge it takes two CTAs per SM, with the largest group that
gives every SM an item, and follows the trajectory of the one-tile-per-CTA
kernel whatever it takes."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, NNN, sc_mcin

pytestmark = pytest.mark.gpu


# groups of 16, 8 and 4 replicas as the replica count allows; one replica
# leaves the one-tile-per-CTA kernel alone
@pytest.mark.parametrize("L,R", [(16, 32), (48, 16), (48, 8), (24, 12), (24, 1)])
def test_default_geometry_keeps_the_trajectory(L, R):
    inp = sc_mcin(L, [(1e-3, NN), (3e-4, NNN)], list(np.geomspace(4.0, 50.0, R)), dm=1e-4)
    h = build_hamiltonian(inp, check=False)
    out = []
    for default in (True, False):
        with Engine(h.n, h.num_atoms, h.supercell, R) as e:
            e.upload(h)
            e.set_temperatures(inp.tems)
            e.set_sweep_kernel("tile")
            T, G, variant = e.tile_geometry()
            if default:
                # edges below 4 have the one-tile-per-CTA kernel only
                assert R % G == 0 and (variant == 2 or R % 4 or T < 4)
            else:
                e.set_tile_geometry(T, 1, 0)
            e.init_spins("rand", seed=4)
            e.sweep(5, 1, seed=6)
            out.append((e.get_spins(), e.rejected()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
