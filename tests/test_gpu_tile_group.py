"""Which replica group the tiled sweep takes by default: with two CTAs per SM at
the model's tile edge, the largest group that gives every SM an item (a tile of
one parity and a group of replicas)."""
import pytest

from espins_gb300.lib import Engine, EspError
from espins_gb300.tables import build_hamiltonian
from helpers import NN, NNN, sc_mcin

pytestmark = pytest.mark.gpu


# every group gives every SM an item, and only those below 16 do (150 items)
@pytest.mark.parametrize("L,R", [((96, 96, 48), 32), ((64, 64, 64), 16), ((40, 40, 48), 16), ((72, 72, 72), 4)])
def test_default_group(L, R):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    inp = sc_mcin(4, [(1e-3, NN), (3e-4, NNN)], [10.0], dm=1e-4)
    inp.supercell_size = list(L)
    h = build_hamiltonian(inp, check=False)
    with Engine(h.n, h.num_atoms, h.supercell, R) as e:
        e.upload(h)
        T, G, variant = e.tile_geometry()
        items = {}
        for g in (4, 8, 16):
            try:
                e.set_tile_geometry(T, g, 2)
            except EspError:
                continue
            items[g] = (L[0] // T) * (L[1] // T) * (L[2] // T) // 8 * (R // g)
    enough = [g for g in items if items[g] >= sms]
    assert T >= 4 and variant == 2 and G == max(enough), (T, G, variant, items)
