"""A lattice of one CTA per replica runs with warps that make trials and fold
measurements, or without them where the replicas fill the SMs: the same
replicas have the same trajectories and measurements either way."""
import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, NNN, sc_mcin

pytestmark = pytest.mark.gpu


# 12 replicas leave every SM one CTA; of 650 an SM has five to run
@pytest.mark.parametrize("L,shells,open_,mode", [(8, [(1e-3, NN), (3e-4, NNN)], False, 0), (6, [(1e-3, NN)], False, 1),
                                                 (7, [(1e-3, NN), (3e-4, NNN)], True, 0)])
def test_replicas_do_not_depend_on_their_number(L, shells, open_, mode):
    few, many = 12, 650
    tems = np.concatenate([np.geomspace(4.0, 60.0, few), np.full(many - few, 20.0)])
    inp = sc_mcin(4, shells, [5.0])
    inp.supercell_size, inp.boundary_open = [L] * 3, open_
    h = build_hamiltonian(inp, check=False)
    v = np.random.default_rng(1).normal(size=(many, h.n, 3))
    s0 = v / np.linalg.norm(v, axis=2, keepdims=True)
    out = []
    for R in (few, many):
        with Engine(h.n, h.num_atoms, h.supercell, R, open_) as e:
            e.upload(h)
            e.set_temperatures(tems[:R])
            e.set_observables(order_axes=np.array([[0.0, 0.6, 0.8]]), staggered_coeff=[-1])
            e.set_spins(s0[:R])
            e.begin(e.schedule(3, 1000, 2, mode=mode, tilt=0.3, seed=6, binning_level=[1, 2]))
            e.advance(9)
            out.append((e.get_spins(), e.collect()))
    (sa, ra), (sb, rb) = out
    assert np.array_equal(sa, sb[:few])
    assert np.array_equal(ra["rejected"], rb["rejected"][:few])
    # sums of the same FP32 terms, in float pairs or more, in another order
    for k in ("data", "obs_data", "binning"):
        assert np.allclose(ra[k], rb[k][:few], rtol=1e-11, atol=1e-13), k
