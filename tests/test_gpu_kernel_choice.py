"""Which kernel sweeps a lattice without parity classes: the automatic choice may
run the cluster-resident kernel's general form, the choice "ell" runs the ELL
kernel colour by colour; both give the same trajectory, and the cluster size
that is reported beside "ell" tells them apart."""
import numpy as np
import pytest

from espins_gb300.lib import Batch, Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, sc_mcin

pytestmark = pytest.mark.gpu

TEMS = [5.0, 20.0, 60.0]


def _engine():
    inp = sc_mcin(4, [(1e-3, NN)], TEMS)
    inp.supercell_size, inp.boundary_open = [9, 8, 7], True
    h = build_hamiltonian(inp, check=False)
    e = Engine(h.n, h.num_atoms, h.supercell, len(TEMS), True)
    e.upload(h)
    e.set_temperatures(TEMS)
    e.init_spins("rand", seed=3)
    return e


def test_the_ell_choice_runs_the_ell_kernel():
    out = []
    for kind in ("auto", "ell"):
        with _engine() as e:
            e.set_sweep_kernel(kind)
            name, cs = e.sweep_kernel()
            assert name == "ell" and (cs > 0) == (kind == "auto")
            n0 = e.launch_count()
            e.sweep(5, 0, seed=4)
            launches = e.launch_count() - n0
            # a launch a colour and sweep, or one for all (and transposes)
            assert launches >= 5 * e.colouring()[1] if kind == "ell" else launches <= 3
            out.append((e.get_spins(), e.rejected()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


def test_batch_tuning_measures_both():
    with _engine() as e:
        e.begin(e.schedule(2, 1000, 1, seed=8))
        with Batch([e]) as b:
            t = b.tune(2)
            assert t["kernel"] == ["ell"] and t["cluster_us"] == [-1.0] and t["ell_us"][0] > 0.0
            name, cs = e.sweep_kernel()
            assert name == "ell"
            b.advance(2)


def test_the_default_cluster_geometry_reports_the_sites_per_thread_it_runs():
    """1,372 sites a colour on one CTA of 512 threads: two sites a thread at a time."""
    h = build_hamiltonian(sc_mcin(14, [(1e-3, NN)], [5.0] * 152), check=False)
    out = []
    for sites in (None, 1, 2):
        with Engine(h.n, h.num_atoms, h.supercell, 152) as e:
            e.upload(h)
            e.set_temperatures([5.0] * 152)
            if sites is None:
                assert e.cluster_geometry() == (1, 512, 2)
            else:
                e.set_cluster_geometry(1, 512, sites)
                assert e.cluster_geometry() == (1, 512, sites)
            e.init_spins("rand", seed=3)
            e.sweep(3, 0, seed=4)
            out.append((e.get_spins(), e.running_energy()))
    for spins, energy in out[1:]:
        assert np.array_equal(spins, out[0][0])
        assert np.array_equal(energy, out[0][1])   # the same sums in the same order
