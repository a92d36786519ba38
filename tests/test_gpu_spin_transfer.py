"""Spin transfers: chunks of a pinned ring that host threads convert while
others are in flight.  What comes back is the FP64 value rounded to FP32, bit
for bit, for arrays below one piece (16 Ki values), of whole and ragged pieces
and chunks, and past the ring's 8 chunks of 1 Mi values; also with two
handles' transfers at once."""
import threading

import numpy as np
import pytest

from espins_gb300.lib import Engine
from espins_gb300.mcin import parse_mcin
from espins_gb300.tables import build_hamiltonian

pytestmark = pytest.mark.gpu


def _round_trips(L, R, seed, out, n=2):
    text = ["begin unit_cell_cart", "1 0 0", "0 1 0", "0 0 1", "end unit_cell_cart", "begin atoms_frac",
            "Fe 0 0 0 1.0", "end atoms_frac", f"supercell_size = {L[0]} {L[1]} {L[2]}", "tems_mode = man",
            f"tems_num = {R}", "tems = " + " ".join(str(2.0 + t) for t in range(R)), "steps_warmup = 1",
            "steps_mc = 1", "steps_measure = 1", "begin jij_parameters", "f1=0,0,0:f2=1,0,0:jij=0.001",
            "f1=0,0,0:f2=-1,0,0:jij=0.001", "end jij_parameters"]
    h = build_hamiltonian(parse_mcin("\n".join(text) + "\n", seedname="sc"))
    rng = np.random.default_rng(seed)
    ok = True
    with Engine(h.n, h.num_atoms, h.supercell, R) as e:
        e.upload(h)
        e.set_temperatures([2.0 + t for t in range(R)])
        for _ in range(n):
            s = rng.normal(size=(R, h.n, 3))
            e.set_spins(s)
            ok &= np.array_equal(e.get_spins(), s.astype(np.float32).astype(np.float64))
    out.append(ok)


# values 3 N R: 24; 16383 and 16386 (a piece, less and more by one or two);
# 49152 = 3 pieces in one chunk; 12 pieces in 3 chunks; 2 chunks, the
# last ragged;
# 8 chunks of 1 Mi and a ragged ninth and tenth
@pytest.mark.parametrize("L,R", [((2, 2, 2), 1), ((43, 127, 1), 1), ((2, 2731, 1), 1), ((32, 32, 16), 1),
                                 ((64, 64, 16), 1), ((32, 32, 17), 2), ((48, 48, 48), 27)])
def test_round_trip(L, R):
    out = []
    _round_trips(L, R, 5, out)
    assert out == [True]


def test_two_handles_at_once():
    out = []
    ts = [threading.Thread(target=_round_trips, args=(L, R, k, out, 4))
          for k, (L, R) in enumerate([((32, 32, 32), 24), ((40, 40, 20), 31)])]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert out == [True, True]
