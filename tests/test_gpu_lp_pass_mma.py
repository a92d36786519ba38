"""The training pass of the mma.sync engine at the edges of its tiles and
chains: batches below one k-step of 32 and one tile of 32 rows, remainders of
both, chains shorter and longer than the four steps in flight and than the
32 rows of a column sum.  Loss and gradient against the FP64 network with
the bounds of BF16 activations (tests/test_gpu_learned.py)."""
import numpy as np
import pytest

import oracle as O
from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, sc_mcin
from test_gpu_lp_step import _bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8, 24, 72, 136, 1160, 4104])
def test_loss_and_gradient_at_the_edges(rows):
    h = build_hamiltonian(sc_mcin(4, [(1e-3, NN)], [5.0]))
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, 12)).astype(np.float32)
    s = rng.normal(size=(rows, 3))
    s /= np.linalg.norm(s, axis=1, keepdims=True)
    t = np.column_stack([s, rng.uniform(0.1, 20.0, rows)]).astype(np.float32)
    with Engine(h.n, h.num_atoms, h.supercell, 1) as e:
        e.upload(h)
        e.set_temperatures([5.0])
        e.lp_init(seed=3)
        e.lp_set_engine("mma")
        p = e.lp_weights().astype(np.float64)
        loss, g = e.lp_loss_grad(x, t)
        loss2, g2 = e.lp_loss_grad(x, t)
    q = p.copy()
    for lo, hi in ((0, 1536), (1664, 18048), (18176, 20736)):
        q[lo:hi] = _bf16(p[lo:hi])
    lo_, go = O.lp_loss_grad(q, _bf16(x), t.astype(np.float64))
    assert abs(loss - lo_) <= 1e-2 * abs(lo_)
    assert np.linalg.norm(g - go) <= 5e-2 * np.linalg.norm(go)
    assert loss == loss2 and np.array_equal(g, g2)
