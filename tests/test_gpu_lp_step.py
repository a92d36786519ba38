"""The fused training step of the learned proposal on the tcgen05 engine
(esp_lp_step.cu) at the edges of its split: batches below one chunk of 64
rows, one chunk and a remainder, parts of 128 rows with a remainder, parts of
more rows than are in flight at once.  Loss and gradient against the FP64
network with the bounds of BF16 activations (tests/test_gpu_learned.py), and a
step of the optimiser against Adam applied to that gradient."""
import numpy as np
import pytest

import oracle as O
from espins_gb300.lib import Engine
from espins_gb300.tables import build_hamiltonian
from helpers import NN, sc_mcin

pytestmark = pytest.mark.gpu


def _bf16(a):
    u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
    return ((u + np.uint32(0x7FFF) + ((u >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)).view(
        np.float32).astype(np.float64)


@pytest.mark.parametrize("rows", [1, 8, 72, 130, 4104, 8200])
def test_loss_and_gradient_at_the_edges_of_the_split(rows):
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
        e.lp_set_engine("tcgen05")
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


def test_first_step_moves_every_weight_by_the_learning_rate():
    """Adam's first step is lr * g / (|g| + eps'), eps' = eps sqrt(1 - beta2)
    / (1 - beta1): the sign of the gradient wherever it is far above eps'."""
    h = build_hamiltonian(sc_mcin(8, [(1e-3, NN)], [5.0, 20.0]))
    with Engine(h.n, h.num_atoms, h.supercell, 2) as e:
        e.upload(h)
        e.set_temperatures([5.0, 20.0])
        e.init_spins("rand", seed=1)
        e.sweep(5, 0, seed=1)
        e.lp_init(seed=2)
        e.lp_set_engine("tcgen05")
        # a training set of one row: every draw is that row
        e.lp_reserve(1)
        assert e.lp_collect(0) == 1
        f, t = e.lp_data(0, 1)
        w0 = e.lp_weights()
        _, g = e.lp_loss_grad(np.repeat(f, 200, axis=0), np.repeat(t, 200, axis=0))
        loss = e.lp_train(1, batch=200, lr=1e-3, seed=7)
        w1 = e.lp_weights()
    assert np.isfinite(loss).all()
    big = np.abs(g) > 1e-4
    assert big.sum() > 100
    # 2^-24 relative of a weight of size one on top of the step itself
    assert np.max(np.abs((w0 - w1)[big] - 1e-3 * np.sign(g[big]))) <= 1e-3 * 1e-3 + 2.0 ** -23
    assert np.array_equal(w0[g == 0.0], w1[g == 0.0])
