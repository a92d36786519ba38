"""Tables of lattices large enough to be merged and built by several threads (on
a host with several cores): every item's row still names the merged list of its
site, rows and coupling lists are numbered across the threads' parts, and a
lattice whose rows do not fit is still refused."""
import numpy as np
import pytest

from helpers import N3, NN, NNN
from test_resident_tables import _check, _sc, lib  # noqa: F401  (lib is a fixture)

J12 = [(1e-3, NN), (3e-4, NNN)]


# parts that end inside a rank, and ranks that end inside a part
@pytest.mark.parametrize("L,cs", [((20, 20, 20), 2), ((16, 18, 26), 5), ((24, 24, 12), 1)])
def test_parity_class_tables_by_threads(lib, L, cs):
    assert _check(lib, _sc(L, J12 + [(-5e-5, N3)], dm=1e-4, bq=2e-5), L, cs, False)[0] == 0


@pytest.mark.parametrize("L,open_,cs", [((21, 20, 19), True, 3), ((17, 19, 23), False, 1), ((41, 37, 1), True, 2)])
def test_general_tables_by_threads(lib, L, open_, cs):
    assert _check(lib, _sc(L, [(1e-3, NN)] if 1 in L else J12, open_, dm=1e-4), L, cs, True, open_)[0] == 0


def test_rows_that_do_not_fit_are_refused(lib):
    L = (21, 21, 21)
    h = _sc(L, J12, True)
    h.jij.val[...] *= np.random.default_rng(0).uniform(0.5, 1.5, size=h.jij.val.shape)
    assert _check(lib, h, L, 2, True, True, limit=12000)[0] == -1
