"""Tables of the cluster-resident sweep for lattices with many neighbours or many
different stencil rows: long-ranged exchange on an even periodic lattice is
taken whatever the length of a site's list, and whatever the number of rows."""
import subprocess

import numpy as np
import pytest

import test_resident_tables as T
from espins_gb300.mcin import parse_mcin
from espins_gb300.tables import build_hamiltonian
from espins_gb300.workloads import lattice_mcin
from helpers import sc_mcin

FCC = [("Fe", p, 1.0) for p in ((0, 0, 0), (0.5, 0.5, 0), (0.5, 0, 0.5), (0, 0.5, 0.5))]


def fcc_shells(n):
    """Offsets of the first n shells of the face-centred lattice, 12, 6, 24, 12, 24, 8, 48 sites."""
    r = np.array([(x, y, z) for x in range(-4, 5) for y in range(-4, 5) for z in range(-4, 5) if (x + y + z) % 2 == 0])
    d = (r ** 2).sum(axis=1)
    return [[tuple(float(c) / 2 for c in v) for v in r[d == s]] for s in sorted(set(d))[1:n + 1]]


def fcc_ham(L, shells, tems=(10.0,), rich=False):
    J = [2e-3, -3e-4, 1e-4, 5e-5, -4e-5, 2e-5, 1e-5]
    sh = fcc_shells(shells)
    text = lattice_mcin(FCC, L, list(zip(J, sh)), tems=list(tems),
                        **({"biquad": (1e-4, sh[0]), "dm": (2e-4, sh[0])} if rich else {}))
    return build_hamiltonian(parse_mcin(text, "fcc"), check=False)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    # rows above 2^14 have their top bit in the highest bit of a descriptor
    drv = T.DRIVER.replace("((d >> 18) & 0x3fff) * t.rstride", "(((d >> 18) & 0x3fff) | ((d >> 63) << 14)) * t.rstride")
    drv = drv.replace("(int)(d >> 60) != i % na", "(int)((d >> 60) & 7) != i % na")
    assert drv.count("d >> 63") == 1 and drv.count("& 7") == 1
    d = tmp_path_factory.mktemp("resident")
    src, so = d / "driver.cpp", d / "driver.so"
    src.write_text(drv)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-I", T.CSRC] +
                   [x for i in T.CUDA_INC for x in ("-I", i)] +
                   [str(src), T.os.path.join(T.CSRC, "esp_resident.cpp"), T.os.path.join(T.CSRC, "esp_tables.cpp"),
                    "-o", str(so)], check=True)
    return T.C.CDLL(str(so))


# 134 neighbours a site (86 with one shell less), equal and unequal slabs
@pytest.mark.parametrize("L,shells,cs", [(6, 7, 1), (6, 6, 1), (8, 7, 3), (10, 7, 5)])
def test_rows_of_more_than_128_neighbours(lib, L, shells, cs):
    assert T._check(lib, fcc_ham(L, shells), (L,) * 3, cs, False)[0] == 0


def test_a_row_for_every_site(lib):
    # neighbours at every odd distance along the axes: no two sites of a class
    # lie alike to the supercell's edges, 17,576 rows on one CTA
    axes = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    shells = [(1e-3 / d, [tuple(s * d * c for c in o) for o in axes for s in ((1, -1) if d < 13 else (1,))])
              for d in range(1, 14, 2)]
    rc, info = T._check(lib, build_hamiltonian(sc_mcin(26, shells, [5.0]), check=False), (26,) * 3, 1, False)
    assert rc == 0
    assert info[0] >= 26 ** 3 * (4 + 39)
