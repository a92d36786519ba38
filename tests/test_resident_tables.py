"""Tables of the cluster-resident sweep (espins_gb300/csrc/esp_resident.cpp):
every item's stencil row, decoded the way the kernel decodes it, must name the
neighbours of its site in merged-list order with their couplings, and every
offset must stay inside a rank's spins.  A small driver compiled with g++ from
the same sources walks the tables."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from espins_gb300.mcin import parse_mcin
from espins_gb300.tables import build_hamiltonian
from espins_gb300.workloads import BCC, BCC1, lattice_mcin
from helpers import N3, NN, NNN, sc_mcin

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "espins_gb300", "csrc")
CUDA_INC = [d for d in (os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/x/x/nvcc")), "include"),
                        "/usr/local/cuda/include") if os.path.exists(os.path.join(d, "cuda_runtime.h"))]

DRIVER = r'''
#include <cmath>
#include <cstdio>
#include <cstring>
#include "esp_resident.h"
using namespace esp;
// 0: as it should be; -1: the lattice is not taken; > 0: the first fault found
extern "C" int check(int N, int na, const int *L, int open, int jm, const int *jn, const int *jb, const double *jv,
                     int bm, const int *bn, const int *bb, const double *bv, int dm, const int *dn, const int *db,
                     const double *dv, const double *mag, int cs, int general, int limit, int *info)
{
    PrepInput in{};
    in.N = N; in.num_atoms = na; in.open_boundary = open != 0; in.mag = mag;
    for (int c = 0; c < 3; ++c) in.L[c] = L[c];
    in.j_maxnb = jm; in.j_nn = jn; in.j_nbors = jb; in.j_val = jv;
    in.b_maxnb = bm; in.b_nn = bn; in.b_nbors = bb; in.b_val = bv;
    in.d_maxnb = dm; in.d_nn = dn; in.d_nbors = db; in.d_val = dv;
    PrepOutput prep;
    std::string err;
    if (prepare_tables(in, prep, err)) return 100;
    int pz = 0, nA = cs;
    if (!general) {
        if (!prep.invariant) return -1;
        const int pairs = L[2] / 2, q = pairs / cs, rem = pairs % cs;
        if (q < 1) return -1;
        pz = 2 * (rem ? q + 1 : q); nA = rem ? rem : cs;
    }
    ResidentHeader head{};
    ResidentTables t;
    if (!build_resident(prep, N, na, L, ResidentSplit{cs, general != 0, pz, nA, limit}, head, t)) return -1;
    info[0] = t.blob_words - t.rows_off; info[1] = t.max_items; info[2] = t.n_big;
    std::vector<char> seen(N, 0);
    std::vector<int> site0(cs + 1, 0);
    for (int q = 0; q < cs; ++q) site0[q + 1] = site0[q] + (q < t.nA ? t.n_big : t.n_small);
    if (site0[cs] != N) return 1;
    for (int q = 0; q < cs; ++q) {
        const int n = site0[q + 1] - site0[q];
        const uint32_t *blob = &t.blob[(size_t)q * t.blob_words];
        ResidentHeader hd;
        std::memcpy(&hd, blob, sizeof(hd));
        if (hd.ncolour != prep.num_colours || hd.colour_start[0] != 0 || hd.colour_start[hd.ncolour] != n) return 2;
        for (int c = 0; c < hd.ncolour; ++c) {
            if (hd.colour_start[c + 1] - hd.colour_start[c] > t.max_items) return 3;
            for (int it = hd.colour_start[c]; it < hd.colour_start[c + 1]; ++it) {
                const uint64_t d = t.desc[site0[q] + it];
                const int l = (int)(d & 0x3ffff) / 12, i = (int)((d >> 32) & 0xfffffff);
                const size_t row = (size_t)((d >> 18) & 0x3fff) * t.rstride;
                if (l >= n || i >= N || (int)(d >> 60) != i % na || prep.colour[i] != c || seen[i]++) return 4;
                if (t.loc2p[site0[q] + l] != prep.inv[i]) return 5;
                if (t.rows_off + row + t.rstride > (size_t)t.blob_words) return 6;
                const uint32_t *rw = blob + t.rows_off + row;
                const int cnt = (int)(rw[0] & 0xffff), nr = (int)(rw[0] >> 16);
                if (4 + cnt > t.rstride || (nr & 1) || (cnt & 1) || cnt > t.jwords || rw[3] != (uint32_t)(i % na)) return 7;
                const float *J = reinterpret_cast<const float *>(blob + sizeof(ResidentHeader) / 4 + rw[1]);
                const float *R = J + t.jwords;
                if (sizeof(ResidentHeader) / 4 + rw[1] + t.jwords + 4 * nr > (size_t)t.rows_off) return 8;
                // the kernel's order of entry words: rich ones, then from the next multiple of 4
                const int p = prep.inv[i];
                int k = 0;
                for (int e = 0; e < cnt; ++e) {
                    if (e == nr) e = (e + 3) & ~3;
                    if (e >= cnt) break;
                    const uint32_t w = rw[4 + e];
                    const bool enc = (rw[2] >> (e / 4 < 31 ? e / 4 : 31)) & 1u;
                    const int off = enc ? (int)w >> 8 : (int)w, own = enc ? (int)(w & 0xff) : 0;
                    const int rn = own ? own - 1 : q;
                    if (rn < 0 || rn >= cs || off % 12) return 9;
                    const int ln = l + off / 12;
                    if (ln < 0 || ln >= site0[rn + 1] - site0[rn]) return 10;
                    const int pn = t.loc2p[site0[rn] + ln];
                    const bool rich = e < nr;
                    const bool zero = J[e] == 0.f && (!rich || (R[4 * e] == 0.f && R[4 * e + 1] == 0.f && R[4 * e + 2] == 0.f && R[4 * e + 3] == 0.f));
                    const size_t o = (size_t)k * N + p;
                    const bool more = k < prep.nnb[p] && prep.nbr[o] != p;
                    if (more && pn == prep.nbr[o] && -J[e] == prep.J[o] &&
                        (rich ? R[4 * e] == (prep.has_b ? prep.B[o] : 0.f) && R[4 * e + 1] == (prep.has_d ? prep.Dx[o] : 0.f) &&
                                    R[4 * e + 2] == (prep.has_d ? prep.Dy[o] : 0.f) && R[4 * e + 3] == (prep.has_d ? prep.Dz[o] : 0.f)
                              : (!prep.has_b || prep.B[o] == 0.f) && (!prep.has_d || (prep.Dx[o] == 0.f && prep.Dy[o] == 0.f && prep.Dz[o] == 0.f)))) {
                        ++k;
                    } else if (!zero || pn != p) {
                        return 11;   // neither the next neighbour nor padding
                    }
                }
                if (k < prep.nnb[p] && prep.nbr[(size_t)k * N + p] != p) return 12;   // a neighbour is missing
            }
        }
    }
    for (int i = 0; i < N; ++i) if (!seen[i]) return 13;
    return 0;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("resident")
    src, so = d / "driver.cpp", d / "driver.so"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-I", CSRC] + [x for i in CUDA_INC for x in ("-I", i)] +
                   [str(src), os.path.join(CSRC, "esp_resident.cpp"), os.path.join(CSRC, "esp_tables.cpp"), "-o", str(so)],
                   check=True)
    return C.CDLL(str(so))


def _check(lib, h, L, cs, general, open_=False, limit=0):
    keep = []

    def p(a, dt):
        keep.append(np.ascontiguousarray(a, dtype=dt))
        return keep[-1].ctypes.data_as(C.c_void_p)

    def ell(t):
        if t is None:
            return [0, None, None, None]
        return [t.nb.shape[0], p(t.nn, np.int32), p(t.nb + 1, np.int32), p(t.val, np.float64)]

    info = (C.c_int * 3)()
    rc = lib.check(h.n, h.num_atoms, p(L, np.int32), int(open_), *ell(h.jij), *ell(h.bij), *ell(h.dij),
                   p(h.mag, np.float64), cs, int(general), limit, info)
    return rc, list(info)


def _sc(L, shells, open_=False, **kw):
    inp = sc_mcin(4, shells, [5.0], **kw)
    inp.supercell_size = list(L)
    inp.boundary_open = open_
    return build_hamiltonian(inp, check=False)


@pytest.mark.parametrize("L,cs", [((4, 4, 4), 1), ((4, 4, 4), 2), ((2, 6, 8), 3), ((12, 12, 12), 5), ((14, 10, 6), 2)])
def test_parity_class_rows_name_the_stencil(lib, L, cs):
    shells = [(1e-3, NN), (3e-4, NNN), (-5e-5, N3)] if min(L) > 2 else [(1e-3, NN[2:])]
    h = _sc(L, shells, **({"dm": 1e-4, "bq": 2e-5} if min(L) > 2 else {}))
    rc, info = _check(lib, h, L, cs, False)
    assert rc == 0
    # one row per class and per side of the lattice's edges, not per site
    assert info[0] <= 8 * 8 * (4 + 36)


def test_parity_class_rows_of_a_two_atom_cell(lib):
    inp = parse_mcin(lattice_mcin(BCC, 8, [(2e-3, BCC1), (5e-4, NN), (-1e-4, NNN)], tems=[10.0], single_ion=-5e-5), "bcc")
    for cs in (1, 2, 3):
        assert _check(lib, build_hamiltonian(inp), (8, 8, 8), cs, False)[0] == 0


@pytest.mark.parametrize("L,open_,cs", [((5, 5, 5), True, 1), ((5, 4, 7), True, 3), ((7, 6, 5), False, 2),
                                        ((6, 6, 6), True, 4), ((9, 5, 1), True, 2), ((11, 3, 3), False, 1)])
def test_general_rows_name_the_merged_lists(lib, L, open_, cs):
    shells = [(1e-3, NN)] if min(L) < 4 else [(1e-3, NN), (3e-4, NNN)]
    h = _sc(L, shells, open_, dm=1e-4)
    assert _check(lib, h, L, cs, True, open_)[0] == 0


def test_a_lattice_with_a_row_per_site_is_left_to_the_other_kernel(lib):
    h = _sc((9, 9, 9), [(1e-3, NN)], True)
    h.jij.val[...] *= np.random.default_rng(0).uniform(0.5, 1.5, size=h.jij.val.shape)
    assert _check(lib, h, (9, 9, 9), 1, True, True, limit=4096)[0] == -1
