// Tables of the cluster-resident sweep: local sites, item descriptors,
// stencil rows and coupling lists of every CTA of a cluster (esp_resident.h).
#include "esp_resident.h"
#include "esp_threads.h"

#include <algorithm>
#include <array>
#include <cstring>
#include <unordered_map>

namespace esp {

namespace {

// Distinct word sequences of one length, numbered in order of appearance.  Most
// sites repeat a sequence of the last few, which are looked at before a hash is
// made.
class WordSet {
public:
    explicit WordSet(int stride) : stride_(stride) {}
    int add(const uint32_t *w)
    {
        if (last_ >= 0 && is(last_, w)) return last_;
        for (int id : recent_)
            if (id >= 0 && is(id, w)) return last_ = id;
        last_ = find(w);
        recent_[turn_++ % recent_.size()] = last_;
        return last_;
    }
    int size() const { return (int)(data_.size() / stride_); }
    const std::vector<uint32_t> &data() const { return data_; }

private:
    bool is(int id, const uint32_t *w) const
    {
        const uint32_t *d = &data_[(size_t)id * stride_];
        for (int i = 0; i < stride_; ++i)
            if (d[i] != w[i]) return false;
        return true;
    }
    int find(const uint32_t *w)
    {
        uint64_t h = 1469598103934665603ull;   // FNV-1a over the words
        for (int i = 0; i < stride_; ++i) h = (h ^ w[i]) * 1099511628211ull;
        std::vector<int> &same = index_[h];
        for (int id : same)
            if (is(id, w)) return id;
        const int id = (int)(data_.size() / stride_);
        data_.insert(data_.end(), w, w + stride_);
        same.push_back(id);
        return id;
    }
    int stride_;
    unsigned turn_ = 0;
    int last_ = -1;
    std::array<int, 8> recent_{-1, -1, -1, -1, -1, -1, -1, -1};
    std::vector<uint32_t> data_;
    std::unordered_map<uint64_t, std::vector<int>> index_;
};

// Where a site lies: its rank and its local index there.
struct Place {
    uint16_t rank, loc;
};

uint32_t bits(float x)
{
    uint32_t u;
    std::memcpy(&u, &x, sizeof(u));
    return u;
}

}  // namespace

bool build_resident(const PrepOutput &prep, int N, int na, const int L[3], const ResidentSplit &sp,
                    const ResidentHeader &head, ResidentTables &out)
{
    const int nc = prep.num_colours, cs = sp.cs;
    if (nc > kMaxResidentColours || cs < 1 || cs > 16 || na > kMaxClusterAtoms) return false;
    out = ResidentTables();
    out.cs = cs;

    // ---- local sites: reference site of (rank, l), and back ----------------
    std::vector<int> site0(cs + 1, 0), ref(N);
    const int Hx = L[0] / 2, Hy = L[1] / 2, ncell = N / na;
    if (sp.general) {
        const int per = ncell / cs, rem = ncell % cs;
        if (per < 1) return false;
        out.nA = rem ? rem : cs;
        out.n_big = (rem ? per + 1 : per) * na;
        out.n_small = per * na;
    } else {
        out.nA = sp.nA;
        out.n_big = Hx * Hy * (sp.pz / 2) * 8 * na;
        out.n_small = Hx * Hy * (sp.pz / 2 - 1) * 8 * na;
    }
    for (int q = 0; q < cs; ++q) site0[q + 1] = site0[q] + (q < out.nA ? out.n_big : out.n_small);
    if (site0[cs] != N || 12 * out.n_big > 0x3ffff || N > 0xfffffff) return false;
    std::vector<Place> place(N);   // by permuted index
    out.loc2p.resize(N);
    for (int q = 0; q < cs; ++q) {
        const int n = site0[q + 1] - site0[q];
        auto put = [&](int l, int i) {
            const int p = prep.inv[i];
            ref[site0[q] + l] = i;
            out.loc2p[site0[q] + l] = p;
            place[p] = Place{(uint16_t)q, (uint16_t)l};
        };
        if (sp.general) {
            // atom-major, and the even x of a row of cells before the odd
            const int c0 = site0[q] / na, c1 = site0[q + 1] / na;
            for (int at = 0, l = 0; at < na; ++at)
                for (int lo = c0; lo < c1;) {
                    const int hi = std::min((lo / L[0] + 1) * L[0], c1);
                    for (int odd = 0; odd < 2; ++odd)
                        for (int c = lo + odd; c < hi; c += 2) put(l++, c * na + at);
                    lo = hi;
                }
        } else {
            const int pcl = n / (8 * na);
            for (int k = 0, l = 0; k < 8 * na; ++k)
                for (int r = 0; r < pcl; ++r) {
                    const int x = 2 * (r % Hx) + ((k >> 2) & 1), y = 2 * ((r / Hx) % Hy) + ((k >> 1) & 1);
                    const int z = slab_z0(sp.pz, sp.nA, q) + 2 * (r / (Hx * Hy)) + (k & 1);
                    put(l++, ((z * L[1] + y) * L[0] + x) * na + (k >> 3));
                }
        }
    }

    // ---- lengths of the neighbour lists -----------------------------------
    // entries, and the rich ones (a prefix up to the last one with a
    // biquadratic or DM coupling): of every site of a general lattice (by
    // permuted index), else of every atom
    struct Extent {
        int n, nr;
        // words of the row: the rich part, then the exchange-only one from the
        // next multiple of 4 on
        int count() const
        {
            const int rich = (nr + 1) & ~1;
            return n > nr ? ((rich + 3) & ~3) + ((n - nr + 1) & ~1) : rich;
        }
    };
    std::vector<Extent> extent(sp.general ? N : na, Extent{0, 0});
    if (sp.general) {
        const bool hb = prep.has_b, hd = prep.has_d;
        for (int p = 0; p < N; ++p) {
            int n = prep.nnb[p];
            while (n > 0 && prep.nbr[(size_t)(n - 1) * N + p] == p) --n;   // padding
            int nr = hb || hd ? n : 0;
            for (; nr > 0; --nr) {
                const size_t o = (size_t)(nr - 1) * N + p;
                if ((hb && prep.B[o] != 0.f) || (hd && (prep.Dx[o] != 0.f || prep.Dy[o] != 0.f || prep.Dz[o] != 0.f))) break;
            }
            extent[p] = Extent{n, nr};
        }
    } else {
        for (int at = 0; at < na; ++at) {
            const auto &st = prep.stencil[at];
            int nr = (int)st.size();
            while (nr > 0 && st[nr - 1].B == 0.f && st[nr - 1].Dx == 0.f && st[nr - 1].Dy == 0.f && st[nr - 1].Dz == 0.f) --nr;
            extent[at] = Extent{(int)st.size(), nr};
        }
    }
    int maxw = 0, maxr = 0, maxn = 0;
    for (const Extent &x : extent) {
        maxw = std::max(maxw, x.count());
        maxr = std::max(maxr, (x.nr + 1) & ~1);
        maxn = std::max(maxn, x.n);
    }
    if (maxw > 0xfff8) return false;   // the counts of a row's header have 16 bits
    out.jwords = std::max(4, (maxw + 3) & ~3);
    const int cstride = out.jwords + 4 * maxr;
    // rows 4 words apart modulo 8, so that the 16-byte reads of lanes with
    // different rows fall in different banks
    out.rstride = 4 + ((maxw + 3) & ~3);
    if (out.rstride % 8 == 0) out.rstride += 4;

    // ---- items --------------------------------------------------------------
    // colour by colour, in the order of the parity classes or of the local
    // sites; both ascend in l within a class, and the classes of a colour
    // ascend too
    std::vector<std::array<int, kMaxResidentColours + 1>> start(cs);
    std::vector<int> order(N);
    size_t entries = 0;
    for (int q = 0; q < cs; ++q) {
        const int n = site0[q + 1] - site0[q];
        std::vector<int> fill(nc + 1, 0);
        for (int l = 0; l < n; ++l) fill[prep.colour[ref[site0[q] + l]] + 1]++;
        for (int c = 0; c < nc; ++c) {
            out.max_items = std::max(out.max_items, fill[c + 1]);
            fill[c + 1] += fill[c];
        }
        for (int c = 0; c <= nc; ++c) start[q][c] = fill[c];
        for (int l = 0; l < n; ++l) order[site0[q] + fill[prep.colour[ref[site0[q] + l]]]++] = l;
    }
    for (const Extent &x : extent) entries += x.n;
    if (!sp.general) entries *= N / na;

    // ---- rows, couplings, descriptors --------------------------------------
    // by several threads, each some of the items with numbers of its own for
    // their rows (by rank) and coupling lists
    struct Part {
        Part(int cs, int rstride, int cstride) : rows(cs, WordSet(rstride)), couplings(cstride) {}
        std::vector<WordSet> rows;
        WordSet couplings;
    };
    const int nparts = work_parts(entries);
    std::vector<Part> parts(nparts, Part(cs, out.rstride, cstride));
    std::vector<char> refused(nparts, 0);
    std::vector<int> row_of(N);   // of an item
    auto first_of = [&](int part) { return (int)((int64_t)N * part / nparts); };
    auto build_part = [&](int part) -> bool {
        Part &my = parts[part];
        std::vector<uint32_t> cw(cstride), rw(out.rstride);
        std::vector<int> nb(maxn);               // permuted index of each neighbour
        std::vector<int> list_of_atom(na, -1);   // coupling lists of the atoms of a parity-class lattice
        // coupling list of the site at permuted index p, words as in its row
        auto list = [&](int p, int at, const Extent &x, int e1) {
            std::fill(cw.begin(), cw.end(), 0u);
            for (int e = 0; e < x.n; ++e) {
                const size_t o = (size_t)e * N + p;
                const int w = e < x.nr ? e : e1 + (e - x.nr);
                const StencilEntry *se = sp.general ? nullptr : &prep.stencil[at][e];
                cw[w] = bits(-(se ? se->J : prep.J[o]));
                if (e < x.nr) {
                    uint32_t *c4 = &cw[out.jwords + 4 * w];
                    c4[0] = bits(se ? se->B : prep.has_b ? prep.B[o] : 0.f);
                    c4[1] = bits(se ? se->Dx : prep.has_d ? prep.Dx[o] : 0.f);
                    c4[2] = bits(se ? se->Dy : prep.has_d ? prep.Dy[o] : 0.f);
                    c4[3] = bits(se ? se->Dz : prep.has_d ? prep.Dz[o] : 0.f);
                }
            }
            return my.couplings.add(cw.data());
        };
        int q = 0;
        for (int it = first_of(part), end = first_of(part + 1); it < end; ++it) {
            while (it >= site0[q + 1]) ++q;
            const int l = order[it], i = ref[site0[q] + l], p = out.loc2p[site0[q] + l], at = i % na;
            const Extent x = extent[sp.general ? p : at];
            if (sp.general) {
                for (int e = 0; e < x.n; ++e) nb[e] = prep.nbr[(size_t)e * N + p];
            } else {
                const int cell = i / na, cx = cell % L[0], cy = (cell / L[0]) % L[1], cz = cell / (L[0] * L[1]);
                auto wrap = [](int v, int len) { return v < 0 ? v + len : v >= len ? v - len : v; };   // |offset| <= len / 2
                const StencilEntry *se = prep.stencil[at].data();
                for (int e = 0; e < x.n; ++e)
                    nb[e] = prep.inv[((wrap(cz + se[e].dz, L[2]) * L[1] + wrap(cy + se[e].dy, L[1])) * L[0] +
                                      wrap(cx + se[e].dx, L[0])) * na + se[e].b];
            }
            // word of entry e: e + the gap after the rich ones
            const int e1 = (((x.nr + 1) & ~1) + 3) & ~3, gap = e1 - x.nr;
            uint32_t far = 0;
            for (int e = 0; e < x.n; ++e)
                if (place[nb[e]].rank != q) far |= 1u << std::min((e < x.nr ? e : e + gap) >> 2, 31);
            std::fill(rw.begin(), rw.end(), 0u);
            for (int e = 0; e < x.n; ++e) {
                const int w = e < x.nr ? e : e + gap;
                const Place there = place[nb[e]];
                const int delta = 12 * ((int)there.loc - l);
                rw[4 + w] = (uint32_t)delta;
                if (far && ((far >> std::min(w >> 2, 31)) & 1u))
                    rw[4 + w] = ((uint32_t)delta << 8) | (uint32_t)(there.rank == q ? 0 : there.rank + 1);
            }
            int li = sp.general ? -1 : list_of_atom[at];
            if (li < 0) {
                li = list(p, at, x, e1);
                if (!sp.general) list_of_atom[at] = li;
            }
            rw[0] = (uint32_t)x.count() | ((uint32_t)((x.nr + 1) & ~1) << 16);
            rw[1] = (uint32_t)li;   // its number here until the parts are put together
            rw[2] = far;
            rw[3] = (uint32_t)at;
            row_of[it] = my.rows[q].add(rw.data());
            if (sp.max_row_words && my.rows[q].size() * out.rstride + my.couplings.size() * cstride > sp.max_row_words) return false;
        }
        return true;
    };
    for_parts(nparts, [&](int part) {
        try {
            refused[part] = !build_part(part);
        } catch (const std::exception &) {
            refused[part] = 1;   // no memory
        }
    });
    for (char r : refused)
        if (r) return false;

    // put together in the items' order, which numbers rows and lists as one
    // thread would
    WordSet couplings(cstride);
    std::vector<std::vector<int>> list_no(nparts);
    std::vector<std::vector<uint32_t>> rank_rows(cs);
    out.desc.resize(N);
    for (int q = 0; q < cs; ++q) {
        WordSet rows(out.rstride);
        for (int part = 0; part < nparts; ++part) {
            const int it0 = std::max(first_of(part), site0[q]), it1 = std::min(first_of(part + 1), site0[q + 1]);
            if (it0 >= it1) continue;
            Part &my = parts[part];
            const std::vector<uint32_t> &lists = my.couplings.data();
            // the part's lists whose first site is of this rank come next
            std::vector<int> &no = list_no[part];
            std::vector<uint32_t> words = my.rows[q].data();
            std::vector<int> row_no(my.rows[q].size());
            for (size_t r = 0; r < row_no.size(); ++r) {
                uint32_t *w = &words[r * out.rstride];
                while (no.size() <= w[1]) no.push_back(couplings.add(&lists[no.size() * cstride]));
                w[1] = (uint32_t)(no[w[1]] * cstride);
                row_no[r] = rows.add(w);
            }
            for (int it = it0; it < it1; ++it) {
                const int l = order[it], i = ref[site0[q] + l], row = row_no[row_of[it]];
                out.desc[it] = (uint64_t)((uint32_t)(12 * l) | ((uint32_t)row << 18)) |
                               ((uint64_t)((uint32_t)i | ((uint32_t)(i % na) << 28) | ((uint32_t)(row >> 14) << 31)) << 32);
            }
        }
        if (rows.size() > 0x8000 ||
            (sp.max_row_words && rows.size() * out.rstride + couplings.size() * cstride > sp.max_row_words))
            return false;
        rank_rows[q] = rows.data();
    }

    // ---- the ranks' blocks -------------------------------------------------
    const int hw = (int)(sizeof(ResidentHeader) / 4);
    out.rows_off = hw + (int)couplings.data().size();
    size_t most = 0;
    for (const auto &r : rank_rows) most = std::max(most, r.size());
    out.blob_words = out.rows_off + (int)most;
    out.blob.assign((size_t)cs * out.blob_words, 0u);
    for (int q = 0; q < cs; ++q) {
        uint32_t *b = &out.blob[(size_t)q * out.blob_words];
        ResidentHeader hd = head;
        hd.ncolour = nc;
        for (int c = 0; c <= nc; ++c) hd.colour_start[c] = start[q][c];
        std::memcpy(b, &hd, sizeof(hd));
        std::memcpy(b + hw, couplings.data().data(), 4 * couplings.data().size());
        std::memcpy(b + out.rows_off, rank_rows[q].data(), 4 * rank_rows[q].size());
    }
    return true;
}

int rows_by_quads(ResidentTables &t)
{
    const int n = (t.blob_words - t.rows_off) / t.rstride;
    std::vector<uint32_t> rows((size_t)n * t.rstride);
    for (int q = 0; q < t.cs; ++q) {
        uint32_t *b = &t.blob[(size_t)q * t.blob_words + t.rows_off];
        std::copy(b, b + rows.size(), rows.begin());
        for (int r = 0; r < n; ++r)
            for (int w = 0; w < t.rstride; ++w)
                b[((size_t)(w / 4) * n + r) * 4 + w % 4] = rows[(size_t)r * t.rstride + w];
    }
    return 4 * n;
}

}  // namespace esp
