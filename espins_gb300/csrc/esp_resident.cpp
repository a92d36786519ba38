// Tables of the cluster-resident sweep: local sites, item descriptors,
// stencil rows and coupling lists of every CTA of a cluster (esp_resident.h).
#include "esp_resident.h"

#include <algorithm>
#include <array>
#include <cstring>
#include <unordered_map>

namespace esp {

namespace {

// Distinct word sequences of one length, numbered in order of appearance.
class WordSet {
public:
    explicit WordSet(int stride) : stride_(stride) {}
    int add(const uint32_t *w)
    {
        uint64_t h = 1469598103934665603ull;   // FNV-1a over the words
        for (int i = 0; i < stride_; ++i) h = (h ^ w[i]) * 1099511628211ull;
        std::vector<int> &same = index_[h];
        for (int id : same)
            if (!std::memcmp(&data_[(size_t)id * stride_], w, sizeof(uint32_t) * stride_)) return id;
        const int id = (int)(data_.size() / stride_);
        data_.insert(data_.end(), w, w + stride_);
        same.push_back(id);
        return id;
    }
    int size() const { return (int)(data_.size() / stride_); }
    const std::vector<uint32_t> &data() const { return data_; }

private:
    int stride_;
    std::vector<uint32_t> data_;
    std::unordered_map<uint64_t, std::vector<int>> index_;
};

struct Entry {
    int site;                    // reference index
    float J, B, Dx, Dy, Dz;
    bool rich() const { return B != 0.f || Dx != 0.f || Dy != 0.f || Dz != 0.f; }
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
    std::vector<int> site0(cs + 1, 0), ref(N), rank_of(N), loc_of(N);
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
    for (int q = 0; q < cs; ++q)
        for (int l = 0; l < site0[q + 1] - site0[q]; ++l) {
            const int n = site0[q + 1] - site0[q];
            int i;
            if (sp.general) {
                // atom-major, and the even x of a row of cells before the odd
                const int ncl = n / na, at = l / ncl;
                int c = site0[q] / na + l % ncl;
                const int row = c / L[0], lo = std::max(row * L[0], site0[q] / na);
                const int hi = std::min((row + 1) * L[0], site0[q + 1] / na);
                const int even = (hi - lo + 1) / 2, k = c - lo;
                c = lo + (k < even ? 2 * k : 2 * (k - even) + 1);
                i = c * na + at;
            } else {
                const int pcl = n / (8 * na);
                const int k = l / pcl, r = l % pcl;
                const int x = 2 * (r % Hx) + ((k >> 2) & 1), y = 2 * ((r / Hx) % Hy) + ((k >> 1) & 1);
                const int z = slab_z0(sp.pz, sp.nA, q) + 2 * (r / (Hx * Hy)) + (k & 1);
                i = ((z * L[1] + y) * L[0] + x) * na + (k >> 3);
            }
            ref[site0[q] + l] = i;
            rank_of[i] = q;
            loc_of[i] = l;
        }
    out.loc2p.resize(N);
    for (int s = 0; s < N; ++s) out.loc2p[s] = prep.inv[ref[s]];

    // ---- neighbours of a reference site in merged-list order ---------------
    std::vector<Entry> nb;
    auto neighbours = [&](int i) {
        nb.clear();
        if (!sp.general) {
            const int cell = i / na, x = cell % L[0], y = (cell / L[0]) % L[1], z = cell / (L[0] * L[1]);
            auto wrap = [](int v, int n) { v %= n; return v < 0 ? v + n : v; };
            for (const StencilEntry &e : prep.stencil[i % na])
                nb.push_back({((wrap(z + e.dz, L[2]) * L[1] + wrap(y + e.dy, L[1])) * L[0] + wrap(x + e.dx, L[0])) * na + e.b,
                              e.J, e.B, e.Dx, e.Dy, e.Dz});
            return;
        }
        const int p = prep.inv[i];
        for (int k = 0; k < prep.nnb[p]; ++k) {
            const size_t o = (size_t)k * N + p;
            if (prep.nbr[o] == p) break;   // padding
            nb.push_back({prep.perm[prep.nbr[o]], prep.J[o], prep.has_b ? prep.B[o] : 0.f, prep.has_d ? prep.Dx[o] : 0.f,
                          prep.has_d ? prep.Dy[o] : 0.f, prep.has_d ? prep.Dz[o] : 0.f});
        }
    };
    // rich entries (a prefix up to the last one), and the words of a row
    auto extents = [&](int &nr, int &cnt) {
        nr = 0;
        for (size_t e = 0; e < nb.size(); ++e)
            if (nb[e].rich()) nr = (int)e + 1;
        const int ne = (int)nb.size() - nr;
        cnt = ((nr + 1) & ~1);
        if (ne) cnt = ((cnt + 3) & ~3) + ((ne + 1) & ~1);
    };
    int maxw = 0, maxr = 0;
    {
        // the longest row: every site of a general lattice, one per atom else
        const int n = sp.general ? N : na;
        for (int i = 0; i < n; ++i) {
            int nr, cnt;
            neighbours(i);
            extents(nr, cnt);
            maxw = std::max(maxw, cnt);
            maxr = std::max(maxr, (nr + 1) & ~1);
        }
    }
    if (maxw > 0xfff8) return false;   // the counts of a row's header have 16 bits
    out.jwords = std::max(4, (maxw + 3) & ~3);
    const int cstride = out.jwords + 4 * maxr;
    // rows 4 words apart modulo 8, so that the 16-byte reads of lanes with
    // different rows fall in different banks
    out.rstride = 4 + ((maxw + 3) & ~3);
    if (out.rstride % 8 == 0) out.rstride += 4;

    // ---- rows, couplings, descriptors --------------------------------------
    out.desc.resize(N);
    WordSet couplings(cstride);
    std::vector<std::vector<uint32_t>> rank_rows(cs);
    std::vector<std::array<int, kMaxResidentColours + 1>> start(cs);
    std::vector<uint32_t> cw(cstride), rw(out.rstride);
    for (int q = 0; q < cs; ++q) {
        WordSet rows(out.rstride);
        const int n = site0[q + 1] - site0[q];
        // items: colour by colour, in the order of the parity classes or of
        // the local sites; both ascend in l within a class, and the classes of
        // a colour ascend too
        std::vector<int> order(n), fill(nc + 1, 0);
        for (int l = 0; l < n; ++l) fill[prep.colour[ref[site0[q] + l]] + 1]++;
        for (int c = 0; c < nc; ++c) {
            out.max_items = std::max(out.max_items, fill[c + 1]);
            fill[c + 1] += fill[c];
        }
        for (int c = 0; c <= nc; ++c) start[q][c] = fill[c];
        for (int l = 0; l < n; ++l) order[fill[prep.colour[ref[site0[q] + l]]]++] = l;
        for (int it = 0; it < n; ++it) {
            const int l = order[it], i = ref[site0[q] + l];
            neighbours(i);
            int nr, cnt;
            extents(nr, cnt);
            std::fill(cw.begin(), cw.end(), 0u);
            std::fill(rw.begin(), rw.end(), 0u);
            uint32_t far = 0;
            const int e1 = (((nr + 1) & ~1) + 3) & ~3;
            auto word_of = [&](size_t e) { return (int)e < nr ? (int)e : e1 + ((int)e - nr); };
            for (size_t e = 0; e < nb.size(); ++e)
                if (rank_of[nb[e].site] != q) far |= 1u << std::min(word_of(e) >> 2, 31);
            for (size_t e = 0; e < nb.size(); ++e) {
                const int w = word_of(e), rn = rank_of[nb[e].site];
                const int delta = 12 * (loc_of[nb[e].site] - l);
                const bool enc = (far >> std::min(w >> 2, 31)) & 1u;
                rw[4 + w] = enc ? ((uint32_t)delta << 8) | (uint32_t)(rn == q ? 0 : rn + 1) : (uint32_t)delta;
                cw[w] = bits(-nb[e].J);
                if ((int)e < nr) {
                    uint32_t *c4 = &cw[out.jwords + 4 * w];
                    c4[0] = bits(nb[e].B); c4[1] = bits(nb[e].Dx); c4[2] = bits(nb[e].Dy); c4[3] = bits(nb[e].Dz);
                }
            }
            rw[0] = (uint32_t)cnt | ((uint32_t)((nr + 1) & ~1) << 16);
            rw[1] = (uint32_t)(couplings.add(cw.data()) * cstride);
            rw[2] = far;
            rw[3] = (uint32_t)(i % na);
            const int row = rows.add(rw.data());
            if (row > 0x7fff || (sp.max_row_words && rows.size() * out.rstride + couplings.size() * cstride > sp.max_row_words))
                return false;
            out.desc[site0[q] + it] =
                (uint64_t)((uint32_t)(12 * l) | ((uint32_t)row << 18)) |
                ((uint64_t)((uint32_t)i | ((uint32_t)(i % na) << 28) | ((uint32_t)(row >> 14) << 31)) << 32);
        }
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
