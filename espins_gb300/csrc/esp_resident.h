// Host-built tables of the cluster-resident sweep (esp_resident.cpp).
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

#include "esp_tables.h"

namespace esp {

constexpr int kMaxClusterAtoms = 8;

// The z planes of a replica over the cs CTAs of its cluster: ranks
// [0, nA) hold pz planes, the others pz - 2 (pz even; nA == cs when every
// slab is equal), so any even Lz with Lz / 2 >= cs splits.  Local sites of a
// rank follow those of the ranks before it in the replica's slab order.
__host__ __device__ inline int slab_planes(int pz, int nA, int q) { return q < nA ? pz : pz - 2; }
__host__ __device__ inline int slab_z0(int pz, int nA, int q) { return q < nA ? q * pz : nA * pz + (q - nA) * (pz - 2); }

// What a CTA of the cluster path knows about its rank's sites, at the start of
// the rank's table block ; followed there by the coupling
// lists and the stencil rows.
constexpr int kMaxResidentColours = 64;
struct ResidentHeader {
    int ncolour, pad[3];
    // items of colour c: descriptors [colour_start[c], colour_start[c+1])
    int colour_start[kMaxResidentColours + 4];
    float4 si[kMaxClusterAtoms];       // (ax, ay, az, Delta)
    float4 fld[kMaxClusterAtoms];      // (f ax, f ay, f az, 0)
    float mag[kMaxClusterAtoms];
};
static_assert(sizeof(ResidentHeader) % 16 == 0, "table parts stay 16-byte aligned");


// The tables of one split of a lattice over the cs CTAs of a cluster.
//
// Local sites.  Parity-class lattices (general == false): the slab of z planes
// of slab_planes / slab_z0, class-major (class k = atom*8 + px*4 + py*2 + pz,
// then half-cell coordinates).  General lattices: whole cells in reference
// order, as equal numbers of cells as possible, atom by atom, and within a
// row of cells along x every second one first: a colour's sites are then close
// to contiguous (cells in order with the atom fastest put the lanes of a
// gather in 8 to 16 of the 32 banks).
//
// Items: a rank's sites colour by colour, class by class (ascending) or in
// local order; desc = (byte offset of the spin | row << 18, reference site |
// atom << 28 | row >> 14 << 31): rows above 2^14, more than shared memory
// holds of any length, need the last bit, and only the variant that reads its
// rows from global memory decodes it.
//
// Stencil rows: sites whose neighbours lie at the same byte offsets from
// their own spin and carry the same couplings share a row: four header words
// (entry words | rich entries << 16, word offset of the coupling list, quads
// of entries that hold a peer CTA's spin, atom), then one word per entry: the
// byte offset, or in those quads (offset << 8) | (owner rank + 1, 0 for this
// CTA).  Entries up to the last one with a biquadratic or DM coupling come
// first, padded to 2 (rich), the exchange-only ones from the next multiple of
// 4 on, padded to 2; padding is the site itself with zero couplings, which
// adds nothing to any sum.  Every entry keeps its place in the merged list.
//
// Coupling lists: -J of every entry word (jwords), then (B, Dx, Dy, Dz) of the
// rich ones.
struct ResidentTables {
    int cs = 0, nA = 0, n_big = 0, n_small = 0;
    int max_items = 0;                  // largest colour of a rank
    int blob_words = 0, rows_off = 0, rstride = 0, jwords = 0;
    std::vector<uint64_t> desc;         // x in the low half
    std::vector<int32_t> loc2p;
    std::vector<uint32_t> blob;         // [rank][blob_words]
    size_t table_bytes(bool rows_smem) const { return (size_t)(rows_smem ? blob_words : rows_off) * 4; }
};

struct ResidentSplit {
    int cs;
    bool general;
    int pz, nA;                         // parity-class slabs
    int max_row_words;                  // give up beyond this many words of rows in a rank (0: no limit)
};

// head: single-ion, field and moment of every atom; the rest is filled here.
// false when the lattice has more colours, entries or rows than the kernel
// takes (a replica that fits its cluster's shared memory has not).
bool build_resident(const PrepOutput &prep, int N, int na, const int L[3], const ResidentSplit &sp,
                    const ResidentHeader &head, ResidentTables &out);

// The ranks' rows from [row][rstride] to [quad][row][4], the order of rows
// that stay in global memory: threads of a warp with rows that follow one
// another read 16 bytes each that do too.  Returns the words of one quad.
int rows_by_quads(ResidentTables &t);

}  // namespace esp
