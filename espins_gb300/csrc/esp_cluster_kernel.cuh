// Cluster-resident sweeps.
//
// One thread-block cluster holds one replica's whole lattice in distributed
// shared memory for the length of a launch: each CTA of the cluster owns a
// slab of z planes of a translation-invariant periodic lattice, stored
// class-major (parity class k = atom*8 + px*4 + py*2 + pz, then half-cell
// coordinates), or some whole cells of any other lattice (odd, open, one
// layer), atom by atom, so a colour pass reads its neighbours from its own or a
// peer CTA's shared memory and writes only its own.  A launch runs `n_meas`
// units of `steps_measure` sweeps, each unit followed by the measurement of mcarlo.F90:536-590 / pt.F90:789-849
// (accumulators, binning, Pm_get histogram), all without touching global
// memory; each CTA reads its slab at the start and writes it back at the end
// as one contiguous block (k_to_slabs / k_from_slabs convert the spin arrays
// around the launch).
//
// Updates, random numbers and the local-field arithmetic are those of
// k_sweep_ell (same colouring, same Philox counter (site, replica, sweep), the
// stencil lists in the merged-list order, the shared explicitly rounded
// trial / field / energy functions), so both kernels produce the same
// trajectory.  Waits are cluster barriers only (hardware, no spinning).
#pragma once
#include <cooperative_groups.h>
#include <type_traits>

#include "esp_cluster.h"
#include "esp_device.cuh"

namespace cg = cooperative_groups;

namespace esp {

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
// Named barriers: wait for, or only announce to, n threads.
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }

// Address, in the cluster's shared-memory window, of what lies at `addr` of
// this CTA's shared memory in the CTA of that rank; and a spin read there.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank)
{
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(d) : "r"(addr), "r"(rank));
    return d;
}
__device__ __forceinline__ void ld_cluster3(uint32_t addr, float &x, float &y, float &z)
{
    asm volatile("ld.shared::cluster.f32 %0, [%3];\n\tld.shared::cluster.f32 %1, [%3+4];\n\t"
                 "ld.shared::cluster.f32 %2, [%3+8];\n"
                 : "=f"(x), "=f"(y), "=f"(z)
                 : "r"(addr)
                 : "memory");
}

// A spin of this CTA's shared memory, by 32-bit address.
__device__ __forceinline__ void ld_shared3(uint32_t addr, float &x, float &y, float &z)
{
    asm volatile("ld.shared.f32 %0, [%3];\n\tld.shared.f32 %1, [%3+4];\n\tld.shared.f32 %2, [%3+8];\n"
                 : "=f"(x), "=f"(y), "=f"(z)
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ uint4 ld_shared_u4(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint2 ld_shared_u2(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 ld_shared_f2(uint32_t addr)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared4(uint32_t addr, float x, float y, float z, float w)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ void st_shared3(uint32_t addr, float x, float y, float z)
{
    asm volatile("st.shared.f32 [%0], %1;\n\tst.shared.f32 [%0+4], %2;\n\tst.shared.f32 [%0+8], %3;\n" ::"r"(addr),
                 "f"(x), "f"(y), "f"(z)
                 : "memory");
}

// Warp-aggregated increments of a shared-memory histogram (1-based bins,
// bin <= 0 adds nothing; every lane of the warp calls together).  Low
// temperatures put almost every cell in one bin: while a warp's 32 cells share
// one bin, and the same bin as its previous call, the count stays in a
// register (one atomic per run instead of one per call); mixed warps add per
// lane.
struct WarpRun {
    int bin = -1;
    unsigned cnt = 0u;
};
__device__ __forceinline__ void hist_add(unsigned *h, WarpRun &run, int bin)
{
    const int b0 = __shfl_sync(0xffffffffu, bin, 0);
    if (__all_sync(0xffffffffu, bin == b0)) {
        if (b0 == run.bin) {
            run.cnt += 32u;
            return;
        }
        if ((threadIdx.x & 31) == 0 && run.bin > 0) atomicAdd(h + (run.bin - 1), run.cnt);
        run.bin = b0;
        run.cnt = 32u;
    } else if (bin > 0) {
        atomicAdd(h + (bin - 1), 1u);
    }
}
__device__ __forceinline__ void hist_flush(unsigned *h, const WarpRun &run)
{
    if ((threadIdx.x & 31) == 0 && run.bin > 0) atomicAdd(h + (run.bin - 1), run.cnt);
}

// HB, HD: the lattice has biquadratic / DM couplings, as compile-time flags so
// the neighbour loop carries no tests for absent terms.  GEN: a lattice
// without the parity-class structure (odd or open), see ResidentTables.  RS:
// the stencil rows are in shared memory (else read from global memory, for
// stencils whose rows do not fit beside the spins).  CL: clusters of more than
// one CTA.  S: sites of a colour pass a thread updates at a time.  PP: the first
// nt_update threads update one site of a colour each, the last warp folds the
// measurements, and the warps between make the next pass's trial spins
// meanwhile.
//
// What bounds it, and why it is written this way.  The spins live in shared
// memory, so HBM is idle.  An update issues 165 thread instructions plus ~10 a
// neighbour (measured: 253 with 6 neighbours, 448 with 26) and the shared
// memory serves 3 wavefronts a neighbour per 32 updates; 16 warps per SM have
// to hide every latency between them:
//  * a neighbour's position is own position + a byte offset from the site's
//    stencil row in shared memory.  Rows are shared by all sites of one
//    class and one side of the lattice's edges (bcc 24^3 on 2 CTAs: 128 rows
//    for 13,824 sites), so they stay in shared memory; the per-site table of
//    neighbour ids they replace streamed from L2 (28 words per site and
//    sweep) with its latency in front of every gather;
//  * entries without biquadratic or DM coupling skip that arithmetic (SC J1 +
//    J2 with biquadratic on J1: 6 of 18 entries have it);
//  * a site's index arithmetic is one 8-byte descriptor (position, row,
//    reference site), loaded one step ahead;
//  * the random numbers and the trial spin of a thread's next site need no
//    neighbour, so they are computed before the barrier that ends a colour
//    pass (between arrive and wait where it is a cluster barrier), and a
//    lattice with few sites runs with as few threads as one site each needs,
//    its measurements folded by a warp that may have none;
//  * S = 2: two sites' instruction streams interleave (SC 48^3 x 32 on 6 CTAs,
//    biquadratic and DM, ten sweeps and measurements: 1053 us with one, 938);
//  * !RS: the rows come out of L2, so they lie quad by quad (the lanes of a
//    warp have rows that follow one another) and, with one site a thread,
//    several quads ahead are in flight.  us for two sweeps and a measurement,
//    a table of neighbour ids / rows one after another / so: fcc with 6 shells
//    12^3 x 40 307 / 375 / 206, 7 shells 10^3 x 40 421 / - / 233, 14^3 x 20 on 2
//    CTAs 623 / - / 584, 2 shells 16^3 x 152 (two sites) 121 / 146 / 115;
//  * PP: where a colour leaves warps of a CTA idle, a pass is one chain of
//    dependent instructions through a few warps (64 spins: 32 sites, one
//    warp).  The trial spins depend on no neighbour, and on the old spin only
//    for cone moves, which no other colour's pass writes: other warps make them
//    a pass ahead.  The fold of a measurement, an FP64 chain longer than a
//    pass, has a warp of its own, which meets the others at the measurements
//    only (64 spins: 5.3 us with the fold in a warp of the passes, 2.3 us so).
// Measured on a GB300, sweeps and measurements of a swap interval, with a table
// of neighbour ids and now: bcc 24^3 x 48 (2 CTAs) 812 -> 660 us, SC 48^3 frustrated x 32 (12
// CTAs) 2530 -> 1810 us, SC 14^3 x 32 with cone moves (2 CTAs, 50 sweeps) 617 ->
// 470 us; two sweeps and a measurement of 64 spins 9.6 -> 2.3 us, of a
// pyrochlore of 256 with order parameter 18.8 -> 7.2 us; general lattices in
// the ELL kernel's place, two sweeps and a measurement of an open 21 x 21 x 7 x
// 60 73 -> 13.6 us, of bcc 25^3 x 16 377 -> 159 us.
// Each thread updates the items tid, tid + NT, ... of a colour in that order
// and adds their dE and dM in that order, in FP32 within a sweep (GEN: every
// term in three floats), whatever the other choices.
template <int S, bool HB, bool HD, bool GEN, bool RS, bool CL, bool PP>
__global__ void __launch_bounds__(kClusterThreads, 1) k_sweep_cluster(const ClusterArgs a)
{
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int csize = (int)cluster.num_blocks();
    const int r = blockIdx.x / csize;  // replica of this cluster
    const int NT = (int)blockDim.x, tid = (int)threadIdx.x;
    const int NU = PP ? a.nt_update : NT;   // threads that update sites
    const int NW = PP ? NT - 32 : NT;       // threads of the passes; PP: the last warp only folds
    const int warp = tid >> 5, lane = tid & 31, nwarps = NT >> 5;
    const int n_local = rank < a.nA ? a.n_big : a.n_small;
    // sites of the ranks before this one
    const size_t site0 = (size_t)rank * a.n_big - (size_t)max(0, rank - a.nA) * (a.n_big - a.n_small);
    const unsigned long long sweep_base = a.sweep_base + (a.ctr ? a.ctr[0] : 0ull);
    const long long meas_base = a.meas_base + (a.ctr ? (long long)a.ctr[2] : 0ll);

    // shared memory: this rank's tables | histograms P(M) [, P(OP), P(SM)] |
    // reduction scratch | spins (smem_words is a multiple of 4, so every part
    // stays 16-byte aligned)
    extern __shared__ __align__(16) unsigned char smem[];
    const ResidentHeader *st = reinterpret_cast<const ResidentHeader *>(smem);
    const uint32_t *gblob = a.blob + (size_t)rank * a.blob_words;
    const uint32_t cpl = (uint32_t)__cvta_generic_to_shared(smem) + (uint32_t)sizeof(ResidentHeader);   // coupling lists
    const uint32_t rows_s = (uint32_t)__cvta_generic_to_shared(smem) + 4u * (uint32_t)a.rows_off;       // RS
    const uint32_t *rows_g = gblob + a.rows_off;                                                        // !RS
    unsigned int *hist = reinterpret_cast<unsigned int *>(smem) + a.smem_words;
    const int nhist = a.obs ? 3 : 1;
    // reduction scratch: [0, 64) warp partials of dE and dM (float pairs, GEN:
    // doubles), [64, 96) of the observables (GEN: [64, 128), doubles), or [0,
    // 112) FP64 at the end; [128, 144) a CTA's totals of a measurement, two
    // buffers by the measurement's parity; [144, 149) the CTA's end-of-launch
    // totals
    double *red = reinterpret_cast<double *>(hist + ((nhist * a.nf + 3) & ~3));
    // the slot's accumulators, kept by rank 0 for the launch (the slot of a
    // replica does not change inside a launch): data, obs data, binning
    // levels, binning sums and variances of E/N, |m| and of |OP|, |SM|
    double *acc = red + kClusterRedDoubles;
    double *c_data = acc, *c_odata = acc + 6;
    int *c_lev = reinterpret_cast<int *>(acc + 12);
    double *c_ls = acc + 12 + kClusterMaxLev / 2, *c_bn = c_ls + 2 * kClusterMaxLev;
    double *c_ols = c_bn + 2 * kClusterMaxLev, *c_obn = c_ols + 2 * kClusterMaxLev;
    float *s3 = reinterpret_cast<float *>(acc + kClusterAccDoubles);   // [n_local][x, y, z]
    const uint32_t s3u = (uint32_t)__cvta_generic_to_shared(s3);

    // ---- set-up: tables and own spins --------------------------------------
    for (int i = tid; i < (a.smem_words >> 2); i += NT)
        reinterpret_cast<uint4 *>(smem)[i] = __ldg(reinterpret_cast<const uint4 *>(gblob) + i);
    for (int i = tid; i < nhist * a.nf; i += NT) hist[i] = 0u;
    // this CTA's slab: one contiguous block of 3 n_local floats, or gathered
    // from the spin arrays
    float *slab = a.slab ? a.slab + ((size_t)r * a.N + site0) * 3 : nullptr;
    if (slab) {
        for (int i = tid; i < 3 * n_local; i += NT) s3[i] = slab[i];
    } else {
        for (int l = tid; l < n_local; l += NT) {
            const size_t g = (size_t)__ldg(a.loc2p + site0 + l) * a.R + r;
            s3[3 * l] = a.sx[g]; s3[3 * l + 1] = a.sy[g]; s3[3 * l + 2] = a.sz[g];
        }
    }
    if constexpr (RS) {
        // the rows' words of peers' spins become offsets in the cluster's
        // shared-memory window, so that a gather there is one addition too
        if (CL) {
            __syncthreads();
            uint32_t *rw = reinterpret_cast<uint32_t *>(smem) + a.rows_off;
            for (int k = tid * a.rstride; k < a.smem_words - a.rows_off; k += NT * a.rstride) {
                const uint32_t far = rw[k + 2];
                for (int e = 0; far != 0u && e < a.rstride - 4; ++e)
                    if ((far >> min(e >> 2, 31)) & 1u) {
                        const uint32_t w = rw[k + 4 + e], q = w & 0xffu;
                        rw[k + 4 + e] = (uint32_t)((int)w >> 8) + (q ? mapa_shared(s3u, q - 1u) - s3u : 0u);
                    }
            }
        }
    }
    const int temp = a.temp_of[r];
    const bool cache = a.measure && a.nlev <= kClusterMaxLev;
    if (rank == 0 && cache) {
        const int nl2 = 2 * a.nlev;
        for (int i = tid; i < 6; i += NT) {
            c_data[i] = a.data[6 * temp + i];
            c_odata[i] = a.obs ? a.obs_data[6 * temp + i] : 0.0;
        }
        for (int i = tid; i < a.nlev; i += NT) c_lev[i] = a.levels[i];
        for (int i = tid; i < nl2; i += NT) {
            c_ls[i] = a.lsum[(size_t)temp * nl2 + i];
            c_bn[i] = a.binning[(size_t)temp * nl2 + i];
            c_ols[i] = a.obs ? a.obs_lsum[(size_t)temp * nl2 + i] : 0.0;
            c_obn[i] = a.obs ? a.obs_bin[(size_t)temp * nl2 + i] : 0.0;
        }
    }
    cluster.sync();

    const float beta = a.beta[temp];
    // sums since the last measurement: of the per-sweep FP32 sums as float
    // pairs, on general lattices of every term in three floats (k_sweep_ell
    // adds them in FP64)
    using Acc = std::conditional_t<GEN, F3, F2>;
    Acc accE{}, accX{}, accY{}, accZ{};
    unsigned long long nrej = 0;
    const float pm_scale = (float)((double)(a.nf - 1) / (a.m_max - a.m_min));
    // replica totals, held by lane 0 of the folding warp of rank 0
    const int fold_warp = nwarps - 1;
    double e_run = 0.0, m_run[3] = {0.0, 0.0, 0.0};
    if (rank == 0 && warp == fold_warp && lane == 0) {
        e_run = a.e_run[r];
        m_run[0] = a.m_run[3 * r]; m_run[1] = a.m_run[3 * r + 1]; m_run[2] = a.m_run[3 * r + 2];
    }

    // A site about to be updated: the address of its spin, its stencil row's
    // header and the address (RS) or word offset of the row's entries, the old
    // spin, the trial spin and the test's uniform.
    struct Site {
        uint32_t own, row;
        uint4 h;
        float ox, oy, oz, nx, ny, nz;
        uint32_t u;
        bool act;
    };
    const uint2 *desc = a.desc + site0;
    const int nc = st->ncolour, wbase = 32 * warp;
    auto row_quad = [&](uint32_t row, int e) -> uint4 {
        return RS ? ld_shared_u4(row + 4u * (uint32_t)e)
                  : __ldg(reinterpret_cast<const uint4 *>(rows_g + row + (uint32_t)(e >> 2) * (uint32_t)a.rows4));
    };
    auto row_pair = [&](uint32_t row, int e) -> uint2 { return ld_shared_u2(row + 4u * (uint32_t)e); };   // RS
    // words of a row in global memory as offsets: (byte offset << 8) | (owner
    // rank + 1, or 0) in the quads the row marks
    auto decode = [&](uint32_t (&w)[4], int n, int e, uint32_t far) {
        if ((far >> min(e >> 2, 31)) & 1u)
            for (int i = 0; i < n; ++i) {
                const uint32_t q = w[i] & 0xffu;
                w[i] = (uint32_t)((int)w[i] >> 8) + (q ? mapa_shared(s3u, q - 1u) - s3u : 0u);
            }
    };
    // row and atom of a descriptor
    auto row_of = [](uint2 d) -> uint32_t { return RS ? d.x >> 18 : (d.x >> 18) | (d.y >> 31) << 14; };
    auto atom_of = [](uint2 d) -> uint32_t { return RS ? d.y >> 28 : (d.y >> 28) & 7u; };
    // PP: trial spins and uniforms of a pass, [parity of the pass][item]
    const uint32_t trials = (s3u + 12u * (uint32_t)a.n_big + 15u) & ~15u;
    // ... and the updating threads' sums of a measurement, [parity][thread][8]
    // (GEN: [12])
    constexpr uint32_t kHandOver = GEN ? 48u : 32u;
    const uint32_t parts = trials + 32u * (uint32_t)NU;
    // What the updating thread itself reads of its next site.
    auto locate = [&](Site &s, uint2 d, bool act) {
        s.own = s3u + (d.x & 0x3ffffu);
        const uint32_t rw = RS ? rows_s + row_of(d) * (4u * (uint32_t)a.rstride) : row_of(d) * 4u;
        s.h = row_quad(rw, 0);
        s.row = rw + (RS ? 16u : (uint32_t)a.rows4);
        s.act = act;
        ld_shared3(s.own, s.ox, s.oy, s.oz);
    };
    // PP, the helping warps: the trials of all items of colour c, sweep `sweep`.
    auto make_trials = [&](int c, unsigned long long sweep, int buf) {
        const int i0 = st->colour_start[c], n = st->colour_start[c + 1] - i0;
        for (int k = tid - NU; k < n; k += NW - NU) {
            const uint2 d = __ldg(desc + i0 + k);
            const Philox4 x = philox4x32_10(d.y & 0xfffffffu, (uint32_t)r, (uint32_t)sweep, (uint32_t)(sweep >> 32), a.rk);
            float ox = 0.f, oy = 0.f, oz = 0.f, nx, ny, nz;
            if (a.mode != 0) ld_shared3(s3u + (d.x & 0x3ffffu), ox, oy, oz);
            if (a.mode == 0) trial_spin(0, a.tilt, st->mag[atom_of(d)], ox, oy, oz, x.x, x.y, nx, ny, nz);
            else trial_spin(1, a.tilt, st->mag[atom_of(d)], ox, oy, oz, x.x, x.y, nx, ny, nz);
            st_shared4(trials + 16u * (uint32_t)(buf * NU + k), nx, ny, nz, __uint_as_float(x.z));
        }
    };
    // Old spin, random numbers and trial spin: everything of an update that
    // does not depend on the neighbours.  The old spin is this thread's own
    // to write (a site is always updated by the same thread), so it may be
    // read before the barrier that ends the previous colour pass.
    auto prepare = [&](Site (&o)[S], const uint2 (&d)[S], const bool (&act)[S], unsigned long long sweep) {
        Philox4 x[S];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            Site &s = o[k];
            locate(s, d[k], act[k]);
            x[k] = philox4x32_10(d[k].y & 0xfffffffu, (uint32_t)r, (uint32_t)sweep, (uint32_t)(sweep >> 32), a.rk);
            s.u = x[k].z;
        }
        if (a.mode == 0) {
#pragma unroll
            for (int k = 0; k < S; ++k)
                trial_spin(0, a.tilt, st->mag[atom_of(d[k])], o[k].ox, o[k].oy, o[k].oz, x[k].x, x[k].y, o[k].nx, o[k].ny, o[k].nz);
        } else {
#pragma unroll
            for (int k = 0; k < S; ++k)
                trial_spin(1, a.tilt, st->mag[atom_of(d[k])], o[k].ox, o[k].oy, o[k].oz, x[k].x, x[k].y, o[k].nx, o[k].ny, o[k].nz);
        }
    };

    // Metropolis update of M prepared sites whose rows have the same entry
    // counts, their instruction streams interleaved: local field from the
    // stencil row, energy change, test (metropolis, get_quant.F90:52-182,
    // delta_energy_get :264-337), each in the arithmetic and order of
    // k_sweep_ell
    auto update = [&](auto mc, const Site *s, float &fE, float &fX, float &fY, float &fZ, unsigned int &rej) {
        constexpr int M = decltype(mc)::value;
        const int cnt = (int)(s[0].h.x & 0xffffu), nr = (int)(s[0].h.x >> 16);
        uint32_t cJ[M], cR[M];
        float g[M][3], q[M][6];
#pragma unroll
        for (int k = 0; k < M; ++k) {
            cJ[k] = cpl + 4u * s[k].h.y;
            cR[k] = cJ[k] + 4u * (uint32_t)a.jwords;
#pragma unroll
            for (int c = 0; c < 3; ++c) g[k][c] = 0.f;
#pragma unroll
            for (int c = 0; c < 6; ++c) q[k][c] = 0.f;
        }
        auto exchange = [&](int k, float nJ, const float (&t)[3]) {
#pragma unroll
            for (int c = 0; c < 3; ++c) g[k][c] = fmaf(nJ, t[c], g[k][c]);
        };
        auto rich = [&](int k, float4 c, const float (&t)[3]) {
            if (HB) bq_form(c.x, t[0], t[1], t[2], q[k][0], q[k][1], q[k][2], q[k][3], q[k][4], q[k][5]);
            if (HD) dm_field(c.y, c.z, c.w, t[0], t[1], t[2], g[k][0], g[k][1], g[k][2]);
        };
        // the spin at word w of site k's row.  In a cluster every spin is read
        // through its shared-memory window, a CTA's own too: as fast there as
        // through the CTA's own window, where telling the two apart cost more
        // (bcc 16^3 x 32 on 2 CTAs: 19.3 us per sweep; 23.7 with a test per
        // pair of entries in the warps that have a peer's spin)
        auto spin = [&](int k, uint32_t w, float (&t)[3]) {
            if constexpr (CL) ld_cluster3(s[k].own + w, t[0], t[1], t[2]);
            else ld_shared3(s[k].own + w, t[0], t[1], t[2]);
        };
        // words of entries e .. e + 3 / e, e + 1 of site k as offsets
        auto offsets = [&](int k, int e, uint32_t (&w)[4]) {
            const uint4 v = row_quad(s[k].row, e);
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        };
        auto offsets2 = [&](int k, int e, uint32_t (&w)[4]) {
            const uint2 v = row_pair(s[k].row, e);
            w[0] = v.x; w[1] = v.y;
        };
        int e = 0;
        if constexpr (!RS) {
            // Rows out of L2: with one site a thread the words of the next Q
            // quads are loaded before the spins of these are read; in a
            // cluster the spins of W quads, some out of a peer's shared memory,
            // before they are used.  The last quad's padding is the site
            // itself without couplings.
            auto walk = [&](auto qc, int end, auto &&use) {
                constexpr int most = decltype(qc)::value;
                constexpr int Q = S > 1 ? 1 : CL ? 2 : most, W = CL && S == 1 && most == 4 ? 2 : 1;
                uint4 next[M][Q];
                auto fetch = [&](int at) {
#pragma unroll
                    for (int k = 0; k < M; ++k)
#pragma unroll
                        for (int j = 0; j < Q; ++j)
                            if (at + 4 * j < end) next[k][j] = row_quad(s[k].row, at + 4 * j);
                };
                if (S == 1) fetch(e);
#pragma unroll 1
                for (; e < end; e += 4 * Q) {
                    if (S > 1) fetch(e);
                    uint4 now[M][Q];
#pragma unroll
                    for (int k = 0; k < M; ++k)
#pragma unroll
                        for (int j = 0; j < Q; ++j) now[k][j] = next[k][j];
                    if (S == 1) fetch(e + 4 * Q);
#pragma unroll
                    for (int j = 0; j < Q; j += W) {
                        float t[W][M][4][3];
#pragma unroll
                        for (int i = 0; i < W; ++i) {
                            const int q = e + 4 * (j + i);
                            if (q >= end) break;
#pragma unroll
                            for (int k = 0; k < M; ++k) {
                                const uint4 v = now[k][j + i];
                                uint32_t w[4] = {v.x, v.y, v.z, v.w};
                                if constexpr (CL) decode(w, 4, q, s[k].h.z);
#pragma unroll
                                for (int c = 0; c < 4; ++c) spin(k, w[c], t[i][k][c]);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < W; ++i) {
                            const int q = e + 4 * (j + i);
                            if (q < end) use(q, t[i]);
                        }
                    }
                }
            };
            if (HB || HD) {
                walk(std::integral_constant<int, 2>{}, nr, [&](int q, const float (&t)[M][4][3]) {
#pragma unroll
                    for (int k = 0; k < M; ++k) {
                        const float4 J = ld_shared_f4(cJ[k] + 4u * (uint32_t)q);
                        const uint32_t c = cR[k] + 16u * (uint32_t)q;
                        exchange(k, J.x, t[k][0]); rich(k, ld_shared_f4(c), t[k][0]);
                        exchange(k, J.y, t[k][1]); rich(k, ld_shared_f4(c + 16u), t[k][1]);
                        if (q + 2 < nr) {
                            exchange(k, J.z, t[k][2]); rich(k, ld_shared_f4(c + 32u), t[k][2]);
                            exchange(k, J.w, t[k][3]); rich(k, ld_shared_f4(c + 48u), t[k][3]);
                        }
                    }
                });
                e = (nr + 3) & ~3;
            }
            walk(std::integral_constant<int, 4>{}, cnt, [&](int q, const float (&t)[M][4][3]) {
#pragma unroll
                for (int k = 0; k < M; ++k) {
                    const float4 J = ld_shared_f4(cJ[k] + 4u * (uint32_t)q);
                    exchange(k, J.x, t[k][0]); exchange(k, J.y, t[k][1]);
                    exchange(k, J.z, t[k][2]); exchange(k, J.w, t[k][3]);
                }
            });
        } else {
            if (HB || HD) {
#pragma unroll(M == 1 ? 3 : 1)
                for (; e < nr; e += 2) {
                    float t[M][2][3];
#pragma unroll
                    for (int k = 0; k < M; ++k) {
                        uint32_t w[4];
                        offsets2(k, e, w);
                        spin(k, w[0], t[k][0]); spin(k, w[1], t[k][1]);
                    }
#pragma unroll
                    for (int k = 0; k < M; ++k) {
                        const float2 J = ld_shared_f2(cJ[k] + 4u * (uint32_t)e);
                        exchange(k, J.x, t[k][0]); rich(k, ld_shared_f4(cR[k] + 16u * (uint32_t)e), t[k][0]);
                        exchange(k, J.y, t[k][1]); rich(k, ld_shared_f4(cR[k] + 16u * (uint32_t)(e + 1)), t[k][1]);
                    }
                }
                e = (e + 3) & ~3;
            }
#pragma unroll 2
            for (; e + 4 <= cnt; e += 4) {
                float t[M][4][3];
#pragma unroll
                for (int k = 0; k < M; ++k) {
                    uint32_t w[4];
                    offsets(k, e, w);
                    spin(k, w[0], t[k][0]); spin(k, w[1], t[k][1]); spin(k, w[2], t[k][2]); spin(k, w[3], t[k][3]);
                }
#pragma unroll
                for (int k = 0; k < M; ++k) {
                    const float4 J = ld_shared_f4(cJ[k] + 4u * (uint32_t)e);
                    exchange(k, J.x, t[k][0]); exchange(k, J.y, t[k][1]);
                    exchange(k, J.z, t[k][2]); exchange(k, J.w, t[k][3]);
                }
            }
            if (e < cnt) {
                float t[M][2][3];
#pragma unroll
                for (int k = 0; k < M; ++k) {
                    uint32_t w[4];
                    offsets2(k, e, w);
                    spin(k, w[0], t[k][0]); spin(k, w[1], t[k][1]);
                }
#pragma unroll
                for (int k = 0; k < M; ++k) {
                    const float2 J = ld_shared_f2(cJ[k] + 4u * (uint32_t)e);
                    exchange(k, J.x, t[k][0]); exchange(k, J.y, t[k][1]);
                }
            }
        }
        float de[M];
#pragma unroll
        for (int k = 0; k < M; ++k) {
            if (a.has_si) si_form(st->si[s[k].h.w], q[k][0], q[k][1], q[k][2], q[k][3], q[k][4], q[k][5]);
            if (a.has_f) {
                const float4 f = st->fld[s[k].h.w];
                g[k][0] = __fadd_rn(g[k][0], f.x); g[k][1] = __fadd_rn(g[k][1], f.y); g[k][2] = __fadd_rn(g[k][2], f.z);
            }
            de[k] = delta_energy(HB || a.has_si, g[k][0], g[k][1], g[k][2], q[k][0], q[k][1], q[k][2], q[k][3], q[k][4],
                                 q[k][5], s[k].ox, s[k].oy, s[k].oz, s[k].nx, s[k].ny, s[k].nz);
        }
#pragma unroll
        for (int k = 0; k < M; ++k)
            if (s[k].act) {
                if (metropolis_accept(beta, de[k], s[k].u)) {
                    st_shared3(s[k].own, s[k].nx, s[k].ny, s[k].nz);
                    const float dx = s[k].nx - s[k].ox, dy = s[k].ny - s[k].oy, dz = s[k].nz - s[k].oz;
                    if constexpr (GEN) {
                        accE = f3_add(accE, de[k]);
                        accX = f3_add(accX, dx); accY = f3_add(accY, dy); accZ = f3_add(accZ, dz);
                    } else {
                        fE += de[k];
                        fX += dx; fY += dy; fZ += dz;
                    }
                } else {
                    ++rej;
                }
            }
    };

    // Rank 0's last warp folds measurement m (the CTAs' totals in buffer m & 1)
    // into the replica totals and the accumulators of mcarlo.F90:536-590 for
    // this temperature slot: lane 0 the sums, one binning level per lane.  The
    // last warp, because small lattices give it the fewest sites (or none), and
    // the fold's FP64 chain then runs beside the other warps' updates.
    auto fold_measurement = [&](const int m) {
        // lane 0 folds the CTAs' sums into the replica totals and the
        // accumulators of mcarlo.F90:536-590 for this temperature
        // slot; the binning levels, independent of one another, go
        // one per lane
        const double rn_inv = a.rn_inv;
        const long long step = meas_base + m + 1;
        double e = 0.0, am = 0.0, aop = 0.0, asm_ = 0.0;
        if (lane == 0) {
            double d4[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int q = 0; q < csize; ++q) {
                const double *pr = cluster.map_shared_rank(red, q);
#pragma unroll
                for (int c = 0; c < 8; ++c) d4[c] += pr[128 + 8 * (m & 1) + c];
            }
            e_run += d4[0];
            m_run[0] += d4[1]; m_run[1] += d4[2]; m_run[2] += d4[3];
            e = e_run;
            const double mx = m_run[0] * rn_inv, my = m_run[1] * rn_inv, mz = m_run[2] * rn_inv;
            const double m2 = mx * mx + my * my + mz * mz;
            const double ee = e * e;
            am = sqrt(m2);
            double *d = cache ? c_data : a.data + 6 * temp;
            d[0] += e; d[1] += ee; d[2] += ee * ee;
            d[3] += am; d[4] += m2; d[5] += m2 * m2;
            if (a.series) {
                double *o = a.series + (((step - 1) % a.series_cap) * a.R + temp) * 2;
                o[0] = e; o[1] = am;
            }
            // orderparam_get / staggered_get (mcarlo.F90:553-568)
            if (a.obs) {
                double *od = cache ? c_odata : a.obs_data + 6 * temp;
                if (a.obs & 1) {
                    const double op = d4[4] * rn_inv;
                    const double o2 = op * op;
                    aop = sqrt(o2);
                    od[0] += aop; od[1] += o2; od[2] += o2 * o2;
                }
                if (a.obs & 2) {
                    const double qx = d4[5] * rn_inv, qy = d4[6] * rn_inv, qz = d4[7] * rn_inv;
                    const double q2 = qx * qx + qy * qy + qz * qz;
                    asm_ = sqrt(q2);
                    od[3] += asm_; od[4] += q2; od[5] += q2 * q2;
                }
            }
        }
        if (a.nlev > 0) {
            e = __shfl_sync(0xffffffffu, e, 0);
            am = __shfl_sync(0xffffffffu, am, 0);
            aop = __shfl_sync(0xffffffffu, aop, 0);
            asm_ = __shfl_sync(0xffffffffu, asm_, 0);
        }
        for (int lv = lane; lv < a.nlev; lv += 32) {
            const size_t g2 = ((size_t)temp * a.nlev + lv) * 2;
            double *ls = cache ? c_ls + 2 * lv : a.lsum + g2;
            double *bn = cache ? c_bn + 2 * lv : a.binning + g2;
            double *ols = !a.obs ? nullptr : (cache ? c_ols + 2 * lv : a.obs_lsum + g2);
            double *obn = !a.obs ? nullptr : (cache ? c_obn + 2 * lv : a.obs_bin + g2);
            ls[0] += e * rn_inv;
            ls[1] += am;
            if (ols) { ols[0] += aop; ols[1] += asm_; }
            const int lev = cache ? c_lev[lv] : a.levels[lv];
            const long long blk = 1LL << lev;
            if ((step & (blk - 1)) == 0) {
                // 1/2^n is exact, so the product equals the division
                const double inv_div = ldexp(1.0, -(a.pt_quirk ? lv + 1 : lev));
                for (int c = 0; c < 2; ++c) {
                    const double v2 = ls[c] * inv_div;
                    bn[c] += v2 * v2;
                    ls[c] = 0.0;
                    if (ols) {
                        const double w2 = ols[c] * inv_div;
                        obn[c] += w2 * w2;
                        ols[c] = 0.0;
                    }
                }
            }
        }
    };
    // Warp partials of the observables' sums, [virtual warp][4] floats (GEN:
    // doubles); PP: two buffers by the measurement's parity, in the place
    // of the warp partials of dE and dM
    auto obs_scratch = [&](int b) -> float * {
        if constexpr (PP) return reinterpret_cast<float *>(red + 64 * b);
        else return reinterpret_cast<float *>(red + 64);
    };
    // GEN, one warp: the sums of n <= 16 warps' doubles [warp][4] into tot[4].
    auto fold_warps = [&](const double *part, int n, double *tot) {
        const int c = lane & 3, w = lane >> 2;
        double x = (w < n ? part[4 * w + c] : 0.0) + (w + 8 < n ? part[4 * (w + 8) + c] : 0.0);
        for (int o = 16; o >= 4; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane < 4) tot[lane] = x;
    };
    // One warp: their totals.
    auto fold_obs = [&](int b, double *tot) {
        const float *redo = obs_scratch(b);
        const int nvw = a.nt_sum >> 5;
        if constexpr (GEN) {
            fold_warps(reinterpret_cast<const double *>(redo), nvw, tot + 4);
            return;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float x = lane < nvw ? redo[4 * lane + c] : 0.f;
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) tot[4 + c] = (double)x;
        }
    };
    int pending = -1;   // measurement whose totals wait for rank 0's fold

    // cells of this CTA, atom at of cell cl at local site at * ncells + cl
    const int ncells = n_local / a.na;

    // the next site to prepare in the thread's sequence of (sweep, colour,
    // round): the warp's first item pw of colour pc, which ends at pe, and its
    // descriptor; lanes past the end take item 0 of the rank and do not commit
    int pc = 0, pw = wbase, pe = st->colour_start[1];
    unsigned long long psweep = sweep_base;
    auto step = [&]() {
        pw += S * NU;
        if (pw >= pe) {
            if (++pc == nc) { pc = 0; ++psweep; }
            pw = st->colour_start[pc] + wbase;
            pe = st->colour_start[pc + 1];
        }
    };
    auto item = [&](uint2 (&d)[S], bool (&act)[S]) {
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const int i = pw + k * NU + lane;
            act[k] = i < pe;
            d[k] = __ldg(desc + (act[k] ? i : 0));
        }
    };
    bool nact[S];
    uint2 nd[S];
    Site cur[S];
    if constexpr (PP) {
        static_assert(!PP || (S == 1 && !CL && RS), "one site per thread, one CTA");
        if (tid < NU) {
            item(nd, nact);
            locate(cur[0], nd[0], nact[0]);
        } else if (tid < NW) {
            make_trials(0, psweep, 0);
        }
        step();
        if (tid < NU) item(nd, nact);
        __syncthreads();
    } else {
        item(nd, nact);
        prepare(cur, nd, nact, psweep);
        step();
        item(nd, nact);
    }
    int tbuf = 0;

    // PP, the last warp: the measurements' sums as the others hand them over, in
    // two buffers (named barriers 2, 3: full, 4, 5: free again), so that the
    // reduction and the FP64 chain of a fold run beside the following passes
    if (PP && warp == fold_warp) {
        for (int m = 0; a.measure && m < a.n_meas; ++m) {
            const int b = m & 1;
            bar_sync(2 + b, NT);
            double *tot = red + 128 + 8 * b;
            if constexpr (GEN) {
                F3 p4[4] = {};
                for (int k = lane; k < NU; k += 32) {
                    const uint32_t at = parts + kHandOver * (uint32_t)(b * NU + k);
                    const float4 u = ld_shared_f4(at), v = ld_shared_f4(at + 16u), w = ld_shared_f4(at + 32u);
                    p4[0] = f3_add(p4[0], F3{u.x, u.y, u.z}); p4[1] = f3_add(p4[1], F3{u.w, v.x, v.y});
                    p4[2] = f3_add(p4[2], F3{v.z, v.w, w.x}); p4[3] = f3_add(p4[3], F3{w.y, w.z, w.w});
                }
                const double x = f3_to_double(f3_warp_sum4(p4));
                if ((lane & 7) == 0) tot[lane >> 3] = x;
            } else {
                F2 p4[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) p4[c] = F2{0.f, 0.f};
                for (int k = lane; k < NU; k += 32) {
                    const uint32_t at = parts + kHandOver * (uint32_t)(b * NU + k);
                    const float4 u = ld_shared_f4(at), v = ld_shared_f4(at + 16u);
                    p4[0] = f2_add(p4[0], F2{u.x, u.y}); p4[1] = f2_add(p4[1], F2{u.z, u.w});
                    p4[2] = f2_add(p4[2], F2{v.x, v.y}); p4[3] = f2_add(p4[3], F2{v.z, v.w});
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    for (int o = 16; o > 0; o >>= 1) p4[c] = f2_add(p4[c], f2_shfl_down(p4[c], o));
                    if (lane == 0) tot[c] = f2_to_double(p4[c]);
                }
            }
            if (a.obs) fold_obs(b, tot);
            __syncwarp();
            fold_measurement(m);
            if (m + 2 < a.n_meas) bar_arrive(4 + b, NT);   // waited for by measurement m + 2
        }
    }
    for (int m = 0; m < (PP && warp == fold_warp ? 0 : a.n_meas); ++m) {
        unsigned int rej = 0;
        for (int sm = 0; sm < a.steps_measure; ++sm) {
            // FP32 sums of one sweep, added to the float pairs after it
            float fE = 0.f, fX = 0.f, fY = 0.f, fZ = 0.f;
            for (int c = 0; c < nc; ++c) {
                if constexpr (PP) {
                    if (tid < NU) {
                        if (st->colour_start[c] + wbase < st->colour_start[c + 1]) {
                            const float4 tr = ld_shared_f4(trials + 16u * (uint32_t)(tbuf * NU + tid));
                            cur[0].nx = tr.x; cur[0].ny = tr.y; cur[0].nz = tr.z;
                            cur[0].u = __float_as_uint(tr.w);
                            update(std::integral_constant<int, 1>{}, cur, fE, fX, fY, fZ, rej);
                        }
                        locate(cur[0], nd[0], nact[0]);
                        step();
                        item(nd, nact);
                    } else {
                        make_trials(pc, psweep, tbuf ^ 1);
                        step();
                    }
                    tbuf ^= 1;
                } else {
                    // at least one round, without an update in a warp that has no
                    // site of this colour
                    int w0 = st->colour_start[c] + wbase;
                    const int e0 = st->colour_start[c + 1];
                    const bool has = w0 < e0;
                    bool last;
                    do {
                        if (has) {
                            const std::integral_constant<int, 1> one{};
                            if constexpr (S == 1) {
                                update(one, cur, fE, fX, fY, fZ, rej);
                            } else {
                                // the second site exists for some lane, and the
                                // rows of both have the same entry counts
                                const bool more = w0 + NT < e0;
                                if (more && __all_sync(0xffffffffu, cur[0].h.x == cur[1].h.x)) {
                                    update(std::integral_constant<int, 2>{}, cur, fE, fX, fY, fZ, rej);
                                } else {
                                    update(one, cur, fE, fX, fY, fZ, rej);
                                    if (more) update(one, cur + 1, fE, fX, fY, fZ, rej);
                                }
                            }
                        }
                        w0 += S * NT;
                        last = w0 >= e0;
                        if (CL && last) cluster_arrive();
                        prepare(cur, nd, nact, psweep);
                        step();
                        item(nd, nact);
                    } while (!last);
                }
                if constexpr (CL) cluster_wait();
                else if constexpr (PP) bar_sync(1, NW);
                else __syncthreads();
                if (pending >= 0) {
                    if (rank == 0 && warp == fold_warp) fold_measurement(pending);
                    pending = -1;
                }
            }
            if constexpr (!GEN) {
                accE = f2_add(accE, fE); accX = f2_add(accX, fX); accY = f2_add(accY, fY); accZ = f2_add(accZ, fZ);
            }
        }
        nrej += rej;
        if (!a.measure) continue;
        if (!PP && a.steps_measure == 0) {
            // no colour pass, so no barrier, since the last measurement
            cluster.sync();
            if (pending >= 0 && rank == 0 && warp == fold_warp) fold_measurement(pending);
        }
        // ---- measurement: cluster-wide sums of dE and dM (and, with the
        // optional measurements, of s.a and c s over the slab) ---------------
        {
            // float pairs within the CTA for dE and dM (FP64 is a slow pipe
            // on this GPU), FP64 across CTAs and into the running totals; GEN:
            // three floats within a warp, FP64 across warps
            Acc p4[4] = {accE, accX, accY, accZ};
            accE = accX = accY = accZ = Acc{};
            float *redf = reinterpret_cast<float *>(red);          // [warp][4 pairs], GEN: [warp][4] doubles
            float *redo = obs_scratch(m & 1);
            if constexpr (PP) {
                if (m >= 2) bar_sync(4 + (m & 1), NT);   // the fold of m - 2 has read this buffer
                if (tid < NU) {
                    const uint32_t at = parts + kHandOver * (uint32_t)((m & 1) * NU + tid);
                    if constexpr (GEN) {
                        st_shared4(at, p4[0].hi, p4[0].mid, p4[0].lo, p4[1].hi);
                        st_shared4(at + 16u, p4[1].mid, p4[1].lo, p4[2].hi, p4[2].mid);
                        st_shared4(at + 32u, p4[2].lo, p4[3].hi, p4[3].mid, p4[3].lo);
                    } else {
                        st_shared4(at, p4[0].hi, p4[0].lo, p4[1].hi, p4[1].lo);
                        st_shared4(at + 16u, p4[2].hi, p4[2].lo, p4[3].hi, p4[3].lo);
                    }
                }
            } else if constexpr (GEN) {
                const double x = f3_to_double(f3_warp_sum4(p4));
                if ((lane & 7) == 0) red[4 * warp + (lane >> 3)] = x;
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    for (int o = 16; o > 0; o >>= 1) p4[c] = f2_add(p4[c], f2_shfl_down(p4[c], o));
                if (lane == 0) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) { redf[8 * warp + 2 * c] = p4[c].hi; redf[8 * warp + 2 * c + 1] = p4[c].lo; }
                }
            }
            const int nvw = a.nt_sum >> 5;
            if (a.obs) {
                // plain FP32 sums over the sites vt, vt + nt_sum, ... of
                // nt_sum virtual threads (the geometry's nominal threads, so
                // that the sums do not depend on the launch's block size)
                for (int vw = warp; vw < nvw; vw += NW >> 5) {
                    F3 q4[4] = {};   // GEN
                    float v[4] = {0.f, 0.f, 0.f, 0.f};
                    if (vw * 32 < n_local) {
                        for (int l = vw * 32 + lane; l < n_local; l += a.nt_sum) {
                            const int at = l / ncells;
                            if constexpr (GEN) {
                                float w[4] = {0.f, 0.f, 0.f, 0.f};
                                obs_add(s3[3 * l], s3[3 * l + 1], s3[3 * l + 2], __ldg(a.obs_atom + at), w[0], w[1], w[2],
                                        w[3]);
#pragma unroll
                                for (int c = 0; c < 4; ++c) q4[c] = f3_add(q4[c], w[c]);
                            } else {
                                obs_add(s3[3 * l], s3[3 * l + 1], s3[3 * l + 2], __ldg(a.obs_atom + at), v[0], v[1], v[2],
                                        v[3]);
                            }
                        }
                        if constexpr (!GEN) {
#pragma unroll
                            for (int c = 0; c < 4; ++c)
                                for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
                        }
                    }
                    if constexpr (GEN) {
                        const double x = f3_to_double(f3_warp_sum4(q4));
                        if ((lane & 7) == 0) reinterpret_cast<double *>(redo)[4 * vw + (lane >> 3)] = x;
                    } else if (lane == 0) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) redo[4 * vw + c] = v[c];
                    }
                }
            }
            if constexpr (!PP) {
                __syncthreads();
                if (warp == 0) {
                    double *tot = red + 128 + 8 * (m & 1);
                    if constexpr (GEN) fold_warps(red, nwarps, tot);
#pragma unroll
                    for (int c = 0; c < (GEN ? 0 : 4); ++c) {
                        F2 x = lane < nwarps ? F2{redf[8 * lane + 2 * c], redf[8 * lane + 2 * c + 1]} : F2{0.f, 0.f};
                        for (int o = 16; o > 0; o >>= 1)
                            if (o < nwarps) x = f2_add(x, f2_shfl_down(x, o));
                        if (lane == 0) tot[c] = f2_to_double(x);   // this CTA's totals
                    }
                    if (a.obs) fold_obs(m & 1, tot);
                }
            }
            // P(M) [P(OP), P(SM)] of this CTA's cells
            if (a.na > 1 || a.obs) {
                const int cl_end = (ncells + 31) & ~31;   // whole warps take part in the vote
                WarpRun run_m, run_op, run_sm;
                for (int cl = tid; cl < cl_end; cl += NW) {
                    int bin = -1, bin_op = -1, bin_sm = -1;
                    if (cl < ncells) {
                        float mx = 0.f, my = 0.f, mz = 0.f, op = 0.f, qx = 0.f, qy = 0.f, qz = 0.f;
                        for (int at = 0; at < a.na; ++at) {
                            const int l = at * ncells + cl;
                            const float ox = s3[3 * l], oy = s3[3 * l + 1], oz = s3[3 * l + 2];
                            mx += ox; my += oy; mz += oz;
                            if (a.obs) obs_add(ox, oy, oz, __ldg(a.obs_atom + at), op, qx, qy, qz);
                        }
                        if (a.na > 1) bin = pm_bin(mx, my, mz, (float)a.m_min, pm_scale, a.nf);
                        if (a.obs & 1) bin_op = pm_bin_value(op, (float)a.m_min, pm_scale, a.nf);
                        if (a.obs & 2) bin_sm = pm_bin(qx, qy, qz, (float)a.m_min, pm_scale, a.nf);
                    }
                    hist_add(hist, run_m, bin);
                    if (a.obs) {
                        hist_add(hist + a.nf, run_op, bin_op);
                        hist_add(hist + 2 * a.nf, run_sm, bin_sm);
                    }
                }
                hist_flush(hist, run_m);
                if (a.obs) {
                    hist_flush(hist + a.nf, run_op);
                    hist_flush(hist + 2 * a.nf, run_sm);
                }
                // every warp has read the cells before the next colour pass
                // writes them
                if constexpr (PP) bar_sync(1, NW);
                else __syncthreads();
            }
            // the totals of this measurement wait in buffer (m & 1) of every
            // CTA; rank 0 folds them after the next cluster barrier (the next
            // colour pass, or the end of the launch), so a measurement adds no
            // cluster barrier of its own
            if constexpr (PP) bar_arrive(2 + (m & 1), NT);   // handed over
            else pending = m;
        }
    }

    // ---- end of launch: totals, rejected counts, histogram, spins ----------
    {
        // warp 0 may still read the last measurement's warp partials, which
        // the warp partials below overwrite
        __syncthreads();
        double v[4];
        if constexpr (GEN) {
            v[0] = f3_to_double(accE); v[1] = f3_to_double(accX); v[2] = f3_to_double(accY); v[3] = f3_to_double(accZ);
        } else {
            v[0] = f2_to_double(accE); v[1] = f2_to_double(accX); v[2] = f2_to_double(accY); v[3] = f2_to_double(accZ);
        }
        unsigned long long nr = nrej;
        for (int c = 0; c < 4; ++c)
            for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
        for (int o = 16; o > 0; o >>= 1) nr += __shfl_down_sync(0xffffffffu, nr, o);
        if (lane == 0) {
            for (int c = 0; c < 4; ++c) red[4 * warp + c] = v[c];
            reinterpret_cast<unsigned long long *>(red + 96)[warp] = nr;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double t4[4] = {0, 0, 0, 0};
            unsigned long long tn = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
                for (int c = 0; c < 4; ++c) t4[c] += red[4 * w + c];
                tn += reinterpret_cast<unsigned long long *>(red + 96)[w];
            }
            for (int c = 0; c < 4; ++c) red[144 + c] = t4[c];
            reinterpret_cast<unsigned long long *>(red)[148] = tn;
        }
        if (a.na > 1)
            for (int i = threadIdx.x; i < a.nf; i += blockDim.x)
                if (hist[i]) atomicAdd(a.pm_counts + (size_t)temp * a.nf + i, (unsigned long long)hist[i]);
        if (a.obs)
            for (int i = threadIdx.x; i < 2 * a.nf; i += blockDim.x)
                if (hist[a.nf + i]) atomicAdd(a.obs_pm + (size_t)temp * 2 * a.nf + i, (unsigned long long)hist[a.nf + i]);
        cluster.sync();
        // the launch's last measurement, then the sums since it
        if (pending >= 0 && rank == 0 && warp == fold_warp) fold_measurement(pending);
        if (rank == 0) __syncthreads();   // the fold's accumulator writes before the write-back below
        if (rank == 0 && warp == fold_warp && lane == 0) {
            double d4[4] = {0, 0, 0, 0};
            unsigned long long tn = 0;
            for (int q = 0; q < csize; ++q) {
                const double *pr = cluster.map_shared_rank(red, q);
                for (int c = 0; c < 4; ++c) d4[c] += pr[144 + c];
                tn += reinterpret_cast<const unsigned long long *>(pr)[148];
            }
            a.e_run[r] = e_run + d4[0];
            a.m_run[3 * r] = m_run[0] + d4[1];
            a.m_run[3 * r + 1] = m_run[1] + d4[2];
            a.m_run[3 * r + 2] = m_run[2] + d4[3];
            a.rej[2 * temp + a.phase] += tn;
        }
        if (rank == 0 && cache) {
            const int nl2 = 2 * a.nlev;
            for (int i = threadIdx.x; i < 6; i += blockDim.x) {
                a.data[6 * temp + i] = c_data[i];
                if (a.obs) a.obs_data[6 * temp + i] = c_odata[i];
            }
            for (int i = threadIdx.x; i < nl2; i += blockDim.x) {
                a.lsum[(size_t)temp * nl2 + i] = c_ls[i];
                a.binning[(size_t)temp * nl2 + i] = c_bn[i];
                if (a.obs) { a.obs_lsum[(size_t)temp * nl2 + i] = c_ols[i]; a.obs_bin[(size_t)temp * nl2 + i] = c_obn[i]; }
            }
        }
    }
    if (slab) {
        for (int i = threadIdx.x; i < 3 * n_local; i += blockDim.x) slab[i] = s3[i];
    } else {
        for (int l = threadIdx.x; l < n_local; l += blockDim.x) {
            const size_t g = (size_t)__ldg(a.loc2p + site0 + l) * a.R + r;
            a.sx[g] = s3[3 * l]; a.sy[g] = s3[3 * l + 1]; a.sz[g] = s3[3 * l + 2];
        }
    }
    // peers may still read this CTA's shared memory until every CTA is done
    cluster.sync();
}

template <int S, bool GEN, bool RS, bool CL, bool PP = false>
ClusterKernel cluster_kernel_t(const ClusterVariant &v)
{
    return v.hb ? (v.hd ? k_sweep_cluster<S, true, true, GEN, RS, CL, PP> : k_sweep_cluster<S, true, false, GEN, RS, CL, PP>)
                : (v.hd ? k_sweep_cluster<S, false, true, GEN, RS, CL, PP> : k_sweep_cluster<S, false, false, GEN, RS, CL, PP>);
}

}  // namespace esp
