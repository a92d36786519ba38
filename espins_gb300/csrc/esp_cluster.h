// Cluster-resident sweep kernel (esp_cluster.cu): arguments and launchers.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "esp_device.cuh"
#include "esp_resident.h"

namespace esp {

constexpr int kClusterThreads = 512;
constexpr int kMaxClasses = 8 * kMaxClusterAtoms;

// Couplings of stencil entry e of parity class k (the neighbour's position
// comes from the index table); padded to 32 bytes.
struct ClusterNbr {
    float J, B, Dx, Dy, Dz, pad0, pad1, pad2;
};

// Everything the kernel needs about the lattice's couplings; the header is
// followed in memory by nclass * maxst ClusterNbr entries (class-major).
struct ClusterStencil {
    int nclass, maxst, ncolour, pad;
    int count[kMaxClasses];            // entries of each class
    float4 si[kMaxClusterAtoms];       // (ax, ay, az, Delta)
    float4 fld[kMaxClusterAtoms];      // (f ax, f ay, f az, 0)
    float mag[kMaxClusterAtoms];
    int colour_start[kMaxClasses + 1]; // classes of colour c: class_order[colour_start[c] .. colour_start[c+1])
    int class_order[kMaxClasses];
};

inline size_t cluster_stencil_bytes(int nclass, int maxst)
{
    return sizeof(ClusterStencil) + (size_t)nclass * maxst * sizeof(ClusterNbr);
}

// Tables of the arguments: esp_resident.h
struct ClusterArgs {
    const uint32_t *blob;           // [rank][blob_words]: header, couplings, rows
    int blob_words, smem_words;     // a rank's block; its part kept in shared memory
    int rows_off, rstride, jwords;  // word offset of the rows, words of a row, of a coupling list's J part
    int rows4;                      // rows in global memory: words of their quads of one number (rows_by_quads)
    // [rank's items, colour by colour]: x = byte offset of the spin | row <<
    // 18, y = reference site | atom << 28 | row >> 14 << 31
    const uint2 *desc;
    int na, N, R;
    int nA, n_big, n_small;         // ranks [0, nA) hold n_big sites, the others n_small
    int has_si, has_f;
    // state: the slabs of every replica, [r][rank][local site][x, y, z],
    // converted from and to the handle's spin arrays around the launch; or,
    // with slab == null (small slabs, where two more launches cost more than
    // they save), the spin arrays themselves, element (p, r) at p*R + r
    float *slab;
    float *sx, *sy, *sz;
    const int32_t *loc2p;           // [rank][local site] -> p
    const int32_t *temp_of;
    const float *beta;
    double *e_run, *m_run;
    unsigned long long *rej;        // [R slots][2]
    int phase;
    // measurement
    int measure, n_meas, steps_measure;
    int nt_sum;                     // the geometry's nominal threads
    int nt_update;                  // threads that update sites (the others make trial spins)
    long long meas_base;
    double *data, *lsum, *binning;
    const int32_t *levels;
    int nlev, pt_quirk;
    unsigned long long *pm_counts;
    double *series;                 // [cap][R slots][2] or null
    long long series_cap;
    int nf;
    double m_min, m_max;
    // random stream
    unsigned long long sweep_base;
    // device counters [sweep, swap, measurement, unit] added to sweep_base
    // and meas_base, or null
    const unsigned long long *ctr;
    double rn_inv;                  // 1 / N
    uint32_t rk[20];                // Philox round keys
    int mode;
    float tilt;
    // optional measurements (mcarlo.F90:553-578): bit 0 order parameter,
    // bit 1 staggered magnetisation
    int obs;
    const float4 *obs_atom;         // [na]: axis (x, y, z), staggered coefficient (w)
    double *obs_data;               // [R slots][6]
    double *obs_lsum, *obs_bin;     // [R slots][nlev][2]
    unsigned long long *obs_pm;     // [R slots][2][nf]
};

// The handle's spin arrays (element (p, r) at p*R + r) to and from the slab
// layout of the cluster path, [r][rank][l][3] with l the kernel's local site
// order: shared-memory transposes of 32 sites x 32 replicas, coalesced on
// both sides.
struct SlabArgs {
    float *sx, *sy, *sz;
    float *slab;
    const int32_t *loc2p;           // [rank][local site] -> p
    int R, nA, cs, N, n_big, n_small;
};
cudaError_t launch_to_slabs(const SlabArgs &a, cudaStream_t st);
cudaError_t launch_from_slabs(const SlabArgs &a, cudaStream_t st);

// nhist: P(M) histogram only (1) or P(M), P(OP), P(SM) (3)
// binning levels whose sums a cluster keeps in shared memory during a launch
// (more levels are updated in global memory)
constexpr int kClusterMaxLev = 32;
// doubles of that cache: data and obs data (12), levels (16), four [level][2] arrays
constexpr int kClusterAccDoubles = 12 + kClusterMaxLev / 2 + 8 * kClusterMaxLev;
// doubles of the reduction scratch before that cache
constexpr int kClusterRedDoubles = 152;
size_t cluster_smem_bytes(int n_local, int nf, int nhist, size_t table_bytes);
// The dynamic shared-memory limit is a property of a kernel function, shared
// by every handle that launches it: raise it to the most the device allows
// next to the kernel's static shared memory (it is an upper bound, not an
// allocation), so that configuring one handle never lowers the limit another
// handle's launches need.  Fails if `need` exceeds that maximum.
inline cudaError_t allow_max_dynamic_smem(const void *kernel, size_t need)
{
    int dev = 0, v = 0;
    cudaFuncAttributes fa{};
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    const long long room = (long long)v - (long long)fa.sharedSizeBytes;
    if (room <= 0 || need > (size_t)room) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room);
}

// Thread geometries of the parity-class path: nt threads per CTA, S sites of
// a colour pass per thread at a time: (256, 1), (512, 1), (512, 2).  nt fixes
// which sites a thread sums (the items tid, tid + nt, ... of a colour, in that
// order, whatever S); a launch whose colours have at most one site per thread
// runs with as many threads as it needs.
bool cluster_threads_ok(int nt, int S);
// Kernel variant: biquadratic / DM terms, general lattice, stencil rows in
// shared memory, two sites of a colour pass per thread at a time, warps that
// make the next pass's trial spins (where it leaves warps free); no effect on
// the results.
struct ClusterVariant {
    bool hb, hd, general, rows_smem, pairs, helpers;
};
// bytes of the trial spins and sums that the warps of such a CTA hand over
inline size_t cluster_helper_bytes(int nt_update, bool general)
{
    return 16 + (size_t)2 * (16 + (general ? 48 : 32)) * nt_update;
}
using ClusterKernel = void (*)(ClusterArgs);
ClusterKernel cluster_kernel_classes_one(const ClusterVariant &v);
ClusterKernel cluster_kernel_classes_many(const ClusterVariant &v);
ClusterKernel cluster_kernel_classes_global(const ClusterVariant &v, int csize);
ClusterKernel cluster_kernel_general_one(const ClusterVariant &v);
ClusterKernel cluster_kernel_general_many(const ClusterVariant &v);
cudaError_t cluster_configure(const ClusterVariant &v, size_t smem, int csize);
// Clusters of csize CTAs of nt threads with `smem` bytes each that fit on the GPU at once.
int cluster_max_active(const ClusterVariant &v, int csize, int nt, size_t smem, int R);
cudaError_t launch_cluster(const ClusterArgs &a, const ClusterVariant &v, int csize, int nt, size_t smem,
                           cudaStream_t st);

}  // namespace esp
