// Monte Carlo kernels for sm_103a.
//
//   k_sweep_ell      one colour class of a Metropolis sweep, every replica
//                    (metropolis + delta_energy_get, get_quant.F90:52-182,264-337)
//   k_energy_part    energy_get (get_quant.F90:186-261) and sum_i s_i per
//                    replica: per-block partials into scratch ...
//   k_energy_reduce  ... reduced in a fixed order (deterministic FP64)
//   k_local_terms    the per-site linear/quadratic coefficients (parity checks)
//   k_obs_part       orderparam_get / staggered_get sums (get_quant.F90:366-422),
//                    reduced by k_energy_reduce
//   k_sc_part        spincorr_get (get_quant.F90:495-540) bin sums per
//                    replica, reduced and accumulated per slot by k_sc_reduce
//   k_sf_part        mcarlo_structure_factor (get_quant.F90:649-717): F(q) per
//                    replica; k_sf_finish projects and accumulates per slot
//   k_measure        per-measurement accumulators and binning
//                    (mcarlo.F90:536-590, pt.F90:789-849)
//   k_pm_hist        Pm_get (get_quant.F90:425-493) as an integer histogram
//   k_pt_swap        pt_swap (pt.F90:1235-1288) on temperature labels
//   k_init_spins     ferro / rand start configurations (mcarlo.F90:271-293)
//   k_spins_in/out   spin_matrix(3,N,slots) <-> the permuted FP32 SoA state
//
// Layout: spins are FP32 SoA (sx, sy, sz), element (p, r) at p*R + r, with p
// the colour-major permuted site index and r the replica.  Consecutive threads
// take consecutive replicas of one site, so spin loads and stores of a warp
// are contiguous and the table entries of a site are read once per warp.
#include "esp_device.cuh"
#include "esp_kernels.h"

namespace esp {

// ---------------------------------------------------------------------------
// Per-block partial sums, no atomics.  Thread t of block b works on replica
// (b*blockDim + t) % R for the whole launch, so the threads of one replica in
// a block are t0, t0+R, ...; thread t < slots (= min(R, blockDim)) sums them
// and adds the result to its block's own slot part[b][t].  Every launch of the
// sweep uses the same grid, so slot (b, t) always belongs to the same block and
// the same replica; k_fold later sums the slots of each replica in block order
// (deterministic) into the running totals.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void add_block_slots(float e, float mx, float my, float mz, unsigned int nrej,
                                                int R, int slots, double *part, unsigned long long *part_rej)
{
    __shared__ double s_part[256][4];
    __shared__ unsigned int s_rej[256];
    const int t = threadIdx.x;
    const int nt = blockDim.x;
    const size_t slot = (size_t)blockIdx.x * slots + t;
    if (R >= nt) {
        double *o = part + 4 * slot;
        o[0] += (double)e; o[1] += (double)mx; o[2] += (double)my; o[3] += (double)mz;
        part_rej[slot] += (unsigned long long)nrej;
        return;
    }
    s_part[t][0] = (double)e; s_part[t][1] = (double)mx; s_part[t][2] = (double)my; s_part[t][3] = (double)mz;
    s_rej[t] = nrej;
    __syncthreads();
    if (t < R) {
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
        unsigned long long nr = 0;
        for (int u = t; u < nt; u += R) {
            a0 += s_part[u][0]; a1 += s_part[u][1]; a2 += s_part[u][2]; a3 += s_part[u][3];
            nr += s_rej[u];
        }
        double *o = part + 4 * slot;
        o[0] += a0; o[1] += a1; o[2] += a2; o[3] += a3;
        part_rej[slot] += nr;
    }
}

// Sum every block's slot of replica r, add it to the running energy /
// magnetisation and to the rejected counter of r's temperature slot, and
// clear the slots.  One block per replica: thread t takes blocks t, t+256, ...
// and a fixed-shape tree combines the threads, so the sum is deterministic.
__global__ void __launch_bounds__(256) k_fold(FoldArgs a)
{
    __shared__ double s_v[4][256];
    __shared__ unsigned long long s_n[256];
    const int r = blockIdx.x;
    double e = 0, mx = 0, my = 0, mz = 0;
    unsigned long long nr = 0;
    // Bound by latency (32 bytes of each of a few blocks a thread): the slots
    // of four blocks are loaded before any is cleared, and the position in the
    // next block follows from the last one's.  608 blocks x 32 replicas: 9 us,
    // 40 us with one block and one 64-bit remainder after the other.
    const int step = (int)((256ll * a.block_threads) % a.R);
    int t = (int)(((long long)r - (long long)threadIdx.x * a.block_threads) % a.R);
    if (t < 0) t += a.R;
    for (int b0 = threadIdx.x; b0 < a.nblocks; b0 += 4 * 256) {
        double2 v[4][2];
        unsigned long long n[4];
        size_t slot[4];
        bool have[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int b = b0 + 256 * j;
            have[j] = b < a.nblocks && t < a.slots;
            if (have[j]) {
                slot[j] = (size_t)b * a.slots + t;
                const double2 *o = reinterpret_cast<const double2 *>(a.part + 4 * slot[j]);
                v[j][0] = o[0];
                v[j][1] = o[1];
                n[j] = a.part_rej[slot[j]];
            }
            t -= step;
            if (t < 0) t += a.R;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!have[j]) continue;
            e += v[j][0].x; mx += v[j][0].y; my += v[j][1].x; mz += v[j][1].y;
            nr += n[j];
            double2 *o = reinterpret_cast<double2 *>(a.part + 4 * slot[j]);
            o[0] = make_double2(0.0, 0.0);
            o[1] = make_double2(0.0, 0.0);
            a.part_rej[slot[j]] = 0ull;
        }
    }
    const int i = threadIdx.x;
    s_v[0][i] = e; s_v[1][i] = mx; s_v[2][i] = my; s_v[3][i] = mz; s_n[i] = nr;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (i < w) {
            for (int c = 0; c < 4; ++c) s_v[c][i] += s_v[c][i + w];
            s_n[i] += s_n[i + w];
        }
        __syncthreads();
    }
    if (i == 0) {
        a.e_run[r] += s_v[0][0];
        a.m_run[3 * r] += s_v[1][0]; a.m_run[3 * r + 1] += s_v[2][0]; a.m_run[3 * r + 2] += s_v[3][0];
        a.rej[2 * a.temp_of[r] + a.phase] += s_n[0];
    }
}

// ---------------------------------------------------------------------------
// One colour class, all replicas.  Grid-stride with a stride that is a
// multiple of R, so each thread keeps one replica for its whole life.
// ---------------------------------------------------------------------------
template <bool HB, bool HD>
__global__ void __launch_bounds__(256) k_sweep_ell(const SweepArgs a)
{
    const int R = a.R;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    const long long S = (nthreads / R) * R;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = tid < S;
    const int r = (int)(tid % R);
    const int temp = a.temp_of[r];
    // FP32 per thread (a few updates each); FP64 from the block sums on
    float accE = 0.f, accX = 0.f, accY = 0.f, accZ = 0.f;
    unsigned int nrej = 0;
    uint32_t sw_lo, sw_hi;
    sweep_index(a, sw_lo, sw_hi);
    if (live) {
        const float beta = a.beta[temp];
        const int pstep = (int)(S / R);
        const bool has_si = a.si != nullptr, has_f = a.fld != nullptr;
        for (int pi = (int)(tid / R); pi < a.n_c; pi += pstep) {
            const int p = a.off_c + pi;
            const size_t idx = (size_t)p * R + r;
            const float ox = a.sx[idx], oy = a.sy[idx], oz = a.sz[idx];
            float gx = 0.f, gy = 0.f, gz = 0.f;
            float qxx = 0.f, qyy = 0.f, qzz = 0.f, qxy = 0.f, qxz = 0.f, qyz = 0.f;
            // entries come in groups of 8 (the host pads every list with
            // zero-coupling entries pointing at the site itself), so each
            // group issues 8 independent index loads and then 24 spin loads
            const int nn = __ldg(a.nnb + p);
            for (int k0 = 0; k0 < nn; k0 += 8) {
                int q[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) q[j] = __ldg(a.nbr + (size_t)(k0 + j) * a.N + p);
                float tx[8], ty[8], tz[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const size_t iq = (size_t)q[j] * R + r;
                    tx[j] = __ldg(a.sx + iq); ty[j] = __ldg(a.sy + iq); tz[j] = __ldg(a.sz + iq);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const size_t e = (size_t)(k0 + j) * a.N + p;
                    const float J = __ldg(a.J + e);
                    gx = fmaf(-J, tx[j], gx); gy = fmaf(-J, ty[j], gy); gz = fmaf(-J, tz[j], gz);
                    if (HB) bq_form(__ldg(a.B + e), tx[j], ty[j], tz[j], qxx, qyy, qzz, qxy, qxz, qyz);
                    // s_k x D_ik (the DM term of delta_energy_get as s_i . (s_k x D))
                    if (HD) dm_field(__ldg(a.Dx + e), __ldg(a.Dy + e), __ldg(a.Dz + e), tx[j], ty[j], tz[j], gx, gy, gz);
                }
            }
            const int orig = __ldg(a.perm + p);
            if (has_si || has_f) {
                const int at = orig % a.num_atoms;
                if (has_si) si_form(__ldg(a.si + at), qxx, qyy, qzz, qxy, qxz, qyz);
                if (has_f) {
                    const float4 f = __ldg(a.fld + at);
                    gx = __fadd_rn(gx, f.x); gy = __fadd_rn(gy, f.y); gz = __fadd_rn(gz, f.z);
                }
            }
            const Philox4 x = philox4x32_10((uint32_t)orig, (uint32_t)r, sw_lo, sw_hi, a.key0, a.key1);
            float nx, ny, nz;
            trial_spin(a.mode, a.tilt, __ldg(a.mag + p), ox, oy, oz, x.x, x.y, nx, ny, nz);
            const float dx = nx - ox, dy = ny - oy, dz = nz - oz;
            // s_new^T Q s_new - s_old^T Q s_old = d^T Q (s_new + s_old)
            const float de = delta_energy(HB || has_si, gx, gy, gz, qxx, qyy, qzz, qxy, qxz, qyz, ox, oy, oz, nx, ny, nz);
            const bool acc = metropolis_accept(beta, de, x.z);
            if (acc) {
                a.sx[idx] = nx; a.sy[idx] = ny; a.sz[idx] = nz;
                accE += de;
                accX += dx; accY += dy; accZ += dz;
            } else {
                ++nrej;
            }
        }
    }
    add_block_slots(accE, accX, accY, accZ, nrej, R, a.slots, a.part, a.part_rej);
}

// ---------------------------------------------------------------------------
// Direct energy and magnetisation, stage 1: thread-local FP64 sums of the
// per-site energies e_i = 1/2 sum_k pair_ik + Delta (s.a)^2 + f.s, then a
// fixed-order block reduction per replica into scratch[block][R][4].
// ---------------------------------------------------------------------------
struct EnergyArgs {
    const int32_t *nnb, *nbr;
    const float *J, *B, *Dx, *Dy, *Dz;
    const int32_t *perm;
    const float4 *si, *fld;
    const float *sx, *sy, *sz;
    double *scratch;          // [gridDim.x][R][4]
    int32_t N, R, num_atoms;
};

// Per-replica sums of the four values in s_acc[t] of this block's threads
// (the replica of thread t is (blockIdx.x * blockDim.x + t) % R, threads at or
// past S hold nothing), in a fixed order, to scratch[block][R][4].
__device__ void store_block_replica_sums(double (*s_acc)[4], long long S, int R, double *scratch)
{
    const int t = threadIdx.x;
    const int base = (int)(((long long)blockIdx.x * blockDim.x) % R);
    for (int rr = t; rr < R; rr += blockDim.x) {
        // first thread of this block holding replica rr
        int u0 = rr - base;
        if (u0 < 0) u0 += R;
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
        for (int u = u0; u < (int)blockDim.x; u += R) {
            const long long g = (long long)blockIdx.x * blockDim.x + u;
            if (g >= S) break;
            a0 += s_acc[u][0]; a1 += s_acc[u][1]; a2 += s_acc[u][2]; a3 += s_acc[u][3];
        }
        double *o = scratch + ((size_t)blockIdx.x * R + rr) * 4;
        o[0] = a0; o[1] = a1; o[2] = a2; o[3] = a3;
    }
}

template <bool HB, bool HD>
__global__ void __launch_bounds__(256) k_energy_part(const EnergyArgs a)
{
    __shared__ double s_acc[256][4];
    const int R = a.R;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    const long long S = (nthreads / R) * R;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0, mx = 0, my = 0, mz = 0;
    if (tid < S) {
        const int r = (int)(tid % R);
        const int pstep = (int)(S / R);
        for (int p = (int)(tid / R); p < a.N; p += pstep) {
            const size_t idx = (size_t)p * R + r;
            const float ox = a.sx[idx], oy = a.sy[idx], oz = a.sz[idx];
            float pair = 0.f;
            // Bound by the latency of the spin loads (out of L2).  Lists are
            // padded to multiples of 8 with the site itself and zero couplings:
            // 8 index loads, then 24 spin loads in flight.  Against one
            // neighbour at a time: 104 -> 84 us for bcc 24^3 x 48 (26
            // neighbours), 3306 -> 2720 us for sc 96 x 96 x 48 x 64; the call
            // 341 -> 289 us for sc 48^3 x 32, 565 -> 455 us x 48.
            const int nn = __ldg(a.nnb + p);
            for (int k0 = 0; k0 < nn; k0 += 8) {
                int q[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) q[j] = __ldg(a.nbr + (size_t)(k0 + j) * a.N + p);
                float sx8[8], sy8[8], sz8[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const size_t iq = (size_t)q[j] * R + r;
                    sx8[j] = __ldg(a.sx + iq); sy8[j] = __ldg(a.sy + iq); sz8[j] = __ldg(a.sz + iq);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const size_t ee = (size_t)(k0 + j) * a.N + p;
                    const float tx = sx8[j], ty = sy8[j], tz = sz8[j];
                    const float d = ox * tx + oy * ty + oz * tz;
                    pair -= __ldg(a.J + ee) * d;
                    if (HB) pair += __ldg(a.B + ee) * d * d;
                    if (HD) {
                        const float cx = oy * tz - oz * ty, cy = oz * tx - ox * tz, cz = ox * ty - oy * tx;
                        pair += __ldg(a.Dx + ee) * cx + __ldg(a.Dy + ee) * cy + __ldg(a.Dz + ee) * cz;
                    }
                }
            }
            float site = 0.5f * pair;
            if (a.si || a.fld) {
                const int at = a.perm[p] % a.num_atoms;
                if (a.si) {
                    const float4 s = a.si[at];
                    const float sa = ox * s.x + oy * s.y + oz * s.z;
                    site += s.w * sa * sa;
                }
                if (a.fld) {
                    const float4 f = a.fld[at];
                    site += f.x * ox + f.y * oy + f.z * oz;
                }
            }
            e += (double)site;
            mx += (double)ox; my += (double)oy; mz += (double)oz;
        }
    }
    const int t = threadIdx.x;
    s_acc[t][0] = e; s_acc[t][1] = mx; s_acc[t][2] = my; s_acc[t][3] = mz;
    __syncthreads();
    store_block_replica_sums(s_acc, S, R, a.scratch);
}

// Stage 1 of the order-parameter / staggered sums: per (site, replica) the
// FP32 products s.a and c s, summed per thread and block in FP64 like the
// energy.
__global__ void __launch_bounds__(256) k_obs_part(const ObsArgs a)
{
    __shared__ double s_acc[256][4];
    const int R = a.R;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    const long long S = (nthreads / R) * R;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double op = 0, qx = 0, qy = 0, qz = 0;
    if (tid < S) {
        const int r = (int)(tid % R);
        const int pstep = (int)(S / R);
        for (int p = (int)(tid / R); p < a.N; p += pstep) {
            const size_t idx = (size_t)p * R + r;
            const float ox = a.sx[idx], oy = a.sy[idx], oz = a.sz[idx];
            const float4 w = __ldg(a.atom + a.perm[p] % a.num_atoms);
            float fo = 0.f, fx = 0.f, fy = 0.f, fz = 0.f;
            obs_add(ox, oy, oz, w, fo, fx, fy, fz);
            op += (double)fo; qx += (double)fx; qy += (double)fy; qz += (double)fz;
        }
    }
    const int t = threadIdx.x;
    s_acc[t][0] = op; s_acc[t][1] = qx; s_acc[t][2] = qy; s_acc[t][3] = qz;
    __syncthreads();
    store_block_replica_sums(s_acc, S, R, a.scratch);
}

// Stage 2: out_e[r] = sum over blocks, out_m[r][3] likewise.  One block per
// replica: thread t takes blocks t, t+256, ... and a fixed-shape tree combines
// the threads, so the sum is deterministic.
__global__ void __launch_bounds__(256) k_energy_reduce(const double *scratch, int nblocks, int R, double *out_e,
                                                       double *out_m)
{
    __shared__ double s_v[4][256];
    const int r = blockIdx.x, t = threadIdx.x;
    double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    for (int b = t; b < nblocks; b += blockDim.x) {
        const double *o = scratch + ((size_t)b * R + r) * 4;
        a0 += o[0]; a1 += o[1]; a2 += o[2]; a3 += o[3];
    }
    s_v[0][t] = a0; s_v[1][t] = a1; s_v[2][t] = a2; s_v[3][t] = a3;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (t < w)
            for (int c = 0; c < 4; ++c) s_v[c][t] += s_v[c][t + w];
        __syncthreads();
    }
    if (t == 0) {
        out_e[r] = s_v[0][0];
        if (out_m) { out_m[3 * r] = s_v[1][0]; out_m[3 * r + 1] = s_v[2][0]; out_m[3 * r + 2] = s_v[3][0]; }
    }
}

// ---------------------------------------------------------------------------
// spincorr_get: bins in pairs per pass (a row of blocks each, so that one
// pass's gather latency hides another's); per item (site, replica) FP32 sums
// over the bin's entries, FP64 per thread and block (like the energy).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_sc_part(const ScArgs a)
{
    __shared__ double s_acc[256][4];
    const int R = a.R, N = a.N;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    const long long S = (nthreads / R) * R;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int pass = blockIdx.y;
    double v[4] = {0, 0, 0, 0};
    if (tid < S) {
        const int r = (int)(tid % R);
        const int pstep = (int)(S / R);
        for (int p = (int)(tid / R); p < N; p += pstep) {
            const size_t idx = (size_t)p * R + r;
            const float ox = a.sx[idx], oy = a.sy[idx], oz = a.sz[idx];
            int off[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) off[q] = __ldg(a.off + (size_t)min(2 * pass + q, a.B) * N + p);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float sum = 0.f, sabs = 0.f;
                // entries in groups of 4 so that their loads overlap
                for (int e = off[q]; e < off[q + 1]; e += 4) {
                    float d[4], w[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const size_t ee = (size_t)min(e + j, off[q + 1] - 1) * N + p;
                        const size_t iq = (size_t)__ldg(a.nb + ee) * R + r;
                        d[j] = ox * a.sx[iq] + oy * a.sy[iq] + oz * a.sz[iq];
                        w[j] = __ldg(a.w + ee);
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (e + j < off[q + 1]) {
                            const float wd = w[j] * d[j];
                            sum += wd;
                            sabs += fabsf(wd);
                        }
                }
                v[2 * q] += (double)sum;
                v[2 * q + 1] += (double)sabs;
            }
        }
    }
    const int t = threadIdx.x;
    s_acc[t][0] = v[0]; s_acc[t][1] = v[1]; s_acc[t][2] = v[2]; s_acc[t][3] = v[3];
    __syncthreads();
    store_block_replica_sums(s_acc, S, R, a.scratch + (size_t)pass * gridDim.x * R * 4);
}

// Block (r, pass): fixed-order sum of the blocks' partials of replica r, then
// for its temperature slot spincorr += S_b, spincorr_abs += A_b, tot_abs +=
// |S_b| (get_quant.F90:535-537) of the pass's two bins.
__global__ void __launch_bounds__(256) k_sc_reduce(const ScArgs a, int nblocks)
{
    __shared__ double s_v[4][256];
    const int r = blockIdx.x, pass = blockIdx.y, t = threadIdx.x, R = a.R;
    const double *base = a.scratch + (size_t)pass * nblocks * R * 4;
    double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    for (int b = t; b < nblocks; b += blockDim.x) {
        const double *o = base + ((size_t)b * R + r) * 4;
        a0 += o[0]; a1 += o[1]; a2 += o[2]; a3 += o[3];
    }
    s_v[0][t] = a0; s_v[1][t] = a1; s_v[2][t] = a2; s_v[3][t] = a3;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (t < w)
            for (int c = 0; c < 4; ++c) s_v[c][t] += s_v[c][t + w];
        __syncthreads();
    }
    const int bin = 2 * pass + t;
    if (t < 2 && bin < a.B) {
        double *acc = a.acc + ((size_t)a.temp_of[r] * a.B + bin) * 3;
        const double sum = s_v[2 * t][0];
        acc[0] += sum;
        acc[1] += s_v[2 * t + 1][0];
        acc[2] += fabs(sum);
    }
}

// ---------------------------------------------------------------------------
// Structure factor F(q) = sum_i s_i e^{iq.r_i} per replica, the sites of each
// sum in order in one FP32 accumulator (so a sum cannot be split): the
// parallelism is (q, replica, component).  A block takes QB q-points x RB
// replicas and walks the sites in tiles, whose phases (shared by the
// replicas) and spins (shared by the q-points) it stages in shared memory, two
// buffers with one barrier per tile; a component's real and imaginary part
// are the lanes of one fma.rn.f32x2.  The phase is exact to 2^-24 of a turn.
//
// Bound: for small meshes the chain of N dependent additions with few warps to
// hide it, so a thread takes one component of one (q, replica) and blocks are
// small (8 q x 8 replicas, 66 blocks for 169 q x 24 replicas); large meshes
// are FP32- and shared-memory-bound, so a thread takes 4 q and all components
// and the block 64 q x 16 replicas, once those blocks fill the GPU.  169 q x 24
// replicas x 3,087 sites: 418 us with 64 q x 4 replicas a block (18 blocks),
// 71 us so, the phases from a table (171 us when each block makes its own).
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long sf_step(const SfArgs &a)
{
    return a.step + (a.ctr ? (long long)*a.ctr : 0ll);
}

__device__ __forceinline__ float2 sf_phase(const SfArgs &a, int i, int qg)
{
    const int4 n = __ldg(a.site_n + i);
    const float4 f = __ldg(a.site_f + i);
    const uint4 qfix = __ldg(a.q_fix + qg);
    const float4 qf = __ldg(a.q_frac + qg);
    // whole cells: exact modulo one turn in 32-bit fixed point
    const uint32_t t = qfix.x * (uint32_t)n.x + qfix.y * (uint32_t)n.y + qfix.z * (uint32_t)n.z;
    const float tw = (float)(int32_t)t * 2.3283064365386963e-10f;   // [-1/2, 1/2) turn
    float tf = qf.x * f.x + qf.y * f.y + qf.z * f.z;
    tf -= rintf(tf);
    float c, sn;
    sincospif(2.f * (tw + tf), &sn, &c);
    return make_float2(c, sn);
}

// the phases of every (site, q)
__global__ void __launch_bounds__(256) k_sf_phases(const SfArgs a, float2 *out)
{
    const long long n = (long long)a.N * a.nq;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
        out[k] = sf_phase(a, (int)(k / a.nq), (int)(k % a.nq));
}

__device__ __forceinline__ float2 sf_fma(float2 x, float2 ph, float2 f)
{
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(x.x), "f"(x.y), "f"(ph.x), "f"(ph.y), "f"(f.x), "f"(f.y));
    return d;
}

// QT q-points and CT components (1 or 3) per thread, tiles of TS sites; TAB:
// the phases are read from a table made once
template <int QB, int RB, int QT, int CT, int TS, bool TAB>
__global__ void __launch_bounds__(QB / QT * RB * 3 / CT) k_sf_part(const SfArgs a)
{
    constexpr int NT = QB / QT * RB * 3 / CT, NQ = QB / QT;
    constexpr int NP = (QB * TS + NT - 1) / NT, NS = (RB * TS + NT - 1) / NT;
    static_assert(CT == 1 || CT == 3, "components per thread");
    if (sf_step(a) % a.every != 0) return;
    __shared__ __align__(16) float2 s_ph[2][TS][QB];
    __shared__ __align__(16) float2 s_sp[2][TS][3][RB];   // a component in both lanes
    const int t = threadIdx.x, tq = t % NQ, tr = (t / NQ) % RB, tc = CT == 1 ? t / (NQ * RB) : 0;
    const int q0 = blockIdx.x * QB, r0 = blockIdx.y * RB;
    float2 f[QT][CT];
#pragma unroll
    for (int k = 0; k < QT; ++k)
#pragma unroll
        for (int c = 0; c < CT; ++c) f[k][c] = make_float2(0.f, 0.f);
    float x[NS], y[NS], z[NS];
    float2 ph_in[TAB ? NP : 1];
    // spins and tabulated phases of the tile from site i0 (in flight while the previous one is summed)
    auto fetch = [&](int i0) {
#pragma unroll
        for (int m = 0; m < NS; ++m) {
            const int k = t + m * NT, i = i0 + k / RB, rg = r0 + k % RB;
            x[m] = y[m] = z[m] = 0.f;
            if (k < RB * TS && i < a.N && rg < a.R) {
                const size_t idx = (size_t)__ldg(a.inv + i) * a.R + rg;
                x[m] = a.sx[idx]; y[m] = a.sy[idx]; z[m] = a.sz[idx];
            }
        }
        if constexpr (TAB) {
#pragma unroll
            for (int m = 0; m < NP; ++m) {
                const int k = t + m * NT, i = i0 + k / QB, qg = q0 + k % QB;
                ph_in[m] = make_float2(0.f, 0.f);
                if (k < QB * TS && i < a.N && qg < a.nq) ph_in[m] = __ldg(a.phase + (size_t)i * a.nq + qg);
            }
        }
    };
    auto stage = [&](int i0, int buf) {
#pragma unroll
        for (int m = 0; m < NS; ++m) {
            const int k = t + m * NT;
            if (k < RB * TS) {
                s_sp[buf][k / RB][0][k % RB] = make_float2(x[m], x[m]);
                s_sp[buf][k / RB][1][k % RB] = make_float2(y[m], y[m]);
                s_sp[buf][k / RB][2][k % RB] = make_float2(z[m], z[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            const int k = t + m * NT, i = i0 + k / QB, qg = q0 + k % QB;
            if (k < QB * TS) {
                if constexpr (TAB) s_ph[buf][k / QB][k % QB] = ph_in[m];
                else s_ph[buf][k / QB][k % QB] = i < a.N && qg < a.nq ? sf_phase(a, i, qg) : make_float2(0.f, 0.f);
            }
        }
    };
    fetch(0);
    stage(0, 0);
    int buf = 0;
    for (int i0 = 0; i0 < a.N; i0 += TS, buf ^= 1) {
        __syncthreads();   // this buffer is staged, the other one read by everyone
        const bool more = i0 + TS < a.N;
        if (more) fetch(i0 + TS);
#pragma unroll 8
        for (int j = 0; j < TS; ++j) {
            float2 sp[CT];
#pragma unroll
            for (int c = 0; c < CT; ++c) sp[c] = s_sp[buf][j][CT == 1 ? tc : c][tr];
#pragma unroll
            for (int k = 0; k < QT; ++k) {
                const float2 ph = s_ph[buf][j][tq + k * NQ];
#pragma unroll
                for (int c = 0; c < CT; ++c) f[k][c] = sf_fma(sp[c], ph, f[k][c]);
            }
        }
        if (more) stage(i0 + TS, buf ^ 1);
    }
#pragma unroll
    for (int k = 0; k < QT; ++k) {
        const int q = q0 + tq + k * NQ, r = r0 + tr;
        if (q < a.nq && r < a.R) {
            float2 *o = reinterpret_cast<float2 *>(a.fq + ((size_t)r * a.nq + q) * 6);
#pragma unroll
            for (int c = 0; c < CT; ++c) o[CT == 1 ? tc : c] = f[k][c];
        }
    }
}

// Per (q, slot): F_perp = F - q (q.F) / q.q, NSF = Re(p.F_perp) / |p|
// (get_quant.F90:693-710), accumulated in FP64.
__global__ void k_sf_finish(const SfArgs a)
{
    if (sf_step(a) % a.every != 0) return;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *a.count += 1;
    if (k >= (long long)a.nq * a.R) return;
    const int q = (int)(k % a.nq), t = (int)(k / a.nq);
    const float4 qc = __ldg(a.q_cart + q);
    if (qc.w != 0.f) return;
    const float *f = a.fq + ((size_t)a.repl_at[t] * a.nq + q) * 6;
    const double qx = qc.x, qy = qc.y, qz = qc.z;
    const double qq = qx * qx + qy * qy + qz * qz;
    const double dre = (f[0] * qx + f[2] * qy + f[4] * qz) / qq;
    const double dim = (f[1] * qx + f[3] * qy + f[5] * qz) / qq;
    const double xr = f[0] - dre * qx, xi = f[1] - dim * qx;
    const double yr = f[2] - dre * qy, yi = f[3] - dim * qy;
    const double zr = f[4] - dre * qz, zi = f[5] - dim * qz;
    const double f2 = xr * xr + xi * xi + yr * yr + yi * yi + zr * zr + zi * zi;
    const double nsf = (a.px * xr + a.py * yr + a.pz * zr) / a.pnorm;
    double *o = a.acc + ((size_t)t * a.nq + q) * 3;
    o[0] += f2;
    o[1] += f2 - nsf * nsf;
    o[2] += nsf * nsf;
}

// ---------------------------------------------------------------------------
// Local terms g_i (3) and Q_i (6) of every (site, replica), FP32.
// ---------------------------------------------------------------------------
template <bool HB, bool HD>
__global__ void k_local_terms(const EnergyArgs a, float *g, float *q)
{
    const long long total = (long long)a.N * a.R;
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < total;
         it += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(it / a.R), r = (int)(it % a.R);
        float gx = 0, gy = 0, gz = 0, qxx = 0, qyy = 0, qzz = 0, qxy = 0, qxz = 0, qyz = 0;
        const int nn = a.nnb[p];
        for (int k = 0; k < nn; ++k) {
            const size_t e = (size_t)k * a.N + p;
            const size_t iq = (size_t)a.nbr[e] * a.R + r;
            const float tx = a.sx[iq], ty = a.sy[iq], tz = a.sz[iq];
            const float J = a.J[e];
            gx = fmaf(-J, tx, gx); gy = fmaf(-J, ty, gy); gz = fmaf(-J, tz, gz);
            if (HB) {
                const float Bv = a.B[e];
                const float bx = Bv * tx, by = Bv * ty, bz = Bv * tz;
                qxx = fmaf(bx, tx, qxx); qyy = fmaf(by, ty, qyy); qzz = fmaf(bz, tz, qzz);
                qxy = fmaf(bx, ty, qxy); qxz = fmaf(bx, tz, qxz); qyz = fmaf(by, tz, qyz);
            }
            if (HD) {
                const float dx = a.Dx[e], dy = a.Dy[e], dz = a.Dz[e];
                gx += ty * dz - tz * dy; gy += tz * dx - tx * dz; gz += tx * dy - ty * dx;
            }
        }
        if (a.si || a.fld) {
            const int at = a.perm[p] % a.num_atoms;
            if (a.si) {
                const float4 s = a.si[at];
                const float dx = s.w * s.x, dy = s.w * s.y, dz = s.w * s.z;
                qxx = fmaf(dx, s.x, qxx); qyy = fmaf(dy, s.y, qyy); qzz = fmaf(dz, s.z, qzz);
                qxy = fmaf(dx, s.y, qxy); qxz = fmaf(dx, s.z, qxz); qyz = fmaf(dy, s.z, qyz);
            }
            if (a.fld) { const float4 f = a.fld[at]; gx += f.x; gy += f.y; gz += f.z; }
        }
        float *go = g + (size_t)it * 3;
        go[0] = gx; go[1] = gy; go[2] = gz;
        float *qo = q + (size_t)it * 6;
        qo[0] = qxx; qo[1] = qyy; qo[2] = qzz; qo[3] = qxy; qo[4] = qxz; qo[5] = qyz;
    }
}

// ---------------------------------------------------------------------------
// Per-measurement accumulators, one thread per temperature slot.
// data[t][6] += E, E^2, E^4, |m|, m^2, m^4 with m = M/N (mcarlo.F90:536-543);
// binning sums as mcarlo.F90:548-590 (pt_quirk: pt.F90:841-849 divides a
// completed block by 2**l, l being the level's position).
// ---------------------------------------------------------------------------
__global__ void k_measure(MeasureArgs a)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.R) return;
    if (a.ctr) a.step += (long long)*a.ctr;
    const int r = a.repl_at[t];
    const double e = a.e_run[r];
    const double mx = a.m_run[3 * r] / (double)a.N;
    const double my = a.m_run[3 * r + 1] / (double)a.N;
    const double mz = a.m_run[3 * r + 2] / (double)a.N;
    const double m2 = mx * mx + my * my + mz * mz;
    const double ee = e * e;
    double *d = a.data + 6 * t;
    d[0] += e; d[1] += ee; d[2] += ee * ee;
    const double am = sqrt(m2);
    d[3] += am; d[4] += m2; d[5] += m2 * m2;
    if (a.series) {
        double *o = a.series + (((a.step - 1) % a.series_cap) * a.R + t) * 2;
        o[0] = e; o[1] = am;
    }
    // orderparam_get / staggered_get of this replica (mcarlo.F90:553-568)
    double aop = 0.0, asm_ = 0.0;
    if (a.obs) {
        double *od = a.obs_data + 6 * t;
        const double *q = a.obs_rep + a.R + 3 * r;
        if (a.obs & 1) {
            const double op = a.obs_rep[r] / (double)a.N;
            const double o2 = op * op;
            aop = sqrt(o2);
            od[0] += aop; od[1] += o2; od[2] += o2 * o2;
        }
        if (a.obs & 2) {
            const double qx = q[0] / (double)a.N, qy = q[1] / (double)a.N, qz = q[2] / (double)a.N;
            const double q2 = qx * qx + qy * qy + qz * qz;
            asm_ = sqrt(q2);
            od[3] += asm_; od[4] += q2; od[5] += q2 * q2;
        }
    }
    if (a.nlev > 0) {
        double *ls = a.lsum + (size_t)t * a.nlev * 2;
        double *bn = a.binning + (size_t)t * a.nlev * 2;
        double *ols = a.obs ? a.obs_lsum + (size_t)t * a.nlev * 2 : nullptr;
        double *obn = a.obs ? a.obs_bin + (size_t)t * a.nlev * 2 : nullptr;
        for (int l = 0; l < a.nlev; ++l) {
            ls[2 * l] += e / (double)a.N;
            ls[2 * l + 1] += am;
            if (ols) { ols[2 * l] += aop; ols[2 * l + 1] += asm_; }
            const long long blk = 1LL << a.levels[l];
            if (a.step % blk == 0) {
                const double div = a.pt_quirk ? (double)(1LL << (l + 1)) : (double)blk;
                for (int c = 0; c < 2; ++c) {
                    const double v = ls[2 * l + c] / div;
                    bn[2 * l + c] += v * v;
                    ls[2 * l + c] = 0.0;
                    if (ols) {
                        const double w = ols[2 * l + c] / div;
                        obn[2 * l + c] += w * w;
                        ols[2 * l + c] = 0.0;
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// P(M) histogram (Pm_get): per unit cell |sum_atoms s| -> bin
// max(nint((|m| - m_min)/(m_max - m_min) * (nf-1)) + 1, 1), counted as
// integers per temperature slot (the reference adds 1/d_m = 100 per hit).
// Block: a tile of cells x all replicas, shared histogram [R][nf] when it fits.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_pm_hist(PmArgs a)
{
    // block (x, y): a chunk of cells x the replica tile [y*rt, y*rt + nrt)
    // per replica of the tile: histograms [nh][nf], P(M) then P(OP), P(SM)
    extern __shared__ unsigned int s_hist[];
    const int R = a.R, nf = a.nf;
    const int nh = a.obs ? 3 : 1;
    const int r0 = blockIdx.y * a.rt;
    const int nrt = min(a.rt, R - r0);
    for (int i = threadIdx.x; i < nrt * nh * nf; i += blockDim.x) s_hist[i] = 0u;
    __syncthreads();
    const float m_min = (float)a.m_min, scale = (float)((double)(nf - 1) / (a.m_max - a.m_min));
    const long long total = (long long)a.ncell * nrt;
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < total;
         it += (long long)gridDim.x * blockDim.x) {
        const int cell = (int)(it / nrt), rr = (int)(it % nrt), r = r0 + rr;
        float mx = 0.f, my = 0.f, mz = 0.f, op = 0.f, qx = 0.f, qy = 0.f, qz = 0.f;
        for (int at = 0; at < a.num_atoms; ++at) {
            const int p = __ldg(a.inv + cell * a.num_atoms + at);
            const size_t idx = (size_t)p * R + r;
            const float sx = a.sx[idx], sy = a.sy[idx], sz = a.sz[idx];
            mx += sx; my += sy; mz += sz;
            if (a.obs) obs_add(sx, sy, sz, __ldg(a.obs_atom + at), op, qx, qy, qz);
        }
        unsigned int *hr = s_hist + (size_t)rr * nh * nf;
        if (a.count_m) atomicAdd(hr + (pm_bin(mx, my, mz, m_min, scale, nf) - 1), 1u);
        if (a.obs & 1) atomicAdd(hr + nf + (pm_bin_value(op, m_min, scale, nf) - 1), 1u);
        if (a.obs & 2) atomicAdd(hr + 2 * nf + (pm_bin(qx, qy, qz, m_min, scale, nf) - 1), 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nrt * nh * nf; i += blockDim.x) {
        const unsigned int c = s_hist[i];
        if (c) {
            const int rr = i / (nh * nf), k = (i / nf) % nh, f = i % nf;
            const int t = a.temp_of[r0 + rr];
            if (k == 0) atomicAdd(a.counts + (size_t)t * nf + f, (unsigned long long)c);
            else atomicAdd(a.obs_counts + ((size_t)t * 2 + (k - 1)) * nf + f, (unsigned long long)c);
        }
    }
}

// ---------------------------------------------------------------------------
// pt_swap on labels: pairs (a, a+1), a = start0, start0+2, ...; one thread.
// x = (1/T_a - 1/T_{a+1}) (E_a - E_{a+1}) with the running energies; accept
// if x > 0 or u < exp(x).  The replicas keep their spins; the slot->replica
// map (the reference's `map`) and replica->slot map are exchanged.
// ---------------------------------------------------------------------------
__global__ void k_pt_swap(PtSwapArgs a)
{
    // pairs are disjoint, one thread each; slots form groups of `group`
    // consecutive temperatures (independent lattices) and pairs never cross
    // a group boundary
    uint32_t idx_lo = a.idx_lo, idx_hi = a.idx_hi;
    int start0 = a.start0;
    if (a.ctr) {
        const unsigned long long idx = (((unsigned long long)a.idx_hi << 32) | a.idx_lo) + a.ctr[1];
        idx_lo = (uint32_t)idx; idx_hi = (uint32_t)(idx >> 32);
        start0 = (int)((a.ctr[3] + (unsigned long long)a.unit_off + 1ull) % 2ull);
    }
    const int per_group = a.group / 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = i / per_group, k = i % per_group;
    if (g >= a.R / a.group) return;
    const int sl = start0 + 2 * k;
    if (sl + 1 >= a.group) return;
    const int s = g * a.group + sl;
    const int ra = a.repl_at[s], rb = a.repl_at[s + 1];
    const double x = (a.inv_t[s] - a.inv_t[s + 1]) * (a.e_run[ra] - a.e_run[rb]);
    a.num_swaps[2 * s] += 1;
    a.num_swaps[2 * (s + 1)] += 1;
    bool swap = x > 0.0;
    if (!swap) {
        const Philox4 v = philox4x32_10((uint32_t)s, idx_lo, idx_hi, 0xFFFFFFFFu, a.key0, a.key1);
        swap = u53(v.x, v.y) < exp(x);
    }
    if (swap) {
        a.repl_at[s] = rb; a.repl_at[s + 1] = ra;
        a.temp_of[rb] = s; a.temp_of[ra] = s + 1;
        a.num_swaps[2 * s + 1] += 1;
        a.num_swaps[2 * (s + 1) + 1] += 1;
    }
}

// ---------------------------------------------------------------------------
// Start configurations: kind 0 ferro (0,0,m); kind 1 rand with
// theta = pi*u1, phi = 2 pi*u2 (mcarlo.F90:279-293), one configuration for
// all replicas as pt.F90:448-459 does.
// ---------------------------------------------------------------------------
// Values e0 .. e0+n-1 of spin_matrix(3, N, slots) (reference site order, slot t
// holding replica repl_at[t]; FP32 staged chunks, or the caller's FP64 array) ->
// the FP32 state, and back.  One thread per value of the chunk, reading or
// writing it contiguously.
template <class T>
__global__ void k_spins_in(const T *stage, const int32_t *inv, const int32_t *repl_at, float *sx, float *sy, float *sz,
                           int N, int R, long long e0, long long n)
{
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long e = e0 + k, ti = e / 3;
        const int c = (int)(e - 3 * ti), t = (int)(ti / N), i = (int)(ti - (long long)t * N);
        const size_t o = (size_t)inv[i] * R + repl_at[t];
        float *dst = c == 0 ? sx : (c == 1 ? sy : sz);
        dst[o] = (float)stage[k];
    }
}

template <class T>
__global__ void k_spins_out(T *stage, const int32_t *inv, const int32_t *repl_at, const float *sx, const float *sy,
                            const float *sz, int N, int R, long long e0, long long n)
{
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long e = e0 + k, ti = e / 3;
        const int c = (int)(e - 3 * ti), t = (int)(ti / N), i = (int)(ti - (long long)t * N);
        const size_t o = (size_t)inv[i] * R + repl_at[t];
        const float *src = c == 0 ? sx : (c == 1 ? sy : sz);
        stage[k] = (T)src[o];
    }
}

__global__ void k_init_spins(const int32_t *perm, const float *mag, float *sx, float *sy, float *sz,
                             int N, int R, int kind, uint32_t k0, uint32_t k1)
{
    const long long total = (long long)N * R;
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < total;
         it += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(it / R);
        const float m = mag[p];
        float x = 0.f, y = 0.f, z = m;
        if (kind == 1) {
            const Philox4 v = philox4x32_10((uint32_t)perm[p], 0xFFFFFFFEu, 0u, 0u, k0, k1);
            const double u1 = (double)v.x * (1.0 / 4294967296.0), u2 = (double)v.y * (1.0 / 4294967296.0);
            double st, ct, sp, cp;
            sincospi(u1, &st, &ct);
            sincospi(2.0 * u2, &sp, &cp);
            x = (float)(m * st * cp); y = (float)(m * st * sp); z = (float)(m * ct);
        }
        sx[it] = x; sy[it] = y; sz[it] = z;
    }
}

// ---------------------------------------------------------------------------
// Host-side launchers
// ---------------------------------------------------------------------------
static int grid_for(long long items, int threads, int max_blocks)
{
    long long b = (items + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > max_blocks) b = max_blocks;
    return (int)b;
}

int sweep_blocks(long long max_items, int R, int max_blocks)
{
    const int threads = 256;
    int blocks = grid_for(max_items, threads, max_blocks);
    // the stride must hold at least one copy of every replica
    const int need = (R + threads - 1) / threads;
    return blocks < need ? need : blocks;
}

cudaError_t launch_fold(const FoldArgs &a, cudaStream_t st)
{
    k_fold<<<a.R, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sweep(const SweepArgs &a, bool hb, bool hd, int blocks, cudaStream_t st)
{
    const int threads = 256;
    if (hb && hd) k_sweep_ell<true, true><<<blocks, threads, 0, st>>>(a);
    else if (hb) k_sweep_ell<true, false><<<blocks, threads, 0, st>>>(a);
    else if (hd) k_sweep_ell<false, true><<<blocks, threads, 0, st>>>(a);
    else k_sweep_ell<false, false><<<blocks, threads, 0, st>>>(a);
    return cudaGetLastError();
}

int energy_blocks(int N, int R, int max_blocks)
{
    const int threads = 256;
    int blocks = grid_for((long long)N * R, threads, max_blocks);
    const int need = (R + threads - 1) / threads;
    return blocks < need ? need : blocks;
}

cudaError_t launch_energy(const EnergyArgsHost &h, double *out_e, double *out_m, int blocks, cudaStream_t st)
{
    EnergyArgs a;
    a.nnb = h.nnb; a.nbr = h.nbr; a.J = h.J; a.B = h.B; a.Dx = h.Dx; a.Dy = h.Dy; a.Dz = h.Dz;
    a.perm = h.perm; a.si = h.si; a.fld = h.fld; a.sx = h.sx; a.sy = h.sy; a.sz = h.sz;
    a.scratch = h.scratch; a.N = h.N; a.R = h.R; a.num_atoms = h.num_atoms;
    const bool hb = h.B != nullptr, hd = h.Dx != nullptr;
    if (hb && hd) k_energy_part<true, true><<<blocks, 256, 0, st>>>(a);
    else if (hb) k_energy_part<true, false><<<blocks, 256, 0, st>>>(a);
    else if (hd) k_energy_part<false, true><<<blocks, 256, 0, st>>>(a);
    else k_energy_part<false, false><<<blocks, 256, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_energy_reduce<<<h.R, 256, 0, st>>>(h.scratch, blocks, h.R, out_e, out_m);
    return cudaGetLastError();
}

cudaError_t launch_obs(const ObsArgs &a, double *out_op, double *out_sm, int blocks, cudaStream_t st)
{
    k_obs_part<<<blocks, 256, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_energy_reduce<<<a.R, 256, 0, st>>>(a.scratch, blocks, a.R, out_op, out_sm);
    return cudaGetLastError();
}

cudaError_t launch_spincorr(const ScArgs &a, int blocks, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    const int npass = (a.B + 1) / 2;
    k_sc_part<<<dim3(blocks, npass), 256, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_sc_reduce<<<dim3(a.R, npass), 256, 0, st>>>(a, blocks);
    return cudaGetLastError();
}

cudaError_t launch_sf_phases(const SfArgs &a, float2 *out, cudaStream_t st)
{
    const long long n = (long long)a.N * a.nq;
    if (n <= 0) return cudaSuccess;
    k_sf_phases<<<grid_for(n, 256, 65536), 256, 0, st>>>(a, out);
    return cudaGetLastError();
}

cudaError_t launch_sfactor(const SfArgs &a, int num_sms, cudaStream_t st)
{
    if (a.nq <= 0) return cudaSuccess;
    const dim3 big((a.nq + 63) / 64, (a.R + 15) / 16), small((a.nq + 7) / 8, (a.R + 7) / 8);
    if ((long long)big.x * big.y >= num_sms) {
        if (a.phase) k_sf_part<64, 16, 4, 3, 16, true><<<big, 256, 0, st>>>(a);
        else k_sf_part<64, 16, 4, 3, 16, false><<<big, 256, 0, st>>>(a);
    } else {
        if (a.phase) k_sf_part<8, 8, 1, 1, 64, true><<<small, 192, 0, st>>>(a);
        else k_sf_part<8, 8, 1, 1, 64, false><<<small, 192, 0, st>>>(a);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const long long n = (long long)a.nq * a.R;
    k_sf_finish<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_local_terms(const EnergyArgsHost &h, float *g, float *q, cudaStream_t st)
{
    EnergyArgs a;
    a.nnb = h.nnb; a.nbr = h.nbr; a.J = h.J; a.B = h.B; a.Dx = h.Dx; a.Dy = h.Dy; a.Dz = h.Dz;
    a.perm = h.perm; a.si = h.si; a.fld = h.fld; a.sx = h.sx; a.sy = h.sy; a.sz = h.sz;
    a.scratch = nullptr; a.N = h.N; a.R = h.R; a.num_atoms = h.num_atoms;
    const int blocks = grid_for((long long)h.N * h.R, 256, 4096);
    const bool hb = h.B != nullptr, hd = h.Dx != nullptr;
    if (hb && hd) k_local_terms<true, true><<<blocks, 256, 0, st>>>(a, g, q);
    else if (hb) k_local_terms<true, false><<<blocks, 256, 0, st>>>(a, g, q);
    else if (hd) k_local_terms<false, true><<<blocks, 256, 0, st>>>(a, g, q);
    else k_local_terms<false, false><<<blocks, 256, 0, st>>>(a, g, q);
    return cudaGetLastError();
}

cudaError_t launch_measure(const MeasureArgs &a, cudaStream_t st)
{
    k_measure<<<(a.R + 127) / 128, 128, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pm(const PmArgs &a0, int max_blocks, cudaStream_t st)
{
    PmArgs a = a0;
    // replica tile: its [rt][nh][nf] histograms fit in 96 KB of shared memory
    const size_t cap = 96 * 1024;
    const int nh = a.obs ? 3 : 1;
    a.rt = (int)(cap / ((size_t)nh * a.nf * sizeof(unsigned int)));
    if (a.rt < 1) return cudaErrorInvalidValue;
    if (a.rt > a.R) a.rt = a.R;
    a.use_shared = 1;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        e = cudaFuncSetAttribute(k_pm_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    const int tiles = (a.R + a.rt - 1) / a.rt;
    // few blocks, many items each: the flush of the block histograms is a
    // global atomic per non-empty bin, so fewer blocks means less contention
    const int cap_blocks = max_blocks / 8 / tiles > 0 ? max_blocks / 8 / tiles : 1;
    int bx = grid_for((long long)a.ncell * a.rt, 256, cap_blocks);
    const size_t smem = (size_t)a.rt * nh * a.nf * sizeof(unsigned int);
    k_pm_hist<<<dim3(bx, tiles), 256, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pt_swap(const PtSwapArgs &a, cudaStream_t st)
{
    if (a.group < 2 || a.R % a.group != 0) return a.group == 1 ? cudaSuccess : cudaErrorInvalidValue;
    const int threads = (a.R / a.group) * (a.group / 2);
    k_pt_swap<<<(threads + 127) / 128, 128, 0, st>>>(a);
    return cudaGetLastError();
}

__global__ void k_bump(unsigned long long *ctr, unsigned long long d0, unsigned long long d1, unsigned long long d2,
                       unsigned long long d3)
{
    ctr[0] += d0; ctr[1] += d1; ctr[2] += d2; ctr[3] += d3;
}

cudaError_t launch_bump(unsigned long long *ctr, const unsigned long long d[4], cudaStream_t st)
{
    k_bump<<<1, 1, 0, st>>>(ctr, d[0], d[1], d[2], d[3]);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_spins_in(const T *stage, const int32_t *inv, const int32_t *repl_at, float *sx, float *sy, float *sz,
                            int N, int R, long long e0, long long n, cudaStream_t st)
{
    k_spins_in<T><<<grid_for(n, 256, 4096), 256, 0, st>>>(stage, inv, repl_at, sx, sy, sz, N, R, e0, n);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_spins_out(T *stage, const int32_t *inv, const int32_t *repl_at, const float *sx, const float *sy,
                             const float *sz, int N, int R, long long e0, long long n, cudaStream_t st)
{
    k_spins_out<T><<<grid_for(n, 256, 4096), 256, 0, st>>>(stage, inv, repl_at, sx, sy, sz, N, R, e0, n);
    return cudaGetLastError();
}

template cudaError_t launch_spins_in<float>(const float *, const int32_t *, const int32_t *, float *, float *, float *, int,
                                            int, long long, long long, cudaStream_t);
template cudaError_t launch_spins_in<double>(const double *, const int32_t *, const int32_t *, float *, float *, float *, int,
                                             int, long long, long long, cudaStream_t);
template cudaError_t launch_spins_out<float>(float *, const int32_t *, const int32_t *, const float *, const float *,
                                             const float *, int, int, long long, long long, cudaStream_t);
template cudaError_t launch_spins_out<double>(double *, const int32_t *, const int32_t *, const float *, const float *,
                                              const float *, int, int, long long, long long, cudaStream_t);

cudaError_t launch_init_spins(const int32_t *perm, const float *mag, float *sx, float *sy, float *sz,
                              int N, int R, int kind, uint64_t seed, cudaStream_t st)
{
    const int blocks = grid_for((long long)N * R, 256, 4096);
    k_init_spins<<<blocks, 256, 0, st>>>(perm, mag, sx, sy, sz, N, R, kind, (uint32_t)seed,
                                         (uint32_t)(seed >> 32));
    return cudaGetLastError();
}

}  // namespace esp
