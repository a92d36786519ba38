// Launchers of the cluster-resident sweep (esp_cluster_kernel.cuh), and the
// transposes between the spin arrays and its slabs.
#include "esp_cluster.h"

namespace esp {

// Sites of rank q and the first of them in a replica's slab order.
__device__ __forceinline__ int slab_sites(const SlabArgs &a, int q) { return q < a.nA ? a.n_big : a.n_small; }
__device__ __forceinline__ size_t slab_site0(const SlabArgs &a, int q)
{
    return (size_t)q * a.n_big - (size_t)max(0, q - a.nA) * (a.n_big - a.n_small);
}

// grid (n_local / 32, cs, R / 32) rounded up, blocks of 32 x 8 threads
__global__ void __launch_bounds__(256) k_to_slabs(const SlabArgs a)
{
    __shared__ float t[3][32][33];   // [component][replica][site]
    __shared__ int rows[32];
    const int l0 = blockIdx.x * 32, q = blockIdx.y, r0 = blockIdx.z * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int nl = slab_sites(a, q);
    const size_t s0 = slab_site0(a, q);
    if (ty == 0) rows[tx] = l0 + tx < nl ? __ldg(a.loc2p + s0 + l0 + tx) : 0;
    __syncthreads();
    for (int j = ty; j < 32; j += 8)
        if (l0 + j < nl && r0 + tx < a.R) {
            const size_t g = (size_t)rows[j] * a.R + r0 + tx;
            t[0][tx][j] = a.sx[g]; t[1][tx][j] = a.sy[g]; t[2][tx][j] = a.sz[g];
        }
    __syncthreads();
    for (int j = ty; j < 32; j += 8)
        if (r0 + j < a.R && l0 + tx < nl) {
            float *o = a.slab + ((size_t)(r0 + j) * a.N + s0 + l0 + tx) * 3;
            o[0] = t[0][j][tx]; o[1] = t[1][j][tx]; o[2] = t[2][j][tx];
        }
}

__global__ void __launch_bounds__(256) k_from_slabs(const SlabArgs a)
{
    __shared__ float t[3][32][33];   // [component][replica][site]
    __shared__ int rows[32];
    const int l0 = blockIdx.x * 32, q = blockIdx.y, r0 = blockIdx.z * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int nl = slab_sites(a, q);
    const size_t s0 = slab_site0(a, q);
    if (ty == 0) rows[tx] = l0 + tx < nl ? __ldg(a.loc2p + s0 + l0 + tx) : 0;
    for (int j = ty; j < 32; j += 8)
        if (r0 + j < a.R && l0 + tx < nl) {
            const float *i = a.slab + ((size_t)(r0 + j) * a.N + s0 + l0 + tx) * 3;
            t[0][j][tx] = i[0]; t[1][j][tx] = i[1]; t[2][j][tx] = i[2];
        }
    __syncthreads();
    for (int j = ty; j < 32; j += 8)
        if (l0 + j < nl && r0 + tx < a.R) {
            const size_t g = (size_t)rows[j] * a.R + r0 + tx;
            a.sx[g] = t[0][tx][j]; a.sy[g] = t[1][tx][j]; a.sz[g] = t[2][tx][j];
        }
}

cudaError_t launch_to_slabs(const SlabArgs &a, cudaStream_t st)
{
    const dim3 grid((a.n_big + 31) / 32, a.cs, (a.R + 31) / 32), block(32, 8);
    k_to_slabs<<<grid, block, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_from_slabs(const SlabArgs &a, cudaStream_t st)
{
    const dim3 grid((a.n_big + 31) / 32, a.cs, (a.R + 31) / 32), block(32, 8);
    k_from_slabs<<<grid, block, 0, st>>>(a);
    return cudaGetLastError();
}

size_t cluster_smem_bytes(int n_local, int nf, int nhist, size_t table_bytes)
{
    return ((table_bytes + 15) & ~(size_t)15) + (size_t)((nhist * nf + 3) & ~3) * sizeof(unsigned int) +
           (size_t)(kClusterRedDoubles + kClusterAccDoubles) * sizeof(double) + (size_t)3 * n_local * sizeof(float);
}

namespace {

ClusterKernel cluster_kernel(const ClusterVariant &v, int csize)
{
    if (v.general) return csize > 1 ? cluster_kernel_general_many(v) : cluster_kernel_general_one(v);
    if (!v.rows_smem) return cluster_kernel_classes_global(v, csize);
    return csize > 1 ? cluster_kernel_classes_many(v) : cluster_kernel_classes_one(v);
}

}  // namespace

bool cluster_threads_ok(int nt, int S) { return (nt == 256 && S == 1) || (nt == 512 && (S == 1 || S == 2)); }

cudaError_t cluster_configure(const ClusterVariant &v, size_t smem, int csize)
{
    const ClusterKernel k = cluster_kernel(v, csize);
    cudaError_t e = allow_max_dynamic_smem(reinterpret_cast<const void *>(k), smem);
    if (e == cudaSuccess && csize > 8) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

int cluster_max_active(const ClusterVariant &v, int csize, int nt, size_t smem, int R)
{
    const ClusterKernel k = cluster_kernel(v, csize);
    if (cluster_configure(v, smem, csize) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(csize * R, 1, 1);
    cfg.blockDim = dim3(nt, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t launch_cluster(const ClusterArgs &a, const ClusterVariant &v, int csize, int nt, size_t smem,
                           cudaStream_t st)
{
    if (nt < 32 || nt > kClusterThreads || nt % 32 != 0) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(csize * a.R, 1, 1);
    cfg.blockDim = dim3(nt, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, cluster_kernel(v, csize), a);
}

}  // namespace esp
