// Instantiations of the cluster-resident sweep: parity-class lattices whose
// stencil rows stay in global memory.  The variants are compiled in several
// translation units side by side.
#include "esp_cluster_kernel.cuh"

namespace esp {

ClusterKernel cluster_kernel_classes_global(const ClusterVariant &v, int csize)
{
    if (csize > 1) return v.pairs ? cluster_kernel_t<2, false, false, true>(v) : cluster_kernel_t<1, false, false, true>(v);
    return v.pairs ? cluster_kernel_t<2, false, false, false>(v) : cluster_kernel_t<1, false, false, false>(v);
}

}  // namespace esp
