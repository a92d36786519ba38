// Instantiations of the cluster-resident sweep: general lattices, one CTA per replica.  The
// variants are compiled in several translation units side by side.
#include "esp_cluster_kernel.cuh"

namespace esp {

ClusterKernel cluster_kernel_general_one(const ClusterVariant &v)
{
    if (v.helpers) return cluster_kernel_t<1, true, true, false, true>(v);
    return v.pairs ? cluster_kernel_t<2, true, true, false>(v) : cluster_kernel_t<1, true, true, false>(v);
}

}  // namespace esp
