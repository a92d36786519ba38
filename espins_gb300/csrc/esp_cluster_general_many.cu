// Instantiations of the cluster-resident sweep: general lattices, several CTAs per replica.  The
// variants are compiled in several translation units side by side.
#include "esp_cluster_kernel.cuh"

namespace esp {

ClusterKernel cluster_kernel_general_many(const ClusterVariant &v)
{
    return v.pairs ? cluster_kernel_t<2, true, true, true>(v) : cluster_kernel_t<1, true, true, true>(v);
}

}  // namespace esp
