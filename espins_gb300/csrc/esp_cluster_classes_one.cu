// Instantiations of the cluster-resident sweep: parity-class lattices, one CTA per replica.  The
// variants are compiled in several translation units side by side.
#include "esp_cluster_kernel.cuh"

namespace esp {

ClusterKernel cluster_kernel_classes_one(const ClusterVariant &v)
{
    if (v.helpers) return cluster_kernel_t<1, false, true, false, true>(v);
    return v.pairs ? cluster_kernel_t<2, false, true, false>(v) : cluster_kernel_t<1, false, true, false>(v);
}

}  // namespace esp
