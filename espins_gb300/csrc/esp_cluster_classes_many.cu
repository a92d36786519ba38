// Instantiations of the cluster-resident sweep: parity-class lattices, several CTAs per replica.  The
// variants are compiled in several translation units side by side.
#include "esp_cluster_kernel.cuh"

namespace esp {

ClusterKernel cluster_kernel_classes_many(const ClusterVariant &v)
{
    return v.pairs ? cluster_kernel_t<2, false, true, true>(v) : cluster_kernel_t<1, false, true, true>(v);
}

}  // namespace esp
