// Instances of the kernel templates, group CLUSTER_SHORT (gf_inst.cuh).
#define GFC_TEMPLATES_ONLY
#include "gf_inst.cuh"

namespace gfc {
GFC_INST_CLUSTER_SHORT(template __global__)
}  // namespace gfc
