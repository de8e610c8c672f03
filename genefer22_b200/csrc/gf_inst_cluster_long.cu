// Instances of the kernel templates, group CLUSTER_LONG (gf_inst.cuh).
#define GFC_TEMPLATES_ONLY
#include "gf_inst.cuh"

namespace gfc {
GFC_INST_CLUSTER_LONG(template __global__)
}  // namespace gfc
