// Instances of the kernel templates, group SMALL (gf_inst.cuh).
#define GFC_TEMPLATES_ONLY
#include "gf_inst.cuh"

namespace gfc {
GFC_INST_SMALL(template __global__)
}  // namespace gfc
