// Instances of the kernel templates, group COLR (gf_inst.cuh).
#define GFC_TEMPLATES_ONLY
#include "gf_inst.cuh"

namespace gfc {
GFC_INST_COLR(template __global__)
}  // namespace gfc
