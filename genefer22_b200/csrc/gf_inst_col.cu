// Instances of the kernel templates, group COL (gf_inst.cuh).
#define GFC_TEMPLATES_ONLY
#include "gf_inst.cuh"

namespace gfc {
GFC_INST_COL(template __global__)
}  // namespace gfc
