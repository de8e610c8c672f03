// Instances of the kernel templates, group ROW_PAIR (gf_inst.cuh).
#define GFC_TEMPLATES_ONLY
#include "gf_inst.cuh"

namespace gfc {
GFC_INST_ROW_PAIR(template __global__)
}  // namespace gfc
