// Instances of the kernel templates, group PCOL (gf_inst.cuh).
#define GFC_TEMPLATES_ONLY
#include "gf_inst.cuh"

namespace gfc {
GFC_INST_PCOL(template __global__)
}  // namespace gfc
