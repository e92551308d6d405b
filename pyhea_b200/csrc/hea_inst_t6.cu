// Kernel instances for 6 species.
#include "hea_inst.cuh"

namespace hea {
const KernelSet &kernel_set_t6() { return kernel_set<6>(); }
}  // namespace hea
