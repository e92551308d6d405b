// Kernel instances for 3 species.
#include "hea_inst.cuh"

namespace hea {
const KernelSet &kernel_set_t3() { return kernel_set<3>(); }
}  // namespace hea
