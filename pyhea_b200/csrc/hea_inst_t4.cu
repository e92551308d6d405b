// Kernel instances for 4 species.
#include "hea_inst.cuh"

namespace hea {
const KernelSet &kernel_set_t4() { return kernel_set<4>(); }
}  // namespace hea
