// Kernel instances for 2 species.
#include "hea_inst.cuh"

namespace hea {
const KernelSet &kernel_set_t2() { return kernel_set<2>(); }
}  // namespace hea
