// Kernel instances for 5 species.
#include "hea_inst.cuh"

namespace hea {
const KernelSet &kernel_set_t5() { return kernel_set<5>(); }
}  // namespace hea
