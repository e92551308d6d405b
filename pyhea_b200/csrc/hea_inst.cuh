// hea_inst.cuh -- the kernel instances of species count T (one translation
// unit per T includes this) as a KernelSet.
#pragma once
#include "hea_kernels.h"
#include "hea_large.cuh"

namespace hea {

// Local-search kernel for species count T and the table's padded shell layout:
// the layouts of the FCC/BCC shell sets (in int4 chunks per shell) have their
// loads unrolled; any other table uses the runtime-layout instance.
template <int T>
McFn pick_mc(int c0, int c1, int c2, int S, bool implicit)
{
    if (implicit) return S == 1 ? mc_kernel<T, ImplicitShells<1>> : S == 2 ? mc_kernel<T, ImplicitShells<2>>
                                                                          : mc_kernel<T, ImplicitShells<3>>;
    if (c0 == 2 && c1 == 0 && c2 == 0) return mc_kernel<T, Shells<2, 0, 0>>;  // BCC, 1 shell
    if (c0 == 2 && c1 == 2 && c2 == 0) return mc_kernel<T, Shells<2, 2, 0>>;  // BCC, 2 shells
    if (c0 == 2 && c1 == 2 && c2 == 3) return mc_kernel<T, Shells<2, 2, 3>>;  // BCC 8/6/12
    if (c0 == 3 && c1 == 0 && c2 == 0) return mc_kernel<T, Shells<3, 0, 0>>;  // FCC, 1 shell
    if (c0 == 3 && c1 == 2 && c2 == 0) return mc_kernel<T, Shells<3, 2, 0>>;  // FCC, 2 shells
    if (c0 == 3 && c1 == 2 && c2 == 3) return mc_kernel<T, Shells<3, 2, 3>>;  // FCC 12/6/12
    if (c0 == 3 && c1 == 2 && c2 == 6) return mc_kernel<T, Shells<3, 2, 6>>;  // FCC 12/6/24
    if (S == 1) return mc_kernel<T, RuntimeShells<1>>;
    if (S == 2) return mc_kernel<T, RuntimeShells<2>>;
    return mc_kernel<T, RuntimeShells<3>>;
}

// The same choice for the HBM-occupancy (cluster) search.
template <int T>
McFn pick_mc_large(int c0, int c1, int c2, int S, bool implicit)
{
    if (implicit)
        return S == 1 ? mc_large_kernel<T, ImplicitShells<1>>
                      : S == 2 ? mc_large_kernel<T, ImplicitShells<2>> : mc_large_kernel<T, ImplicitShells<3>>;
    if (c0 == 2 && c1 == 2 && c2 == 3) return mc_large_kernel<T, Shells<2, 2, 3>>;
    if (c0 == 3 && c1 == 2 && c2 == 3) return mc_large_kernel<T, Shells<3, 2, 3>>;
    if (c0 == 3 && c1 == 2 && c2 == 6) return mc_large_kernel<T, Shells<3, 2, 6>>;
    if (S == 1) return mc_large_kernel<T, RuntimeShells<1>>;
    if (S == 2) return mc_large_kernel<T, RuntimeShells<2>>;
    return mc_large_kernel<T, RuntimeShells<3>>;
}

template <int T>
const KernelSet &kernel_set()
{
    static const KernelSet ks = {
        {nullptr, generate_kernel<T, 1>, generate_kernel<T, 2>, generate_kernel<T, 3>},
        large_generate_kernel<T>,
        {nullptr, large_recount_kernel<T, 1>, large_recount_kernel<T, 2>, large_recount_kernel<T, 3>},
        {nullptr, large_fitness_kernel<T, 1>, large_fitness_kernel<T, 2>, large_fitness_kernel<T, 3>},
        pick_mc<T>,
        pick_mc_large<T>,
    };
    return ks;
}

}  // namespace hea
