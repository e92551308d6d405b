// hea_kernels.h -- the search kernels of one species count as function tables.
// Each species count's instances are compiled in a translation unit of their
// own (hea_inst_t2.cu .. hea_inst_t6.cu), so the library's units build side by side.
#pragma once
#include "hea_search.cuh"

namespace hea {

using GenFn = void (*)(const SearchConst, const GenArgs);
using McFn = void (*)(const SearchConst, const McArgs);
using LGenFn = void (*)(const SearchConst, uint8_t *, const int32_t *, uint32_t);
using LRecFn = void (*)(const SearchConst, const int4 *, const uint8_t *, const int32_t *, int32_t *, uint64_t *);
using LFitFn = void (*)(const SearchConst, const int32_t *, int, const int32_t *, double *);

struct KernelSet {
    GenFn gen[kMaxShells + 1];  // by shell count
    LGenFn lgen;
    LRecFn lrec[kMaxShells + 1];
    LFitFn lfit[kMaxShells + 1];
    // local search for the table's padded shell layout (int4 chunks per shell) or implicit neighbours
    McFn (*mc)(int c0, int c1, int c2, int S, bool implicit);
    McFn (*mc_large)(int c0, int c1, int c2, int S, bool implicit);
};

const KernelSet &kernel_set_t2();
const KernelSet &kernel_set_t3();
const KernelSet &kernel_set_t4();
const KernelSet &kernel_set_t5();
const KernelSet &kernel_set_t6();

}  // namespace hea
