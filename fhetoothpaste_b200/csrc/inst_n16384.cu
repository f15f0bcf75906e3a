// Kernel instantiations for N = 16384: one rotation per cluster of 4 CTAs of 4096
// coefficients each (cluster_ntt.cuh; 1024 threads per CTA, 4 coefficients per
// thread), for the rotation (row-by-row multiply-accumulate: the digit stage does not
// fit beside 4096 coefficients) and the key-switching modes; compiled as a separate
// unit so the ring sizes build in parallel.
#include "br_kernels.cuh"
#include "dispatch.h"
#include "ks_kernels.cuh"
#include "misc_kernels.cuh"

namespace tp {

static_assert(br_cluster_logs(14) == 2, "cluster size of this unit");

const void* br_kernel_ptr_14(int variant, int loge, int dl, bool r4) {
    if (r4 || loge != 2 || dl != 0) return nullptr;
    switch (variant) {
        case kCggiBinary: return (const void*)br_kernel<14, kCggiBinary, 2, 0, 2>;
        case kCggiTernary: return (const void*)br_kernel<14, kCggiTernary, 2, 0, 2>;
        default: return (const void*)br_kernel<14, kBmmpBinary, 2, 0, 2>;
    }
}

const void* br_wide_kernel_ptr_14(int variant, int logs) {
    if (logs == 3)
        return variant == kCggiBinary    ? (const void*)br_kernel<14, kCggiBinary, 2, 0, 3, false, 2>
               : variant == kCggiTernary ? (const void*)br_kernel<14, kCggiTernary, 2, 0, 3, false, 2>
                                         : (const void*)br_kernel<14, kBmmpBinary, 2, 0, 3, false, 2>;
    return nullptr;
}

const void* ks_kernel_ptr_14(int mode, int loge) {
    if (loge != 2) return nullptr;  // clusters run with 4 coefficients per thread
    switch (mode) {
        case kKsRlwe: return (const void*)ks_kernel<14, kKsRlwe, 2, 2>;
        case kKsAuto: return (const void*)ks_kernel<14, kKsAuto, 2, 2>;
        case kKsMerge: return (const void*)ks_kernel<14, kKsMerge, 2, 2>;
        case kKsTrace: return (const void*)ks_kernel<14, kKsTrace, 2, 2>;
        default: return (const void*)ks_kernel<14, kKsSplit, 2, 2>;
    }
}

const void* ntt_kernel_ptr_14(bool forward) {
    return forward ? (const void*)ntt_cluster_kernel<14, true, 2>
                   : (const void*)ntt_cluster_kernel<14, false, 2>;
}

}  // namespace tp
