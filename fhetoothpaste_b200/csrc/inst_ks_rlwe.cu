// Digit-staged RLWE key-switch kernels (compiled as a separate unit).
#include "dispatch.h"
#include "ks_rlwe_kernel.cuh"

namespace tp {
namespace {

template <int LOGN>
const void* pick(uint32_t digits) {
    switch (digits) {
        case 2: return (const void*)ks_rlwe_kernel<LOGN, 2>;
        case 3: return (const void*)ks_rlwe_kernel<LOGN, 3>;
        case 4: return (const void*)ks_rlwe_kernel<LOGN, 4>;
        default: return nullptr;
    }
}

}  // namespace

const void* ks_rlwe_kernel_ptr(int logn, uint32_t digits) {
    return logn == 10 ? pick<10>(digits) : logn == 11 ? pick<11>(digits) : logn == 12 ? pick<12>(digits) : nullptr;
}

}  // namespace tp
