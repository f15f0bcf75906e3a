// Double-precision key-switch kernels (compiled as a separate unit).
#include "fft_host.h"
#include "ks_fft_kernel.cuh"

namespace tp {
namespace {

template <int LOGN>
const void* pick(uint32_t digits, int limbs) {
    switch (digits * 10 + limbs) {
        case 23: return (const void*)ks_fft_kernel<LOGN, 2, 3>;
        case 24: return (const void*)ks_fft_kernel<LOGN, 2, 4>;
        case 33: return (const void*)ks_fft_kernel<LOGN, 3, 3>;
        case 34: return (const void*)ks_fft_kernel<LOGN, 3, 4>;
        case 43: return (const void*)ks_fft_kernel<LOGN, 4, 3>;
        case 44: return (const void*)ks_fft_kernel<LOGN, 4, 4>;
        default: return nullptr;
    }
}

}  // namespace

const void* ks_fft_kernel_ptr(int logn, uint32_t digits, int limbs) {
    return logn == 10 ? pick<10>(digits, limbs) : logn == 11 ? pick<11>(digits, limbs) : nullptr;
}

}  // namespace tp
