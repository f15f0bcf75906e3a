// RLWE -> RLWE key switching of a batch (lib/src/operators/rlwe_conversion.cpp:224-249), digit-staged:
// the words of ks_kernel<.., kKsRlwe, ..> with all digits' transforms before the products.
//
// What bounds it: the integer pipes (a digit's transform is 32 instructions a butterfly), and with
// them, in the row-by-row form, the latency of the transforms' passes: its running sums and the next
// key words keep 118 registers a thread, so one block of 16 warps per SM at N = 2048. Here a thread's
// own slots of every digit but the last wait in shared memory (no barrier: nobody else reads
// them), the forward loop needs 64 registers, and 1024 threads are resident per SM. The products
// of a slot are then summed exactly over the digits (WideAcc) and reduced once. Microseconds for
// 4096 ciphertexts (row by row -> here): N = 1024, l = 4 189 -> 162; N = 2048, l = 4 426 -> 338, l = 2
// 269 -> 195; N = 4096, l = 3 832 -> 575; one ciphertext, N = 2048, l = 4 18.6 -> 16.5.
#pragma once

#include "ks_kernels.cuh"

namespace tp {

// Shared memory of a block, in words: forward twiddles, two exchange buffers, digits - 1 rows.
__host__ __device__ constexpr size_t ks_rlwe_smem_words(int logn, int dl) { return (size_t)(3 + dl - 1) << logn; }

template <int LOGN, int DL>
__global__ void __launch_bounds__(1 << (LOGN - 2), 1 << (12 - LOGN)) ks_rlwe_kernel(const KsKernelParams prm) {
    constexpr int N = 1 << LOGN, T = N / 4;
    static_assert(LOGN <= 12, "one block per ciphertext");
    extern __shared__ __align__(16) uint64_t smem[];
    uint64_t* tw = smem;
    uint64_t* buf0 = smem + N;
    uint64_t* buf1 = smem + 2 * N;
    uint64_t* rows = smem + 3 * N;  // digit d of this thread's slot pair jp at d N + (jp T + t) 2
    const int t = threadIdx.x;
    for (int i = t; i < N; i += T) tw[i] = prm.tw_fwd[i];
    __syncthreads();
    int sel = 0;
    for (uint64_t it = blockIdx.x; it < prm.items; it += gridDim.x) {
        const uint64_t* in = prm.in + it * prm.in_stride;
        uint64_t* out = prm.out + it * prm.out_stride;
        uint64_t a[4], x[1][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] = gl_add(in[t + j * T], prm.corr);
#pragma unroll 1
        for (int d = 0; d < DL; ++d) {
            const uint32_t sh = prm.dshift[d];
            const uint64_t mk = prm.dmask[d], dl = prm.ddelta[d];
            if (prm.small_digits) {
                ntt_pass0_digit(a, sh, mk, dl, prm.small_digits, x[0]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) x[0][j] = gl_sub((a[j] >> sh) & mk, dl);
                fwd_pass_math<LOGN, 0, 1, 2, 0, true>(x, t, tw);
            }
            ntt_forward_after_pass0<LOGN, 1, 2, 0, true>(x, t, sel ? buf1 : buf0, tw);
            sel ^= 1;
            if (d + 1 < DL) {
#pragma unroll
                for (int jp = 0; jp < 2; ++jp)
                    *reinterpret_cast<ulonglong2*>(rows + d * N + (jp * T + t) * 2) =
                        make_ulonglong2(x[0][2 * jp], x[0][2 * jp + 1]);
            }
        }
        // out -= KS; out.B += in.B (rlwe_conversion.cpp:243-248); slots 4 t + 2 jp and the next
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                ulonglong2* o = reinterpret_cast<ulonglong2*>(out + c * N + 4 * t + 2 * jp);
                ulonglong2 v = *o, kv[DL];
#pragma unroll
                for (int d = 0; d < DL; ++d)
                    kv[d] = __ldg(reinterpret_cast<const ulonglong2*>(prm.key + (uint64_t)d * (2 * N) +
                                                                      ((c * 2 + jp) * T + t) * 2));
                WideAcc s0, s1;
                wide_zero(s0);
                wide_zero(s1);
#pragma unroll
                for (int d = 0; d < DL; ++d) {
                    const ulonglong2 r = d + 1 < DL
                                             ? *reinterpret_cast<const ulonglong2*>(rows + d * N + (jp * T + t) * 2)
                                             : make_ulonglong2(x[0][2 * jp], x[0][2 * jp + 1]);
                    wide_mad(s0, r.x, kv[d].x);
                    wide_mad(s1, r.y, kv[d].y);
                }
                v.x = gl_sub(v.x, wide_reduce(s0));
                v.y = gl_sub(v.y, wide_reduce(s1));
                if (c == 1) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(in + N + 4 * t + 2 * jp);
                    v.x = gl_add(v.x, b.x);
                    v.y = gl_add(v.y, b.y);
                }
                *o = v;
            }
        }
    }
}

}  // namespace tp
