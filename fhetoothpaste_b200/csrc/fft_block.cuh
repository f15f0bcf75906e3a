// Exact negacyclic products over the integers with double-precision transforms.
//
// A gadget digit is a small integer polynomial and a key polynomial splits into a few
// balanced limbs (k = k_0 + k_1 B + k_2 B^2 ..., |k_i| <= B/2), so each coefficient of
// digit * limb mod X^N + 1 is an integer far below 2^51. A complex FFT in double
// precision gives it with an absolute error below 1/2 (the bound is checked for every
// key, fft_error_bound), so rounding to the nearest integer recovers it exactly, and the
// limbs recombine mod p to the very words the modular transforms give. A butterfly costs
// 6 to 8 FP64 instructions against 32 integer ones for a Goldilocks butterfly, and a
// transform has n = N/2 complex points instead of N words.
//
// Folding: z_j = a_j + i a_{j+n}, j < n, evaluated at the n roots of x^n = i, which are
// x_e = w^(1 + 4 brv(e)) with w = exp(2 pi i / 2N). X^n - i splits into X^(n/2) -+ r with
// r^2 = i and so on, as the modular transform does: every butterfly is (u + w v, u - w v)
// with one twiddle per block of a level, tw[m + b] for block b of the level with m blocks.
//
// One polynomial is transformed by n/16 threads, 16 complex points (64 registers) each,
// in three passes over an in-place shared-memory buffer: the first levels (3 or 4) on
// elements t + i n/16, then 3 levels inside blocks of 64 (4 inside blocks of 128 at n = 2048)
// and 3 levels inside blocks of 8.
// Twiddles of odd blocks are i times their even neighbour's and need no table entry.
#pragma once

#include <stdint.h>

#include "gl_arith.cuh"

namespace tp {

// First-pass twiddles (block index below 16), the same for every size; kernel parameters,
// so that the FP64 instructions read them as constant operands.
struct FftHead {
    double2 fwd[16];  // (cos, tan) of tw[k]
    double2 inv[16];  // (cos, sin) of tw[k]
};

// The later passes' tables (double2): pass 2 has 2^min(k-6, 4) blocks, pass 3 n/8, with four
// entries each (first level, second, third for the two even children) or, for a pass 2 of four
// levels, eight (and the four even grandchildren).
__host__ __device__ constexpr int fft_blocks2(int logk) { return 1 << (logk < 10 ? logk - 6 : 4); }
__host__ __device__ constexpr int fft_entries2(int logk) { return logk > 10 ? 8 : 4; }
__host__ __device__ constexpr int fft_table_len(int logk) {
    return fft_entries2(logk) * fft_blocks2(logk) + 4 * (1 << (logk - 3));
}

// Position of element e in a polynomial's buffer, in 16-byte units: the unit inside each
// 128-byte line is permuted so that every pass and the slot-wise reads are conflict-free.
__device__ __forceinline__ int fft_pos(int e) {
    const int line = e >> 3;
    return (line << 3) | ((e & 7) ^ (line & 7) ^ (((line >> 3) & 1) << 2));
}

// v *= (1 + i t): the butterfly's product up to the factor c that its FMAs apply.
__device__ __forceinline__ double2 fft_ratio(double2 v, double t) {
    return make_double2(fma(-t, v.y, v.x), fma(t, v.x, v.y));
}
// (u, v) <- (u + w v, u - w v), w = c (1 + i t): six FMAs.
__device__ __forceinline__ void fft_bfly(double2& u, double2& v, double2 ct) {
    const double2 y = fft_ratio(v, ct.y);
    v = make_double2(fma(-ct.x, y.x, u.x), fma(-ct.x, y.y, u.y));
    u = make_double2(fma(ct.x, y.x, u.x), fma(ct.x, y.y, u.y));
}
// The same with twiddle i w.
__device__ __forceinline__ void fft_bfly_i(double2& u, double2& v, double2 ct) {
    const double2 y = fft_ratio(v, ct.y);
    v = make_double2(fma(ct.x, y.y, u.x), fma(-ct.x, y.x, u.y));
    u = make_double2(fma(-ct.x, y.y, u.x), fma(ct.x, y.x, u.y));
}
// Backward: (u, v) <- (u + v, (u - v) conj(w)), w = (re, im).
__device__ __forceinline__ void fft_ibfly(double2& u, double2& v, double2 w) {
    const double dx = u.x - v.x, dy = u.y - v.y;
    u = make_double2(u.x + v.x, u.y + v.y);
    v = make_double2(fma(dx, w.x, dy * w.y), fma(dy, w.x, -(dx * w.y)));
}
// conj(i w) = -i conj(w).
__device__ __forceinline__ void fft_ibfly_i(double2& u, double2& v, double2 w) {
    const double dx = u.x - v.x, dy = u.y - v.y;
    u = make_double2(u.x + v.x, u.y + v.y);
    v = make_double2(fma(dy, w.x, -(dx * w.y)), -fma(dx, w.x, dy * w.y));
}

// Three levels on eight points (distances 4, 2, 1) inside one block, twiddles w[0] (first
// level), w[1] (second, block 2b), w[2], w[3] (third, blocks 4b and 4b + 2).
__device__ __forceinline__ void fft_radix8(double2 (&x)[8], const double2 (&w)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) fft_bfly(x[k], x[k + 4], w[0]);
    fft_bfly(x[0], x[2], w[1]);
    fft_bfly(x[1], x[3], w[1]);
    fft_bfly_i(x[4], x[6], w[1]);
    fft_bfly_i(x[5], x[7], w[1]);
    fft_bfly(x[0], x[1], w[2]);
    fft_bfly_i(x[2], x[3], w[2]);
    fft_bfly(x[4], x[5], w[3]);
    fft_bfly_i(x[6], x[7], w[3]);
}
__device__ __forceinline__ void fft_iradix8(double2 (&x)[8], const double2 (&w)[4]) {
    fft_ibfly(x[0], x[1], w[2]);
    fft_ibfly_i(x[2], x[3], w[2]);
    fft_ibfly(x[4], x[5], w[3]);
    fft_ibfly_i(x[6], x[7], w[3]);
    fft_ibfly(x[0], x[2], w[1]);
    fft_ibfly(x[1], x[3], w[1]);
    fft_ibfly_i(x[4], x[6], w[1]);
    fft_ibfly_i(x[5], x[7], w[1]);
#pragma unroll
    for (int k = 0; k < 4; ++k) fft_ibfly(x[k], x[k + 4], w[0]);
}

// Four levels on sixteen points (distances 8, 4, 2, 1) inside one block, twiddles as above and
// w[4] .. w[7] for the fourth level's blocks 8b, 8b + 2, 8b + 4, 8b + 6.
__device__ __forceinline__ void fft_radix16(double2 (&x)[16], const double2* w, int stride) {
    const double2 w0 = w[0], w1 = w[stride];
#pragma unroll
    for (int k = 0; k < 8; ++k) fft_bfly(x[k], x[k + 8], w0);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        fft_bfly(x[k], x[k + 4], w1);
        fft_bfly_i(x[k + 8], x[k + 12], w1);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const double2 w2 = w[(2 + q) * stride];
#pragma unroll
        for (int k = 8 * q; k < 8 * q + 2; ++k) {
            fft_bfly(x[k], x[k + 2], w2);
            fft_bfly_i(x[k + 4], x[k + 6], w2);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double2 w3 = w[(4 + q) * stride];
        fft_bfly(x[4 * q], x[4 * q + 1], w3);
        fft_bfly_i(x[4 * q + 2], x[4 * q + 3], w3);
    }
}
__device__ __forceinline__ void fft_iradix16(double2 (&x)[16], const double2* w, int stride) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double2 w3 = w[(4 + q) * stride];
        fft_ibfly(x[4 * q], x[4 * q + 1], w3);
        fft_ibfly_i(x[4 * q + 2], x[4 * q + 3], w3);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const double2 w2 = w[(2 + q) * stride];
#pragma unroll
        for (int k = 8 * q; k < 8 * q + 2; ++k) {
            fft_ibfly(x[k], x[k + 2], w2);
            fft_ibfly_i(x[k + 4], x[k + 6], w2);
        }
    }
    const double2 w0 = w[0], w1 = w[stride];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        fft_ibfly(x[k], x[k + 4], w1);
        fft_ibfly_i(x[k + 8], x[k + 12], w1);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) fft_ibfly(x[k], x[k + 8], w0);
}

// LOGK = log2 n (9, 10 or 11), 16 points per thread.
template <int LOGK>
struct Fft {
    static constexpr int n = 1 << LOGK;
    static constexpr int T = n / 16;          // threads per polynomial
    static constexpr int HEAD = LOGK < 10 ? LOGK - 6 : 4;  // levels of the first pass
    static constexpr bool MID16 = LOGK > 10;  // the second pass has four levels
    static_assert(LOGK >= 9 && LOGK <= 11, "built for 512, 1024 and 2048 points");

    // Barrier of one polynomial's threads (group g of the block).
    static __device__ __forceinline__ void group_sync(int g) {
        if constexpr (T == 32) {
            (void)g;
            __syncwarp();
        } else {
            asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(T) : "memory");
        }
    }

    // First pass: x[i] is element t + i T.
    static __device__ __forceinline__ void head(double2 (&x)[16], const FftHead& h) {
#pragma unroll
        for (int s = 0; s < HEAD; ++s) {
            const int d = 8 >> s;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if ((i & d) == 0) {
                    const int k = (1 << s) + i / (2 * d);
                    if ((k & 1) && s > 0) fft_bfly_i(x[i], x[i + d], h.fwd[k - 1]);
                    else fft_bfly(x[i], x[i + d], h.fwd[k]);
                }
        }
    }
    static __device__ __forceinline__ void ihead(double2 (&x)[16], const FftHead& h) {
#pragma unroll
        for (int s = HEAD - 1; s >= 0; --s) {
            const int d = 8 >> s;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if ((i & d) == 0) {
                    const int k = (1 << s) + i / (2 * d);
                    if ((k & 1) && s > 0) fft_ibfly_i(x[i], x[i + d], h.inv[k - 1]);
                    else fft_ibfly(x[i], x[i + d], h.inv[k]);
                }
        }
    }

    static __device__ __forceinline__ void load_tw(double2 (&w)[4], const double2* tab, int blocks, int b) {
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = tab[q * blocks + b];
    }

    // The levels after the first pass, in place on `buf` but for the output: slot e goes to
    // put(e, value). tab = pass 2 then pass 3 entries.
    template <typename Put>
    static __device__ __forceinline__ void tail(double2* buf, const double2* tab, int t, int g, Put&& put) {
        constexpr int B2 = fft_blocks2(LOGK), B3 = n / 8;
        double2 x[8], w[4];
        if constexpr (MID16) {
            double2 y[16];
            const int e0 = ((t >> 3) << 7) + (t & 7);
#pragma unroll
            for (int k = 0; k < 16; ++k) y[k] = buf[fft_pos(e0 + 8 * k)];
            fft_radix16(y, tab + (t >> 3), B2);
#pragma unroll
            for (int k = 0; k < 16; ++k) buf[fft_pos(e0 + 8 * k)] = y[k];
        } else {
            load_tw(w, tab, B2, t >> 2);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e0 = ((t >> 2) << 6) + (t & 3) + 4 * q;
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = buf[fft_pos(e0 + 8 * k)];
                fft_radix8(x, w);
#pragma unroll
                for (int k = 0; k < 8; ++k) buf[fft_pos(e0 + 8 * k)] = x[k];
            }
        }
        group_sync(g);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int b = t + q * T;
            load_tw(w, tab + fft_entries2(LOGK) * B2, B3, b);
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = buf[fft_pos(8 * b + k)];
            fft_radix8(x, w);
#pragma unroll
            for (int k = 0; k < 8; ++k) put(8 * b + k, x[k]);
        }
    }
    // The inverse of tail, in place but for its input: slot e is read at *at(e). Ends before the
    // barrier that ihead's reads need.
    template <typename At>
    static __device__ __forceinline__ void itail(double2* buf, const double2* tab, int t, int g, At&& at) {
        constexpr int B2 = fft_blocks2(LOGK), B3 = n / 8;
        double2 x[8], w[4];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int b = t + q * T;
            load_tw(w, tab + fft_entries2(LOGK) * B2, B3, b);
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = *at(8 * b + k);
            fft_iradix8(x, w);
#pragma unroll
            for (int k = 0; k < 8; ++k) buf[fft_pos(8 * b + k)] = x[k];
        }
        group_sync(g);
        if constexpr (MID16) {
            double2 y[16];
            const int e0 = ((t >> 3) << 7) + (t & 7);
#pragma unroll
            for (int k = 0; k < 16; ++k) y[k] = buf[fft_pos(e0 + 8 * k)];
            fft_iradix16(y, tab + (t >> 3), B2);
#pragma unroll
            for (int k = 0; k < 16; ++k) buf[fft_pos(e0 + 8 * k)] = y[k];
        } else {
            load_tw(w, tab, B2, t >> 2);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e0 = ((t >> 2) << 6) + (t & 3) + 4 * q;
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = buf[fft_pos(e0 + 8 * k)];
                fft_iradix8(x, w);
#pragma unroll
                for (int k = 0; k < 8; ++k) buf[fft_pos(e0 + 8 * k)] = x[k];
            }
        }
    }
};

// ---- limbs ----------------------------------------------------------------------------

// Balanced limb base: L limbs of base B cover (-p/2, p/2). ceil(p^(1/3)) and 2^16.
__host__ __device__ constexpr uint32_t fft_limb_base(int limbs) { return limbs == 3 ? 2642246u : 65536u; }

// Adding 1.5 2^52 rounds a double of magnitude below 2^51 to the nearest integer v and
// leaves 2^51 + v in its 52 mantissa bits.
constexpr double kFftRound = 6755399441055744.0;
__device__ __forceinline__ uint64_t fft_round(double v) {
    return (uint64_t)__double_as_longlong(v + kFftRound) & 0xFFFFFFFFFFFFFull;
}
// 2^51 (1 + B + ... + B^(L-1)) mod p, what the offsets above add to the recombined limbs.
__host__ __device__ constexpr uint64_t fft_round_offset(int limbs) {
    unsigned __int128 s = 0, b = 1;
    for (int l = 0; l < limbs; ++l) {
        s += b << 51;
        b *= fft_limb_base(limbs);
    }
    return (uint64_t)(s % kP);
}
// sum_l (c_l - 2^51) B^l mod p, c_l below 2^52.
template <int L>
__device__ __forceinline__ uint64_t fft_recombine(const uint64_t (&c)[L]) {
    static_assert(L == 3 || L == 4, "three or four limbs");
    constexpr uint64_t off = fft_round_offset(L);
    uint64_t s;
    if constexpr (L == 3) {
        constexpr uint32_t B = fft_limb_base(3);
        // Horner in 32-bit words: c2 B + c1 < 2^75, times B plus c0 < 2^96
        const uint64_t p0 = (uint64_t)lo32(c[2]) * B + lo32(c[1]);
        const uint64_t p1 = (uint64_t)hi32(c[2]) * B + hi32(c[1]) + hi32(p0);
        const uint64_t q0 = (uint64_t)lo32(p0) * B + lo32(c[0]);
        const uint64_t q1 = (uint64_t)lo32(p1) * B + hi32(c[0]) + hi32(q0);
        const uint32_t q2 = hi32(p1) * B + hi32(q1);
        s = gl_reduce96(lo32(q0), lo32(q1), q2);
    } else {
        const unsigned __int128 v = (((unsigned __int128)c[3] << 48) + ((unsigned __int128)c[2] << 32)) +
                                    (((unsigned __int128)c[1] << 16) + c[0]);
        s = gl_reduce128((uint32_t)v, (uint32_t)(v >> 32), (uint32_t)(v >> 64), (uint32_t)(v >> 96));
    }
    return gl_sub(s, off);
}

}  // namespace tp
