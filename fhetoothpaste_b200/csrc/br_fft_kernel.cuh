// CGGI blind rotation with double-precision transforms (fft_block.cuh): same words as
// br_kernels.cuh, whose modular transforms it replaces where the key passes the error
// bound (binary and ternary, 2 to 4 digits; one block and the pair at N = 1024 and 2048, clusters at
// 1024 to 4096, halves on two blocks at 4096).
//
// One block per rotation, the accumulator in shared memory as coefficients (pairs j,
// j + N/2) for all n iterations. Per iteration (cggi_blind_rotation.cpp:364-432):
//   digits of the accumulator (binary: of (X^-a - 1) acc) -> 2l forward FFTs at once ->
//   per slot the 2l rows times the key's limbs (ternary: E_lo - X^a E_hi) -> 2L backward
//   FFTs at once -> round, recombine the L limbs mod p -> acc += G (ternary: the two
//   terms (X^-a - 1) E_lo + (X^a - 1) E_hi = (X^-a - 1)(E_lo - X^a E_hi), the outer
//   factor applied to the recombined coefficients, exactly).
// The products by monomials outside the transforms are index shifts.
//
// What bounds it: the key words grow from 8 bytes a coefficient to 8 per limb (1.18 MB an
// iteration, ternary N = 2048); by clock counters in the kernel the products take 45% of an
// iteration, which is 71 of the 75 bytes a clock that a copy loop on every SM gets from L2. The FP64
// pipe is busy for a third of the time, and the rest are the transforms' passes through shared memory
// and their barriers (L1 and shared memory at 66 to 85% of their peak, by ncu). Measured against the
// modular kernels: ternary N = 2048, n = 630, 4096 rotations 452.7 -> 317.3 ms; 1024
// bootstraps of binary N = 1024, n = 500 55.7 -> 40.6 ms.
//
// The key stream, 16 bytes per slot, component, limb and row, is read from L2 straight
// into registers several steps ahead of its use.
#pragma once

#include "br_kernels.cuh"
#include "fft_block.cuh"
#include "mbar.cuh"

namespace tp {

struct BrFftParams {
    const double2* key;       // [it][limb][m < 8][row][component][lane < n/8]
    const double2* tab_fwd;   // pass tables, fft_table_len(log2 n) entries
    const double2* tab_inv;
    const double2* roots;     // 2N: exp(2 pi i k / 2N)
    const uint64_t* lwes;
    uint64_t lwe_stride;
    const uint64_t* accs;
    uint64_t acc_stride;
    uint64_t* out;            // coefficients
    uint64_t batch;
    uint32_t n;
    uint64_t corr;
    uint32_t dshift[8];
    uint64_t dmask[8];
    uint64_t ddelta[8];
    unsigned int* err;
    const unsigned int* exact;  // recorded launches: runs only while *exact is not 0 (the key passes the bound)
    FftHead head;
};

__host__ __device__ constexpr int br_fft_threads(int logn, int dl, int limbs) {
    return (1 << (logn - 4)) * (dl > limbs ? dl : limbs);
}
// The products of a slot replace its digits in place, but other threads may still read those:
// a thread holds its products in registers until all are done, except the first of its eight
// slots', which go to a spare area as far as shared memory allows (one block per SM from
// N = 2048 up, two below; 4 KB are left for the LWE words).
__host__ __device__ constexpr size_t br_fft_base_bytes(int logn, int dl, int limbs) {
    return ((size_t)(2 * (dl > limbs ? dl : limbs)) << (logn - 1)) * 16 + ((size_t)2 << (logn - 1)) * 16 +
           (size_t)2 * fft_table_len(logn - 1) * 16 + 8 * 16;
}
__host__ __device__ constexpr int br_fft_spare(int logn, int dl, int limbs) {
    const size_t room = (logn >= 11 ? 227u * 1024u : 113u * 1024u) - 4096 - br_fft_base_bytes(logn, dl, limbs);
    const int m = (int)(room / ((size_t)2 * limbs * (1 << (logn - 4)) * 16));
    return m > 8 ? 8 : m;
}
// Shared memory in bytes: transform buffers (max(2l, 2L) polynomials), accumulator, pass
// tables of both directions, the iteration's eight monomial factors, the spare area, LWE
// words (32-bit).
__host__ __device__ constexpr size_t br_fft_smem(int logn, int dl, int limbs, uint32_t n) {
    return br_fft_base_bytes(logn, dl, limbs) +
           (size_t)2 * limbs * br_fft_spare(logn, dl, limbs) * (1 << (logn - 4)) * 16 + (((size_t)n + 4) / 4) * 16;
}

// Asks for `bytes` (a multiple of 16, 16-byte aligned) in L2.
__device__ __forceinline__ void l2_prefetch(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// A key word pair. Volatile loads stay as far ahead of their use as the code puts them; other
// forms sink towards it in the assembler (ternary N = 2048: 35.3k clocks an iteration, against
// 50.2k for ld.global.nc and 41.9k for that with a warp barrier after each batch).
__device__ __forceinline__ double2 key_ld(const double2* p) {
    double2 v;
    asm volatile("ld.volatile.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// The pair (coefficients j, j + n) of X^-s a, s < 4n, from a's pairs.
template <int LOGK, typename Load>
__device__ __forceinline__ ulonglong2 rot_pair(Load&& at, uint32_t j, uint32_t s) {
    const uint32_t idx = j + s;
    const ulonglong2 v = at(idx & ((1u << LOGK) - 1u));
    const uint32_t q = (idx >> LOGK) & 3u;
    const uint64_t a = (q & 1u) ? v.y : v.x, b = (q & 1u) ? v.x : v.y;
    return make_ulonglong2((q & 2u) ? gl_neg(a) : a, (q == 1u || q == 2u) ? gl_neg(b) : b);
}

// This thread's 16 points (pairs j = tg + i TG) of one digit of the pairs at v: (v >> sh) & mk -
// off (off carries 2^52).
template <int LOGK>
__device__ __forceinline__ void digit_points(double2 (&x)[16], const ulonglong2* v, int tg, uint32_t sh, uint32_t mk,
                                             double off) {
    constexpr int TG = Fft<LOGK>::T;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const ulonglong2 p = v[tg + i * TG];
        x[i] = make_double2(__hiloint2double(0x43300000, (int)((uint32_t)(p.x >> sh) & mk)) - off,
                            __hiloint2double(0x43300000, (int)((uint32_t)(p.y >> sh) & mk)) - off);
    }
}
// Pair u of (X^-a - 1) acc, half u / n: what binary CGGI decomposes (mux_operator.cpp:144-150).
// Every digit of a half needs it, so the block forms it once (each digit for itself took a third
// of the forward phase: binary N = 2048, l = 4, 11.7k clocks against 8.7k).
template <int LOGK>
__device__ __forceinline__ ulonglong2 rotated_difference(const ulonglong2* acc, uint32_t u, uint32_t a) {
    const ulonglong2* ah = acc + (u & (1u << LOGK));
    const ulonglong2 v = acc[u], w = rot_pair<LOGK>([&](uint32_t k) { return ah[k]; }, u & ((1u << LOGK) - 1u), a);
    return make_ulonglong2(gl_sub(w.x, v.x), gl_sub(w.y, v.y));
}
// s += x k
__device__ __forceinline__ void cmac(double2& s, double2 x, double2 k) {
    s.x = fma(x.x, k.x, s.x);
    s.y = fma(x.x, k.y, s.y);
    s.x = fma(-x.y, k.y, s.x);
    s.y = fma(x.y, k.x, s.y);
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
// lo - w hi
__device__ __forceinline__ double2 csubmul(double2 lo, double2 w, double2 hi) {
    return make_double2(fma(w.y, hi.y, fma(-w.x, hi.x, lo.x)), fma(-w.y, hi.x, fma(-w.x, hi.y, lo.y)));
}
// Rounded limbs (in place of the products in buf) to words G mod p; acc += G (binary) or
// (X^-a - 1) G (ternary), over H halves. All T threads; ends with a barrier.
template <int LOGK, int VARIANT, int L, int T, int H = 2>
__device__ __forceinline__ void recombine_update(double2* buf, ulonglong2* acc, int t, uint32_t a) {
    constexpr int n = 1 << LOGK;
    const ulonglong2* wb = reinterpret_cast<const ulonglong2*>(buf);
    ulonglong2* gb = reinterpret_cast<ulonglong2*>(buf);
    constexpr int U = (H * n + T - 1) / T;
    ulonglong2 gv[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
        const int u = t + k * T;
        if ((H * n) % T == 0 || u < H * n) {
            const int h = u >> LOGK, pos = fft_pos(u & (n - 1));
            uint64_t cx[L], cy[L];
#pragma unroll
            for (int l = 0; l < L; ++l) {
                const ulonglong2 v = wb[(h * L + l) * n + pos];
                cx[l] = v.x;
                cy[l] = v.y;
            }
            gv[k] = make_ulonglong2(fft_recombine<L>(cx), fft_recombine<L>(cy));
            if constexpr (VARIANT == kCggiBinary) {
                // acc += ExtProd (mux_operator.cpp:151)
                const ulonglong2 v = acc[u];
                acc[u] = make_ulonglong2(gl_add(v.x, gv[k].x), gl_add(v.y, gv[k].y));
            } else {
                gb[(h * L) * n + pos] = gv[k];
            }
        }
    }
    __syncthreads();
    if constexpr (VARIANT == kCggiTernary) {
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int u = t + k * T;
            if ((H * n) % T == 0 || u < H * n) {
                const ulonglong2* gh = gb + (u >> LOGK) * (L * n);
                const ulonglong2 w = rot_pair<LOGK>([&](uint32_t j) { return gh[fft_pos((int)j)]; }, u & (n - 1), a);
                const ulonglong2 v = acc[u];
                acc[u] = make_ulonglong2(gl_add(v.x, gl_sub(w.x, gv[k].x)), gl_add(v.y, gl_sub(w.y, gv[k].y)));
            }
        }
        __syncthreads();
    }
}

template <int LOGN, int VARIANT, int DL, int L>
__global__ void __launch_bounds__(br_fft_threads(LOGN, DL, L), LOGN <= 10 ? 2 : 1)
br_fft_kernel(const __grid_constant__ BrFftParams prm) {
    static_assert(VARIANT == kCggiBinary || VARIANT == kCggiTernary, "CGGI only");
    constexpr int LOGK = LOGN - 1;
    using F = Fft<LOGK>;
    constexpr int N = 1 << LOGN, n = F::n, TG = F::T;
    constexpr int G = br_rgsw_per_group(VARIANT);
    constexpr int C = 2 * G, R = 2 * DL;
    constexpr int T = br_fft_threads(LOGN, DL, L);
    constexpr int P = 2 * (DL > L ? DL : L);   // polynomial buffers
    constexpr int LANES = n / 8;
    constexpr int SPARE = br_fft_spare(LOGN, DL, L);
    constexpr uint32_t MASK2N = 2u * N - 1u;
    constexpr bool SIGNED = VARIANT != kCggiBinary;

    if (prm.exact && !*prm.exact) return;
    extern __shared__ __align__(16) uint64_t smem[];
    double2* buf = reinterpret_cast<double2*>(smem);                   // P n
    ulonglong2* acc = reinterpret_cast<ulonglong2*>(buf + P * n);      // 2 n: plus corr (signed)
    double2* tab_f = reinterpret_cast<double2*>(acc + 2 * n);
    double2* tab_i = tab_f + fft_table_len(LOGK);
    double2* mono_s = tab_i + fft_table_len(LOGK);
    double2* spare = mono_s + 8;               // products of the first SPARE slot eighths
    uint32_t* lwe_s = reinterpret_cast<uint32_t*>(spare + 2 * L * SPARE * LANES);

    const int t = threadIdx.x;
    const int grp = t / TG, tg = t % TG;       // transform group, thread in it
    const int limb = t / LANES, lane = t % LANES;
    for (int i = t; i < fft_table_len(LOGK); i += T) {
        tab_f[i] = prm.tab_fwd[i];
        tab_i[i] = prm.tab_inv[i];
    }

    for (uint64_t b = blockIdx.x; b < prm.batch; b += gridDim.x) {
        __syncthreads();  // previous ciphertext done with lwe_s / acc
        const uint64_t* lwe = prm.lwes + b * prm.lwe_stride;
        bool bad = false;
        for (uint32_t i = t; i <= prm.n; i += T) {
            const uint64_t v = lwe[i];
            bad |= v > MASK2N;
            lwe_s[i] = (uint32_t)v & MASK2N;
        }
        if (bad) atomicOr(prm.err, 1u);
        __syncthreads();
        {
            // acc = acc_in X^b (cggi_blind_rotation.cpp:242,333-358), plus the signed digits' corrector
            const uint64_t* ain = prm.accs + b * prm.acc_stride;
            const uint32_t s = (2u * N - lwe_s[prm.n]) & MASK2N;
            for (int u = t; u < 2 * n; u += T) {
                const uint64_t* a = ain + (u >> LOGK) * N;
                ulonglong2 v = rot_pair<LOGK>(
                    [&](uint32_t j) { return make_ulonglong2(gl_canon(a[j]), gl_canon(a[j + n])); }, u & (n - 1), s);
                if constexpr (SIGNED) v = make_ulonglong2(gl_add(v.x, prm.corr), gl_add(v.y, prm.corr));
                acc[u] = v;
            }
        }
        __syncthreads();

        // This block's share of an iteration's key, requested into L2 two iterations ahead: all
        // blocks walk the key at the same pace, so without it each of them waits for HBM.
        auto prefetch = [&](uint32_t it) {
            constexpr uint32_t bytes = (uint32_t)L * 8 * R * C * LANES * 16;
            const uint32_t share = ((bytes + gridDim.x - 1) / gridDim.x + 127u) & ~127u;
            const uint32_t off = blockIdx.x * share;
            if (it < prm.n && off < bytes) l2_prefetch(reinterpret_cast<const char*>(prm.key) + (uint64_t)it * bytes + off,
                                                       min(share, bytes - off));
        };
        if (t == 0) {
            prefetch(0);
            prefetch(1);
        }
#pragma unroll 1
        for (uint32_t it = 0; it < prm.n; ++it) {
            if (t == 0) prefetch(it + 2);
            const uint32_t a = lwe_s[it];
            if (a == 0) continue;  // cggi_blind_rotation.cpp:369-370

            if constexpr (VARIANT == kCggiTernary) {
                // X^a in slot e = lane + m LANES: w^(a (1 + 4 brv(e))), brv(e) = 8 brv(lane) + brv3(m);
                // the factors of m, read after the next barrier (the last readers are behind it)
                if (t < 8) mono_s[t] = __ldg(prm.roots + ((4u * a * (__brev((uint32_t)t) >> 29)) & MASK2N));
            }

            // ---- digits and forward transforms: group grp takes digit grp % DL of half grp / DL ----
            const ulonglong2* src = acc;
            if constexpr (!SIGNED) {
                ulonglong2* d = reinterpret_cast<ulonglong2*>(buf);
                for (int u = t; u < 2 * n; u += T) d[u] = rotated_difference<LOGK>(acc, u, a);
                src = d;
                __syncthreads();
            }
            double2 x[16];
            if (grp < R) {
                const int h = grp / DL, d = grp - h * DL;
                digit_points<LOGK>(x, src + h * n, tg, prm.dshift[d], (uint32_t)prm.dmask[d],
                                   4503599627370496.0 + (SIGNED ? (double)prm.ddelta[d] : 0.0));
            }
            if constexpr (!SIGNED) __syncthreads();  // the differences are read before the transforms overwrite them
            if (grp < R) {
                F::head(x, prm.head);
                double2* pb = buf + grp * n;
#pragma unroll
                for (int i = 0; i < 16; ++i) pb[fft_pos(tg + i * TG)] = x[i];
                F::group_sync(grp);
                F::tail(pb, tab_f, tg, grp, [&](int e, double2 v) { pb[fft_pos(e)] = v; });
            }

            // ---- slot-wise products; this thread's slots lane + m LANES, one limb ----
            double2 o[2][8 - SPARE];
            {
                // Rows go in batches of BR: a batch's key words are requested while the one before it
                // is multiplied, which keeps 8 to 12 16-byte loads per thread in flight.
                constexpr int BR = C == 4 ? (R % 3 == 0 ? 3 : 2) : (R % 4 == 0 ? 4 : R), NB = 8 * R / BR;
                static_assert(R % BR == 0, "a batch lies in one slot");
                const double2* kp = prm.key + (((uint64_t)it * L + limb) * (8 * R * C)) * LANES + lane;
                double2 kv[2][BR][C];
                auto load = [&](int q, double2 (&k)[BR][C]) {
#pragma unroll
                    for (int r = 0; r < BR; ++r)
#pragma unroll
                        for (int c = 0; c < C; ++c) k[r][c] = key_ld(kp + ((q * BR + r) * C + c) * LANES);
                };
                double2 wb = make_double2(1.0, 0.0);
                const bool on = limb < L;
                if (on) {
                    load(0, kv[0]);
                    if constexpr (VARIANT == kCggiTernary)
                        wb = __ldg(prm.roots + ((a * (1u + 32u * (__brev((uint32_t)lane) >> (35 - LOGK)))) & MASK2N));
                }
                __syncthreads();
                if (on) {
                    double2 s[C];
#pragma unroll
                    for (int q = 0; q < NB; ++q) {
                        const int m = q * BR / R, pos = fft_pos(lane + m * LANES);
                        if (q + 1 < NB) load(q + 1, kv[(q + 1) & 1]);
                        if (q * BR % R == 0) {
#pragma unroll
                            for (int c = 0; c < C; ++c) s[c] = make_double2(0.0, 0.0);
                        }
#pragma unroll
                        for (int r = 0; r < BR; ++r) {
                            const double2 x = buf[(q * BR % R + r) * n + pos];
#pragma unroll
                            for (int c = 0; c < C; ++c) cmac(s[c], x, kv[q & 1][r][c]);
                        }
                        if ((q + 1) * BR % R != 0) continue;
                        double2 v[2] = {s[0], s[1]};
                        if constexpr (VARIANT == kCggiTernary) {
                            const double2 w = cmul(wb, mono_s[m]);
#pragma unroll
                            for (int h = 0; h < 2; ++h) v[h] = csubmul(s[h], w, s[C - 2 + h]);
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (m < SPARE) spare[(h * L + limb) * (SPARE * LANES) + pos] = v[h];
                            else o[h][m - SPARE] = v[h];
                        }
                    }
                }
                __syncthreads();  // every read of the digits' slots before the products take their place
                if (on) {
#pragma unroll
                    for (int m = SPARE; m < 8; ++m) {
                        const int pos = fft_pos(lane + m * LANES);
#pragma unroll
                        for (int h = 0; h < 2; ++h) buf[(h * L + limb) * n + pos] = o[h][m - SPARE];
                    }
                }
                __syncthreads();
            }

            // ---- backward transforms, rounded coefficients back in place ----
            if (grp < 2 * L) {
                double2* pb = buf + grp * n;
                F::itail(pb, tab_i, tg, grp, [&](int e) {
                    return (e < SPARE * LANES ? spare + grp * (SPARE * LANES) : pb) + fft_pos(e);
                });
                F::group_sync(grp);
                double2 x[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = pb[fft_pos(tg + i * TG)];
                F::ihead(x, prm.head);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    *reinterpret_cast<ulonglong2*>(pb + fft_pos(tg + i * TG)) =
                        make_ulonglong2(fft_round(x[i].x), fft_round(x[i].y));
            }
            __syncthreads();

            // ---- limbs to words mod p; accumulator ----
            recombine_update<LOGK, VARIANT, L, T>(buf, acc, t, a);
        }

        uint64_t* res = prm.out + b * (2ull * N);
        for (int u = t; u < 2 * n; u += T) {
            ulonglong2 v = acc[u];
            if constexpr (SIGNED) v = make_ulonglong2(gl_sub(v.x, prm.corr), gl_sub(v.y, prm.corr));
            uint64_t* r = res + (u >> LOGK) * N + (u & (n - 1));
            r[0] = v.x;
            r[n] = v.y;
        }
    }
}

// ---------------------------------------------------------------------------
// Two rotations on a cluster of two blocks, for throughput: block c rotates ciphertext c of the
// pair and multiplies the slots of half c of both, so that each block reads half the key (the
// key stream from L2 takes 45% of an iteration of the one-block form). Per iteration the blocks
// exchange half of their digits' slots and half of their products through distributed shared
// memory, 48 KB each at ternary N = 2048, with two cluster barriers: the digits of the other
// block's half go to its receive area, free since the barrier after the last products; products
// go where their block's digits of that half have been sent away from. Digits travel as bulk
// copies (the transform's own stores, a 128-byte line apart from lane to lane, took 4.7k clocks for 48 KB).
// Ternary N = 2048, n = 630, 4096 rotations: 317 -> 298 ms over the one-block form.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr size_t br_fft_pair_base_bytes(int logn, int dl, int limbs) {
    const size_t k = (size_t)1 << (logn - 1);
    return ((2 * (dl > limbs ? dl : limbs)) * k + dl * k + 2 * k + 9) * 16;  // buffers, receive area, accumulator, factors, barrier
}
__host__ __device__ constexpr size_t br_fft_pair_limit(int logn) { return logn >= 11 ? 227u * 1024u : 113u * 1024u; }
__host__ __device__ constexpr bool br_fft_pair_tabs(int logn, int dl, int limbs) {  // pass tables in shared memory
    return br_fft_pair_base_bytes(logn, dl, limbs) + 2 * fft_table_len(logn - 1) * 16 + 4096 <= br_fft_pair_limit(logn);
}
// Eighths of the slots whose own products go to a spare area (see br_fft_spare).
__host__ __device__ constexpr int br_fft_pair_spare(int logn, int dl, int limbs) {
    if (!br_fft_pair_tabs(logn, dl, limbs)) return 0;
    const size_t room = br_fft_pair_limit(logn) - 4096 - br_fft_pair_base_bytes(logn, dl, limbs) -
                        2 * fft_table_len(logn - 1) * 16;
    const int m = (int)(room / ((size_t)2 * limbs * (1 << (logn - 4)) * 16));
    return m > 4 ? 4 : m;
}
__host__ __device__ constexpr size_t br_fft_pair_smem(int logn, int dl, int limbs, uint32_t n) {
    return br_fft_pair_base_bytes(logn, dl, limbs) +
           (br_fft_pair_tabs(logn, dl, limbs) ? 2 * fft_table_len(logn - 1) * 16 : 0) +
           (size_t)2 * limbs * br_fft_pair_spare(logn, dl, limbs) * (1 << (logn - 4)) * 16 + ((2 * (size_t)(n + 1) + 7) / 8) * 16;
}

template <int LOGN, int VARIANT, int DL, int L>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(br_fft_threads(LOGN, DL, L), LOGN <= 10 ? 2 : 1)
br_fft_pair_kernel(const __grid_constant__ BrFftParams prm) {
    static_assert(VARIANT == kCggiBinary || VARIANT == kCggiTernary, "CGGI only");
    constexpr int LOGK = LOGN - 1;
    using F = Fft<LOGK>;
    constexpr int N = 1 << LOGN, n = F::n, TG = F::T;
    constexpr int G = br_rgsw_per_group(VARIANT);
    constexpr int C = 2 * G, R = 2 * DL;
    constexpr int T = br_fft_threads(LOGN, DL, L);
    constexpr int P = 2 * (DL > L ? DL : L);
    constexpr int LANES = n / 8, M = 4;        // slots of this block per thread
    constexpr int SPARE = br_fft_pair_spare(LOGN, DL, L);
    constexpr bool TABS = br_fft_pair_tabs(LOGN, DL, L);
    constexpr uint32_t MASK2N = 2u * N - 1u;
    constexpr bool SIGNED = VARIANT != kCggiBinary;

    if (prm.exact && !*prm.exact) return;
    extern __shared__ __align__(16) uint64_t smem[];
    double2* buf = reinterpret_cast<double2*>(smem);                   // P n
    double2* recv = buf + P * n;                                       // R n/2: the other rotation's digits
    ulonglong2* acc = reinterpret_cast<ulonglong2*>(recv + R * (n / 2));  // 2 n: plus corr (signed)
    double2* mono_s = reinterpret_cast<double2*>(acc + 2 * n);         // [rotation][m < 4]
    uint64_t* bar = reinterpret_cast<uint64_t*>(mono_s + 8);           // the other block's digits have come
    double2* spare = mono_s + 9;
    double2* tabs = spare + 2 * L * SPARE * LANES;
    uint16_t* lwe_s = reinterpret_cast<uint16_t*>(tabs + (TABS ? 2 * fft_table_len(LOGK) : 0));  // [rotation][n + 1]

    auto cluster = cooperative_groups::this_cluster();
    const int c = (int)cluster.block_rank();
    const int t = threadIdx.x;
    const int grp = t / TG, tg = t % TG;
    const int limb = t / LANES, lane = t % LANES;
    const double2* tab_f = prm.tab_fwd;
    const double2* tab_i = prm.tab_inv;
    if constexpr (TABS) {
        for (int i = t; i < fft_table_len(LOGK); i += T) {
            tabs[i] = prm.tab_fwd[i];
            tabs[fft_table_len(LOGK) + i] = prm.tab_inv[i];
        }
        tab_f = tabs;
        tab_i = tabs + fft_table_len(LOGK);
    }
    uint32_t phase = 0;
    bool ok = true;  // a wait for the other block's digits ran out
    if (t == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    double2* buf_peer = cluster.map_shared_rank(buf, (unsigned)(c ^ 1));
    cluster.sync();  // both blocks running, their barriers set, before remote stores

    for (uint64_t b0 = blockIdx.x & ~1ull; b0 < prm.batch; b0 += gridDim.x) {
        const uint64_t b = b0 + c;
        __syncthreads();
        bool bad = false;
#pragma unroll
        for (int r = 0; r < 2; ++r) {  // both rotations' words; a missing one is all zeros and written nowhere
            const uint64_t* lwe = prm.lwes + (b0 + r) * prm.lwe_stride;
            const bool have = b0 + r < prm.batch;
            for (uint32_t i = t; i <= prm.n; i += T) {
                const uint64_t v = have ? lwe[i] : 0;
                bad |= v > MASK2N;
                lwe_s[r * (prm.n + 1) + i] = (uint16_t)(v & MASK2N);
            }
        }
        if (bad && c == 0) atomicOr(prm.err, 1u);
        __syncthreads();
        {
            const uint64_t* ain = prm.accs + b * prm.acc_stride;
            const uint32_t s = (2u * N - lwe_s[c * (prm.n + 1) + prm.n]) & MASK2N;
            for (int u = t; u < 2 * n; u += T) {
                ulonglong2 v = make_ulonglong2(0, 0);
                if (b < prm.batch) {
                    const uint64_t* a = ain + (u >> LOGK) * N;
                    v = rot_pair<LOGK>([&](uint32_t j) { return make_ulonglong2(gl_canon(a[j]), gl_canon(a[j + n])); },
                                       u & (n - 1), s);
                }
                if constexpr (SIGNED) v = make_ulonglong2(gl_add(v.x, prm.corr), gl_add(v.y, prm.corr));
                acc[u] = v;
            }
        }
        __syncthreads();

        auto prefetch = [&](uint32_t it) {  // this block's share of an iteration's key, as in the one-block form
            constexpr uint32_t bytes = (uint32_t)L * 8 * R * C * LANES * 16;
            const uint32_t share = ((bytes + gridDim.x - 1) / gridDim.x + 127u) & ~127u;
            const uint32_t off = blockIdx.x * share;
            if (it < prm.n && off < bytes) l2_prefetch(reinterpret_cast<const char*>(prm.key) + (uint64_t)it * bytes + off,
                                                       min(share, bytes - off));
        };
        if (t == 0) {
            prefetch(0);
            prefetch(1);
        }
#pragma unroll 1
        for (uint32_t it = 0; it < prm.n; ++it) {
            if (t == 0) prefetch(it + 2);
            const uint32_t ar[2] = {lwe_s[it], lwe_s[prm.n + 1 + it]};
            if (ar[0] == 0 && ar[1] == 0) continue;  // one rotation alone at 0 adds (X^0 - 1) G = 0
            const uint32_t a = c ? ar[1] : ar[0];
            if (t == 0) mbar_expect(bar, R * (n / 2) * 16);

            if constexpr (VARIANT == kCggiTernary) {
                // factors of this block's m (see br_fft_kernel), both rotations
                if (t < 8)
                    mono_s[t] = __ldg(prm.roots + ((4u * (t < 4 ? ar[0] : ar[1]) *
                                                    (__brev((uint32_t)(c * M + (t & 3))) >> 29)) & MASK2N));
            }

            // ---- digits and forward transforms; the other half's slots to the other block ----
            const ulonglong2* src = acc;
            if constexpr (!SIGNED) {
                ulonglong2* d = reinterpret_cast<ulonglong2*>(buf);
                for (int u = t; u < 2 * n; u += T) d[u] = rotated_difference<LOGK>(acc, u, a);
                src = d;
                __syncthreads();
            }
            double2 x[16];
            if (grp < R) {
                const int h = grp / DL, d = grp - h * DL;
                digit_points<LOGK>(x, src + h * n, tg, prm.dshift[d], (uint32_t)prm.dmask[d],
                                   4503599627370496.0 + (SIGNED ? (double)prm.ddelta[d] : 0.0));
            }
            if constexpr (!SIGNED) __syncthreads();  // the differences are read before the transforms overwrite them
            if (grp < R) {
                F::head(x, prm.head);
                double2* pb = buf + grp * n;
#pragma unroll
                for (int i = 0; i < 16; ++i) pb[fft_pos(tg + i * TG)] = x[i];
                F::group_sync(grp);
                F::tail(pb, tab_f, tg, grp, [&](int e, double2 v) { pb[fft_pos(e)] = v; });
                bulk_fence();
                F::group_sync(grp);
                if (tg == 0)
                    bulk_to_block(recv + grp * (n / 2), pb + (c ^ 1) * (n / 2), n / 2 * 16, bar, (uint32_t)(c ^ 1));
            }

            // ---- slot-wise products, slots lane + (4 c + m) LANES of both rotations, one limb ----
            double2 o[2][M - SPARE + 1];
            {
                constexpr int BR = 2, NB = M * R / BR;
                const double2* kp = prm.key + ((((uint64_t)it * L + limb) * 8 + c * M) * (R * C)) * LANES + lane;
                double2 kv[2][BR][C];
                auto load = [&](int q, double2 (&k)[BR][C]) {
#pragma unroll
                    for (int r = 0; r < BR; ++r)
#pragma unroll
                        for (int cc = 0; cc < C; ++cc) k[r][cc] = key_ld(kp + ((q * BR + r) * C + cc) * LANES);
                };
                double2 wb[2];
                const bool on = limb < L;
                if (on) {
                    load(0, kv[0]);
                    if constexpr (VARIANT == kCggiTernary) {
                        const uint32_t e = 1u + 32u * (__brev((uint32_t)lane) >> (35 - LOGK));
                        wb[0] = __ldg(prm.roots + ((ar[0] * e) & MASK2N));
                        wb[1] = __ldg(prm.roots + ((ar[1] * e) & MASK2N));
                    }
                }
                __syncthreads();
                ok = ok && mbar_wait(bar, phase);
                phase ^= 1;
                if (on) {
                    double2 s[2][C];
#pragma unroll
                    for (int q = 0; q < NB; ++q) {
                        const int m = q * BR / R, pos = fft_pos(lane + (c * M + m) * LANES),
                                  rpos = fft_pos(lane + m * LANES);
                        if (q + 1 < NB) load(q + 1, kv[(q + 1) & 1]);
                        if (q * BR % R == 0) {
#pragma unroll
                            for (int cc = 0; cc < C; ++cc) s[0][cc] = s[1][cc] = make_double2(0.0, 0.0);
                        }
#pragma unroll
                        for (int r = 0; r < BR; ++r) {
                            const double2 x0 = buf[(q * BR % R + r) * n + pos];
                            const double2 x1 = recv[(q * BR % R + r) * (n / 2) + rpos];
#pragma unroll
                            for (int cc = 0; cc < C; ++cc) {
                                cmac(s[0][cc], x0, kv[q & 1][r][cc]);
                                cmac(s[1][cc], x1, kv[q & 1][r][cc]);
                            }
                        }
                        if ((q + 1) * BR % R != 0) continue;
                        if constexpr (VARIANT == kCggiTernary) {
                            // rotation of s[0] is c, of s[1] the other
                            const double2 w0 = cmul(c ? wb[1] : wb[0], mono_s[c * 4 + m]);
                            const double2 w1 = cmul(c ? wb[0] : wb[1], mono_s[(c ^ 1) * 4 + m]);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                s[0][h] = csubmul(s[0][h], w0, s[0][C - 2 + h]);
                                s[1][h] = csubmul(s[1][h], w1, s[1][C - 2 + h]);
                            }
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            buf_peer[(h * L + limb) * n + pos] = s[1][h];
                            if (m < SPARE) spare[(h * L + limb) * (SPARE * LANES) + rpos] = s[0][h];
                            else o[h][m - SPARE] = s[0][h];
                        }
                    }
                }
                cluster.sync();  // both blocks' reads of the digits done, products of the other half here
                if (on) {
#pragma unroll
                    for (int m = SPARE; m < M; ++m)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            buf[(h * L + limb) * n + fft_pos(lane + (c * M + m) * LANES)] = o[h][m - SPARE];
                }
                __syncthreads();
            }

            // ---- backward transforms, rounded coefficients back in place ----
            if (grp < 2 * L) {
                double2* pb = buf + grp * n;
                F::itail(pb, tab_i, tg, grp, [&](int e) {
                    const int el = e - c * (n / 2);
                    return el >= 0 && el < SPARE * LANES ? spare + grp * (SPARE * LANES) + fft_pos(el) : pb + fft_pos(e);
                });
                F::group_sync(grp);
                double2 x[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = pb[fft_pos(tg + i * TG)];
                F::ihead(x, prm.head);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    *reinterpret_cast<ulonglong2*>(pb + fft_pos(tg + i * TG)) =
                        make_ulonglong2(fft_round(x[i].x), fft_round(x[i].y));
            }
            __syncthreads();

            recombine_update<LOGK, VARIANT, L, T>(buf, acc, t, a);
        }

        if (b < prm.batch) {
            uint64_t* res = prm.out + b * (2ull * N);
            for (int u = t; u < 2 * n; u += T) {
                ulonglong2 v = acc[u];
                if constexpr (SIGNED) v = make_ulonglong2(gl_sub(v.x, prm.corr), gl_sub(v.y, prm.corr));
                uint64_t* r = res + (u >> LOGK) * N + (u & (n - 1));
                r[0] = v.x;
                r[n] = v.y;
            }
        }
    }
    if (!ok) atomicOr(prm.err, 2u);
    cluster.sync();  // no block leaves while the other may still store to it
}

// ---------------------------------------------------------------------------
// A few rotations: one rotation per cluster of CS blocks, for latency. One block alone reads
// its key at a third of the rate that a full GPU's blocks get (they share lines on the way
// from L2) and runs every transform itself. Here block c transforms the polynomials c PP ..
// c PP + PP - 1 (PP = 1 at eight blocks), multiplies the slots [c n/CS, (c + 1) n/CS) and
// recombines the same range of coefficients. Four exchanges an iteration, all as bulk copies
// between the blocks' shared memory that complete on the receiver's barriers (cluster barriers
// behind remote stores took 1.0k to 1.4k clocks each): digit slots to their blocks, products to
// the blocks of their limbs, rounded limbs to the blocks of their coefficients, words mod p to the
// blocks whose digits need them. Every block takes part in each exchange that another block's
// next step waits for, so an area's next contents are sent only after its last reads: digits i + 1
// follow words i of all blocks, which follow their products i, and so on round the cycle.
// N = 4096, n = 60, one rotation on eight blocks against two: ternary l = 3 1.66 -> 0.74 ms,
// binary l = 4 1.44 -> 0.75.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int br_fft_cluster_polys(int dl, int limbs, int cs) {
    return (2 * (dl > limbs ? dl : limbs) + cs - 1) / cs;
}
// A thread multiplies the slots lane + m LANES of one limb: n/8 lanes, at N = 4096 n/16 (512
// threads keep 128 registers each).
__host__ __device__ constexpr int br_fft_cluster_lanes(int logn) { return 1 << (logn - (logn > 11 ? 5 : 4)); }
__host__ __device__ constexpr int br_fft_cluster_threads(int logn, int limbs) { return br_fft_cluster_lanes(logn) * limbs; }
// At N = 4096 (eight blocks, one polynomial each) a block keeps only the accumulator half and the
// words that its digit is of, and reads the pass tables through L1.
__host__ __device__ constexpr int br_fft_cluster_halves(int logn) { return logn > 11 ? 1 : 2; }
// Forward and backward buffers (PP polynomials each), digit slots (2l n/CS), limb and word
// areas (2L n/CS, also the products on their way out; 2n), accumulator (2n), words on their way out
// (2 n/CS), pass tables, monomial factors, barriers, LWE words.
__host__ __device__ constexpr size_t br_fft_cluster_smem(int logn, int dl, int limbs, int cs, uint32_t n) {
    const size_t k = (size_t)1 << (logn - 1);
    const int halves = br_fft_cluster_halves(logn);
    return (2 * br_fft_cluster_polys(dl, limbs, cs) * k + (2 * dl + 2 * limbs + 2) * (k / cs) + 2 * halves * k +
            (halves == 2 ? 2 * fft_table_len(logn - 1) : 0) + 10) * 16 + (((size_t)n + 4) / 4) * 16;
}

template <int LOGN, int VARIANT, int DL, int L, int CS>
__global__ void __launch_bounds__(br_fft_cluster_threads(LOGN, L), 1)
br_fft_cluster_kernel(const __grid_constant__ BrFftParams prm) {
    static_assert(VARIANT == kCggiBinary || VARIANT == kCggiTernary, "CGGI only");
    constexpr int LOGK = LOGN - 1;
    using F = Fft<LOGK>;
    constexpr int N = 1 << LOGN, n = F::n, TG = F::T;
    constexpr int G = br_rgsw_per_group(VARIANT);
    constexpr int C = 2 * G, R = 2 * DL;
    constexpr int LANES = br_fft_cluster_lanes(LOGN), T = LANES * L, NS = n / CS, M = NS / LANES;
    constexpr int KL = n / 8, KM = 8 / CS, SUB = KL / LANES;  // the key's lanes, its m per block, m here per key m
    constexpr int PP = br_fft_cluster_polys(DL, L, CS);
    constexpr int H = br_fft_cluster_halves(LOGN);            // accumulator halves kept
    constexpr uint32_t MASK2N = 2u * N - 1u;
    constexpr bool SIGNED = VARIANT != kCggiBinary;
    // products and limbs as bulk copies, or (fewer blocks, more words to each) as remote stores behind
    // a cluster barrier
    constexpr bool BULK = CS == 8, WORDS = CS == 8 || LOGN == 10;
    static_assert(8 % CS == 0 && PP * TG <= T - 32, "block shape");
    static_assert(H == 2 || (CS == 8 && PP == 1), "one half: one polynomial per block");

    if (prm.exact && !*prm.exact) return;
    extern __shared__ __align__(16) uint64_t smem[];
    double2* work = reinterpret_cast<double2*>(smem);                  // PP n
    double2* inv = work + PP * n;                                      // PP n
    double2* dig = inv + PP * n;                                       // R NS
    ulonglong2* lim = reinterpret_cast<ulonglong2*>(dig + R * NS);     // 2L NS
    ulonglong2* gb = lim + 2 * L * NS;                                 // 2 n
    ulonglong2* acc = gb + H * n;                                      // H n: plus corr (signed)
    ulonglong2* gs = acc + H * n;                                      // 2 NS
    double2* tabs = reinterpret_cast<double2*>(gs + 2 * NS);
    double2* mono_s = tabs + (H == 2 ? 2 * fft_table_len(LOGK) : 0);
    uint64_t* bar = reinterpret_cast<uint64_t*>(mono_s + 8);           // [4]: digits, products, limbs, words have come
    uint32_t* lwe_s = reinterpret_cast<uint32_t*>(mono_s + 10);

    auto cluster = cooperative_groups::this_cluster();
    const int c = (int)cluster.block_rank();
    const int t = threadIdx.x;
    const int grp = t / TG, tg = t % TG;
    const int limb = t / LANES, lane = t % LANES;
    const double2* tab_f = prm.tab_fwd;
    const double2* tab_i = prm.tab_inv;
    if constexpr (H == 2) {
        for (int i = t; i < fft_table_len(LOGK); i += T) {
            tabs[i] = prm.tab_fwd[i];
            tabs[fft_table_len(LOGK) + i] = prm.tab_inv[i];
        }
        tab_f = tabs;
        tab_i = tabs + fft_table_len(LOGK);
    }
    auto half = [](int h) { return H == 2 ? h * n : 0; };  // where half h starts in acc and gb
    // blocks whose forward polynomials are digits of half h
    auto first_of = [](int h) { return h * DL / PP; };
    auto last_of = [](int h) { return (h * DL + DL - 1) / PP; };
    const uint32_t own_halves = (c >= first_of(0) && c <= last_of(0) ? 1 : 0) + (c >= first_of(1) && c <= last_of(1) ? 1 : 0);
    const uint32_t own_limbs = c * PP >= 2 * L ? 0 : min(PP, 2 * L - c * PP);  // limb polynomials transformed back here
    uint32_t phase = 0;
    bool ok = true;  // a wait for the other blocks ran out
    if (t == 0) {
        for (int q = 0; q < 4; ++q) mbar_init(bar + q, 1);
        mbar_init_fence();
    }
    cluster.sync();  // every block of the cluster running, its barriers set, before copies to it

    const uint64_t clusters = gridDim.x / CS;
    for (uint64_t b = blockIdx.x / CS; b < prm.batch; b += clusters) {
        __syncthreads();
        const uint64_t* lwe = prm.lwes + b * prm.lwe_stride;
        bool bad = false;
        for (uint32_t i = t; i <= prm.n; i += T) {
            const uint64_t v = lwe[i];
            bad |= v > MASK2N;
            lwe_s[i] = (uint32_t)v & MASK2N;
        }
        if (bad) atomicOr(prm.err, 1u);
        __syncthreads();
        {
            // acc = acc_in X^b, plus the signed digits' corrector
            const uint64_t* ain = prm.accs + b * prm.acc_stride;
            const uint32_t s = (2u * N - lwe_s[prm.n]) & MASK2N;
            const int h0 = H == 2 || c < DL ? 0 : 1;  // the half kept (H = 1)
            for (int u = t; u < H * n; u += T) {
                const uint64_t* a = ain + (h0 + (u >> LOGK)) * N;
                ulonglong2 v = rot_pair<LOGK>(
                    [&](uint32_t j) { return make_ulonglong2(gl_canon(a[j]), gl_canon(a[j + n])); }, u & (n - 1), s);
                if constexpr (SIGNED) v = make_ulonglong2(gl_add(v.x, prm.corr), gl_add(v.y, prm.corr));
                acc[u] = v;
            }
        }
        cluster.sync();  // every block has read the accumulator before one writes its result over it

        auto prefetch = [&](uint32_t it) {  // this block's slots of an iteration's key, one thread per limb
            constexpr uint32_t per = (uint32_t)R * C * KL * 16;
            const uint32_t l = (uint32_t)(t - (T - 32));  // of a warp that has no transform
            if (it < prm.n && l < L)
                l2_prefetch(reinterpret_cast<const char*>(prm.key) + (((uint64_t)it * L + l) * 8 + c * KM) * per, KM * per);
        };
        prefetch(0);
        prefetch(1);
#pragma unroll 1
        for (uint32_t it = 0; it < prm.n; ++it) {
            prefetch(it + 2);
            const uint32_t a = lwe_s[it];
            if (a == 0) continue;
            if (t == T - 1) {
                mbar_expect(bar, R * NS * 16);
                if (BULK && own_limbs) mbar_expect(bar + 1, own_limbs * n * 16);
                if constexpr (BULK) mbar_expect(bar + 2, 2 * L * NS * 16);
                if (WORDS && own_halves) mbar_expect(bar + 3, own_halves * n * 16);
            }

            // ---- digits and forward transforms, slots to their blocks ----
            const int p = c * PP + grp;
            const ulonglong2* src = acc;
            if constexpr (!SIGNED) {
                // in the words' area, which is written again only after this block's digits have gone
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (c >= first_of(h) && c <= last_of(h))
                        for (int u = t; u < n; u += T) gb[half(h) + u] = rotated_difference<LOGK>(acc, half(h) + u, a);
                src = gb;
                __syncthreads();
            }
            if (grp < PP && p < R) {
                const int h = p / DL, d = p - h * DL;
                double2 x[16];
                digit_points<LOGK>(x, src + half(h), tg, prm.dshift[d], (uint32_t)prm.dmask[d],
                                   4503599627370496.0 + (SIGNED ? (double)prm.ddelta[d] : 0.0));
                F::head(x, prm.head);
                double2* pb = work + grp * n;
#pragma unroll
                for (int i = 0; i < 16; ++i) pb[fft_pos(tg + i * TG)] = x[i];
                F::group_sync(grp);
                F::tail(pb, tab_f, tg, grp, [&](int e, double2 v) { pb[fft_pos(e)] = v; });
                bulk_fence();
                F::group_sync(grp);
                if (tg < CS) bulk_to_block(dig + p * NS, pb + tg * NS, NS * 16, bar, (uint32_t)tg);
            } else if (VARIANT == kCggiTernary && t >= T - KM) {
                const int km = t - (T - KM);
                mono_s[km] = __ldg(prm.roots + ((4u * a * (__brev((uint32_t)(c * KM + km)) >> 29)) & MASK2N));
            }

            // ---- slot-wise products; slots lane + (c M + mm) LANES, one limb ----
            // the key's lane of mm is lane + (mm % SUB) LANES, its m is c KM + mm / SUB
            constexpr int BR = H == 1 ? 2 : C == 4 ? (R % 3 == 0 ? 3 : 2) : (R % 4 == 0 ? 4 : R), NB = M * R / BR;
            const double2* kp = prm.key + ((((uint64_t)it * L + limb) * 8 + c * KM) * (R * C)) * KL + lane;
            double2 kv[2][BR][C];
            auto load = [&](int q, double2 (&k)[BR][C]) {
#pragma unroll
                for (int r = 0; r < BR; ++r)
#pragma unroll
                    for (int cc = 0; cc < C; ++cc) {
                        const int mm = q * BR / R, row = q * BR % R + r;
                        k[r][cc] = key_ld(kp + ((mm / SUB * R + row) * C + cc) * KL + mm % SUB * LANES);
                    }
            };
            load(0, kv[0]);
            double2 wb[SUB];
            if constexpr (VARIANT == kCggiTernary) {
#pragma unroll
                for (int q = 0; q < SUB; ++q)
                    wb[q] = __ldg(prm.roots + ((a * (1u + 32u * (__brev((uint32_t)(lane + q * LANES)) >> (35 - LOGK)))) & MASK2N));
            }
            __syncthreads();
            ok = ok && mbar_wait(bar, phase);
            double2 s[C];
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                const int mm = q * BR / R, pos = fft_pos(c * NS + lane + mm * LANES) - c * NS;
                if (q + 1 < NB) load(q + 1, kv[(q + 1) & 1]);
                if (q * BR % R == 0) {
#pragma unroll
                    for (int cc = 0; cc < C; ++cc) s[cc] = make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int r = 0; r < BR; ++r) {
                    const double2 x = dig[(q * BR % R + r) * NS + pos];
#pragma unroll
                    for (int cc = 0; cc < C; ++cc) cmac(s[cc], x, kv[q & 1][r][cc]);
                }
                if ((q + 1) * BR % R != 0) continue;
                double2 v[2] = {s[0], s[1]};
                if constexpr (VARIANT == kCggiTernary) {
                    const double2 w = cmul(wb[mm % SUB], mono_s[mm / SUB]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) v[h] = csubmul(s[h], w, s[C - 2 + h]);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int qo = h * L + limb;
                    if constexpr (BULK) reinterpret_cast<double2*>(lim)[qo * NS + pos] = v[h];
                    else cluster.map_shared_rank(inv, (unsigned)(qo / PP))[(qo % PP) * n + c * NS + pos] = v[h];
                }
            }
            if constexpr (BULK) {
                bulk_fence();
                __syncthreads();
                if (t < 2 * L)
                    bulk_to_block(inv + (t % PP) * n + c * NS, lim + t * NS, NS * 16, bar + 1, (uint32_t)(t / PP));
            } else {
                cluster.sync();
            }

            // ---- backward transforms, rounded limbs to the blocks of their coefficients ----
            if (grp < PP && p < 2 * L) {
                if constexpr (BULK) ok = ok && mbar_wait(bar + 1, phase);
                double2* pb = inv + grp * n;
                F::itail(pb, tab_i, tg, grp, [&](int e) { return pb + fft_pos(e); });
                F::group_sync(grp);
                double2 x[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = pb[fft_pos(tg + i * TG)];
                F::ihead(x, prm.head);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int pos = fft_pos(tg + i * TG);
                    const ulonglong2 r = make_ulonglong2(fft_round(x[i].x), fft_round(x[i].y));
                    if constexpr (BULK) *reinterpret_cast<ulonglong2*>(pb + pos) = r;
                    else cluster.map_shared_rank(lim, (unsigned)(pos / NS))[p * NS + pos % NS] = r;
                }
                if constexpr (BULK) {
                    bulk_fence();
                    F::group_sync(grp);
                    if (tg < CS) bulk_to_block(lim + p * NS, pb + tg * NS, NS * 16, bar + 2, (uint32_t)tg);
                }
            }
            if constexpr (!BULK) cluster.sync();

            // ---- words mod p to the blocks that need their half ----
            if constexpr (BULK) ok = ok && mbar_wait(bar + 2, phase);
            for (int u = t; u < 2 * NS; u += T) {
                const int h = u / NS, j = fft_pos(c * NS + u % NS) - c * NS;
                uint64_t cx[L], cy[L];
#pragma unroll
                for (int l = 0; l < L; ++l) {
                    const ulonglong2 v = lim[(h * L + l) * NS + j];
                    cx[l] = v.x;
                    cy[l] = v.y;
                }
                const ulonglong2 gw = make_ulonglong2(fft_recombine<L>(cx), fft_recombine<L>(cy));
                if constexpr (WORDS) gs[u] = gw;
                else
                    for (int q = first_of(h); q <= last_of(h); ++q)
                        cluster.map_shared_rank(gb, (unsigned)q)[half(h) + c * NS + u % NS] = gw;
            }
            if constexpr (WORDS) {
                bulk_fence();
                __syncthreads();
            } else {
                cluster.sync();
            }
            if (WORDS && t < 2 * CS) {
                const int h = t / CS, q = t % CS;
                if (q >= first_of(h) && q <= last_of(h))
                    bulk_to_block(gb + half(h) + c * NS, gs + h * NS, NS * 16, bar + 3, (uint32_t)q);
            }

            // ---- accumulator halves of this block ----
            if (WORDS && own_halves) ok = ok && mbar_wait(bar + 3, phase);
            phase ^= 1;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (c < first_of(h) || c > last_of(h)) continue;
                const ulonglong2* gh = gb + half(h);
                for (int u = t; u < n; u += T) {
                    const ulonglong2 v = acc[half(h) + u], g = gh[u];
                    if constexpr (VARIANT == kCggiBinary) {
                        acc[half(h) + u] = make_ulonglong2(gl_add(v.x, g.x), gl_add(v.y, g.y));
                    } else {
                        const ulonglong2 w = rot_pair<LOGK>([&](uint32_t j) { return gh[j]; }, u, a);
                        acc[half(h) + u] = make_ulonglong2(gl_add(v.x, gl_sub(w.x, g.x)), gl_add(v.y, gl_sub(w.y, g.y)));
                    }
                }
            }
            __syncthreads();
        }

        uint64_t* res = prm.out + b * (2ull * N);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (c != last_of(h)) continue;
            for (int u = t; u < n; u += T) {
                ulonglong2 v = acc[half(h) + u];
                if constexpr (SIGNED) v = make_ulonglong2(gl_sub(v.x, prm.corr), gl_sub(v.y, prm.corr));
                res[h * N + u] = v.x;
                res[h * N + u + n] = v.y;
            }
        }
    }
    if (!ok) atomicOr(prm.err, 2u);
    cluster.sync();  // no block leaves while its copies to others are under way
}

// ---------------------------------------------------------------------------
// N = 4096: one rotation on a cluster of two blocks, block c holding accumulator half c (both
// halves with their digits' transforms, 6 x 32 KB at l = 3, do not fit one SM). Block c transforms
// the l digits of its half, multiplies slot half c of all 2l digits for both halves and all limbs,
// and transforms, rounds and recombines the L limb polynomials of its half, so that only slots
// cross: half of the digits' as bulk copies, half of the products as stores. The pass tables are
// read through L1 (no shared memory is left for them). 74 clusters are resident; ternary, l = 3, n
// = 60: 74 rotations 4.01 -> 1.58 ms, 148 4.02 -> 3.2 (modular -> here). Key batches 1 / 2 / 3
// ahead: 1.70 / 1.66 / 1.58 ms. Up to 15 rotations run on eight blocks each, above.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int br_fft_halves_threads(int logn, int limbs) { return (1 << (logn - 5)) * limbs; }
// Transform buffers (L polynomials), receive area (l half polynomials), accumulator half, monomial
// factors, barrier, LWE words (16-bit).
__host__ __device__ constexpr size_t br_fft_halves_smem(int logn, int dl, int limbs, uint32_t n) {
    const size_t k = (size_t)1 << (logn - 1);
    return (limbs * k + dl * (k / 2) + k + 5) * 16 + ((size_t)(n + 1 + 7) / 8) * 16;
}

template <int LOGN, int VARIANT, int DL, int L>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(br_fft_halves_threads(LOGN, L), 1)
br_fft_halves_kernel(const __grid_constant__ BrFftParams prm) {
    static_assert(VARIANT == kCggiBinary || VARIANT == kCggiTernary, "CGGI only");
    constexpr int LOGK = LOGN - 1;
    using F = Fft<LOGK>;
    constexpr int N = 1 << LOGN, n = F::n, TG = F::T;
    constexpr int G = br_rgsw_per_group(VARIANT);
    constexpr int C = 2 * G, R = 2 * DL;
    constexpr int T = br_fft_halves_threads(LOGN, L);
    constexpr int LANES = n / 16, M = 8;       // slots c n/2 + lane + m LANES of this thread, one limb
    constexpr uint32_t MASK2N = 2u * N - 1u;
    constexpr bool SIGNED = VARIANT != kCggiBinary;
    static_assert(DL <= L && TG * L == T && LANES * L == T, "block shape");

    if (prm.exact && !*prm.exact) return;
    extern __shared__ __align__(16) uint64_t smem[];
    double2* buf = reinterpret_cast<double2*>(smem);                     // L n
    double2* recv = buf + L * n;                                         // DL n/2: the other half's digits
    ulonglong2* acc = reinterpret_cast<ulonglong2*>(recv + DL * (n / 2));  // n: plus corr (signed)
    double2* mono_s = reinterpret_cast<double2*>(acc + n);               // 4: factors of the key's m = 4 c + q
    uint64_t* bar = reinterpret_cast<uint64_t*>(mono_s + 4);
    uint16_t* lwe_s = reinterpret_cast<uint16_t*>(mono_s + 5);

    auto cluster = cooperative_groups::this_cluster();
    const int c = (int)cluster.block_rank();
    const int t = threadIdx.x;
    const int grp = t / TG, tg = t % TG;
    const int limb = t / LANES, lane = t % LANES;
    uint32_t phase = 0;
    bool ok = true;  // a wait for the other block's digits ran out
    if (t == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    double2* buf_peer = cluster.map_shared_rank(buf, (unsigned)(c ^ 1));
    cluster.sync();  // both blocks running, their barriers set, before remote stores

    for (uint64_t b = blockIdx.x >> 1; b < prm.batch; b += gridDim.x >> 1) {
        __syncthreads();
        const uint64_t* lwe = prm.lwes + b * prm.lwe_stride;
        bool bad = false;
        for (uint32_t i = t; i <= prm.n; i += T) {
            const uint64_t v = lwe[i];
            bad |= v > MASK2N;
            lwe_s[i] = (uint16_t)(v & MASK2N);
        }
        if (bad && c == 0) atomicOr(prm.err, 1u);
        __syncthreads();
        {
            // acc = half c of acc_in X^b, plus the signed digits' corrector
            const uint64_t* a = prm.accs + b * prm.acc_stride + (uint64_t)c * N;
            const uint32_t s = (2u * N - lwe_s[prm.n]) & MASK2N;
            for (int u = t; u < n; u += T) {
                ulonglong2 v = rot_pair<LOGK>(
                    [&](uint32_t j) { return make_ulonglong2(gl_canon(a[j]), gl_canon(a[j + n])); }, u, s);
                if constexpr (SIGNED) v = make_ulonglong2(gl_add(v.x, prm.corr), gl_add(v.y, prm.corr));
                acc[u] = v;
            }
        }
        __syncthreads();

        auto prefetch = [&](uint32_t it) {  // this block's share of an iteration's key, as in the one-block form
            constexpr uint32_t bytes = (uint32_t)L * 8 * R * C * (n / 8) * 16;
            const uint32_t share = ((bytes + gridDim.x - 1) / gridDim.x + 127u) & ~127u;
            const uint32_t off = blockIdx.x * share;
            if (it < prm.n && off < bytes) l2_prefetch(reinterpret_cast<const char*>(prm.key) + (uint64_t)it * bytes + off,
                                                       min(share, bytes - off));
        };
        if (t == 0) {
            prefetch(0);
            prefetch(1);
        }
#pragma unroll 1
        for (uint32_t it = 0; it < prm.n; ++it) {
            if (t == 0) prefetch(it + 2);
            const uint32_t a = lwe_s[it];
            if (a == 0) continue;
            if (t == 0) mbar_expect(bar, DL * (n / 2) * 16);
            if constexpr (VARIANT == kCggiTernary) {
                if (t < 4) mono_s[t] = __ldg(prm.roots + ((4u * a * (__brev((uint32_t)(4 * c + t)) >> 29)) & MASK2N));
            }

            // ---- digits and forward transforms; the other half's slots to the other block ----
            const ulonglong2* src = acc;
            if constexpr (!SIGNED) {
                ulonglong2* d = reinterpret_cast<ulonglong2*>(buf);
                for (int u = t; u < n; u += T) d[u] = rotated_difference<LOGK>(acc, u, a);
                src = d;
                __syncthreads();
            }
            double2 x[16];
            if (grp < DL)
                digit_points<LOGK>(x, src, tg, prm.dshift[grp], (uint32_t)prm.dmask[grp],
                                   4503599627370496.0 + (SIGNED ? (double)prm.ddelta[grp] : 0.0));
            if constexpr (!SIGNED) __syncthreads();
            if (grp < DL) {
                F::head(x, prm.head);
                double2* pb = buf + grp * n;
#pragma unroll
                for (int i = 0; i < 16; ++i) pb[fft_pos(tg + i * TG)] = x[i];
                F::group_sync(grp);
                F::tail(pb, prm.tab_fwd, tg, grp, [&](int e, double2 v) { pb[fft_pos(e)] = v; });
                bulk_fence();
                F::group_sync(grp);
                if (tg == 0)
                    bulk_to_block(recv + grp * (n / 2), pb + (c ^ 1) * (n / 2), n / 2 * 16, bar, (uint32_t)(c ^ 1));
            }

            // ---- slot-wise products, one limb; rows of half c from buf, of the other from recv ----
            double2 o[M];
            {
                // slot lane + m LANES of this half is lane' = lane + (m & 1) LANES of the key's 4 c + m / 2
                const double2* kp = prm.key + (((uint64_t)it * L + limb) * 8 + 4 * c) * (R * C) * (n / 8) + lane;
                constexpr int BR = C == 4 ? 1 : 2, NB = M * R / BR;  // four loads a batch, AH batches ahead
                constexpr int AH = 3;
                static_assert(R % BR == 0, "a batch lies in one slot");
                double2 kv[AH + 1][BR][C];
                auto load = [&](int q, double2 (&k)[BR][C]) {
                    const int m = q * BR / R, r0 = q * BR % R;
#pragma unroll
                    for (int r = 0; r < BR; ++r)
#pragma unroll
                        for (int cc = 0; cc < C; ++cc)
                            k[r][cc] = key_ld(kp + (((m >> 1) * R + r0 + r) * C + cc) * (n / 8) + (m & 1) * LANES);
                };
#pragma unroll
                for (int q = 0; q < AH; ++q) load(q, kv[q]);
                double2 wb[2];
                if constexpr (VARIANT == kCggiTernary) {
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        wb[q] = __ldg(prm.roots + ((a * (1u + 32u * (__brev((uint32_t)(lane + q * LANES)) >> (35 - LOGK)))) & MASK2N));
                }
                __syncthreads();
                ok = ok && mbar_wait(bar, phase);
                phase ^= 1;
                double2 s[C];
#pragma unroll
                for (int q = 0; q < NB; ++q) {
                    const int m = q * BR / R, r0 = q * BR % R;
                    const int el = lane + m * LANES, e = c * (n / 2) + el;
                    if (q + AH < NB) load(q + AH, kv[(q + AH) % (AH + 1)]);
                    if (r0 == 0) {
#pragma unroll
                        for (int cc = 0; cc < C; ++cc) s[cc] = make_double2(0.0, 0.0);
                    }
#pragma unroll
                    for (int k = 0; k < BR; ++k) {
                        const int r = r0 + k;
                        const double2 xv = (r / DL) == c ? buf[(r % DL) * n + fft_pos(e)]
                                                         : recv[(r % DL) * (n / 2) + fft_pos(el)];
#pragma unroll
                        for (int cc = 0; cc < C; ++cc) cmac(s[cc], xv, kv[q % (AH + 1)][k][cc]);
                    }
                    if (r0 + BR != R) continue;
                    double2 v[2] = {s[0], s[1]};
                    if constexpr (VARIANT == kCggiTernary) {
                        const double2 w = cmul(wb[m & 1], mono_s[m >> 1]);
#pragma unroll
                        for (int h = 0; h < 2; ++h) v[h] = csubmul(s[h], w, s[C - 2 + h]);
                    }
                    buf_peer[limb * n + fft_pos(e)] = c ? v[0] : v[1];
                    o[m] = c ? v[1] : v[0];
                }
                cluster.sync();  // both blocks' reads of the digits done, products of the other half's slots here
#pragma unroll
                for (int m = 0; m < M; ++m) buf[limb * n + fft_pos(c * (n / 2) + lane + m * LANES)] = o[m];
                __syncthreads();
            }

            // ---- backward transforms, rounded coefficients back in place ----
            {
                double2* pb = buf + grp * n;
                F::itail(pb, prm.tab_inv, tg, grp, [&](int e) { return pb + fft_pos(e); });
                F::group_sync(grp);
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = pb[fft_pos(tg + i * TG)];
                F::ihead(x, prm.head);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    *reinterpret_cast<ulonglong2*>(pb + fft_pos(tg + i * TG)) =
                        make_ulonglong2(fft_round(x[i].x), fft_round(x[i].y));
            }
            __syncthreads();
            recombine_update<LOGK, VARIANT, L, T, 1>(buf, acc, t, a);
        }

        uint64_t* res = prm.out + b * (2ull * N) + (uint64_t)c * N;
        for (int u = t; u < n; u += T) {
            ulonglong2 v = acc[u];
            if constexpr (SIGNED) v = make_ulonglong2(gl_sub(v.x, prm.corr), gl_sub(v.y, prm.corr));
            res[u] = v.x;
            res[u + n] = v.y;
        }
    }
    if (!ok) atomicOr(prm.err, 2u);
    cluster.sync();  // no block leaves while the other may still store to it
}

}  // namespace tp
