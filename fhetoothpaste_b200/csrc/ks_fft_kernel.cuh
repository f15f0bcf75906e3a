// Automorphism key switches whose result stays in the coefficient domain (packing merges,
// trace steps, truncation splits; ks_kernels.cuh) with double-precision transforms
// (fft_block.cuh): same words, N = 1024 and 2048, where the key passes the error bound.
//
// One block per item. The modular kernel transforms l digits and the automorphism's B part
// forward and two sums backward; here nothing but the digit products passes through the
// evaluation domain: l forward FFTs at once, the slots' l rows times the key's limbs, 2L
// backward FFTs at once, and the recombined words are added to the coefficients that the
// item's loads left in shared memory. The key (512 KB at N = 2048, l = L = 4) is read from L2
// by every block at the same time, like the rotation's.
#pragma once

#include "br_fft_kernel.cuh"
#include "ks_kernels.cuh"

namespace tp {

struct KsFftParams {
    KsKernelParams ks;        // `key` unused
    const double2* key;       // [limb][m < 8][row][half][lane < n/8]
    const double2* tab_fwd;
    const double2* tab_inv;
    int mode;                 // kKsMerge, kKsTrace or kKsSplit
    FftHead head;
};

__host__ __device__ constexpr int ks_fft_threads(int logn, int limbs) { return (1 << (logn - 4)) * limbs; }
// Transform buffers (2L polynomials), the item's A difference (later the first products), its
// sums (2n) and B difference, pass tables.
__host__ __device__ constexpr size_t ks_fft_smem(int logn, int limbs) {
    return (((size_t)2 * limbs + 4) << (logn - 1)) * 16 + (size_t)2 * fft_table_len(logn - 1) * 16;
}

template <int LOGN, int DL, int L>
__global__ void __launch_bounds__(ks_fft_threads(LOGN, L), LOGN <= 10 ? 2 : 1)
ks_fft_kernel(const __grid_constant__ KsFftParams prm) {
    constexpr int LOGK = LOGN - 1;
    using F = Fft<LOGK>;
    constexpr int N = 1 << LOGN, n = F::n, TG = F::T, LANES = n / 8, T = LANES * L;
    static_assert(T == TG * 2 * L && DL <= 2 * L, "block shape");

    if (prm.ks.exact && !*prm.ks.exact) return;
    extern __shared__ __align__(16) uint64_t smem[];
    double2* buf = reinterpret_cast<double2*>(smem);                  // 2L n
    ulonglong2* as = reinterpret_cast<ulonglong2*>(buf + 2 * L * n);  // n: aut(diff).A plus corr
    double2* spare = reinterpret_cast<double2*>(as);                  // the first eighth's products
    uint64_t* base = reinterpret_cast<uint64_t*>(as + n);             // 2N: sums
    ulonglong2* bs = as + 3 * n;                                      // n: aut(diff).B
    double2* tab_f = reinterpret_cast<double2*>(bs + n);
    double2* tab_i = tab_f + fft_table_len(LOGK);
    static_assert(2 * L * LANES <= n, "the first eighth's products fit over the A difference");

    const KsKernelParams& ks = prm.ks;
    const int t = threadIdx.x;
    const int grp = t / TG, tg = t % TG;
    const int limb = t / LANES, lane = t % LANES;
    for (int i = t; i < fft_table_len(LOGK); i += T) {
        tab_f[i] = prm.tab_fwd[i];
        tab_i[i] = prm.tab_inv[i];
    }
    const bool merge = prm.mode == kKsMerge;

    for (uint64_t it = blockIdx.x; it < ks.items; it += gridDim.x) {
        __syncthreads();
        uint64_t* out = ks.out + it * ks.out_stride;
        // ---- sums (kept) and differences (in the transform buffers) of the item's nodes: all global
        // reads of the item, coalesced; the next item's nodes are requested into L2 ----
        uint64_t* diff = reinterpret_cast<uint64_t*>(buf);  // 2N
        constexpr int W = (N + T - 1) / T;
        auto store = [&](int k, uint64_t r, uint64_t l, bool wrap) {
            if (merge) {
                if (wrap) l = gl_neg(l);
                diff[k] = gl_sub(r, l);
                base[k] = gl_add(r, l);
            } else {
                diff[k] = r;
                base[k] = r;
            }
        };
        if (ks.leaf) {
            // leaf of row x: A = (x_0, -x_{N-1}, .., -x_1) / N, B = (x_N, 0, .., 0) / N
            const uint64_t len = 1ull << ks.leaf_log, p = it >> (ks.leaf_log - 1), q = it & (len / 2 - 1);
            auto row_of = [&](uint32_t c) {
                return ks.leaf + (p * len + (((uint32_t)len - 1) ^ (__brev(c) >> (32 - ks.leaf_log)))) * (N + 1);
            };
            const uint64_t* left = row_of((uint32_t)(2 * q));
            const uint64_t* right = row_of((uint32_t)(2 * q) + 1);
            uint64_t r[W], l[W];
            auto leaf = [](uint64_t x, uint32_t k) { return gl_div_pow2<LOGN>(k ? gl_neg(x) : x); };
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const uint32_t m = t + k * T, ml = (m - ks.shift) & (N - 1);
                if (N % T != 0 && m >= N) continue;
                r[k] = right[m ? N - m : 0];
                l[k] = left[ml ? N - ml : 0];
            }
            const uint64_t rb = gl_div_pow2<LOGN>(right[N]), lb = gl_div_pow2<LOGN>(left[N]);
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const uint32_t m = t + k * T, ml = (m - ks.shift) & (N - 1);
                if (N % T != 0 && m >= N) continue;
                store(m, leaf(r[k], m), leaf(l[k], ml), m < ks.shift);
                store(N + m, m ? 0 : rb, ml ? 0 : lb, false);  // X^shift moves b to `shift` below N
            }
        } else {
            const uint64_t* left;
            const uint64_t* right;
            auto nodes_of = [&](uint64_t item) {
                left = ks.in + item * ks.in_stride;
                right = left + (merge ? ks.right_offset : 0);
                if (merge && ks.pairs) {
                    const uint64_t pk = item / ks.pair_count, q = item % ks.pair_count;
                    const uint32_t ls = ks.pairs[2 * q], rs = ks.pairs[2 * q + 1];
                    const uint64_t* nodes = ks.in + pk * ks.prev_count * ks.in_stride;
                    left = ls == kNoNode ? ks.zero : nodes + ls * ks.in_stride;
                    right = rs == kNoNode ? ks.zero : nodes + rs * ks.in_stride;
                }
            };
            if (t == 0 && it + gridDim.x < ks.items) {
                nodes_of(it + gridDim.x);
                if (((uintptr_t)right & 15) == 0) l2_prefetch(right, 2 * N * 8);
                if (merge && ((uintptr_t)left & 15) == 0) l2_prefetch(left, 2 * N * 8);
            }
            nodes_of(it);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint64_t r[W], l[W];
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const uint32_t m = t + k * T;
                    if (N % T != 0 && m >= N) continue;
                    r[k] = right[h * N + m];
                    l[k] = merge ? left[h * N + ((m - ks.shift) & (N - 1))] : 0;
                }
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const uint32_t m = t + k * T;
                    if (N % T == 0 || m < N) store(h * N + m, r[k], l[k], m < ks.shift);
                }
            }
        }
        __syncthreads();
        // ---- the differences under the automorphism: coefficient m comes from m t^-1 ----
#pragma unroll
        for (int j = t; j < n; j += T) {
            uint64_t d[2][2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t i = ((uint32_t)(j + q * n) * ks.auto_index_inv) & (2 * N - 1), src = i & (N - 1);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint64_t v = diff[h * N + src];
                    d[h][q] = i >= N ? gl_neg(v) : v;
                }
            }
            as[j] = make_ulonglong2(gl_add(d[0][0], ks.corr), gl_add(d[0][1], ks.corr));
            bs[j] = make_ulonglong2(d[1][0], d[1][1]);
        }
        __syncthreads();

        // ---- digits and forward transforms ----
        if (grp < DL) {
            const uint32_t sh = ks.dshift[grp];
            const uint32_t mk = (uint32_t)ks.dmask[grp];
            const double off = 4503599627370496.0 + (double)ks.ddelta[grp];
            double2 x[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const ulonglong2 v = as[tg + i * TG];
                x[i] = make_double2(__hiloint2double(0x43300000, (int)((uint32_t)(v.x >> sh) & mk)) - off,
                                    __hiloint2double(0x43300000, (int)((uint32_t)(v.y >> sh) & mk)) - off);
            }
            F::head(x, prm.head);
            double2* pb = buf + grp * n;
#pragma unroll
            for (int i = 0; i < 16; ++i) pb[fft_pos(tg + i * TG)] = x[i];
            F::group_sync(grp);
            F::tail(pb, tab_f, tg, grp, [&](int e, double2 v) { pb[fft_pos(e)] = v; });
        }

        // ---- slot-wise products, slots lane + m LANES of one limb ----
        {
            constexpr int BR = DL % 2 == 0 ? 2 : DL, NB = 8 * DL / BR;
            const double2* kp = prm.key + (uint64_t)limb * (8 * DL * 2) * LANES + lane;
            double2 kv[2][BR][2], o[2][7], s[2];
            auto load = [&](int q, double2 (&k)[BR][2]) {
#pragma unroll
                for (int r = 0; r < BR; ++r)
#pragma unroll
                    for (int h = 0; h < 2; ++h) k[r][h] = key_ld(kp + ((q * BR + r) * 2 + h) * LANES);
            };
            load(0, kv[0]);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                const int m = q * BR / DL, pos = fft_pos(lane + m * LANES);
                if (q + 1 < NB) load(q + 1, kv[(q + 1) & 1]);
                if (q * BR % DL == 0) s[0] = s[1] = make_double2(0.0, 0.0);
#pragma unroll
                for (int r = 0; r < BR; ++r) {
                    const double2 x = buf[(q * BR % DL + r) * n + pos];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const double2 k = kv[q & 1][r][h];
                        s[h].x = fma(x.x, k.x, s[h].x);
                        s[h].y = fma(x.x, k.y, s[h].y);
                        s[h].x = fma(-x.y, k.y, s[h].x);
                        s[h].y = fma(x.y, k.x, s[h].y);
                    }
                }
                if ((q + 1) * BR % DL != 0) continue;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (m == 0) spare[(h * L + limb) * LANES + pos] = s[h];
                    else o[h][m - 1] = s[h];
                }
            }
            __syncthreads();  // every read of the digits' slots before the products take their place
#pragma unroll
            for (int m = 1; m < 8; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) buf[(h * L + limb) * n + fft_pos(lane + m * LANES)] = o[h][m - 1];
            __syncthreads();
        }

        // ---- backward transforms, rounded limbs in place ----
        {
            double2* pb = buf + grp * n;
            F::itail(pb, tab_i, tg, grp, [&](int e) { return (e < LANES ? spare + grp * LANES : pb) + fft_pos(e); });
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

        // ---- words mod p: y = -KS.A | aut(diff).B - KS.B, added to the sums ----
        const ulonglong2* wb = reinterpret_cast<const ulonglong2*>(buf);
#pragma unroll
        for (int u = t; u < 2 * n; u += T) {
            const int h = u >> LOGK, j = u & (n - 1), pos = fft_pos(j);
            uint64_t cx[L], cy[L];
#pragma unroll
            for (int l = 0; l < L; ++l) {
                const ulonglong2 v = wb[(h * L + l) * n + pos];
                cx[l] = v.x;
                cy[l] = v.y;
            }
            uint64_t y[2] = {fft_recombine<L>(cx), fft_recombine<L>(cy)};
            if (h == 0) {
                y[0] = gl_neg(y[0]);
                y[1] = gl_neg(y[1]);
            } else {
                const ulonglong2 v = bs[j];
                y[0] = gl_sub(v.x, y[0]);
                y[1] = gl_sub(v.y, y[1]);
            }
            const uint64_t sv[2] = {base[h * N + j], base[h * N + j + n]};
            out[h * N + j] = gl_add(sv[0], y[0]);
            out[h * N + j + n] = gl_add(sv[1], y[1]);
            if (prm.mode == kKsSplit) {  // the other child: X^-shift (x - y)
                uint64_t* out1 = out + ks.right_offset + h * N;
                const uint64_t z[2] = {gl_sub(sv[0], y[0]), gl_sub(sv[1], y[1])};
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const uint32_t m = (uint32_t)(j + q * n);
                    if (m >= ks.shift) out1[m - ks.shift] = z[q];
                    else out1[m + N - ks.shift] = gl_neg(z[q]);
                }
            }
        }
    }
}

}  // namespace tp
