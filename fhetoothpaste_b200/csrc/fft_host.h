// Host side of the double-precision transforms (fft_block.cuh): tables, key
// transforms, the exactness bound, kernel lookup. Library-internal.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_block.cuh"

namespace tp {

// Device tables of one (device, n = 2^logk points); shared by every context, kept.
struct FftTables {
    int device, logk;
    double2* pass_fwd;   // fft_table_len(logk)
    double2* pass_inv;
    double2* roots;      // exp(2 pi i k / 4n), k < 4n
    double4* dd;         // tw[k] in double-double (re.h, re.l, im.h, im.l), k < n
    FftHead head;
};
cudaError_t fft_tables(int device, int logk, const FftTables** out);

// Upper bound on the absolute error of a product coefficient before rounding: `rows`
// digit polynomials of coefficients at most dmax against limb polynomials of squared
// 2-norm at most norm2, `sets` such sums combined with unit weights. Below 1/2 every
// coefficient rounds to the exact integer. With u = 2^-53 and S = sets rows dmax
// sqrt(N) sqrt(norm2), errors in the 2-norm forward and summed over slots after it:
//   forward, per level: 4u (rounding of v (1 + i t), of c and of t: u |v| each, of the
//     sum: u), relative in the 2-norm, which the butterflies scale;
//   key: u (transformed in double-double);
//   products: each of the 2 rows FMAs of a component rounds the terms before it:
//     sqrt(2) (rows + 1) u on average over rows of equal norm;
//   combining two sets: 6u (X^a from two rounded roots: 3.4u; two FMAs);
//   backward, per level: 3.71u of the slots' absolute sum (sum: u, product: 2u,
//     twiddle: 0.71u), and (1/n) sum |E_e| <= S by Cauchy-Schwarz.
// The magnitude condition of the rounding (below 2^51) is part of the test.
bool fft_exact(int logk, uint32_t rows, double dmax, double norm2, int limbs, int sets);

// The squared norm that the largest limb polynomial of a key of `polys` polynomials of uniformly
// random words exceeds in `share` of the keys.
double fft_random_norm2(int logk, int limbs, uint64_t polys, double share);

// Limb counts in the order of preference: the fewest (less key to read, fewer transforms) whose bound
// one key of a thousand fails, four where most keys pass, three where most keys pass.
struct FftLimbs { int limbs; double share; };
constexpr FftLimbs kFftLimbs[] = {{3, 1e-3}, {4, 0.5}, {3, 0.5}};

// Whether a key's transforms of `bytes` may be allocated out of `room` free bytes.
constexpr bool fft_key_fits(uint64_t bytes, uint64_t room) { return bytes <= room / 8; }
static_assert(fft_key_fits(1, 8) && !fft_key_fits(2, 15) && fft_key_fits(1ull << 32, 1ull << 35));

// Transforms `polys` key polynomials of N = 2n canonical coefficient words: polynomial
// first + i sits at src + i N and is ((it G + g) rows + r) 2 + h of the key, stored as
// [it][limb][m < 8][r][2g + h][lane < n/8] double2 (slot lane + m n/8), scaled by 1/n.
// *norm2 is raised to the largest squared 2-norm of a limb polynomial.
void fft_key_launch(double2* dst, const uint64_t* src, uint64_t polys, uint64_t first, uint32_t G, uint32_t rows,
                    int limbs, const FftTables& tab, unsigned long long* norm2, cudaStream_t st);

const void* br_fft_kernel_ptr(int logn, int variant, uint32_t digits, int limbs);
// One rotation on a cluster of two blocks, an accumulator half each (N = 4096).
const void* br_fft_halves_ptr(int logn, int variant, uint32_t digits, int limbs);
// Two rotations on a cluster of two blocks.
const void* br_fft_pair_ptr(int logn, int variant, uint32_t digits, int limbs);
// One rotation on a cluster of cs blocks (2, 4 or 8; nullptr where not built).
const void* br_fft_cluster_ptr(int logn, int variant, uint32_t digits, int limbs, int cs);

// Key switches with coefficient results (ks_fft_kernel.cuh).
const void* ks_fft_kernel_ptr(int logn, uint32_t digits, int limbs);

}  // namespace tp
