// Tables, key transforms and the exactness bound of the double-precision transforms.
#include "fft_host.h"

#include <cmath>
#include <mutex>
#include <vector>

#include "br_fft_kernel.cuh"

namespace tp {
namespace {

uint32_t rev(uint32_t x, int bits) {
    uint32_t r = 0;
    for (int i = 0; i < bits; ++i) r |= ((x >> i) & 1u) << (bits - 1 - i);
    return r;
}

// tw[k], k = m + b: exp(i pi (1/(4m) + brv(b)/m)), the square root of block b's constant.
long double tw_angle(uint32_t k) {
    int lg = 0;
    while ((2u << lg) <= k) ++lg;
    const uint32_t m = 1u << lg, b = k - m;
    return acosl(-1.0L) * (0.25L + (long double)rev(b, lg)) / (long double)m;
}

std::mutex g_mu;
std::vector<FftTables*> g_tabs;

struct Dd { double h, l; };
__device__ __forceinline__ Dd dd_norm(double a, double b) {
    const double s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ Dd dd_add(Dd a, Dd b) {
    const double s = a.h + b.h;
    const double z = s - a.h;
    return dd_norm(s, (a.h - (s - z)) + (b.h - z) + (a.l + b.l));
}
__device__ __forceinline__ Dd dd_mul(Dd a, Dd b) {
    const double p = a.h * b.h;
    return dd_norm(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
__device__ __forceinline__ Dd dd_neg(Dd a) { return {-a.h, -a.l}; }

// One block per limb of a key polynomial, transformed by radix-2 levels in shared memory
// in double-double arithmetic (relative error near 2^-100), so that the stored doubles
// carry one rounding. Run once per key upload; bound by FP64 (about 150 operations a
// butterfly): 15120 polynomials of N = 2048 (three limbs) take a few milliseconds against
// the upload's tens.
__global__ void __launch_bounds__(256) fft_key_kernel(double2* __restrict__ dst, const uint64_t* __restrict__ src,
                                                      uint64_t polys, uint64_t first, uint32_t G, uint32_t rows,
                                                      int logk, int limbs, const double4* __restrict__ tw,
                                                      unsigned long long* __restrict__ norm2) {
    extern __shared__ double4 z[];  // n points (re.h, re.l, im.h, im.l)
    __shared__ unsigned long long part[8];
    const uint32_t n = 1u << logk, lanes = n >> 3;
    const int64_t base = fft_limb_base(limbs);
    const double scale = 1.0 / (double)n;
    for (uint64_t item = blockIdx.x; item < polys * limbs; item += gridDim.x) {
        const uint64_t p = item / limbs;
        const int l = (int)(item % limbs);
        const uint64_t* a = src + p * (2ull * n);
        const uint64_t id = first + p;
        const uint32_t h = (uint32_t)(id & 1), C = 2 * G;
        const uint64_t rig = id >> 1;
        const uint32_t r = (uint32_t)(rig % rows);
        const uint32_t g = (uint32_t)((rig / rows) % G);
        const uint64_t it = rig / rows / G;
        // limb l, balanced, of the word's representative in (-p/2, p/2)
        auto limb = [&](uint64_t x) -> int64_t {
            int64_t v = x > kP / 2 ? -(int64_t)(kP - x) : (int64_t)x;
            for (int q = 0;; ++q) {
                if (q == limbs - 1) return v;
                int64_t d = v % base;
                if (d > base / 2) d -= base;
                if (d < -(base / 2)) d += base;
                if (q == l) return d;
                v = (v - d) / base;
            }
        };
        unsigned long long sq = 0;
        __syncthreads();  // the previous limb's points are stored
        for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
            const int64_t x = limb(a[j]), y = limb(a[j + n]);
            sq += (unsigned long long)(x * x) + (unsigned long long)(y * y);
            z[j] = make_double4((double)x, 0.0, (double)y, 0.0);
        }
        for (int lg = 0; lg < logk; ++lg) {
            __syncthreads();
            const uint32_t m = 1u << lg, half = n >> (lg + 1);
            for (uint32_t q = threadIdx.x; q < n / 2; q += blockDim.x) {
                const uint32_t b = q / half, i0 = (q & (half - 1)) + b * 2 * half, i1 = i0 + half;
                const double4 w = tw[m + b], u = z[i0], v = z[i1];
                const Dd wr{w.x, w.y}, wi{w.z, w.w}, vr{v.x, v.y}, vi{v.z, v.w}, ur{u.x, u.y}, ui{u.z, u.w};
                const Dd pr = dd_add(dd_mul(wr, vr), dd_neg(dd_mul(wi, vi)));
                const Dd pi = dd_add(dd_mul(wr, vi), dd_mul(wi, vr));
                const Dd ar = dd_add(ur, pr), ai = dd_add(ui, pi);
                const Dd br = dd_add(ur, dd_neg(pr)), bi = dd_add(ui, dd_neg(pi));
                z[i0] = make_double4(ar.h, ar.l, ai.h, ai.l);
                z[i1] = make_double4(br.h, br.l, bi.h, bi.l);
            }
        }
        __syncthreads();
        double2* out = dst + (it * limbs + l) * (8ull * rows * C * lanes);
        for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) {
            const uint32_t m = e / lanes, lane = e & (lanes - 1);
            out[((uint64_t)(m * rows + r) * C + (2 * g + h)) * lanes + lane] =
                make_double2(z[e].x * scale, z[e].z * scale);
        }
        for (int o = 16; o; o >>= 1) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sq;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; ++w) sq += part[w];
            atomicMax(norm2, sq);
        }
    }
}

template <int LOGN, int VARIANT>
const void* pick_pair(uint32_t digits, int limbs) {
    switch (digits * 10 + limbs) {
        case 23: return (const void*)br_fft_pair_kernel<LOGN, VARIANT, 2, 3>;
        case 24: return (const void*)br_fft_pair_kernel<LOGN, VARIANT, 2, 4>;
        case 33: return (const void*)br_fft_pair_kernel<LOGN, VARIANT, 3, 3>;
        case 34: return (const void*)br_fft_pair_kernel<LOGN, VARIANT, 3, 4>;
        case 43: return (const void*)br_fft_pair_kernel<LOGN, VARIANT, 4, 3>;
        case 44: return (const void*)br_fft_pair_kernel<LOGN, VARIANT, 4, 4>;
        default: return nullptr;
    }
}

template <int LOGN, int VARIANT, int CS>
const void* pick_cluster(uint32_t digits, int limbs) {
    switch (digits * 10 + limbs) {
        case 23: return (const void*)br_fft_cluster_kernel<LOGN, VARIANT, 2, 3, CS>;
        case 24: return (const void*)br_fft_cluster_kernel<LOGN, VARIANT, 2, 4, CS>;
        case 33: return (const void*)br_fft_cluster_kernel<LOGN, VARIANT, 3, 3, CS>;
        case 34: return (const void*)br_fft_cluster_kernel<LOGN, VARIANT, 3, 4, CS>;
        case 43: return (const void*)br_fft_cluster_kernel<LOGN, VARIANT, 4, 3, CS>;
        case 44: return (const void*)br_fft_cluster_kernel<LOGN, VARIANT, 4, 4, CS>;
        default: return nullptr;
    }
}
template <int VARIANT>
const void* pick_cluster(int logn, uint32_t digits, int limbs, int cs) {
    if (logn == 10)
        return cs == 2   ? pick_cluster<10, VARIANT, 2>(digits, limbs)
               : cs == 4 ? pick_cluster<10, VARIANT, 4>(digits, limbs)
                         : pick_cluster<10, VARIANT, 8>(digits, limbs);
    if (logn == 12 && cs == 8 && limbs == 4)
        return digits == 2   ? (const void*)br_fft_cluster_kernel<12, VARIANT, 2, 4, 8>
               : digits == 3 ? (const void*)br_fft_cluster_kernel<12, VARIANT, 3, 4, 8>
               : digits == 4 ? (const void*)br_fft_cluster_kernel<12, VARIANT, 4, 4, 8>
                             : nullptr;
    if (logn == 11 && cs >= 4)
        return cs == 4 ? pick_cluster<11, VARIANT, 4>(digits, limbs) : pick_cluster<11, VARIANT, 8>(digits, limbs);
    return nullptr;
}

template <int LOGN, int VARIANT>
const void* pick(uint32_t digits, int limbs) {
    switch (digits * 10 + limbs) {
        case 23: return (const void*)br_fft_kernel<LOGN, VARIANT, 2, 3>;
        case 24: return (const void*)br_fft_kernel<LOGN, VARIANT, 2, 4>;
        case 33: return (const void*)br_fft_kernel<LOGN, VARIANT, 3, 3>;
        case 34: return (const void*)br_fft_kernel<LOGN, VARIANT, 3, 4>;
        case 43: return (const void*)br_fft_kernel<LOGN, VARIANT, 4, 3>;
        case 44: return (const void*)br_fft_kernel<LOGN, VARIANT, 4, 4>;
        default: return nullptr;
    }
}

}  // namespace

const void* br_fft_kernel_ptr(int logn, int variant, uint32_t digits, int limbs) {
    if (variant == kCggiBinary)
        return logn == 10 ? pick<10, kCggiBinary>(digits, limbs) : logn == 11 ? pick<11, kCggiBinary>(digits, limbs) : nullptr;
    if (variant == kCggiTernary)
        return logn == 10 ? pick<10, kCggiTernary>(digits, limbs) : logn == 11 ? pick<11, kCggiTernary>(digits, limbs) : nullptr;
    return nullptr;
}

const void* br_fft_halves_ptr(int logn, int variant, uint32_t digits, int limbs) {
    if (logn != 12 || limbs != 4 || digits < 2 || digits > 4) return nullptr;
    if (variant == kCggiBinary)
        return digits == 2   ? (const void*)br_fft_halves_kernel<12, kCggiBinary, 2, 4>
               : digits == 3 ? (const void*)br_fft_halves_kernel<12, kCggiBinary, 3, 4>
                             : (const void*)br_fft_halves_kernel<12, kCggiBinary, 4, 4>;
    if (variant == kCggiTernary)
        return digits == 2   ? (const void*)br_fft_halves_kernel<12, kCggiTernary, 2, 4>
               : digits == 3 ? (const void*)br_fft_halves_kernel<12, kCggiTernary, 3, 4>
                             : (const void*)br_fft_halves_kernel<12, kCggiTernary, 4, 4>;
    return nullptr;
}

const void* br_fft_pair_ptr(int logn, int variant, uint32_t digits, int limbs) {
    if (variant == kCggiBinary)
        return logn == 10 ? pick_pair<10, kCggiBinary>(digits, limbs) : logn == 11 ? pick_pair<11, kCggiBinary>(digits, limbs) : nullptr;
    if (variant == kCggiTernary)
        return logn == 10 ? pick_pair<10, kCggiTernary>(digits, limbs) : logn == 11 ? pick_pair<11, kCggiTernary>(digits, limbs) : nullptr;
    return nullptr;
}

const void* br_fft_cluster_ptr(int logn, int variant, uint32_t digits, int limbs, int cs) {
    if (variant == kCggiBinary) return pick_cluster<kCggiBinary>(logn, digits, limbs, cs);
    if (variant == kCggiTernary) return pick_cluster<kCggiTernary>(logn, digits, limbs, cs);
    return nullptr;
}

cudaError_t fft_tables(int device, int logk, const FftTables** out) {
    std::lock_guard<std::mutex> lk(g_mu);
    for (auto* t : g_tabs)
        if (t->device == device && t->logk == logk) {
            *out = t;
            return cudaSuccess;
        }
    const uint32_t n = 1u << logk, B2 = (uint32_t)fft_blocks2(logk), B3 = n / 8, len = (uint32_t)fft_table_len(logk);
    auto ratio = [](uint32_t k) {
        const long double a = tw_angle(k);
        return make_double2((double)cosl(a), (double)(sinl(a) / cosl(a)));
    };
    auto plain = [](uint32_t k) {
        const long double a = tw_angle(k);
        return make_double2((double)cosl(a), (double)sinl(a));
    };
    std::vector<double2> f(len), v(len), roots(4 * n);
    std::vector<double4> dd(n);
    auto fill = [&](uint32_t off, uint32_t blocks, int entries) {
        for (uint32_t b = 0; b < blocks; ++b) {
            const uint32_t k[8] = {blocks + b,             2 * blocks + 2 * b,     4 * blocks + 4 * b,     4 * blocks + 4 * b + 2,
                                   8 * blocks + 8 * b,     8 * blocks + 8 * b + 2, 8 * blocks + 8 * b + 4, 8 * blocks + 8 * b + 6};
            for (int q = 0; q < entries; ++q) {
                f[off + q * blocks + b] = ratio(k[q]);
                v[off + q * blocks + b] = plain(k[q]);
            }
        }
    };
    fill(0, B2, fft_entries2(logk));
    fill(fft_entries2(logk) * B2, B3, 4);
    for (uint32_t k = 0; k < 4 * n; ++k) {
        const long double a = acosl(-1.0L) * (long double)k / (long double)(2 * n);
        roots[k] = make_double2((double)cosl(a), (double)sinl(a));
    }
    dd[0] = make_double4(1.0, 0.0, 0.0, 0.0);
    for (uint32_t k = 1; k < n; ++k) {
        const long double c = cosl(tw_angle(k)), s = sinl(tw_angle(k));
        const double ch = (double)c, sh = (double)s;
        dd[k] = make_double4(ch, (double)(c - (long double)ch), sh, (double)(s - (long double)sh));
    }
    auto* t = new FftTables();
    t->device = device;
    t->logk = logk;
    t->head.fwd[0] = t->head.inv[0] = make_double2(1.0, 0.0);
    for (uint32_t k = 1; k < 16; ++k) {
        t->head.fwd[k] = ratio(k);
        t->head.inv[k] = plain(k);
    }
    cudaError_t e = cudaSuccess;
    auto put = [&](auto** dst, const auto& src) {
        if (e == cudaSuccess) e = cudaMalloc(dst, src.size() * sizeof(src[0]));
        if (e == cudaSuccess) e = cudaMemcpy(*dst, src.data(), src.size() * sizeof(src[0]), cudaMemcpyHostToDevice);
    };
    put(&t->pass_fwd, f);
    put(&t->pass_inv, v);
    put(&t->roots, roots);
    put(&t->dd, dd);
    if (e != cudaSuccess) {
        cudaFree(t->pass_fwd);
        cudaFree(t->pass_inv);
        cudaFree(t->roots);
        cudaFree(t->dd);
        delete t;
        return e;
    }
    g_tabs.push_back(t);
    *out = t;
    return cudaSuccess;
}

bool fft_exact(int logk, uint32_t rows, double dmax, double norm2, int limbs, int sets) {
    const double N = std::ldexp(1.0, logk + 1);
    const double s = sets * (double)rows * dmax * std::sqrt(N) * std::sqrt(norm2);
    const double units = 4.0 * logk + 1.0 + std::sqrt(2.0) * (rows + 1.0) + (sets > 1 ? 6.0 : 0.0) + 3.71 * logk;
    const double largest = sets * (double)rows * N * dmax * (fft_limb_base(limbs) / 2 + 2.0);
    return s * units * std::ldexp(1.0, -53) < 0.49 && largest < std::ldexp(1.0, 51);
}

double fft_random_norm2(int logk, int limbs, uint64_t polys, double share) {
    // N squares of numbers uniform in [-b/2, b/2]: mean N b^2 / 12, deviation sqrt(0.8 / N) of it, close
    // to normal; the largest of m such sums exceeds z deviations in m Q(z) of the keys (m Q(z) small)
    const double b = (double)fft_limb_base(limbs), N = std::ldexp(1.0, logk + 1), m = (double)polys * limbs;
    double lo = 0.0, hi = 20.0;
    for (int i = 0; i < 60; ++i) {
        const double z = 0.5 * (lo + hi);
        (m * 0.5 * std::erfc(z / std::sqrt(2.0)) > share ? lo : hi) = z;
    }
    return N * b * b / 12.0 * (1.0 + hi * std::sqrt(0.8 / N));
}

void fft_key_launch(double2* dst, const uint64_t* src, uint64_t polys, uint64_t first, uint32_t G, uint32_t rows,
                    int limbs, const FftTables& tab, unsigned long long* norm2, cudaStream_t st) {
    const size_t smem = sizeof(double4) << tab.logk;  // 32 KB at 1024 points
    if (smem > 48u * 1024u)
        cudaFuncSetAttribute(fft_key_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const uint64_t items = polys * limbs;
    const unsigned blocks = (unsigned)(items < 4096 ? items : 4096);
    fft_key_kernel<<<blocks, 256, smem, st>>>(dst, src, polys, first, G, rows, tab.logk, limbs, tab.dd, norm2);
}

}  // namespace tp
