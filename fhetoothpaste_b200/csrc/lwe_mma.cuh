// LWE -> LWE key switching as an 8-bit matrix product on the tensor cores (tcgen05).
//
// The sum over input coefficients i and digits j of raw_ij(row) * ksk[i][j][col]
// (lwe_conversion.cpp:205-239; the signed offset is a constant per column, see
// lwe_ks_kernel) is a contraction of length K = n_in * l over integers: digits below 2^16
// are one or two byte planes, a key word is eight bytes, and a product of byte matrices
// with K <= 33024 is exact in 32-bit sums (255^2 K < 2^31). Output word (row, col) is
//   sum_{d < planes} sum_{b < 8} 2^(8 (d + b)) (plane_d . key_b)[row][col]  mod p,
// so the tile's columns are the bytes of 32 output words and each digit plane has its own
// accumulator: both planes' products share one key tile.
//
// Three launches: digit planes of the batch (K-major bytes), the product, and the sum over
// the splits of K with the output update. The product runs on 128 x 256 tiles (128
// ciphertexts, 32 words) with 128-byte K steps: 64 KB of TMA loads (three stages) against
// 1084 clocks of the tensor pipe, 60 of the 75 bytes a clock that an SM gets from L2; two
// accumulators of 256 columns fill TMEM. K is split over several blocks per tile where the
// tiles alone leave the last wave, or the GPU, idle. Measured against lwe_ks_kernel (2048 -> 630,
// base 2^16, l = 4): 4096 ciphertexts 10.80 ms -> 0.329 ms (the product alone 0.242 ms: 1.40 P byte
// products a second, the tensor pipe busy three quarters of the time), 100 of them 1803 -> 25 us,
// one 1764 -> 25 us. A context's first call maps its workspace as well: 1.3 ms at this size.
#pragma once

#include <cuda.h>
#include <stdint.h>

#include "gl_arith.cuh"
#include "ks_util_kernels.cuh"
#include "lwe_mma_plan.h"
#include "mbar.cuh"

namespace tp {

constexpr int kMmaStages = 3;
constexpr int kMmaThreads = 192;                                // warps 0-3 epilogue, 4 loads, 5 products
__host__ __device__ constexpr size_t mma_stage_bytes(int planes) { return (size_t)(planes * kMmaRows + kMmaCols) * kMmaK; }
__host__ __device__ constexpr size_t mma_smem(int planes) { return kMmaStages * mma_stage_bytes(planes) + 1024 + 128; }

struct LweMmaParams {
    uint64_t* part;       // splits x rows x width partial sums, canonical
    uint32_t rows, rows_pad, width, steps, splits;
    int* err;             // host-mapped: set when a wait ran out
};

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
// K-major operand tile, rows of 128 bytes in the 128-byte swizzle (8-row atoms of 1024 bytes).
__device__ __forceinline__ uint64_t mma_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// u8 x u8 -> s32, M = 128, N = 256, both K-major.
constexpr uint32_t kMmaIdesc = (2u << 4) | ((uint32_t)(kMmaCols >> 3) << 17) | ((uint32_t)(kMmaRows >> 4) << 24);

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(kMmaIdesc), "r"((uint32_t)accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t (&v)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
}

// Block (m, n, split): rows 128 m.., words 32 n.., K steps of its share.
template <int PLANES>
__global__ void __launch_bounds__(kMmaThreads, 1)
lwe_mma_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap,
               const __grid_constant__ LweMmaParams prm) {
    extern __shared__ uint8_t raw[];
    uint8_t* base = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    constexpr uint32_t stage_bytes = (uint32_t)mma_stage_bytes(PLANES);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + kMmaStages * stage_bytes);
    uint64_t* empty = full + kMmaStages;
    uint64_t* done = empty + kMmaStages;
    uint32_t* tmem_s = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t share = (prm.steps + prm.splits - 1) / prm.splits;
    const uint32_t s0 = blockIdx.z * share;
    const uint32_t steps = s0 < prm.steps ? min(share, prm.steps - s0) : 0u;
    constexpr uint32_t tmem_cols = PLANES * kMmaCols;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMmaStages; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        mbar_init(done, 1);
        mbar_init_fence();
    }
    if (warp == 5)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_s)),
                     "n"(tmem_cols)
                     : "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_s;

    bool ok = true;
    if (warp == 4) {
        if (lane == 0) {
            uint32_t i = 0;
            for (; i < steps && ok; ++i) {
                const uint32_t s = i % kMmaStages, ph = (i / kMmaStages) & 1;
                ok = mbar_wait(empty + s, ph ^ 1);
                if (!ok) break;
                uint8_t* st = base + s * stage_bytes;
                mbar_expect(full + s, stage_bytes);
                const int x = (int)((s0 + i) * kMmaK);
#pragma unroll
                for (int d = 0; d < PLANES; ++d)
                    tma_load_2d(st + d * (kMmaRows * kMmaK), &amap, x, (int)(d * prm.rows_pad + blockIdx.x * kMmaRows),
                                full + s);
                tma_load_2d(st + PLANES * (kMmaRows * kMmaK), &bmap, x, (int)(blockIdx.y * kMmaCols), full + s);
            }
            if (!ok)  // the copies in flight land before the block leaves
                for (uint32_t j = i > kMmaStages ? i - kMmaStages : 0; j < i; ++j)
                    mbar_wait(full + j % kMmaStages, (j / kMmaStages) & 1);
        }
    } else if (warp == 5) {
        if (lane == 0) {
            for (uint32_t i = 0; i < steps && ok; ++i) {
                const uint32_t s = i % kMmaStages, ph = (i / kMmaStages) & 1;
                ok = mbar_wait(full + s, ph);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a = smem_u32(base + s * stage_bytes);
                const uint64_t bd = mma_desc(a + PLANES * (kMmaRows * kMmaK));
#pragma unroll
                for (int k = 0; k < kMmaK / 32; ++k)
#pragma unroll
                    for (int d = 0; d < PLANES; ++d)
                        mma_i8(tmem + d * kMmaCols, mma_desc(a + d * (kMmaRows * kMmaK)) + 2 * k, bd + 2 * k,
                               i > 0 || k > 0);
                mma_commit(empty + s);
            }
            mma_commit(done);
        }
    } else if (steps) {
        ok = mbar_wait(done, 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t row = blockIdx.x * kMmaRows + threadIdx.x;
        const uint32_t col0 = blockIdx.y * kMmaWords;
        uint64_t* dst = prm.part + ((uint64_t)blockIdx.z * prm.rows + row) * prm.width + col0;
#pragma unroll 1
        for (int w = 0; w < kMmaWords; w += 2) {
            uint32_t v[PLANES][16];
            __syncwarp();
#pragma unroll
            for (int d = 0; d < PLANES; ++d)
                tmem_ld16(v[d], tmem + ((uint32_t)(warp * 32) << 16) + d * kMmaCols + w * 8);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                // sum_b 2^(8b) (v0 + 2^8 v1), below 2^97
                unsigned __int128 sum = 0;
#pragma unroll
                for (int b = 7; b >= 0; --b) {
                    uint64_t tb = v[0][q * 8 + b];
                    if constexpr (PLANES == 2) tb += (uint64_t)v[PLANES - 1][q * 8 + b] << 8;
                    sum = (sum << 8) + tb;
                }
                if (ok && row < prm.rows && col0 + w + q < prm.width)
                    dst[w + q] = gl_reduce128((uint32_t)sum, (uint32_t)(sum >> 32), (uint32_t)(sum >> 64),
                                              (uint32_t)(sum >> 96));
            }
        }
    }
    if (!ok) *(volatile int*)prm.err = 1;
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 5) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(tmem_cols) : "memory");
    }
}

// tp_debug_lwe_timeout: a wait on a barrier that nothing completes, reported as lwe_mma_kernel reports its own.
__global__ void lwe_timeout_kernel(int* err) {
    __shared__ uint64_t bar;
    mbar_init(&bar, 1);
    mbar_init_fence();
    if (!mbar_wait(&bar, 0, 64)) *(volatile int*)err = 1;
}

// Byte planes of the digits of rows row0 .. row0 + rows - 1: plane d, row r, position
// k = i l + j holds byte d of (x_i + corr) >> dshift[j] & dmask[j]; zero past n_in l. A
// thread makes 16 neighbouring positions (16-byte stores).
template <int PLANES>
__global__ void __launch_bounds__(256) lwe_digits_kernel(uint8_t* __restrict__ planes, const LweKsParams prm,
                                                         uint64_t row0, uint32_t rows, uint32_t rows_pad,
                                                         uint32_t kpad) {
    const uint32_t quads = kpad / 16, L = prm.digits;
    const uint64_t total = (uint64_t)rows * quads;
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < total;
         q += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(q / quads), k0 = (uint32_t)(q - (uint64_t)r * quads) * 16;
        uint32_t lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
        uint32_t i = k0 / L, j = k0 - i * L;
        uint64_t x = i < prm.n_in ? gl_add(lwe_ks_in_word(prm, row0 + r, i), prm.corr) : 0;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const uint32_t v = i < prm.n_in ? (uint32_t)((x >> prm.dshift[j]) & prm.dmask[j]) : 0u;
            lo[e / 4] |= (v & 255u) << (8 * (e % 4));
            hi[e / 4] |= (v >> 8) << (8 * (e % 4));
            if (++j == L) {
                j = 0;
                ++i;
                if (e < 15 && i < prm.n_in) x = gl_add(lwe_ks_in_word(prm, row0 + r, i), prm.corr);
            }
        }
        uint8_t* d = planes + (uint64_t)r * kpad + k0;
        *reinterpret_cast<uint4*>(d) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        if constexpr (PLANES == 2)
            *reinterpret_cast<uint4*>(d + (uint64_t)rows_pad * kpad) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    }
}

// Key bytes, K-major: row col * 8 + b of kpad bytes holds byte b of ksk[k][col], zero past K.
__global__ void __launch_bounds__(256) lwe_key_bytes_kernel(uint8_t* __restrict__ dst, const uint64_t* __restrict__ ksk,
                                                            uint32_t K, uint32_t kpad, uint32_t width) {
    const uint64_t total = (uint64_t)width * (kpad / 16);
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < total;
         q += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t col = (uint32_t)(q % width), k0 = (uint32_t)(q / width) * 16;
        uint32_t b[8][4] = {};
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const uint64_t v = k0 + e < K ? ksk[(uint64_t)(k0 + e) * width + col] : 0;
#pragma unroll
            for (int c = 0; c < 8; ++c) b[c][e / 4] |= (uint32_t)((v >> (8 * c)) & 255u) << (8 * (e % 4));
        }
#pragma unroll
        for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(dst + ((uint64_t)col * 8 + c) * kpad + k0) =
                make_uint4(b[c][0], b[c][1], b[c][2], b[c][3]);
    }
}

// Output update from the splits' partial sums (the end of lwe_ks_kernel).
__global__ void __launch_bounds__(256) lwe_mma_finish_kernel(const LweKsParams prm, const uint64_t* __restrict__ part,
                                                             uint64_t row0, uint32_t rows, uint32_t splits) {
    const uint32_t width = prm.n_out + 1;
    const uint64_t total = (uint64_t)rows * width;
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < total;
         q += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(q / width), col = (uint32_t)(q - (uint64_t)r * width);
        uint64_t sum = part[q];
        for (uint32_t s = 1; s < splits; ++s) sum = gl_add(sum, part[s * total + q]);
        lwe_ks_store(prm, row0 + r, col, gl_sub(sum, prm.cterm[col]));
    }
}

}  // namespace tp
