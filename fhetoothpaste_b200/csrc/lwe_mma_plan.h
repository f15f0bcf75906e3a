// How a tensor-core LWE key switch (lwe_mma.cuh) is cut into passes, tiles and splits: host arithmetic only.
#pragma once

#include <stdint.h>

#include <algorithm>

namespace tp {

constexpr int kMmaRows = 128, kMmaCols = 256, kMmaK = 128;      // block tile, bytes of K per step
constexpr int kMmaWords = kMmaCols / 8;                         // output words per tile
constexpr uint32_t kMmaMaxSteps = 258;                          // 255^2 * 128 * 258 < 2^31

// Ciphertexts of `width` words, digits of `planes` bytes: two byte planes at most, and the words' tiles
// are the grid's second dimension.
constexpr bool lwe_mma_fits(int planes, uint64_t width) {
    return planes <= 2 && (width + kMmaWords - 1) / kMmaWords <= 65535;
}

// One pass of the key switch over up to `rows` ciphertexts.
struct LweMmaPlan {
    uint32_t rows, rows_pad, splits;
    uint64_t plane_bytes, part_bytes;  // digit planes, then partial sums
    uint64_t bytes() const { return plane_bytes + part_bytes; }
};

// kpad: bytes of K (a multiple of kMmaK); width: output words of a ciphertext.
inline LweMmaPlan lwe_mma_plan(int planes, uint32_t kpad, uint32_t width, uint64_t batch, uint64_t sms) {
    LweMmaPlan p{};
    // at most 256 MB of digit planes at a time
    const uint64_t most = std::max<uint64_t>(1, (256ull << 20) / ((uint64_t)planes * kpad * kMmaRows)) * kMmaRows;
    p.rows = (uint32_t)std::min(batch, most);
    p.rows_pad = (p.rows + kMmaRows - 1) / kMmaRows * kMmaRows;
    const uint32_t steps = kpad / kMmaK;
    const uint64_t tiles = (uint64_t)(p.rows_pad / kMmaRows) * ((width + kMmaWords - 1) / kMmaWords);
    // splits of K: the fewest block-steps over the waves, a block costing about six steps
    // beside its share (fill, drain, epilogue); at least enough for exact 32-bit sums
    const uint32_t least = (steps + kMmaMaxSteps - 1) / kMmaMaxSteps;
    uint64_t best = ~0ull;
    for (uint32_t s = least; s <= steps && s <= std::max(64u, least); ++s) {
        const uint32_t share = (steps + s - 1) / s;
        if ((steps + share - 1) / share != s) continue;  // every split has steps
        const uint64_t cost = (tiles * s + sms - 1) / sms * (share + 6) + s / 4;
        if (cost < best) {
            best = cost;
            p.splits = s;
        }
    }
    p.plane_bytes = (uint64_t)planes * p.rows_pad * kpad;
    p.part_bytes = (uint64_t)p.splits * p.rows * width * 8;
    return p;
}

}  // namespace tp
