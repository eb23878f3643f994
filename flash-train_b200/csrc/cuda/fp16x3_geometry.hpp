// How the prepared form cuts a product into tiles and K slices. Pure arithmetic: the platform lays launches out by it, and
// large_group.hpp estimates times with it.
#ifndef FTCUDA_FP16X3_GEOMETRY_HPP_
#define FTCUDA_FP16X3_GEOMETRY_HPP_

#include <cstdint>

namespace ftcuda {
namespace fp16x3 {

constexpr std::uint32_t kBlockK = 64;   // K elements of one block: 128 bytes of FP16, one swizzle row
constexpr int kTileM            = 256;  // rows of a CTA pair's tile
constexpr int kMaxTileN         = 256;

inline std::uint64_t divideUp(std::uint64_t x, std::uint64_t y) { return (x + y - 1) / y; }

struct Geometry {
    std::uint32_t tile_n, splits, blocks_per_split;
    double cycles;
};

// SM cycles of one K block of a tile: a K step of 16 is three MMAs of tile_n / 2 cycles each, or the
// shared-memory traffic behind them (operand fetches and TMA writes at 128 bytes a cycle) where that is longer, which it is
// under 192 columns.
inline double blockCycles(std::uint32_t tile_n) {
    const double mma = 1.5 * tile_n, smem = 160.0 + 0.625 * tile_n;
    return 4.0 * (mma > smem ? mma : smem);
}

// Tile width and K slices of the least modelled cost, in SM cycles: a tile costs about 4000 beside its K blocks (pipeline fill,
// last drain, output); K slices cost a second kernel and their sums' way through memory.
inline Geometry chooseGeometry(std::uint64_t m, std::uint64_t n, std::uint64_t k_blocks, std::uint64_t pairs) {
    // Slice counts that K can be cut into, in multiples of four blocks.
    std::uint32_t counts[32];
    std::uint64_t lengths[32];
    int candidates = 0;
    for (std::uint32_t splits = 1; splits <= 32; ++splits) {
        const std::uint64_t per_split = splits == 1 ? k_blocks : divideUp(divideUp(k_blocks, splits), 4) * 4;
        if (splits > 1 && divideUp(k_blocks, per_split) != splits) { continue; }
        counts[candidates]    = splits;
        lengths[candidates++] = per_split;
    }
    const double outputs = static_cast<double>(m) * static_cast<double>(n);
    Geometry best{kMaxTileN, 1, static_cast<std::uint32_t>(k_blocks), 0.0};
    for (std::uint32_t width = kMaxTileN; width >= 64; width -= 16) {
        const std::uint64_t tiles  = divideUp(m, kTileM) * divideUp(n, width);
        const double block_cycles  = blockCycles(width);
        const double share         = static_cast<double>(tiles) / static_cast<double>(pairs);
        const double multiplying   = share * static_cast<double>(k_blocks) * block_cycles;
        for (int i = 0; i < candidates; ++i) {
            const std::uint32_t splits = counts[i];
            if (tiles * splits >= (1ULL << 31)) { break; }
            const double combining = splits > 1 ? 8000.0 + outputs * (8.0 * splits + 4.0) / 3500.0 : 0.0;
            // What it costs at least, with no wave part-filled, grows with the slices: no later count can be better either.
            // (The factor covers the rounding of this sum.)
            if (best.cycles != 0.0 && (multiplying + share * splits * 4000.0 + combining) * (1.0 - 1e-9) > best.cycles) { break; }
            const double cycles =
                static_cast<double>(divideUp(tiles * splits, pairs)) * (static_cast<double>(lengths[i]) * block_cycles + 4000.0) + combining;
            if (best.cycles == 0.0 || cycles < best.cycles) {
                best = Geometry{width, splits, static_cast<std::uint32_t>(lengths[i]), cycles};
            }
        }
    }
    return best;
}

}  // namespace fp16x3
}  // namespace ftcuda

#endif
