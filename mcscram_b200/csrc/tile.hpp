// tile.hpp -- arguments of the tile kernel (k_tile in kernels.cuh).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace mcg {
namespace dev {

struct TileArgs {
    const uint4 *be;               // needed events {pdag + 1, event + 1, thr lo, thr hi}: node slots [0, n_be)
    const uint4 *gates;            // gate i (slot n_be + i), layer by layer: kind | inverted << 2 | k << 8 | counter
                                   // bits << 16 | tallies << 20, in_begin, input pairs, tally index (or list offset)
    const uint32_t *in;            // inputs, an even number per gate: the slot's byte offset | complemented;
                                   // the last slot is the empty input (zeros)
    const uint32_t *layer;         // n_layers + 1 gate indices
    const uint32_t *tally_list;
    const uint2 *be_tally;         // tallied events {slot, tally index}
    uint32_t n_be, n_slots, n_layers, n_be_tally, n_tally, tally_in_smem;
    uint32_t iteration_first, n_iterations;
    uint64_t word_begin, word_count;
    unsigned long long *ones;
};

constexpr uint32_t kTileLanes = 32;
constexpr uint32_t kTileOr = 0, kTileXor = 1, kTileAtleast = 2;  // gate kinds (AND forms through De Morgan)

}  // namespace dev
}  // namespace mcg
