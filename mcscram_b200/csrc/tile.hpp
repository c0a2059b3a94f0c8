// tile.hpp -- arguments of the tile kernel (k_tile in kernels.cuh).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace mcg {
namespace dev {

struct TileArgs {
    const uint4 *be;               // needed events, segment by segment: {pdag + 1, event + 1, thr lo,
                                   // thr hi | first word of the slot << 1}
    const uint4 *gates;            // gates, layer by layer: kind | inverted << 2 | k << 8 | counter
                                   // bits << 16 | tallies << 20, in_begin, input pairs | first word of the slot << 16,
                                   // tally index (or list offset)
    const uint32_t *in;            // inputs, an even number per gate: the slot's byte offset | complemented;
                                   // the last slot is the empty input (zeros)
    const uint32_t *layer;         // gate indices
    const uint2 *segment;          // {events' end, layers' end}
    const uint32_t *tally_list;
    const uint2 *be_tally;         // tallied events {slot, tally index}
    uint32_t n_slots, n_segments, n_be_tally, n_tally, tally_in_smem;
    uint32_t iteration_first, n_iterations;
    uint64_t word_begin, word_count;
    unsigned long long *ones;
};

constexpr uint32_t kTileLanes = 32;
constexpr uint32_t kTileOr = 0, kTileXor = 1, kTileAtleast = 2;  // gate kinds (AND forms through De Morgan)

// Batched instances in tiles (k_batch_tile): tables of all trees, concatenated.
struct BatchTileTree {
    uint32_t n_be, n_segments, n_be_tally;
    uint32_t gate_off, layer_off, in_off, be_tally_off, seg_off, event_off;
};

// Up to kTileInstances instances of one tree that follow each other.
struct BatchTileGroup {
    uint32_t tree, first, size;
    uint32_t pad;
    uint64_t rec_off;  // its event records, in events
};

constexpr uint32_t kTileInstances = 16;
constexpr uint32_t kTileRow = kTileInstances * kTileLanes * 8;  // bytes of a node's row: [instance][half][word] u32
constexpr uint32_t kTileRec = 5;                                // uint4 per event record: 16 thresholds, then
                                                                // {largest, all-ones mask, pdag + 1, event + 1}
constexpr int kBatchTileThreads = 512, kBatchTileBlocks = 2;    // per block, blocks per SM
constexpr uint32_t kBatchTileOut = 8 * 32 * 16;                 // bytes of staged outputs per warp

struct BatchTileArgs {
    const BatchTileTree *trees;
    const BatchTileGroup *groups;
    const uint4 *recs;
    const uint4 *gates;            // as TileArgs but for the last two fields, input pairs and the gate's slot; row 0
                                   // is the empty input
    const uint32_t *in, *layer;
    const uint2 *segment;          // {events' end, layers' end}
    const uint32_t *event_slot;
    const uint2 *be_tally;         // tallied events {slot, tallies}
    uint64_t tiles, words;         // per instance
    uint64_t items;
    uint32_t iteration;
    unsigned char *scratch;        // per block: a row per slot
    uint64_t scratch_stride;
    unsigned long long *queue;     // zero before the launch
    unsigned long long *ones;      // per instance
};

}  // namespace dev
}  // namespace mcg
