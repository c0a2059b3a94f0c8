// tile_cost.hpp -- the choice between the tile kernels and the interpreters, for a
// pass of the fused mode and for a run of batched instances (host side; no CUDA
// calls).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#include <vector_types.h>

#include "tile.hpp"

namespace mcg {

// SM clocks of a pass.  The tile kernel's layers each cost a block a barrier and
// a chain of table loads, however few gates they have, and the blocks of an SM
// come to them together; the interpreter has no barrier, but every warp walks
// every op.  So deep graphs of few events are the interpreter's where the words
// are many: 800 gates in a chain over 60 events on 262,144 words take 15.4 ms in
// tiles and 2.6 there; 2,048 words 0.37 and 0.90.  The coefficients are fitted to
// both kernels on graphs of 4 to 2,000 events, 2 to 800 layers and fan-ins of 2
// to 24, 2,048 to 2^20 words (within 12 % for eight of ten); over 1,833 passes of
// 507 graphs the choice was more than 10 % behind the better kernel in 9.
struct TileCost {
    uint64_t sms = 1, blocks = 1;      // blocks: per SM, in long passes
    uint64_t events = 0, inputs = 0;   // inputs: records of all gates
    uint64_t rounds = 0, pairs = 0;    // over the layers: gates per warp of the one with most, input pairs of the widest gate
    uint64_t ops = 0;                  // of the interpreter's program, about
    bool l1 = true;                    // the blocks leave the SM some L1 for the tables

    // layer: gate indices; gates: .z's low half the input pairs; block_bytes: shared memory of a block
    TileCost() = default;
    TileCost(const std::vector<uint32_t> &layer, const std::vector<uint4> &gates, size_t n_events, size_t n_inputs,
             size_t n_tally, uint32_t n_sms, uint32_t threads, size_t block_bytes)
        : sms(n_sms), blocks(1024 / threads), events(n_events), inputs(n_inputs),
          ops(n_inputs + 2 * gates.size() + n_tally), l1(blocks * block_bytes <= (200u << 10)) {
        const uint32_t warps = threads / 32;
        for (size_t l = 0; l + 1 < layer.size(); ++l) {
            uint32_t widest = 0;
            for (uint32_t i = layer[l]; i < layer[l + 1]; ++i) widest = std::max(widest, gates[i].z & 0xFFFFu);
            pairs += widest;
            rounds += (layer[l + 1] - layer[l] + warps - 1) / warps;
        }
    }
    uint64_t tile(uint64_t words) const {
        const uint64_t tiles = (words + 31) / 32;
        uint64_t b = blocks;
        while (b > 1 && tiles < sms * b) b /= 2;
        return (tiles + sms * b - 1) / (sms * b) * (b * (318 * events + 3 * inputs) + 1500 + 580 * rounds + (l1 ? 55 : 111) * pairs);
    }
    uint64_t interpreter(uint64_t words) const {
        const uint64_t warps = (words + 256 * sms - 1) / (256 * sms) * 8;  // blocks of eight warps
        return std::max(warps * (390 * events + 20 * ops), 3900 * events + 500 * ops - 120 * inputs);
    }
    bool interpreter_is_faster(uint64_t words) const { return interpreter(words) < tile(words); }
    bool interpreter_may_be_faster() const { return interpreter_is_faster(1ull << 32); }
};

// The same for batched instances, per tree.  The batch tile kernel shares an
// event's generator calls between up to 16 instances and the interpreter between
// four, but each of its layers is a barrier and a walk through rows in the L2, so
// that few instances of deep trees on many words are the interpreter's: two
// instances of a chain of 522 gates over 360 events on 204,067 words take 11.7 ms
// in tiles and 6.5 there, one of 200 events on 4,096 words 0.14 and 1.6.
// Coefficients fitted to both on 60 graphs of 10 to 3,000 events, 1 to 32
// instances and 2,048 to 131,072 words: of 1,428 runs 36 are more than 4 % behind
// the better kernel, 11 more than 15 %.
struct BatchTreeCost {
    uint64_t events = 0, segments = 0, inputs = 0, ops = 0;
    uint64_t rounds[3] = {0, 0, 0};        // over the layers: gates per warp, with 1, 2 and 4 quads of instances a gate
    uint64_t pairs = 0;                    // over the layers: input pairs of the widest gate
    uint64_t counts = 0, widest_count = 0; // of k-of-n gates: input pairs times counter bits, of all and of the layers' widest

    BatchTreeCost() = default;
    // layer: gate indices; gates: their records (.x: kind and counter bits, .z: input pairs)
    BatchTreeCost(const std::vector<uint32_t> &layer, const std::vector<uint4> &gates, size_t n_events, size_t n_segments,
                  size_t n_inputs, size_t n_ops)
        : events(n_events), segments(n_segments), inputs(n_inputs), ops(n_ops) {
        constexpr uint32_t warps = dev::kBatchTileThreads / 32;
        for (size_t l = 0; l + 1 < layer.size(); ++l) {
            uint64_t widest = 0, widest_k = 0;
            for (uint32_t i = layer[l]; i < layer[l + 1]; ++i) {
                const uint64_t n = gates[i].z;
                if ((gates[i].x & 3u) == dev::kTileAtleast) {
                    widest_k = std::max(widest_k, n * ((gates[i].x >> 16) & 0xFu));
                    counts += n * ((gates[i].x >> 16) & 0xFu);
                } else {
                    widest = std::max(widest, n);
                }
            }
            pairs += widest;
            widest_count += widest_k;
            for (uint32_t q = 0; q < 3; ++q) rounds[q] += (layer[l + 1] - layer[l] + (warps >> q) - 1) / (warps >> q);
        }
    }
    // Clocks of a block for 32 words of `size` instances, two blocks on its SM.
    uint64_t tile(uint32_t size) const {
        const uint64_t quads = (size + 3) / 4;
        return (size > 8 ? 1315 : size > 4 ? 1037 : 835) * events + 1450 * rounds[quads > 2 ? 2 : quads - 1] + 110 * pairs +
               30 * inputs * quads + 4590 * segments + 55 * widest_count + 157 * counts * quads;
    }
    // Clocks of an SM for a warp's 32 words of `share` instances (4 or 1), and of such a warp on its own.
    uint64_t interpreter(uint32_t share) const {
        return share > 1 ? 455 * events + 42 * ops + 65 * counts : 303 * events + 19 * ops + 14 * counts;
    }
    uint64_t interpreter_alone(uint32_t share) const {
        return share > 1 ? 14200 * events + 1325 * ops : 7900 * events + 730 * ops;
    }
};

}  // namespace mcg
