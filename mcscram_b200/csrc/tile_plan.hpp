// tile_plan.hpp -- a graph as the tile kernels evaluate it (host side).
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

#include "graph.hpp"
#include "mcg.h"
#include "tile.hpp"

namespace mcg {

// The nodes some tally depends on, as slots of the tile kernels: events in
// their order, then gates layer by layer.  NOT and NULL gates read their last
// input only.  Inputs are slot << 1 | complemented, kEmptyInput pads every
// gate to an even number of them.
constexpr uint32_t kEmptyInput = 0xFFFFFFFFu;
struct TilePlan {
    std::vector<uint32_t> event;                 // slot -> event
    std::vector<uint4> gates;
    std::vector<uint32_t> in, layer{0}, tally_list;
    std::vector<uint2> be_tally;
    uint32_t slots() const { return (uint32_t)(event.size() + gates.size()); }
    bool fits = true;  // the records' fields
    // An input as the kernels read it: the byte offset of its slot's row
    // (slots start at `first`, the empty input is row `empty`) | complemented.
    static uint32_t byte_record(uint32_t rec, uint32_t row_bytes, uint32_t first, uint32_t empty) {
        return rec == kEmptyInput ? empty * row_bytes : ((rec >> 1) + first) * row_bytes | (rec & 1u);
    }
};

inline TilePlan plan_tile(const Graph &g) {
    TilePlan t;
    const uint32_t nb = g.n_be;
    auto first_input = [&](uint32_t i) {
        const bool last_only = (g.gate_op[i] == MCG_NOT || g.gate_op[i] == MCG_NULL) && g.gate_in_count[i] > 0;
        return last_only ? g.gate_in_count[i] - 1 : 0u;
    };
    std::vector<uint32_t> slot(g.n_nodes(), 0), depth(g.n_gates, 0);
    std::vector<char> needed(g.n_nodes(), 0);
    for (uint32_t v : g.tally_nodes) needed[v] = 1;
    for (uint32_t i = g.n_gates; i-- > 0;) {
        if (!needed[nb + i]) continue;
        for (uint32_t j = first_input(i); j < g.gate_in_count[i]; ++j) needed[g.inputs[g.gate_in_begin[i] + j]] = 1;
    }
    std::vector<std::vector<uint32_t>> layers, tallies(g.n_nodes());
    for (uint32_t i = 0; i < g.n_gates; ++i) {
        if (!needed[nb + i]) continue;
        for (uint32_t j = first_input(i); j < g.gate_in_count[i]; ++j) {
            const uint32_t c = g.inputs[g.gate_in_begin[i] + j];
            if (c >= nb) depth[i] = std::max(depth[i], depth[c - nb] + 1);
        }
        if (layers.size() <= depth[i]) layers.resize(depth[i] + 1);
        layers[depth[i]].push_back(i);
    }
    for (uint32_t k = 0; k < (uint32_t)g.tally_nodes.size(); ++k) tallies[g.tally_nodes[k]].push_back(k);
    for (uint32_t e = 0; e < nb; ++e) {
        if (!needed[e]) continue;
        slot[e] = (uint32_t)t.event.size();
        t.event.push_back(e);
        for (uint32_t k : tallies[e]) t.be_tally.push_back(make_uint2(slot[e], k));
    }
    uint32_t next = (uint32_t)t.event.size();
    for (const auto &layer : layers) {
        for (uint32_t i : layer) slot[nb + i] = next++;
        for (uint32_t i : layer) {
            const uint8_t op = g.gate_op[i];
            const uint32_t n = g.gate_in_count[i], from = first_input(i);
            const bool and_type = op == MCG_AND || op == MCG_NAND;  // AND = ~OR(~x), NAND = OR(~x)
            const bool inverted = op == MCG_AND || op == MCG_NOR || op == MCG_NOT;
            const uint32_t kind = op == MCG_ATLEAST ? dev::kTileAtleast
                                  : op == MCG_XOR   ? dev::kTileXor
                                                    : dev::kTileOr;
            uint32_t nbits = 0;
            while (nbits < 8 && (n >> nbits) != 0) ++nbits;
            const std::vector<uint32_t> &mine = tallies[nb + i];
            if (mine.size() > 0xFFFu) t.fits = false;
            t.gates.push_back(make_uint4(kind | (inverted ? 4u : 0u) | ((g.gate_k[i] & 0xFFu) << 8) |
                                             (std::max(nbits, 1u) << 16) | ((uint32_t)mine.size() << 20),
                                         (uint32_t)t.in.size(), (n - from + 1) / 2,
                                         mine.size() == 1 ? mine[0] : (uint32_t)t.tally_list.size()));
            if (mine.size() > 1) t.tally_list.insert(t.tally_list.end(), mine.begin(), mine.end());
            for (uint32_t j = from; j < n; ++j) {
                const bool negated = j >= n - g.gate_neg_count[i];
                t.in.push_back(slot[g.inputs[g.gate_in_begin[i] + j]] << 1 | (uint32_t)(negated != and_type));
            }
            if ((n - from) % 2) t.in.push_back(kEmptyInput);
        }
        t.layer.push_back((uint32_t)t.gates.size());
    }
    return t;
}

}  // namespace mcg
