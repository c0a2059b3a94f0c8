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

// What both plans need of a graph: NOT and NULL gates' first read input, the
// needed nodes, each node's tallies.
struct TileNeeds {
    const Graph &g;
    std::vector<char> needed;
    std::vector<std::vector<uint32_t>> tallies;

    explicit TileNeeds(const Graph &graph) : g(graph), needed(graph.n_nodes(), 0), tallies(graph.n_nodes()) {
        for (uint32_t v : g.tally_nodes) needed[v] = 1;
        for (uint32_t i = g.n_gates; i-- > 0;) {
            if (!needed[g.n_be + i]) continue;
            for (uint32_t j = first_input(i); j < g.gate_in_count[i]; ++j) needed[input(i, j)] = 1;
        }
        for (uint32_t k = 0; k < (uint32_t)g.tally_nodes.size(); ++k) tallies[g.tally_nodes[k]].push_back(k);
    }
    uint32_t input(uint32_t i, uint32_t j) const { return g.inputs[g.gate_in_begin[i] + j]; }
    uint32_t first_input(uint32_t i) const {
        const bool last_only = (g.gate_op[i] == MCG_NOT || g.gate_op[i] == MCG_NULL) && g.gate_in_count[i] > 0;
        return last_only ? g.gate_in_count[i] - 1 : 0u;
    }
    // Appends gate i to the plan's tables; slot: of each node.
    void emit(TilePlan &t, uint32_t i, const std::vector<uint32_t> &slot) const {
        const uint8_t op = g.gate_op[i];
        const uint32_t n = g.gate_in_count[i], from = first_input(i);
        const bool and_type = op == MCG_AND || op == MCG_NAND;  // AND = ~OR(~x), NAND = OR(~x)
        const bool inverted = op == MCG_AND || op == MCG_NOR || op == MCG_NOT;
        const uint32_t kind = op == MCG_ATLEAST ? dev::kTileAtleast : op == MCG_XOR ? dev::kTileXor : dev::kTileOr;
        uint32_t nbits = 0;
        while (nbits < 8 && (n >> nbits) != 0) ++nbits;
        const std::vector<uint32_t> &mine = tallies[g.n_be + i];
        if (mine.size() > 0xFFFu) t.fits = false;
        t.gates.push_back(make_uint4(kind | (inverted ? 4u : 0u) | ((g.gate_k[i] & 0xFFu) << 8) |
                                         (std::max(nbits, 1u) << 16) | ((uint32_t)mine.size() << 20),
                                     (uint32_t)t.in.size(), (n - from + 1) / 2,
                                     mine.size() == 1 ? mine[0] : (uint32_t)t.tally_list.size()));
        if (mine.size() > 1) t.tally_list.insert(t.tally_list.end(), mine.begin(), mine.end());
        for (uint32_t j = from; j < n; ++j) {
            const bool negated = j >= n - g.gate_neg_count[i];
            t.in.push_back(slot[input(i, j)] << 1 | (uint32_t)(negated != and_type));
        }
        if ((n - from) % 2) t.in.push_back(kEmptyInput);
    }
};

inline TilePlan plan_tile(const Graph &g) {
    TilePlan t;
    const uint32_t nb = g.n_be;
    const TileNeeds needs(g);
    std::vector<uint32_t> slot(g.n_nodes(), 0), depth(g.n_gates, 0);
    std::vector<std::vector<uint32_t>> layers;
    for (uint32_t i = 0; i < g.n_gates; ++i) {
        if (!needs.needed[nb + i]) continue;
        for (uint32_t j = needs.first_input(i); j < g.gate_in_count[i]; ++j) {
            const uint32_t c = needs.input(i, j);
            if (c >= nb) depth[i] = std::max(depth[i], depth[c - nb] + 1);
        }
        if (layers.size() <= depth[i]) layers.resize(depth[i] + 1);
        layers[depth[i]].push_back(i);
    }
    for (uint32_t e = 0; e < nb; ++e) {
        if (!needs.needed[e]) continue;
        slot[e] = (uint32_t)t.event.size();
        t.event.push_back(e);
        for (uint32_t k : needs.tallies[e]) t.be_tally.push_back(make_uint2(slot[e], k));
    }
    uint32_t next = (uint32_t)t.event.size();
    for (const auto &layer : layers) {
        for (uint32_t i : layer) slot[nb + i] = next++;
        for (uint32_t i : layer) needs.emit(t, i, slot);
        t.layer.push_back((uint32_t)t.gates.size());
    }
    return t;
}

// The plan of the kernels whose rows are used again (the batch tile kernel, the
// strip kernel, the tile kernel on large trees): the gates in depth-first postorder, cut into segments
// that each sample their own new events (`events` of them, if so many are
// left) and then evaluate their gates.  A node's row is free again after the
// layer that reads it last (by_layer; else after the segment, whose gates may
// then be taken in any order that respects their inputs) and is the next one
// to be written, so that rows mostly stay in the L2 from writer to reader and
// their memory is mostly never written back.
constexpr uint32_t kSegmentEvents = 96;
struct SegmentPlan {
    TilePlan tile;                    // tile.layer over all segments; slots from 0
    std::vector<uint2> segment;       // per segment: its events' and its layers' end
    std::vector<uint32_t> event_slot, gate_slot;
    std::vector<uint32_t> gate;       // gate ids, in tile.gates' order
    uint32_t slots = 0;
};

// `round`: segments are filled up to whole multiples of so many events with the
// next one's first.
inline SegmentPlan plan_segments(const Graph &g, uint32_t events, bool by_layer, uint32_t round = 1) {
    SegmentPlan p;
    TilePlan &t = p.tile;
    const uint32_t nb = g.n_be;
    const TileNeeds needs(g);
    // postorder over the needed gates, the child with the most gates below it
    // first (its temporary rows then overlap the fewest others)
    std::vector<uint64_t> weight(g.n_gates, 1);
    for (uint32_t i = 0; i < g.n_gates; ++i)
        for (uint32_t j = needs.first_input(i); j < g.gate_in_count[i]; ++j)
            if (needs.input(i, j) >= nb)
                weight[i] = std::min<uint64_t>(weight[i] + weight[needs.input(i, j) - nb], 1ull << 40);
    std::vector<uint32_t> order, children;
    std::vector<char> state(g.n_gates, 0);  // 1: expanded, 2: in order
    std::vector<uint32_t> stack;
    for (uint32_t v : g.tally_nodes)
        if (v >= nb) stack.push_back(v - nb);
    std::reverse(stack.begin(), stack.end());
    while (!stack.empty()) {
        const uint32_t i = stack.back();
        if (state[i] == 0) {
            state[i] = 1;
            children.clear();
            for (uint32_t j = needs.first_input(i); j < g.gate_in_count[i]; ++j) {
                const uint32_t c = needs.input(i, j);
                if (c >= nb && state[c - nb] == 0) children.push_back(c - nb);
            }
            std::stable_sort(children.begin(), children.end(),
                             [&](uint32_t x, uint32_t y) { return weight[x] < weight[y]; });
            stack.insert(stack.end(), children.begin(), children.end());
        } else {
            stack.pop_back();
            if (state[i] == 1) {
                state[i] = 2;
                order.push_back(i);
            }
        }
    }
    // segments: each gate's segment and layer in it, each event's segment
    struct Segment {
        std::vector<uint32_t> events;
        std::vector<std::vector<uint32_t>> layers;
    };
    std::vector<Segment> segs(1);
    std::vector<char> sampled(nb, 0);
    std::vector<uint32_t> seg_of(g.n_gates, 0), depth(g.n_gates, 0);
    for (uint32_t i : order) {
        if (segs.back().events.size() >= events) segs.emplace_back();
        Segment &s = segs.back();
        seg_of[i] = (uint32_t)segs.size();
        for (uint32_t j = needs.first_input(i); j < g.gate_in_count[i]; ++j) {
            const uint32_t c = needs.input(i, j);
            if (c < nb) {
                if (!sampled[c]) s.events.push_back(c);
                sampled[c] = 1;
            } else if (seg_of[c - nb] == seg_of[i]) {
                depth[i] = std::max(depth[i], depth[c - nb] + 1);
            }
        }
        if (s.layers.size() <= depth[i]) s.layers.resize(depth[i] + 1);
        s.layers[depth[i]].push_back(i);
    }
    for (uint32_t e = 0; e < nb; ++e)
        if (needs.needed[e] && !sampled[e]) segs.back().events.push_back(e);
    for (size_t k = 0; k + 1 < segs.size(); ++k) {
        std::vector<uint32_t> &to = segs[k].events, &from = segs[k + 1].events;
        const size_t n = std::min<size_t>((round - to.size() % round) % round, from.size());
        to.insert(to.end(), from.begin(), from.begin() + (std::ptrdiff_t)n);
        from.erase(from.begin(), from.begin() + (std::ptrdiff_t)n);
    }
    // reads left of each node; tallied events keep their rows (counted at the end)
    std::vector<uint32_t> reads(g.n_nodes(), 0);
    for (uint32_t i : order)
        for (uint32_t j = needs.first_input(i); j < g.gate_in_count[i]; ++j) ++reads[needs.input(i, j)];
    for (uint32_t e = 0; e < nb; ++e)
        if (!needs.tallies[e].empty()) ++reads[e];
    std::vector<uint32_t> slot(g.n_nodes(), 0), free_slots, dead;
    auto take = [&](uint32_t v) {
        if (free_slots.empty()) {
            slot[v] = p.slots++;
        } else {
            slot[v] = free_slots.back();
            free_slots.pop_back();
        }
    };
    for (Segment &s : segs) {
        for (uint32_t e : s.events) {
            take(e);
            t.event.push_back(e);
            p.event_slot.push_back(slot[e]);
        }
        for (const auto &layer : s.layers) {
            for (uint32_t i : layer) {
                take(nb + i);
                p.gate.push_back(i);
                p.gate_slot.push_back(slot[nb + i]);
                needs.emit(t, i, slot);
            }
            for (uint32_t i : layer) {
                for (uint32_t j = needs.first_input(i); j < g.gate_in_count[i]; ++j)
                    if (--reads[needs.input(i, j)] == 0) dead.push_back(slot[needs.input(i, j)]);
                if (reads[nb + i] == 0) dead.push_back(slot[nb + i]);
            }
            if (by_layer) {
                free_slots.insert(free_slots.end(), dead.begin(), dead.end());
                dead.clear();
            }
            t.layer.push_back((uint32_t)t.gates.size());
        }
        free_slots.insert(free_slots.end(), dead.begin(), dead.end());
        dead.clear();
        p.segment.push_back(make_uint2((uint32_t)t.event.size(), (uint32_t)t.layer.size() - 1));
    }
    for (uint32_t e = 0; e < nb; ++e)
        for (uint32_t k : needs.tallies[e]) t.be_tally.push_back(make_uint2(slot[e], k));
    return p;
}

}  // namespace mcg
