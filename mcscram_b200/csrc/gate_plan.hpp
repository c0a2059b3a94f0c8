// gate_plan.hpp -- a graph's gates as the staged pipeline's gate kernel
// evaluates them (host side; no CUDA calls).
#pragma once
#include <algorithm>
#include <cstdint>
#include <numeric>
#include <vector>

#include <vector_types.h>

#include "graph.hpp"
#include "mcg.h"

namespace mcg {

// Gate kinds.  AND, NAND, OR, NOR, one-of-n and n-of-n gates are ORs of
// complemented or plain inputs with a complemented or plain result (De
// Morgan), NOT and NULL ORs of their last input.  k-of-n gates with k or
// n - k + 1 at most 4 keep that many running "at least j" words (kGateChain);
// the others count in bit slices.
constexpr uint32_t kGateOr = 0, kGateXor = 1, kGateChain = 2, kGateCount = 3;
constexpr uint32_t kGateFlip = 0x80000000u;  // input record: node | kGateFlip if it is read complemented
constexpr uint32_t kGateParts = 64;

// About what a block of 32 warps takes per gate (ns) and per input (tenths of
// it), fitted to passes of one block per tile with 50 to 8,000 gates of 2 to 60
// inputs: latency, as a block's warps wait for the rows of one gate each.
constexpr uint32_t kGateNs = 20, kInputNs = 16, kCountGateNs = 47, kCountInputNs = 63;

struct GatePlan {
    // Gates layer by layer, in a layer part by part, two records each:
    // {kind | inverted << 2 | k << 8 | counter bits << 16, first further input, inputs, output node} and the
    // first four inputs.  Inputs are padded to a multiple of 4 with copies of the last one.
    std::vector<uint4> gates;
    std::vector<uint32_t> in;        // inputs from the fifth on, 4-aligned per gate
    std::vector<uint2> tally;        // per gate {its tally (of several: their offset in tally_list), count}
    std::vector<uint32_t> tally_list;
    // Parts: sets of gates that read no gate of another part, and behind the last
    // one all of them as one.  Part p's layers are layer[part[p]] ..
    // layer[part[p + 1] - 1], each a gate range [layer[l].x, layer[l].y).
    std::vector<uint32_t> part;
    std::vector<uint2> layer;
    uint32_t parts() const { return (uint32_t)part.size() - 2; }
    uint32_t largest = 0;            // gates of the largest part
    uint64_t block_ns = 0;           // about what a block of 32 warps takes for the costliest part's
    bool counts = false;             // some gate is a kGateCount
};

// `depth`: each gate's layer, from 1 on.
inline GatePlan plan_gates(const Graph &g, const std::vector<uint32_t> &depth) {
    GatePlan t;
    const uint32_t nb = g.n_be, ng = g.n_gates;
    std::vector<uint32_t> root(ng);
    std::iota(root.begin(), root.end(), 0u);
    auto find = [&](uint32_t i) {
        while (root[i] != i) i = root[i] = root[root[i]];
        return i;
    };
    for (uint32_t i = 0; i < ng; ++i)
        for (uint32_t j = 0; j < g.gate_in_count[i]; ++j) {
            const uint32_t c = g.inputs[g.gate_in_begin[i] + j];
            if (c >= nb) root[find(i)] = find(c - nb);
        }
    // components, the largest first, each to the part with the fewest gates
    std::vector<uint32_t> size(ng, 0), comps, part_of(ng, 0);
    for (uint32_t i = 0; i < ng; ++i) ++size[find(i)];
    for (uint32_t i = 0; i < ng; ++i)
        if (size[i]) comps.push_back(i);
    std::stable_sort(comps.begin(), comps.end(), [&](uint32_t x, uint32_t y) { return size[x] > size[y]; });
    // As many parts as the largest component leaves evenly loaded: every part is
    // a block per tile, and small components in parts of their own are blocks
    // with next to nothing to do (2,905 gates of which most are in one component,
    // 3,173 words: 0.19 ms, in 64 parts 0.32).
    const uint32_t even = comps.empty() ? 1u : (ng + size[comps[0]] - 1) / size[comps[0]];
    const uint32_t n_parts = std::min(kGateParts, even);
    std::vector<uint64_t> load(n_parts, 0);
    for (uint32_t c : comps) {
        const uint32_t p = (uint32_t)(std::min_element(load.begin(), load.end()) - load.begin());
        load[p] += size[c];
        part_of[c] = p;
    }
    t.largest = (uint32_t)*std::max_element(load.begin(), load.end());
    for (uint32_t i = 0; i < ng; ++i) part_of[i] = part_of[find(i)];
    // by layer, in a layer by part: two counting sorts
    auto sorted = [&](const std::vector<uint32_t> &from, const std::vector<uint32_t> &key) {
        std::vector<uint32_t> at(*std::max_element(key.begin(), key.end()) + 2, 0), to(ng);
        for (uint32_t k : key) ++at[k + 1];
        std::partial_sum(at.begin(), at.end(), at.begin());
        for (uint32_t i : from) to[at[key[i]]++] = i;
        return to;
    };
    std::vector<uint32_t> order(ng);
    std::iota(order.begin(), order.end(), 0u);
    if (ng) order = sorted(sorted(order, part_of), depth);
    // the gates' tallies: gate i's are tally[tally_at[i]] .. tally[tally_at[i + 1] - 1]
    std::vector<uint32_t> tally_at(ng + 1, 0), tally(g.tally_nodes.size());
    for (uint32_t v : g.tally_nodes)
        if (v >= nb) ++tally_at[v - nb + 1];
    std::partial_sum(tally_at.begin(), tally_at.end(), tally_at.begin());
    std::vector<uint32_t> next(tally_at);
    for (uint32_t k = 0; k < (uint32_t)g.tally_nodes.size(); ++k)
        if (g.tally_nodes[k] >= nb) tally[next[g.tally_nodes[k] - nb]++] = k;
    t.gates.reserve(2 * (size_t)ng);
    t.tally.reserve(ng);

    std::vector<uint32_t> rec;
    std::vector<uint64_t> cost(n_parts, 0);
    std::vector<std::vector<uint2>> layers(n_parts + 1);  // per part, then of all
    for (uint32_t at = 0; at < ng; ++at) {
        const uint32_t i = order[at];
        const uint8_t op = g.gate_op[i];
        const uint32_t n = g.gate_in_count[i], k = g.gate_k[i] & 0xFFu;
        const bool last_only = (op == MCG_NOT || op == MCG_NULL) && n > 0;
        bool and_type = op == MCG_AND || op == MCG_NAND;  // AND = ~OR(~x), NAND = OR(~x)
        bool inverted = op == MCG_AND || op == MCG_NOR || op == MCG_NOT;
        uint32_t kind = op == MCG_XOR ? kGateXor : kGateOr, kk = k, nbits = 0;
        if (op == MCG_ATLEAST) {
            kind = kGateCount;
            if (n <= 255 && k >= 1 && k <= n) {
                // at least k of x = not (at least n - k + 1 of ~x)
                const uint32_t co = n - k + 1;
                and_type = inverted = co < k;
                kk = std::min(k, co);
                if (kk == 1) kind = kGateOr;
                else if (kk <= 4) kind = kGateChain;
                else and_type = inverted = false, kk = k;
            }
            while (nbits < 8 && (n >> nbits) != 0) ++nbits;
        }
        t.counts |= kind == kGateCount;
        rec.clear();
        for (uint32_t j = last_only ? n - 1 : 0u; j < n; ++j) {
            const bool negated = j >= n - g.gate_neg_count[i];
            rec.push_back(g.inputs[g.gate_in_begin[i] + j] | (negated != and_type ? kGateFlip : 0u));
        }
        const uint32_t count = (uint32_t)rec.size();
        t.gates.push_back(make_uint4(kind | (inverted ? 4u : 0u) | (kk << 8) | (std::max(nbits, 1u) << 16),
                                     (uint32_t)t.in.size(), count, nb + i));
        while (rec.size() < 4 || rec.size() % 4) rec.push_back(count ? rec[count - 1] : 0u);
        t.gates.push_back(make_uint4(rec[0], rec[1], rec[2], rec[3]));
        t.in.insert(t.in.end(), rec.begin() + 4, rec.end());
        cost[part_of[i]] += kind == kGateCount ? kCountGateNs + (uint64_t)count * kCountInputNs / 10
                                               : kGateNs + (uint64_t)count * kInputNs / 10;
        const uint32_t *mine = tally.data() + tally_at[i], n_mine = tally_at[i + 1] - tally_at[i];
        t.tally.push_back(make_uint2(n_mine == 1 ? mine[0] : (uint32_t)t.tally_list.size(), n_mine));
        if (n_mine > 1) t.tally_list.insert(t.tally_list.end(), mine, mine + n_mine);
        const uint32_t last = at ? order[at - 1] : i;
        const bool same_layer = at && depth[last] == depth[i];
        auto put = [&](std::vector<uint2> &ranges, bool same) {
            if (same) ++ranges.back().y;
            else ranges.push_back(make_uint2(at, at + 1));
        };
        put(layers[part_of[i]], same_layer && part_of[last] == part_of[i]);
        put(layers[n_parts], same_layer);
    }
    for (const auto &ranges : layers) {
        t.part.push_back((uint32_t)t.layer.size());
        t.layer.insert(t.layer.end(), ranges.begin(), ranges.end());
    }
    t.block_ns = *std::max_element(cost.begin(), cost.end());
    t.part.push_back((uint32_t)t.layer.size());
    return t;
}

}  // namespace mcg
