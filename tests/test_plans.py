"""The plans that the strip, staged, tile and batch kernels follow, walked on the
CPU (compiled here against the plans' own headers): every node's value is the
definition's, whatever rows are used again, in any order the kernels may take
the gates of a layer or segment."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <cuda_runtime.h>
#include "gate_plan.hpp"
#include "tile_plan.hpp"

using namespace mcg;
static std::mt19937_64 rng;
static uint32_t below(uint32_t n) { return (uint32_t)(rng() % n); }

[[noreturn]] static void wrong(const char *what, uint32_t at) {
    std::printf("wrong: %s %u\n", what, at);
    std::exit(1);
}

// n_gates gates of every connective with negated tails, empty and wide ones; `reach`: a gate reads the `reach` nodes
// before it and events up to its share of them (0: any node before it); `roots`: gates that nothing has read yet are
// read first, so that the last gate reaches nearly all of them.
static Graph random_graph(uint32_t n_be, uint32_t n_gates, uint32_t reach, bool roots, int tallies) {
    Graph g;
    g.n_be = n_be;
    g.n_gates = n_gates;
    for (uint32_t e = 0; e < n_be; ++e) {
        g.be_pdag_idx.push_back((int32_t)e + 2);
        g.be_event_idx.push_back(e);
        g.be_threshold.push_back(1u << 31);
    }
    std::vector<uint32_t> unread;
    for (uint32_t j = 0; j < n_gates; ++j) {
        const uint8_t op = (uint8_t)below(8);
        static const uint32_t sizes[] = {1, 2, 2, 3, 3, 4, 5, 7, 9, 12};
        uint32_t n = sizes[below(10)];
        if (!roots && below(20) == 0) n = 0;
        if (below(60) == 0) n = 20 + below(300);
        if (j + 1 == n_gates && roots) n = std::max<uint32_t>(n, (uint32_t)unread.size());
        g.gate_op.push_back(op);
        g.gate_k.push_back(below(n + 3));
        g.gate_in_begin.push_back((uint32_t)g.inputs.size());
        g.gate_in_count.push_back(n);
        g.gate_neg_count.push_back(below(n + 1));
        for (uint32_t i = 0; i < n; ++i) {
            uint32_t v;
            if (roots && !unread.empty() && (i == n - 1 || below(2))) {
                v = unread.back();
                unread.pop_back();
            } else if (j && below(2)) {
                const uint32_t span = reach ? std::min(reach, j) : j;
                v = n_be + j - 1 - below(span);
            } else {
                const uint64_t most = reach ? std::max<uint64_t>(1, (uint64_t)(j + 1) * n_be / n_gates) : n_be;
                v = below((uint32_t)std::min<uint64_t>(most, n_be));
            }
            g.inputs.push_back(v);
        }
        if (roots) unread.push_back(n_be + j);
    }
    const uint32_t nn = n_be + n_gates;
    if (tallies == 0) g.tally_nodes = {nn - 1};
    else if (tallies == 1) for (uint32_t v = 0; v < nn; ++v) g.tally_nodes.push_back(v);
    else for (uint32_t i = 0; i < 25; ++i) g.tally_nodes.push_back(below(nn));  // some twice
    const std::string err = g.validate();
    if (!err.empty()) {
        std::printf("%s\n", err.c_str());
        std::exit(2);
    }
    return g;
}

static uint64_t count_at_least(const std::vector<uint64_t> &x, uint32_t k) {  // as the reference: counts modulo 256
    uint64_t r = 0;
    for (int b = 0; b < 64; ++b) {
        uint8_t c = 0;
        for (uint64_t v : x) c = (uint8_t)(c + ((v >> b) & 1u));
        if (c >= (uint8_t)k) r |= 1ull << b;
    }
    return r;
}

// The definition: every node's word.
static std::vector<uint64_t> values(const Graph &g) {
    std::vector<uint64_t> val(g.n_nodes());
    for (uint32_t e = 0; e < g.n_be; ++e) val[e] = rng() & rng();
    for (uint32_t j = 0; j < g.n_gates; ++j) {
        std::vector<uint64_t> x;
        for (uint32_t i = 0; i < g.gate_in_count[j]; ++i) {
            const uint64_t v = val[g.inputs[g.gate_in_begin[j] + i]];
            x.push_back(i >= g.gate_in_count[j] - g.gate_neg_count[j] ? ~v : v);
        }
        const uint8_t op = g.gate_op[j];
        uint64_t r = op == MCG_AND || op == MCG_NAND ? ~0ull : 0ull;
        for (uint64_t v : x)
            r = op == MCG_AND || op == MCG_NAND ? r & v : op == MCG_OR || op == MCG_NOR ? r | v : op == MCG_XOR ? r ^ v : v;
        if (op == MCG_ATLEAST) r = count_at_least(x, g.gate_k[j] & 0xFFu);
        val[g.n_be + j] = op == MCG_NAND || op == MCG_NOR || op == MCG_NOT ? ~r : r;
    }
    return val;
}

static std::vector<uint32_t> shuffled(uint32_t from, uint32_t to) {
    std::vector<uint32_t> o;
    for (uint32_t i = from; i < to; ++i) o.push_back(i);
    std::shuffle(o.begin(), o.end(), rng);
    return o;
}

// A gate of a tile plan from the rows.
static uint64_t tile_gate(const TilePlan &t, uint32_t i, const std::vector<uint64_t> &rows) {
    const uint4 m = t.gates[i];
    const uint32_t kind = m.x & 3u, kk = (m.x >> 8) & 0xFFu, nbits = (m.x >> 16) & 0xFu;
    std::vector<uint64_t> x;
    for (uint32_t p = 0; p < 2 * m.z; ++p) {
        const uint32_t rec = t.in[m.y + p];
        if (rec == kEmptyInput) x.push_back(0);
        else x.push_back((rec & 1u) ? ~rows[rec >> 1] : rows[rec >> 1]);
    }
    uint64_t r = 0;
    if (kind == dev::kTileAtleast) {
        uint32_t real = 0;
        for (uint32_t p = 0; p < 2 * m.z; ++p) real += t.in[m.y + p] != kEmptyInput;
        if (nbits < 8 && (real >> nbits)) wrong("counter bits of gate", i);
        r = count_at_least(x, kk);
    } else {
        for (uint64_t v : x) r = kind == dev::kTileXor ? r ^ v : r | v;
    }
    return (m.x & 4u) ? ~r : r;
}

struct Tallies {
    const Graph &g;
    const std::vector<uint64_t> &val;
    std::vector<char> seen;
    Tallies(const Graph &graph, const std::vector<uint64_t> &v) : g(graph), val(v), seen(graph.tally_nodes.size(), 0) {}
    void give(uint32_t idx, uint64_t word) {
        if (idx >= seen.size() || seen[idx]) wrong("tally twice or out of range", idx);
        seen[idx] = 1;
        if (word != val[g.tally_nodes[idx]]) wrong("value of tally", idx);
    }
    void all() {
        for (uint32_t i = 0; i < seen.size(); ++i)
            if (!seen[i]) wrong("missing tally", i);
    }
};

static void give_gate(Tallies &out, const TilePlan &t, uint32_t i, uint64_t r) {
    const uint32_t n = t.gates[i].x >> 20;
    if (n == 1) out.give(t.gates[i].w, r);
    else
        for (uint32_t k = 0; k < n; ++k) out.give(t.tally_list[t.gates[i].w + k], r);
}

static void walk_tile(const Graph &g, const std::vector<uint64_t> &val) {
    const TilePlan t = plan_tile(g);
    std::vector<uint64_t> rows(t.slots(), 0xDEADull);
    Tallies out(g, val);
    for (uint32_t i = 0; i < t.event.size(); ++i) rows[i] = val[t.event[i]];
    for (size_t l = 0; l + 1 < t.layer.size(); ++l)
        for (uint32_t i : shuffled(t.layer[l], t.layer[l + 1])) {
            const uint64_t r = tile_gate(t, i, rows);
            rows[t.event.size() + i] = r;
            give_gate(out, t, i, r);
        }
    for (const uint2 &x : t.be_tally) out.give(x.y, rows[x.x]);
    out.all();
}

// Returns the plan's segments.
static size_t walk_segments(const Graph &g, const std::vector<uint64_t> &val, uint32_t events, bool by_layer,
                            uint32_t round) {
    const SegmentPlan p = plan_segments(g, events, by_layer, round);
    const TilePlan &t = p.tile;
    std::vector<uint64_t> rows(p.slots, 0xDEADull);
    Tallies out(g, val);
    uint32_t e = 0, l = 0;
    for (const uint2 &seg : p.segment) {
        std::vector<char> written(p.slots, 0);
        for (uint32_t i : shuffled(e, seg.x)) {
            if (written[p.event_slot[i]]) wrong("row of two events", i);
            written[p.event_slot[i]] = 1;
            rows[p.event_slot[i]] = val[t.event[i]];
        }
        e = seg.x;
        if (by_layer) {
            for (; l < seg.y; ++l) {  // the gates of a layer at once, in any order
                for (uint32_t i : shuffled(t.layer[l], t.layer[l + 1])) {
                    const uint64_t r = tile_gate(t, i, rows);
                    rows[p.gate_slot[i]] = r;
                    give_gate(out, t, i, r);
                    if (r != val[g.n_be + p.gate[i]]) wrong("gate", p.gate[i]);
                }
            }
        } else {  // the gates of a segment in any order that has their inputs
            const uint32_t q0 = t.layer[l], q1 = t.layer[seg.y];
            l = seg.y;
            std::vector<int> pos(g.n_gates, -1), done(q1 - q0, 0);
            for (uint32_t q = q0; q < q1; ++q) pos[p.gate[q]] = (int)(q - q0);
            for (uint32_t left = q1 - q0; left;)
                for (uint32_t q : shuffled(q0, q1)) {
                    if (done[q - q0] || below(2)) continue;
                    const uint32_t i = p.gate[q];
                    const bool last_only = (g.gate_op[i] == MCG_NOT || g.gate_op[i] == MCG_NULL) && g.gate_in_count[i];
                    bool ready = true;
                    for (uint32_t j = last_only ? g.gate_in_count[i] - 1 : 0; j < g.gate_in_count[i]; ++j) {
                        const uint32_t c = g.inputs[g.gate_in_begin[i] + j];
                        if (c >= g.n_be && pos[c - g.n_be] >= 0 && !done[pos[c - g.n_be]]) ready = false;
                    }
                    if (!ready) continue;
                    const uint64_t r = tile_gate(t, q, rows);
                    rows[p.gate_slot[q]] = r;
                    give_gate(out, t, q, r);
                    done[q - q0] = 1;
                    --left;
                }
        }
    }
    for (const uint2 &x : t.be_tally) out.give(x.y, rows[x.x]);
    out.all();
    return p.segment.size();
}

static uint64_t staged_gate(const GatePlan &t, uint32_t i, const std::vector<uint64_t> &rows) {
    const uint4 m = t.gates[2 * i], q = t.gates[2 * i + 1];
    const uint32_t kind = m.x & 3u, kk = (m.x >> 8) & 0xFFu, nbits = (m.x >> 16) & 0xFu;
    std::vector<uint64_t> x;
    for (uint32_t j = 0; j < m.z; ++j) {
        const uint32_t rec = j == 0 ? q.x : j == 1 ? q.y : j == 2 ? q.z : j == 3 ? q.w : t.in[m.y + j - 4];
        x.push_back((rec & kGateFlip) ? ~rows[rec & ~kGateFlip] : rows[rec & ~kGateFlip]);
    }
    uint64_t r = 0;
    if (kind == kGateChain) {
        if (kk < 2 || kk > 4) wrong("chain", i);
        r = count_at_least(x, kk);
    } else if (kind == kGateCount) {
        if (!t.counts || (nbits < 8 && (m.z >> nbits))) wrong("counter", i);
        r = count_at_least(x, kk);
    } else {
        for (uint64_t v : x) r = kind == kGateXor ? r ^ v : r | v;
    }
    return (m.x & 4u) ? ~r : r;
}

static void walk_parts(const Graph &g, const std::vector<uint64_t> &val) {
    std::vector<uint32_t> depth(g.n_gates, 1);
    for (uint32_t j = 0; j < g.n_gates; ++j)
        for (uint32_t i = 0; i < g.gate_in_count[j]; ++i) {
            const uint32_t c = g.inputs[g.gate_in_begin[j] + i];
            if (c >= g.n_be) depth[j] = std::max(depth[j], depth[c - g.n_be] + 1);
        }
    const GatePlan t = plan_gates(g, depth);
    for (int merged = 0; merged < 2; ++merged) {
        std::vector<uint64_t> rows(g.n_nodes(), 0xDEADull);
        std::copy(val.begin(), val.begin() + g.n_be, rows.begin());
        Tallies out(g, val);
        for (uint32_t k = 0; k < g.tally_nodes.size(); ++k)
            if (g.tally_nodes[k] < g.n_be) out.give(k, val[g.tally_nodes[k]]);  // a kernel of their own
        for (uint32_t p : merged ? std::vector<uint32_t>{t.parts()} : shuffled(0, t.parts()))
            for (uint32_t l = t.part[p]; l < t.part[p + 1]; ++l)
                for (uint32_t i : shuffled(t.layer[l].x, t.layer[l].y)) {
                    const uint64_t r = staged_gate(t, i, rows);
                    rows[t.gates[2 * i].w] = r;
                    const uint2 x = t.tally[i];
                    if (x.y == 1) out.give(x.x, r);
                    else
                        for (uint32_t k = 0; k < x.y; ++k) out.give(t.tally_list[x.x + k], r);
                }
        if (rows != val) wrong("staged rows, merged", (uint32_t)merged);
        out.all();
    }
}

// Parts of a plan over separate trees of so many gates (each a chain).
static void parts_of(int n, char **sizes) {
    Graph g;
    g.n_be = 1;
    g.be_pdag_idx = {2};
    g.be_event_idx = {0};
    g.be_threshold = {1};
    std::vector<uint32_t> depth;
    for (int t = 0; t < n; ++t)
        for (int i = 0; i < std::atoi(sizes[t]); ++i) {
            g.gate_op.push_back(MCG_NULL);
            g.gate_k.push_back(0);
            g.gate_in_begin.push_back((uint32_t)g.inputs.size());
            g.gate_in_count.push_back(1);
            g.gate_neg_count.push_back(0);
            g.inputs.push_back(i ? g.n_gates : 0);
            ++g.n_gates;
            depth.push_back((uint32_t)i + 1);
        }
    const GatePlan t = plan_gates(g, depth);
    std::printf("ok %u %u\n", t.parts(), t.largest);
}

int main(int argc, char **argv) {
    if (!std::strcmp(argv[1], "parts")) {
        parts_of(argc - 2, argv + 2);
        return 0;
    }
    const uint32_t n_be = (uint32_t)std::atoi(argv[1]), n_gates = (uint32_t)std::atoi(argv[2]);
    const uint32_t reach = (uint32_t)std::atoi(argv[3]);
    size_t most = 0;
    (void)argc;
    for (int seed = 0; seed < 12; ++seed) {
        rng.seed((uint64_t)seed * 7919 + n_be);
        const Graph g = random_graph(n_be, n_gates, reach, seed % 2 == 0, seed % 3);
        const std::vector<uint64_t> val = values(g);
        walk_tile(g, val);
        walk_parts(g, val);
        for (uint32_t events : {8u, 96u, 256u, 384u})
            for (int form = 0; form < 3; ++form)
                most = std::max(most, walk_segments(g, val, events, form != 0, form == 2 ? 32 : 1));
    }
    std::printf("ok %zu\n", most);
}
"""


@pytest.fixture(scope="module")
def walker(tmp_path_factory):
    d = tmp_path_factory.mktemp("plans")
    (d / "walk.cc").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'mcscram_b200/csrc'}", "-I/usr/local/cuda/include", str(d / "walk.cc"),
                    str(ROOT / "mcscram_b200/csrc/graph.cpp"), "-o", str(d / "walk")], check=True)
    return d / "walk"


@pytest.mark.parametrize("n_be,n_gates,reach,segments", [(1, 1, 0, 1), (3, 40, 0, 1), (40, 60, 0, 2), (95, 200, 30, 5),
                                                         (385, 300, 40, 10), (1600, 1000, 40, 10),
                                                         (1600, 1000, 0, 10), (5000, 3000, 100, 10)])
def test_every_plan_gives_every_value(walker, n_be, n_gates, reach, segments):
    r = subprocess.run([str(walker), str(n_be), str(n_gates), str(reach)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
    assert int(r.stdout.split()[1]) >= segments  # the most that a plan had, at 8 events each


@pytest.mark.parametrize("sizes,parts,largest", [([7], 1, 7), ([5] * 16, 16, 5), ([5] * 200, 64, 20), ([1000] + [1] * 900, 2, 1000),
                                                 ([60, 60, 1, 2, 3], 3, 60), ([40, 30, 20, 10], 3, 40)])
def test_parts_are_evenly_loaded(walker, sizes, parts, largest):
    """A part is a block per tile: trees of a few gates beside large ones share one."""
    r = subprocess.run([str(walker), "parts", *map(str, sizes)], capture_output=True, text=True, check=True)
    assert r.stdout.split() == ["ok", str(parts), str(largest)]
