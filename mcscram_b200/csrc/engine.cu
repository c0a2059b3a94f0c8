// engine.cu -- the mcg_* engine entry points of include/mcg.h.
//
// One engine = one flattened PDAG on one device and stream.  It owns the
// device copies of the compiled fused program, the layered-mode tables, the
// tally counters and the fused kernel's scratch.  Replaces the device-memory
// ownership and pass submission of the reference's layer_manager
// (src/mc/queue/layer_manager.tpp:203-301) and its queueables
// (src/mc/queue/queueable.h:206-273, 725-731).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "engine_internal.hpp"
#include "error.hpp"
#include "graph.hpp"
#include "kernels.cuh"
#include "mcg.h"
#include "mcg_tune.h"
#include "program.hpp"
#include "smem_limit.hpp"
#include "staged_run.hpp"
#include "tile_plan.hpp"

namespace {

// Bit packing of the sampler: the carry chain measured faster than compares on B200 (register-only sampler).
constexpr int kPackForm = 1;
using mcg::internal::kDefaultChunkWords;
using mcg::internal::kFusedThreads;

#define MCG_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t err_ = (call);                                                              \
        if (err_ != cudaSuccess) {                                                              \
            cudaGetLastError(); /* reported here, and not by the next launch's check */         \
            return mcg::fail(err_ == cudaErrorMemoryAllocation ? MCG_ERR_OOM : MCG_ERR_CUDA,    \
                             std::string(#call) + ": " + cudaGetErrorString(err_));             \
        }                                                                                       \
    } while (0)

template <typename T>
cudaError_t upload(T **dptr, const std::vector<T> &v) {
    *dptr = nullptr;
    if (v.empty()) return cudaSuccess;
    cudaError_t e = cudaMalloc((void **)dptr, v.size() * sizeof(T));
    if (e != cudaSuccess) return e;
    return cudaMemcpy(*dptr, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
}

// The engines' large work buffers (strip and fused scratch, staged chunk
// buffers: gigabytes for a large tree) are kept per device when an engine is
// destroyed (it has synchronised its streams by then), and the next engine
// takes the smallest kept buffer that fits instead of allocating.  What does
// not fit comes from cudaMalloc; at most kKeptBuffers buffers and
// kKeptBytes bytes are kept per device, and a failed allocation first
// frees the kept ones.  mcg_trim_memory frees them all.
constexpr size_t kKeptBuffers = 2;
constexpr size_t kKeptBytes = 33ull << 30;  // two chunk buffers of 16 GiB, with 1 GiB of hit weights behind one

struct KeptBuffer {
    void *ptr;
    size_t bytes;
};
std::mutex g_kept_mutex;
std::vector<std::vector<KeptBuffer>> g_kept;  // per device

std::vector<KeptBuffer> &kept_on(int device) {
    if (g_kept.size() <= (size_t)device) g_kept.resize((size_t)device + 1);
    return g_kept[device];
}

void free_kept(int device) {
    std::vector<KeptBuffer> drop;
    {
        std::lock_guard<std::mutex> lock(g_kept_mutex);
        drop.swap(kept_on(device));
    }
    for (const KeptBuffer &b : drop) cudaFree(b.ptr);
}

cudaError_t work_alloc(mcg_engine *e, void **ptr, size_t bytes) {
    *ptr = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_kept_mutex);
        std::vector<KeptBuffer> &kept = kept_on(e->device);
        size_t best = kept.size();
        for (size_t i = 0; i < kept.size(); ++i)
            if (kept[i].bytes >= bytes && (best == kept.size() || kept[i].bytes < kept[best].bytes)) best = i;
        if (best < kept.size()) {
            *ptr = kept[best].ptr;
            e->work_bytes[*ptr] = kept[best].bytes;
            kept.erase(kept.begin() + (std::ptrdiff_t)best);
            return cudaSuccess;
        }
    }
    cudaError_t err = cudaMalloc(ptr, bytes);
    if (err == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        free_kept(e->device);
        err = cudaMalloc(ptr, bytes);
    }
    if (err == cudaSuccess) e->work_bytes[*ptr] = bytes;
    return err;
}

void work_free(mcg_engine *e, void *ptr) {
    if (!ptr) return;
    const size_t bytes = e->work_bytes[ptr];
    std::vector<KeptBuffer> drop;
    {
        std::lock_guard<std::mutex> lock(g_kept_mutex);
        std::vector<KeptBuffer> &kept = kept_on(e->device);
        kept.push_back({ptr, bytes});
        size_t total = 0;
        for (const KeptBuffer &b : kept) total += b.bytes;
        while (!kept.empty() && (kept.size() > kKeptBuffers || total > kKeptBytes)) {
            auto smallest = std::min_element(kept.begin(), kept.end(),
                                             [](const KeptBuffer &a, const KeptBuffer &b) { return a.bytes < b.bytes; });
            total -= smallest->bytes;
            drop.push_back(*smallest);
            kept.erase(smallest);
        }
    }
    for (const KeptBuffer &b : drop) cudaFree(b.ptr);
}

}  // namespace

extern "C" mcg_status mcg_trim_memory(int device) {
    mcg::clear_error();
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || device < 0 || device >= n_dev) {
        cudaGetLastError();
        return mcg::fail(MCG_ERR_INVALID, "mcg_trim_memory: device ordinal out of range");
    }
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    free_kept(device);
    cudaSetDevice(prev);
    return MCG_OK;
}

namespace {

// Strip mode's program: segments of events and gates (plan_segments), the
// gates of each in groups of up to kStripGroup that the kernel evaluates
// together (no gate of a group reads another, so all their input loads can be
// in flight at once).  AND, OR, NAND and NOR gates of at most
// kStripGroupMaxIn inputs, one-of-n and n-of-n among them, and NOT and NULL
// gates (of their last input) take the OR form r = outinv ^ OR_i (x_i ^
// flip_i) (De Morgan: AND = ~OR(~x), NAND = OR(~x)); flip_i also carries the
// input's negation.  A group is taken from the gates whose inputs are there,
// four of one fan-in if there are so many, so that its slots are mostly full.
// Every other gate (XOR, other ATLEAST, wider gates) is a group of one
// evaluated by strip_gate.  Each group is two uint4 records: its header and
// the output rows of its gates.
//
// 384 events per segment: the blocks of a launch start together, and where
// all of them sampled all events and then evaluated all gates, the gates'
// loads had little to hide under.  2^20 words of the 5,000-event tree: 190.8
// ms; with one segment 197.7 (layer by layer 193.9), with 48 events per
// segment, whose groups are less full, 197.1, with 96 to 768 190.7 to 191.
constexpr uint32_t kStripSegmentEvents = 384;

mcg_status build_strip_program(mcg_engine *e) {
    using mcg::dev::kStripGroup;
    using mcg::dev::kStripGroupMaxIn;
    const mcg::Graph &g = e->graph;
    constexpr uint32_t kRowBytes = mcg::dev::kStripLanes * (uint32_t)sizeof(uint64_t);
    const mcg::SegmentPlan plan = mcg::plan_segments(g, kStripSegmentEvents, false);
    if ((uint64_t)plan.slots + 1 > 0xFFFFFFFFull / kRowBytes)
        return mcg::fail(MCG_ERR_INVALID, "strip mode: too many nodes");
    e->strip_rows = plan.slots + 1;
    const uint32_t empty = plan.slots * kRowBytes;
    const uint32_t nb = g.n_be;
    std::vector<uint4> be, tab_be, groups, ginfo, single;
    std::vector<uint2> segment, be_tally;
    std::vector<uint32_t> gin, inputs, tally_list;
    for (size_t i = 0; i < plan.tile.event.size(); ++i) {
        const uint32_t v = plan.tile.event[i];
        const uint4 r = make_uint4((uint32_t)g.be_pdag_idx[v] + 1u, g.be_event_idx[v] + 1u,
                                   (uint32_t)g.be_threshold[v], (uint32_t)(g.be_threshold[v] >> 32));
        tab_be.push_back(r);
        be.push_back(make_uint4(plan.event_slot[i] * kRowBytes, r.y, r.z, r.w));
    }
    for (const uint2 &t : plan.tile.be_tally) be_tally.push_back(make_uint2(t.x * kRowBytes, t.y));
    std::vector<std::vector<uint32_t>> tallies(g.n_gates);
    for (uint32_t t = 0; t < (uint32_t)g.tally_nodes.size(); ++t)
        if (g.tally_nodes[t] >= nb) tallies[g.tally_nodes[t] - nb].push_back(t);
    // A row is used again by later segments, so the rows of a gate's inputs
    // are those of its segment: kept per node as the segments go by.
    std::vector<uint32_t> row(g.n_nodes(), 0);
    std::vector<uint32_t> waiting(g.n_gates, 0);  // inputs of the gate that this segment still has to evaluate
    std::vector<std::vector<uint32_t>> readers(g.n_gates);
    std::vector<char> here(g.n_gates, 0);
    auto last_only = [&](uint32_t i) { return g.gate_op[i] == MCG_NOT || g.gate_op[i] == MCG_NULL; };
    auto first = [&](uint32_t i) { return last_only(i) && g.gate_in_count[i] ? g.gate_in_count[i] - 1 : 0u; };
    auto fan_in = [&](uint32_t i) { return g.gate_in_count[i] - first(i); };
    // 0: a group of its own, 1: OR form of the inputs, 2: of their complements
    auto or_form = [&](uint32_t i) -> int {
        const uint8_t op = g.gate_op[i];
        const uint32_t n = g.gate_in_count[i], k = g.gate_k[i] & 0xFFu;
        if (last_only(i)) return 1;
        if (n > kStripGroupMaxIn) return 0;
        if (op == MCG_OR || op == MCG_NOR || (op == MCG_ATLEAST && k == 1 && n >= 1)) return 1;
        if (op == MCG_AND || op == MCG_NAND || (op == MCG_ATLEAST && k == n && n >= 1)) return 2;
        return 0;
    };
    auto inverted = [&](uint32_t i) {  // of the OR form
        const uint8_t op = g.gate_op[i];
        return op == MCG_AND || op == MCG_NOR || op == MCG_NOT || (op == MCG_ATLEAST && or_form(i) == 2);
    };
    auto info = [&](uint32_t i, uint32_t own) {
        ginfo.push_back(make_uint4(row[nb + i], (uint32_t)tally_list.size(), (uint32_t)tallies[i].size(), own));
        tally_list.insert(tally_list.end(), tallies[i].begin(), tallies[i].end());
    };
    uint32_t ev = 0, layer = 0;
    for (const uint2 &seg : plan.segment) {
        for (; ev < seg.x; ++ev) row[plan.tile.event[ev]] = plan.event_slot[ev] * kRowBytes;
        const uint32_t q0 = plan.tile.layer[layer], q1 = plan.tile.layer[seg.y];
        layer = seg.y;
        std::vector<uint32_t> ready[kStripGroupMaxIn + 1], own;  // by fan-in; groups of one
        auto offer = [&](uint32_t i) { (or_form(i) ? ready[fan_in(i)] : own).push_back(i); };
        for (uint32_t q = q0; q < q1; ++q) {
            const uint32_t i = plan.gate[q];
            here[i] = 1;
            row[nb + i] = plan.gate_slot[q] * kRowBytes;
        }
        for (uint32_t q = q0; q < q1; ++q) {
            const uint32_t i = plan.gate[q];
            for (uint32_t j = first(i); j < g.gate_in_count[i]; ++j) {
                const uint32_t c = g.inputs[g.gate_in_begin[i] + j];
                if (c >= nb && here[c - nb]) {
                    ++waiting[i];
                    readers[c - nb].push_back(i);
                }
            }
            if (!waiting[i]) offer(i);
        }
        auto done = [&](uint32_t i) {
            for (uint32_t r : readers[i])
                if (--waiting[r] == 0) offer(r);
        };
        for (uint32_t left = q1 - q0; left;) {
            if (!own.empty()) {
                const uint32_t i = own.back();
                own.pop_back();
                groups.push_back(make_uint4(1u | (1u << 24), 0u, (uint32_t)ginfo.size(), 0u));
                groups.push_back(make_uint4(row[nb + i], 0u, 0u, 0u));
                info(i, (uint32_t)single.size());
                const uint32_t n = g.gate_in_count[i];
                uint32_t nbits = 0;
                while (nbits < 8 && (n >> nbits) != 0) ++nbits;
                single.push_back(make_uint4((uint32_t)g.gate_op[i] | ((g.gate_k[i] & 0xFFu) << 8) |
                                                (std::max(nbits, 1u) << 16),
                                            (uint32_t)inputs.size(), n, g.gate_neg_count[i]));
                for (uint32_t j = 0; j < n; ++j) inputs.push_back(row[g.inputs[g.gate_in_begin[i] + j]]);
                done(i);
                --left;
                continue;
            }
            uint32_t most = 0;  // the fan-in of most ready gates
            for (uint32_t f = 1; f <= kStripGroupMaxIn; ++f)
                if (ready[f].size() > ready[most].size()) most = f;
            std::vector<uint32_t> pick;
            auto take = [&](std::vector<uint32_t> &from) {
                while (pick.size() < kStripGroup && !from.empty()) {
                    pick.push_back(from.back());
                    from.pop_back();
                }
            };
            if (ready[most].size() >= kStripGroup) take(ready[most]);
            else
                for (uint32_t f = kStripGroupMaxIn + 1; f-- > 0;) take(ready[f]);
            const uint32_t cnt = (uint32_t)pick.size();
            uint32_t maxn = 0, outinv = 0, outs[kStripGroup] = {0u, 0u, 0u, 0u};
            for (uint32_t j = 0; j < cnt; ++j) {
                maxn = std::max(maxn, fan_in(pick[j]));
                if (inverted(pick[j])) outinv |= 1u << j;
                outs[j] = row[nb + pick[j]];
            }
            groups.push_back(make_uint4(cnt | (maxn << 8), (uint32_t)gin.size(), (uint32_t)ginfo.size(), outinv));
            groups.push_back(make_uint4(outs[0], outs[1], outs[2], outs[3]));
            for (uint32_t s = 0; s < maxn; ++s) {
                for (uint32_t j = 0; j < kStripGroup; ++j) {
                    uint32_t rec = empty;
                    if (j < cnt && s < fan_in(pick[j])) {
                        const uint32_t i = pick[j], at = first(i) + s, n = g.gate_in_count[i];
                        const bool negated = at >= n - g.gate_neg_count[i];
                        rec = row[g.inputs[g.gate_in_begin[i] + at]] | (uint32_t)(negated != (or_form(i) == 2));
                    }
                    gin.push_back(rec);
                }
            }
            for (uint32_t i : pick) info(i, 0u);
            for (uint32_t i : pick) done(i);
            left -= cnt;
        }
        for (uint32_t q = q0; q < q1; ++q) {
            here[plan.gate[q]] = 0;
            readers[plan.gate[q]].clear();
        }
        segment.push_back(make_uint2(ev, (uint32_t)groups.size() / 2));
    }
    e->n_strip_be = (uint32_t)be.size();
    e->n_strip_segments = (uint32_t)segment.size();
    e->n_strip_be_tally = (uint32_t)be_tally.size();
    MCG_CUDA(upload(&e->d_strip_be, be));
    MCG_CUDA(upload(&e->d_strip_table_be, tab_be));
    MCG_CUDA(upload(&e->d_strip_segment, segment));
    MCG_CUDA(upload(&e->d_strip_single, single));
    MCG_CUDA(upload(&e->d_strip_inputs, inputs));
    MCG_CUDA(upload(&e->d_strip_groups, groups));
    MCG_CUDA(upload(&e->d_strip_gin, gin));
    MCG_CUDA(upload(&e->d_strip_ginfo, ginfo));
    MCG_CUDA(upload(&e->d_strip_be_tally, be_tally));
    MCG_CUDA(upload(&e->d_gate_tally_list, tally_list));
    return MCG_OK;
}

mcg_status build_layered_tables(mcg_engine *e) {
    const mcg::Graph &g = e->graph;
    std::vector<uint4> be(g.n_be);
    for (uint32_t i = 0; i < g.n_be; ++i) {
        be[i] = make_uint4((uint32_t)g.be_pdag_idx[i] + 1u, g.be_event_idx[i] + 1u, (uint32_t)g.be_threshold[i],
                           (uint32_t)(g.be_threshold[i] >> 32));
    }
    std::vector<uint4> meta(g.n_gates);
    std::vector<uint32_t> layer(g.n_gates, 1);
    uint32_t n_layers = 0;
    for (uint32_t i = 0; i < g.n_gates; ++i) {
        meta[i] = make_uint4((uint32_t)g.gate_op[i] | ((g.gate_k[i] & 0xFFu) << 8), g.gate_in_begin[i],
                             g.gate_in_count[i], g.gate_neg_count[i]);
        uint32_t l = 1;
        for (uint32_t j = 0; j < g.gate_in_count[i]; ++j) {
            const uint32_t c = g.inputs[g.gate_in_begin[i] + j];
            if (c >= g.n_be) l = std::max(l, layer[c - g.n_be] + 1);
        }
        layer[i] = l;
        n_layers = std::max(n_layers, l);
    }
    // Gate ids grouped by layer (layer 1 .. n_layers), like the reference's
    // LayeredTopologicalOrder depth (src/preprocessor.cc:130-171).
    std::vector<uint32_t> counts(n_layers + 2, 0);
    for (uint32_t i = 0; i < g.n_gates; ++i) counts[layer[i]]++;
    e->layer_offsets.assign(n_layers + 1, 0);
    for (uint32_t l = 1; l <= n_layers; ++l) e->layer_offsets[l] = e->layer_offsets[l - 1] + counts[l];
    std::vector<uint32_t> cursor(e->layer_offsets.begin(), e->layer_offsets.end());
    std::vector<uint32_t> order(g.n_gates);
    for (uint32_t i = 0; i < g.n_gates; ++i) order[cursor[layer[i] - 1]++] = i;

    std::vector<uint32_t> be_nodes, be_idx;
    for (uint32_t t = 0; t < (uint32_t)g.tally_nodes.size(); ++t) {
        if (g.tally_nodes[t] < g.n_be) {
            be_nodes.push_back(g.tally_nodes[t]);
            be_idx.push_back(t);
        }
    }
    e->n_be_tally = (uint32_t)be_nodes.size();
    if (e->mode == MCG_MODE_STRIP) {
        mcg_status st = build_strip_program(e);
        if (st != MCG_OK) return st;
    } else if (e->mode == MCG_MODE_STAGED) {
        const mcg::GatePlan plan = mcg::plan_gates(g, layer);
        e->n_gate_parts = plan.parts();
        e->n_gate_layers = plan.part[plan.parts() + 1] - plan.part[plan.parts()];
        e->gates_largest_part = plan.largest;
        e->gate_block_ns = plan.block_ns;
        e->gates_count = plan.counts;
        MCG_CUDA(upload(&e->d_gates, plan.gates));
        MCG_CUDA(upload(&e->d_gate_in, plan.in));
        MCG_CUDA(upload(&e->d_gate_tally, plan.tally));
        MCG_CUDA(upload(&e->d_gate_tally_list, plan.tally_list));
        MCG_CUDA(upload(&e->d_gate_part, plan.part));
        MCG_CUDA(upload(&e->d_gate_layer, plan.layer));
    }
    MCG_CUDA(upload(&e->d_be_tally_nodes, be_nodes));
    MCG_CUDA(upload(&e->d_be_tally_idx, be_idx));

    MCG_CUDA(upload(&e->d_be, be));
    MCG_CUDA(upload(&e->d_meta, meta));
    MCG_CUDA(upload(&e->d_inputs, g.inputs));
    MCG_CUDA(upload(&e->d_tally_nodes, g.tally_nodes));
    MCG_CUDA(upload(&e->d_layer_gates, order));
    return MCG_OK;
}

dim3 rows_grid(uint64_t words, uint32_t rows, uint32_t threads) {
    const uint32_t bx = (uint32_t)((words + threads - 1) / threads);
    uint32_t by = rows, bz = 1;
    while (by > 65535u) {
        bz *= 2;
        by = (rows + bz - 1) / bz;
    }
    return dim3(bx, by, bz);
}

// Materialises every node's words for one pass over [word_begin, word_begin + W)
// into d_buf (reference dataflow).
mcg_status layered_eval(mcg_engine *e, uint32_t iteration, uint64_t word_begin, uint64_t W) {
    const mcg::Graph &g = e->graph;
    const uint64_t need = (uint64_t)g.n_nodes() * W;
    if (need > e->buf_words) {
        if (e->d_buf) cudaFree(e->d_buf);
        e->d_buf = nullptr;
        e->buf_words = 0;
        MCG_CUDA(cudaMalloc((void **)&e->d_buf, std::max<uint64_t>(need, 1) * sizeof(uint64_t)));
        e->buf_words = need;
    }
    const uint32_t t3 = (iteration + 1u) << 6;
    if (g.n_be > 0) {
        mcg::dev::k_layer_be<kPackForm><<<rows_grid(W, g.n_be, 256), 256, 0, e->stream>>>(
            e->d_be, g.n_be, W, word_begin, t3, e->d_buf);
        ++e->launches;
    }
    for (size_t l = 0; l + 1 < e->layer_offsets.size(); ++l) {
        const uint32_t n = e->layer_offsets[l + 1] - e->layer_offsets[l];
        if (n == 0) continue;
        mcg::dev::k_layer_gates<<<rows_grid(W, n, 256), 256, 0, e->stream>>>(
            e->d_meta, e->d_inputs, e->d_layer_gates + e->layer_offsets[l], n, g.n_be, W, e->d_buf);
        ++e->launches;
    }
    MCG_CUDA(cudaGetLastError());
    return MCG_OK;
}

using FusedKernel = void (*)(mcg::dev::FusedArgs);

// Register budget follows the CTAs wanted per SM (65536 / (256 * n) per thread).
FusedKernel fused_kernel(uint32_t ctas_per_sm) {
    switch (ctas_per_sm) {
        case 1: return mcg::dev::k_fused<kFusedThreads, 1, kPackForm>;
        case 3: return mcg::dev::k_fused<kFusedThreads, 3, kPackForm>;
        case 4: return mcg::dev::k_fused<kFusedThreads, 4, kPackForm>;
        default: return mcg::dev::k_fused<kFusedThreads, 2, kPackForm>;
    }
}

// Host-only compilation of the fused program (launch shape from the options).
mcg_status compile_fused(mcg_engine *e, const mcg_run_desc &run) {
    mcg::DeviceShape prop;
    MCG_CUDA(mcg::device_shape(&prop, e->device));
    if (run.block_threads != 0 && run.block_threads != kFusedThreads)
        return mcg::fail(MCG_ERR_INVALID, "block_threads must be 0 or 256");
    e->nt = kFusedThreads;
    // 4 CTAs per SM measured fastest on the 200- and the 5,000-event trees
    const uint32_t ctas_per_sm = run.ctas_per_sm ? run.ctas_per_sm : 4u;
    if (ctas_per_sm < 1 || ctas_per_sm > 4) return mcg::fail(MCG_ERR_INVALID, "ctas_per_sm must be 1..4");
    e->ctas_per_sm = ctas_per_sm;
    const size_t smem_cap = std::min<size_t>(prop.sharedMemPerBlockOptin, prop.sharedMemPerMultiprocessor / ctas_per_sm) -
                            1024;  // per-CTA reserve
    const uint64_t n_tally = e->graph.tally_nodes.size();
    size_t tally_bytes = n_tally * sizeof(unsigned long long);
    e->tally_in_smem = tally_bytes <= smem_cap / 2;
    if (!e->tally_in_smem) tally_bytes = 0;
    const size_t slot_bytes = (size_t)e->nt * sizeof(uint64_t);
    uint32_t budget = (uint32_t)((smem_cap - tally_bytes) / slot_bytes);
    if (run.smem_slots == MCG_SMEM_SLOTS_NONE) budget = 0;
    else if (run.smem_slots) budget = std::min(budget, run.smem_slots);
    const std::string err = mcg::compile_program(e->graph, budget, e->prog);
    if (!err.empty()) return mcg::fail(MCG_ERR_INVALID, err);
    e->smem_bytes = (uint32_t)(e->prog.smem_slots * slot_bytes + tally_bytes);
    e->grid = (uint32_t)prop.multiProcessorCount * ctas_per_sm;
    e->scratch_stride = (uint64_t)e->grid * e->nt;
    e->chunk_words = run.chunk_words ? run.chunk_words : kDefaultChunkWords;
    e->prog_compiled = true;
    return MCG_OK;
}

using TileKernel = void (*)(const mcg::dev::TileArgs);
TileKernel tile_kernel(uint32_t threads) {
    switch (threads) {
        case 256: return mcg::dev::k_tile<256, kPackForm>;
        case 512: return mcg::dev::k_tile<512, kPackForm>;
        default: return mcg::dev::k_tile<1024, kPackForm>;
    }
}

template <typename T>
mcg_status upload_tile(mcg_engine *e, const T **dptr, const std::vector<T> &v) {
    T *p = nullptr;
    MCG_CUDA(upload(&p, v));
    if (p) e->tile_tables.push_back(p);
    *dptr = p;
    return MCG_OK;
}

// Fused mode's default shape where 32 words of every needed node (about 880 on
// a B200), or of every one that is live at a time in segments, have room in
// shared memory: e->tile, or not.  233,937
// words, all gates tallied: 1,030 events in segments 9.1 ms, the interpreter
// 13.9; 2,500 events 23.5 and 36.3; 4,096 words of them 0.22 and 2.75, 0.50 and
// 7.3 ms.
mcg_status setup_tile(mcg_engine *e) {
    const mcg::Graph &g = e->graph;
    mcg::DeviceShape dev;
    MCG_CUDA(mcg::device_shape(&dev, e->device));
    constexpr uint32_t kSlotBytes = mcg::dev::kTileLanes * sizeof(uint64_t);
    // the most, and so the smallest, blocks that share an SM's 1,024 threads
    // and its shared memory; the tally counters go to shared memory where
    // they fit as well
    uint32_t threads = 0;
    uint64_t room = 0, words = 0;
    auto fit = [&](uint64_t slots) {
        words = (slots + 1) * kSlotBytes;  // and the empty input
        for (uint32_t nt : {256u, 512u, 1024u}) {
            const uint64_t own = (nt / 32u) * mcg::dev::kEventTableStride * sizeof(uint2);
            const uint64_t most = std::min<uint64_t>(
                dev.sharedMemPerBlockOptin, dev.sharedMemPerMultiprocessor / (1024u / nt) - dev.reservedSharedMemPerBlock);
            if (words + own > most) continue;
            threads = nt;
            room = most - own;
            return true;
        }
        return false;
    };
    mcg::TilePlan t = mcg::plan_tile(g);
    uint32_t slots = t.slots();
    std::vector<uint32_t> event_slot(t.event.size()), gate_slot(t.gates.size());
    std::vector<uint2> segment{make_uint2((uint32_t)t.event.size(), (uint32_t)t.layer.size() - 1)};
    for (uint32_t i = 0; i < slots; ++i) (i < t.event.size() ? event_slot[i] : gate_slot[i - t.event.size()]) = i;
    if (!fit(slots)) {
        // segments: as long as their rows fit, since each has its own layers to wait for
        for (uint32_t events : {256u, 96u}) {
            mcg::SegmentPlan p = mcg::plan_segments(g, events, true, 32);
            slots = p.slots;
            if (!fit(slots)) continue;
            t = std::move(p.tile);
            segment = std::move(p.segment);
            event_slot = std::move(p.event_slot);
            gate_slot = std::move(p.gate_slot);
            break;
        }
    }
    if (!threads || !t.fits) return MCG_OK;
    for (uint32_t &rec : t.in) rec = t.byte_record(rec, kSlotBytes, 0, slots);
    for (size_t i = 0; i < t.gates.size(); ++i) {
        if (t.gates[i].z > 0xFFFFu) return MCG_OK;
        t.gates[i].z |= gate_slot[i] * mcg::dev::kTileLanes << 16;
    }
    const uint64_t counters = g.tally_nodes.size() * sizeof(unsigned long long);
    mcg::dev::TileArgs &a = e->tile_args;
    a = mcg::dev::TileArgs{};
    a.tally_in_smem = words + counters <= room ? 1u : 0u;
    e->tile_smem = (uint32_t)(words + (a.tally_in_smem ? counters : 0));
    mcg_status st = MCG_OK;
    for (uint32_t nt = threads; nt <= 1024u && st == MCG_OK; nt *= 2) st = mcg::set_smem_limit(tile_kernel(nt), e->tile_smem);
    if (st != MCG_OK) return st;
    std::vector<uint4> be(t.event.size());
    for (size_t i = 0; i < be.size(); ++i) {
        const uint32_t v = t.event[i];
        be[i] = make_uint4((uint32_t)g.be_pdag_idx[v] + 1u, g.be_event_idx[v] + 1u, (uint32_t)g.be_threshold[v],
                           (uint32_t)(g.be_threshold[v] >> 32) | event_slot[i] * mcg::dev::kTileLanes << 1);
    }
    if ((st = upload_tile(e, &a.be, be)) != MCG_OK || (st = upload_tile(e, &a.gates, t.gates)) != MCG_OK ||
        (st = upload_tile(e, &a.in, t.in)) != MCG_OK || (st = upload_tile(e, &a.layer, t.layer)) != MCG_OK ||
        (st = upload_tile(e, &a.tally_list, t.tally_list)) != MCG_OK ||
        (st = upload_tile(e, &a.be_tally, t.be_tally)) != MCG_OK ||
        (st = upload_tile(e, &a.segment, segment)) != MCG_OK)
        return st;
    a.n_slots = slots + 1;
    a.n_segments = (uint32_t)segment.size();
    a.n_be_tally = (uint32_t)t.be_tally.size();
    a.n_tally = (uint32_t)g.tally_nodes.size();
    e->tile_threads = threads;
    e->tile_sms = (uint32_t)dev.multiProcessorCount;
    e->tile = true;
    e->tile_cost = mcg::TileCost(t.layer, t.gates, t.event.size(), t.in.size(), g.tally_nodes.size(), e->tile_sms, threads,
                                 e->tile_smem + (threads / 32) * sizeof(uint2) * mcg::dev::kEventTableStride +
                                     dev.reservedSharedMemPerBlock);
    return MCG_OK;
}

uint64_t tiles_of(uint64_t words) { return (words + mcg::dev::kTileLanes - 1) / mcg::dev::kTileLanes; }

// Threads of the tile kernel's blocks in a pass: a pass with fewer tiles than
// resident blocks gives each of them more warps (4,096 words of a 60-event tree
// are 128 tiles: 18.2 us with 1,024 threads each, 23.3 us with 256).
uint32_t tile_pass_threads(const mcg_engine *e, uint64_t words) {
    uint32_t threads = e->tile_threads;
    while (threads < 1024u && tiles_of(words) < (uint64_t)e->tile_sms * (1024u / threads)) threads *= 2;
    return threads;
}

// Whether a launch over so many words of a fused-mode engine is the tile kernel's.
bool takes_tile(const mcg_engine *e, uint64_t words) {
    return e->tile && (!e->d_ops || !e->tile_cost.interpreter_is_faster(words));
}

mcg_status launch_tile(mcg_engine *e, uint32_t it_first, uint32_t n_it, uint64_t word_begin, uint64_t count) {
    mcg::dev::TileArgs a = e->tile_args;
    a.iteration_first = it_first;
    a.n_iterations = n_it;
    a.word_begin = word_begin;
    a.word_count = count;
    a.ones = e->d_tally;
    const uint64_t tiles = tiles_of(count);
    const uint32_t threads = tile_pass_threads(e, count);
    const uint32_t grid = (uint32_t)std::min<uint64_t>((uint64_t)e->tile_sms * (1024u / threads),
                                                       std::max<uint64_t>(tiles, 1));
    tile_kernel(threads)<<<grid, threads, e->tile_smem, e->stream>>>(a);
    ++e->launches;
    MCG_CUDA(cudaGetLastError());
    return MCG_OK;
}

mcg_status setup_interpreter(mcg_engine *e, const mcg_run_desc &run) {
    mcg_status st = compile_fused(e, run);
    if (st != MCG_OK) return st;
    st = mcg::set_smem_limit(fused_kernel(e->ctas_per_sm), e->smem_bytes);
    if (st != MCG_OK) return st;
    if (e->prog.global_slots)
        MCG_CUDA(work_alloc(e, (void **)&e->d_scratch,
                            (size_t)e->prog.global_slots * e->scratch_stride * sizeof(uint64_t)));
    MCG_CUDA(upload(reinterpret_cast<mcg::Op **>(&e->d_ops), e->prog.ops));
    return MCG_OK;
}

mcg_status setup_fused(mcg_engine *e, const mcg_run_desc &run) {
    // the default shape (no slot count, block size or residency of its own)
    if (!run.smem_slots && !run.block_threads && (!run.ctas_per_sm || run.ctas_per_sm == 4)) {
        const mcg_status ts = setup_tile(e);
        if (ts != MCG_OK) return ts;
    }
    if (!e->tile) return setup_interpreter(e, run);
    e->ctas_per_sm = 4;
    e->chunk_words = run.chunk_words ? run.chunk_words : kDefaultChunkWords;
    // next to the tile kernel where some passes are the interpreter's, and where there is room for it
    if (!e->tile_cost.interpreter_may_be_faster()) return MCG_OK;
    const mcg_status st = setup_interpreter(e, run);
    if (st != MCG_ERR_OOM) return st;
    mcg::clear_error();
    return MCG_OK;
}

// From a block of so many words per SM on, gate blocks take two words per lane:
// half the loads and instructions per word.  Fewer words are one per lane, for
// twice the blocks (32,768 words of the 5,000-event tree: 6.23 ms, one word per
// lane 6.55; 2,048 words of a 500-event tree: no difference).
constexpr uint64_t kWideGateWords = 64;
constexpr uint32_t kStripBlocksPerSm = 6, kStripFewBlocks = 4;

mcg_status setup_staged(mcg_engine *e, const mcg_run_desc &run,
                        const std::function<uint64_t(uint64_t)> &extra_words) {
    const mcg::Graph &g = e->graph;
    const uint64_t nn = std::max<uint64_t>(g.n_nodes(), 1);
    // two chunk buffers, together at most ~48 GB by default
    uint64_t words = run.layered_max_words ? run.layered_max_words : (24ull << 30) / (nn * sizeof(uint64_t));
    words = std::max<uint64_t>(256, std::min<uint64_t>(words, 1ull << 20));
    words = (words + 255) / 256 * 256;
    e->stage_words = words;
    const uint64_t extra = extra_words ? extra_words(words) : 0;
    e->stage_extra_words = extra;
    MCG_CUDA(work_alloc(e, (void **)&e->d_stage[0], (nn * words + extra) * sizeof(uint64_t)));
    MCG_CUDA(work_alloc(e, (void **)&e->d_stage[1], nn * words * sizeof(uint64_t)));
    if (extra) e->d_stage_extra = e->d_stage[0] + nn * words;
    MCG_CUDA(cudaMalloc((void **)&e->d_event_table,
                        std::max<uint64_t>(e->graph.n_be, 1) * mcg::dev::kEventTableStride * sizeof(uint2)));
    // Cap the resident sampler blocks per SM through their shared-memory
    // footprint, so gate-phase blocks (memory bound) can run next to them.
    mcg::DeviceShape prop;
    MCG_CUDA(mcg::device_shape(&prop, e->device));
    const uint32_t blocks = run.sampler_blocks_per_sm ? run.sampler_blocks_per_sm : 8u;
    if (blocks < 1 || blocks > 8) return mcg::fail(MCG_ERR_INVALID, "sampler_blocks_per_sm must be 1..8");
    e->sampler_smem = blocks >= 8 ? 0u : (uint32_t)(prop.sharedMemPerMultiprocessor / blocks - 2048);
    const mcg_status lim = mcg::set_smem_limit(mcg::dev::k_stage_be<kPackForm>,
                                               e->sampler_smem);
    if (lim != MCG_OK) return lim;
    // Gate blocks of a chunk that the next one is sampled beside: two per SM, as
    // they would otherwise fill the SMs' registers and stop the sampling while
    // they wait for memory.  300,001 words of a 1,003-event tree in three
    // chunks: 11.12 ms with all blocks at once, 10.84 ms with 3 per SM, 10.79
    // with 2 or 1.5, 10.94 with 1.  Trees with so many gates per event that the
    // gate phase is the longer one get all blocks.
    const uint64_t traffic = g.inputs.size() + g.n_gates;
    e->gates_beside_sampler = traffic <= 8ull * g.n_be;
    e->gate_sms = (uint32_t)prop.multiProcessorCount;
    // The gate phase of chunk k runs while chunk k+1 is sampled: giving its
    // stream the higher priority lets its (memory-bound) blocks be scheduled
    // in between the sampler's blocks instead of after all of them.
    int prio_low = 0, prio_high = 0;
    MCG_CUDA(cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high));
    MCG_CUDA(cudaStreamCreateWithPriority(&e->s_a, cudaStreamNonBlocking, prio_low));
    MCG_CUDA(cudaStreamCreateWithPriority(&e->s_b, cudaStreamNonBlocking, prio_high));
    for (cudaEvent_t *ev : {&e->ev_fork, &e->ev_a[0], &e->ev_a[1], &e->ev_b[0], &e->ev_b[1], &e->ev_join_a,
                            &e->ev_join_b})
        MCG_CUDA(cudaEventCreateWithFlags(ev, cudaEventDisableTiming));
    return MCG_OK;
}

// Strip kernel for a residency target: fewer blocks per SM give each thread
// more registers (6: 40, 5: 48, 4: 64).
using StripKernel = void (*)(mcg::dev::StripArgs);
StripKernel strip_kernel(uint32_t blocks_per_sm) {
    switch (blocks_per_sm) {
        case 4: return mcg::dev::k_strip<kPackForm, 4>;
        case 5: return mcg::dev::k_strip<kPackForm, 5>;
        default: return mcg::dev::k_strip<kPackForm, 6>;
    }
}

mcg_status setup_strip(mcg_engine *e, const mcg_run_desc &run) {
    const mcg::Graph &g = e->graph;
    mcg::DeviceShape prop;
    MCG_CUDA(mcg::device_shape(&prop, e->device));
    const uint32_t target = run.ctas_per_sm ? run.ctas_per_sm : kStripBlocksPerSm;
    if (target < 4 || target > 6) return mcg::fail(MCG_ERR_INVALID, "strip mode: ctas_per_sm must be 0 or 4..6");
    e->strip_blocks = target;
    const uint64_t n_tally = g.tally_nodes.size();
    // tally counters in shared memory while the target residency still fits
    const uint64_t tally_bytes = n_tally * sizeof(unsigned long long);
    const uint64_t per_block = prop.sharedMemPerMultiprocessor / target - 2048;
    e->strip_smem = tally_bytes <= per_block ? (uint32_t)tally_bytes : 0u;
    const StripKernel kern = strip_kernel(target);
    const mcg_status lim = mcg::set_smem_limit(kern, e->strip_smem);
    if (lim != MCG_OK) return lim;
    int per_sm = 0;
    MCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, mcg::dev::kStripThreads, e->strip_smem));
    if (per_sm < 1) return mcg::fail(MCG_ERR_INVALID, "strip kernel does not fit on an SM");
    e->strip_grid = (uint32_t)(prop.multiProcessorCount * per_sm);
    if (!run.ctas_per_sm) {
        const mcg_status few = mcg::set_smem_limit(strip_kernel(kStripFewBlocks), e->strip_smem);
        if (few != MCG_OK) return few;
        e->strip_few = kStripFewBlocks * (uint64_t)prop.multiProcessorCount;
    }
    const uint64_t warps = (uint64_t)e->strip_grid * (mcg::dev::kStripThreads / 32);
    const uint64_t bytes = warps * e->strip_rows * mcg::dev::kStripLanes * sizeof(uint64_t);
    MCG_CUDA(work_alloc(e, (void **)&e->d_strip_scratch, bytes));
    MCG_CUDA(cudaMalloc((void **)&e->d_queue, sizeof(unsigned long long)));
    MCG_CUDA(cudaMalloc((void **)&e->d_event_table,
                        std::max<uint64_t>(g.n_be, 1) * mcg::dev::kEventTableStride * sizeof(uint2)));
    return MCG_OK;
}

// One persistent launch per pass on the engine stream.
mcg_status run_strip(mcg_engine *e, uint32_t it_first, uint32_t n_it, uint64_t word_begin, uint64_t count) {
    const mcg::Graph &g = e->graph;
    mcg::dev::StripArgs a{};
    a.be = e->d_strip_be;
    a.table = e->d_event_table;
    a.segment = e->d_strip_segment;
    a.n_segments = e->n_strip_segments;
    a.rows = e->strip_rows;
    a.single = e->d_strip_single;
    a.inputs = e->d_strip_inputs;
    a.groups = e->d_strip_groups;
    a.gin = e->d_strip_gin;
    a.ginfo = e->d_strip_ginfo;
    a.tally_list = e->d_gate_tally_list;
    a.be_tally = e->d_strip_be_tally;
    a.n_be_tally = e->n_strip_be_tally;
    a.n_tally = (uint32_t)g.tally_nodes.size();
    a.tally_in_smem = e->strip_smem ? 1u : 0u;
    a.ones = e->d_tally;
    a.scratch = e->d_strip_scratch;
    a.word_begin = word_begin;
    a.word_count = count;
    a.queue = e->d_queue;
    // No more blocks than strips: they then lie one to an SM, two to an SM and so
    // on, where of a full grid any blocks take the strips.  At up to four strips
    // per SM the kernel for four blocks, whose threads have 64 registers, is the
    // faster one.  958 events, 27,987 words: 1.95 ms (five blocks 2.07, full grid
    // 5.4); 151,552 words: 5.38 (five blocks 5.53, full grid of six 7.9).
    const uint64_t strips = (count + mcg::dev::kStripThreads - 1) / mcg::dev::kStripThreads;
    const uint32_t blocks = strips <= e->strip_few ? kStripFewBlocks : e->strip_blocks;
    const uint32_t grid = (uint32_t)std::min<uint64_t>(e->strip_grid, std::max<uint64_t>(strips, 1));
    for (uint32_t it = 0; it < n_it; ++it) {
        const uint32_t iteration = it_first + it;
        if (e->n_strip_be > 0 && e->table_iteration != iteration) {
            const uint64_t n = (uint64_t)e->n_strip_be * mcg::dev::kEventTableStride;
            mcg::dev::k_event_table<<<(uint32_t)((n + 255) / 256), 256, 0, e->stream>>>(
                e->d_strip_table_be, e->n_strip_be, (iteration + 1u) << 6, e->d_event_table);
            ++e->launches;
            e->table_iteration = iteration;
        }
        MCG_CUDA(cudaMemsetAsync(e->d_queue, 0, sizeof(unsigned long long), e->stream));
        cudaEvent_t p0 = nullptr, p1 = nullptr;
        if (e->profile_a) {
            if (e->prof_used == e->prof_events.size()) {
                cudaEvent_t x, y;
                MCG_CUDA(cudaEventCreate(&x));
                MCG_CUDA(cudaEventCreate(&y));
                e->prof_events.push_back({x, y});
            }
            p0 = e->prof_events[e->prof_used].first;
            p1 = e->prof_events[e->prof_used].second;
            ++e->prof_used;
            MCG_CUDA(cudaEventRecord(p0, e->stream));
        }
        strip_kernel(blocks)<<<grid, mcg::dev::kStripThreads, e->strip_smem, e->stream>>>(a);
        ++e->launches;
        if (p1) MCG_CUDA(cudaEventRecord(p1, e->stream));
        MCG_CUDA(cudaGetLastError());
    }
    return MCG_OK;
}

using StageGatesKernel = void (*)(const mcg::dev::StageGateArgs);
StageGatesKernel stage_gates_kernel(bool wide, bool count, bool split) {
    using mcg::dev::k_stage_gates;
    if (split) return count ? k_stage_gates<1, true, true> : k_stage_gates<1, false, true>;
    if (wide) return count ? k_stage_gates<2, true, false> : k_stage_gates<2, false, false>;
    return count ? k_stage_gates<1, true, false> : k_stage_gates<1, false, false>;
}

// Blocks that share the gates of a layer and tile, a launch per layer; 0: every
// layer in one launch, a block per tile and part.  The one launch leaves most of
// the chip idle where a pass has few tiles, and its blocks walk all gates of a
// part (gate_block_ns) where a launch per layer costs about 4 us, and more the
// more tiles share the rows.  The line is where the two sides crossed for 50 to
// 8,000 gates of 2 to 60 inputs in 2 to 50 layers: 64 words of 8,000 gates of 6
// inputs in 5 layers 57 us by layers and 283 in one launch, 256 words of 3,000 of
// 20 inputs 70 and 198, 2,048 words of 2,000 k-of-16 gates in 40 layers 378 and
// 370; from 3,000 words on one launch is the faster one but for layers of
// hundreds of gates.
constexpr uint64_t kGateLaunchNs = 4000;
uint32_t gate_splits(const mcg_engine *e, uint64_t tiles, uint64_t blocks) {
    if (2 * blocks > e->gate_sms ||
        e->gate_block_ns * e->gate_sms <= kGateLaunchNs * e->n_gate_layers * (e->gate_sms + 3 * blocks))
        return 0;
    const uint64_t wanted = (e->graph.n_gates / e->n_gate_layers + 7) / 8;  // a gate per warp of 256 threads
    const uint64_t most = (8ull * e->gate_sms + tiles - 1) / tiles;
    return (uint32_t)std::max<uint64_t>(1, std::min(wanted, most));
}

// One chunk: phase A (sampling) on s_a into buffer `set`, phase B (gates and
// tallies) on s_b once A is done; `last`: no chunk follows it.  A reuses a buffer only after the B that
// read it (two chunks earlier) has finished.
mcg_status staged_chunk(mcg_engine *e, uint64_t k, uint32_t iteration, uint64_t word_begin, uint64_t W,
                        bool last) {
    const mcg::Graph &g = e->graph;
    const int set = (int)(k & 1);
    uint64_t *buf = e->d_stage[set];
    const uint64_t stride = (W + 1) / 2 * 2;  // rows of an even length take 16-byte loads
    if (k >= 2) MCG_CUDA(cudaStreamWaitEvent(e->s_a, e->ev_b[set], 0));
    const uint32_t t3 = (iteration + 1u) << 6;
    const uint4 *be_tab = e->d_be_sample ? e->d_be_sample : e->d_be;
    if (g.n_be > 0 && e->table_iteration != iteration) {
        // s_a is in order: earlier sampler launches finish before the table changes
        const uint64_t n = (uint64_t)g.n_be * mcg::dev::kEventTableStride;
        mcg::dev::k_event_table<<<(uint32_t)((n + 255) / 256), 256, 0, e->s_a>>>(be_tab, g.n_be, t3,
                                                                                           e->d_event_table);
        ++e->launches;
        e->table_iteration = iteration;
    }
    if (g.n_be > 0) {
        // events per thread: fewer where the last wave of blocks would leave much
        // of the chip idle (2,048 words of 500 events: 185 us for the call, 188 with 4)
        const uint64_t waves = (uint64_t)g.n_be * ((W + 511) / 512) / (4ull * e->gate_sms);
        const uint32_t ept = waves >= 32 ? 4u : waves >= 16 ? 2u : 1u;
        const uint32_t groups = (g.n_be + ept - 1) / ept;
        cudaEvent_t p0 = nullptr, p1 = nullptr;
        if (e->profile_a) {
            if (e->prof_used == e->prof_events.size()) {
                cudaEvent_t a, b;
                MCG_CUDA(cudaEventCreate(&a));
                MCG_CUDA(cudaEventCreate(&b));
                e->prof_events.push_back({a, b});
            }
            p0 = e->prof_events[e->prof_used].first;
            p1 = e->prof_events[e->prof_used].second;
            ++e->prof_used;
            MCG_CUDA(cudaEventRecord(p0, e->s_a));
        }
        mcg::dev::k_stage_be<kPackForm><<<rows_grid((W + 1) / 2, groups, 256), 256, e->sampler_smem, e->s_a>>>(
            be_tab, e->d_event_table, g.n_be, ept, W, stride, word_begin, buf);
        ++e->launches;
        if (p1) MCG_CUDA(cudaEventRecord(p1, e->s_a));
    }
    if (e->sample_hook) {
        const mcg_status st = e->sample_hook(e->s_a, buf, W, stride, word_begin);
        if (st != MCG_OK) return st;
    }
    MCG_CUDA(cudaEventRecord(e->ev_a[set], e->s_a));
    MCG_CUDA(cudaStreamWaitEvent(e->s_b, e->ev_a[set], 0));
    if (g.n_gates > 0) {
        mcg::dev::StageGateArgs a{};
        a.gates = e->d_gates;
        a.in = e->d_gate_in;
        a.tally = e->d_gate_tally;
        a.tally_list = e->d_gate_tally_list;
        a.part = e->d_gate_part;
        a.layer = e->d_gate_layer;
        a.words = W;
        a.stride = stride;
        a.buf = buf;
        a.ones = e->d_tally;
        const bool wide = W >= kWideGateWords * e->gate_sms;
        uint64_t tiles = (W + (wide ? 63 : 31)) / (wide ? 64 : 32);
        // Warps per block: the fewer blocks share the chip, the more of a
        // layer's gates a block takes at a time.  Blocks are counted at the
        // largest part's gates, which a small part's blocks do not wait for.
        // 16 trees of very different sizes on 1,434 words: 0.49 ms with 512
        // threads, 0.90 with 256; 640 words of them: 0.25 ms with 1,024, 0.83
        // with 256.  512 blocks (32,768 words of one tree): 0.65 ms with 256.
        const uint64_t blocks = tiles * g.n_gates / std::max<uint32_t>(e->gates_largest_part, 1);
        const uint32_t threads = blocks >= 3ull * e->gate_sms ? 256u : blocks >= 2ull * e->gate_sms ? 512u : 1024u;
        if (!last && e->gates_beside_sampler) tiles = std::min<uint64_t>(tiles, 2ull * e->gate_sms);
        const uint32_t splits = gate_splits(e, tiles, blocks);
        const StageGatesKernel kern = stage_gates_kernel(wide, e->gates_count, splits > 0);
        if (!splits) {
            a.layers = e->n_gate_layers;
            kern<<<dim3((uint32_t)tiles, e->n_gate_parts), threads, 0, e->s_b>>>(a);
            ++e->launches;
        } else {
            a.part_first = e->n_gate_parts;  // all parts as one
            for (a.layers = 1; a.first < e->n_gate_layers; ++a.first) {
                kern<<<dim3((uint32_t)tiles, 1, splits), 256, 0, e->s_b>>>(a);
                ++e->launches;
            }
        }
    }
    if (e->n_be_tally) {
        dim3 grid = rows_grid(1, e->n_be_tally, 256);
        grid.x = (uint32_t)std::min<uint64_t>((W + 255) / 256, 64);
        mcg::dev::k_layer_tally<<<grid, 256, 0, e->s_b>>>(e->d_be_tally_nodes, e->n_be_tally, W, stride, buf, e->d_tally,
                                                          e->d_be_tally_idx);
        ++e->launches;
    }
    if (e->chunk_hook) {
        const mcg_status st = e->chunk_hook(e->s_b, buf, W, stride);
        if (st != MCG_OK) return st;
    }
    MCG_CUDA(cudaEventRecord(e->ev_b[set], e->s_b));
    MCG_CUDA(cudaGetLastError());
    return MCG_OK;
}

// Forks the staged streams from the engine stream, so that the chunks follow
// earlier work on it.
mcg_status staged_fork(mcg_engine *e) {
    MCG_CUDA(cudaEventRecord(e->ev_fork, e->stream));
    MCG_CUDA(cudaStreamWaitEvent(e->s_a, e->ev_fork, 0));
    MCG_CUDA(cudaStreamWaitEvent(e->s_b, e->ev_fork, 0));
    return MCG_OK;
}

// Chunks of n_it passes; *chunk counts them from the fork on (0 there), since
// a buffer waits for the gates of the chunk before last.  `more`: chunks of
// another call follow before the join.
mcg_status staged_chunks(mcg_engine *e, uint64_t *chunk, uint32_t it_first, uint32_t n_it, uint64_t word_begin,
                         uint64_t count, bool more) {
    for (uint32_t it = 0; it < n_it; ++it) {
        for (uint64_t off = 0; off < count; ++*chunk) {
            const uint64_t n = std::min<uint64_t>(e->stage_words, count - off);
            const mcg_status st = staged_chunk(e, *chunk, it_first + it, word_begin + off, n,
                                               !more && it + 1 == n_it && off + n == count);
            if (st != MCG_OK) return st;
            off += n;
        }
    }
    return MCG_OK;
}

mcg_status staged_join(mcg_engine *e) {
    MCG_CUDA(cudaEventRecord(e->ev_join_a, e->s_a));
    MCG_CUDA(cudaEventRecord(e->ev_join_b, e->s_b));
    MCG_CUDA(cudaStreamWaitEvent(e->stream, e->ev_join_a, 0));
    MCG_CUDA(cudaStreamWaitEvent(e->stream, e->ev_join_b, 0));
    return MCG_OK;
}

mcg_status run_staged_impl(mcg_engine *e, uint32_t it_first, uint32_t n_it, uint64_t word_begin, uint64_t count) {
    uint64_t chunk = 0;
    return mcg::forked_run([&] { return staged_fork(e); },
                           [&] { return staged_chunks(e, &chunk, it_first, n_it, word_begin, count, false); },
                           [&] { return staged_join(e); });
}

mcg_status launch_fused(mcg_engine *e, uint32_t it_first, uint32_t n_it, uint64_t word_begin, uint64_t count) {
    mcg::dev::FusedArgs a;
    a.ops = e->d_ops;
    a.smem_slots = e->prog.smem_slots;
    a.scratch = e->d_scratch;
    a.scratch_stride = e->scratch_stride;
    a.tally = e->d_tally;
    a.n_tally = (uint32_t)e->graph.tally_nodes.size();
    a.tally_in_smem = e->tally_in_smem ? 1u : 0u;
    a.iteration_first = it_first;
    a.n_iterations = n_it;
    a.word_begin = word_begin;
    a.word_count = count;
    const uint64_t want = (count + e->nt - 1) / e->nt;
    const uint32_t grid = (uint32_t)std::min<uint64_t>(e->grid, std::max<uint64_t>(want, 1));
    fused_kernel(e->ctas_per_sm)<<<grid, e->nt, e->smem_bytes, e->stream>>>(a);
    ++e->launches;
    MCG_CUDA(cudaGetLastError());
    return MCG_OK;
}

void release(mcg_engine *e) {
    // the side streams' work ends before their buffers go back to the pool
    if (e->s_a) cudaStreamSynchronize(e->s_a);
    if (e->s_b) cudaStreamSynchronize(e->s_b);
    if (e->stream) cudaStreamSynchronize(e->stream);
    work_free(e, e->d_scratch);
    work_free(e, e->d_stage[0]);
    work_free(e, e->d_stage[1]);
    work_free(e, e->d_strip_scratch);
    for (void *p : e->tile_tables) cudaFree(p);
    cudaFree(e->d_ops);
    cudaFree(e->d_tally);
    cudaFree(e->d_be);
    cudaFree(e->d_meta);
    cudaFree(e->d_inputs);
    cudaFree(e->d_tally_nodes);
    cudaFree(e->d_layer_gates);
    cudaFree(e->d_buf);
    cudaFree(e->d_strip_be);
    cudaFree(e->d_strip_table_be);
    cudaFree(e->d_strip_segment);
    cudaFree(e->d_strip_single);
    cudaFree(e->d_strip_inputs);
    cudaFree(e->d_strip_be_tally);
    cudaFree(e->d_gate_tally);
    cudaFree(e->d_gates);
    cudaFree(e->d_gate_in);
    cudaFree(e->d_gate_part);
    cudaFree(e->d_gate_layer);
    cudaFree(e->d_gate_tally_list);
    cudaFree(e->d_be_tally_nodes);
    cudaFree(e->d_be_tally_idx);
    cudaFree(e->d_event_table);
    cudaFree(e->d_queue);
    cudaFree(e->d_strip_groups);
    cudaFree(e->d_strip_gin);
    cudaFree(e->d_strip_ginfo);
    for (int i = 0; i < 2; ++i) {
        if (e->ev_snap[i]) cudaEventDestroy(e->ev_snap[i]);
    }
    for (cudaEvent_t ev : {e->ev_fork, e->ev_a[0], e->ev_a[1], e->ev_b[0], e->ev_b[1], e->ev_join_a, e->ev_join_b})
        if (ev) cudaEventDestroy(ev);
    for (auto &pe : e->prof_events) {
        cudaEventDestroy(pe.first);
        cudaEventDestroy(pe.second);
    }
    if (e->s_a) cudaStreamDestroy(e->s_a);
    if (e->s_b) cudaStreamDestroy(e->s_b);
    if (e->own_stream && e->stream) cudaStreamDestroy(e->stream);
}

}  // namespace

namespace mcg {
namespace internal {
mcg_status run_staged(mcg_engine *e, uint32_t it_first, uint32_t n_it, uint64_t word_begin, uint64_t count) {
    return run_staged_impl(e, it_first, n_it, word_begin, count);
}
mcg_status fork_staged(mcg_engine *e) { return staged_fork(e); }
mcg_status add_staged(mcg_engine *e, uint64_t *chunk, uint32_t iteration, uint64_t word_begin, uint64_t count,
                      bool more) {
    return staged_chunks(e, chunk, iteration, 1, word_begin, count, more);
}
mcg_status join_staged(mcg_engine *e) { return staged_join(e); }
}  // namespace internal
}  // namespace mcg

mcg_status mcg::internal::create_with_extra(const mcg_graph_desc *graph, const mcg_run_desc *run_in,
                                            const std::function<uint64_t(uint64_t)> &extra_words, mcg_engine **out) {
    mcg::clear_error();
    if (!graph || !out) return mcg::fail(MCG_ERR_INVALID, "graph and out must not be NULL");
    *out = nullptr;
    mcg_run_desc run{};
    if (run_in) run = *run_in;
    if (run.mode > MCG_MODE_FUSED) return mcg::fail(MCG_ERR_INVALID, "unknown mode");
    auto *e = new (std::nothrow) mcg_engine();
    if (!e) return mcg::fail(MCG_ERR_OOM, "host allocation failed");
    const std::string err = mcg::Graph::from_desc(*graph, e->graph);
    if (!err.empty()) {
        delete e;
        return mcg::fail(MCG_ERR_INVALID, err);
    }
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev == 0) {
        cudaGetLastError();
        delete e;
        return mcg::fail(MCG_ERR_NO_DEVICE, "no CUDA device visible");
    }
    if (run.device < 0 || run.device >= n_dev) {
        delete e;
        return mcg::fail(MCG_ERR_INVALID, "device ordinal out of range");
    }
    if (run.mode == MCG_MODE_AUTO) {
        // the launch shape tuned (or cached) for this tree shape on this device
        mcg_tune_choice ch{};
        const mcg_status ts = mcg_tune(graph, &run, run.tune_pass_words, nullptr, nullptr, &ch);
        if (ts != MCG_OK) {
            delete e;
            return ts;
        }
        run.mode = ch.mode;
        run.ctas_per_sm = ch.ctas_per_sm;
        run.layered_max_words = ch.layered_max_words;
        run.smem_slots = 0;
        run.chunk_words = 0;
        run.sampler_blocks_per_sm = 0;
        mcg::clear_error();
    }
    e->device = run.device;
    e->mode = run.mode;
    e->run_desc = run;
    e->layered_max_words = run.layered_max_words;
    mcg_status st = MCG_OK;
    do {
        if (cudaSetDevice(e->device) != cudaSuccess) {
            st = mcg::fail(MCG_ERR_CUDA, "cudaSetDevice failed");
            break;
        }
        if (run.stream) {
            e->stream = (cudaStream_t)run.stream;
        } else {
            if (cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) != cudaSuccess) {
                st = mcg::fail(MCG_ERR_CUDA, "cudaStreamCreate failed");
                break;
            }
            e->own_stream = true;
        }
        const size_t nt = std::max<size_t>(e->graph.tally_nodes.size(), 1);
        // the counters and, behind them, two snapshot slots (mcg_snapshot_tallies)
        if (cudaMalloc((void **)&e->d_tally, 3 * nt * sizeof(unsigned long long)) != cudaSuccess ||
            cudaMemset(e->d_tally, 0, nt * sizeof(unsigned long long)) != cudaSuccess) {
            cudaGetLastError();
            st = mcg::fail(MCG_ERR_OOM, "tally allocation failed");
            break;
        }
        st = build_layered_tables(e);
        if (st != MCG_OK) break;
        // the fused program is compiled here only for the fused mode (on request otherwise)
        if (e->mode == MCG_MODE_FUSED) st = setup_fused(e, run);
        else if (e->mode == MCG_MODE_STAGED) st = setup_staged(e, run, extra_words);
        else if (e->mode == MCG_MODE_STRIP) st = setup_strip(e, run);
    } while (false);
    if (st != MCG_OK) {
        release(e);
        delete e;
        return st;
    }
    *out = e;
    return MCG_OK;
}

extern "C" {

mcg_status mcg_create(const mcg_graph_desc *graph, const mcg_run_desc *run, mcg_engine **out) {
    return mcg::internal::create_with_extra(graph, run, {}, out);
}

mcg_status mcg_engine_launch_shape(mcg_engine *e, uint32_t *mode, uint32_t *ctas_per_sm) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    if (mode) *mode = e->mode;
    if (ctas_per_sm)
        *ctas_per_sm = e->mode == MCG_MODE_STRIP ? e->strip_blocks : e->mode == MCG_MODE_FUSED ? e->ctas_per_sm : 0u;
    return MCG_OK;
}

mcg_status mcg_fused_kernel(mcg_engine *e, uint64_t word_count, uint32_t *tile_threads, uint32_t *segments) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    if (e->mode != MCG_MODE_FUSED) return mcg::fail(MCG_ERR_STATE, "not a fused-mode engine");
    const bool tile = takes_tile(e, std::min<uint64_t>(word_count, e->chunk_words));
    if (tile_threads) *tile_threads = tile ? tile_pass_threads(e, std::min<uint64_t>(word_count, e->chunk_words)) : 0u;
    if (segments) *segments = e->tile ? e->tile_args.n_segments : 0u;
    return MCG_OK;
}

mcg_status mcg_destroy(mcg_engine *e) {
    mcg::clear_error();
    if (!e) return MCG_OK;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    release(e);
    delete e;
    return MCG_OK;
}

mcg_status mcg_run(mcg_engine *e, uint32_t iteration_first, uint32_t n_iterations, uint64_t word_begin,
                   uint64_t word_count) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    if (word_begin + word_count > (1ull << 32) || word_begin + word_count < word_begin)
        return mcg::fail(MCG_ERR_INVALID, "word range exceeds the 32-bit sample counter");
    if ((uint64_t)iteration_first + n_iterations + 1 >= (1ull << 26))
        return mcg::fail(MCG_ERR_INVALID, "iteration exceeds the 26-bit pass counter field");
    if (n_iterations == 0 || word_count == 0) return MCG_OK;
    MCG_CUDA(cudaSetDevice(e->device));
    if (e->mode == MCG_MODE_STAGED) {
        const mcg_status st = run_staged_impl(e, iteration_first, n_iterations, word_begin, word_count);
        if (st != MCG_OK) return st;
    } else if (e->mode == MCG_MODE_STRIP) {
        const mcg_status st = run_strip(e, iteration_first, n_iterations, word_begin, word_count);
        if (st != MCG_OK) return st;
    } else if (e->mode == MCG_MODE_FUSED) {
        for (uint64_t off = 0; off < word_count; off += e->chunk_words) {
            const uint64_t n = std::min<uint64_t>(e->chunk_words, word_count - off);
            const mcg_status st = (takes_tile(e, n) ? launch_tile : launch_fused)(e, iteration_first, n_iterations,
                                                                                  word_begin + off, n);
            if (st != MCG_OK) return st;
        }
    } else {
        const uint64_t nn = std::max<uint64_t>(e->graph.n_nodes(), 1);
        uint64_t W = e->layered_max_words ? e->layered_max_words : std::max<uint64_t>((8ull << 30) / (nn * 8), 1024);
        W = std::min<uint64_t>(W, word_count);
        const uint32_t n_tally = (uint32_t)e->graph.tally_nodes.size();
        for (uint32_t it = 0; it < n_iterations; ++it) {
            for (uint64_t off = 0; off < word_count; off += W) {
                const uint64_t n = std::min<uint64_t>(W, word_count - off);
                mcg_status st = layered_eval(e, iteration_first + it, word_begin + off, n);
                if (st != MCG_OK) return st;
                if (n_tally) {
                    const uint32_t bx = (uint32_t)std::min<uint64_t>((n + 255) / 256, 64);
                    dim3 grid = rows_grid(1, n_tally, 256);
                    grid.x = bx;
                    mcg::dev::k_layer_tally<<<grid, 256, 0, e->stream>>>(e->d_tally_nodes, n_tally, n, n, e->d_buf,
                                                                         e->d_tally, nullptr);
                    ++e->launches;
                    MCG_CUDA(cudaGetLastError());
                }
            }
        }
    }
    e->total_bits += (uint64_t)n_iterations * word_count * 64ull;
    return MCG_OK;
}

mcg_status mcg_synchronize(mcg_engine *e) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    MCG_CUDA(cudaSetDevice(e->device));
    MCG_CUDA(cudaStreamSynchronize(e->stream));
    return MCG_OK;
}

mcg_status mcg_read_tallies(mcg_engine *e, uint64_t *ones, uint64_t *total_bits) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    MCG_CUDA(cudaSetDevice(e->device));
    MCG_CUDA(cudaStreamSynchronize(e->stream));
    if (ones && !e->graph.tally_nodes.empty()) {
        MCG_CUDA(cudaMemcpy(ones, e->d_tally, e->graph.tally_nodes.size() * sizeof(uint64_t), cudaMemcpyDeviceToHost));
    }
    if (total_bits) *total_bits = e->total_bits;
    return MCG_OK;
}

mcg_status mcg_tally_device_ptr(mcg_engine *e, uint64_t **ones_dev) {
    mcg::clear_error();
    if (!e || !ones_dev) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    *ones_dev = reinterpret_cast<uint64_t *>(e->d_tally);
    return MCG_OK;
}

mcg_status mcg_set_tallies(mcg_engine *e, const uint64_t *ones, uint64_t total_bits) {
    mcg::clear_error();
    if (!e || !ones) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    MCG_CUDA(cudaSetDevice(e->device));
    MCG_CUDA(cudaStreamSynchronize(e->stream));
    if (!e->graph.tally_nodes.empty())
        MCG_CUDA(cudaMemcpy(e->d_tally, ones, e->graph.tally_nodes.size() * sizeof(uint64_t), cudaMemcpyHostToDevice));
    e->total_bits = total_bits;
    return MCG_OK;
}

mcg_status mcg_snapshot_tallies(mcg_engine *e, uint32_t slot) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    if (slot > 1) return mcg::fail(MCG_ERR_INVALID, "slot must be 0 or 1");
    MCG_CUDA(cudaSetDevice(e->device));
    const size_t n = std::max<size_t>(e->graph.tally_nodes.size(), 1);
    if (!e->ev_snap[slot]) MCG_CUDA(cudaEventCreateWithFlags(&e->ev_snap[slot], cudaEventDisableTiming));
    // device-side copy into the slot behind the counters: no host buffer to pin
    MCG_CUDA(cudaMemcpyAsync(e->d_tally + (1 + slot) * n, e->d_tally, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice,
                             e->stream));
    MCG_CUDA(cudaEventRecord(e->ev_snap[slot], e->stream));
    e->snap_total[slot] = e->total_bits;
    return MCG_OK;
}

mcg_status mcg_snapshot_read(mcg_engine *e, uint32_t slot, uint64_t *ones, uint64_t *total_bits) {
    mcg::clear_error();
    if (!e || !ones || !total_bits) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (slot > 1 || !e->ev_snap[slot]) return mcg::fail(MCG_ERR_STATE, "no snapshot in this slot");
    MCG_CUDA(cudaSetDevice(e->device));
    MCG_CUDA(cudaEventSynchronize(e->ev_snap[slot]));
    // the slot is not written by the passes behind the snapshot: this copy does not wait for them
    const size_t n = std::max<size_t>(e->graph.tally_nodes.size(), 1);
    if (!e->graph.tally_nodes.empty())
        MCG_CUDA(cudaMemcpy(ones, e->d_tally + (1 + slot) * n, e->graph.tally_nodes.size() * sizeof(uint64_t),
                            cudaMemcpyDeviceToHost));
    *total_bits = e->snap_total[slot];
    return MCG_OK;
}

mcg_status mcg_reset_tallies(mcg_engine *e) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    MCG_CUDA(cudaSetDevice(e->device));
    MCG_CUDA(cudaMemsetAsync(e->d_tally, 0, std::max<size_t>(e->graph.tally_nodes.size(), 1) * sizeof(uint64_t),
                             e->stream));
    e->total_bits = 0;
    return MCG_OK;
}

mcg_status mcg_dump_words(mcg_engine *e, uint32_t iteration, uint64_t word_begin, uint64_t n_words, uint64_t *out) {
    mcg::clear_error();
    if (!e || !out) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (word_begin + n_words > (1ull << 32)) return mcg::fail(MCG_ERR_INVALID, "word range exceeds the sample counter");
    if (n_words == 0) return MCG_OK;
    MCG_CUDA(cudaSetDevice(e->device));
    mcg_status st = layered_eval(e, iteration, word_begin, n_words);
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaStreamSynchronize(e->stream));
    MCG_CUDA(cudaMemcpy(out, e->d_buf, (size_t)e->graph.n_nodes() * n_words * sizeof(uint64_t), cudaMemcpyDeviceToHost));
    return MCG_OK;
}

mcg_status mcg_program_info_get(mcg_engine *e, mcg_program_info *info) {
    mcg::clear_error();
    if (!e || !info) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (!e->prog_compiled) {
        MCG_CUDA(cudaSetDevice(e->device));
        mcg_run_desc rd = e->run_desc;
        rd.ctas_per_sm = 0;  // the other modes' value means something else
        const mcg_status st = compile_fused(e, rd);
        if (st != MCG_OK) return st;
    }
    info->n_ops = e->prog.ops.size();
    info->smem_slots = e->prog.smem_slots;
    info->global_slots = e->prog.global_slots;
    info->max_live = e->prog.max_live;
    info->block_threads = e->nt;
    info->grid_ctas = e->grid;
    info->scratch_bytes = (uint64_t)e->prog.global_slots * e->scratch_stride * sizeof(uint64_t);
    info->smem_bytes = e->smem_bytes;
    info->n_inline_be = e->prog.n_inline_be;
    return MCG_OK;
}

mcg_status mcg_launch_count(mcg_engine *e, uint64_t *launches) {
    mcg::clear_error();
    if (!e || !launches) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    *launches = e->launches;
    return MCG_OK;
}

mcg_status mcg_time_runs(mcg_engine *e, uint32_t iteration_first, uint64_t word_begin, uint64_t word_count,
                         uint32_t repeats, double *ms_per_run) {
    mcg::clear_error();
    if (!e || !ms_per_run || repeats == 0) return mcg::fail(MCG_ERR_INVALID, "bad argument");
    MCG_CUDA(cudaSetDevice(e->device));
    cudaEvent_t a, b;
    MCG_CUDA(cudaEventCreate(&a));
    MCG_CUDA(cudaEventCreate(&b));
    MCG_CUDA(cudaEventRecord(a, e->stream));
    for (uint32_t r = 0; r < repeats; ++r) {
        const mcg_status st = mcg_run(e, iteration_first + r, 1, word_begin, word_count);
        if (st != MCG_OK) {
            cudaEventDestroy(a);
            cudaEventDestroy(b);
            return st;
        }
    }
    MCG_CUDA(cudaEventRecord(b, e->stream));
    MCG_CUDA(cudaEventSynchronize(b));
    float ms = 0;
    MCG_CUDA(cudaEventElapsedTime(&ms, a, b));
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    *ms_per_run = (double)ms / repeats;
    return MCG_OK;
}

mcg_status mcg_sampler_peak(int32_t device, uint64_t n_events, uint64_t n_words, uint32_t repeats,
                            double *words_per_second) {
    mcg::clear_error();
    if (!words_per_second || n_events == 0 || n_words == 0 || repeats == 0 || n_events > 0xFFFFFFFFull ||
        n_words > 0xFFFFFFFFull)
        return mcg::fail(MCG_ERR_INVALID, "bad argument");
    MCG_CUDA(cudaSetDevice(device));
    uint64_t *sink = nullptr;
    uint2 *table = nullptr;
    MCG_CUDA(cudaMalloc((void **)&sink, n_words * sizeof(uint64_t)));
    if (cudaMalloc((void **)&table, n_events * mcg::dev::kEventTableStride * sizeof(uint2)) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(sink);
        return mcg::fail(MCG_ERR_OOM, "sampler table allocation failed");
    }
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const uint64_t nt = n_events * mcg::dev::kEventTableStride;
    mcg::dev::k_peak_table<<<(uint32_t)((nt + 255) / 256), 256>>>((uint32_t)n_events, 2u << 6, table);
    const uint32_t blocks = (uint32_t)((n_words + 255) / 256);
    // warm-up
    mcg::dev::k_sampler_peak<kPackForm><<<blocks, 256>>>((uint32_t)n_events, n_words, table, sink);
    cudaEventRecord(a);
    for (uint32_t r = 0; r < repeats; ++r)
        mcg::dev::k_sampler_peak<kPackForm><<<blocks, 256>>>((uint32_t)n_events, n_words, table, sink);
    cudaEventRecord(b);
    cudaError_t err = cudaEventSynchronize(b);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(table);
    cudaFree(sink);
    if (err != cudaSuccess) return mcg::fail(MCG_ERR_CUDA, cudaGetErrorString(err));
    *words_per_second = (double)n_events * (double)n_words * repeats / (ms * 1e-3);
    return MCG_OK;
}

mcg_status mcg_sampler_peak_shared(int32_t device, uint64_t n_events, uint64_t n_words, uint32_t repeats,
                                   uint32_t instances, double *instance_words_per_second) {
    mcg::clear_error();
    if (!instance_words_per_second || n_events == 0 || n_words == 0 || repeats == 0 || n_events > 0xFFFFFFFFull ||
        n_words > 0xFFFFFFFFull || (instances != 1 && instances != 4))
        return mcg::fail(MCG_ERR_INVALID, "bad argument");
    MCG_CUDA(cudaSetDevice(device));
    uint64_t *sink = nullptr;
    MCG_CUDA(cudaMalloc((void **)&sink, n_words * sizeof(uint64_t)));
    auto launch = [&] {
        const uint32_t blocks = (uint32_t)((n_words + 255) / 256);
        if (instances == 4)
            mcg::dev::k_sampler_peak_shared<kPackForm, 4><<<blocks, 256>>>((uint32_t)n_events, n_words, sink);
        else
            mcg::dev::k_sampler_peak_shared<kPackForm, 1><<<blocks, 256>>>((uint32_t)n_events, n_words, sink);
    };
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    launch();  // warm-up
    cudaEventRecord(a);
    for (uint32_t r = 0; r < repeats; ++r) launch();
    cudaEventRecord(b);
    cudaError_t err = cudaEventSynchronize(b);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(sink);
    if (err != cudaSuccess) return mcg::fail(MCG_ERR_CUDA, cudaGetErrorString(err));
    *instance_words_per_second = (double)n_events * (double)n_words * instances * repeats / (ms * 1e-3);
    return MCG_OK;
}

mcg_status mcg_profile_sampler(mcg_engine *e, int32_t enable) {
    mcg::clear_error();
    if (!e) return mcg::fail(MCG_ERR_INVALID, "engine is NULL");
    e->profile_a = enable != 0;
    e->prof_used = 0;
    return MCG_OK;
}

mcg_status mcg_profile_sampler_read(mcg_engine *e, uint64_t *launches, double *total_ms) {
    mcg::clear_error();
    if (!e || !launches || !total_ms) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    MCG_CUDA(cudaSetDevice(e->device));
    MCG_CUDA(cudaStreamSynchronize(e->stream));
    double sum = 0;
    for (size_t i = 0; i < e->prof_used; ++i) {
        float ms = 0;
        MCG_CUDA(cudaEventElapsedTime(&ms, e->prof_events[i].first, e->prof_events[i].second));
        sum += ms;
    }
    *launches = e->prof_used;
    *total_ms = sum;
    return MCG_OK;
}

const char *mcg_version(void) { return "mcg 0.2 (sm_100a)"; }

}  // extern "C"
