// batch.cu -- batched instances in one persistent, graph-captured launch
// (include/mcg_batch.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <string>
#include <vector>

#include "batch_tile.cuh"
#include "error.hpp"
#include "graph.hpp"
#include "kernels.cuh"
#include "mcg_batch.h"
#include "program.hpp"
#include "smem_limit.hpp"
#include "tile_cost.hpp"
#include "tile_plan.hpp"

namespace {

constexpr int kThreads = 256;
constexpr int kPackForm = 1;
// Instances of one tree that differ only in thresholds (uncertainty draws)
// share their Philox calls kShare at a time (k_fused_batch_k) unless a tree
// has an ATLEAST gate of more than kShareAtleastMaxIn inputs (the four-wide
// interpreter counts ATLEAST inputs in four bit slices per instance).
constexpr uint32_t kShare = 4;
constexpr uint32_t kShareAtleastMaxIn = 15;

#define MCG_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t err_ = (call);                                                              \
        if (err_ != cudaSuccess) {                                                              \
            cudaGetLastError(); /* reported here, and not by the next launch's check */         \
            return mcg::fail(err_ == cudaErrorMemoryAllocation ? MCG_ERR_OOM : MCG_ERR_CUDA,    \
                             std::string(#call) + ": " + cudaGetErrorString(err_));             \
        }                                                                                       \
    } while (0)

using BatchKernel = void (*)(mcg::dev::BatchArgs);

BatchKernel batch_kernel(uint32_t ctas_per_sm, uint32_t share, bool atleast) {
    if (share == kShare && atleast) {
        switch (ctas_per_sm) {
            case 2: return mcg::dev::k_fused_batch_k<kThreads, 2, kPackForm, kShare, true>;
            case 3: return mcg::dev::k_fused_batch_k<kThreads, 3, kPackForm, kShare, true>;
            default: return mcg::dev::k_fused_batch_k<kThreads, 4, kPackForm, kShare, true>;
        }
    }
    if (share == kShare) {
        switch (ctas_per_sm) {
            case 2: return mcg::dev::k_fused_batch_k<kThreads, 2, kPackForm, kShare, false>;
            case 3: return mcg::dev::k_fused_batch_k<kThreads, 3, kPackForm, kShare, false>;
            default: return mcg::dev::k_fused_batch_k<kThreads, 4, kPackForm, kShare, false>;
        }
    }
    switch (ctas_per_sm) {
        case 2: return mcg::dev::k_fused_batch<kThreads, 2, kPackForm>;
        case 3: return mcg::dev::k_fused_batch<kThreads, 3, kPackForm>;
        default: return mcg::dev::k_fused_batch<kThreads, 4, kPackForm>;
    }
}

template <typename T>
cudaError_t ensure(T **p, uint64_t &cap, uint64_t n) {
    if (n <= cap && *p) return cudaSuccess;
    if (*p) cudaFree(*p);
    *p = nullptr;
    cap = 0;
    cudaError_t e = cudaMalloc((void **)p, std::max<uint64_t>(n, 1) * sizeof(T));
    if (e == cudaSuccess) cap = std::max<uint64_t>(n, 1);
    return e;
}

}  // namespace

struct mcg_batch {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    uint32_t ctas_per_sm = 4;
    uint32_t share = 1;  // instances per work item (kShare or 1)
    bool atleast = false; // the shared kernel needs its ATLEAST counters
    std::vector<mcg::Graph> trees;
    std::vector<uint32_t> tree_op_offset;
    uint32_t smem_slots = 0, max_global = 0, grid = 0, smem_bytes = 0;
    uint64_t total_ops = 0;
    uint4 *d_ops = nullptr;
    uint32_t *d_tree_off = nullptr;
    uint64_t *d_scratch = nullptr;       // of the interpreter (interpreter_scratch)
    uint64_t scratch_stride = 0;
    unsigned int *d_queue = nullptr;
    // per-run buffers
    uint32_t *d_inst_tree = nullptr;
    uint64_t cap_inst = 0, cap_inst2 = 0, cap_thr = 0, cap_ones = 0;
    uint64_t *d_thr_off = nullptr;
    uint64_t *d_thr = nullptr;
    unsigned long long *d_ones = nullptr;
    uint32_t *d_group_first = nullptr, *d_group_size = nullptr;
    uint64_t cap_grp = 0, cap_grp2 = 0;
    uint32_t n_groups = 0;
    // tiles (the default shape): all trees' tables, and per run the groups and their event records
    bool tile = false;
    unsigned char *d_tile_rows = nullptr;
    uint32_t tile_blocks = 0;
    std::vector<mcg::dev::BatchTileTree> tile_trees;
    std::vector<mcg::BatchTreeCost> cost;  // per tree
    mcg::dev::BatchTileArgs tile_args{};
    std::vector<void *> tile_tables;
    const uint2 *d_event = nullptr;
    const uint32_t *d_event_node = nullptr, *d_event_off = nullptr;
    mcg::dev::BatchTileGroup *d_tile_groups = nullptr;
    uint4 *d_tile_recs = nullptr;
    uint64_t cap_tile_groups = 0, cap_tile_recs = 0;
    uint32_t n_tile_groups = 0, tile_most_events = 0;
    // graph
    cudaGraphExec_t graph = nullptr;
    bool g_tile = false;
    uint32_t g_instances = 0, g_iteration = 0;
    uint64_t g_words = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    uint64_t launches = 0;
    double last_ms = 0.0;
};

namespace {

void drop_graph(mcg_batch *b) {
    if (b->graph) cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
}

// Gives all of the tile kernel's memory back.
void drop_tile(mcg_batch *b) {
    drop_graph(b);
    for (void *p : b->tile_tables) cudaFree(p);
    b->tile_tables.clear();
    cudaFree(b->d_tile_groups);
    cudaFree(b->d_tile_recs);
    cudaFree(b->d_tile_rows);
    b->d_tile_groups = nullptr;
    b->d_tile_recs = nullptr;
    b->d_tile_rows = nullptr;
    b->cap_tile_groups = b->cap_tile_recs = 0;
    b->tile = false;
}

// A per-run buffer of n elements; the captured graph goes with a buffer it reads.
template <typename T>
cudaError_t grow(mcg_batch *b, T **p, uint64_t &cap, uint64_t n) {
    if (n <= cap && *p) return cudaSuccess;
    drop_graph(b);
    return ensure(p, cap, n);
}

void release(mcg_batch *b) {
    drop_tile(b);
    cudaFree(b->d_ops);
    cudaFree(b->d_tree_off);
    cudaFree(b->d_scratch);
    cudaFree(b->d_queue);
    cudaFree(b->d_inst_tree);
    cudaFree(b->d_thr_off);
    cudaFree(b->d_thr);
    cudaFree(b->d_ones);
    cudaFree(b->d_group_first);
    cudaFree(b->d_group_size);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
}

template <typename T>
mcg_status upload_table(mcg_batch *b, const T **dptr, const std::vector<T> &v) {
    void *p = nullptr;
    MCG_CUDA(cudaMalloc(&p, std::max<size_t>(v.size(), 1) * sizeof(T)));
    b->tile_tables.push_back(p);
    if (!v.empty()) MCG_CUDA(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    *dptr = (const T *)p;
    return MCG_OK;
}

// The tile kernel's scratch: a row of 4 KB per slot of the largest tree for each
// of the two blocks of every SM, held as long as the batch (84 MB for trees of
// 60 events, 0.4 GB for 2,000, 1.5 GB for the 5,000-event tree; the interpreter
// 26 MB, 1.0 and 5.3 GB).  Above this much the interpreter takes the batch.
constexpr uint64_t kTileScratchMost = 16ull << 30;

// Tables of k_batch_tile; leaves b->tile false where the interpreter has to
// take the batch (rows too large).  Out of memory is the caller's to handle.
mcg_status setup_tile(mcg_batch *b, const mcg::DeviceShape &prop) {
    using namespace mcg::dev;
    std::vector<uint4> gates;
    std::vector<uint32_t> in, layer, event_node, event_off, event_slot;
    std::vector<uint2> event, be_tally, segment;
    uint64_t most_slots = 0;
    for (const auto &g : b->trees) {
        const mcg::SegmentPlan plan = mcg::plan_segments(g, mcg::kSegmentEvents, true);
        const mcg::TilePlan &t = plan.tile;
        if (!t.fits || in.size() + t.in.size() > 0xFFFFFFFFull) return MCG_OK;
        most_slots = std::max<uint64_t>(most_slots, plan.slots + 1ull);
        if (most_slots * kTileRow > 0xFFFFFFFFull) return MCG_OK;
        BatchTileTree x{};
        x.n_be = (uint32_t)t.event.size();
        x.n_segments = (uint32_t)plan.segment.size();
        x.seg_off = (uint32_t)segment.size();
        x.event_off = (uint32_t)event_slot.size();
        x.gate_off = (uint32_t)gates.size();
        x.layer_off = (uint32_t)layer.size();
        x.in_off = (uint32_t)in.size();
        x.be_tally_off = (uint32_t)be_tally.size();
        for (const uint2 &s : t.be_tally) {  // {slot, tallies}: the slot's tallies follow each other
            if (be_tally.size() > x.be_tally_off && be_tally.back().x == s.x + 1u) ++be_tally.back().y;
            else be_tally.push_back(make_uint2(s.x + 1u, 1u));
        }
        x.n_be_tally = (uint32_t)be_tally.size() - x.be_tally_off;
        gates.insert(gates.end(), t.gates.begin(), t.gates.end());
        for (size_t i = 0; i < t.gates.size(); ++i) gates[x.gate_off + i].w = plan.gate_slot[i] + 1u;
        for (uint32_t v : plan.event_slot) event_slot.push_back(v + 1u);
        segment.insert(segment.end(), plan.segment.begin(), plan.segment.end());
        layer.insert(layer.end(), t.layer.begin(), t.layer.end());
        for (uint32_t rec : t.in) in.push_back(mcg::TilePlan::byte_record(rec, kTileRow, 1, 0));
        event_off.push_back((uint32_t)event.size());
        for (uint32_t e : t.event) {
            event.push_back(make_uint2((uint32_t)g.be_pdag_idx[e] + 1u, g.be_event_idx[e] + 1u));
            event_node.push_back(e);
        }
        b->tile_most_events = std::max(b->tile_most_events, x.n_be);
        b->tile_trees.push_back(x);
        const size_t k = b->cost.size(), ops_end = k + 1 < b->trees.size() ? b->tree_op_offset[k + 1] : b->total_ops;
        b->cost.emplace_back(t.layer, t.gates, t.event.size(), plan.segment.size(), t.in.size(),
                             ops_end - b->tree_op_offset[k]);
    }
    const uint64_t stride = most_slots * kTileRow;
    const uint64_t blocks = (uint64_t)prop.multiProcessorCount * kBatchTileBlocks;
    if (stride * blocks > kTileScratchMost) return MCG_OK;
    MCG_CUDA(cudaMalloc((void **)&b->d_tile_rows, stride * blocks));
    b->tile_blocks = (uint32_t)blocks;
    BatchTileArgs &a = b->tile_args;
    mcg_status st;
    if ((st = upload_table(b, &a.trees, b->tile_trees)) != MCG_OK || (st = upload_table(b, &a.gates, gates)) != MCG_OK ||
        (st = upload_table(b, &a.in, in)) != MCG_OK || (st = upload_table(b, &a.layer, layer)) != MCG_OK ||
        (st = upload_table(b, &a.be_tally, be_tally)) != MCG_OK || (st = upload_table(b, &a.segment, segment)) != MCG_OK ||
        (st = upload_table(b, &a.event_slot, event_slot)) != MCG_OK || (st = upload_table(b, &b->d_event, event)) != MCG_OK ||
        (st = upload_table(b, &b->d_event_node, event_node)) != MCG_OK ||
        (st = upload_table(b, &b->d_event_off, event_off)) != MCG_OK)
        return st;
    st = mcg::set_smem_limit(k_batch_tile, (kBatchTileThreads / 32) * kBatchTileOut);
    if (st != MCG_OK) return st;
    a.scratch = b->d_tile_rows;
    a.scratch_stride = stride;
    b->tile = true;
    return MCG_OK;
}

// The interpreter's scratch, from its first run on.
mcg_status interpreter_scratch(mcg_batch *b) {
    if (!b->max_global || b->d_scratch) return MCG_OK;
    void *p = nullptr;
    MCG_CUDA(cudaMalloc(&p, (size_t)b->max_global * b->share * b->scratch_stride * sizeof(uint64_t)));
    b->d_scratch = static_cast<uint64_t *>(p);
    return MCG_OK;
}

// From here on the interpreter runs the batch: it needs less memory where few
// values are live, and no records per group.
mcg_status use_interpreter(mcg_batch *b) {
    cudaGetLastError();
    mcg::clear_error();
    drop_tile(b);
    return interpreter_scratch(b);
}

// Whether the interpreter is the faster one for a run (tile_cost.hpp).
bool interpreter_is_faster(const mcg_batch *b, uint32_t n_inst, const uint32_t *inst_tree, uint64_t words) {
    const uint64_t tiles = (words + mcg::dev::kTileLanes - 1) / mcg::dev::kTileLanes;
    const uint64_t slabs = (words + kThreads - 1) / kThreads, sms = b->tile_blocks / mcg::dev::kBatchTileBlocks;
    uint64_t tile = 0, tile_least = 0, interp = 0, interp_least = 0;
    for (uint32_t i = 0; i < n_inst;) {
        const mcg::BatchTreeCost &c = b->cost[inst_tree[i]];
        uint32_t n = 1;
        while (i + n < n_inst && inst_tree[i + n] == inst_tree[i]) ++n;
        i += n;
        interp += (n + b->share - 1) / b->share * slabs * (kThreads / 32) * c.interpreter(b->share);
        interp_least = std::max(interp_least, c.interpreter_alone(b->share));
        for (uint32_t left = n; left;) {
            const uint32_t size = std::min(left, mcg::dev::kTileInstances);
            left -= size;
            tile += tiles * c.tile(size);
            tile_least = std::max(tile_least, c.tile(size) / 2);  // alone on its SM
        }
    }
    return std::max(interp / sms, interp_least) < std::max(tile / b->tile_blocks, tile_least);
}

mcg_status setup(mcg_batch *b, const mcg_run_desc &run) {
    MCG_CUDA(cudaSetDevice(b->device));
    mcg::DeviceShape prop;
    MCG_CUDA(mcg::device_shape(&prop, b->device));
    b->ctas_per_sm = run.ctas_per_sm ? run.ctas_per_sm : 4u;
    if (b->ctas_per_sm < 2 || b->ctas_per_sm > 4) return mcg::fail(MCG_ERR_INVALID, "ctas_per_sm must be 2..4");
    b->share = kShare;
    for (const auto &g : b->trees)
        for (size_t i = 0; i < g.gate_op.size(); ++i)
            if (g.gate_op[i] == MCG_ATLEAST) {
                if (g.gate_in_count[i] <= kShareAtleastMaxIn) b->atleast = true;
                else b->share = 1;
            }
    // What one of ctas_per_sm resident CTAs may take: the SM's shared memory
    // shared out, less the per-block reservation and the kernel's static
    // shared memory (its work-item slot), so that all of them stay resident.
    cudaFuncAttributes fa{};
    MCG_CUDA(cudaFuncGetAttributes(&fa, reinterpret_cast<const void *>(batch_kernel(b->ctas_per_sm, b->share,
                                                                                     b->atleast))));
    const size_t cap = std::min<size_t>(prop.sharedMemPerBlockOptin,
                                        prop.sharedMemPerMultiprocessor / b->ctas_per_sm -
                                            prop.reservedSharedMemPerBlock) -
                       fa.sharedSizeBytes;
    // a slot holds one word per instance of a work item
    uint32_t budget = (uint32_t)(cap / (kThreads * sizeof(uint64_t) * b->share));
    if (run.smem_slots == MCG_SMEM_SLOTS_NONE) budget = 0;
    else if (run.smem_slots) budget = std::min(budget, run.smem_slots);
    std::vector<mcg::Op> all;
    for (const auto &g : b->trees) {
        mcg::Program prog;
        const std::string err = mcg::compile_program(g, budget, prog, true);
        if (!err.empty()) return mcg::fail(MCG_ERR_INVALID, err);
        b->tree_op_offset.push_back((uint32_t)all.size());
        all.insert(all.end(), prog.ops.begin(), prog.ops.end());
        b->smem_slots = std::max(b->smem_slots, prog.smem_slots);
        b->max_global = std::max(b->max_global, prog.global_slots);
    }
    if (all.size() >= 0xFFFFFFFFull) return mcg::fail(MCG_ERR_INVALID, "programs too large");
    b->total_ops = all.size();
    b->smem_bytes = b->smem_slots * b->share * kThreads * (uint32_t)sizeof(uint64_t);
    b->grid = (uint32_t)prop.multiProcessorCount * b->ctas_per_sm;
    b->scratch_stride = (uint64_t)b->grid * kThreads;
    MCG_CUDA(cudaMalloc((void **)&b->d_ops, all.size() * sizeof(mcg::Op)));
    MCG_CUDA(cudaMemcpy(b->d_ops, all.data(), all.size() * sizeof(mcg::Op), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMalloc((void **)&b->d_tree_off, b->tree_op_offset.size() * sizeof(uint32_t)));
    MCG_CUDA(cudaMemcpy(b->d_tree_off, b->tree_op_offset.data(), b->tree_op_offset.size() * sizeof(uint32_t),
                        cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMalloc((void **)&b->d_queue, sizeof(unsigned long long)));
    mcg_status ts = MCG_OK;
    if (!run.smem_slots && !run.ctas_per_sm) ts = setup_tile(b, prop);  // the default shape
    if (ts == MCG_ERR_OOM || (ts == MCG_OK && !b->tile)) ts = use_interpreter(b);
    if (ts != MCG_OK) return ts;
    const mcg_status lim = mcg::set_smem_limit(batch_kernel(b->ctas_per_sm, b->share, b->atleast), b->smem_bytes);
    if (lim != MCG_OK) return lim;
    if (run.stream) {
        b->stream = (cudaStream_t)run.stream;
    } else {
        MCG_CUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
        b->own_stream = true;
    }
    MCG_CUDA(cudaEventCreate(&b->ev0));
    MCG_CUDA(cudaEventCreate(&b->ev1));
    return MCG_OK;
}

// Captures [zero queue, zero ones, persistent launch] for the current shapes.
mcg_status capture(mcg_batch *b, bool tile, uint32_t n_inst, uint32_t iteration, uint64_t words) {
    drop_graph(b);
    mcg::dev::BatchArgs a;
    a.ops = b->d_ops;
    a.tree_op_offset = b->d_tree_off;
    a.inst_tree = b->d_inst_tree;
    a.inst_thr_offset = b->d_thr_off;
    a.thr = b->d_thr;
    a.n_instances = n_inst;
    a.slabs_per_instance = (uint32_t)((words + kThreads - 1) / kThreads);
    a.words_per_instance = words;
    a.iteration = iteration;
    a.smem_slots = b->smem_slots;
    a.scratch = b->d_scratch;
    a.scratch_stride = b->scratch_stride;
    a.queue = b->d_queue;
    a.inst_ones = b->d_ones;
    a.group_first = b->d_group_first;
    a.group_size = b->d_group_size;
    a.n_groups = b->n_groups;
    cudaGraph_t g = nullptr;
    MCG_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(b->d_queue, 0, sizeof(unsigned long long), b->stream);
    cudaMemsetAsync(b->d_ones, 0, (size_t)n_inst * sizeof(unsigned long long), b->stream);
    if (tile) {
        using namespace mcg::dev;
        BatchTileArgs t = b->tile_args;
        t.groups = b->d_tile_groups;
        t.recs = b->d_tile_recs;
        t.words = words;
        t.tiles = (words + kTileLanes - 1) / kTileLanes;
        t.items = t.tiles * b->n_tile_groups;
        t.iteration = iteration;
        t.queue = reinterpret_cast<unsigned long long *>(b->d_queue);
        t.ones = b->d_ones;
        const dim3 grid(b->n_tile_groups, std::min(64u, std::max(1u, (b->tile_most_events + 255u) / 256u)));
        k_batch_records<<<grid, 256, 0, b->stream>>>(b->d_tile_groups, b->d_event, b->d_event_node, b->d_event_off,
                                                     t.trees, b->d_thr_off, b->d_thr, b->d_tile_recs);
        k_batch_tile<<<(uint32_t)std::min<uint64_t>(b->tile_blocks, t.items), kBatchTileThreads,
                       (kBatchTileThreads / 32) * kBatchTileOut, b->stream>>>(t);
    } else {
        batch_kernel(b->ctas_per_sm, b->share, b->atleast)<<<b->grid, kThreads, b->smem_bytes, b->stream>>>(a);
    }
    const cudaError_t launch_err = cudaGetLastError();
    const cudaError_t end_err = cudaStreamEndCapture(b->stream, &g);
    if (launch_err != cudaSuccess || end_err != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return mcg::fail(MCG_ERR_CUDA, std::string("batch capture: ") +
                                           cudaGetErrorString(launch_err != cudaSuccess ? launch_err : end_err));
    }
    const cudaError_t inst_err = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (inst_err != cudaSuccess) return mcg::fail(MCG_ERR_CUDA, cudaGetErrorString(inst_err));
    b->g_tile = tile;
    b->g_instances = n_inst;
    b->g_iteration = iteration;
    b->g_words = words;
    return MCG_OK;
}

// A validated run in tiles or by the interpreter, from its groups to its results
// on the host.
mcg_status run_instances(mcg_batch *b, bool tile, uint32_t n_inst, const uint32_t *inst_tree, const uint64_t *thr_offset,
                         const uint64_t *thresholds, uint64_t n_thr, uint32_t iteration, uint64_t words,
                         uint64_t *ones) {
    // groups of up to `share` consecutive instances of one tree (up to 16 in tiles)
    const uint32_t most = tile ? mcg::dev::kTileInstances : b->share;
    std::vector<uint32_t> gfirst, gsize;
    for (uint32_t i = 0; i < n_inst;) {
        uint32_t n = 1;
        while (n < most && i + n < n_inst && inst_tree[i + n] == inst_tree[i]) ++n;
        gfirst.push_back(i);
        gsize.push_back(n);
        i += n;
    }
    MCG_CUDA(grow(b, &b->d_inst_tree, b->cap_inst, n_inst));
    MCG_CUDA(grow(b, &b->d_thr_off, b->cap_inst2, n_inst));
    MCG_CUDA(grow(b, &b->d_thr, b->cap_thr, n_thr));
    MCG_CUDA(grow(b, &b->d_ones, b->cap_ones, n_inst));
    MCG_CUDA(grow(b, &b->d_group_first, b->cap_grp, gfirst.size()));
    MCG_CUDA(grow(b, &b->d_group_size, b->cap_grp2, gsize.size()));
    if (b->n_groups != (uint32_t)gfirst.size()) drop_graph(b);
    b->n_groups = (uint32_t)gfirst.size();
    std::vector<mcg::dev::BatchTileGroup> groups;
    if (tile) {
        // the costliest first (events, and about as much again for every 20
        // instances), so that the last items of the queue are small
        std::vector<uint32_t> order(gfirst.size());
        for (uint32_t i = 0; i < (uint32_t)order.size(); ++i) order[i] = i;
        auto cost = [&](uint32_t i) { return (uint64_t)b->tile_trees[inst_tree[gfirst[i]]].n_be * (20u + gsize[i]); };
        std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return cost(x) > cost(y); });
        uint64_t recs = 0;
        for (uint32_t i : order) {
            const uint32_t t = inst_tree[gfirst[i]];
            groups.push_back({t, gfirst[i], gsize[i], 0u, recs});
            recs += b->tile_trees[t].n_be;
        }
        MCG_CUDA(grow(b, &b->d_tile_groups, b->cap_tile_groups, groups.size()));
        MCG_CUDA(grow(b, &b->d_tile_recs, b->cap_tile_recs, std::max<uint64_t>(recs, 1) * mcg::dev::kTileRec));
        b->n_tile_groups = (uint32_t)groups.size();
        MCG_CUDA(cudaMemcpyAsync(b->d_tile_groups, groups.data(), groups.size() * sizeof(groups[0]),
                                 cudaMemcpyHostToDevice, b->stream));
    }
    MCG_CUDA(cudaMemcpyAsync(b->d_group_first, gfirst.data(), gfirst.size() * sizeof(uint32_t),
                             cudaMemcpyHostToDevice, b->stream));
    MCG_CUDA(cudaMemcpyAsync(b->d_group_size, gsize.data(), gsize.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                             b->stream));
    MCG_CUDA(cudaMemcpyAsync(b->d_inst_tree, inst_tree, n_inst * sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream));
    MCG_CUDA(cudaMemcpyAsync(b->d_thr_off, thr_offset, n_inst * sizeof(uint64_t), cudaMemcpyHostToDevice, b->stream));
    MCG_CUDA(cudaMemcpyAsync(b->d_thr, thresholds, n_thr * sizeof(uint64_t), cudaMemcpyHostToDevice, b->stream));
    if (!b->graph || b->g_tile != tile || b->g_instances != n_inst || b->g_iteration != iteration || b->g_words != words) {
        const mcg_status st = capture(b, tile, n_inst, iteration, words);
        if (st != MCG_OK) return st;
    }
    MCG_CUDA(cudaEventRecord(b->ev0, b->stream));
    MCG_CUDA(cudaGraphLaunch(b->graph, b->stream));
    MCG_CUDA(cudaEventRecord(b->ev1, b->stream));
    ++b->launches;
    MCG_CUDA(cudaMemcpyAsync(ones, b->d_ones, n_inst * sizeof(uint64_t), cudaMemcpyDeviceToHost, b->stream));
    MCG_CUDA(cudaStreamSynchronize(b->stream));
    float ms = 0;
    MCG_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
    b->last_ms = ms;
    return MCG_OK;
}

}  // namespace

extern "C" {

mcg_status mcg_batch_create(const mcg_graph_desc *trees, uint32_t n_trees, const mcg_run_desc *run_in,
                            mcg_batch **out) {
    mcg::clear_error();
    if (!trees || !out || n_trees == 0) return mcg::fail(MCG_ERR_INVALID, "trees and out must be given");
    *out = nullptr;
    mcg_run_desc run{};
    if (run_in) run = *run_in;
    auto b = std::make_unique<mcg_batch>();
    for (uint32_t t = 0; t < n_trees; ++t) {
        mcg::Graph g;
        const std::string err = mcg::Graph::from_desc(trees[t], g);
        if (!err.empty()) return mcg::fail(MCG_ERR_INVALID, "tree " + std::to_string(t) + ": " + err);
        if (g.tally_nodes.empty()) return mcg::fail(MCG_ERR_INVALID, "tree " + std::to_string(t) + ": no tally node");
        b->trees.push_back(std::move(g));
    }
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev == 0) {
        cudaGetLastError();
        return mcg::fail(MCG_ERR_NO_DEVICE, "no CUDA device visible");
    }
    b->device = run.device;
    const mcg_status st = setup(b.get(), run);
    if (st != MCG_OK) {
        release(b.get());
        return st;
    }
    *out = b.release();
    return MCG_OK;
}

mcg_status mcg_batch_destroy(mcg_batch *b) {
    mcg::clear_error();
    if (!b) return MCG_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    release(b);
    delete b;
    return MCG_OK;
}

mcg_status mcg_batch_run(mcg_batch *b, uint32_t n_inst, const uint32_t *inst_tree, const uint64_t *thr_offset,
                         const uint64_t *thresholds, uint64_t n_thr, uint32_t iteration, uint64_t words,
                         uint64_t *ones) {
    mcg::clear_error();
    if (!b || !inst_tree || !thr_offset || !thresholds || !ones) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (n_inst == 0 || words == 0) return MCG_OK;
    if (words > 0xFFFFFFFFull) return mcg::fail(MCG_ERR_INVALID, "words_per_instance exceeds the sample counter");
    const uint64_t slabs = (words + kThreads - 1) / kThreads;
    if ((uint64_t)n_inst * slabs >= 0xFFFFFFFFull) return mcg::fail(MCG_ERR_INVALID, "too many work items");
    if ((uint64_t)iteration + 2 >= (1ull << 26)) return mcg::fail(MCG_ERR_INVALID, "iteration out of range");
    for (uint32_t i = 0; i < n_inst; ++i) {
        if (inst_tree[i] >= b->trees.size()) return mcg::fail(MCG_ERR_INVALID, "instance tree out of range");
        if (thr_offset[i] + b->trees[inst_tree[i]].n_be > n_thr)
            return mcg::fail(MCG_ERR_INVALID, "instance thresholds out of range");
    }
    for (uint64_t k = 0; k < n_thr; ++k)
        if (thresholds[k] > (1ull << 32)) return mcg::fail(MCG_ERR_INVALID, "threshold above 2^32");
    MCG_CUDA(cudaSetDevice(b->device));
    bool tile = b->tile && !interpreter_is_faster(b, n_inst, inst_tree, words);
    mcg_status st = tile ? MCG_OK : interpreter_scratch(b);
    if (st == MCG_ERR_OOM && b->tile) {  // no room for the interpreter next to the tile kernel's memory
        mcg::clear_error();
        tile = true;
        st = MCG_OK;
    }
    if (st != MCG_OK) return st;
    st = run_instances(b, tile, n_inst, inst_tree, thr_offset, thresholds, n_thr, iteration, words, ones);
    if (st == MCG_ERR_OOM && tile) {  // a buffer did not fit there
        st = use_interpreter(b);
        if (st == MCG_OK)
            st = run_instances(b, false, n_inst, inst_tree, thr_offset, thresholds, n_thr, iteration, words, ones);
    }
    return st;
}

mcg_status mcg_batch_kernel(mcg_batch *b, uint32_t n_inst, const uint32_t *inst_tree, uint64_t words, int32_t *tiles) {
    mcg::clear_error();
    if (!b || !inst_tree || !tiles) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    for (uint32_t i = 0; i < n_inst; ++i)
        if (inst_tree[i] >= b->trees.size()) return mcg::fail(MCG_ERR_INVALID, "instance tree out of range");
    *tiles = b->tile && !interpreter_is_faster(b, n_inst, inst_tree, words) ? 1 : 0;
    return MCG_OK;
}

mcg_status mcg_batch_info_get(mcg_batch *b, mcg_batch_info *info) {
    mcg::clear_error();
    if (!b || !info) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    info->n_trees = (uint32_t)b->trees.size();
    info->smem_slots = b->smem_slots;
    info->max_global_slots = b->max_global;
    info->grid_ctas = b->grid;
    info->total_ops = b->total_ops;
    info->launches = b->launches;
    info->last_kernel_ms = b->last_ms;
    info->instances_per_item = b->share;
    return MCG_OK;
}

}  // extern "C"

// Tree sizes for the uncertainty driver (ua.cpp).
uint32_t mcg_batch_tree_count(const mcg_batch *b) { return (uint32_t)b->trees.size(); }
uint32_t mcg_batch_tree_n_be(const mcg_batch *b, uint32_t t) { return b->trees[t].n_be; }
