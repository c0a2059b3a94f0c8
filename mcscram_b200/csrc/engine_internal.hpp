// engine_internal.hpp -- the engine object shared by engine.cu and is.cu.
#pragma once
#include <cuda_runtime.h>

#include <functional>
#include <utility>
#include <unordered_map>
#include <vector>

#include "graph.hpp"
#include "mcg.h"
#include "program.hpp"
#include "tile_cost.hpp"
#include "tile.hpp"

namespace mcg {
namespace internal {
constexpr int kFusedThreads = 256;
constexpr uint64_t kDefaultChunkWords = 1ull << 21;
}  // namespace internal
}  // namespace mcg

struct mcg_engine {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    std::unordered_map<void *, size_t> work_bytes;  // sizes of the kept-buffer cache's allocations
    uint32_t mode = MCG_MODE_FUSED;
    mcg::Graph graph;
    mcg::Program prog;

    // fused
    uint4 *d_ops = nullptr;
    uint64_t *d_scratch = nullptr;
    uint64_t scratch_stride = 0;
    uint32_t nt = mcg::internal::kFusedThreads;
    uint32_t ctas_per_sm = 2;
    uint32_t grid = 0;
    uint32_t smem_bytes = 0;
    bool tally_in_smem = false;
    uint64_t chunk_words = mcg::internal::kDefaultChunkWords;

    // tile kernel (fused mode, small trees): its tables and launch shape
    bool tile = false;
    mcg::dev::TileArgs tile_args{};        // device pointers and sizes; the pass is filled in per launch
    std::vector<void *> tile_tables;
    uint32_t tile_threads = 0, tile_smem = 0, tile_sms = 0;
    mcg::TileCost tile_cost;               // its and the interpreter's time for a pass (tile_plan.hpp)

    // tallies
    unsigned long long *d_tally = nullptr;
    uint64_t total_bits = 0;

    // layered
    uint4 *d_be = nullptr;
    uint4 *d_meta = nullptr;
    uint32_t *d_inputs = nullptr;
    uint32_t *d_tally_nodes = nullptr;
    uint32_t *d_layer_gates = nullptr;
    std::vector<uint32_t> layer_offsets;  // into d_layer_gates, size n_layers + 1
    uint64_t *d_buf = nullptr;
    uint64_t buf_words = 0;
    uint64_t layered_max_words = 0;

    // staged
    uint4 *d_gates = nullptr;           // the gate kernel's tables (gate_plan.hpp)
    uint32_t *d_gate_in = nullptr;
    uint2 *d_gate_tally = nullptr;      // per gate {offset, count} into d_gate_tally_list
    uint32_t *d_gate_part = nullptr;
    uint2 *d_gate_layer = nullptr;
    uint32_t n_gate_parts = 0;
    uint32_t n_gate_layers = 0;
    uint32_t gates_largest_part = 0;    // gates
    uint64_t gate_block_ns = 0;         // a block's walk over the costliest part (gate_plan.hpp)
    bool gates_count = false;           // some gate counts in bit slices
    uint32_t gate_sms = 0;              // SMs of the device
    bool gates_beside_sampler = false;  // few gate blocks while the next chunk is sampled
    uint32_t *d_gate_tally_list = nullptr;
    uint32_t *d_be_tally_nodes = nullptr;  // tallied basic events
    uint32_t *d_be_tally_idx = nullptr;
    uint32_t n_be_tally = 0;
    uint64_t *d_stage[2] = {nullptr, nullptr};
    uint2 *d_event_table = nullptr;     // per-pass sampler table, n_be x kEventTableStride
    uint32_t table_iteration = 0xFFFFFFFFu;
    const uint4 *d_be_sample = nullptr;  // basic-event table the sampler phase reads (d_be unless overridden)
    // optional work queued on the gate stream after each chunk's gate phase (buffer, W, row stride)
    std::function<mcg_status(cudaStream_t, const uint64_t *, uint64_t, uint64_t)> chunk_hook;
    // optional work queued on the sampler stream after a chunk's basic-event
    // words are written and before its gates read them (buffer, W, row stride, word_begin)
    std::function<mcg_status(cudaStream_t, uint64_t *, uint64_t, uint64_t, uint64_t)> sample_hook;
    uint32_t sampler_smem = 0;          // dynamic smem that caps sampler blocks per SM
    uint64_t stage_words = 0;           // words per chunk the stage buffers hold
    uint64_t *d_stage_extra = nullptr;  // extra words the creator asked for, behind the first stage buffer
    uint64_t stage_extra_words = 0;
    cudaStream_t s_a = nullptr, s_b = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_a[2] = {nullptr, nullptr}, ev_b[2] = {nullptr, nullptr};
    cudaEvent_t ev_join_a = nullptr, ev_join_b = nullptr;
    // strip
    uint64_t *d_strip_scratch = nullptr;   // per warp strip_rows x 32 words
    unsigned long long *d_queue = nullptr; // strip counter
    // its program (build_strip_program), as StripArgs has it
    uint4 *d_strip_be = nullptr, *d_strip_table_be = nullptr;
    uint2 *d_strip_segment = nullptr, *d_strip_be_tally = nullptr;
    uint4 *d_strip_single = nullptr, *d_strip_groups = nullptr, *d_strip_ginfo = nullptr;
    uint32_t *d_strip_inputs = nullptr, *d_strip_gin = nullptr;
    uint32_t n_strip_be = 0, n_strip_segments = 0, n_strip_be_tally = 0, strip_rows = 1;
    uint32_t strip_grid = 0;
    uint64_t strip_few = 0;                // up to so many strips the four-block kernel runs
    uint32_t strip_smem = 0;               // tally counters in shared memory (0: global atomics)
    uint32_t strip_blocks = 6;             // resident blocks per SM the kernel is built for

    cudaEvent_t ev_snap[2] = {nullptr, nullptr};  // tally snapshots (slots behind d_tally)
    uint64_t snap_total[2] = {0, 0};

    mcg_run_desc run_desc{};                  // options the engine was created with
    bool prog_compiled = false;               // fused program compiled (fused mode, or on request)
    bool profile_a = false;                   // time every sampler-phase launch
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof_events;
    size_t prof_used = 0;

    uint64_t launches = 0;
};


namespace mcg {
namespace internal {

// mcg_create for an engine whose first stage buffer carries `extra_words(words
// per chunk)` 64-bit words behind it (d_stage_extra; staged mode only): room
// that comes and goes with the kept work buffers instead of an allocation.
mcg_status create_with_extra(const mcg_graph_desc *graph, const mcg_run_desc *run,
                             const std::function<uint64_t(uint64_t)> &extra_words, mcg_engine **out);

// Staged pass over [word_begin, word_begin + count) for n_it passes (engine.cu).
mcg_status run_staged(mcg_engine *e, uint32_t it_first, uint32_t n_it, uint64_t word_begin, uint64_t count);

// The same in parts: several word ranges, each with its own hooks and event
// table, whose sampling runs under the gates and hooks of the range before.
// *chunk is 0 at the fork; `more`: another range follows before the join.
mcg_status fork_staged(mcg_engine *e);
mcg_status add_staged(mcg_engine *e, uint64_t *chunk, uint32_t iteration, uint64_t word_begin, uint64_t count,
                      bool more);
mcg_status join_staged(mcg_engine *e);

}  // namespace internal
}  // namespace mcg
