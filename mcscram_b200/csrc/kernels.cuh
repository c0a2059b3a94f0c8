// kernels.cuh -- sm_100a kernels of the Monte Carlo engine.
//
//  k_tile        fused mode, trees that fit in shared memory: a block evaluates
//                32 words of every node at a time, its warps share out events
//                and gates; one launch per pass.
//  k_fused       persistent interpreter: each thread owns one sample word per
//                slab and walks the compiled node program (program_format.h):
//                Philox sampling in registers, gates in an accumulator,
//                shared-memory value slots, popcount tallies reduced per warp
//                into shared-memory counters and flushed once per CTA.
//  k_layer_be    reference dataflow, basic events: one word per thread
//                (src/mc/kernel/basic_event.h:125-142)
//  k_layer_gates reference dataflow, one layer of gates
//                (src/mc/kernel/gate.h:299-362, ATLEAST 506-555)
//  k_layer_tally reference dataflow, tallies (src/mc/kernel/tally.h:322-361)
//  k_sampler_peak register-only sampler: the fused kernel's speed of light.
#pragma once
#include <cstdint>

#include "gate_plan.hpp"
#include "mcg.h"
#include "philox.cuh"
#include "program_format.h"
#include "tile.hpp"

namespace mcg {
namespace dev {

constexpr uint64_t kAllOnes = ~0ull;

// Bit-sliced 8-bit counters (mod 256, like the reference's uint8 count).
// Bit-sliced count of up to 15 inputs (4 slices); count >= k for k <= 15.
struct SlicedCount4 {
    uint64_t c0 = 0, c1 = 0, c2 = 0, c3 = 0;
    __device__ __forceinline__ void add(uint64_t v) {
        const uint64_t t = c0 & v;
        c0 ^= v;
        const uint64_t t1 = c1 & t;
        c1 ^= t;
        const uint64_t t2 = c2 & t1;
        c2 ^= t1;
        c3 ^= t2;
    }
    __device__ __forceinline__ uint64_t ge(uint32_t k) const {
        const uint64_t c[4] = {c0, c1, c2, c3};
        uint64_t gt = 0, eq = kAllOnes;
#pragma unroll
        for (int b = 3; b >= 0; --b) {
            if ((k >> b) & 1u) {
                eq &= c[b];
            } else {
                gt |= eq & c[b];
                eq &= ~c[b];
            }
        }
        return gt | eq;
    }
};

struct SlicedCount {
    uint64_t c[8];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int b = 0; b < 8; ++b) c[b] = 0;
    }
    __device__ __forceinline__ void add(uint64_t v, uint32_t nbits) {
        uint64_t carry = v;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            if ((uint32_t)b < nbits) {
                const uint64_t t = c[b] & carry;
                c[b] ^= carry;
                carry = t;
            }
        }
    }
    // Per-lane (count >= k) for an 8-bit k.
    __device__ __forceinline__ uint64_t ge(uint32_t k) const {
        uint64_t gt = 0, eq = kAllOnes;
#pragma unroll
        for (int b = 7; b >= 0; --b) {
            if ((k >> b) & 1u) {
                eq &= c[b];
            } else {
                gt |= eq & c[b];
                eq &= ~c[b];
            }
        }
        return gt | eq;
    }
};

__device__ __forceinline__ uint64_t load_slot(uint32_t ref, const uint64_t *my_slots, const uint64_t *my_scratch,
                                              uint32_t nt, uint64_t stride) {
    if (ref & kSlotGlobal) return my_scratch[(uint64_t)(ref & kSlotIndexMask) * stride];
    return my_slots[(uint32_t)ref * nt];
}

__device__ __forceinline__ void store_slot(uint32_t ref, uint64_t v, uint64_t *my_slots, uint64_t *my_scratch,
                                           uint32_t nt, uint64_t stride) {
    if (ref == kNoSlot) return;
    if (ref & kSlotGlobal) my_scratch[(uint64_t)(ref & kSlotIndexMask) * stride] = v;
    else my_slots[(uint32_t)ref * nt] = v;
}

// Walks one node program for this thread's sample word.  With THR_TABLE the
// basic-event ops carry an index into thr (a per-instance uint64 threshold
// table) instead of the threshold itself.  tally(index, count) is called by
// lane 0 of each warp with the warp's popcount sum for a TALLY op.
template <int NT, int PF, bool THR_TABLE, bool SPLIT, class Tally>
__device__ __forceinline__ void interpret(const uint4 *__restrict__ ops, const WordCtx &ctx, uint32_t t3, bool valid,
                                          uint64_t *my_slots, uint64_t *my_scratch, uint64_t stride,
                                          const uint64_t *__restrict__ thr, Tally &&tally) {
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t acc = 0, last = 0;
    uint32_t conn = 0, kk = 0, nbits = 0;
    SlicedCount cnt;
    cnt.clear();
    const uint4 *p = ops;
    uint4 op = __ldg(p);
    while (true) {
        const uint4 nxt = __ldg(p + 1);
        const uint32_t code = op.x & kOpMask;
        if (code == kOpHalt) break;
        // Value of the op: one sampler call site keeps the unrolled Philox
        // body in the instruction cache once.
        uint64_t v = 0;
        if (code == kOpInBe || code == kOpBeDef) {
            if constexpr (THR_TABLE) {
                const uint64_t t = thr[op.z];
                if (t >= (1ull << 32)) v = kAllOnes;
                else if (t == 0) v = 0;
                else v = be_word<PF, SPLIT>(op.y, op.w, ctx, t3, (uint32_t)t);
            } else {
                v = be_word<PF, SPLIT>(op.y, op.w, ctx, t3, op.z);
            }
        } else if (code == kOpInSlot) {
            v = load_slot(op.y, my_slots, my_scratch, NT, stride);
        } else if (code == kOpInConst || code == kOpConstDef) {
            v = ((uint64_t)op.z << 32) | op.y;
        }
        if (code == kOpInBe || code == kOpInSlot || code == kOpInConst) {
            if (op.x & kNegBit) v = ~v;
            switch (conn) {
                case MCG_AND: case MCG_NAND: acc &= v; break;
                case MCG_OR: case MCG_NOR: acc |= v; break;
                case MCG_XOR: acc ^= v; break;
                case MCG_ATLEAST: cnt.add(v, nbits); break;
                default: acc = v; break;  // NOT, NULL: the last input wins
            }
        } else if (code == kOpBeDef || code == kOpConstDef) {
            last = v;
            store_slot(op.x >> 8, last, my_slots, my_scratch, NT, stride);
        } else if (code == kOpBegin) {
            conn = (op.x >> 8) & 0xFFu;
            kk = (op.x >> 16) & 0xFFu;
            nbits = (op.x >> 24) & 0xFu;
            acc = (conn == MCG_AND || conn == MCG_NAND) ? kAllOnes : 0ull;
            if (conn == MCG_ATLEAST) cnt.clear();
        } else if (code == kOpEnd) {
            if (conn == MCG_ATLEAST) last = cnt.ge(kk);
            else if (conn == MCG_NAND || conn == MCG_NOR || conn == MCG_NOT) last = ~acc;
            else last = acc;
            store_slot(op.y, last, my_slots, my_scratch, NT, stride);
        } else if (code == kOpTally) {
            uint32_t c = valid ? (uint32_t)__popcll(last) : 0u;
            c = __reduce_add_sync(0xFFFFFFFFu, c);
            if (lane == 0) tally(op.y, c);
        }
        op = nxt;
        ++p;
    }
}

struct FusedArgs {
    const uint4 *ops;
    uint32_t smem_slots;
    uint64_t *scratch;        // [global_slots][grid * NT]
    uint64_t scratch_stride;  // grid * NT of the allocation
    unsigned long long *tally;
    uint32_t n_tally;
    uint32_t tally_in_smem;
    uint32_t iteration_first;
    uint32_t n_iterations;
    uint64_t word_begin;
    uint64_t word_count;
};

template <int NT, int MINB, int PF>
__global__ void __launch_bounds__(NT, MINB) k_fused(FusedArgs a) {
    extern __shared__ __align__(16) uint64_t smem[];
    const uint32_t tid = threadIdx.x;
    unsigned long long *s_tally = reinterpret_cast<unsigned long long *>(smem + (size_t)a.smem_slots * NT);
    if (a.tally_in_smem) {
        for (uint32_t i = tid; i < a.n_tally; i += NT) s_tally[i] = 0ull;
        __syncthreads();
    }
    unsigned long long *tally = a.tally_in_smem ? s_tally : a.tally;
    const uint64_t gtid = (uint64_t)blockIdx.x * NT + tid;
    const uint64_t total_threads = (uint64_t)gridDim.x * NT;
    uint64_t *my_slots = smem + tid;
    uint64_t *my_scratch = a.scratch + gtid;
    auto add = [tally](uint32_t idx, uint32_t c) { atomicAdd(&tally[idx], (unsigned long long)c); };

    for (uint32_t it = 0; it < a.n_iterations; ++it) {
        const uint32_t t3 = (a.iteration_first + it + 1u) << 6;
        for (uint64_t base = 0; base < a.word_count; base += total_threads) {
            const uint64_t j = base + gtid;
            const WordCtx ctx = make_word_ctx((uint32_t)(a.word_begin + j));
            interpret<NT, PF, false, MINB == 4>(a.ops, ctx, t3, j < a.word_count, my_slots, my_scratch,
                                                a.scratch_stride, nullptr, add);
        }
    }
    if (a.tally_in_smem) {
        __syncthreads();
        for (uint32_t i = tid; i < a.n_tally; i += NT) {
            const unsigned long long c = s_tally[i];
            if (c) atomicAdd(&a.tally[i], c);
        }
    }
}

// Batched instances (uncertainty analysis): a persistent work queue over
// (instance, slab) items; an instance runs its tree's program with its own
// threshold table over words [0, words_per_instance) of pass `iteration`
// and counts the ones of every TALLY op into inst_ones[instance].
struct BatchArgs {
    const uint4 *ops;                  // all tree programs, concatenated
    const uint32_t *tree_op_offset;    // first op of each tree's program
    const uint32_t *inst_tree;         // tree of each instance
    const uint64_t *inst_thr_offset;   // first threshold of each instance
    const uint64_t *thr;               // thresholds (uint64, 0 .. 2^32)
    uint32_t n_instances;
    uint32_t slabs_per_instance;
    uint64_t words_per_instance;
    uint32_t iteration;
    uint32_t smem_slots;
    uint64_t *scratch;
    uint64_t scratch_stride;
    unsigned int *queue;               // next item; zero before the launch
    unsigned long long *inst_ones;
    // k_fused_batch_k: groups of up to K consecutive instances of one tree
    const uint32_t *group_first;
    const uint32_t *group_size;
    uint32_t n_groups;
};

template <int NT, int MINB, int PF>
__global__ void __launch_bounds__(NT, MINB) k_fused_batch(BatchArgs a) {
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ unsigned int s_item;
    const uint32_t tid = threadIdx.x;
    const uint64_t gtid = (uint64_t)blockIdx.x * NT + tid;
    uint64_t *my_slots = smem + tid;
    uint64_t *my_scratch = a.scratch + gtid;
    const uint32_t t3 = (a.iteration + 1u) << 6;
    const unsigned int n_items = a.n_instances * a.slabs_per_instance;
    while (true) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(a.queue, 1u);
        __syncthreads();
        const unsigned int item = s_item;
        if (item >= n_items) break;
        const uint32_t inst = item / a.slabs_per_instance;
        const uint64_t j = (uint64_t)(item % a.slabs_per_instance) * NT + tid;
        const WordCtx ctx = make_word_ctx((uint32_t)j);
        unsigned long long *ones = a.inst_ones + inst;
        auto add = [ones](uint32_t, uint32_t c) { atomicAdd(ones, (unsigned long long)c); };
        interpret<NT, PF, true, false>(a.ops + a.tree_op_offset[a.inst_tree[inst]], ctx, t3, j < a.words_per_instance,
                                    my_slots, my_scratch, a.scratch_stride, a.thr + a.inst_thr_offset[inst], add);
    }
}

// Slot planes of the K-wide interpreter: slot s of instance k at [s * K + k].
template <int K>
__device__ __forceinline__ uint64_t load_slot_k(uint32_t ref, int k, const uint64_t *my_slots,
                                                const uint64_t *my_scratch, uint32_t nt, uint64_t stride) {
    if (ref & kSlotGlobal) return my_scratch[((uint64_t)(ref & kSlotIndexMask) * K + k) * stride];
    return my_slots[((uint32_t)ref * K + k) * nt];
}

template <int K>
__device__ __forceinline__ void store_slot_k(uint32_t ref, int k, uint64_t v, uint64_t *my_slots,
                                             uint64_t *my_scratch, uint32_t nt, uint64_t stride) {
    if (ref == kNoSlot) return;
    if (ref & kSlotGlobal) my_scratch[((uint64_t)(ref & kSlotIndexMask) * K + k) * stride] = v;
    else my_slots[((uint32_t)ref * K + k) * nt] = v;
}

// The interpreter over K instances of one tree that differ only in their
// thresholds (draws of an uncertainty analysis): every op acts on K words, a
// basic event's 16 Philox calls run once and are compared with the K
// instances' thresholds (thr[k][op.z]), so word k equals what interpret gives
// instance k.  With ATL, ATLEAST gates of at most 15 inputs count in four
// bit slices per instance; without it the program must have no ATLEAST gate
// (the batch runs wider ones one instance at a time).  tally(k, count) is
// called by lane 0 with instance k's warp popcount sum.
template <int NT, int PF, int K, bool ATL, class Tally>
__device__ __forceinline__ void interpret_k(const uint4 *__restrict__ ops, const WordCtx &ctx, uint32_t t3,
                                            bool valid, uint64_t *my_slots, uint64_t *my_scratch, uint64_t stride,
                                            const uint64_t *const *thr, Tally &&tally) {
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t acc[K], last[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = last[k] = 0ull;
    SlicedCount4 cnt[K];
    uint32_t conn = 0, kk = 0;
    const uint4 *p = ops;
    uint4 op = __ldg(p);
    while (true) {
        const uint4 nxt = __ldg(p + 1);
        const uint32_t code = op.x & kOpMask;
        if (code == kOpHalt) break;
        uint64_t v[K];
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = 0ull;
        if (code == kOpInBe || code == kOpBeDef) {
            uint32_t t32[K];
            uint32_t ones = 0, zeros = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint64_t t = thr[k][op.z];
                t32[k] = (uint32_t)t;
                if (t >= (1ull << 32)) {
                    ones |= 1u << k;
                    t32[k] = 1u;
                } else if (t == 0) {
                    zeros |= 1u << k;
                    t32[k] = 1u;
                }
            }
            if ((ones | zeros) != (1u << K) - 1u) be_words<PF, K>(op.y, op.w, ctx, t3, t32, v);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if ((ones >> k) & 1u) v[k] = kAllOnes;
                else if ((zeros >> k) & 1u) v[k] = 0ull;
            }
        } else if (code == kOpInSlot) {
#pragma unroll
            for (int k = 0; k < K; ++k) v[k] = load_slot_k<K>(op.y, k, my_slots, my_scratch, NT, stride);
        } else if (code == kOpInConst || code == kOpConstDef) {
#pragma unroll
            for (int k = 0; k < K; ++k) v[k] = ((uint64_t)op.z << 32) | op.y;
        }
        if (code == kOpInBe || code == kOpInSlot || code == kOpInConst) {
            if (op.x & kNegBit) {
#pragma unroll
                for (int k = 0; k < K; ++k) v[k] = ~v[k];
            }
            switch (conn) {
                case MCG_AND: case MCG_NAND:
#pragma unroll
                    for (int k = 0; k < K; ++k) acc[k] &= v[k];
                    break;
                case MCG_OR: case MCG_NOR:
#pragma unroll
                    for (int k = 0; k < K; ++k) acc[k] |= v[k];
                    break;
                case MCG_XOR:
#pragma unroll
                    for (int k = 0; k < K; ++k) acc[k] ^= v[k];
                    break;
                case MCG_ATLEAST:
                    if constexpr (ATL) {
#pragma unroll
                        for (int k = 0; k < K; ++k) cnt[k].add(v[k]);
                    }
                    break;
                default:  // NOT, NULL: the last input wins
#pragma unroll
                    for (int k = 0; k < K; ++k) acc[k] = v[k];
                    break;
            }
        } else if (code == kOpBeDef || code == kOpConstDef) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                last[k] = v[k];
                store_slot_k<K>(op.x >> 8, k, last[k], my_slots, my_scratch, NT, stride);
            }
        } else if (code == kOpBegin) {
            conn = (op.x >> 8) & 0xFFu;
            kk = (op.x >> 16) & 0xFFu;
            const uint64_t init = (conn == MCG_AND || conn == MCG_NAND) ? kAllOnes : 0ull;
#pragma unroll
            for (int k = 0; k < K; ++k) acc[k] = init;
            if constexpr (ATL) {
                if (conn == MCG_ATLEAST) {
#pragma unroll
                    for (int k = 0; k < K; ++k) cnt[k] = SlicedCount4{};
                }
            }
        } else if (code == kOpEnd) {
            const bool inv = conn == MCG_NAND || conn == MCG_NOR || conn == MCG_NOT;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (ATL && conn == MCG_ATLEAST) last[k] = kk > 15 ? 0ull : cnt[k].ge(kk);  // at most 15 inputs
                else last[k] = inv ? ~acc[k] : acc[k];
                store_slot_k<K>(op.y, k, last[k], my_slots, my_scratch, NT, stride);
            }
        } else if (code == kOpTally) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, valid ? (uint32_t)__popcll(last[k]) : 0u);
                if (lane == 0) tally((uint32_t)k, c);
            }
        }
        op = nxt;
        ++p;
    }
}

// Batched instances K at a time: a work item is (group, slab), a group up to
// K consecutive instances of one tree; missing members of a short group
// repeat its first instance's thresholds and add nothing to any tally.
template <int NT, int MINB, int PF, int K, bool ATL>
__global__ void __launch_bounds__(NT, MINB) k_fused_batch_k(BatchArgs a) {
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ unsigned int s_item;
    const uint32_t tid = threadIdx.x;
    const uint64_t gtid = (uint64_t)blockIdx.x * NT + tid;
    uint64_t *my_slots = smem + tid;
    uint64_t *my_scratch = a.scratch + gtid;
    const uint32_t t3 = (a.iteration + 1u) << 6;
    const unsigned int n_items = a.n_groups * a.slabs_per_instance;
    while (true) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(a.queue, 1u);
        __syncthreads();
        const unsigned int item = s_item;
        if (item >= n_items) break;
        const uint32_t grp = item / a.slabs_per_instance;
        const uint64_t j = (uint64_t)(item % a.slabs_per_instance) * NT + tid;
        const uint32_t first = a.group_first[grp], n = a.group_size[grp];
        const uint64_t *thr[K];
#pragma unroll
        for (int k = 0; k < K; ++k) thr[k] = a.thr + a.inst_thr_offset[first + ((uint32_t)k < n ? (uint32_t)k : 0u)];
        const WordCtx ctx = make_word_ctx((uint32_t)j);
        unsigned long long *ones = a.inst_ones + first;
        auto add = [ones, n](uint32_t k, uint32_t c) {
            if (k < n) atomicAdd(ones + k, (unsigned long long)c);
        };
        interpret_k<NT, PF, K, ATL>(a.ops + a.tree_op_offset[a.inst_tree[first]], ctx, t3, j < a.words_per_instance,
                                   my_slots, my_scratch, a.scratch_stride, thr, add);
    }
}

// ---------------------------------------------------------------------------
// Reference dataflow (layered).  Node words live in buf[node * W + w].

// Basic events: be[e] = {pdag_idx+1, event_idx+1, thr_lo, thr_hi}.
template <int PF>
__global__ void __launch_bounds__(256) k_layer_be(const uint4 *__restrict__ be, uint32_t n_be, uint64_t W,
                                                  uint64_t word_begin, uint32_t t3, uint64_t *__restrict__ buf) {
    const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t e = blockIdx.y + gridDim.y * blockIdx.z;
    if (w >= W || e >= n_be) return;
    const uint4 r = be[e];
    const uint64_t thr = ((uint64_t)r.w << 32) | r.z;
    uint64_t v;
    if (thr == 0) v = 0;
    else if (thr >= (1ull << 32)) v = kAllOnes;
    else v = be_word<PF>(r.x, r.y, make_word_ctx((uint32_t)(word_begin + w)), t3, (uint32_t)thr);
    buf[(uint64_t)e * W + w] = v;
}

// One layer of gates; gate ids listed in layer_gates.  meta[g] = {op | k<<8, in_begin, in_count, neg_count}.
// ATLEAST counts each bit lane with a uint8 counter, as the reference kernel does.
static __global__ void __launch_bounds__(256) k_layer_gates(const uint4 *__restrict__ meta, const uint32_t *__restrict__ inputs,
                                                     const uint32_t *__restrict__ layer_gates, uint32_t n_layer,
                                                     uint32_t n_be, uint64_t W, uint64_t *__restrict__ buf) {
    const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t li = blockIdx.y + gridDim.y * blockIdx.z;
    if (w >= W || li >= n_layer) return;
    const uint32_t gi = layer_gates[li];
    const uint4 m = meta[gi];
    const uint32_t op = m.x & 0xFFu;
    const uint32_t n = m.z;
    const uint32_t off = n - m.w;
    const uint32_t *in = inputs + m.y;
    uint64_t r;
    if (op == MCG_ATLEAST) {
        const uint8_t k = (uint8_t)(m.x >> 8);
        r = 0;
        for (uint32_t lane = 0; lane < 64; ++lane) {
            const uint64_t mask = 1ull << lane;
            uint8_t cnt = 0;
            for (uint32_t i = 0; i < n; ++i) {
                const uint64_t v = buf[(uint64_t)in[i] * W + w];
                cnt += (uint8_t)((((i < off) ? v : ~v) & mask) ? 1 : 0);
            }
            if (cnt >= k) r |= mask;
        }
    } else {
        r = (op == MCG_AND || op == MCG_NAND) ? kAllOnes : 0ull;
        for (uint32_t i = 0; i < n; ++i) {
            uint64_t v = buf[(uint64_t)in[i] * W + w];
            if (i >= off) v = ~v;
            if (op == MCG_OR || op == MCG_NOR) r |= v;
            else if (op == MCG_AND || op == MCG_NAND) r &= v;
            else if (op == MCG_XOR) r ^= v;
            else r = v;
        }
        if (op == MCG_NAND || op == MCG_NOR || op == MCG_NOT) r = ~r;
    }
    buf[(uint64_t)(n_be + gi) * W + w] = r;
}

// Tallies: popcount, block reduction, one atomic per block and node.
// tally_idx (optional) maps row t of tally_nodes to its counter.
static __global__ void __launch_bounds__(256) k_layer_tally(const uint32_t *__restrict__ tally_nodes, uint32_t n_tally,
                                                     uint64_t W, uint64_t stride, const uint64_t *__restrict__ buf,
                                                     unsigned long long *__restrict__ ones,
                                                     const uint32_t *__restrict__ tally_idx) {
    __shared__ uint32_t warp_sums[8];
    const uint32_t t = blockIdx.y + gridDim.y * blockIdx.z;
    if (t >= n_tally) return;
    uint32_t c = 0;
    const uint64_t *row = buf + (uint64_t)tally_nodes[t] * stride;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < W; w += (uint64_t)gridDim.x * blockDim.x)
        c += (uint32_t)__popcll(row[w]);
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if ((threadIdx.x & 31u) == 0) warp_sums[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long s = 0;
        for (uint32_t i = 0; i < (blockDim.x >> 5); ++i) s += warp_sums[i];
        if (s) atomicAdd(&ones[tally_idx ? tally_idx[t] : t], s);
    }
}

// ---------------------------------------------------------------------------
// Staged pipeline.  Phase A samples basic-event words into buf rows
// [0, n_be); phase B evaluates the gates into rows n_be + g, with tallies fused.

// Per-pass event table (philox.cuh): thread (e, g) fills entry g of event e.
static __global__ void __launch_bounds__(256) k_event_table(const uint4 *__restrict__ be, uint32_t n_be, uint32_t t3,
                                                     uint2 *__restrict__ table) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)n_be * kEventTableStride) return;
    const uint32_t e = (uint32_t)(i / kEventTableStride);
    const int g = (int)(i % kEventTableStride);
    event_table_entry(be[e].x, t3, g, table[i]);
}

// Phase A: thread (w, group) samples words 2 w and 2 w + 1 of events
// [group * ept, + ept) using the pass's event table.  Launched with dynamic
// shared memory that only caps the blocks per SM, leaving room for gate-phase
// blocks.  Bound by the sampler's instructions: two words per thread share the
// table's loads and leave 64 registers to a thread, in four blocks per SM
// (300,001 words of the 1,003-event tree with its gates: 10.48 ms; one word per
// thread in six blocks of 40 registers 10.72, two in three or five blocks
// 10.63, four in two or three 10.61 and 10.65).
template <int PF>
__global__ void __launch_bounds__(256, 4) k_stage_be(const uint4 *__restrict__ be, const uint2 *__restrict__ table,
                                                     uint32_t n_be, uint32_t ept, uint64_t W, uint64_t stride,
                                                     uint64_t word_begin, uint64_t *__restrict__ buf) {
    const uint64_t w = 2 * ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x);
    const uint32_t e0 = (blockIdx.y + gridDim.y * blockIdx.z) * ept;
    if (w >= W || e0 >= n_be) return;
    const WordCtx ctx[2] = {make_word_ctx((uint32_t)(word_begin + w)), make_word_ctx((uint32_t)(word_begin + w + 1))};
    const uint32_t end = min(e0 + ept, n_be);
#pragma unroll 1
    for (uint32_t e = e0; e < end; ++e) {
        const uint4 r = be[e];
        uint64_t v[2];
        if (r.w != 0) v[0] = v[1] = kAllOnes;           // threshold 2^32
        else if (r.z == 0) v[0] = v[1] = 0;             // threshold 0
        else be_words_tab<PF, 2>(r.y, ctx, GlobalTable{table + (uint64_t)e * kEventTableStride}, r.z, v);
        uint64_t *out = buf + (uint64_t)e * stride + w;
        // The pipeline's rows have room for an even number of words.  The other branch
        // stays for any stride's sake: without it the sampler is scheduled 0.7 % slower
        // (300,001 words of the 1,003-event tree 10.44 -> 10.52 ms).
        if (stride % 2 == 0) {
            *reinterpret_cast<ulonglong2 *>(out) = make_ulonglong2(v[0], v[1]);
        } else {
            out[0] = v[0];
            if (w + 1 < W) out[1] = v[1];
        }
    }
}

// Phase B: every layer of gates in one launch, or a launch per layer for few words
// of many gates (gate_splits).  A block takes 32 * WPL words
// (lane = WPL neighbouring words, one load each of a row) of one part
// (gate_plan.hpp); its warps share out the gates of a layer, and a block
// barrier ends the layer.  A block's gates read rows that the block or phase A
// wrote, so no layer waits for the whole chip, and a pass of few words has no
// launch per layer.  Bound by memory (5.4 TB/s of rows read and written) where
// it runs alone on many words, by the latency of a gate's rows on few; under
// the sampling of the next chunk it costs the issue slots of 166 instructions
// per gate and 64 words.  32,768 words of the 5,000-event tree (20 layers):
// 0.65 ms, 0.96 with a launch per layer.
constexpr int kGateThreadsMost = 1024;
struct StageGateArgs {
    const uint4 *gates;
    const uint32_t *in;
    const uint2 *tally;
    const uint32_t *tally_list;
    const uint32_t *part;
    const uint2 *layer;
    uint64_t words, stride;  // per row: words in use, words from row to row
    uint32_t part_first;     // part of blockIdx.y = 0
    uint32_t first, layers;  // the layers that the launch takes of every part
    uint64_t *buf;
    unsigned long long *ones;
};

// WPL words of a row, in 32-bit halves.
template <int WPL>
struct GateRow {
    uint32_t w[2 * WPL];
};

template <int WPL>
__device__ __forceinline__ GateRow<WPL> gate_load(const char *col, uint32_t stride, uint32_t rec) {
    const char *p = col + (uint64_t)(rec & ~kGateFlip) * stride;
    GateRow<WPL> r;
    if constexpr (WPL == 2) {
        const uint4 v = *reinterpret_cast<const uint4 *>(p);
        r.w[0] = v.x, r.w[1] = v.y, r.w[2] = v.z, r.w[3] = v.w;
    } else {
        const uint2 v = *reinterpret_cast<const uint2 *>(p);
        r.w[0] = v.x, r.w[1] = v.y;
    }
    return r;
}

// Calls f(half, value) for every input of a gate, U loads in flight.  The
// records behind the last input repeat it: their value is the input's again
// (PAD: 0).
template <int WPL, int U, bool PAD, class F>
__device__ __forceinline__ void gate_inputs(const char *col, uint32_t stride, uint32_t n, uint4 q, const uint4 *more,
                                            F f) {
#pragma unroll 1
    for (uint32_t j = 0; j < n;) {
        const uint32_t rec[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (uint32_t u0 = 0; u0 < 4; u0 += U) {
            if (U < 4 && u0 && j + u0 >= n) break;
            GateRow<WPL> x[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) x[u] = gate_load<WPL>(col, stride, rec[u0 + u]);
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t flip = (uint32_t)((int32_t)rec[u0 + u] >> 31);
                const uint32_t keep = j + u0 + u < n ? 0xFFFFFFFFu : 0u;
#pragma unroll
                for (int h = 0; h < 2 * WPL; ++h) f(h, PAD ? (x[u].w[h] ^ flip) & keep : x[u].w[h] ^ flip);
            }
        }
        j += 4;
        if (j < n) q = *more++;
    }
}

// A 64-bit word of a k-of-n gate, counted in eight bit slices, four inputs at a
// time through full adders.  Not inlined, and in a kernel of its own for graphs
// that have such gates (COUNT): 131,072 words of 600 OR gates of 12 inputs take
// 1.37 ms in the other one, 1.45 in this one, 1.59 with the counting inlined.
// Bound by the rows' loads on few words, by the counting on many: 131,072 words
// of 600 gates of 60 inputs 8.4 ms; 28.7 one input and 32 bits at a time, 19.0
// one input and 64 bits at a time with a thread per word.
static __device__ __noinline__ uint2 gate_count(const char *col, uint32_t stride, const uint4 m, uint4 q,
                                                const uint4 *more) {
    const uint32_t n = m.z, kk = (m.x >> 8) & 0xFFu, nbits = (m.x >> 16) & 0xFu;
    uint32_t c[8][2] = {};
#pragma unroll 1
    for (uint32_t j = 0; j < n;) {
        const uint32_t rec[4] = {q.x, q.y, q.z, q.w};
        GateRow<1> x[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) x[u] = gate_load<1>(col, stride, rec[u]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                v[u] = j + u < n ? x[u].w[h] ^ (uint32_t)((int32_t)rec[u] >> 31) : 0u;
            const uint32_t t0 = (c[0][h] & v[0]) | (c[0][h] & v[1]) | (v[0] & v[1]);
            c[0][h] ^= v[0] ^ v[1];
            const uint32_t t1 = (c[0][h] & v[2]) | (c[0][h] & v[3]) | (v[2] & v[3]);
            c[0][h] ^= v[2] ^ v[3];
            uint32_t t = (c[1][h] & t0) | (c[1][h] & t1) | (t0 & t1);
            c[1][h] ^= t0 ^ t1;
#pragma unroll
            for (uint32_t b = 2; b < 8; ++b) {
                if (b < nbits) {
                    const uint32_t s = c[b][h] & t;
                    c[b][h] ^= t;
                    t = s;
                }
            }
        }
        j += 4;
        if (j < n) q = *more++;
    }
    uint32_t r[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t gt = 0, eq = 0xFFFFFFFFu;
#pragma unroll
        for (int b = 7; b >= 0; --b) {
            if ((kk >> b) & 1u) {
                eq &= c[b][h];
            } else {
                gt |= eq & c[b][h];
                eq &= ~c[b][h];
            }
        }
        r[h] = gt | eq;
    }
    return make_uint2(r[0], r[1]);
}

// A gate's words: m and q are its two records.  COUNT: of a graph with gates
// that count in bit slices.
template <int WPL, bool COUNT>
__device__ __forceinline__ GateRow<WPL> gate_words(const char *col, uint32_t stride, const uint4 &m, const uint4 &q,
                                                   const uint32_t *in) {
    constexpr int H = 2 * WPL;
    GateRow<WPL> r;
#pragma unroll
    for (int h = 0; h < H; ++h) r.w[h] = 0;
    const uint32_t kind = m.x & 3u, kk = (m.x >> 8) & 0xFFu;
    const uint4 *more = reinterpret_cast<const uint4 *>(in + m.y);
    if (kind == kGateOr && m.z == 2) {
        const GateRow<WPL> x = gate_load<WPL>(col, stride, q.x), y = gate_load<WPL>(col, stride, q.y);
        const uint32_t fx = (uint32_t)((int32_t)q.x >> 31), fy = (uint32_t)((int32_t)q.y >> 31);
#pragma unroll
        for (int h = 0; h < H; ++h) r.w[h] = (x.w[h] ^ fx) | (y.w[h] ^ fy);
    } else if (kind == kGateOr) {
        gate_inputs<WPL, 4, false>(col, stride, m.z, q, more, [&](int h, uint32_t v) { r.w[h] |= v; });
    } else if (kind == kGateXor) {
        gate_inputs<WPL, 4, true>(col, stride, m.z, q, more, [&](int h, uint32_t v) { r.w[h] ^= v; });
    } else if (!COUNT || kind == kGateChain) {
        // c[j]: at least j + 1 so far; r: at least kk
        uint32_t c[3][H] = {};
        const uint32_t two = kk == 2 ? 0xFFFFFFFFu : 0u, three = kk == 3 ? 0xFFFFFFFFu : 0u;
        gate_inputs<WPL, 2, true>(col, stride, m.z, q, more, [&](int h, uint32_t v) {
            const uint32_t below = (c[0][h] & two) | (c[1][h] & three) | (c[2][h] & ~(two | three));
            r.w[h] |= below & v;
            c[2][h] |= c[1][h] & v;
            c[1][h] |= c[0][h] & v;
            c[0][h] |= v;
        });
    } else if constexpr (COUNT) {
#pragma unroll
        for (int w = 0; w < WPL; ++w) {
            const uint2 x = gate_count(col + 8 * w, stride, m, q, more);
            r.w[2 * w] = x.x, r.w[2 * w + 1] = x.y;
        }
    }
    const uint32_t inverted = (m.x & 4u) ? 0xFFFFFFFFu : 0u;
#pragma unroll
    for (int h = 0; h < H; ++h) r.w[h] ^= inverted;
    return r;
}

// SPLIT: a launch of one layer, whose gates the blocks of blockIdx.z share (the
// other launches carry no stride and offset of it through their layers: 800
// layers of a gate each on 2,048 words 0.48 ms, 0.50 with them).
template <int WPL, bool COUNT, bool SPLIT>
__global__ void __launch_bounds__(kGateThreadsMost) k_stage_gates(const __grid_constant__ StageGateArgs a) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t warps = blockDim.x >> 5;
    const uint32_t stride = (uint32_t)(a.stride * sizeof(uint64_t));
    const uint32_t step = SPLIT ? warps * gridDim.z : warps, mine0 = SPLIT ? blockIdx.z * warps + warp : warp;
    const uint32_t *part = a.part + a.part_first + blockIdx.y;
    const uint32_t l_begin = part[0] + a.first, l_end = min(l_begin + a.layers, part[1]);
    if (l_begin >= l_end) return;
    const uint32_t tiles = (uint32_t)((a.words + 32 * WPL - 1) / (32 * WPL));
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t w0 = ((uint64_t)tile * 32u + lane) * WPL;
        const bool valid = w0 < a.words, both = w0 + (WPL - 1) < a.words;
        const bool whole = ((uint64_t)tile + 1) * (32 * WPL) <= a.words;
        // lanes behind the end read the row's first words and store nothing
        char *col = reinterpret_cast<char *>(a.buf + (valid ? w0 : 0));
        uint32_t l = l_begin;
        uint2 range = a.layer[l];
        uint32_t i = range.x + mine0;
        uint4 m{}, q{};
        auto head = [&](uint32_t g) {
            m = a.gates[2 * (uint64_t)g];
            q = a.gates[2 * (uint64_t)g + 1];
        };
        if (i < range.y) head(i);
        for (;;) {
            // the warp's next gate, in this layer or the next: its records are
            // loaded under this gate's rows
            const bool mine = i < range.y, last = i + step >= range.y;
            const uint4 cm = m, cq = q;
            const uint32_t gate = i;
            i += step;
            if (last && ++l < l_end) {
                range = a.layer[l];
                i = range.x + mine0;
            }
            if (i < range.y) head(i);
            if (mine) {
                const uint2 t = a.tally[gate];
                const GateRow<WPL> r = gate_words<WPL, COUNT>(col, stride, cm, cq, a.in);
                char *out = col + (uint64_t)cm.w * stride;
                if (valid) {
                    if constexpr (WPL == 2)
                        *reinterpret_cast<uint4 *>(out) = make_uint4(r.w[0], r.w[1], r.w[2], r.w[3]);
                    else
                        *reinterpret_cast<uint2 *>(out) = make_uint2(r.w[0], r.w[1]);
                }
                if (t.y) {
                    uint32_t n = __popc(r.w[0]) + __popc(r.w[1]), n2 = 0;
                    if constexpr (WPL == 2) n2 = __popc(r.w[2]) + __popc(r.w[3]);
                    n = whole ? n + n2 : (valid ? n : 0u) + (both ? n2 : 0u);
                    n = __reduce_add_sync(0xFFFFFFFFu, n);
                    if (lane == 0 && n) {
                        if (t.y == 1) atomicAdd(&a.ones[t.x], (unsigned long long)n);
                        else
                            for (uint32_t j = 0; j < t.y; ++j)
                                atomicAdd(&a.ones[a.tally_list[t.x + j]], (unsigned long long)n);
                    }
                }
            }
            if (last) {
                __syncthreads();
                if (l == l_end) break;
            }
        }
    }
}

// Strip mode: one persistent kernel per pass.  A block takes strips of 256
// consecutive words from a queue; warp w owns words [32 w, 32 w + 32) of
// the strip and a private scratch block of rows of 32 words.  Lane l samples
// its word of a segment's events (one Philox word per event, event table of
// the pass), evaluates the segment's gates for the same word, adds the
// popcounts of tallied nodes into the block's shared-memory counters, and goes
// on to the next segment; rows are used again (build_strip_program).  A lane
// only reads the column it wrote, so the only barrier is the strip hand-out:
// the eight warps of a block walk the events together (the table rows they
// read stay in L1), while the blocks on an SM drift apart, so the
// memory-bound gate work of some blocks runs under the multiply-bound
// sampling of the others.  Bound by the issue of the sampler's instructions
// (703 per event and warp) and the gates' (46): 2^20 words of the 5,000-event
// tree take 188.0 ms; 193.9 with all events before all gates and 8-byte table
// loads.
constexpr int kStripLanes = 32;
constexpr int kStripThreads = 256;

struct StripArgs {
    const uint4 *be;              // in segment order: {row, event + 1, thr lo, thr hi}
    const uint2 *table;           // event table of the pass, in the same order
    const uint2 *segment;         // {events' end, groups' end}
    uint32_t n_segments;
    uint32_t rows;                // of a warp's scratch block; the last one holds zeros
    const uint4 *single;          // gates of their own: op | k << 8 | nbits << 16, in_begin, in_count, neg_count
    const uint32_t *inputs;       // their inputs: rows
    const uint4 *groups;          // per group two records: {count | fan-in << 8 | single << 24, gin offset,
                                  // ginfo offset, outinv} and the output rows of its gates
    const uint32_t *gin;          // group inputs, slot-major, kStripGroup records per slot: row | flip
    const uint4 *ginfo;           // per grouped gate: {output row, tally offset, tally count, single gate}
    const uint32_t *tally_list;
    const uint2 *be_tally;        // tallied events {row, tally index}
    uint32_t n_be_tally;
    uint32_t n_tally;
    uint32_t tally_in_smem;
    unsigned long long *ones;
    uint64_t *scratch;            // per warp: rows x 32 words
    uint64_t word_begin, word_count;
    unsigned long long *queue;
};

__device__ __forceinline__ void strip_tally(const StripArgs &a, unsigned long long *s_ones, uint32_t idx,
                                            uint32_t c) {
    if (a.tally_in_smem) atomicAdd(&s_ones[idx], (unsigned long long)c);
    else atomicAdd(&a.ones[idx], (unsigned long long)c);
}

// Gate groups of the strip kernel: up to kStripGroup gates that read none of
// each other, evaluated together in the OR form
// r = outinv ^ OR_i (x_i ^ flip_i).  A row is its byte offset in the warp's
// scratch block; an input record is the row | flip, an empty slot the row of
// zeros.
constexpr uint32_t kStripGroup = 4;
constexpr uint32_t kStripGroupMaxIn = 8;
static_assert(kStripGroup == 4, "k_strip's group loop packs four gates' tallies into two reductions");

__device__ __forceinline__ uint64_t &strip_row(const uint64_t *col, uint32_t row) {
    return *reinterpret_cast<uint64_t *>(reinterpret_cast<unsigned char *>(const_cast<uint64_t *>(col)) + row);
}

__device__ __forceinline__ uint64_t strip_in(const uint64_t *col, uint32_t rec) {
    return strip_row(col, rec & ~1u) ^ (uint64_t)(-(int64_t)(rec & 1u));
}

// Tally of one gate word column: warp sum of the valid lanes' popcounts,
// added by lane 0 to every tally slot of the node.
__device__ __forceinline__ void strip_gate_tally(const StripArgs &a, unsigned long long *s_ones, const uint4 &f,
                                                 uint64_t r, bool valid, uint32_t lane) {
    if (f.z) {
        const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, valid ? (uint32_t)__popcll(r) : 0u);
        if (lane == 0 && c)
            for (uint32_t j = 0; j < f.z; ++j) strip_tally(a, s_ones, a.tally_list[f.y + j], c);
    }
}


// Not inlined: the one-gate path (ATLEAST counters, wide fan-in loops) then
// keeps its registers to itself, and k_strip's sampler and gate groups spill
// 36 bytes instead of 376 at 40 registers.
static __device__ __noinline__ uint64_t strip_gate(const StripArgs &a, const uint64_t *col, uint32_t gi) {
    constexpr uint32_t kMaxIn = 8;
    const uint4 m = a.single[gi];
    const uint32_t op = m.x & 0xFFu, kk = (m.x >> 8) & 0xFFu, nbits = (m.x >> 16) & 0xFu;
    const uint32_t n = m.z, off = n - m.w;
    const uint32_t *in = a.inputs + m.y;
    if (op == MCG_ATLEAST) {
        if (n <= kMaxIn) {
            // counts of at most 8 fit 4 slices; k > 8 can never be reached
            SlicedCount4 cnt;
#pragma unroll
            for (uint32_t i0 = 0; i0 < kMaxIn; i0 += 4) {
                uint64_t v[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    if (i0 + j < n) v[j] = strip_row(col, in[i0 + j]);
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    if (i0 + j < n) cnt.add(i0 + j >= off ? ~v[j] : v[j]);
            }
            return kk > 8 ? 0ull : cnt.ge(kk);
        }
        SlicedCount cnt;
        cnt.clear();
        for (uint32_t i = 0; i < n; ++i) {
            const uint64_t x = strip_row(col, in[i]);
            cnt.add(i >= off ? ~x : x, nbits);
        }
        return cnt.ge(kk);
    }
    uint64_t acc = (op == MCG_AND || op == MCG_NAND) ? kAllOnes : 0ull;
    if (n <= kMaxIn) {
#pragma unroll
        for (uint32_t i0 = 0; i0 < kMaxIn; i0 += 4) {
            uint64_t v[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (i0 + j < n) v[j] = strip_row(col, in[i0 + j]);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                if (i0 + j < n) {
                    const uint64_t x = i0 + j >= off ? ~v[j] : v[j];
                    if (op == MCG_OR || op == MCG_NOR) acc |= x;
                    else if (op == MCG_AND || op == MCG_NAND) acc &= x;
                    else if (op == MCG_XOR) acc ^= x;
                    else acc = x;
                }
            }
        }
    } else {
        for (uint32_t i = 0; i < n; ++i) {
            uint64_t x = strip_row(col, in[i]);
            if (i >= off) x = ~x;
            if (op == MCG_OR || op == MCG_NOR) acc |= x;
            else if (op == MCG_AND || op == MCG_NAND) acc &= x;
            else if (op == MCG_XOR) acc ^= x;
            else acc = x;
        }
    }
    return (op == MCG_NAND || op == MCG_NOR || op == MCG_NOT) ? ~acc : acc;
}

template <int PF, int MINB>
__global__ void __launch_bounds__(kStripThreads, MINB) k_strip(StripArgs a) {
    extern __shared__ unsigned long long s_ones[];
    __shared__ unsigned long long s_strip;
    const uint32_t lane = threadIdx.x & 31u;
    if (a.tally_in_smem)
        for (uint32_t i = threadIdx.x; i < a.n_tally; i += blockDim.x) s_ones[i] = 0;
    const uint64_t gwarp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    uint64_t *col = a.scratch + gwarp * (uint64_t)a.rows * kStripLanes + lane;
    col[(uint64_t)(a.rows - 1) * kStripLanes] = 0;
    const uint64_t n_strips = (a.word_count + kStripThreads - 1) / kStripThreads;
    for (;;) {
        __syncthreads();  // s_strip is free again (and the tally counters are zeroed)
        if (threadIdx.x == 0) s_strip = atomicAdd(a.queue, 1ull);
        __syncthreads();
        const unsigned long long strip = s_strip;
        if (strip >= n_strips) break;
        const uint64_t wl = strip * kStripThreads + threadIdx.x;
        const bool valid = wl < a.word_count;
        const WordCtx ctx = make_word_ctx((uint32_t)(a.word_begin + wl));
        uint32_t e = 0, gq = 0;
#pragma unroll 1
        for (uint32_t sg = 0; sg < a.n_segments; ++sg) {
            const uint2 end = a.segment[sg];
#pragma unroll 1
            for (; e < end.x; ++e) {
                const uint4 r = a.be[e];
                uint64_t v;
                if (r.w != 0) v = kAllOnes;
                else if (r.z == 0) v = 0;
                else v = be_word_tab<PF>(r.y, ctx, GlobalTable{a.table + (uint64_t)e * kEventTableStride}, r.z);
                strip_row(col, r.x) = v;
            }
            // no gate of a group reads another, so the loads of a whole group
            // are in flight together and its outputs are stored after them
#pragma unroll 1
            for (; gq < end.y; ++gq) {
                const uint4 h = a.groups[2 * gq];
                if (h.x >> 24) {
                    const uint4 f = a.ginfo[h.z];
                    const uint64_t r = strip_gate(a, col, f.w);
                    strip_row(col, f.x) = r;
                    strip_gate_tally(a, s_ones, f, r, valid, lane);
                    continue;
                }
                const uint32_t cnt = h.x & 0xFFu, maxn = (h.x >> 8) & 0xFFFFu;
                const uint4 *rec = reinterpret_cast<const uint4 *>(a.gin + h.y);
                uint64_t acc[kStripGroup] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 2
                for (uint32_t sl = 0; sl < maxn; ++sl) {
                    const uint4 rr = rec[sl];
                    acc[0] |= strip_in(col, rr.x);
                    acc[1] |= strip_in(col, rr.y);
                    acc[2] |= strip_in(col, rr.z);
                    acc[3] |= strip_in(col, rr.w);
                }
                const uint4 out = a.groups[2 * gq + 1];
                uint32_t pc[kStripGroup];
#pragma unroll
                for (uint32_t j = 0; j < kStripGroup; ++j) {
                    const uint64_t r = ((h.w >> j) & 1u) ? ~acc[j] : acc[j];
                    pc[j] = valid && j < cnt ? (uint32_t)__popcll(r) : 0u;
                    const uint32_t node = j == 0 ? out.x : j == 1 ? out.y : j == 2 ? out.z : out.w;
                    if (j < cnt) strip_row(col, node) = r;
                }
                // tallies: two gates' warp sums (at most 32 x 64 each) per 32-bit
                // reduction, then lane j adds gate j's sum to its tally slots
                const uint32_t s01 = __reduce_add_sync(0xFFFFFFFFu, pc[0] | (pc[1] << 16));
                const uint32_t s23 = __reduce_add_sync(0xFFFFFFFFu, pc[2] | (pc[3] << 16));
                if (lane < cnt) {
                    const uint4 f = a.ginfo[h.z + lane];
                    const uint32_t c = ((lane < 2 ? s01 : s23) >> (16 * (lane & 1u))) & 0xFFFFu;
                    if (f.z && c)
                        for (uint32_t t = 0; t < f.z; ++t) strip_tally(a, s_ones, a.tally_list[f.y + t], c);
                }
            }
        }
        for (uint32_t j = 0; j < a.n_be_tally; ++j) {
            const uint2 t = a.be_tally[j];
            const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, valid ? (uint32_t)__popcll(strip_row(col, t.x)) : 0u);
            if (lane == 0 && c) strip_tally(a, s_ones, t.y, c);
        }
    }
    __syncthreads();
    if (a.tally_in_smem)
        for (uint32_t i = threadIdx.x; i < a.n_tally; i += blockDim.x)
            if (s_ones[i]) atomicAdd(&a.ones[i], s_ones[i]);
}

// Tile kernel (fused mode, trees whose live node words fit in shared memory): a
// block evaluates 32 sample words (lane = word) of every needed node at a
// time, the whole pass in one launch.  Its warps share out the events of a
// segment (small trees: of the tree), then the gates of each of its layers.
// Nothing but the counters leaves the SM, an event's
// table entries are made by the warp that samples it (18 lanes, one product
// each: 1.5 % of the sampling), and a pass spreads over events x words, so
// that 4,096 words of a small tree already keep every SM busy where the
// interpreter had 16 blocks.  1,024 threads per SM in all (64 registers each),
// in as many blocks as the tile's size allows: one block's layers run under
// the sampling of another.  Bound by the sampler's multiplies (0.86 of the
// register-only sampler; the rest is gate work and the last, partly filled
// round of events).  262,221 words of the 200-event tree: 2.00 ms, the
// interpreter 2.67 ms; 233,937 words of a 1,030-event tree in segments 9.1 ms
// and 13.9; 4,096 words of a 60-event tree: 18 us of kernel where the
// staged pipeline ran nine launches.
// An input record's word: x, or its complement.
__device__ __forceinline__ uint64_t tile_in(const uint64_t *col, uint32_t rec) {
    const uint64_t x = *reinterpret_cast<const uint64_t *>(reinterpret_cast<const unsigned char *>(col) + (rec & ~1u));
    return x ^ (uint64_t)(-(int64_t)(rec & 1u));
}

// An event's table entries in shared memory, two to a 16-byte load.
struct SharedTable {
    const uint4 *tab;
    __device__ __forceinline__ uint2 operator()(int g) const {
        const uint4 q = tab[g >> 1];
        return g & 1 ? make_uint2(q.z, q.w) : make_uint2(q.x, q.y);
    }
};

template <int NT, int PF>
__global__ void __launch_bounds__(NT, 1024 / NT) k_tile(const __grid_constant__ TileArgs a) {
    constexpr uint32_t kWarps = NT / 32;
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ uint4 s_tab[kWarps][kEventTableStride / 2];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t *col = smem + lane;
    unsigned long long *s_ones = reinterpret_cast<unsigned long long *>(smem + (size_t)a.n_slots * kTileLanes);
    if (a.tally_in_smem)
        for (uint32_t i = threadIdx.x; i < a.n_tally; i += NT) s_ones[i] = 0;
    if (warp == 0) col[(a.n_slots - 1) * kTileLanes] = 0;  // the empty input
    __syncthreads();
    // one warp per tallied node and tile: the shared counters need no atomics
    auto add = [&](uint32_t t, uint32_t c) {
        if (a.tally_in_smem) s_ones[t] += c;
        else atomicAdd(&a.ones[t], (unsigned long long)c);
    };
    const uint64_t tiles = (a.word_count + kTileLanes - 1) / kTileLanes;
    for (uint32_t it = 0; it < a.n_iterations; ++it) {
        const uint32_t t3 = (a.iteration_first + it + 1u) << 6;
        for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const uint64_t wl = tile * kTileLanes + lane;
            const bool valid = wl < a.word_count;
            const WordCtx ctx = make_word_ctx((uint32_t)(a.word_begin + wl));
            uint32_t e_begin = 0, l = 0;
            for (uint32_t sg = 0; sg < a.n_segments; ++sg) {
                const uint2 end = a.segment[sg];
#pragma unroll 1
                for (uint32_t e = e_begin + warp; e < end.x; e += kWarps) {
                    const uint4 r = a.be[e];
                    uint64_t v;
                    if (r.w & 1u) {
                        v = kAllOnes;
                    } else if (r.z == 0) {
                        v = 0;
                    } else {
                        __syncwarp();  // the last event's entries have been read
                        if (lane < (uint32_t)kEventTableStride)
                            event_table_entry(r.x, t3, (int)lane, reinterpret_cast<uint2 *>(s_tab[warp])[lane]);
                        __syncwarp();
                        v = be_word_tab<PF>(r.y, ctx, SharedTable{s_tab[warp]}, r.z);
                    }
                    col[r.w >> 1] = v;
                }
                __syncthreads();
                for (; l < end.y; ++l) {
                    const uint32_t gates_end = a.layer[l + 1];
                    for (uint32_t i = a.layer[l] + warp; i < gates_end; i += kWarps) {
                        const uint4 m = a.gates[i];
                        const uint32_t kind = m.x & 3u;
                        const uint2 *in = reinterpret_cast<const uint2 *>(a.in + m.y);
                        const uint32_t pairs = m.z & 0xFFFFu;
                        uint64_t r = 0;
                        if (kind == kTileOr) {
#pragma unroll 2
                            for (uint32_t j = 0; j < pairs; ++j) {
                                const uint2 s = in[j];
                                r |= tile_in(col, s.x) | tile_in(col, s.y);
                            }
                        } else if (kind == kTileXor) {
                            for (uint32_t j = 0; j < pairs; ++j) {
                                const uint2 s = in[j];
                                r ^= tile_in(col, s.x) ^ tile_in(col, s.y);
                            }
                        } else {
                            const uint32_t kk = (m.x >> 8) & 0xFFu, nbits = (m.x >> 16) & 0xFu;
                            if (nbits <= 4) {  // at most 15 inputs
                                SlicedCount4 cnt;
                                for (uint32_t j = 0; j < pairs; ++j) {
                                    const uint2 s = in[j];
                                    cnt.add(tile_in(col, s.x));
                                    cnt.add(tile_in(col, s.y));
                                }
                                r = kk > 15 ? 0ull : cnt.ge(kk);
                            } else {
                                SlicedCount cnt;
                                cnt.clear();
                                for (uint32_t j = 0; j < pairs; ++j) {
                                    const uint2 s = in[j];
                                    cnt.add(tile_in(col, s.x), nbits);
                                    cnt.add(tile_in(col, s.y), nbits);
                                }
                                r = cnt.ge(kk);
                            }
                        }
                        if (m.x & 4u) r = ~r;
                        col[m.z >> 16] = r;
                        const uint32_t nt = m.x >> 20;  // tallies of the gate: one (its index), or a list
                        if (nt) {
                            const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, valid ? (uint32_t)__popcll(r) : 0u);
                            if (lane == 0 && c) {
                                if (nt == 1) add(m.w, c);
                                else
                                    for (uint32_t j = 0; j < nt; ++j) add(a.tally_list[m.w + j], c);
                            }
                        }
                    }
                    __syncthreads();
                }
                e_begin = end.x;
            }
            for (uint32_t j = warp; j < a.n_be_tally; j += kWarps) {
                const uint2 t = a.be_tally[j];
                const uint32_t c =
                    __reduce_add_sync(0xFFFFFFFFu, valid ? (uint32_t)__popcll(col[t.x * kTileLanes]) : 0u);
                if (lane == 0 && c) add(t.y, c);
            }
            if (a.n_be_tally) __syncthreads();  // the words are free again
        }
    }
    __syncthreads();
    if (a.tally_in_smem)
        for (uint32_t i = threadIdx.x; i < a.n_tally; i += NT)
            if (s_ones[i]) atomicAdd(&a.ones[i], s_ones[i]);
}

// Register-only sampler: thread w generates words (e, w) for n_events events
// (event e: pdag_idx + 1 = e + 3, event_idx + 1 = e + 1, table row e) and
// xors them together; one store per thread keeps the work alive.  Same
// sampler code as the product's sampling kernel.
template <int PF>
__global__ void __launch_bounds__(256) k_sampler_peak(uint32_t n_events, uint64_t n_words,
                                                      const uint2 *__restrict__ table, uint64_t *__restrict__ sink) {
    const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= n_words) return;
    const WordCtx ctx = make_word_ctx((uint32_t)w);
    uint64_t x = 0;
    for (uint32_t e = 0; e < n_events; ++e) {
        const uint32_t thr = 0x01000000u + (e * 0x9E3779B9u >> 8);  // spread of probabilities
        x ^= be_word_tab<PF>(e + 1u, ctx, GlobalTable{table + (uint64_t)e * kEventTableStride}, thr);
    }
    sink[w] = x;
}

// Register-only sampler of the shared batch path: thread w generates words
// (e, w) of K instances per Philox evaluation (be_words, the sampler the
// batch interpreters call) and xors them together.
template <int PF, int K>
__global__ void __launch_bounds__(256) k_sampler_peak_shared(uint32_t n_events, uint64_t n_words,
                                                             uint64_t *__restrict__ sink) {
    const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= n_words) return;
    const WordCtx ctx = make_word_ctx((uint32_t)w);
    uint64_t x = 0;
    for (uint32_t e = 0; e < n_events; ++e) {
        uint32_t thr[K];
        uint64_t out[K];
#pragma unroll
        for (int k = 0; k < K; ++k) thr[k] = 0x01000000u + ((e * 0x9E3779B9u + (uint32_t)k * 0x7F4A7C15u) >> 8);
        be_words<PF, K>(e + 3u, e + 1u, ctx, 2u << 6, thr, out);
#pragma unroll
        for (int k = 0; k < K; ++k) x ^= out[k];
    }
    sink[w] = x;
}

// Event table for k_sampler_peak's synthetic events.
static __global__ void __launch_bounds__(256) k_peak_table(uint32_t n_events, uint32_t t3, uint2 *__restrict__ table) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)n_events * kEventTableStride) return;
    const uint32_t e = (uint32_t)(i / kEventTableStride);
    event_table_entry(e + 3u, t3, (int)(i % kEventTableStride), table[i]);
}

}  // namespace dev
}  // namespace mcg
