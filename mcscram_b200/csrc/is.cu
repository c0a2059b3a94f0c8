// is.cu -- importance-sampling engine (include/mcg_is.h).
//
// Sampling and gate evaluation are the staged pipeline's kernels, fed with
// the proposal thresholds; a weights kernel queued after each chunk's gate
// phase turns every top-event hit into an FP64 likelihood ratio.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <string>
#include <vector>

#include "engine_internal.hpp"
#include "error.hpp"
#include "mcg_is.h"
#include "smem_limit.hpp"
#include "staged_run.hpp"

namespace {

#define MCG_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t err_ = (call);                                                              \
        if (err_ != cudaSuccess) {                                                              \
            cudaGetLastError(); /* reported here, and not by the next launch's check */         \
            return mcg::fail(err_ == cudaErrorMemoryAllocation ? MCG_ERR_OOM : MCG_ERR_CUDA,    \
                             std::string(#call) + ": " + cudaGetErrorString(err_));             \
        }                                                                                       \
    } while (0)

constexpr int kWeightThreads = 128;  // four warps: four neighbouring words are one 32-byte sector of a row

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}

__device__ void atomic_max_double(double *addr, double v) {
    unsigned long long *a = reinterpret_cast<unsigned long long *>(addr);
    unsigned long long old = *a;
    while (__longlong_as_double((long long)old) < v) {
        const unsigned long long prev = atomicCAS(a, old, (unsigned long long)__double_as_longlong(v));
        if (prev == old) break;
        old = prev;
    }
}

// Likelihood ratios: many independent trees in one graph (or one tree), tree
// k owning basic events [be_begin[k], be_begin[k + 1]) and tallied root
// root_row[k].  One warp per (tree, word), see k_is_weights.
// A pass may draw its words from several proposals (components c = 0 ..
// n_comp - 1, component 0 the main one, c taking a share pi_c of the
// words).  Every sample is then weighted by the balance heuristic of
// multiple importance sampling, whichever component drew it:
//     w = p(x) / sum_c pi_c q_c(x),
//     log w = -logsumexp_c(ln pi_c - log(p / q_c)(x)),
// which is unbiased and keeps w <= p / (pi_c q_c) for every c.
constexpr int kMaxComponents = 8;

// ---------------------------------------------------------------------------
// Cut-set component: importance sampling of a union of rare events over the
// cut sets of a tree (the "at least one event" mixture of Owen, Maximov &
// Chertkov).  For a tree of AND / OR / ATLEAST / pass-through gates without
// shared nodes, S(node) is the sum over its minimal cut sets of the product
// of their events' probabilities (event: p; AND: product; OR: sum; ATLEAST
// k: k-th elementary symmetric sum of the children's S).  A sample picks a
// cut set C with probability prod_{i in C} p_i / S(top) by descending from
// the top (OR: one child with probability S(child)/S(OR); AND: every child;
// ATLEAST: a k-subset with probability proportional to the product of its
// members' S), forces C's events to fail and draws the other events at their
// nominal probabilities.  Its density is
//     q(x) = p(x) N(x) / S(top),
// N(x) = the number of minimal cut sets contained in x (event: x_i; AND:
// product; OR: sum; ATLEAST: k-th elementary symmetric sum of the children's
// counts), so log(p/q) = log S(top) - log N(x); N(x) >= 1 wherever the top
// event fires, which bounds the weight of this component by S(top) / pi.
//
// Basic events read by several gates (gates still read by one gate each)
// are drawn first, z_i = 1 with a proposal probability r_i, and the tree is
// then one of private events with the shared ones as constants: S_z(node)
// uses z_i for a shared event's leaves (a leaf with z_i = 1 holds the empty
// cut set), and the descent and forcing above run on that conditioned tree
// (no forcing when S_z(top) = 0: z leaves no cut set).  The density is
//     q(x) = r(z) p(x_private) N(x) / S_z(top),
// with N(x) the same count (a shared leaf counts x_i), so
//     log(p/q) = log(p(z) / r(z)) + log S_z(top) - log N(x).
// S_z differs from S_0 (all z_i = 0) only above the shared leaves with
// z_i = 1, so S_z is evaluated by a descent that enters only those gates and
// takes S_0 for every other one.  In the forcing kernel a gate is entered
// when its range of shared-leaf occurrences (the leaves in depth-first
// order) holds one of the sample's z_i = 1 occurrences; in the weights
// kernel when its companion gate fired (an OR over the shared leaves below
// the gate, evaluated with the other gates).
constexpr int kCutStack = 256;     // descent stack of one sample (node ids)
constexpr int kCountDepth = 32;    // frames of the N(x) and S_z evaluations
constexpr int kCutMaxK = 8;        // ATLEAST thresholds the count frames hold
constexpr int kCutMaxN = 32;       // ATLEAST fan-in above shared leaves (suffix sums in registers)
constexpr int kZOcc = 32;          // z_i = 1 occurrences a sample keeps for pruning (more: no pruning)
constexpr uint32_t kNoNode = 0xFFFFFFFFu;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {  // the SplitMix64 finaliser
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Uniform in [0, 1) number `draw` of the stream `base`.
__device__ __forceinline__ double cut_uniform(uint64_t base, uint32_t draw) {
    return (double)(mix64(base + (uint64_t)draw * 0x9E3779B97F4A7C15ull) >> 11) * 0x1.0p-53;
}

struct CutArgs {
    uint64_t *buf;
    uint64_t W, stride, word_begin;  // words of the chunk, row stride of buf
    uint32_t n_inst, n_be;
    const uint32_t *root_row;      // per tree
    const uint4 *gate;             // per gate: op | k << 8, in_begin, in_count, table offset
    const uint32_t *inputs;
    const double *S;               // per node: S_0
    const double *tab;             // OR: cumulative S_0(child) / S_0(OR); ATLEAST: E[j][r] = e_r(S_j..S_n-1)
    const unsigned char *tree_ok;  // per tree: drawn by the component (else its samples stay nominal)
    const unsigned char *shared;   // per basic event: read by several gates
    const uint2 *gate_occ;         // per gate: [lo, hi) of the shared-leaf occurrences below it
    const uint32_t *z_begin;       // per tree: its shared events are z_event[z_begin[k] .. z_begin[k + 1])
    const uint32_t *z_event;
    const uint64_t *q;             // per basic event: a shared event z_i = 1 with probability q / 2^32
    const uint32_t *z_occ_begin;   // per shared event: its occurrences z_occ[z_occ_begin[j] .. z_occ_begin[j + 1])
    const uint32_t *z_occ;
    uint64_t seed;
    unsigned int *error;
};

// Values of gates already evaluated for one sample: open addressing over
// kMemoSlots node ids with at most kMemoProbes probes, so a full table costs
// a few loads per lookup (a sample that sets many shared events evaluates
// hundreds of gates); values that find no slot are simply not kept.  A bit
// per slot says that it holds a value, so a new sample clears 32 bytes: the
// table is per-thread memory, and clearing its keys moved 2.2 GB of it
// through DRAM for 629,000 samples (1.5 ms of the kernel's 1.6).
constexpr int kMemoBits = 8;
constexpr int kMemoSlots = 1 << kMemoBits;
constexpr int kMemoProbes = 8;
struct GateMemo {
    uint32_t key[kMemoSlots];
    double val[kMemoSlots];
    uint32_t used[kMemoSlots / 32];
    __device__ void clear() {
#pragma unroll
        for (int i = 0; i < kMemoSlots / 32; ++i) used[i] = 0;
    }
    __device__ bool holds(uint32_t h) const { return (used[h >> 5] >> (h & 31u)) & 1u; }
    __device__ bool get(uint32_t node, double &v) {
        uint32_t h = (node * 2654435761u) >> (32 - kMemoBits);
        for (int i = 0; i < kMemoProbes; ++i, h = (h + 1) & (kMemoSlots - 1)) {
            if (!holds(h)) return false;
            if (key[h] == node) {
                v = val[h];
                return true;
            }
        }
        return false;
    }
    __device__ void put(uint32_t node, double v) {
        uint32_t h = (node * 2654435761u) >> (32 - kMemoBits);
        for (int i = 0; i < kMemoProbes; ++i, h = (h + 1) & (kMemoSlots - 1)) {
            if (!holds(h) || key[h] == node) {
                used[h >> 5] |= 1u << (h & 31u);
                key[h] = node;
                val[h] = v;
                return;
            }
        }
    }
};

// The AND / OR / ATLEAST recursion (product, sum, k-th elementary symmetric
// sum) from gate `root`: a basic event x gives leaf(x), a gate x is entered
// when enter(x) holds and gives other(x) otherwise; memo holds values of
// gates evaluated before (the same recursion gives the same value).  Returns
// -1 when the tree is deeper than the frames hold.  The frame being worked
// on (node, next input, accumulator, gate record) stays in registers; only
// the suspended ancestors and the ATLEAST k-subset sums are in local memory.
template <class Leaf, class Enter, class Other>
__device__ double tree_eval(uint32_t root, const uint4 *gate, const uint32_t *inputs, uint32_t n_be, Leaf leaf,
                            Enter enter, Other other, GateMemo &memo) {
    double known;
    if (memo.get(root, known)) return known;
    struct Suspended {
        uint32_t node, j;
        double acc;
    };
    Suspended st[kCountDepth];
    double dp[kCountDepth][kCutMaxK + 1];  // the k-subset sums of an ATLEAST frame at each depth
    int sp = 0;                            // depth of the current frame
    uint32_t node = root, j = 0;
    uint4 g = gate[root - n_be];
    uint32_t op = g.x & 0xFFu, kk = (g.x >> 8) & 0xFFu;
    double acc = op == MCG_AND ? 1.0 : 0.0;
    auto start = [&]() {  // the k-subset sums of a new ATLEAST frame at depth sp
        if (op == MCG_ATLEAST) {
            dp[sp][0] = 1.0;
            for (uint32_t r = 1; r <= kk && r <= (uint32_t)kCutMaxK; ++r) dp[sp][r] = 0.0;
        }
    };
    auto deliver = [&](double v) {
        if (op == MCG_AND) {
            acc *= v;
        } else if (op == MCG_ATLEAST) {
            for (int r = (int)kk; r >= 1; --r) dp[sp][r] += dp[sp][r - 1] * v;
        } else {
            acc += v;
        }
    };
    start();
    for (;;) {
        if (j < g.z) {
            const uint32_t x = inputs[g.y + j++];
            if (x < n_be) {
                deliver(leaf(x));
                continue;
            }
            if (!enter(x)) {
                deliver(other(x));
                continue;
            }
            if (memo.get(x, known)) {
                deliver(known);
                continue;
            }
            if (sp + 1 == kCountDepth) return -1.0;
            st[sp] = Suspended{node, j, acc};
            ++sp;
            node = x;
            j = 0;
            g = gate[x - n_be];
            op = g.x & 0xFFu;
            kk = (g.x >> 8) & 0xFFu;
            acc = op == MCG_AND ? 1.0 : 0.0;
            start();
            continue;
        }
        const double v = op == MCG_ATLEAST ? dp[sp][kk] : acc;
        memo.put(node, v);
        if (sp == 0) return v;
        --sp;
        node = st[sp].node;
        j = st[sp].j;
        acc = st[sp].acc;
        g = gate[node - n_be];
        op = g.x & 0xFFu;
        kk = (g.x >> 8) & 0xFFu;
        deliver(v);
    }
}

// The stream of sample b of word w of tree k.
__device__ __forceinline__ uint64_t cut_base(const CutArgs &a, uint32_t k, uint64_t w, uint32_t b) {
    uint64_t base = mix64(a.seed ^ ((uint64_t)k << 32));
    base = mix64(base ^ (a.word_begin + w));
    return mix64(base ^ (uint64_t)b);
}

// Draws the shared events, kDrawEvents of them and kDrawWords words per
// block: a warp takes a word, lane l its samples l and l + 32, and the two
// ballots of a draw are the event's word.  Every shared event of the tree
// draws from the stream zbase of the sample.  Bound by the two 64-bit hashes
// per lane and draw; drawn inside k_cut_force, one sample per thread, the
// trees with the most shared events held their SMs long after the others
// were done.
constexpr uint32_t kDrawEvents = 32, kDrawWords = 32;
__global__ void __launch_bounds__(256) k_cut_draw(const __grid_constant__ CutArgs a, uint32_t n_z) {
    __shared__ uint64_t s_word[kDrawEvents][kDrawWords + 1];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t j0 = blockIdx.x * kDrawEvents, j1 = min(n_z, j0 + kDrawEvents);
    const uint64_t w0 = (uint64_t)blockIdx.y * kDrawWords;  // at most 2^20 words a chunk
    uint32_t k0 = 0, hi = a.n_inst;  // the tree of j0: z_begin[k0] <= j0 < z_begin[k0 + 1]
    while (hi - k0 > 1) {
        const uint32_t mid = (k0 + hi) / 2;
        if (a.z_begin[mid] <= j0) k0 = mid;
        else hi = mid;
    }
    for (uint32_t i = warp; i < kDrawWords && w0 + i < a.W; i += 8) {
        uint32_t k = k0, first = 0, end = 0;
        uint64_t zbase[2] = {0, 0};
        for (uint32_t j = j0; j < j1; ++j) {
            if (j >= end) {  // the first event, or the first of the next tree that has any
                while (a.z_begin[k + 1] <= j) ++k;
                first = a.z_begin[k];
                end = a.z_begin[k + 1];
#pragma unroll
                for (int h = 0; h < 2; ++h) zbase[h] = mix64(cut_base(a, k, w0 + i, lane + 32u * h) ^ 0x2545F4914F6CDD1Dull);
            }
            const uint64_t add = (uint64_t)(j - first + 1) * 0x9E3779B97F4A7C15ull, thr = a.q[a.z_event[j]];
            const uint32_t lo = __ballot_sync(0xFFFFFFFFu, (mix64(zbase[0] + add) >> 32) < thr);
            const uint32_t up = __ballot_sync(0xFFFFFFFFu, (mix64(zbase[1] + add) >> 32) < thr);
            if (lane == 0) s_word[j - j0][i] = ((uint64_t)up << 32) | lo;
        }
    }
    __syncthreads();
    for (uint32_t j = j0 + warp; j < j1; j += 8)
        if (w0 + lane < a.W) a.buf[(uint64_t)a.z_event[j] * a.stride + w0 + lane] = s_word[j - j0][lane];
}

// One thread per (tree, word, sample): collects the sample's shared events
// (drawn by k_cut_draw), then descends from the tree's top on the conditioned
// tree and ORs the sample's bit into the words of the chosen cut set's
// private events.
__global__ void __launch_bounds__(256) k_cut_force(CutArgs a) {
    const uint64_t item = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= (uint64_t)a.n_inst * a.W * 64) return;
    const uint32_t b = (uint32_t)(item & 63u);
    const uint64_t wi = item >> 6;
    const uint64_t w = wi % a.W;
    const uint32_t k = (uint32_t)(wi / a.W);
    if (!a.tree_ok[k]) return;  // a tree the component cannot draw: nominal samples
    const uint64_t base = cut_base(a, k, w, b);
    uint32_t draw = 0;
    const unsigned long long bit = 1ull << b;
    const uint32_t n_be = a.n_be;
    // the occurrences of the tree's shared events that the sample sets, in
    // the events' order: a warp holds 32 samples of one word, so its lanes
    // read 32 events' words at once and pass on the ones set in any sample
    uint32_t occ[kZOcc];
    int n_occ = 0;
    bool prune = true;
    const uint32_t lane = threadIdx.x & 31u, half = b & 32u;
    const uint32_t z0 = a.z_begin[k], z1 = a.z_begin[k + 1];
    for (uint32_t j0 = z0; j0 < z1; j0 += 32) {
        uint32_t x = 0;
        if (j0 + lane < z1) x = (uint32_t)(a.buf[(uint64_t)a.z_event[j0 + lane] * a.stride + w] >> half);
        for (uint32_t m = __ballot_sync(0xFFFFFFFFu, x != 0); m; m &= m - 1) {
            const int src = __ffs((int)m) - 1;
            if (!((__shfl_sync(0xFFFFFFFFu, x, src) >> lane) & 1u)) continue;
            const uint32_t j = j0 + (uint32_t)src;
            for (uint32_t o = a.z_occ_begin[j]; prune && o < a.z_occ_begin[j + 1]; ++o) {
                if (n_occ == kZOcc) {
                    prune = false;
                    break;
                }
                const uint32_t v = a.z_occ[o];
                int q = n_occ++;
                while (q > 0 && occ[q - 1] > v) {
                    occ[q] = occ[q - 1];
                    --q;
                }
                occ[q] = v;
            }
        }
    }
    // a gate whose subtree holds a z_i = 1 leaf (every gate with shared leaves
    // below when the sample has too many to keep)
    auto affected = [&](uint32_t node) -> bool {
        const uint2 r = a.gate_occ[node - n_be];
        if (r.x >= r.y) return false;
        if (!prune) return true;
        for (int q = 0; q < n_occ; ++q)
            if (occ[q] >= r.x) return occ[q] < r.y;
        return false;
    };
    auto leaf = [&](uint32_t x) -> double {
        return a.shared[x] ? (double)((a.buf[(uint64_t)x * a.stride + w] >> b) & 1ull) : a.S[x];
    };
    auto s0 = [&](uint32_t x) -> double { return a.S[x]; };
    GateMemo memo;
    memo.clear();
    auto sz = [&](uint32_t x) -> double {  // S_z of any node
        if (x < n_be) return leaf(x);
        if (!affected(x)) return a.S[x];
        const double v = tree_eval(x, a.gate, a.inputs, n_be, leaf, affected, s0, memo);
        if (v < 0.0) atomicOr(a.error, 4u);
        return v;
    };
    uint32_t stack[kCutStack];
    int sp = 0;
    const uint32_t root = a.root_row[k];
    if (!(sz(root) > 0.0)) return;  // z leaves no cut set: nominal private events
    stack[sp++] = root;
    while (sp) {
        const uint32_t node = stack[--sp];
        if (node < n_be) {
            if (!a.shared[node])
                atomicOr(reinterpret_cast<unsigned long long *>(a.buf + (uint64_t)node * a.stride + w), bit);
            continue;
        }
        const uint4 g = a.gate[node - n_be];
        const uint32_t op = g.x & 0xFFu, kk = (g.x >> 8) & 0xFFu, n = g.z;
        const uint32_t *in = a.inputs + g.y;
        const double *tab = a.tab + g.w;
        const bool cond = affected(node);
        if (op == MCG_OR) {
            const double u = cut_uniform(base, ++draw);
            uint32_t j = 0;
            if (!cond) {
                while (j + 1 < n && u >= tab[j]) ++j;
            } else {  // shares of S_z: the children's sum, then the first child whose cumulative share passes u
                double cz[kCutMaxN];  // the children's S_z, kept from the sum (wider gates evaluate twice)
                double tot = 0.0;
                for (uint32_t c = 0; c < n; ++c) {
                    const double v = sz(in[c]);
                    if (c < (uint32_t)kCutMaxN) cz[c] = v;
                    tot += v;
                }
                double cum = 0.0;
                for (; j + 1 < n; ++j) {
                    cum += j < (uint32_t)kCutMaxN ? cz[j] : sz(in[j]);
                    if (u * tot < cum) break;
                }
            }
            if (sp == kCutStack) { atomicOr(a.error, 1u); return; }
            stack[sp++] = in[j];
        } else if (op == MCG_ATLEAST) {
            double v[kCutMaxN], E[(kCutMaxN + 1) * (kCutMaxK + 1)];
            const double *Et = tab;
            if (cond) {  // E[j][r] = e_r(S_z of children j .. n - 1)
                if (n > (uint32_t)kCutMaxN) { atomicOr(a.error, 4u); return; }
                for (uint32_t c = 0; c < n; ++c) v[c] = sz(in[c]);
                for (uint32_t r = 0; r <= kk; ++r) E[(uint64_t)n * (kk + 1) + r] = r == 0 ? 1.0 : 0.0;
                for (int c = (int)n - 1; c >= 0; --c)
                    for (uint32_t r = 0; r <= kk; ++r) {
                        double e = E[(uint64_t)(c + 1) * (kk + 1) + r];
                        if (r > 0) e += v[c] * E[(uint64_t)(c + 1) * (kk + 1) + r - 1];
                        E[(uint64_t)c * (kk + 1) + r] = e;
                    }
                Et = E;
            }
            uint32_t r = kk;
            for (uint32_t j = 0; j < n && r > 0; ++j) {
                bool take = n - j == r;
                if (!take) {  // P(take j | r still to take) = S_j E[j+1][r-1] / E[j][r]
                    const double e0 = Et[(uint64_t)j * (kk + 1) + r], e1 = Et[(uint64_t)(j + 1) * (kk + 1) + r - 1];
                    take = cut_uniform(base, ++draw) * e0 < (cond ? v[j] : a.S[in[j]]) * e1;
                }
                if (take) {
                    if (sp == kCutStack) { atomicOr(a.error, 1u); return; }
                    stack[sp++] = in[j];
                    --r;
                }
            }
        } else {  // AND and pass-through gates: every input
            for (uint32_t j = 0; j < n; ++j) {
                if (sp == kCutStack) { atomicOr(a.error, 1u); return; }
                stack[sp++] = in[j];
            }
        }
    }
}

inline uint64_t mix64_host(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

struct IsBatchArgs {
    const uint64_t *buf;
    uint64_t W;                    // row stride of buf
    uint64_t w_begin, w_count;     // the words of this launch
    uint32_t n_inst;
    uint32_t words_per_warp;       // words a warp takes
    uint32_t n_comp;               // 1 .. kMaxComponents
    uint32_t n_be;                 // stride of a[] and C[] between components
    const uint32_t *be_begin;      // n_inst + 1
    const uint32_t *root_row;      // n_inst
    const double *a;               // [n_comp][n_be]
    const double *C;               // [n_comp][n_inst]
    double log_pi[kMaxComponents];
    int cut_comp;                  // component drawn by cut sets, or -1: its log(p/q) is
                                   // C + acc (the shared events' log(p(z) / r(z))) + log S_z - log N(x)
    const double *cut_logS;        // per tree: log S_0(top)
    const uint4 *cut_gate;         // per gate (see CutArgs)
    const double *cut_S;           // per node: S_0
    const unsigned char *cut_tree_ok;  // per tree: drawn by the component (else its density there is p)
    const unsigned char *shared;   // per basic event: read by several gates
    const uint32_t *companion;     // per gate: node of the OR over the shared leaves below it, or kNoNode
    const uint32_t *inputs;
    uint32_t n_be_nodes;           // basic events of the joined graph (node ids below are events)
    unsigned int *error;
    double *sums;                  // per tree: sum w, sum w^2, hits, max log w
    double *weights;               // [n_inst][w_count][64]: the hits' weights for k_is_ce, or null
    double *ce;                    // per event, or null
};

constexpr int kWeightWarps = kWeightThreads / 32;

// The suspended frames of a warp's walk (the same for all of its lanes).
struct WalkFrame {
    uint64_t mask;     // samples of the word that the frame is evaluated for
    uint32_t node, j;  // gate, next input
};

// Values of the recursion of tree_eval for all samples of one word at once:
// lane l evaluates samples l and l + 32 (v[0], v[1]), the warp walks the
// union of the gates its samples enter, so there is no divergence and the
// inputs of a gate are read by 32 lanes at once.  mask holds the samples to
// evaluate; a lane outside a frame's mask carries values nobody reads.
//   COUNT: N(x), entered through fired gates, a leaf gives its own bit; only
//          inputs that fired in some sample of the mask are visited (the
//          others add 0, and multiply an AND that did not fire).
//   else:  S_z, entered through gates whose companion fired, every other
//          input gives S_0 (a shared leaf its bit).
// The order of the inputs, and with it every rounding, is tree_eval's.
// Returns false when the tree is deeper than the frames hold.
template <bool COUNT>
__device__ bool word_eval(const IsBatchArgs &p, const uint64_t *col, uint32_t root, uint64_t root_mask,
                          WalkFrame *stack, double (&v)[2]) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nbn = p.n_be_nodes;
    double st_acc[kCountDepth][2];               // suspended accumulators
    double dp[kCountDepth][kCutMaxK + 1][2];     // the k-subset sums of an ATLEAST frame at each depth
    int sp = 0;
    uint32_t node = root, j = 0;
    uint64_t mask = root_mask;
    uint4 g = p.cut_gate[root - nbn];
    uint32_t op = g.x & 0xFFu, kk = (g.x >> 8) & 0xFFu;
    double acc[2];
    auto start = [&]() {
        acc[0] = acc[1] = op == MCG_AND ? 1.0 : 0.0;
        if (op == MCG_ATLEAST) {
            dp[sp][0][0] = dp[sp][0][1] = 1.0;
            for (uint32_t r = 1; r <= kk && r <= (uint32_t)kCutMaxK; ++r) dp[sp][r][0] = dp[sp][r][1] = 0.0;
        }
    };
    auto deliver = [&](double x0, double x1) {
        if (op == MCG_AND) {
            acc[0] *= x0;
            acc[1] *= x1;
        } else if (op == MCG_ATLEAST) {
            for (int r = (int)kk; r >= 1; --r) {
                dp[sp][r][0] += dp[sp][r - 1][0] * x0;
                dp[sp][r][1] += dp[sp][r - 1][1] * x1;
            }
        } else {
            acc[0] += x0;
            acc[1] += x1;
        }
    };
    auto bit = [&](uint64_t x, int h) -> bool { return (x >> (lane + 32u * h)) & 1ull; };
    // the inputs [base, base + 32) of the current gate, one per lane: node id,
    // the word that says in which samples it is entered (a leaf: fired), S_0
    uint32_t base = 0xFFFFFFFFu, cid = 0, live = 0;
    uint64_t cword = 0;
    double cval = 0.0;
    uint4 cgate = make_uint4(0u, 0u, 0u, 0u);  // a gate input's record, for the walk into it
    auto load = [&](uint32_t b) {
        base = b;
        cword = 0;
        cval = 0.0;
        cid = b + lane < g.z ? p.inputs[g.y + b + lane] : kNoNode;
        if (cid != kNoNode) {
            if (cid >= nbn) cgate = p.cut_gate[cid - nbn];
            if (COUNT) {
                cword = col[(uint64_t)cid * p.W] & mask;
            } else if (cid < nbn) {
                if (p.shared[cid]) cword = col[(uint64_t)cid * p.W] & mask;
                else cval = p.cut_S[cid];
            } else {
                const uint32_t c = p.companion[cid - nbn];
                if (c != kNoNode) cword = col[(uint64_t)c * p.W] & mask;
                cval = p.cut_S[cid];
            }
        }
        live = __ballot_sync(0xFFFFFFFFu, COUNT ? cword != 0 : cid != kNoNode);
    };
    start();
    load(0);
    for (;;) {
        const uint32_t rest = j - base < 32u ? live & (0xFFFFFFFFu << (j - base)) : 0u;
        if (rest) {
            const int s = __ffs((int)rest) - 1;
            j = base + (uint32_t)s + 1u;
            const uint32_t x = __shfl_sync(0xFFFFFFFFu, cid, s);
            const uint64_t xw = __shfl_sync(0xFFFFFFFFu, cword, s);
            if (COUNT) {
                if (x < nbn) {
                    deliver(bit(xw, 0) ? 1.0 : 0.0, bit(xw, 1) ? 1.0 : 0.0);
                    continue;
                }
            } else {
                const double c = __shfl_sync(0xFFFFFFFFu, cval, s);
                if (x < nbn || xw == 0) {
                    // a shared leaf has S_0 = 0, so its bit is all of its value
                    deliver(x < nbn && bit(xw, 0) ? 1.0 : c, x < nbn && bit(xw, 1) ? 1.0 : c);
                    continue;
                }
            }
            if (sp + 1 == kCountDepth) return false;
            if (lane == 0) stack[sp] = WalkFrame{mask, node, j};
            st_acc[sp][0] = acc[0];
            st_acc[sp][1] = acc[1];
            ++sp;
            node = x;
            j = 0;
            mask = xw;
            g.x = __shfl_sync(0xFFFFFFFFu, cgate.x, s);
            g.y = __shfl_sync(0xFFFFFFFFu, cgate.y, s);
            g.z = __shfl_sync(0xFFFFFFFFu, cgate.z, s);
            op = g.x & 0xFFu;
            kk = (g.x >> 8) & 0xFFu;
            start();
            load(0);
            continue;
        }
        if (base + 32u < g.z) {
            j = base + 32u;
            load(j);
            continue;
        }
        double r[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) r[h] = op == MCG_ATLEAST ? dp[sp][kk][h] : acc[h];
        if (sp == 0) {
            v[0] = r[0];
            v[1] = r[1];
            return true;
        }
        // back to the parent: samples that did not enter this gate get its other value
        const double c = COUNT ? 0.0 : p.cut_S[node];
#pragma unroll
        for (int h = 0; h < 2; ++h) r[h] = bit(mask, h) ? r[h] : c;
        --sp;
        __syncwarp();
        const WalkFrame f = stack[sp];
        __syncwarp();
        node = f.node;
        j = f.j;
        mask = f.mask;
        acc[0] = st_acc[sp][0];
        acc[1] = st_acc[sp][1];
        g = p.cut_gate[node - nbn];
        op = g.x & 0xFFu;
        kk = (g.x >> 8) & 0xFFu;
        deliver(r[0], r[1]);
        // more inputs of the parent are read again (from L1: the walk has just been there)
        if (j < g.z) load(j / 32u * 32u);
        else base = (g.z + 31u) / 32u * 32u, live = 0;
    }
}

// One warp per (tree, word): lane l owns samples l and l + 32.  The events'
// words are read 128 rows at a time (row-major, so the warps of a block, which
// take neighbouring words, share their sectors), and only events that fired in
// a sample in which the tree's top event fired touch the FP64 sums, in the
// events' order.  Then the cut-set terms (word_eval), the balance heuristic
// and the weights of the two samples, and the sums of the warp's words reduced
// once per block.  Bound by the walks' instructions (issue slots 45 % busy, the
// rest latency).  16 trees of 55 to 9,956 events with shared events, 2,048
// words, 1.2 million hits: 1.9 ms with k_is_ce's 0.3 ms behind it, where one
// thread per word (or eight), with the 64 samples' sums in local memory, a
// walk per sample and the cross-entropy sums in the same kernel, took 20 ms.
// A word's samples over two or four warps: 1.9 and 2.7 ms (their walks visit
// nearly the same gates), so a word stays with one warp.
template <int NC>
__global__ void __launch_bounds__(kWeightThreads, NC <= 2 ? 8 : 4) k_is_weights(const __grid_constant__ IsBatchArgs p) {
    __shared__ WalkFrame s_stack[kWeightWarps][kCountDepth];
    __shared__ double s_sum[kWeightWarps][4];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t per_block = (uint64_t)kWeightWarps * p.words_per_warp;
    const uint64_t blocks_per_tree = (p.w_count + per_block - 1) / per_block;
    const uint32_t k = (uint32_t)(blockIdx.x / blocks_per_tree);
    const uint64_t first = (blockIdx.x % blocks_per_tree) * per_block;
    const uint32_t b0 = p.be_begin[k], b1 = p.be_begin[k + 1], root = p.root_row[k];
    const bool cut = p.cut_comp >= 0, cut_ok = cut && p.cut_tree_ok[k];
    double lsum = 0.0, lsum2 = 0.0, lhits = 0.0, lmax = -INFINITY;
    for (uint32_t i = 0; i < p.words_per_warp; ++i) {
        const uint64_t wl = first + (uint64_t)i * kWeightWarps + warp;  // the block's warps take neighbouring words
        if (wl >= p.w_count) break;
        const uint64_t *col = p.buf + p.w_begin + wl;
        const uint64_t top = col[(uint64_t)root * p.W];
        if (top == 0) continue;  // uniform across the warp
        double s[NC][2];
#pragma unroll
        for (int c = 0; c < NC; ++c) s[c][0] = s[c][1] = 0.0;
        for (uint32_t e0 = b0; e0 < b1; e0 += 128) {
            uint64_t x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t e = e0 + 32u * u + lane;
                x[u] = e < b1 ? col[(uint64_t)e * p.W] & top : 0ull;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                uint32_t m = __ballot_sync(0xFFFFFFFFu, x[u] != 0);
                if (!m) continue;
                double av[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    av[c] = x[u] && c < (int)p.n_comp ? p.a[(uint64_t)c * p.n_be + e0 + 32u * u + lane] : 0.0;
                for (; m; m &= m - 1) {
                    const int src = __ffs((int)m) - 1;
                    const uint64_t xe = __shfl_sync(0xFFFFFFFFu, x[u], src);
                    const bool f0 = (xe >> lane) & 1ull, f1 = (xe >> (lane + 32u)) & 1ull;
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const double a = __shfl_sync(0xFFFFFFFFu, av[c], src);
                        if (f0) s[c][0] += a;
                        if (f1) s[c][1] += a;
                    }
                }
            }
        }
        double n_cut[2] = {1.0, 1.0}, log_sz[2] = {0.0, 0.0};
        if (cut_ok) {
            log_sz[0] = log_sz[1] = p.cut_logS[k];
            if (root < p.n_be_nodes) {  // the top is an event: one cut set (a shared one's S_z is 1)
                if (p.shared[root]) log_sz[0] = log_sz[1] = 0.0;
            } else {
                if (!word_eval<true>(p, col, root, top, s_stack[warp], n_cut)) n_cut[0] = n_cut[1] = -1.0;
                const uint32_t comp = p.companion[root - p.n_be_nodes];
                const uint64_t ent = comp != kNoNode ? col[(uint64_t)comp * p.W] & top : 0ull;
                if (ent) {  // samples with a shared leaf z_i = 1 below the top: S_z(top)
                    double sz[2] = {0.0, 0.0};
                    if (!word_eval<false>(p, col, root, ent, s_stack[warp], sz)) sz[0] = sz[1] = -1.0;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if ((ent >> (lane + 32u * h)) & 1ull) {
                            if (!(sz[h] > 0.0)) atomicOr(p.error, 2u);
                            log_sz[h] = log(fmax(sz[h], 1e-300));
                        }
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!((top >> (lane + 32u * h)) & 1ull)) continue;
            double lw_cut = 0.0;
            if (cut) {
                double s_cut = 0.0;
#pragma unroll
                for (int c = 0; c < NC; ++c) s_cut = c == p.cut_comp ? s[c][h] : s_cut;
                lw_cut = p.C[(uint64_t)p.cut_comp * p.n_inst + k] + s_cut;
                if (cut_ok) {
                    if (!(n_cut[h] >= 1.0)) atomicOr(p.error, 2u);  // too deep, or a failure without a cut set
                    lw_cut += log_sz[h];
                    if (n_cut[h] > 1.0) lw_cut -= log(n_cut[h]);
                }
            }
            double lw = p.cut_comp == 0 ? lw_cut : p.C[k] + s[0][h];
            if (NC > 1 && p.n_comp > 1) {
                // -logsumexp_c(ln pi_c - log(p/q_c))
                double u[NC], hi = -INFINITY;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    u[c] = -INFINITY;
                    if (c < (int)p.n_comp) {
                        u[c] = p.log_pi[c] -
                               (c == p.cut_comp ? lw_cut : p.C[(uint64_t)c * p.n_inst + k] + s[c][h]);
                        hi = fmax(hi, u[c]);
                    }
                }
                double sum = 0.0;
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (c < (int)p.n_comp) sum += u[c] == hi ? 1.0 : exp(u[c] - hi);
                lw = -(hi + log(sum));
            }
            const double wv = exp(lw);
            if (p.weights) p.weights[((uint64_t)k * p.w_count + wl) * 64u + lane + 32u * h] = wv;
            lsum += wv;
            lsum2 += wv * wv;
            lhits += 1.0;
            lmax = fmax(lmax, lw);
        }
    }
    lsum = warp_sum(lsum);
    lsum2 = warp_sum(lsum2);
    lhits = warp_sum(lhits);
    lmax = warp_max(lmax);
    if (lane == 0) {
        s_sum[warp][0] = lsum;
        s_sum[warp][1] = lsum2;
        s_sum[warp][2] = lhits;
        s_sum[warp][3] = lmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[4] = {0.0, 0.0, 0.0, -INFINITY};
        for (int q = 0; q < kWeightWarps; ++q) {
            t[0] += s_sum[q][0];
            t[1] += s_sum[q][1];
            t[2] += s_sum[q][2];
            t[3] = fmax(t[3], s_sum[q][3]);
        }
        if (t[2] != 0.0) {
            double *out = p.sums + 4ull * k;
            atomicAdd(&out[0], t[0]);
            atomicAdd(&out[1], t[1]);
            atomicAdd(&out[2], t[2]);
            atomic_max_double(&out[3], t[3]);
        }
    }
}

// Cross-entropy numerators, sum over hits of w x_i: one warp per event and
// share of the words, reading the weights k_is_weights left of the samples
// where the event and the top event fired, and one reduction per warp (inside
// the weights kernel it was one per event and 32 words, with an FP64 atomic
// each: 5.4 ms of the 20).  32 U words at a time; bound by the latency of the
// weights, so the words an event fires in often are read four at a time, and few
// events' words are shared out to more warps (launch_weights): 4,096 words of 60
// events at 0.3 take 21 us, 131 a word at a time in shares of 256.
template <int U>
__global__ void __launch_bounds__(kWeightThreads) k_is_ce(const __grid_constant__ IsBatchArgs p, uint32_t n_events) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t e = blockIdx.x * kWeightWarps + (threadIdx.x >> 5);
    if (e >= n_events) return;
    uint32_t lo = 0, hi = p.n_inst;  // the tree: be_begin[lo] <= e < be_begin[lo + 1]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (p.be_begin[mid] <= e) lo = mid;
        else hi = mid;
    }
    const uint64_t *row = p.buf + (uint64_t)e * p.W + p.w_begin;
    const uint64_t *top = p.buf + (uint64_t)p.root_row[lo] * p.W + p.w_begin;
    const double *weights = p.weights + (uint64_t)lo * p.w_count * 64u;
    double c = 0.0;
    const uint64_t step = 32ull * U * gridDim.y;
    for (uint64_t w0 = 32ull * U * blockIdx.y; w0 < p.w_count; w0 += step) {
        uint64_t x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t w = w0 + 32u * u + lane;
            x[u] = w < p.w_count ? row[w] : 0ull;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t w = w0 + 32u * u + lane;
            if (x[u]) x[u] &= top[w];
            // a word with few samples is its lane's; a dense one (an event whose proposal is near 1/2) is read by
            // all lanes together, two weights each
            const bool dense = __popcll(x[u]) > 3;
            uint32_t m = __ballot_sync(0xFFFFFFFFu, dense);
            if (!dense)
                for (uint64_t b = x[u]; b; b &= b - 1)
                    c += weights[w * 64u + (uint32_t)__ffsll((long long)b) - 1u];
            while (m) {
                double v[4][2];
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // past the last dense word: lane 0's, with no sample
                    const int src = m ? __ffs((int)m) - 1 : 0;
                    const uint64_t xe = __shfl_sync(0xFFFFFFFFu, x[u], src) & (m ? ~0ull : 0ull);
                    m &= m - 1;
                    const double *ww = weights + (w0 + 32u * u + (uint32_t)src) * 64u + lane;
                    v[k][0] = (xe >> lane) & 1ull ? ww[0] : 0.0;
                    v[k][1] = (xe >> (lane + 32u)) & 1ull ? ww[32] : 0.0;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    c += v[k][0];
                    c += v[k][1];
                }
            }
        }
    }
    if (!__any_sync(0xFFFFFFFFu, c != 0.0)) return;
    c = warp_sum(c);
    if (lane == 0) {
        if (gridDim.y == 1) p.ce[e] += c;
        else atomicAdd(&p.ce[e], c);
    }
}

// Size of the buffer between the two kernels (behind the engine's first stage
// buffer), for chunks of `words` words: 64 weights per tree and word, `most` in
// all or those of 32 words; longer chunks are taken in several launches.
constexpr uint64_t kHitWeights = 1ull << 27;  // 1 GiB
uint64_t hit_weight_words(uint32_t n_inst, uint64_t words, uint64_t most) {
    return 64ull * n_inst * std::min<uint64_t>(words, std::max<uint64_t>(32, most / (64ull * n_inst)));
}

// create(most): a handle with so many hit weights; with the least of them, and
// without the buffers kept on the device, where there is no room for that.
template <class Create>
mcg_status create_with_room(int device, Create create) {
    const mcg_status st = create(kHitWeights);
    if (st != MCG_ERR_OOM) return st;
    cudaGetLastError();
    mcg_trim_memory(device);
    return create(0);
}

// Queues both kernels for one chunk of W words.
cudaError_t launch_weights(IsBatchArgs p, uint64_t W, uint32_t n_events, uint64_t weight_words, int sms,
                           cudaStream_t s) {
    for (uint64_t at = 0; at < W; at += p.w_count) {
        p.w_begin = at;
        p.w_count = p.ce ? std::min<uint64_t>(W - at, weight_words) : W - at;
        // a warp takes one word, and several where a launch has far more words than the chip runs at once: fewer
        // atomics on a tree's four sums
        const uint64_t words = (uint64_t)p.n_inst * p.w_count;
        p.words_per_warp = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(16, words / ((uint64_t)sms * 64 * 4)));
        const uint64_t per_block = (uint64_t)kWeightWarps * p.words_per_warp;
        const uint32_t blocks = (uint32_t)(p.n_inst * ((p.w_count + per_block - 1) / per_block));
        if (p.n_comp == 1) k_is_weights<1><<<blocks, kWeightThreads, 0, s>>>(p);
        else if (p.n_comp == 2) k_is_weights<2><<<blocks, kWeightThreads, 0, s>>>(p);
        else if (p.n_comp <= 4) k_is_weights<4><<<blocks, kWeightThreads, 0, s>>>(p);
        else k_is_weights<kMaxComponents><<<blocks, kWeightThreads, 0, s>>>(p);
        if (p.ce && n_events) {
            const uint32_t eb = (n_events + kWeightWarps - 1) / kWeightWarps;
            // shares of at most 256 words: the events whose proposal is near 1/2 read every word and would be a
            // long tail (16 trees of 55 to 9,956 events, 2,048 words: 0.31 ms, 0.75 with 1,024 words); of as few as
            // 32 where the events do not give every SM 16 warps
            uint32_t split = 1;
            while (p.w_count / split > 256 ||
                   (p.w_count / split > 32 && (uint64_t)n_events * split < 16ull * (uint64_t)sms))
                split *= 2;
            (p.w_count / split < 128 ? k_is_ce<1> : k_is_ce<4>)<<<dim3(eb, split), kWeightThreads, 0, s>>>(p, n_events);
        }
        const cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

// Inputs of a run from its proposal thresholds, one block per (tree,
// component): the sampler's table beq, the log-ratio terms at the quantised
// probabilities
//     a_i = ln(p_i / q_i) - l_i,  l_i = ln((1 - p_i) / (1 - q_i)),
// and the tree's constant C = sum_i l_i (threads take events at a fixed
// stride and are summed in a fixed order: the same thresholds give the same
// C).  Component 0's blocks also reset the tree's sums.  On the device
// because four logarithms per event and component took the host 2 ms for two
// components of 30,000 events, and the terms 24 bytes per event of upload
// where the thresholds are 8.
struct RatioArgs {
    const uint4 *be;               // nominal table {pdag + 1, event + 1, thr lo, thr hi}
    const uint64_t *q;             // [n_comp][n_be]
    const uint32_t *be_begin;      // n_inst + 1
    uint32_t n_be, n_inst;
    int cut_comp;                  // its shared events are drawn by k_cut_draw: the sampler leaves them 0
    const unsigned char *drawn;    // per basic event: such an event (cut_comp >= 0)
    uint4 *beq;                    // [n_comp][n_be]
    double *a, *C;                 // [n_comp][n_be], [n_comp][n_inst]
    double *sums, *ce;             // ce may be null
};

constexpr int kRatioThreads = 256;
__global__ void __launch_bounds__(kRatioThreads) k_ratio_terms(RatioArgs r) {
    __shared__ double s_part[kRatioThreads / 32];
    const uint32_t k = blockIdx.x, c = blockIdx.y;
    const uint32_t b1 = r.be_begin[k + 1];
    const uint64_t row = (uint64_t)c * r.n_be;
    constexpr double kTwo32 = 4294967296.0;
    double l = 0.0;
    for (uint32_t i = r.be_begin[k] + threadIdx.x; i < b1; i += kRatioThreads) {
        const uint4 n = r.be[i];
        const uint64_t tp = ((uint64_t)n.w << 32) | n.z, tq = r.q[row + i];
        const bool zero = (int)c == r.cut_comp && r.drawn[i];
        r.beq[row + i] = make_uint4(n.x, n.y, zero ? 0u : (uint32_t)tq, zero ? 0u : (uint32_t)(tq >> 32));
        double a = 0.0;
        if (tp != 0 && tp < (1ull << 32)) {
            const double p = (double)tp / kTwo32, q = (double)tq / kTwo32;
            const double l1 = log1p(-p) - log1p(-q);
            a = log(p) - log(q) - l1;
            l += l1;
        }
        r.a[row + i] = a;
        if (c == 0 && r.ce) r.ce[i] = 0.0;
    }
    l = warp_sum(l);
    if ((threadIdx.x & 31u) == 0) s_part[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kRatioThreads / 32; ++w) t += s_part[w];
        r.C[(uint64_t)c * r.n_inst + k] = t;
        if (c == 0) {
            double *out = r.sums + 4ull * k;
            out[0] = out[1] = out[2] = 0.0;
            out[3] = -INFINITY;
        }
    }
}

// A proposal threshold must lie in [1, 2^32 - 1], or equal a constant nominal
// one; returns the first event where it does not, or n_be.
uint32_t bad_threshold(const mcg::Graph &g, const uint64_t *q_thr) {
    for (uint32_t i = 0; i < g.n_be; ++i) {
        const uint64_t tp = g.be_threshold[i], tq = q_thr[i];
        const bool fixed = tp == 0 || tp >= (1ull << 32);
        if (fixed ? tq != tp : (tq == 0 || tq >= (1ull << 32))) return i;
    }
    return g.n_be;
}

mcg_status check_thresholds(const mcg::Graph &g, const uint64_t *q_thr) {
    const uint32_t i = bad_threshold(g, q_thr);
    if (i == g.n_be) return MCG_OK;
    return mcg::fail(MCG_ERR_INVALID, "proposal threshold " + std::to_string(i) +
                                          " must lie in [1, 2^32 - 1] (or equal a constant nominal one)");
}

// The engine as it is outside of a run: no hooks, its own event table.
void plain_sampling(mcg_engine *e) {
    e->chunk_hook = nullptr;
    e->sample_hook = nullptr;
    e->d_be_sample = nullptr;
    e->table_iteration = 0xFFFFFFFFu;
}

}  // namespace

struct mcg_is {
    mcg_engine *engine = nullptr;
    uint64_t *d_q = nullptr;     // proposal thresholds
    uint4 *d_be_q = nullptr;     // in the sampler's table layout
    double *d_a = nullptr;       // per-event log-ratio increments
    double *d_sums = nullptr;    // 4 doubles, and behind them
    double *d_ce = nullptr;      // the per-event CE numerators: read back in one copy
    double *d_C = nullptr;       // the constant of the log-ratio
    uint32_t *d_tree = nullptr;  // the one tree of k_is_weights: its events [0, n_be), its root row
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

// Chunk size of the importance-sampling engines when the caller leaves it
// at 0: the staged engine's budget (two chunk buffers of up to 24 GB each),
// but at most 2^17 words per chunk.  A small tree would otherwise take
// 2^20-word chunks of tens of GB that its calls never fill, and these
// engines are created and destroyed as trees converge; large joined graphs
// keep their budget-sized chunks (fewer, fuller launches).
static void default_chunk(const mcg_graph_desc &graph, mcg_run_desc &run) {
    if (run.layered_max_words) return;
    const uint64_t nn = std::max<uint64_t>((uint64_t)graph.n_be + graph.n_gates, 1);
    run.layered_max_words = std::min<uint64_t>(1ull << 17, std::max<uint64_t>(256, (24ull << 30) / (nn * 8)));
}

// Frees everything; keeps the error message a failed create has just set.
static void release_is(mcg_is *is) {
    const std::string keep = mcg::last_error();
    if (is->engine) {
        cudaSetDevice(is->engine->device);
        cudaStreamSynchronize(is->engine->stream);
    }
    cudaFree(is->d_be_q);
    cudaFree(is->d_q);
    cudaFree(is->d_a);
    cudaFree(is->d_sums);
    cudaFree(is->d_C);
    cudaFree(is->d_tree);
    if (is->ev0) cudaEventDestroy(is->ev0);
    if (is->ev1) cudaEventDestroy(is->ev1);
    if (is->engine) mcg_destroy(is->engine);
    delete is;
    mcg::last_error() = keep;
}

// A single-tree handle with so many hit weights (hit_weight_words).
static mcg_status create_is(const mcg_graph_desc *graph, const mcg_run_desc &run, uint64_t most, mcg_is **out) {
    auto is = std::unique_ptr<mcg_is, void (*)(mcg_is *)>(new mcg_is, release_is);
    mcg_status st = mcg::internal::create_with_extra(
        graph, &run, [most](uint64_t words) { return hit_weight_words(1, words, most); }, &is->engine);
    if (st != MCG_OK) return st;
    mcg_engine *e = is->engine;
    const uint32_t nb = e->graph.n_be;
    MCG_CUDA(cudaMalloc((void **)&is->d_be_q, std::max<uint32_t>(nb, 1) * sizeof(uint4)));
    MCG_CUDA(cudaMalloc((void **)&is->d_a, std::max<uint32_t>(nb, 1) * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&is->d_q, std::max<uint32_t>(nb, 1) * sizeof(uint64_t)));
    MCG_CUDA(cudaMalloc((void **)&is->d_sums, (4ull + nb) * sizeof(double)));
    is->d_ce = is->d_sums + 4;
    MCG_CUDA(cudaMalloc((void **)&is->d_C, sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&is->d_tree, 3 * sizeof(uint32_t)));
    const uint32_t tree[3] = {0u, nb, e->graph.tally_nodes[0]};
    MCG_CUDA(cudaMemcpy(is->d_tree, tree, sizeof(tree), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaEventCreate(&is->ev0));
    MCG_CUDA(cudaEventCreate(&is->ev1));
    *out = is.release();
    return MCG_OK;
}

extern "C" {

mcg_status mcg_is_create(const mcg_graph_desc *graph, const mcg_run_desc *run_in, mcg_is **out) {
    mcg::clear_error();
    if (!graph || !out) return mcg::fail(MCG_ERR_INVALID, "graph and out must not be NULL");
    *out = nullptr;
    if (graph->n_tally != 1) return mcg::fail(MCG_ERR_INVALID, "the tally list must hold exactly the top event");
    mcg_run_desc run{};
    if (run_in) run = *run_in;
    run.mode = MCG_MODE_STAGED;
    default_chunk(*graph, run);
    // the entry point's limit, before any of the engine's buffers is taken (a
    // device that does not exist is refused by the engine's creation)
    mcg::DeviceShape prop;
    if (mcg::device_shape(&prop, run.device) != cudaSuccess) cudaGetLastError();
    else if (2ull * graph->n_be * sizeof(double) > prop.sharedMemPerBlockOptin)
        return mcg::fail(MCG_ERR_INVALID, "too many basic events for a single-tree handle (mcg_is_batch_create with one "
                                          "tree takes them)");
    return create_with_room(run.device, [&](uint64_t most) { return create_is(graph, run, most, out); });
}

mcg_status mcg_is_destroy(mcg_is *is) {
    mcg::clear_error();
    if (is) release_is(is);
    return MCG_OK;
}

mcg_status mcg_is_run(mcg_is *is, const uint64_t *q_thr, uint32_t iteration, uint64_t word_begin, uint64_t word_count,
                      mcg_is_result *result, double *ce_num) {
    mcg::clear_error();
    if (!is || !q_thr || !result) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    mcg_engine *e = is->engine;
    const mcg::Graph &g = e->graph;
    const uint32_t nb = g.n_be;
    if (word_begin + word_count > (1ull << 32)) return mcg::fail(MCG_ERR_INVALID, "word range exceeds the counter");
    const mcg_status bad = check_thresholds(g, q_thr);
    if (bad != MCG_OK) return bad;
    MCG_CUDA(cudaSetDevice(e->device));
    MCG_CUDA(cudaMemcpyAsync(is->d_q, q_thr, nb * sizeof(uint64_t), cudaMemcpyHostToDevice, e->stream));
    const bool want_ce = ce_num != nullptr;
    const mcg::AtExit plain_again([e] { plain_sampling(e); });
    e->d_be_sample = is->d_be_q;
    e->table_iteration = 0xFFFFFFFFu;  // the sampler table follows the proposal
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
    IsBatchArgs args{};
    RatioArgs ra{};
    ra.be = e->d_be;
    ra.q = is->d_q;
    ra.be_begin = is->d_tree;
    ra.n_be = nb;
    ra.n_inst = 1;
    ra.cut_comp = -1;
    ra.beq = is->d_be_q;
    ra.a = is->d_a;
    ra.C = is->d_C;
    ra.sums = is->d_sums;
    ra.ce = want_ce ? is->d_ce : nullptr;
    k_ratio_terms<<<1, kRatioThreads, 0, e->stream>>>(ra);
    MCG_CUDA(cudaGetLastError());
    args.n_inst = args.n_comp = 1;
    args.n_be = args.n_be_nodes = nb;
    args.be_begin = is->d_tree;
    args.root_row = is->d_tree + 2;
    args.a = is->d_a;
    args.C = is->d_C;
    args.cut_comp = -1;
    args.sums = is->d_sums;
    args.weights = want_ce ? reinterpret_cast<double *>(e->d_stage_extra) : nullptr;
    args.ce = want_ce ? is->d_ce : nullptr;
    const uint64_t weight_words = e->stage_extra_words / 64u;
    e->chunk_hook = [=](cudaStream_t s, const uint64_t *buf, uint64_t W, uint64_t stride) -> mcg_status {
        IsBatchArgs p = args;
        p.buf = buf;
        p.W = stride;
        const cudaError_t err = launch_weights(p, W, nb, weight_words, sms, s);
        if (err != cudaSuccess) return mcg::fail(MCG_ERR_CUDA, std::string("k_is_weights: ") + cudaGetErrorString(err));
        return MCG_OK;
    };
    MCG_CUDA(cudaEventRecord(is->ev0, e->stream));
    const mcg_status st = mcg::internal::run_staged(e, iteration, 1, word_begin, word_count);
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaEventRecord(is->ev1, e->stream));
    std::vector<double> sums(4ull + (want_ce ? nb : 0));
    MCG_CUDA(cudaMemcpyAsync(sums.data(), is->d_sums, sums.size() * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    MCG_CUDA(cudaStreamSynchronize(e->stream));
    if (want_ce) std::copy(sums.begin() + 4, sums.end(), ce_num);
    float ms = 0;
    MCG_CUDA(cudaEventElapsedTime(&ms, is->ev0, is->ev1));
    std::memset(result, 0, sizeof(*result));
    const double n = (double)word_count * 64.0;
    result->samples = word_count * 64;
    result->hits = (uint64_t)sums[2];
    result->sum_w = sums[0];
    result->sum_w2 = sums[1];
    result->estimate = sums[0] / n;
    const double var = std::max(0.0, sums[1] / n - result->estimate * result->estimate);
    result->std_err = n > 1 ? std::sqrt(var / (n - 1.0)) : 0.0;
    result->rel_err = result->estimate > 0 ? result->std_err / result->estimate : INFINITY;
    result->ess = sums[1] > 0 ? sums[0] * sums[0] / sums[1] : 0.0;
    result->max_log_w = sums[3];
    result->kernel_ms = ms;
    return MCG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Batched importance sampling over many trees joined into one graph.

struct mcg_is_batch {
    mcg_engine *engine = nullptr;
    uint32_t n_inst = 0;
    uint32_t n_comp_cap = 0;             // components the device arrays hold
    std::vector<uint32_t> be_begin;
    uint64_t *d_q = nullptr;             // [n_comp][n_be] proposal thresholds
    uint4 *d_be_q = nullptr;             // [n_comp][n_be] sampler tables
    double *d_a = nullptr;               // [n_comp][n_be]
    double *d_C = nullptr;               // [n_comp][n_inst]
    double *d_sums = nullptr;
    double *d_ce = nullptr;
    uint32_t *d_be_begin = nullptr;
    uint32_t *d_root = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // cut-set component (built on first use)
    bool cut_ready = false;
    uint4 *d_cut_gate = nullptr;
    double *d_cut_S = nullptr, *d_cut_tab = nullptr, *d_cut_logS = nullptr;
    unsigned int *d_cut_error = nullptr;
    // shared basic events of the cut-set component: companion gates appended
    // to the graph at creation (the caller's gates are the first n_gates_in)
    uint32_t n_gates_in = 0;
    bool companions = false;
    std::vector<uint32_t> companion;     // per gate of the caller: its companion node, or kNoNode
    std::vector<unsigned char> shared;   // per basic event
    std::vector<unsigned char> tree_gates_ok;  // per tree: gates the component takes (companions built for it)
    std::vector<unsigned char> tree_ok;  // per tree: the cut-set component draws it (else its samples stay nominal)
    unsigned char *d_tree_ok = nullptr;
    std::vector<uint32_t> z_event;       // shared events, tree by tree
    std::vector<uint64_t> cut_q;         // per run: the component's thresholds
    unsigned char *d_shared = nullptr, *d_drawn = nullptr;
    uint2 *d_gate_occ = nullptr;
    uint32_t *d_companion = nullptr, *d_z_begin = nullptr, *d_z_event = nullptr;
    uint32_t *d_z_occ_begin = nullptr, *d_z_occ = nullptr;
};

namespace {

// Frees everything; keeps the error message a failed create has just set.
void release_batch(mcg_is_batch *b) {
    const std::string keep = mcg::last_error();
    if (b->engine) {
        cudaSetDevice(b->engine->device);
        cudaStreamSynchronize(b->engine->stream);
    }
    cudaFree(b->d_q);
    cudaFree(b->d_be_q);
    cudaFree(b->d_a);
    cudaFree(b->d_C);
    cudaFree(b->d_sums);
    cudaFree(b->d_ce);
    cudaFree(b->d_be_begin);
    cudaFree(b->d_root);
    cudaFree(b->d_cut_gate);
    cudaFree(b->d_cut_S);
    cudaFree(b->d_cut_tab);
    cudaFree(b->d_cut_logS);
    cudaFree(b->d_cut_error);
    for (void *q : {(void *)b->d_tree_ok, (void *)b->d_shared, (void *)b->d_gate_occ, (void *)b->d_companion, (void *)b->d_z_begin,
                    (void *)b->d_z_event, (void *)b->d_z_occ_begin, (void *)b->d_z_occ,
                    (void *)b->d_drawn})
        cudaFree(q);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->engine) mcg_destroy(b->engine);
    mcg::last_error() = keep;
}

// Every gate must read nodes of one tree only, and root k must belong to
// tree k: the owner of each node is propagated from the event ranges.
std::string check_partition(const mcg::Graph &g, const std::vector<uint32_t> &be_begin) {
    const uint32_t n_inst = (uint32_t)be_begin.size() - 1;
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    std::vector<uint32_t> owner(g.n_nodes(), kNone);
    for (uint32_t k = 0; k < n_inst; ++k)
        for (uint32_t i = be_begin[k]; i < be_begin[k + 1]; ++i) owner[i] = k;
    for (uint32_t j = 0; j < g.n_gates; ++j) {
        uint32_t o = kNone;
        for (uint32_t s = 0; s < g.gate_in_count[j]; ++s) {
            const uint32_t x = owner[g.inputs[g.gate_in_begin[j] + s]];
            if (x == kNone) continue;
            if (o != kNone && x != o) return "gate " + std::to_string(j) + " reads nodes of two trees";
            o = x;
        }
        owner[g.n_be + j] = o;
    }
    for (uint32_t k = 0; k < n_inst; ++k) {
        const uint32_t r = g.tally_nodes[k];
        if (owner[r] != k && !(owner[r] == kNone && be_begin[k] == be_begin[k + 1]))
            return "tallied node " + std::to_string(k) + " is not a node of tree " + std::to_string(k);
    }
    return std::string();
}

// Trees the cut-set component can draw: every gate AND / OR / ATLEAST /
// pass-through without complemented inputs and read by one gate at most
// (tree_ok[t]).  For those of them with basic events read by several gates,
// companion gates: for every gate with a shared event's leaf below it, an OR
// over those leaves and over its child gates' companions, appended after the
// caller's gates (the tallies stay the trees' tops).  The weights kernel
// reads a companion's word to see which gates a sample's z_i = 1 leaves
// reach.  Returns whether any companion was added.
struct Augmented {
    std::vector<uint8_t> op;
    std::vector<uint32_t> k, begin, count, neg, inputs;
    std::vector<int32_t> pdag;
    std::vector<uint32_t> companion;  // per caller's gate
    std::vector<unsigned char> tree_ok;
    mcg_graph_desc desc{};
};

bool add_companions(const mcg_graph_desc &d, uint32_t n_inst, const uint32_t *be_begin, Augmented &a) {
    const uint64_t nb = d.n_be, ng = d.n_gates, nn = nb + ng;
    std::vector<uint32_t> fanout(nn, 0), owner(nn, kNoNode);
    for (uint64_t i = 0; i < d.n_inputs; ++i)
        if (d.inputs[i] < nn) ++fanout[d.inputs[i]];
    for (uint32_t t = 0; t < n_inst; ++t)
        for (uint32_t i = be_begin[t]; i < be_begin[t + 1]; ++i) owner[i] = t;
    a.tree_ok.assign(n_inst, 1);
    for (uint64_t j = 0; j < ng; ++j) {
        uint32_t o = kNoNode;
        const bool in_range = (uint64_t)d.gate_in_begin[j] + d.gate_in_count[j] <= d.n_inputs;
        for (uint32_t c = 0; in_range && c < d.gate_in_count[j]; ++c) {
            const uint32_t x = d.inputs[d.gate_in_begin[j] + c];
            if (x < nn && owner[x] != kNoNode) o = owner[x];
        }
        owner[nb + j] = o;
        const uint8_t op = d.gate_op[j];
        if (o != kNoNode && (!in_range || fanout[nb + j] > 1 || d.gate_neg_count[j] ||
                             !(op == MCG_AND || op == MCG_OR || op == MCG_ATLEAST || op == MCG_NULL)))
            a.tree_ok[o] = 0;
    }
    bool any_shared = false;
    for (uint64_t i = 0; i < nb; ++i) any_shared |= fanout[i] > 1 && owner[i] != kNoNode && a.tree_ok[owner[i]];
    a.companion.assign(ng, kNoNode);
    if (!any_shared) return false;
    a.op.assign(d.gate_op, d.gate_op + ng);
    a.k.assign(d.gate_k, d.gate_k + ng);
    a.begin.assign(d.gate_in_begin, d.gate_in_begin + ng);
    a.count.assign(d.gate_in_count, d.gate_in_count + ng);
    a.neg.assign(d.gate_neg_count, d.gate_neg_count + ng);
    a.inputs.assign(d.inputs, d.inputs + d.n_inputs);
    if (d.gate_pdag_idx) a.pdag.assign(d.gate_pdag_idx, d.gate_pdag_idx + ng);
    for (uint64_t j = 0; j < ng; ++j) {
        if (owner[nb + j] == kNoNode || !a.tree_ok[owner[nb + j]]) continue;
        std::vector<uint32_t> in;
        for (uint32_t c = 0; c < d.gate_in_count[j]; ++c) {
            const uint32_t x = d.inputs[d.gate_in_begin[j] + c];
            if (x < nb ? fanout[x] > 1 : (x - nb < j && a.companion[x - nb] != kNoNode))
                in.push_back(x < nb ? x : a.companion[x - nb]);
        }
        if (in.empty()) continue;
        a.companion[j] = (uint32_t)(nb + a.op.size());
        a.op.push_back(MCG_OR);
        a.k.push_back(0);
        a.begin.push_back((uint32_t)a.inputs.size());
        a.count.push_back((uint32_t)in.size());
        a.neg.push_back(0);
        if (d.gate_pdag_idx) a.pdag.push_back(-1);
        a.inputs.insert(a.inputs.end(), in.begin(), in.end());
    }
    a.desc = d;
    a.desc.n_gates = (uint32_t)a.op.size();
    a.desc.gate_op = a.op.data();
    a.desc.gate_k = a.k.data();
    a.desc.gate_in_begin = a.begin.data();
    a.desc.gate_in_count = a.count.data();
    a.desc.gate_neg_count = a.neg.data();
    a.desc.inputs = a.inputs.data();
    a.desc.n_inputs = a.inputs.size();
    a.desc.gate_pdag_idx = d.gate_pdag_idx ? a.pdag.data() : nullptr;
    return true;
}

// A handle over n_inst trees with so many hit weights (hit_weight_words).
mcg_status create_is_batch(const mcg_graph_desc *graph, uint32_t n_inst, const uint32_t *be_begin,
                           const mcg_run_desc &run, uint64_t most, mcg_is_batch **out) {
    auto b = std::unique_ptr<mcg_is_batch, void (*)(mcg_is_batch *)>(new mcg_is_batch, [](mcg_is_batch *x) {
        release_batch(x);
        delete x;
    });
    b->n_inst = n_inst;
    b->be_begin.assign(be_begin, be_begin + n_inst + 1);
    b->n_gates_in = graph->n_gates;
    Augmented aug;
    b->companions = add_companions(*graph, n_inst, be_begin, aug);
    b->companion = aug.companion;
    b->tree_gates_ok = aug.tree_ok;
    mcg_status st = mcg::internal::create_with_extra(
        b->companions ? &aug.desc : graph, &run,
        [n_inst, most](uint64_t words) { return hit_weight_words(n_inst, words, most); }, &b->engine);
    if (st != MCG_OK) return st;
    const mcg::Graph &g = b->engine->graph;
    const std::string bad = check_partition(g, b->be_begin);
    if (!bad.empty()) return mcg::fail(MCG_ERR_INVALID, bad);
    const uint32_t nb = std::max<uint32_t>(g.n_be, 1);
    MCG_CUDA(cudaSetDevice(b->engine->device));
    MCG_CUDA(cudaMalloc((void **)&b->d_ce, nb * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&b->d_sums, 4ull * n_inst * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&b->d_be_begin, (n_inst + 1ull) * sizeof(uint32_t)));
    MCG_CUDA(cudaMalloc((void **)&b->d_root, n_inst * sizeof(uint32_t)));
    MCG_CUDA(cudaMemcpy(b->d_be_begin, be_begin, (n_inst + 1ull) * sizeof(uint32_t), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_root, g.tally_nodes.data(), n_inst * sizeof(uint32_t), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaEventCreate(&b->ev0));
    MCG_CUDA(cudaEventCreate(&b->ev1));
    *out = b.release();
    return MCG_OK;
}

}  // namespace

extern "C" {

mcg_status mcg_is_batch_create(const mcg_graph_desc *graph, uint32_t n_inst, const uint32_t *be_begin,
                               const mcg_run_desc *run_in, mcg_is_batch **out) {
    mcg::clear_error();
    if (!graph || !be_begin || !out) return mcg::fail(MCG_ERR_INVALID, "graph, be_begin and out must not be NULL");
    *out = nullptr;
    if (n_inst == 0) return mcg::fail(MCG_ERR_INVALID, "no trees");
    if (graph->n_tally != n_inst) return mcg::fail(MCG_ERR_INVALID, "the tally list must hold one top event per tree");
    if (be_begin[0] != 0 || be_begin[n_inst] != graph->n_be)
        return mcg::fail(MCG_ERR_INVALID, "be_begin must start at 0 and end at n_be");
    for (uint32_t k = 0; k < n_inst; ++k)
        if (be_begin[k + 1] < be_begin[k]) return mcg::fail(MCG_ERR_INVALID, "be_begin must not decrease");
    mcg_run_desc run{};
    if (run_in) run = *run_in;
    run.mode = MCG_MODE_STAGED;
    default_chunk(*graph, run);
    return create_with_room(run.device,
                            [&](uint64_t most) { return create_is_batch(graph, n_inst, be_begin, run, most, out); });
}

mcg_status mcg_is_batch_destroy(mcg_is_batch *b) {
    mcg::clear_error();
    if (!b) return MCG_OK;
    release_batch(b);
    delete b;
    return MCG_OK;
}

}  // extern "C"

namespace {

// Tables of the cut-set component (see k_cut_force): every gate AND, OR,
// ATLEAST (k <= 8) or pass-through without complemented inputs and read by
// one gate at most; basic events read by several gates are the shared
// events z of their tree (the graph then carries companion gates); S(top) > 0
// for every tree.
mcg_status build_cut_tables(mcg_is_batch *b) {
    const mcg::Graph &g = b->engine->graph;
    const uint32_t nb = g.n_be, ng_all = g.n_gates, ng = b->n_gates_in, nn = g.n_nodes();
    std::vector<uint32_t> fanout(nn, 0), owner(nn, kNoNode);
    for (uint32_t j = 0; j < ng; ++j)
        for (uint32_t c = 0; c < g.gate_in_count[j]; ++c) ++fanout[g.inputs[g.gate_in_begin[j] + c]];
    for (uint32_t t = 0; t < b->n_inst; ++t)
        for (uint32_t i = b->be_begin[t]; i < b->be_begin[t + 1]; ++i) owner[i] = t;
    for (uint32_t j = 0; j < ng; ++j)
        for (uint32_t c = 0; c < g.gate_in_count[j]; ++c) {
            const uint32_t o = owner[g.inputs[g.gate_in_begin[j] + c]];
            if (o != kNoNode) owner[nb + j] = o;
        }
    // Trees the component cannot draw keep nominal samples in its words (their
    // density there is p); it fails only when it can draw none of them.
    std::vector<unsigned char> &ok = b->tree_ok;
    ok.assign(b->n_inst, 1);
    std::string why;
    auto reject = [&](uint32_t node, const std::string &msg) {
        const uint32_t t = owner[node];
        if (t == kNoNode || !ok[t]) return;
        ok[t] = 0;
        if (why.empty()) why = msg;
    };
    // a shared basic event needs its tree's companion gates (built when every gate of the tree qualified)
    for (uint32_t i = 0; i < nb + ng; ++i)
        if (fanout[i] > 1 && owner[i] != kNoNode &&
            (i >= nb || !b->companions || owner[i] >= b->tree_gates_ok.size() || !b->tree_gates_ok[owner[i]]))
            reject(i, "cut-set sampling needs trees: node " + std::to_string(i) + " is read by several gates");
    b->shared.assign(nb, 0);
    for (uint32_t i = 0; i < nb; ++i) b->shared[i] = fanout[i] > 1 && owner[i] != kNoNode && ok[owner[i]];
    // S_0 (shared events at 0) for the tables; S with every event at p for the check
    std::vector<double> S(nn, 0.0), Sp(nn, 0.0), tab;
    std::vector<uint4> gate(std::max<uint32_t>(ng_all, 1), make_uint4(0, 0, 0, 0));
    for (uint32_t i = 0; i < nb; ++i) {
        const uint64_t t = g.be_threshold[i];
        Sp[i] = t >= (1ull << 32) ? 1.0 : (double)t / 4294967296.0;
        S[i] = b->shared[i] ? 0.0 : Sp[i];
    }
    auto elementary = [](const std::vector<double> &v, uint32_t k, std::vector<double> &E) {
        const uint32_t n = (uint32_t)v.size();  // E[j][r] = e_r(v_j, ..., v_{n-1}), j = n .. 0
        E.assign((size_t)(n + 1) * (k + 1), 0.0);
        E[(size_t)n * (k + 1)] = 1.0;
        for (int c = (int)n - 1; c >= 0; --c)
            for (uint32_t r = 0; r <= k; ++r) {
                double e = E[(size_t)(c + 1) * (k + 1) + r];
                if (r > 0) e += v[c] * E[(size_t)(c + 1) * (k + 1) + r - 1];
                E[(size_t)c * (k + 1) + r] = e;
            }
    };
    std::vector<double> vals, valp, E, Ep;
    for (uint32_t j = 0; j < ng; ++j) {
        const uint32_t op = g.gate_op[j], n = g.gate_in_count[j], k = g.gate_k[j] & 0xFFu;
        const uint32_t *in = g.inputs.data() + g.gate_in_begin[j];
        if (g.gate_neg_count[j] || !(op == MCG_AND || op == MCG_OR || op == MCG_ATLEAST || op == MCG_NULL))
            reject(nb + j, "cut-set sampling needs AND/OR/ATLEAST gates without complemented inputs; gate " +
                               std::to_string(j) + " is not one");
        if (op == MCG_ATLEAST && k > (uint32_t)kCutMaxK) reject(nb + j, "cut-set sampling: ATLEAST threshold above 8");
        if (owner[nb + j] == kNoNode || !ok[owner[nb + j]]) continue;  // its tree keeps nominal samples
        gate[j] = make_uint4(op | (k << 8), g.gate_in_begin[j], n, (uint32_t)tab.size());
        vals.assign(n, 0.0);
        valp.assign(n, 0.0);
        for (uint32_t c = 0; c < n; ++c) vals[c] = S[in[c]], valp[c] = Sp[in[c]];
        double v = 0.0, vp = 0.0;
        if (op == MCG_AND) {
            v = vp = 1.0;
            for (uint32_t c = 0; c < n; ++c) v *= vals[c], vp *= valp[c];
        } else if (op == MCG_OR) {
            for (uint32_t c = 0; c < n; ++c) v += vals[c], vp += valp[c];
            double cum = 0.0;
            for (uint32_t c = 0; c < n; ++c) {
                cum += vals[c];
                tab.push_back(v > 0 ? cum / v : 1.0);
            }
        } else if (op == MCG_ATLEAST) {
            elementary(vals, k, E);
            elementary(valp, k, Ep);
            v = E[k];
            vp = Ep[k];
            tab.insert(tab.end(), E.begin(), E.end());
        } else {  // pass-through
            v = n ? vals[n - 1] : 0.0;
            vp = n ? valp[n - 1] : 0.0;
        }
        S[nb + j] = v;
        Sp[nb + j] = vp;
    }
    for (uint32_t j = ng; j < ng_all; ++j)  // companions: never entered by the descent or the evaluations
        gate[j] = make_uint4(MCG_OR, g.gate_in_begin[j], g.gate_in_count[j], 0);
    std::vector<double> logS(b->n_inst, 0.0);
    for (uint32_t t = 0; t < b->n_inst; ++t) {
        if (!ok[t]) continue;
        const double st = Sp[g.tally_nodes[t]];
        if (!(st > 0.0) || !std::isfinite(st)) {
            ok[t] = 0;
            if (why.empty()) why = "cut-set sampling: tree " + std::to_string(t) + " has no cut set";
            continue;
        }
        logS[t] = std::log(S[g.tally_nodes[t]]);  // -inf when every cut set holds a shared event
    }
    // shared-leaf occurrences in depth-first order from every top: each gate's
    // subtree holds the range [lo, hi) of them
    std::vector<uint2> occ_range(std::max<uint32_t>(ng_all, 1), make_uint2(0, 0));
    std::vector<std::vector<uint32_t>> occ_of(nb);
    uint32_t pos = 0;
    for (uint32_t t = 0; t < b->n_inst; ++t) {
        const uint32_t root = g.tally_nodes[t];
        if (root < nb || !ok[t]) continue;
        std::vector<std::pair<uint32_t, uint32_t>> st{{root, 0}};
        occ_range[root - nb].x = pos;
        while (!st.empty()) {
            auto &top = st.back();
            const uint32_t j = top.first - nb;
            if (top.second < g.gate_in_count[j]) {
                const uint32_t x = g.inputs[g.gate_in_begin[j] + top.second++];
                if (x < nb) {
                    if (b->shared[x]) occ_of[x].push_back(pos++);
                } else {
                    occ_range[x - nb].x = pos;
                    st.push_back({x, 0});
                }
            } else {
                occ_range[j].y = pos;
                const uint32_t op = g.gate_op[j];
                if (op == MCG_ATLEAST && occ_range[j].y > occ_range[j].x && g.gate_in_count[j] > (uint32_t)kCutMaxN) {
                    ok[t] = 0;
                    if (why.empty())
                        why = "cut-set sampling: ATLEAST gate " + std::to_string(j) +
                              " above shared events has more than 32 inputs";
                }
                st.pop_back();
            }
        }
    }
    bool any = false;
    for (uint32_t t = 0; t < b->n_inst; ++t) any |= ok[t] != 0;
    if (!any) return mcg::fail(MCG_ERR_INVALID, why.empty() ? std::string("cut-set sampling: no tree qualifies") : why);
    std::vector<uint32_t> z_begin(b->n_inst + 1, 0), z_occ_begin{0}, z_occ;
    b->z_event.clear();
    for (uint32_t t = 0; t < b->n_inst; ++t) {
        z_begin[t] = (uint32_t)b->z_event.size();
        for (uint32_t i = b->be_begin[t]; i < b->be_begin[t + 1]; ++i) {
            if (!b->shared[i] || !ok[t]) continue;
            b->z_event.push_back(i);
            z_occ.insert(z_occ.end(), occ_of[i].begin(), occ_of[i].end());
            z_occ_begin.push_back((uint32_t)z_occ.size());
        }
    }
    z_begin[b->n_inst] = (uint32_t)b->z_event.size();
    std::vector<uint32_t> comp(std::max<uint32_t>(ng, 1), kNoNode);
    if (b->companions) std::copy(b->companion.begin(), b->companion.end(), comp.begin());
    if (tab.empty()) tab.push_back(0.0);
    const uint64_t nz = std::max<uint64_t>(b->z_event.size(), 1);
    if (z_occ.empty()) z_occ.push_back(0);
    MCG_CUDA(cudaMalloc((void **)&b->d_cut_gate, gate.size() * sizeof(uint4)));
    MCG_CUDA(cudaMalloc((void **)&b->d_cut_S, nn * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&b->d_cut_tab, tab.size() * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&b->d_cut_logS, b->n_inst * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&b->d_cut_error, sizeof(unsigned int)));
    MCG_CUDA(cudaMalloc((void **)&b->d_shared, std::max<uint32_t>(nb, 1)));
    MCG_CUDA(cudaMalloc((void **)&b->d_tree_ok, b->n_inst));
    MCG_CUDA(cudaMemcpy(b->d_tree_ok, ok.data(), b->n_inst, cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMalloc((void **)&b->d_gate_occ, occ_range.size() * sizeof(uint2)));
    MCG_CUDA(cudaMalloc((void **)&b->d_companion, comp.size() * sizeof(uint32_t)));
    MCG_CUDA(cudaMalloc((void **)&b->d_z_begin, z_begin.size() * sizeof(uint32_t)));
    MCG_CUDA(cudaMalloc((void **)&b->d_z_event, nz * sizeof(uint32_t)));
    MCG_CUDA(cudaMalloc((void **)&b->d_z_occ_begin, z_occ_begin.size() * sizeof(uint32_t)));
    MCG_CUDA(cudaMalloc((void **)&b->d_z_occ, z_occ.size() * sizeof(uint32_t)));
    std::vector<unsigned char> drawn(std::max<uint32_t>(nb, 1), 0);
    for (uint32_t i : b->z_event) drawn[i] = 1;
    MCG_CUDA(cudaMalloc((void **)&b->d_drawn, drawn.size()));
    MCG_CUDA(cudaMemcpy(b->d_drawn, drawn.data(), drawn.size(), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_cut_gate, gate.data(), gate.size() * sizeof(uint4), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_cut_S, S.data(), nn * sizeof(double), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_cut_tab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_cut_logS, logS.data(), b->n_inst * sizeof(double), cudaMemcpyHostToDevice));
    if (nb) MCG_CUDA(cudaMemcpy(b->d_shared, b->shared.data(), nb, cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_gate_occ, occ_range.data(), occ_range.size() * sizeof(uint2), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_companion, comp.data(), comp.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_z_begin, z_begin.data(), z_begin.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    if (!b->z_event.empty())
        MCG_CUDA(cudaMemcpy(b->d_z_event, b->z_event.data(), b->z_event.size() * sizeof(uint32_t),
                            cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_z_occ_begin, z_occ_begin.data(), z_occ_begin.size() * sizeof(uint32_t),
                        cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemcpy(b->d_z_occ, z_occ.data(), z_occ.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    b->cut_ready = true;
    return MCG_OK;
}

// Device arrays for n_comp components, grown on demand.
mcg_status ensure_components(mcg_is_batch *b, uint32_t n_comp) {
    if (n_comp <= b->n_comp_cap) return MCG_OK;
    const uint64_t nb = std::max<uint32_t>(b->engine->graph.n_be, 1);
    cudaFree(b->d_q);
    cudaFree(b->d_be_q);
    cudaFree(b->d_a);
    cudaFree(b->d_C);
    b->d_q = nullptr;
    b->d_be_q = nullptr;
    b->d_a = b->d_C = nullptr;
    b->n_comp_cap = 0;
    MCG_CUDA(cudaMalloc((void **)&b->d_q, n_comp * nb * sizeof(uint64_t)));
    MCG_CUDA(cudaMalloc((void **)&b->d_be_q, n_comp * nb * sizeof(uint4)));
    MCG_CUDA(cudaMalloc((void **)&b->d_a, n_comp * nb * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&b->d_C, (uint64_t)n_comp * b->n_inst * sizeof(double)));
    b->n_comp_cap = n_comp;
    return MCG_OK;
}

}  // namespace

extern "C" {

mcg_status mcg_is_batch_run(mcg_is_batch *b, const uint64_t *q_thr, uint32_t n_def, const uint64_t *q_def,
                            const uint64_t *words_def, uint64_t words_cutset, const uint64_t *q_cutset,
                            uint32_t iteration, uint64_t word_begin, uint64_t word_count, double *tree_sums,
                            double *ce_num, double *kernel_ms) {
    mcg::clear_error();
    if (!b || !q_thr || !tree_sums) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (n_def + 1 > (uint32_t)kMaxComponents)
        return mcg::fail(MCG_ERR_INVALID, "at most " + std::to_string(kMaxComponents - 1) + " defensive proposals");
    if (n_def && (!q_def || !words_def)) return mcg::fail(MCG_ERR_INVALID, "n_defensive > 0 needs q_defensive and words");
    uint64_t def_total = words_cutset;
    for (uint32_t c = 0; c < n_def; ++c) def_total += words_def[c];
    if (def_total > word_count) return mcg::fail(MCG_ERR_INVALID, "defensive and cut-set words exceed word_count");
    if (words_cutset && n_def + 2 > (uint32_t)kMaxComponents)
        return mcg::fail(MCG_ERR_INVALID, "at most " + std::to_string(kMaxComponents - 2) +
                                              " defensive proposals next to the cut-set component");
    mcg_engine *e = b->engine;
    const mcg::Graph &g = e->graph;
    if (word_begin + word_count > (1ull << 32) || word_begin + word_count < word_begin)
        return mcg::fail(MCG_ERR_INVALID, "word range exceeds the 32-bit sample counter");
    if ((uint64_t)iteration + 2 >= (1ull << 26))
        return mcg::fail(MCG_ERR_INVALID, "iteration exceeds the 26-bit pass counter field");
    const uint32_t n_inst = b->n_inst;
    const uint64_t nb = g.n_be;
    // Components that draw words: the main proposal (if it gets any) and
    // every defensive proposal with words.  A single component needs no mixture.
    std::vector<const uint64_t *> comp_q;
    std::vector<uint64_t> comp_words;
    if (word_count - def_total > 0) {
        comp_q.push_back(q_thr);
        comp_words.push_back(word_count - def_total);
    }
    for (uint32_t c = 0; c < n_def; ++c)
        if (words_def[c]) {
            comp_q.push_back(q_def + (uint64_t)c * nb);
            comp_words.push_back(words_def[c]);
        }
    int cut_comp = -1;
    if (words_cutset) {  // shared events from q_cutset, nominal private events plus a forced cut set per sample
        if (!b->cut_ready) {
            MCG_CUDA(cudaSetDevice(e->device));
            const mcg_status cs = build_cut_tables(b);
            if (cs != MCG_OK) return cs;
        }
        b->cut_q.assign(g.be_threshold.begin(), g.be_threshold.end());
        for (uint32_t i : b->z_event) {
            const uint64_t tp = g.be_threshold[i];
            if (q_cutset && tp != 0 && tp < (1ull << 32)) b->cut_q[i] = q_cutset[i];
        }
        cut_comp = (int)comp_q.size();
        comp_q.push_back(b->cut_q.data());
        comp_words.push_back(words_cutset);
    }
    if (comp_q.empty()) comp_q.push_back(q_thr), comp_words.push_back(0);
    const uint32_t nc = (uint32_t)comp_q.size();
    MCG_CUDA(cudaSetDevice(e->device));
    mcg_status st = ensure_components(b, nc);
    if (st != MCG_OK) return st;
    for (uint32_t c = 0; c < nc; ++c) {
        st = check_thresholds(g, comp_q[c]);
        if (st != MCG_OK) return st;
    }
    for (uint32_t c = 0; c < nc && nb; ++c)
        MCG_CUDA(cudaMemcpyAsync(b->d_q + c * nb, comp_q[c], nb * sizeof(uint64_t), cudaMemcpyHostToDevice, e->stream));
    RatioArgs ra{};
    ra.be = e->d_be;
    ra.q = b->d_q;
    ra.be_begin = b->d_be_begin;
    ra.n_be = (uint32_t)nb;
    ra.n_inst = n_inst;
    ra.cut_comp = cut_comp;
    ra.drawn = b->d_drawn;
    ra.beq = b->d_be_q;
    ra.a = b->d_a;
    ra.C = b->d_C;
    ra.sums = b->d_sums;
    ra.ce = ce_num ? b->d_ce : nullptr;
    k_ratio_terms<<<dim3(n_inst, nc), kRatioThreads, 0, e->stream>>>(ra);
    MCG_CUDA(cudaGetLastError());
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
    IsBatchArgs args{};
    args.n_inst = n_inst;
    args.n_comp = nc;
    args.n_be = (uint32_t)nb;
    args.be_begin = b->d_be_begin;
    args.root_row = b->d_root;
    args.a = b->d_a;
    args.C = b->d_C;
    for (uint32_t c = 0; c < nc; ++c)
        args.log_pi[c] = nc > 1 ? std::log((double)comp_words[c] / (double)word_count) : 0.0;
    args.sums = b->d_sums;
    args.ce = ce_num ? b->d_ce : nullptr;
    args.weights = ce_num ? reinterpret_cast<double *>(e->d_stage_extra) : nullptr;
    const uint64_t weight_words = e->stage_extra_words / (64ull * n_inst);
    args.cut_comp = cut_comp;
    args.cut_logS = b->d_cut_logS;
    args.cut_gate = b->d_cut_gate;
    args.cut_S = b->d_cut_S;
    args.cut_tree_ok = b->d_tree_ok;
    args.shared = b->d_shared;
    args.companion = b->d_companion;
    args.inputs = e->d_inputs;
    args.n_be_nodes = g.n_be;
    args.error = b->d_cut_error;
    if (cut_comp >= 0) MCG_CUDA(cudaMemsetAsync(b->d_cut_error, 0, sizeof(unsigned int), e->stream));
    const mcg::AtExit plain_again([e] { plain_sampling(e); });
    e->chunk_hook = [=](cudaStream_t s, const uint64_t *buf, uint64_t W, uint64_t stride) -> mcg_status {
        IsBatchArgs p = args;
        p.buf = buf;
        p.W = stride;
        const cudaError_t err = launch_weights(p, W, (uint32_t)nb, weight_words, sms, s);
        if (err != cudaSuccess)
            return mcg::fail(MCG_ERR_CUDA, std::string("k_is_weights: ") + cudaGetErrorString(err));
        return MCG_OK;
    };
    MCG_CUDA(cudaEventRecord(b->ev0, e->stream));
    // component c draws the next comp_words[c] words with its own sampler
    // table; it is sampled (and forced) under the gates and weights of the
    // component before it, which wait for memory for most of their time
    // (16 trees, 2,048 words, two components: 6.82 -> 6.45 ms)
    uint64_t off = 0, chunk = 0;
    uint32_t last_comp = 0;
    for (uint32_t c = 0; c < nc; ++c)
        if (comp_words[c]) last_comp = c;
    std::function<mcg_status(cudaStream_t, uint64_t *, uint64_t, uint64_t, uint64_t)> cut_hook;
    if (cut_comp >= 0) {
        CutArgs ca{};
        ca.n_inst = n_inst;
        ca.n_be = g.n_be;
        ca.root_row = b->d_root;
        ca.gate = b->d_cut_gate;
        ca.inputs = e->d_inputs;
        ca.S = b->d_cut_S;
        ca.tab = b->d_cut_tab;
        ca.tree_ok = b->d_tree_ok;
        ca.shared = b->d_shared;
        ca.gate_occ = b->d_gate_occ;
        ca.z_begin = b->d_z_begin;
        ca.z_event = b->d_z_event;
        ca.q = b->d_q + (uint64_t)cut_comp * nb;
        ca.z_occ_begin = b->d_z_occ_begin;
        ca.z_occ = b->d_z_occ;
        ca.seed = mix64_host(((uint64_t)iteration << 32) ^ 0x5bd1e995u);
        ca.error = b->d_cut_error;
        const uint32_t n_z = (uint32_t)b->z_event.size();
        cut_hook = [=](cudaStream_t s, uint64_t *buf, uint64_t W, uint64_t stride, uint64_t wb) -> mcg_status {
            CutArgs x = ca;
            x.buf = buf;
            x.W = W;
            x.stride = stride;
            x.word_begin = wb;
            const uint64_t threads = (uint64_t)x.n_inst * W * 64;
            if (n_z) {
                const dim3 grid((n_z + kDrawEvents - 1) / kDrawEvents, (uint32_t)((W + kDrawWords - 1) / kDrawWords));
                k_cut_draw<<<grid, 256, 0, s>>>(x, n_z);
            }
            k_cut_force<<<(uint32_t)((threads + 255) / 256), 256, 0, s>>>(x);
            const cudaError_t err = cudaGetLastError();
            if (err != cudaSuccess) return mcg::fail(MCG_ERR_CUDA, std::string("k_cut_force: ") + cudaGetErrorString(err));
            return MCG_OK;
        };
    }
    auto add_components = [&]() -> mcg_status {
        for (uint32_t c = 0; c < nc; ++c) {
            if (!comp_words[c]) continue;
            e->d_be_sample = b->d_be_q + c * nb;
            e->table_iteration = 0xFFFFFFFFu;  // the sampler table follows the component
            e->sample_hook = (int)c == cut_comp ? cut_hook : nullptr;
            const mcg_status added =
                mcg::internal::add_staged(e, &chunk, iteration, word_begin + off, comp_words[c], c != last_comp);
            if (added != MCG_OK) return added;
            off += comp_words[c];
        }
        return MCG_OK;
    };
    st = mcg::forked_run([&] { return mcg::internal::fork_staged(e); }, add_components,
                         [&] { return mcg::internal::join_staged(e); });
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaEventRecord(b->ev1, e->stream));
    MCG_CUDA(cudaMemcpyAsync(tree_sums, b->d_sums, 4ull * n_inst * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    if (ce_num && nb)
        MCG_CUDA(cudaMemcpyAsync(ce_num, b->d_ce, nb * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    unsigned int cut_error = 0;
    if (cut_comp >= 0)
        MCG_CUDA(cudaMemcpyAsync(&cut_error, b->d_cut_error, sizeof(unsigned int), cudaMemcpyDeviceToHost, e->stream));
    MCG_CUDA(cudaStreamSynchronize(e->stream));
    if (cut_error & 1u) return mcg::fail(MCG_ERR_STATE, "cut-set descent deeper than its stack (256 nodes)");
    if (cut_error & 2u)
        return mcg::fail(MCG_ERR_STATE, "cut-set count failed (tree deeper than 32 levels, or a failure without "
                                        "a cut set)");
    if (cut_error & 4u)
        return mcg::fail(MCG_ERR_STATE, "cut-set descent above shared events failed (tree deeper than 32 levels)");
    if (kernel_ms) {
        float ms = 0.f;
        MCG_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
        *kernel_ms = ms;
    }
    return MCG_OK;
}

}  // extern "C"
