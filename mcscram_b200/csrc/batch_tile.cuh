// batch_tile.cuh -- the tile kernel of batched instances (batch.cu).
#pragma once
#include "kernels.cuh"

namespace mcg {
namespace dev {

// ---------------------------------------------------------------------------
// Batched instances in tiles.  The instances of a tree differ in their
// thresholds only, so the generator's outputs are made once for up to 16 of
// them.  A work item is (group of instances, 32 words); a block's warps share
// out the (event, half word) pairs, then each layer's (gate, four instances).
// Node words lie in a scratch row per slot, [instance][half][word], private to
// the block and written again by its next item.
//
// For a (event, half word) a warp makes 32 outputs per lane, stages them in
// shared memory and marks the ones below the largest of the group's
// thresholds; only those (a few per lane: probabilities are small) are
// compared with every instance's threshold.  Comparing all outputs with every
// threshold cost the interpreter half of its time at four instances.
// 512 threads, two blocks per SM: one block's gates run under the sampling of
// the other (16 trees of 32 to 6,909 events, 16 draws, 16,384 words: 37.5 ms
// where one block of 1,024 threads took 48.2 and the interpreter 120).  A tree
// is taken in segments of about 96 events and their gates, and rows are used
// again (plan_segments): 107 GB of rows to and from memory in that run and not
// 177; segments of 64, 192 and 384 events are 0.5 to 5 % slower.  Bound by the
// issue of the generator's and the compares' instructions (0.57 of the slots,
// as the sampler alone): that run takes 35.4 ms, 101 instances of the
// 200-event tree on 4,096 words 0.66 ms (0.73 before the segments and the
// compares' adds; the interpreter 2.06).

// Thread (event of a group): its record from the instances' tables.
static __global__ void __launch_bounds__(256) k_batch_records(const BatchTileGroup *__restrict__ groups,
                                                              const uint2 *__restrict__ event,
                                                              const uint32_t *__restrict__ event_node,
                                                              const uint32_t *__restrict__ event_off,
                                                              const BatchTileTree *__restrict__ trees,
                                                              const uint64_t *__restrict__ thr_off,
                                                              const uint64_t *__restrict__ thr,
                                                              uint4 *__restrict__ recs) {
    const BatchTileGroup g = groups[blockIdx.x];
    const uint32_t n_be = trees[g.tree].n_be, off = event_off[g.tree];
    for (uint32_t e = blockIdx.y * blockDim.x + threadIdx.x; e < n_be; e += gridDim.y * blockDim.x) {
        const uint32_t node = event_node[off + e];
        uint32_t t[kTileInstances], most = 0, all = 0;
#pragma unroll
        for (uint32_t k = 0; k < kTileInstances; ++k) {
            const uint64_t x = k < g.size ? thr[thr_off[g.first + k] + node] : 0ull;
            if (x >= (1ull << 32)) all |= 1u << k;
            t[k] = x >= (1ull << 32) ? 0u : (uint32_t)x;
            most = max(most, t[k]);
        }
        uint4 *r = recs + (g.rec_off + e) * kTileRec;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) r[q] = make_uint4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
        const uint2 x = event[off + e];
        r[4] = make_uint4(most, all, x.x, x.y);
    }
}

// acc gets the bit, which it does not hold yet, where v < t.  An add and not
// an or: adds take half the issue time of logic operations.
__device__ __forceinline__ void add_if_below(uint32_t &acc, uint32_t v, uint32_t t, uint32_t bit) {
    asm("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %1, %2;\n\t@p add.u32 %0, %0, %3;\n\t}" : "+r"(acc) : "r"(v), "r"(t), "r"(bit));
}

// The marked outputs of a lane against the first KG thresholds of the record;
// stores the half words of the group's `size` instances.
template <int KG>
__device__ __forceinline__ void batch_compare(const uint4 *__restrict__ rec, uint32_t all, uint32_t marked,
                                              const uint32_t *out, uint32_t size, uint32_t *row) {
    uint32_t t[KG], acc[KG];
#pragma unroll
    for (int q = 0; q < KG / 4; ++q) {
        const uint4 x = rec[q];
        t[4 * q] = x.x;
        t[4 * q + 1] = x.y;
        t[4 * q + 2] = x.z;
        t[4 * q + 3] = x.w;
    }
#pragma unroll
    for (int k = 0; k < KG; ++k) acc[k] = 0;
    for (uint32_t left = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)__popc(marked)); left; --left) {
        // the highest marked output; a lane with none left gets b = -1, whose bit is 0 (PTX shifts clamp)
        const uint32_t b = 31u - (uint32_t)__clz((int)marked);
        uint32_t bit;
        asm("shl.b32 %0, 1, %1;" : "=r"(bit) : "r"(b));
        marked ^= bit;
        const uint32_t v = out[((b & 28u) << 5) + (b & 3u)];
#pragma unroll
        for (int k = 0; k < KG; ++k) add_if_below(acc[k], v, t[k], bit);
    }
    if (all) {
#pragma unroll
        for (int k = 0; k < KG; ++k)
            if ((all >> k) & 1u) acc[k] = 0xFFFFFFFFu;
    }
    if (size == KG) {
#pragma unroll
        for (int k = 0; k < KG; ++k) row[k * 64] = acc[k];
    } else {
#pragma unroll
        for (int k = 0; k < KG; ++k)
            if ((uint32_t)k < size) row[k * 64] = acc[k];
    }
}

__device__ __forceinline__ uint4 tile_in4(const unsigned char *base, uint32_t rec) {
    uint4 x = *reinterpret_cast<const uint4 *>(base + (rec & ~1u));
    const uint32_t f = 0u - (rec & 1u);
    return make_uint4(x.x ^ f, x.y ^ f, x.z ^ f, x.w ^ f);
}

// r |= x ^ f, one three-input operation per 32 bits.
__device__ __forceinline__ void tile_or4(uint4 &r, const uint4 &x, uint32_t f) {
    r = make_uint4(r.x | (x.x ^ f), r.y | (x.y ^ f), r.z | (x.z ^ f), r.w | (x.w ^ f));
}

// An ATLEAST or XOR gate for 32 words of two instances (16 lanes and 16 bytes each).
__device__ __noinline__ uint4 tile_gate4(const uint4 m, const uint2 *__restrict__ in, const unsigned char *base) {
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    if ((m.x & 3u) == kTileXor) {
        for (uint32_t j = 0; j < m.z; ++j) {
            const uint2 s = in[j];
            const uint4 x = tile_in4(base, s.x), y = tile_in4(base, s.y);
            r = make_uint4(r.x ^ x.x ^ y.x, r.y ^ x.y ^ y.y, r.z ^ x.z ^ y.z, r.w ^ x.w ^ y.w);
        }
    } else {
        // counted 64 bits at a time, so that the slices stay in registers
        const uint32_t kk = (m.x >> 8) & 0xFFu, nbits = (m.x >> 16) & 0xFu;
        uint64_t w[2];
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            SlicedCount cnt;
            cnt.clear();
            for (uint32_t j = 0; j < 2 * m.z; ++j) {
                const uint32_t s = reinterpret_cast<const uint32_t *>(in)[j];
                const uint64_t x = *reinterpret_cast<const uint64_t *>(base + (s & ~1u) + 8 * h);
                cnt.add(s & 1u ? ~x : x, nbits);
            }
            const uint64_t g = cnt.ge(kk);
            if (h == 0) w[0] = g;
            else w[1] = g;
        }
        r = make_uint4((uint32_t)w[0], (uint32_t)(w[0] >> 32), (uint32_t)w[1], (uint32_t)(w[1] >> 32));
    }
    return r;
}

static __global__ void __launch_bounds__(kBatchTileThreads, kBatchTileBlocks) k_batch_tile(const __grid_constant__ BatchTileArgs a) {
    constexpr uint32_t kWarps = kBatchTileThreads / 32;
    extern __shared__ __align__(16) unsigned char smem_out[];
    __shared__ uint2 s_tab[kWarps][10];
    __shared__ unsigned long long s_item;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned char *rows = a.scratch + blockIdx.x * a.scratch_stride;
    uint4 *out = reinterpret_cast<uint4 *>(smem_out + warp * kBatchTileOut) + lane;  // [call][lane]
    if (threadIdx.x < kTileRow / 16) reinterpret_cast<uint4 *>(rows)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    const uint32_t t3 = (a.iteration + 1u) << 6;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(a.queue, 1ull);
        __syncthreads();
        const unsigned long long item = s_item;
        if (item >= a.items) break;
        const BatchTileGroup g = a.groups[item / a.tiles];
        const BatchTileTree t = a.trees[g.tree];
        const uint64_t w0 = (item % a.tiles) * kTileLanes;
        const WordCtx ctx = make_word_ctx((uint32_t)(w0 + lane));
        // a lane's 16 bytes of a row: words (4 * lane) % 32 .. + 3 of one half of instance lane / 16
        const uint32_t wl = (4u * lane) & 31u;
        const uint32_t live = a.words - w0 > wl ? (uint32_t)min((unsigned long long)(a.words - w0 - wl), 4ull) : 0u;
        auto count = [&](const uint4 &r, uint32_t k, uint32_t tallies) {
            uint32_t c = (live > 0 ? __popc(r.x) : 0) + (live > 1 ? __popc(r.y) : 0) + (live > 2 ? __popc(r.z) : 0) +
                         (live > 3 ? __popc(r.w) : 0);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
            if ((lane & 15u) == 0 && k < g.size && c) atomicAdd(&a.ones[g.first + k], (unsigned long long)c * tallies);
        };
        const uint32_t quads = (g.size + 3) / 4;
        unsigned char *lane_base = rows + lane * 16u;  // instance lane / 16, and + 512 bytes the two after it
        // a warp's four instances of every gate it takes: from k on
        const uint32_t quad_bits = quads > 2 ? 2u : quads - 1u, k = 4 * (warp & ((1u << quad_bits) - 1u));
        unsigned char *src = lane_base + k * 256u;
        const bool more = k + 2 < g.size;
        uint32_t e_begin = 0, l_begin = 0;
        for (uint32_t sg = 0; sg < t.n_segments; ++sg) {
            const uint2 end = a.segment[t.seg_off + sg];
#pragma unroll 1
            for (uint32_t u = 2 * e_begin + warp; u < 2 * end.x; u += kWarps) {
                const uint32_t half = u & 1u;
                const uint4 *rec = a.recs + (g.rec_off + (u >> 1)) * kTileRec;
                const uint4 r = rec[4];
                uint32_t marked = 0;
                __syncwarp();  // the last pair's entries and outputs have been read
                if (r.x) {
                    if (lane < 9) event_table_entry(r.z, t3, lane < 8 ? (int)(8 * half + lane) : 16, s_tab[warp][lane]);
                    __syncwarp();
                    uint32_t ge = 0;
                    half_word_outputs(
                        r.w, ctx, s_tab[warp][8].x, [&](int c) { return s_tab[warp][c]; },
                        [&](int c, uint32_t o0, uint32_t o1, uint32_t o2, uint32_t o3) {
                            out[c * 32] = make_uint4(o0, o1, o2, o3);
                            ge = shift_in_ge(ge, o3, r.x);
                            ge = shift_in_ge(ge, o2, r.x);
                            ge = shift_in_ge(ge, o1, r.x);
                            ge = shift_in_ge(ge, o0, r.x);
                        });
                    // call c is at nibble 7 - c: reverse the nibbles, and "below" is not ">="
                    ge = ((ge & 0x0F0F0F0Fu) << 4) | ((ge >> 4) & 0x0F0F0F0Fu);
                    marked = ~__byte_perm(ge, 0, 0x0123);
                }
                unsigned char *event_row = rows + (uint64_t)a.event_slot[t.event_off + (u >> 1)] * kTileRow;
                uint32_t *row = reinterpret_cast<uint32_t *>(event_row) + half * 32u + lane;
                const uint32_t *mine = reinterpret_cast<const uint32_t *>(out);
                if (g.size > 8) batch_compare<16>(rec, r.y, marked, mine, g.size, row);
                else if (g.size > 4) batch_compare<8>(rec, r.y, marked, mine, g.size, row);
                else batch_compare<4>(rec, r.y, marked, mine, g.size, row);
            }
            __syncthreads();
            for (uint32_t l = l_begin; l < end.y; ++l) {
                const uint32_t begin = a.layer[t.layer_off + l];
                const uint32_t gates_end = k < g.size ? a.layer[t.layer_off + l + 1] : 0u;
                for (uint32_t i = begin + (warp >> quad_bits); i < gates_end; i += kWarps >> quad_bits) {
                    const uint4 m = a.gates[t.gate_off + i];
                    const uint2 *in = reinterpret_cast<const uint2 *>(a.in + t.in_off + m.y);
                    unsigned char *dst = src + (uint64_t)m.w * kTileRow;
                    uint4 r0 = make_uint4(0u, 0u, 0u, 0u), r1 = r0;
                    if ((m.x & 3u) == kTileOr) {
                        // both pairs of instances at once: eight loads in flight
                        if (more) {
#pragma unroll 2
                            for (uint32_t j = 0; j < m.z; ++j) {
                                const uint2 s = in[j];
                                const uint4 *p = reinterpret_cast<const uint4 *>(src + (s.x & ~1u));
                                const uint4 *q = reinterpret_cast<const uint4 *>(src + (s.y & ~1u));
                                const uint4 p0 = p[0], p1 = p[32], q0 = q[0], q1 = q[32];
                                const uint32_t fp = 0u - (s.x & 1u), fq = 0u - (s.y & 1u);
                                tile_or4(r0, p0, fp);
                                tile_or4(r1, p1, fp);
                                tile_or4(r0, q0, fq);
                                tile_or4(r1, q1, fq);
                            }
                        } else {
#pragma unroll 2
                            for (uint32_t j = 0; j < m.z; ++j) {
                                const uint2 s = in[j];
                                tile_or4(r0, tile_in4(src, s.x), 0u);
                                tile_or4(r0, tile_in4(src, s.y), 0u);
                            }
                        }
                    } else {
                        r0 = tile_gate4(m, in, src);
                        if (more) r1 = tile_gate4(m, in, src + 512);
                    }
                    if (m.x & 4u) {
                        r0 = make_uint4(~r0.x, ~r0.y, ~r0.z, ~r0.w);
                        r1 = make_uint4(~r1.x, ~r1.y, ~r1.z, ~r1.w);
                    }
                    *reinterpret_cast<uint4 *>(dst) = r0;
                    if (more) *reinterpret_cast<uint4 *>(dst + 512) = r1;
                    const uint32_t nt = m.x >> 20;
                    if (nt) {
                        count(r0, k + lane / 16u, nt);
                        if (more) count(r1, k + 2 + lane / 16u, nt);
                    }
                }
                __syncthreads();
            }
            e_begin = end.x;
            l_begin = end.y;
        }
        for (uint32_t u = warp; u < t.n_be_tally * quads; u += kWarps) {
            const uint2 x = a.be_tally[t.be_tally_off + u / quads];
            const uint32_t k = 4 * (u % quads);
            for (uint32_t p = 0; p < 2 && k + 2 * p < g.size; ++p)
                count(*reinterpret_cast<const uint4 *>(lane_base + (uint64_t)x.x * kTileRow + (k + 2 * p) * 256u),
                      k + 2 * p + lane / 16u, x.y);
        }
    }
}

}  // namespace dev
}  // namespace mcg
