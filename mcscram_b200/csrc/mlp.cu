// mlp.cu -- the importance-sampling proposal network (include/mcg_is.h).
//
// 16 features -> 64 -> 64 -> 1, ReLU, sigmoid; BF16 operands, FP32
// accumulation.  Every dense product -- the two hidden layers forward, the
// back-propagated hidden gradient, and the weight and bias gradients -- is a
// tcgen05.mma on the fifth-generation tensor cores with its accumulator in
// tensor memory (TMEM); the output layer (64 -> 1), the sigmoid and the loss
// are per-row work on the CUDA cores.
//
// A CTA of 256 threads works on tiles of 128 rows: TMEM lane r holds row r, and
// threads r and r + 128 (warps w and w + 4 read the same lanes) each take half
// of its units.  Bias, ReLU and the ReLU's derivative are per thread; the
// output dot product runs on from the first thread's half to the second's, in
// the order of the units, and the second computes the row's loss.  Feature rows arrive by bulk copies (cp.async.bulk with an
// mbarrier transaction count), the next tile's while the current one is
// computed.  One elected thread issues the MMAs and commits them to an
// mbarrier the others wait on (bounded waits: a wait that runs out sets an
// error flag the host reads, and the CTA releases its TMEM and returns).
//
// Shared-memory operands use the tensor cores' no-swizzle canonical layout:
// a tile of rows x units (BF16) is stored as 8 x 8 blocks of 128 contiguous
// bytes, line i of a block holding row 8 rb + i's units 8 ub .. 8 ub + 7,
// blocks ordered row-block-major.  The same bytes serve as a K-major operand
// (rows as M, units as K) and as an MN-major one (units as M or N, rows as
// K); only the descriptor's two block strides differ.  The weight gradients
// reduce over rows, so they are products with K = rows whose accumulators
// stay in TMEM across all of a CTA's tiles:
//   G1 = [dH2 | H2]^T [H1 | 1 | dz]  ->  dW2^T, db2 (rows 0..63), dW3 (rows 64..127, column 65)
//   G2 = [dH1 | dH2]^T [X | 1]       ->  dW1^T, db1 (rows 0..63; rows 64..127 unused)
// Each CTA writes one partial gradient and a second kernel sums them in CTA
// order (the same rows give the same gradient bit for bit).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "error.hpp"
#include "mcg_is.h"

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

constexpr int kIn = MCG_MLP_IN;       // 16
constexpr int kHid = MCG_MLP_HIDDEN;  // 64
// parameter offsets (FP32 master layout)
constexpr int kOffW1 = 0;                  // [16][64]
constexpr int kOffB1 = kOffW1 + kIn * kHid;   // [64]
constexpr int kOffW2 = kOffB1 + kHid;         // [64][64]
constexpr int kOffB2 = kOffW2 + kHid * kHid;  // [64]
constexpr int kOffW3 = kOffB2 + kHid;         // [64]
constexpr int kOffB3 = kOffW3 + kHid;         // [1]
constexpr int kParams = kOffB3 + 1;
static_assert(kParams == MCG_MLP_PARAMS, "parameter layout");

typedef __nv_bfloat16 bf16;

// BF16 copies of the weights as the kernels' shared memory holds them (one bulk
// copy brings W1 and W2 in): W1 [hidden][feature] and W2 [out][in] in the
// operand layout below (8 x 8 blocks of 128 bytes), then W3[64].
constexpr int kPackW1 = 0;
constexpr int kPackW2 = kPackW1 + kHid * kIn;
constexpr int kPackW3 = kPackW2 + kHid * kHid;
constexpr int kPackSize = kPackW3 + kHid;
constexpr uint32_t kPackBytes = (uint32_t)kPackW3 * 2u;  // of W1 and W2

// Element (row n, column k) of a packed operand with `cols` columns.
__host__ __device__ constexpr int pack_at(int n, int k, int cols) {
    return ((n >> 3) * (cols >> 3) + (k >> 3)) * 64 + (n & 7) * 8 + (k & 7);
}

// Place of parameter i's BF16 copy, or -1 (biases).
__host__ __device__ constexpr int pack_index(int i) {
    if (i < kOffB1) return kPackW1 + pack_at((i - kOffW1) % kHid, (i - kOffW1) / kHid, kIn);
    if (i >= kOffW2 && i < kOffB2) return kPackW2 + pack_at((i - kOffW2) % kHid, (i - kOffW2) / kHid, kHid);
    if (i >= kOffW3 && i < kOffB3) return kPackW3 + i - kOffW3;
    return -1;
}

constexpr int kTile = 128;     // rows per tile: the MMA's M, TMEM lanes
// 8 warps, warp w reading TMEM lanes 32 (w % 4) .. + 31.  The kernels are a chain of short steps per tile, bound by
// its latency and by the instructions of the row-wise steps at two CTAs per SM (the tensor pipe is busy 18 % of its
// active cycles).  The gradient of 250,000 rows: 50.2 us with one thread per row; 45.8 with two;
// 44.7 with the weight gradients issued by a second thread and waited for on barriers of their own; 35.4 with the
// row-wise steps on BF16 pairs, one add per descriptor and the weights brought in by one bulk copy (2,001 rows, one
// tile per CTA: 14.9 -> 8.0 us).
constexpr int kThreads = 256;
constexpr int kCtasPerSm = 2;  // two CTAs of 256 TMEM columns fill the SM's 512
constexpr uint32_t kTmemCols = 256;
// TMEM columns (FP32 accumulators, 128 lanes each)
constexpr uint32_t kColD1 = 0;    // X W1; later dH2 W2^T
constexpr uint32_t kColD2 = 64;   // H1 W2
constexpr uint32_t kColG1 = 128;  // 80 columns, accumulated over the CTA's tiles
constexpr uint32_t kColG2 = 208;  // 32 columns, accumulated over the CTA's tiles
// units per row of the shared-memory tiles
constexpr int kUnitsX = 32;   // X (16) | 1 | 0 ...            (B of G2, A of layer 1)
constexpr int kUnitsE = 80;   // H1 (64) | 1 | dz | 0 ...      (A of layer 2, B of G1)
constexpr int kUnitsC = 192;  // dH1 (64) | dH2 (64) | H2 (64) (A of dH2 W2^T, G1, G2)
constexpr uint32_t kRowBlockX = kUnitsX / 8 * 128;  // bytes between row blocks
constexpr uint32_t kRowBlockE = kUnitsE / 8 * 128;
constexpr uint32_t kRowBlockC = kUnitsC / 8 * 128;
constexpr uint64_t kWaitNs = 2000000000ull;  // bound of every mbarrier wait (2 s)

struct alignas(128) TcSmem {
    float stage[kTile * kIn];  // the next tile's feature rows as the bulk copy leaves them
    bf16 x[2][kTile * kUnitsX];  // two X tiles: a tile's G2 product may still read one while the next is filled
    bf16 e[kTile * kUnitsE];
    bf16 c[kTile * kUnitsC];
    alignas(128) bf16 w1[kHid * kIn];  // B of layer 1: N = hidden, K = feature (K-major)
    bf16 w2[kHid * kHid];    // right behind w1; B of layer 2: N = out, K = in (K-major); of dH2 W2^T: N = in, K = out (MN-major)
    float b1[kHid], b2[kHid], w3[kHid], w3b[kHid];
    float z[kTile], d[kTile];  // a row's half dot product, its dL/dz
    float red[2][kTile / 32];
    unsigned long long bar_mma, bar_end, bar_rows, bar_w, bar_g1, bar_g2, bar_abort[2];
    uint32_t tmem;
};

// --- PTX wrappers --------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(unsigned long long *bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the phase with the given parity to complete, for kWaitNs at most.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = now_ns();
    while (!mbar_try(bar, parity)) {
        if (now_ns() - t0 > kWaitNs) return false;
    }
    return true;
}

// Bulk copy of `bytes` (a multiple of 16, 16-byte aligned ends) into shared
// memory, completing a transaction on bar.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, unsigned long long *bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// Shared-memory matrix descriptor, no swizzle: lbo = bytes between core
// matrices along K, sbo = bytes between core matrices along M/N.  The high
// word is a constant of the operand, and the K steps of a product only move
// the address field: one add each (made anew per step, the descriptors took
// the issuing thread about 90 clocks per MMA).
struct Desc {
    uint32_t lo, hi;
    __device__ __forceinline__ Desc step(uint32_t bytes) const { return Desc{lo + (bytes >> 4), hi}; }
    __device__ __forceinline__ uint64_t bits() const { return ((uint64_t)hi << 32) | lo; }
};

__device__ __forceinline__ Desc sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return Desc{((addr >> 4) & 0x3FFFu) | (((lbo >> 4) & 0x3FFFu) << 16),
                ((sbo >> 4) & 0x3FFFu) | (1u << 14)};  // version 1 (sm_100)
}

// Instruction descriptor: BF16 A and B, FP32 accumulator, M = 128, N = n;
// a_mn / b_mn select the MN-major form of an operand.
__host__ __device__ constexpr uint32_t idesc(int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTile >> 4) << 24);
}

// D (+)= A B, issued by one thread.
__device__ __forceinline__ void umma(uint32_t d, Desc a, Desc b, uint32_t id, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a.bits()), "l"(b.bits()), "r"(id), "r"((uint32_t)accumulate)
        : "memory");
}

// Arrives on bar once every MMA this thread issued before has completed.
__device__ __forceinline__ void umma_commit(unsigned long long *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

#define MCG_R8(i) "=r"(r[i]), "=r"(r[i + 1]), "=r"(r[i + 2]), "=r"(r[i + 3]), "=r"(r[i + 4]), "=r"(r[i + 5]), \
                  "=r"(r[i + 6]), "=r"(r[i + 7])

// 32 or 16 consecutive FP32 columns of this thread's TMEM lane; the wait is
// in the same statement, so the registers are valid when it returns.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n"
        : MCG_R8(0), MCG_R8(8), MCG_R8(16), MCG_R8(24)
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n"
        : MCG_R8(0), MCG_R8(8)
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
#undef MCG_R8

// --- tile layout ---------------------------------------------------------

// The 16 bytes holding units 8 ub .. 8 ub + 7 of row r in a tile of `units` per row.
template <int Units>
__device__ __forceinline__ uint4 *chunk(bf16 *tile, int r, int ub) {
    return reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(tile) +
                                     ((uint32_t)((r >> 3) * (Units / 8) + ub) << 7) + ((uint32_t)(r & 7) << 4));
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);  // a in the low half (lower unit)
    return *reinterpret_cast<const uint32_t *>(&h);
}

// 0xFFFF in each half of a BF16 pair that is above 0.
__device__ __forceinline__ uint32_t positive2(uint32_t h) {
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
    return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162 *>(&h), zero);
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}

// --- shared steps of the forward and gradient kernels ---------------------

// Biases and W3; the constant zero units of the X and E tiles.  Called by all
// threads before the first barrier; W1 and W2 follow by bulk copy (load_weights).
__device__ void setup_operands(TcSmem &s, const bf16 *__restrict__ pack, const float *__restrict__ params) {
    const int tid = threadIdx.x, i = tid % kHid;
    if (tid < kHid) s.b1[i] = params[kOffB1 + i];
    else if (tid < 2 * kHid) s.b2[i] = params[kOffB2 + i];
    else if (tid < 3 * kHid) s.w3[i] = params[kOffW3 + i];
    else s.w3b[i] = __bfloat162float(pack[kPackW3 + i]);
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    *chunk<kUnitsX>(s.x[tid / kTile], tid % kTile, 3) = zero;  // units 24..31
    if (tid < kTile) *chunk<kUnitsE>(s.e, tid, 9) = zero;      // units 72..79
}

// Thread 0: W1 and W2, completing bar_w; it waits for them before its first MMA.
__device__ __forceinline__ void load_weights(TcSmem &s, const bf16 *__restrict__ pack) {
    bulk_load(s.w1, pack + kPackW1, kPackBytes, &s.bar_w);
}

// TMEM allocation (warp 0) and mbarriers (thread 0); returns after the
// barrier that publishes both.
__device__ uint32_t setup_tmem_and_barriers(TcSmem &s) {
    const int tid = threadIdx.x;
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s.tmem)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(&s.bar_mma, 1);
        mbar_init(&s.bar_end, 1);
        mbar_init(&s.bar_rows, 1);
        mbar_init(&s.bar_w, 1);
        mbar_init(&s.bar_abort[0], 1);
        mbar_init(&s.bar_abort[1], 1);
        mbar_init(&s.bar_g1, 1);
        mbar_init(&s.bar_g2, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    return s.tmem;
}

// Barrier that also agrees on ok across the CTA; a failure anywhere ends the
// tile loop in every thread with ok = false.
#define MCG_SYNC_OR_BREAK()                    \
    if (!__syncthreads_and(ok)) {              \
        ok = false;                            \
        break;                                 \
    }

__device__ void release_tmem(uint32_t tmem) {
    tc_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// Thread 0: the bulk copy of tile `tile`'s feature rows into the stage
// (the copy of the CTA's j-th tile completes phase j of bar_rows).
__device__ __forceinline__ void load_rows(TcSmem &s, const float *__restrict__ feat, uint32_t n, uint32_t tile) {
    const uint32_t row0 = tile * kTile;
    const uint32_t rows = min((uint32_t)kTile, n - row0);
    bulk_load(s.stage, feat + (uint64_t)row0 * kIn, rows * kIn * (uint32_t)sizeof(float), &s.bar_rows);
}

// Row r's eight features of `half` (zero past n) from the stage into X tile xb;
// the first half also writes the ones unit.
__device__ __forceinline__ void rows_to_x(TcSmem &s, int xb, int r, int half, bool valid) {
    const float4 *src = reinterpret_cast<const float4 *>(s.stage + r * kIn + 8 * half);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 a = valid ? src[0] : zero, b = valid ? src[1] : zero;
    bf16 *x = s.x[xb];
    *chunk<kUnitsX>(x, r, half) = make_uint4(pack2(a.x, a.y), pack2(a.z, a.w), pack2(b.x, b.y), pack2(b.z, b.w));
    if (half == 0) *chunk<kUnitsX>(x, r, 2) = make_uint4(valid ? 0x3F80u : 0u, 0u, 0u, 0u);  // unit 16 = 1.0
}

// Thread 0: D1 = X W1 (one K = 16 step) from X tile xb.
__device__ __forceinline__ void issue_layer1(TcSmem &s, uint32_t tmem, int xb) {
    umma(tmem + kColD1, sdesc(smem_addr(s.x[xb]), 128, kRowBlockX), sdesc(smem_addr(s.w1), 128, 2 * 128),
         idesc(kHid, false, false), false);
}

// G2 += [dH1 | dH2]^T [X | 1] for the tile whose X tile is xb and whose dH1,
// dH2 are in the C tile (K = rows, both operands MN-major).
__device__ __forceinline__ void issue_g2(TcSmem &s, uint32_t tmem, int xb, bool accumulate) {
    const Desc a = sdesc(smem_addr(s.c), kRowBlockC, 128), b = sdesc(smem_addr(s.x[xb]), kRowBlockX, 128);
#pragma unroll
    for (int k = 0; k < kTile / 16; ++k)
        umma(tmem + kColG2, a.step(2 * kRowBlockC * k), b.step(2 * kRowBlockX * k), idesc(32, true, true),
             accumulate || k > 0);
}

// G1 += [dH2 | H2]^T [H1 | 1 | d]: K = rows, both operands MN-major.
__device__ __forceinline__ void issue_g1(TcSmem &s, uint32_t tmem, bool accumulate) {
    const Desc a = sdesc(smem_addr(s.c) + 8 * 128, kRowBlockC, 128), b = sdesc(smem_addr(s.e), kRowBlockE, 128);
#pragma unroll
    for (int k = 0; k < kTile / 16; ++k)
        umma(tmem + kColG1, a.step(2 * kRowBlockC * k), b.step(2 * kRowBlockE * k), idesc(80, true, true),
             accumulate || k > 0);
}

// Thread 0: dH2 W2^T into D1's columns: A = dH2 (K-major, K = out), B = W2
// read as N = in, K = out (MN-major).
__device__ __forceinline__ void issue_dh1(TcSmem &s, uint32_t tmem) {
    const Desc a = sdesc(smem_addr(s.c) + 8 * 128, 128, kRowBlockC), b = sdesc(smem_addr(s.w2), (kHid / 8) * 128, 128);
#pragma unroll
    for (int k = 0; k < kHid / 16; ++k)
        umma(tmem + kColD1, a.step(256 * k), b.step(2 * (kHid / 8) * 128 * k), idesc(kHid, false, true), k > 0);
}

// Thread 0: D2 = H1 W2 (four K = 16 steps).
__device__ __forceinline__ void issue_layer2(TcSmem &s, uint32_t tmem) {
    const Desc a = sdesc(smem_addr(s.e), 128, kRowBlockE), b = sdesc(smem_addr(s.w2), 128, (kHid / 8) * 128);
#pragma unroll
    for (int k = 0; k < kHid / 16; ++k)
        umma(tmem + kColD2, a.step(256 * k), b.step(256 * k), idesc(kHid, false, false), k > 0);
}

// H1 = relu(D1 + b1), units 32 half .. + 31 of row r, into the E tile.
__device__ __forceinline__ void epilogue_h1(TcSmem &s, uint32_t t_row, int r, int half) {
    float v[32];
    tmem_ld32(t_row + kColD1 + 32 * half, v);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        float h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = fmaxf(v[8 * g + j] + s.b1[32 * half + 8 * g + j], 0.f);
        *chunk<kUnitsE>(s.e, r, 4 * half + g) = pack8(h);
    }
}

// H2 = relu(D2 + b2), units 32 half .. + 31 of row r, as BF16 pairs into h and,
// with STORE, into the C tile; returns z = H2 . W3 + b3 (BF16 operands, FP32
// sums in unit order) in the second half's threads.  All threads call it: the
// first half's sums cross a barrier.
template <bool STORE>
__device__ __forceinline__ float epilogue_h2(TcSmem &s, uint32_t t_row, int r, int half, float b3, uint32_t (&h)[16]) {
    float v[32];
    tmem_ld32(t_row + kColD2 + 32 * half, v);
#pragma unroll
    for (int j = 0; j < 16; ++j)
        h[j] = pack2(fmaxf(v[2 * j] + s.b2[32 * half + 2 * j], 0.f), fmaxf(v[2 * j + 1] + s.b2[32 * half + 2 * j + 1], 0.f));
    auto dot = [&](float z, const float *w) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            z = fmaf(__uint_as_float(h[j] << 16), w[2 * j], z);
            z = fmaf(__uint_as_float(h[j] & 0xFFFF0000u), w[2 * j + 1], z);
        }
        return z;
    };
    float z = b3;
    if (half == 0) {
        z = dot(z, s.w3b);
        s.z[r] = z;
    }
    if constexpr (STORE) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
            *chunk<kUnitsC>(s.c, r, 16 + 4 * half + g) = make_uint4(h[4 * g], h[4 * g + 1], h[4 * g + 2], h[4 * g + 3]);
    }
    __syncthreads();
    if (half == 1) z = dot(s.z[r], s.w3b + 32);
    return z;
}

// Error exit (a wait ran out), the two threads that issue work: record it, let
// the bulk copies still in flight land (thread 0's: the weights, and the CTA's
// tiles [waited, issued)) and let every MMA the thread issued finish, so that shared memory
// and TMEM are no longer in use when the CTA leaves.
__device__ void on_timeout(TcSmem &s, int *err, int issuer, uint32_t waited, uint32_t issued) {
    atomicExch(err, 1);
    if (issuer == 0) mbar_wait(&s.bar_w, 0);
    for (uint32_t j = waited; j < issued; ++j) mbar_wait(&s.bar_rows, j & 1);
    umma_commit(&s.bar_abort[issuer]);
    mbar_wait(&s.bar_abort[issuer], 0);
}

// q = sigmoid(network(features)) for rows [0, n): persistent CTAs over 128-row tiles.
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    k_mlp_forward(const bf16 *__restrict__ pack, const float *__restrict__ params, const float *__restrict__ feat,
                  uint32_t n, float *__restrict__ q, int *__restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    TcSmem &s = *reinterpret_cast<TcSmem *>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, r = tid % kTile, half = tid / kTile;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    const uint32_t my_tiles = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    setup_operands(s, pack, params);
    const uint32_t tmem = setup_tmem_and_barriers(s);
    const uint32_t t_row = tmem + ((uint32_t)(warp % 4 * 32) << 16);
    const float b3 = params[kOffB3];
    uint32_t issued = 0;  // bulk copies issued (thread 0)
    bool ok = true;
    if (tid == 0) {
        load_weights(s, pack);
        if (my_tiles > 0) load_rows(s, feat, n, blockIdx.x);
        issued = my_tiles > 0 ? 1 : 0;
        ok = mbar_wait(&s.bar_w, 0);
    }
    uint32_t ph = 0, i = 0;
    for (; i < my_tiles; ++i) {
        const uint32_t tile = blockIdx.x + i * gridDim.x;
        const uint32_t row = tile * kTile + r;
        ok = mbar_wait(&s.bar_rows, i & 1) && ok;
        rows_to_x(s, 0, r, half, row < n);
        fence_async_smem();
        tc_before_sync();
        MCG_SYNC_OR_BREAK();
        tc_after_sync();
        if (tid == 0) {
            if (i + 1 < my_tiles) {  // every thread has read the stage
                load_rows(s, feat, n, tile + gridDim.x);
                ++issued;
            }
            issue_layer1(s, tmem, 0);
            umma_commit(&s.bar_mma);
        }
        ok = mbar_wait(&s.bar_mma, ph) && ok;
        ph ^= 1;
        tc_after_sync();
        epilogue_h1(s, t_row, r, half);
        fence_async_smem();
        tc_before_sync();
        MCG_SYNC_OR_BREAK();
        tc_after_sync();
        if (tid == 0) {
            issue_layer2(s, tmem);
            umma_commit(&s.bar_mma);
        }
        ok = mbar_wait(&s.bar_mma, ph) && ok;
        ph ^= 1;
        tc_after_sync();
        uint32_t h[16];
        const float z = epilogue_h2<false>(s, t_row, r, half, b3, h);
        if (ok && half == 1 && row < n) q[row] = 1.f / (1.f + __expf(-z));
        tc_before_sync();  // the next tile's layer 2 overwrites D2 after the next barrier
    }
    ok = __syncthreads_and(ok) != 0;
    if (!ok && tid == 0) on_timeout(s, err, 0, i, issued);
    release_tmem(tmem);
}

// Weighted BCE gradient of rows [0, n): persistent CTAs, CTA b taking tiles
// b, b + gridDim.x, ...; its gradient (kParams floats, then the loss) goes to
// partial[b * (kParams + 1) ..], every entry written once.  Thread 0 issues the
// products the tile's chain waits for, thread kTile (warp 4) the weight
// gradients: a tile's G1 once dH2, H2, H1 and d are published, its G2 with the
// next tile's layer 1 (or after the last tile).  Their commits go to barriers
// of their own, waited for where the operands are written again: G1's (E, and
// the H2 and dH2 units of C) before the next tile's H1, G2's (dH1 and dH2; its
// X tile alternates) before the next tile's dH2.
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    k_mlp_grad(const bf16 *__restrict__ pack, const float *__restrict__ params, const float *__restrict__ feat,
               const float *__restrict__ tgt, const float *__restrict__ wts, float inv_wsum_host,
               const float *__restrict__ inv_wsum_dev, uint32_t n, float *__restrict__ partial, int *__restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    TcSmem &s = *reinterpret_cast<TcSmem *>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = tid % kTile, half = tid / kTile;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    const uint32_t my_tiles = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    setup_operands(s, pack, params);
    const uint32_t tmem = setup_tmem_and_barriers(s);
    const uint32_t t_row = tmem + ((uint32_t)(warp % 4 * 32) << 16);
    const float b3 = params[kOffB3];
    uint32_t issued = 0;  // bulk copies issued (thread 0)
    bool ok = true;
    if (tid == 0) {
        load_weights(s, pack);
        if (my_tiles > 0) load_rows(s, feat, n, blockIdx.x);
        issued = my_tiles > 0 ? 1 : 0;
        ok = mbar_wait(&s.bar_w, 0);
    }
    const float inv_wsum = inv_wsum_dev ? *inv_wsum_dev : inv_wsum_host;
    float loss = 0.f, gb3 = 0.f;
    uint32_t ph = 0, i = 0;
    for (; i < my_tiles; ++i) {
        const uint32_t tile = blockIdx.x + i * gridDim.x;
        const int xb = (int)(i & 1);
        const uint32_t row = tile * kTile + r;
        const bool valid = row < n;
        const float tv = valid ? tgt[row] : 0.f;
        const float wv = valid ? (wts ? wts[row] : 1.f) * inv_wsum : 0.f;
        ok = mbar_wait(&s.bar_rows, i & 1) && ok;
        rows_to_x(s, xb, r, half, valid);  // the X tile tile i - 2 used: its G2 was waited for before tile i - 1's dH2
        fence_async_smem();
        tc_before_sync();
        MCG_SYNC_OR_BREAK();
        tc_after_sync();
        if (tid == 0) {
            if (i + 1 < my_tiles) {  // every thread has read the stage
                load_rows(s, feat, n, tile + gridDim.x);
                ++issued;
            }
            issue_layer1(s, tmem, xb);
            umma_commit(&s.bar_mma);
        } else if (tid == kTile && i > 0) {
            issue_g2(s, tmem, xb ^ 1, i > 1);
            umma_commit(&s.bar_g2);
        }
        ok = mbar_wait(&s.bar_mma, ph) && ok;
        if (i > 0) ok = mbar_wait(&s.bar_g1, (i - 1) & 1) && ok;
        ph ^= 1;
        tc_after_sync();
        epilogue_h1(s, t_row, r, half);
        fence_async_smem();
        tc_before_sync();
        MCG_SYNC_OR_BREAK();
        tc_after_sync();
        if (tid == 0) {
            issue_layer2(s, tmem);
            umma_commit(&s.bar_mma);
        }
        ok = mbar_wait(&s.bar_mma, ph) && ok;
        ph ^= 1;
        tc_after_sync();
        uint32_t h[16];
        const float z = epilogue_h2<true>(s, t_row, r, half, b3, h);
        // dL/dz = w (q - t) / sum w, by the row's second thread; [1, d] into units 64, 65 of E
        float qv = 0.f;
        if (half == 1) {
            float d = 0.f;
            if (valid) {
                qv = 1.f / (1.f + __expf(-z));
                d = wv * (qv - tv);
            }
            gb3 += d;
            s.d[r] = d;
            *chunk<kUnitsE>(s.e, r, 8) = make_uint4(pack2(valid ? 1.f : 0.f, d), 0u, 0u, 0u);
        }
        __syncthreads();
        // dH2 = d W3 where H2 > 0, into units 64..127 of C
        if (i > 0) ok = mbar_wait(&s.bar_g2, (i - 1) & 1) && ok;
        const float d = s.d[r];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            uint32_t q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float *w = s.w3 + 32 * half + 8 * g + 2 * j;
                q[j] = pack2(d * w[0], d * w[1]) & positive2(h[4 * g + j]);
            }
            *chunk<kUnitsC>(s.c, r, 8 + 4 * half + g) = make_uint4(q[0], q[1], q[2], q[3]);
        }
        fence_async_smem();
        tc_before_sync();
        MCG_SYNC_OR_BREAK();
        tc_after_sync();
        if (tid == 0) {
            issue_dh1(s, tmem);
            umma_commit(&s.bar_mma);
        } else if (tid == kTile) {
            issue_g1(s, tmem, i > 0);
            umma_commit(&s.bar_g1);
        }
        if (half == 1 && valid) {  // the loss, while the product runs
            const float qc = fminf(fmaxf(qv, 1e-7f), 1.f - 1e-7f);
            loss -= wv * (tv * __logf(qc) + (1.f - tv) * __logf(1.f - qc));
        }
        ok = mbar_wait(&s.bar_mma, ph) && ok;
        ph ^= 1;
        tc_after_sync();
        // dH1 = D1 where H1 > 0, into units 0..63 of C
        float v[32];
        tmem_ld32(t_row + kColD1 + 32 * half, v);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const uint4 h1 = *chunk<kUnitsE>(s.e, r, 4 * half + g);
            *chunk<kUnitsC>(s.c, r, 4 * half + g) =
                make_uint4(pack2(v[8 * g], v[8 * g + 1]) & positive2(h1.x), pack2(v[8 * g + 2], v[8 * g + 3]) & positive2(h1.y),
                           pack2(v[8 * g + 4], v[8 * g + 5]) & positive2(h1.z),
                           pack2(v[8 * g + 6], v[8 * g + 7]) & positive2(h1.w));
        }
        fence_async_smem();  // published by the next barrier, before this tile's G2 is issued
        tc_before_sync();
    }
    ok = __syncthreads_and(ok) != 0;
    if (ok && i > 0) {
        tc_after_sync();
        if (tid == kTile) {  // its commit covers every G1 and G2 before
            issue_g2(s, tmem, (int)((i - 1) & 1), i > 1);
            umma_commit(&s.bar_end);
        }
        ok = mbar_wait(&s.bar_end, 0);
        ok = __syncthreads_and(ok) != 0;
    }
    float *out = partial + (uint64_t)blockIdx.x * (kParams + 1);
    if (ok) {
        tc_after_sync();
        // row tid of G1: out unit tid of dW2^T (tid < 64), or H2 unit tid - 64 against d; of G2: hidden unit tid of
        // dW1^T.  With no tile the accumulators were never written.
        if (tid < kTile) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float v[32];
                tmem_ld32(t_row + kColG1 + 32 * c, v);
                if (tid < kHid)
#pragma unroll
                    for (int j = 0; j < 32; ++j) out[kOffW2 + (32 * c + j) * kHid + tid] = i ? v[j] : 0.f;
            }
            float w[16], v[32];
            tmem_ld16(t_row + kColG1 + 64, w);
            tmem_ld32(t_row + kColG2, v);
            if (tid < kHid) {
                out[kOffB2 + tid] = i ? w[0] : 0.f;
#pragma unroll
                for (int f = 0; f < kIn; ++f) out[kOffW1 + f * kHid + tid] = i ? v[f] : 0.f;
                out[kOffB1 + tid] = i ? v[16] : 0.f;
            } else {
                out[kOffW3 + tid - kHid] = i ? w[1] : 0.f;
            }
        }
    } else if (tid == 0) {
        on_timeout(s, err, 0, i, issued);
    } else if (tid == kTile) {
        on_timeout(s, err, 1, 0, 0);
    }
    // loss and db3: sums over the rows' second threads
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o);
        gb3 += __shfl_xor_sync(0xFFFFFFFFu, gb3, o);
    }
    if (half == 1 && lane == 0) {
        s.red[0][warp - kTile / 32] = loss;
        s.red[1][warp - kTile / 32] = gb3;
    }
    __syncthreads();
    if (tid == 0) {
        float l = 0.f, g = 0.f;
        for (int w = 0; w < kTile / 32; ++w) {
            l += s.red[0][w];
            g += s.red[1][w];
        }
        out[kOffB3] = g;
        out[kParams] = l;
    }
    release_tmem(tmem);
}

// Sum over the CTAs of partial[b][i] (i = kParams: the loss), in the block's
// threads p < kReduceCols, entry blockIdx.x * kReduceCols + p.  A block of
// 1,024 threads brings 32 entries of all partials into shared memory (ten
// loads in flight per thread), then sums them in a fixed order -- group g's
// partials b = g, g + 8, ..., and the eight sums in g order -- so the same
// partials give the same gradient bit for bit.
constexpr int kReduceCols = 32, kReduceGroups = 8, kReduceThreads = 1024;
__device__ __forceinline__ float reduce_entry(const float *__restrict__ partial, uint32_t blocks) {
    extern __shared__ float s_partial[];  // [blocks][kReduceCols]
    __shared__ float part[kReduceGroups][kReduceCols];
    const int p = threadIdx.x % kReduceCols, g = threadIdx.x / kReduceCols;
    const int i = blockIdx.x * kReduceCols + p;
#pragma unroll 10
    for (uint32_t b = g; b < blocks; b += kReduceThreads / kReduceCols)
        s_partial[b * kReduceCols + p] = i <= kParams ? partial[(uint64_t)b * (kParams + 1) + i] : 0.f;
    __syncthreads();
    if (g < kReduceGroups) {
        float v = 0.f;
        for (uint32_t b = g; b < blocks; b += kReduceGroups) v += s_partial[b * kReduceCols + p];
        part[g][p] = v;
    }
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < kReduceGroups; ++k) t += part[k][p];
    return t;
}

// The gradient (kParams entries) and behind it the loss.
__global__ void __launch_bounds__(kReduceThreads)
    k_mlp_reduce(const float *__restrict__ partial, uint32_t blocks, float *__restrict__ grad) {
    const float t = reduce_entry(partial, blocks);
    const int i = blockIdx.x * kReduceCols + threadIdx.x;
    if (threadIdx.x < kReduceCols && i <= kParams) grad[i] = t;
}

// A training step behind the gradient kernel: the gradient's sum, Adam and the
// BF16 operand copy of each parameter, entry by entry (one launch where the
// sum, Adam and the copy were three: 13.1 -> 9.5 us of a step at 250,000 rows).
__global__ void __launch_bounds__(kReduceThreads)
    k_mlp_step(const float *__restrict__ partial, uint32_t blocks, float *__restrict__ p, float *__restrict__ m,
               float *__restrict__ v, float lr, float b1c, float b2c, bf16 *__restrict__ pack, float *__restrict__ loss) {
    const float gi = reduce_entry(partial, blocks);
    const int i = blockIdx.x * kReduceCols + threadIdx.x;
    if (threadIdx.x >= kReduceCols || i > kParams) return;
    if (i == kParams) {
        *loss = gi;
        return;
    }
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / b1c) / (sqrtf(vi / b2c) + 1e-8f);
    p[i] = pi;
    const int at = pack_index(i);
    if (at >= 0) pack[at] = __float2bfloat16(pi);
}

// 1 / sum of the row weights (FP64, fixed order): kSumBlocks partial sums, then
// their sum.  On the device for many rows: the host's serial sum took 0.3 ms
// of a call with 250,000.
constexpr int kSumBlocks = 64, kSumThreads = 256;
constexpr uint32_t kHostSumRows = 1u << 15;
__global__ void __launch_bounds__(kSumThreads) k_weight_sum(const float *__restrict__ w, uint32_t n,
                                                            double *__restrict__ part) {
    __shared__ double s_part[kSumThreads / 32];
    double t = 0.0;
    for (uint64_t i = (uint64_t)blockIdx.x * kSumThreads + threadIdx.x; i < n; i += (uint64_t)kSumBlocks * kSumThreads)
        t += w[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kSumThreads / 32; ++k) t += s_part[k];
        part[blockIdx.x] = t;
    }
}

__global__ void k_weight_inverse(const double *__restrict__ part, float *__restrict__ inv) {
    double t = 0.0;
    for (int k = 0; k < kSumBlocks; ++k) t += part[k];
    *inv = t > 0.0 ? (float)(1.0 / t) : 0.f;
}

// FP32 master weights -> BF16 operand copies.
__global__ void k_mlp_pack(const float *__restrict__ p, bf16 *__restrict__ pack) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    const int at = pack_index(i);
    if (at >= 0) pack[at] = __float2bfloat16(p[i]);
}

}  // namespace

struct mcg_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    float *d_params = nullptr, *d_m = nullptr, *d_v = nullptr;
    // results, in one buffer so that a call reads its own and the flag back in one copy: the gradient, the loss,
    // the flag that a kernel sets whose tensor-core or copy wait ran out, the forward pass's q
    float *d_grad = nullptr, *d_loss = nullptr, *d_q = nullptr;
    int *d_err = nullptr;        // 0 but between a kernel that gave up and the end of its call (check_waits)
    std::vector<float> host_q;   // flag and q of a short forward pass
    double *d_wpart = nullptr;   // k_weight_sum's partial sums
    float *d_inv_wsum = nullptr; // 1 / sum of the call's row weights, or
    float inv_wsum = 0.f;        // summed on the host
    bool inv_on_device = false;
    bf16 *d_pack = nullptr;
    float *d_feat = nullptr, *d_tgt = nullptr, *d_w = nullptr;
    float *d_partial = nullptr;  // [ctas][kParams + 1] per-CTA gradients and losses
    uint32_t ctas = 0;           // persistent CTAs of the forward and gradient kernels
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;  // around the steps of the last mcg_mlp_train
    double train_ms = 0.0;
    uint32_t cap = 0, cap_q = 0;
    uint64_t adam_t = 0;
};

namespace {

// Up to so many rows a forward pass reads the flag and q in one copy through the
// host; a second copy costs about as much as moving so many values there.
constexpr uint32_t kStagedRows = 1u << 15;

// The results' buffer for n rows; its flag is 0.
mcg_status ensure_results(mcg_mlp *m, uint32_t n) {
    if (n <= m->cap_q) return MCG_OK;
    m->cap_q = 0;
    cudaFree(m->d_grad);
    m->d_grad = m->d_loss = m->d_q = nullptr;
    m->d_err = nullptr;
    float *p = nullptr;
    MCG_CUDA(cudaMalloc((void **)&p, (kParams + 2ull + n) * sizeof(float)));
    m->d_grad = p;
    m->d_loss = p + kParams;
    m->d_err = reinterpret_cast<int *>(m->d_loss + 1);
    m->d_q = m->d_loss + 2;
    MCG_CUDA(cudaMemsetAsync(m->d_err, 0, sizeof(int), m->stream));
    m->cap_q = n;
    return MCG_OK;
}

mcg_status ensure_rows(mcg_mlp *m, uint32_t n) {
    if (n <= m->cap) return MCG_OK;
    cudaFree(m->d_feat);
    cudaFree(m->d_tgt);
    cudaFree(m->d_w);
    m->d_feat = m->d_tgt = m->d_w = nullptr;
    m->cap = 0;
    MCG_CUDA(cudaMalloc((void **)&m->d_feat, (size_t)n * kIn * sizeof(float)));
    MCG_CUDA(cudaMalloc((void **)&m->d_tgt, (size_t)n * sizeof(float)));
    MCG_CUDA(cudaMalloc((void **)&m->d_w, (size_t)n * sizeof(float)));
    const mcg_status st = ensure_results(m, n);
    if (st != MCG_OK) return st;
    m->cap = n;
    return MCG_OK;
}

// After a synchronised call that read the flag `err`: did one of its kernels
// give up on a tensor-core or copy wait?  The flag is cleared for the next call.
mcg_status check_waits(mcg_mlp *m, int err) {
    if (!err) return MCG_OK;
    MCG_CUDA(cudaMemsetAsync(m->d_err, 0, sizeof(int), m->stream));
    return mcg::fail(MCG_ERR_CUDA, "proposal network: a tensor-core or bulk-copy wait timed out (results invalid)");
}

mcg_status pack(mcg_mlp *m) {
    k_mlp_pack<<<(kParams + 255) / 256, 256, 0, m->stream>>>(m->d_params, m->d_pack);
    MCG_CUDA(cudaGetLastError());
    return MCG_OK;
}

// The gradient kernel over the uploaded rows; returns its CTAs (partial gradients).
mcg_status grad_partials(mcg_mlp *m, uint32_t n, bool has_w, uint32_t &blocks) {
    const uint32_t tiles = (n + kTile - 1) / kTile;
    blocks = std::max<uint32_t>(1, std::min<uint32_t>(tiles, m->ctas));
    k_mlp_grad<<<blocks, kThreads, sizeof(TcSmem), m->stream>>>(m->d_pack, m->d_params, m->d_feat, m->d_tgt,
                                                               has_w ? m->d_w : nullptr, m->inv_wsum,
                                                               m->inv_on_device ? m->d_inv_wsum : nullptr, n,
                                                               m->d_partial, m->d_err);
    MCG_CUDA(cudaGetLastError());
    return MCG_OK;
}

constexpr uint32_t kReduceBlocks = (kParams + 1 + kReduceCols - 1) / kReduceCols;

// The call's rows to the device, and 1 / sum of their weights.
mcg_status upload_rows(mcg_mlp *m, const float *feat, const float *tgt, const float *w, uint32_t n) {
    mcg_status st = ensure_rows(m, n);
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaMemcpyAsync(m->d_feat, feat, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    if (!tgt) return MCG_OK;
    MCG_CUDA(cudaMemcpyAsync(m->d_tgt, tgt, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    if (w) MCG_CUDA(cudaMemcpyAsync(m->d_w, w, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    m->inv_on_device = w && n >= kHostSumRows;
    if (m->inv_on_device) {
        k_weight_sum<<<kSumBlocks, kSumThreads, 0, m->stream>>>(m->d_w, n, m->d_wpart);
        k_weight_inverse<<<1, 1, 0, m->stream>>>(m->d_wpart, m->d_inv_wsum);
        MCG_CUDA(cudaGetLastError());
        return MCG_OK;
    }
    double ws = n;
    if (w) {
        ws = 0.0;
        for (uint32_t i = 0; i < n; ++i) ws += w[i];
    }
    m->inv_wsum = ws > 0 ? (float)(1.0 / ws) : 0.f;
    return MCG_OK;
}

}  // namespace

extern "C" {

mcg_status mcg_mlp_create(int32_t device, uint64_t seed, mcg_mlp **out) {
    mcg::clear_error();
    if (!out) return mcg::fail(MCG_ERR_INVALID, "out is NULL");
    *out = nullptr;
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev == 0) {
        cudaGetLastError();
        return mcg::fail(MCG_ERR_NO_DEVICE, "no CUDA device visible");
    }
    auto m = std::make_unique<mcg_mlp>();
    m->device = device;
    MCG_CUDA(cudaSetDevice(device));
    MCG_CUDA(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    MCG_CUDA(cudaMalloc((void **)&m->d_params, kParams * sizeof(float)));
    MCG_CUDA(cudaMalloc((void **)&m->d_wpart, kSumBlocks * sizeof(double)));
    MCG_CUDA(cudaMalloc((void **)&m->d_inv_wsum, sizeof(float)));
    MCG_CUDA(cudaMalloc((void **)&m->d_m, kParams * sizeof(float)));
    MCG_CUDA(cudaMalloc((void **)&m->d_v, kParams * sizeof(float)));
    MCG_CUDA(cudaMalloc((void **)&m->d_pack, kPackSize * sizeof(bf16)));
    MCG_CUDA(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TcSmem)));
    MCG_CUDA(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TcSmem)));
    // two CTAs per SM need the largest shared-memory carveout
    MCG_CUDA(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    MCG_CUDA(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    int sms = 0, smem_sm = 0, reserved = 0;
    MCG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    MCG_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
    MCG_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device));
    // CTAs that fit an SM's shared memory, at most two: each holds 256 of the
    // SM's 512 TMEM columns
    const int per_sm = smem_sm / (int)(sizeof(TcSmem) + reserved);
    m->ctas = (uint32_t)std::max(1, sms * std::min(std::max(per_sm, 1), kCtasPerSm));
    // the reduction holds 32 entries of every CTA's partial gradient
    const size_t most = (48u << 10) - sizeof(float) * kReduceGroups * kReduceCols;
    m->ctas = std::min<uint32_t>(m->ctas, (uint32_t)(most / (kReduceCols * sizeof(float))));
    MCG_CUDA(cudaMalloc((void **)&m->d_partial, (size_t)m->ctas * (kParams + 1) * sizeof(float)));
    mcg_status st = ensure_results(m.get(), kStagedRows);
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaEventCreate(&m->ev0));
    MCG_CUDA(cudaEventCreate(&m->ev1));
    // He-style initialisation from a seeded host generator
    std::vector<float> p(kParams, 0.f);
    std::mt19937_64 rng(seed);
    std::normal_distribution<float> nd(0.f, 1.f);
    for (int i = 0; i < kIn * kHid; ++i) p[kOffW1 + i] = nd(rng) * std::sqrt(2.f / kIn);
    for (int i = 0; i < kHid * kHid; ++i) p[kOffW2 + i] = nd(rng) * std::sqrt(2.f / kHid);
    for (int i = 0; i < kHid; ++i) p[kOffW3 + i] = nd(rng) * std::sqrt(1.f / kHid);
    MCG_CUDA(cudaMemcpy(m->d_params, p.data(), kParams * sizeof(float), cudaMemcpyHostToDevice));
    MCG_CUDA(cudaMemset(m->d_m, 0, kParams * sizeof(float)));
    MCG_CUDA(cudaMemset(m->d_v, 0, kParams * sizeof(float)));
    st = pack(m.get());
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaStreamSynchronize(m->stream));
    *out = m.release();
    return MCG_OK;
}

mcg_status mcg_mlp_destroy(mcg_mlp *m) {
    mcg::clear_error();
    if (!m) return MCG_OK;
    cudaSetDevice(m->device);
    cudaStreamSynchronize(m->stream);
    cudaFree(m->d_params);
    cudaFree(m->d_grad);
    cudaFree(m->d_m);
    cudaFree(m->d_v);
    cudaFree(m->d_wpart);
    cudaFree(m->d_inv_wsum);
    cudaFree(m->d_pack);
    cudaFree(m->d_feat);
    cudaFree(m->d_tgt);
    cudaFree(m->d_w);
    cudaFree(m->d_partial);
    if (m->ev0) cudaEventDestroy(m->ev0);
    if (m->ev1) cudaEventDestroy(m->ev1);
    cudaStreamDestroy(m->stream);
    delete m;
    return MCG_OK;
}

mcg_status mcg_mlp_set_params(mcg_mlp *m, const float *params) {
    mcg::clear_error();
    if (!m || !params) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    MCG_CUDA(cudaSetDevice(m->device));
    MCG_CUDA(cudaMemcpyAsync(m->d_params, params, kParams * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MCG_CUDA(cudaMemsetAsync(m->d_m, 0, kParams * sizeof(float), m->stream));
    MCG_CUDA(cudaMemsetAsync(m->d_v, 0, kParams * sizeof(float), m->stream));
    m->adam_t = 0;
    mcg_status st = pack(m);
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaStreamSynchronize(m->stream));
    return MCG_OK;
}

mcg_status mcg_mlp_get_params(mcg_mlp *m, float *params) {
    mcg::clear_error();
    if (!m || !params) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    MCG_CUDA(cudaSetDevice(m->device));
    MCG_CUDA(cudaMemcpyAsync(params, m->d_params, kParams * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MCG_CUDA(cudaStreamSynchronize(m->stream));
    return MCG_OK;
}

mcg_status mcg_mlp_forward(mcg_mlp *m, const float *features, uint32_t n, float *q_out) {
    mcg::clear_error();
    if (!m || !features || !q_out) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (n == 0) return MCG_OK;
    MCG_CUDA(cudaSetDevice(m->device));
    mcg_status st = upload_rows(m, features, nullptr, nullptr, n);
    if (st != MCG_OK) return st;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    k_mlp_forward<<<std::min(tiles, m->ctas), kThreads, sizeof(TcSmem), m->stream>>>(m->d_pack, m->d_params,
                                                                                     m->d_feat, n, m->d_q, m->d_err);
    MCG_CUDA(cudaGetLastError());
    if (n <= kStagedRows) {
        m->host_q.resize(n + 1u);
        MCG_CUDA(cudaMemcpyAsync(m->host_q.data(), m->d_err, (n + 1u) * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
        MCG_CUDA(cudaStreamSynchronize(m->stream));
        int err;
        std::memcpy(&err, m->host_q.data(), sizeof(err));
        std::memcpy(q_out, m->host_q.data() + 1, (size_t)n * sizeof(float));
        return check_waits(m, err);
    }
    int err = 0;
    MCG_CUDA(cudaMemcpyAsync(q_out, m->d_q, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MCG_CUDA(cudaMemcpyAsync(&err, m->d_err, sizeof(err), cudaMemcpyDeviceToHost, m->stream));
    MCG_CUDA(cudaStreamSynchronize(m->stream));
    return check_waits(m, err);
}

mcg_status mcg_mlp_grad(mcg_mlp *m, const float *features, const float *targets, const float *weights, uint32_t n,
                        float *grad_out, float *loss_out) {
    mcg::clear_error();
    if (!m || !features || !targets || !grad_out) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (n == 0) return mcg::fail(MCG_ERR_INVALID, "no rows");
    MCG_CUDA(cudaSetDevice(m->device));
    mcg_status st = upload_rows(m, features, targets, weights, n);
    if (st != MCG_OK) return st;
    uint32_t blocks = 0;
    st = grad_partials(m, n, weights != nullptr, blocks);
    if (st != MCG_OK) return st;
    k_mlp_reduce<<<kReduceBlocks, kReduceThreads, blocks * kReduceCols * sizeof(float), m->stream>>>(m->d_partial, blocks, m->d_grad);
    MCG_CUDA(cudaGetLastError());
    float out[kParams + 2];  // gradient, loss, flag
    MCG_CUDA(cudaMemcpyAsync(out, m->d_grad, sizeof(out), cudaMemcpyDeviceToHost, m->stream));
    MCG_CUDA(cudaStreamSynchronize(m->stream));
    std::memcpy(grad_out, out, kParams * sizeof(float));
    const float loss = out[kParams];
    int err;
    std::memcpy(&err, out + kParams + 1, sizeof(err));
    st = check_waits(m, err);
    if (st != MCG_OK) return st;
    if (loss_out) *loss_out = loss;
    return MCG_OK;
}

mcg_status mcg_mlp_train(mcg_mlp *m, const float *features, const float *targets, const float *weights, uint32_t n,
                         uint32_t steps, float lr, float *loss_out) {
    mcg::clear_error();
    if (!m || !features || !targets) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    if (n == 0) return mcg::fail(MCG_ERR_INVALID, "no rows");
    MCG_CUDA(cudaSetDevice(m->device));
    mcg_status st = upload_rows(m, features, targets, weights, n);
    if (st != MCG_OK) return st;
    MCG_CUDA(cudaEventRecord(m->ev0, m->stream));
    for (uint32_t s = 0; s < steps; ++s) {
        uint32_t blocks = 0;
        st = grad_partials(m, n, weights != nullptr, blocks);
        if (st != MCG_OK) return st;
        ++m->adam_t;
        const float b1c = 1.f - std::pow(0.9f, (float)m->adam_t);
        const float b2c = 1.f - std::pow(0.999f, (float)m->adam_t);
        k_mlp_step<<<kReduceBlocks, kReduceThreads, blocks * kReduceCols * sizeof(float), m->stream>>>(
            m->d_partial, blocks, m->d_params, m->d_m, m->d_v, lr, b1c, b2c, m->d_pack, m->d_loss);
    }
    MCG_CUDA(cudaGetLastError());
    MCG_CUDA(cudaEventRecord(m->ev1, m->stream));
    float out[2];  // loss, flag
    MCG_CUDA(cudaMemcpyAsync(out, m->d_loss, sizeof(out), cudaMemcpyDeviceToHost, m->stream));
    MCG_CUDA(cudaStreamSynchronize(m->stream));
    float ms = 0.f;
    MCG_CUDA(cudaEventElapsedTime(&ms, m->ev0, m->ev1));
    m->train_ms = ms;
    int err;
    std::memcpy(&err, out + 1, sizeof(err));
    st = check_waits(m, err);
    if (st != MCG_OK) return st;
    if (loss_out) *loss_out = out[0];
    return MCG_OK;
}

mcg_status mcg_mlp_train_time(mcg_mlp *m, double *ms) {
    mcg::clear_error();
    if (!m || !ms) return mcg::fail(MCG_ERR_INVALID, "NULL argument");
    *ms = m->train_ms;
    return MCG_OK;
}

}  // extern "C"
