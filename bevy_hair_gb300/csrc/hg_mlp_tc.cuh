// The shading surrogate's network on the 5th-generation tensor cores
// (tcgen05): 128 rows per MMA (M = 128), accumulators in tensor memory,
// operands in shared memory.  Same network and numerics as hg_mlp.cuh
// (FP16 weights and activations, FP32 accumulation), with the biases folded
// into the products: every layer's input carries two constant-1 columns whose
// weights are the FP16 high and low parts of the bias, which keeps the bias
// to ~2^-22 relative.
//
// A "chain" is one warpgroup (4 warps, 128 threads; thread r owns row r) that
// runs one evaluation at a time in 104 TMEM columns: the accumulator (64), the
// hidden activations (32 columns of FP16 pairs) and the inputs (8).  Per layer
// one thread issues the MMAs and commits them to the chain's mbarrier; the 128
// threads wait (bounded), read their row of the accumulator with tcgen05.ld,
// apply ReLU + FP16 conversion and store it as the next layer's A operand
// with tcgen05.st.  A CTA holds four chains (512 threads) and all of the SM's
// 512 TMEM columns; while one chain converts, the tensor core runs another's
// layer.
//
// The A operand lives in tensor memory because shared-memory bandwidth bounds
// the alternative: with N = 64, an MMA that reads A (128 x 80) from shared
// memory moves 30 KB per layer for 1.3 MFLOP, and every activation is stored
// there first.  Only the weights (10 KB a layer) and the constant bias columns
// stay in shared memory.  The elected lane takes the MMAs' operands from values
// that are the same in the whole warp by construction (broadcast from lane 0):
// from per-thread registers each MMA took ~100 cycles to issue.  Against two
// evaluations a chain with A in shared memory (same outputs, bit for bit):
// 1,000,003 rows 112 -> 48 us (with row-wise stores), shade model 1 at
// 1920 x 1080 with 9 lights 391 -> 263 us.
//
// Shared-memory operand layout (K-major, no swizzle): 8 x 16-byte core
// matrices; element (row, k) at (row/8)*SBO + (k/8)*LBO + (row%8)*16 + (k%8)*2
// with LBO = 128 (core matrices adjacent along K are contiguous) and
// SBO = (K/8)*128.  A operands in TMEM: row r in lane r, elements 2j and 2j+1
// in column j.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "hg_mlp.cuh"

namespace hg {
namespace mlp {
namespace tc {

constexpr uint32_t kM = 128;
constexpr uint32_t kKin = 16;   // 10 inputs, 2 bias columns, 4 zeros
constexpr uint32_t kKhid = 80;  // 64 activations, 2 bias columns, 14 zeros
constexpr uint32_t kLbo = 128;
constexpr uint32_t kSboIn = (kKin / 8) * 128, kSboHid = (kKhid / 8) * 128;
// Shared-memory byte offsets of one CTA.
constexpr uint32_t kOffW1 = 0;
constexpr uint32_t kOffW2 = kOffW1 + kHid * kKin * 2;
constexpr uint32_t kOffW3 = kOffW2 + kHid * kKhid * 2;
constexpr uint32_t kOffW4 = kOffW3 + kHid * kKhid * 2;
constexpr uint32_t kOffW5 = kOffW4 + kHid * kKhid * 2;
constexpr uint32_t kWeightBytes = kOffW5 + kOut * kKhid * 2;  // 35,328
constexpr uint32_t kOffOnes = kWeightBytes;                   // 128 x 16: two columns of ones, the bias input
constexpr uint32_t kChains = 4;                               // warpgroups per CTA
constexpr uint32_t kOffStage = kOffOnes + kM * kKin * 2;      // per warp 32 x 13 floats: output rows (infer)
constexpr uint32_t kStageFloats = 32 * (kUsedOut + 1);
constexpr uint32_t kOffBar = kOffStage + 4 * kChains * kStageFloats * 4;  // kChains mbarriers, then the TMEM address
constexpr uint32_t kOffSlot = kOffBar + 8 * kChains;
constexpr uint32_t kSmemBytes = kOffSlot + 16;
constexpr uint32_t kTmemCols = 512;
// TMEM columns of a chain.
constexpr uint32_t kChainCols = 128, kColAcc = 0, kColHid = 64, kColIn = 96;
constexpr uint32_t kThreads = 128 * kChains;
static_assert(kSmemBytes <= 232448, "shared memory per CTA");
static_assert(kWeightBytes % 128 == 0 && kOffStage % 128 == 0 && kOffBar % 8 == 0, "tile alignment");
static_assert(kChains * kChainCols <= kTmemCols && kColHid + kHid / 2 <= kColIn && kColIn + kKin / 2 <= kChainCols,
              "tensor memory columns");
// Instruction descriptors (kind::f16): D F32, A and B F16, both K-major, M = 128.
constexpr uint32_t kIdescHid = (1u << 4) | ((64u >> 3) << 17) | ((kM >> 4) << 24);
constexpr uint32_t kIdescOut = (1u << 4) | ((16u >> 3) << 17) | ((kM >> 4) << 24);
// Bounded waits: iterations of mbarrier.try_wait before a chain gives up.
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr uint32_t kErrTimeout = 2u;

__device__ __forceinline__ uint32_t canon(uint32_t row, uint32_t k, uint32_t sbo) {
    return (row >> 3) * sbo + (k >> 3) * kLbo + (row & 7u) * 16u + (k & 7u) * 2u;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start, LBO, SBO (all >> 4), version 1,
// base offset 0, no swizzle.
__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(kLbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot_saddr, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot_saddr), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same with the A operand (128 x 16 FP16, 8 columns) in tensor memory.
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void commit(uint32_t mbar_saddr) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar_saddr)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t mbar_saddr, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(mbar_saddr), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }

// Wait for phase `parity` of the mbarrier, at most kWaitLimit polls.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar_saddr, uint32_t parity) {
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar_saddr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Barrier over one warpgroup (named barrier `id`, 128 threads) that returns
// the OR of `pred` over its threads.
__device__ __forceinline__ bool group_sync_or(uint32_t id, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 q, %1, 0;\nbar.red.or.pred p, %2, 128, q;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(id)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t v[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t v[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// The value, unknown to the optimiser: keeps it from making a copy of the
// caller's loop for either outcome of a test on it.
__device__ __forceinline__ uint32_t opaque(uint32_t v) {
    asm volatile("" : "+r"(v));
    return v;
}

// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r != 0;
}

// This thread's row (lane) of 32 or 8 adjacent columns.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t v[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t v[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// The weight tiles of the CTA (every thread takes part): W[n][k] in the
// canonical layout, the two bias columns (FP16 high and low parts) after the
// real inputs.  A unit of 8 columns of a row is 16 contiguous bytes on both
// sides; element by element this took 6 us more of every launch.
__device__ __forceinline__ void load_weights(uint8_t* smem, const __half* __restrict__ w16,
                                             const float* __restrict__ params, int tid, int nthreads) {
    auto bias = [](float b) {
        const __half hi = __float2half_rn(b), lo = __float2half_rn(b - __half2float(hi));
        return (uint32_t)__half_as_ushort(hi) | (uint32_t)__half_as_ushort(lo) << 16;
    };
    for (int i = tid; i < (int)(kHid * kKin / 8); i += nthreads) {
        const uint32_t n = i / (kKin / 8), k = i % (kKin / 8) * 8;
        uint4 v = *reinterpret_cast<const uint4*>(w16 + kW1 + n * kIn + k);
        if (k == 8u) {  // inputs 8, 9, then the bias columns 10, 11
            v.y = bias(params[kB1 + n]);
            v.z = v.w = 0u;
        }
        *reinterpret_cast<uint4*>(smem + kOffW1 + canon(n, k, kSboIn)) = v;
    }
    const int woff[4] = {kW2, kW3, kW4, kW5}, boff[4] = {kB2, kB3, kB4, kB5};
    const uint32_t soff[4] = {kOffW2, kOffW3, kOffW4, kOffW5};
    for (int l = 0; l < 4; ++l)
        for (int i = tid; i < (int)((l < 3 ? kHid : kOut) * kKhid / 8); i += nthreads) {
            const uint32_t n = i / (kKhid / 8), k = i % (kKhid / 8) * 8;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (k < (uint32_t)kHid) v = *reinterpret_cast<const uint4*>(w16 + woff[l] + n * kHid + k);
            else if (k == (uint32_t)kHid) v.x = bias(params[boff[l] + n]);
            *reinterpret_cast<uint4*>(smem + soff[l] + canon(n, k, kSboHid)) = v;
        }
}
static_assert(kW1 % 8 == 0 && kW2 % 8 == 0 && kW3 % 8 == 0 && kW4 % 8 == 0 && kW5 % 8 == 0 && kUsedIn == 10 &&
                  kIn % 8 == 0,
              "16-byte weight rows; inputs 8 and 9 share their block with the bias columns");

struct Chain {
    uint32_t w;       // shared address of the weights
    uint32_t mbar;    // shared address of the mbarrier
    uint32_t tmem;    // TMEM address of the chain's columns, at this warp's lanes
    uint32_t cols;    // the same at lane 0
    uint32_t lead;    // 1 in the warpgroup's first warp, one lane of which issues the MMAs
    uint32_t phase;   // parity of the mbarrier's next phase
    uint32_t bar_id;  // named barrier of the warpgroup
    uint32_t row;     // this thread's row, 0..127
};

// One layer's MMAs (the chain's first thread): KSTEPS products of 16 columns of
// the A operand at TMEM column `a`, then, for hidden inputs, the bias columns.
template <uint32_t KSTEPS, bool BIAS>
__device__ __forceinline__ void issue(const Chain& c, uint32_t a, uint32_t w_off, uint32_t w_sbo, uint32_t idesc) {
#pragma unroll
    for (uint32_t ks = 0; ks < KSTEPS; ++ks)
        mma_ts(c.cols + kColAcc, c.cols + a + 8u * ks, desc(c.w + w_off + ks * 2u * kLbo, w_sbo), idesc, ks);
    if (BIAS)
        mma(c.cols + kColAcc, desc(c.w + kOffOnes, kSboIn), desc(c.w + w_off + KSTEPS * 2u * kLbo, w_sbo), idesc, 1u);
    commit(c.mbar);
}

// The network on the row's normalised inputs: y receives this thread's 12
// outputs.  Every thread of the warpgroup calls it.  Returns false (for the
// whole warpgroup) when an MMA did not complete in time; the chain is then
// unusable.
__device__ __forceinline__ bool forward(Chain& c, const float x[kUsedIn], float y[kUsedOut]) {
    {
        const uint32_t in[8] = {pack_h2(x[0], x[1]), pack_h2(x[2], x[3]), pack_h2(x[4], x[5]), pack_h2(x[6], x[7]),
                                pack_h2(x[8], x[9]), 0x3C003C00u,         0u,                  0u};
        tmem_st8(c.tmem + kColIn, in);
    }
    tmem_wait_st();
    fence_before();
    if (group_sync_or(c.bar_id, false)) return false;
    if (opaque(c.lead)) {
        fence_after();
        if (elect_one()) issue<1, false>(c, kColIn, kOffW1, kSboIn, kIdescHid);
    }
#pragma unroll
    for (int layer = 0; layer < 4; ++layer) {
        const bool ok = mbar_wait(c.mbar, c.phase);
        if (ok) c.phase ^= 1u;  // after a timeout the phase stays the outstanding one
        fence_after();
        uint32_t h[kHid / 2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t v[32];
            tmem_ld32(c.tmem + kColAcc + 32u * half, v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j)
                h[16 * half + j] = pack_relu(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
        }
        tmem_st32(c.tmem + kColHid, h);
        tmem_wait_st();
        fence_before();
        if (group_sync_or(c.bar_id, !ok)) return false;
        if (opaque(c.lead)) {
            fence_after();
            const uint32_t w = layer == 0 ? kOffW2 : layer == 1 ? kOffW3 : layer == 2 ? kOffW4 : kOffW5;
            if (elect_one()) issue<4, true>(c, kColHid, w, kSboHid, layer < 3 ? kIdescHid : kIdescOut);
        }
    }
    const bool ok = mbar_wait(c.mbar, c.phase);
    if (ok) c.phase ^= 1u;
    fence_after();
    uint32_t o[16];
    tmem_ld16(c.tmem + kColAcc, o);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < kUsedOut; ++i) y[i] = __uint_as_float(o[i]);
    fence_before();
    return !group_sync_or(c.bar_id, !ok);
}

// CTA set-up: weights, the constant bias input, mbarriers, TMEM.  Every thread
// calls it; returns this thread's chain.
__device__ __forceinline__ Chain setup(uint8_t* smem, const __half* w16, const float* params) {
    const uint32_t tid = threadIdx.x;
    // broadcast from lane 0, so that the compiler knows it to be the same in
    // the whole warp: the MMAs take their operands from uniform registers
    const uint32_t warp = __shfl_sync(0xffffffffu, tid >> 5, 0), g = warp >> 2;
    const uint32_t base = smem_addr(smem);
    Chain c;
    c.lead = (warp & 3u) == 0u ? 1u : 0u;
    c.w = base;
    c.bar_id = 1u + g;
    c.row = tid & 127u;
    c.mbar = base + kOffBar + 8u * g;
    c.phase = 0;
    load_weights(smem, w16, params, (int)tid, (int)blockDim.x);
    for (uint32_t i = tid; i < kM * kKin / 8u; i += blockDim.x)  // columns 0, 1 of every row are 1
        *reinterpret_cast<uint4*>(smem + kOffOnes + canon(i >> 1, (i & 1u) * 8u, kSboIn)) =
            make_uint4((i & 1u) ? 0u : 0x3C003C00u, 0u, 0u, 0u);
    if (tid == 0) {
        for (uint32_t k = 0; k < kChains; ++k) mbar_init(base + kOffBar + 8u * k, 1);
        fence_mbar_init();
    }
    if (tid < 32) {
        tmem_alloc(base + kOffSlot, kTmemCols);
        tmem_relinquish();
    }
    fence_proxy_async();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tbase =
        __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(smem + kOffSlot), 0);
    c.cols = tbase + g * kChainCols;
    c.tmem = c.cols + ((c.row & ~31u) << 16);
    return c;
}

// CTA tear-down after every chain has finished (or given up): bounded waits
// for a failed chain's outstanding commits, then the TMEM is freed.
__device__ __forceinline__ void teardown(uint8_t* smem, Chain& c, bool failed) {
    if (failed) (void)mbar_wait(c.mbar, c.phase);
    fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        fence_after();
        tmem_dealloc(*reinterpret_cast<volatile uint32_t*>(smem + kOffSlot), kTmemCols);
    }
}

}  // namespace tc
}  // namespace mlp
}  // namespace hg
