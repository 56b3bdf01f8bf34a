// Prefill dequant-GEMM on the 5th-generation tensor cores (sm_100a):
//   Y[M,N] (bf16) = X[M,K] (bf16) . dequant(W[N,K])^T, fp32 accumulation in tensor memory.
//
// Replaces C-ML's "dequantize the whole weight to an fp32 temporary, then a scalar
// triple loop" (src/nn/qlora.c:264-317) and its dequantize-at-load + fp32 matmul
// (src/core/gguf.c:271-295, src/ops/ir/execution.c:989-1052).
//
// A tile is 128 weight rows (the MMA "M" side, operand A) by NX <= 256 activation rows (the MMA "N" side, operand B), or 256 weight rows
// by 257 to 512 activation rows, which a pair of CTAs shares (cta_group::2: a CTA expands 128 weight rows and holds half of the
// activations, two MMAs into two halves of tensor memory). K in slabs of 64. Where the small tiles are fewer than the SMs, a cluster
// of 2 to 8 CTAs shares the K of a tile: their sums meet in distributed shared memory, every CTA adds and finishes its part of the
// columns in rank order (no scratch in global memory, no second launch, the same result every time).
//   warp 0      one lane issues TMA tensor loads of the bf16 activation slab (128B swizzle, boxes of up to 256 rows)
//   warp 1      allocates tensor memory; an elected lane (of the pair's first CTA) issues tcgen05.mma (kind::f16, 128 or 256 x NX x 16);
//               in the second CTA it passes on that the CTA's slab is ready
//   warps 2..17 expand the packed weights to bf16 in the canonical K-major 128B-swizzled layout the MMA reads, two groups of eight
//               the slabs in turn; they are the epilogue too: tcgen05.ld, then Y or the cluster's sum
// What bounds it: up to 256 activation rows the expansion (a slab of 128 x 64 weights takes 0.37 us for Q4_0, 0.54 for NF4, 0.63 for
// Q8_0, about as long as its instructions at half an instruction a cycle and scheduler) beside about 4 us to start and 2.5 to 4 for a
// cluster's sum; above, the MMA: a slab of 256 x 512 x 64 takes a pair 1,090 cycles, the tensor cores 1,024 of them. Pairs halve what an SM
// reads of the activations (every 128 weight rows used to read all of them: 1.4 GB from L2 at 2,048 rows of 11008x4096) and the
// expansion per MMA. The issuing warp is the next limit: with a barrier for each box, or an arrival released for the cluster, a slab took
// 1,440 cycles. Hence the tile: as many activation rows as fill the SMs in whole waves (pick_shape).
// Packed weights and scales come by plain loads into registers, three slabs of the group ahead. Each thread keeps one
// block index and no other address, and the issuing warp counts its stages: with 64-bit addresses, zeroed registers and a vote
// in every wait a slab took 0.60 instead of 0.40 us, with a division per slab in the issuing warp 0.54.
// The cluster's sum: a thread has four weight rows of a column, reads all ranks' sums in 16-byte pieces that are in flight together, and
// stores 8 or 16 bytes; one value and one rank after the other, with a last barrier that waited for the stores, it took 1.1 to 2.2 us more
// (3.5 for NF4 at 511 rows). A table of NF4's code pairs in shared memory instead of permutes was slower (4096x4096 77 rows 17.5 18.2).
// What an output is multiplied with or added to is requested before the wait for the accumulators or with the cluster's sums, then a
// batch ahead; requested with the batch itself, it put a memory latency into each: SwiGLU 11008x4096 77 rows 34.3 31.1, 512 67.7 62.3,
// 2048 174 158 (without SwiGLU 30.8, 49.2, 130: the rest is the division and exponential of every output), onto a residual 4096x11008
// 512 48.4 45.5, 4096x4096 512 25.4 22.6, stored as fp32 4096x4096 77 13.9 12.9.
// us a call, weights from memory, bf16 output, before and after the pairs and this sum:
//   Q4_0 4096x4096    M = 77 15.1 13.9, 512 25.6 23.4, 2048 56.0 49.6      11008x4096  77 31.3 30.8, 512 57.0 49.8, 2048 159 130
//   Q4_0 4096x11008   M = 77 25.9 24.5, 512 49.0 46.1, 2048 142 124        32000x4096  77 59.7 59.6, 512 111 97.6, 2048 408 357
//   NF4 4096x4096     M = 77 17.5 16.1, 512 30.1 26.7, 2048 58.8 50.5      Q8_0 4096x4096  77 18.0 17.4, 512 30.8 30.1, 2048 65.6 52.1
//   Q8_0 7000x5120    M = 600 87.6 53.9
// Expansion:
//   Q4_0  a byte permute drops two nibbles into the mantissas of two bf16 halves (0x43nn = 128 + n), one packed subtract gives
//         n - 8 exactly, one packed multiply applies the block scale
//   NF4   the two bytes of a code value by byte permutes over a table of 16 in registers, one packed multiply by the block scale
//   Q8_0  a byte permuted into an fp32 mantissa, one multiply-add, rounded once
// Q4_0 and NF4 therefore round twice (scale or code value to bf16, then the product); the path's
// tolerance is 1e-2 of the largest output. No load is multicast; a pair's commits arrive at the
// barriers of both its CTAs. Every wait on an mbarrier is bounded; on expiry the CTA raises a status flag (cmlb200_gemm_status), waits for its
// copies and MMAs in flight (each has a barrier of its own), frees its tensor memory and returns.
#include <cuda.h>
#include <mutex>
#include <type_traits>
#include "common.cuh"

namespace {

constexpr int BK = 64;              // K slab: 64 bf16 = one 128-byte swizzle row
constexpr int DQ_WARPS = 16;
constexpr int DQ_THREADS = DQ_WARPS * 32;
constexpr int THREADS = 64 + DQ_THREADS;
constexpr int A_BYTES = 128 * BK * 2;           // 16 KB: 128 expanded weight rows
constexpr int BN = 128;             // weight rows of a tile
constexpr int B_ROWS = 256;         // activation rows of a box and an MMA
constexpr int B_BYTES = B_ROWS * BK * 2;        // 32 KB
constexpr int AHEAD = 3;                        // slabs whose packed weights a thread has requested
#ifndef CML_GEMM_SPIN_LIMIT
#define CML_GEMM_SPIN_LIMIT (1u << 22)          // (a test builds this file with a limit that runs out)
#endif
constexpr uint32_t SPIN_LIMIT = CML_GEMM_SPIN_LIMIT;
constexpr uint32_t DRAIN_LIMIT = 1u << 22;

// A group always comes back to the same stages, so a parity wait is never two phases from its barrier. A stage holds both operands of a
// slab. PAIR: two boxes of activations, of which a CTA holds half the rows each.
template <int TYPE, bool PAIR> struct Cfg {
    static constexpr int RAWB = (TYPE == CMLB200_Q8_0) ? 64 : 32;       // packed bytes per row and slab
    static constexpr int GROUPS = 2, GROUP_WARPS = DQ_WARPS / GROUPS;
    static constexpr int STAGES = 4, BOXES = PAIR ? 2 : 1;
    static constexpr int BOX_BYTES = PAIR ? B_BYTES / 2 : B_BYTES;
    // offsets from the 1024-byte aligned base
    static constexpr int a_off = 0;
    static constexpr int b_off = STAGES * A_BYTES;
    static constexpr int bar_off = b_off + STAGES * B_BYTES;
    static constexpr int nbars = 3 * STAGES + 2;
    static constexpr int total = bar_off + 8 * nbars + 32;
    static_assert(total + 1024 <= 227 * 1024, "the stages do not fit shared memory");
};

__device__ int g_gemm_status = 0;   // 0 = ok; otherwise a code identifying the wait that expired

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait. Returns false (and raises the abort flag) when the limit is hit or when
// another role already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
        if (mbar_try(bar, parity)) return true;
        if (it > 1024) {
            if (*abort_flag) return false;
            __nanosleep(32);
        }
    }
    *abort_flag = code;
    atomicCAS(&g_gemm_status, 0, code);
    return false;
}
// Waits for something that is under way whoever has aborted: a copy of this CTA, or its last MMAs.
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < DRAIN_LIMIT && !mbar_try(bar, parity); ++it)
        if (it > 1024) __nanosleep(32);
}
// Every lane waits on the barrier itself (each reader of bytes that a tensor load wrote has to
// observe the barrier's phase on its own); the verdict is then made warp-uniform so that no lane
// is left behind at a __syncwarp.
__device__ __noinline__ bool warp_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    bool mine = false;
    for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
        if (mbar_try(bar, parity)) { mine = true; break; }
        if (it > 1024) {
            if (*abort_flag) break;
            __nanosleep(32);
        }
    }
    if (!mine && !*abort_flag) { *abort_flag = code; atomicCAS(&g_gemm_status, 0, code); }
    return __all_sync(0xffffffffu, mine);
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    return warp_wait_slow(bar, parity, abort_flag, code);
}

__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr) {
    // K-major, 128-byte swizzle: 8-row groups 1024 B apart (SBO), LBO unused (=1), version 1
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// PAIR: for both CTAs of a pair, from the first one's issuing lane; a commit arrives at the barrier of either
template <bool PAIR>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    if (PAIR)
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
    else
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    if (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Arrives at the same barrier of the pair's first CTA. What the arrival stands for lies in this SM's own memory, which its half of the
// MMA reads: released for the CTA. (A release for the cluster holds the warp up for 1,400 cycles, and a slab with it.)
__device__ __forceinline__ void mbar_arrive_first(uint32_t bar) {
    asm volatile("{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %0, 0;\n mbarrier.arrive.shared::cluster.b64 _, [a];\n}\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&f)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; j++) f[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t bf162_mul(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf162_sub(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}

// Expand the 32 weights this thread owns (row n, K offset k0 + 32*h) into four 16-byte
// chunks of bf16, in element order. `raw`: the thread's packed bytes (16, or 32 for Q8_0).
template <int TYPE>
__device__ __forceinline__ void expand32(const uint4* raw, float scale, uint4 (&out)[4]) {
    if (TYPE == CMLB200_Q8_0) {
        // (2^15 + q + 128) scale - (2^15 + 128) scale: the second product is exact (20 bits), so the difference is q scale, which is
        // exact too (19 bits)
        const float offset = -32896.0f * scale;
        const uint32_t w[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
        auto each = [&](auto value) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t o[4];
#pragma unroll
                for (int p = 0; p < 4; p++) {            // 2^15 + (q + 128) as fp32 has the byte in its mantissa
                    const uint32_t u = w[2 * c + (p >> 1)] ^ 0x80808080u;
                    o[p] = pack_bf16(value(__uint_as_float(__byte_perm(u, 0x47000000u, p & 1 ? 0x7424 : 0x7404))),
                                     value(__uint_as_float(__byte_perm(u, 0x47000000u, p & 1 ? 0x7434 : 0x7414))));
                }
                out[c] = make_uint4(o[0], o[1], o[2], o[3]);
            }
        };
        if (fabsf(scale) <= 65504.0f) each([&](float v) { return fmaf(v, scale, offset); });
        else each([&](float v) { return (v - 32896.0f) * scale; });      // infinite weights
    } else if (TYPE == CMLB200_NF4) {
        // word i = bytes 4i..4i+3 = elements 8i..8i+7, the even one in the high nibble. Low and high bytes of the 16 code values
        // as bf16, four to a word; a permute looks up eight entries, a second one picks by the index's top bit
        const uint32_t w[4] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w};
        const uint32_t s2 = pack_bf16(scale, scale);
        constexpr uint32_t L0 = 0xca063280u, L1 = 0x00bb3d92u, L2 = 0xad7c25a3u, L3 = 0x803910e2u;
        constexpr uint32_t H0 = 0xbebfbfbfu, H1 = 0x00bdbebeu, H2 = 0x3e3e3e3du, H3 = 0x3f3f3f3eu;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            uint32_t o[4];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const uint32_t v = p ? w[c] >> 16 : w[c];
                const uint32_t e = v & 0x7777u, pick = ((v >> 1) & 0x4444u) | 0x3210u;
                const uint32_t lo = __byte_perm(__byte_perm(L0, L1, e), __byte_perm(L2, L3, e), pick);
                const uint32_t hi = __byte_perm(__byte_perm(H0, H1, e), __byte_perm(H2, H3, e), pick);
                o[2 * p] = bf162_mul(__byte_perm(lo, hi, 0x4051), s2);
                o[2 * p + 1] = bf162_mul(__byte_perm(lo, hi, 0x6273), s2);
            }
            out[c] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    } else {
        // Q4_0: byte j -> element j (low nibble) and j+16 (high nibble). 0x43nn as bf16 is 128 + n.
        const uint32_t w[4] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w};
        const uint32_t s2 = pack_bf16(scale, scale);
        const uint32_t bias = 0x43084308u;                 // (136, 136): 128 + n - 136 = n - 8
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t l4 = w[i] & 0x0F0F0F0Fu, h4 = (w[i] >> 4) & 0x0F0F0F0Fu;
            lo[2 * i] = bf162_mul(bf162_sub(__byte_perm(l4, 0x43434343u, 0x4140), bias), s2);
            lo[2 * i + 1] = bf162_mul(bf162_sub(__byte_perm(l4, 0x43434343u, 0x4342), bias), s2);
            hi[2 * i] = bf162_mul(bf162_sub(__byte_perm(h4, 0x43434343u, 0x4140), bias), s2);
            hi[2 * i + 1] = bf162_mul(bf162_sub(__byte_perm(h4, 0x43434343u, 0x4342), bias), s2);
        }
        out[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        out[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        out[2] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        out[3] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
    }
}

// What happens to a finished output value (the sum over all of K) at flat index i of [M, N]:
//   GEMM_OUT_BF16    stored as bf16                         (the plain product)
//   GEMM_OUT_F32     stored as fp32                         (Q/K/V: RoPE and attention read fp32)
//   GEMM_ACC_F32     added to an fp32 array                 (attention-out and FFN-down onto the residual,
//                                                            src/nn/llama.c:523-530, 538-543)
//   GEMM_SWIGLU_BF16 silu(gate[i]) * value stored as bf16   (the up projection finishing SwiGLU,
//                                                            src/nn/llama.c:126-155; gate may be the output array)
enum { GEMM_OUT_BF16 = 0, GEMM_OUT_F32 = 1, GEMM_ACC_F32 = 2, GEMM_SWIGLU_BF16 = 3 };
// CNT finished values `step` places apart (neighbouring activation rows of one weight row; or, 1 apart, the other way round), of which
// `count` exist, `at` the first one's place. What they are multiplied with or added to comes first, by a call of its own, so that
// those loads are in flight together and beside others. (Reductions in global memory, which load nothing, make zeros of sums below 2^-126.)
template <int CNT>
__device__ __forceinline__ void operands(const void* out, const __nv_bfloat16* gate, int mode, size_t at, int step, int count, uint32_t (&w)[CNT]) {
    if (mode == GEMM_SWIGLU_BF16) {
        // (a gate of one where there is none: its division is done as well, and what a register happens to hold sends it the long way
        // round. 9152x1280, 758 rows, 48.8 us so; a guard around every output instead made whole tiles 4 % slower)
#pragma unroll
        for (int j = 0; j < CNT; j++) {
            w[j] = 0x3f80u;
            if (j < count) w[j] = reinterpret_cast<const uint16_t*>(gate)[at + (size_t)j * step];
        }
    } else if (mode == GEMM_ACC_F32) {
#pragma unroll
        for (int j = 0; j < CNT; j++)
            if (j < count) w[j] = static_cast<const uint32_t*>(out)[at + (size_t)j * step];
    }
}
template <int CNT>
__device__ __forceinline__ void combine(int mode, const uint32_t (&w)[CNT], float (&v)[CNT]) {
    if (mode == GEMM_SWIGLU_BF16) {
#pragma unroll
        for (int j = 0; j < CNT; j++) {
            const float g = __uint_as_float(w[j] << 16);
            v[j] *= g / (1.0f + expf(-g));
        }
    } else if (mode == GEMM_ACC_F32) {
#pragma unroll
        for (int j = 0; j < CNT; j++) v[j] += __uint_as_float(w[j]);
    }
}
template <int CNT>
__device__ __forceinline__ void store(void* out, int mode, size_t at, int step, int count, const float (&v)[CNT]) {
    if (mode == GEMM_OUT_BF16 || mode == GEMM_SWIGLU_BF16) {
        __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out) + at;
#pragma unroll
        for (int j = 0; j < CNT; j++, o += step)
            if (j < count) *o = __float2bfloat16_rn(v[j]);
    } else {
        float* o = static_cast<float*>(out) + at;
#pragma unroll
        for (int j = 0; j < CNT; j++, o += step)
            if (j < count) *o = v[j];
    }
}
// The same of four neighbouring weight rows in one activation row, all there, in memory aligned to them
__device__ __forceinline__ void operands4(const void* out, const __nv_bfloat16* gate, int mode, size_t at, uint32_t (&w)[4]) {
    if (mode == GEMM_SWIGLU_BF16) {
        const uint2 g = *reinterpret_cast<const uint2*>(gate + at);
        w[0] = g.x & 0xffffu; w[1] = g.x >> 16; w[2] = g.y & 0xffffu; w[3] = g.y >> 16;
    } else if (mode == GEMM_ACC_F32) {
        const uint4 h = *reinterpret_cast<const uint4*>(static_cast<const uint32_t*>(out) + at);
        w[0] = h.x; w[1] = h.y; w[2] = h.z; w[3] = h.w;
    }
}
__device__ __forceinline__ void store4(void* out, int mode, size_t at, const float (&v)[4]) {
    if (mode == GEMM_OUT_BF16 || mode == GEMM_SWIGLU_BF16)
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(out) + at) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    else *reinterpret_cast<float4*>(static_cast<float*>(out) + at) = make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ uint4 ld_weights(const uint4* p) {        // the row's next slabs come into L2 along with it
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

struct GemmArgs {
    const uint8_t* qs;
    const void* scales;
    void* out;
    const __nv_bfloat16* gate;
    int mode, M, N, K, NX, tiles_m, tiles, nf4_block, nf4_shift;
};

template <int TYPE, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap xmap, const GemmArgs p) {
    using C = Cfg<TYPE, PAIR>;
    constexpr int STAGES = C::STAGES, RAWB = C::RAWB;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem), bars = sbase + C::bar_off;
    auto full_a = [&](int s) { return bars + 8 * s; };               // (a pair's first CTA: and all that the second one has for the slab)
    auto full_b = [&](int s) { return bars + 8 * (STAGES + s); };
    auto empty = [&](int s) { return bars + 8 * (2 * STAGES + s); };
    const uint32_t done_bar = bars + 8 * (C::nbars - 2), free_bar = bars + 8 * (C::nbars - 1);      // accumulators finished / read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::bar_off + 8 * C::nbars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::bar_off + 8 * C::nbars + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KB = (p.K + BK - 1) / BK;                 // K % 64 == 32: the last slab's upper half is zero
    const int n_lo = min(p.NX, B_ROWS), n_hi = p.NX - n_lo;              // activation rows of the first and the second MMA
    // a cluster shares the K of a tile; CTAs without one walk over several tiles
    uint32_t rank, ranks;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    // a pair has 256 weight rows of a tile, 128 in either CTA, and either holds half of the activations that both multiply with
    const int second = PAIR ? (int)rank : 0, BM = PAIR ? 2 * BN : BN;
    const int first_tile = blockIdx.x / ranks, step = gridDim.x / ranks;
    if (PAIR) { rank = 0; ranks = 1; }
    const int kb0 = KB * rank / ranks, kb1 = KB * (rank + 1) / ranks, nkb = kb1 - kb0;
    const int my_tiles = first_tile < p.tiles ? (p.tiles - first_tile + step - 1) / step : 0, slabs = my_tiles * nkb;
    uint32_t tmem_cols = 32;
    while ((int)tmem_cols < p.NX) tmem_cols <<= 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(full_a(s), C::GROUP_WARPS + (PAIR && !second ? 1 : 0)); mbar_init(full_b(s), 1); mbar_init(empty(s), 1); }
        mbar_init(done_bar, 1);
        mbar_init(free_bar, PAIR ? 2 * DQ_WARPS : DQ_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                         ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                         ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");      // its barriers and columns, too
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer: activation slabs (operand B) ----------------
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int it = 0, s = 0, kb = kb0, tile = first_tile;              // counters instead of divisions
            uint32_t phase = 1;
            for (; it < slabs; it++) {
                const uint32_t bar = full_b(s), to = sbase + C::b_off + s * B_BYTES;
                const int y = (tile % p.tiles_m) * p.NX;
                if (!mbar_wait(empty(s), phase, abort_flag, 1)) break;
                mbar_expect_tx(bar, (uint32_t)n_lo * BK * 2);
                if (PAIR) {
                    tma_load_2d(to, &xmap, kb * BK, y + second * (n_lo / 2), bar);
                    tma_load_2d(to + C::BOX_BYTES, &xmap, kb * BK, y + B_ROWS + second * (n_hi / 2), bar);
                } else tma_load_2d(to, &xmap, kb * BK, y, bar);
                if (++s == STAGES) { s = 0; phase ^= 1; }
                if (++kb == kb1) { kb = kb0; tile += step; }
            }
            for (int i = max(0, it - STAGES); i < it; i++) mbar_drain(full_b(i % STAGES), (i / STAGES) & 1);      // no copy outlives its CTA
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: the warp stays converged, an elected lane issues ----
        const uint32_t ibase = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BM >> 4) << 24);
        const uint32_t idesc = ibase | ((uint32_t)(n_lo >> 3) << 17), idesc_hi = ibase | ((uint32_t)(n_hi >> 3) << 17);
        bool ok = true;
        int s = 0, seg = 0;
        uint32_t phase = 0;
        // (the boxes first: they are there earlier, so their wait hides behind the expansion's)
        auto slab_there = [&]() { return warp_wait(full_b(s), phase, abort_flag, 4) && warp_wait(full_a(s), phase, abort_flag, 3); };
        if (PAIR && second) {                                              // tells the first CTA what has come to this one
            for (int it = 0; it < slabs && ok; it++) {
                ok = slab_there();
                if (ok && lane == 0) mbar_arrive_first(full_a(s));
                __syncwarp();
                if (++s == STAGES) { s = 0; phase ^= 1; }
            }
            seg = my_tiles;
        }
        const bool issues = !(PAIR && second);
        for (; seg < my_tiles && ok; seg++) {
            if (seg) ok = warp_wait(free_bar, (seg - 1) & 1, abort_flag, 7);
            for (int i = 0; i < nkb && ok; i++) {
                ok = slab_there();
                if (!ok) break;
                const uint64_t adesc = make_desc_sw128(sbase + C::a_off + s * A_BYTES), bdesc = make_desc_sw128(sbase + C::b_off + s * B_BYTES);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
#pragma unroll
                    for (int box = 0; box < C::BOXES; box++)
#pragma unroll
                        for (int kk = 0; kk < BK / 16; kk++)               // 32 bytes inside the swizzle row per K=16 step
                            umma_f16<PAIR>(tmem_base + (uint32_t)(box * B_ROWS), adesc + (uint64_t)(2 * kk), bdesc + (uint64_t)(box * (C::BOX_BYTES >> 4) + 2 * kk),
                                           box ? idesc_hi : idesc, (i | kk) ? 1u : 0u);
                    umma_commit<PAIR>(empty(s));
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; phase ^= 1; }
            }
            if (elect_one()) umma_commit<PAIR>(done_bar);      // arrives once every MMA issued so far has retired
            __syncwarp();
        }
        if (issues && !ok && seg > 0) mbar_drain(done_bar, (seg - 1) & 1);          // tensor memory and the stages outlive the MMAs
    } else {
        // ---------------- weight expansion (operand A), then epilogue ----------------
        const int dqw = warp - 2, grp = dqw / C::GROUP_WARPS, tg = (dqw % C::GROUP_WARPS) * 32 + lane;
        const int h = tg & 1, row = tg >> 1;                         // this thread's 32 weights of a slab: row, half
        const int row_blocks = p.K / 32;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint8_t* a_row[4];
#pragma unroll
        for (int c = 0; c < 4; c++) a_row[c] = smem + C::a_off + (row >> 3) * 1024 + (row & 7) * 128 + (((4 * h + c) ^ (row & 7)) << 4);
        // packed weights come straight into registers, AHEAD slabs before they are expanded
        // place in the weight of the next slab to request: its slab within the tile, its block index (32 weights); the last slab's
        // upper half may lie past the row's end (K % 64 == 32): a scale of zero stands for it
        int ftile = first_tile, fkb = kb0 + grp;
        const int flim = min(kb1, h ? row_blocks / 2 : (row_blocks + 1) / 2);
        uint32_t fblk = 0;
        auto place = [&]() {
            while (fkb >= kb1) { fkb -= nkb; ftile += step; }
            fblk = (uint32_t)min(ftile / p.tiles_m * BM + second * BN + row, p.N - 1) * (uint32_t)row_blocks + 2u * (uint32_t)fkb + (uint32_t)h;
        };
        place();
        uint4 raw[AHEAD][RAWB / 32];
        typedef typename std::conditional<TYPE == CMLB200_NF4, float, uint16_t>::type Scale;
        Scale scale[AHEAD];
#pragma unroll
        for (int d = 0; d < AHEAD; d++)
#pragma unroll
            for (int i = 0; i < RAWB / 32; i++) raw[d][i] = make_uint4(0u, 0u, 0u, 0u);
        auto fetch = [&](uint4 (&r)[RAWB / 32], Scale& sc) {
            if (fkb < flim && ftile < p.tiles) {
                const uint4* src = reinterpret_cast<const uint4*>(p.qs) + (size_t)fblk * (RAWB / 32);
#pragma unroll
                for (int i = 0; i < RAWB / 32; i++) r[i] = ld_weights(src + i);
                if (TYPE == CMLB200_NF4) {
                    const uint32_t at = p.nf4_shift >= 0 ? fblk >> p.nf4_shift : (uint32_t)((size_t)fblk * 32 / (size_t)p.nf4_block);
                    sc = __ldg(reinterpret_cast<const float*>(p.scales) + at);
                } else sc = __ldg(reinterpret_cast<const uint16_t*>(p.scales) + fblk);
            } else sc = 0;
            fblk += 2 * C::GROUPS;
            fkb += C::GROUPS;
            if (fkb >= kb1) place();
        };
        bool ok = true;
        // one slab: out of the registers of its slot (known when compiling: nothing moves between registers, which would wait for loads)
        auto slab = [&](uint4 (&r)[RAWB / 32], Scale& sc, int it) {
            uint4 out[4];
            float f;
            if constexpr (TYPE == CMLB200_NF4) f = sc;
            else f = cml_half_to_float(sc);
            expand32<TYPE>(r, f, out);                                // (past the end of a row: zeros meet zero-filled activations)
            fetch(r, sc);
            const int s = it % STAGES;
            ok = warp_wait(empty(s), ((it / STAGES) & 1) ^ 1, abort_flag, 5);
            if (!ok) return;
#pragma unroll
            for (int c = 0; c < 4; c++) *reinterpret_cast<uint4*>(a_row[c] + s * A_BYTES) = out[c];
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full_a(s));
        };
        static_assert(AHEAD == 3, "the loop below names the slots");
#pragma unroll
        for (int d = 0; d < AHEAD; d++) fetch(raw[d], scale[d]);
        const int q = warp & 3, part = dqw >> 2;                     // epilogue: tensor memory lanes 32q.., columns 16 part + 64 i
        float* const own = reinterpret_cast<float*>(smem);           // [NX][128]: this CTA's sums, where the stages were
        int it = grp, slot = 0, ends = 0;                            // this group's next slab, its slot, the slab behind the tile
        for (int seg = 0; seg < my_tiles && ok; seg++) {
            const int tile = first_tile + seg * step, n0 = tile / p.tiles_m * BM + second * BN, m0 = (tile % p.tiles_m) * p.NX;
            ends += nkb;
            for (; it < ends && ok; it += C::GROUPS) {
                if (slot == 0) slab(raw[0], scale[0], it);
                else if (slot == 1) slab(raw[1], scale[1], it);
                else slab(raw[2], scale[2], it);
                slot = slot == 2 ? 0 : slot + 1;
            }
            const int r = q * 32 + lane, there = ranks == 1 && n0 + r < p.N ? p.M - m0 : 0;
            auto place = [&](int c) { return (size_t)(m0 + c) * p.N + n0 + r; };
            uint32_t w[16];
            auto ahead = [&](int c) { operands(p.out, p.gate, p.mode, place(c), p.N, min(p.NX, there) - c, w); };
            ahead(part * 16);
            ok = ok && warp_wait(done_bar, seg & 1, abort_flag, 6);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // ---- D[n][m] (lane = weight row, column = activation row) -> Y[m][n], or into shared memory for the cluster
            if (ok) {
                for (int c0 = part * 16; c0 < p.NX; c0 += 64) {
                    float f[16];
                    tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, f);
                    if (ranks == 1) {
                        combine(p.mode, w, f);
                        ahead(c0 + 64);
                        store(p.out, p.mode, place(c0), p.N, min(p.NX, there) - c0, f);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) own[(c0 + j) * 128 + r] = f[j];
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_first(free_bar);
                else mbar_arrive(free_bar);
            }
        }
    }
    if (ranks > 1) {                                                 // one tile, its K over the cluster: CTA r adds and finishes its share of the columns
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int n0 = first_tile / p.tiles_m * BN, m0 = (first_tile % p.tiles_m) * p.NX;
        if (warp >= 2 && !*abort_flag) {
            const int cols = min(p.NX, p.M - m0), per = (cols + (int)ranks - 1) / (int)ranks, c0 = (int)rank * per;
            const int r = lane * 4, quads = n0 + r < p.N ? (min(cols, c0 + per) - c0) * 32 : 0;      // four weight rows of a column each
            const bool whole = p.N % 4 == 0 && ((uintptr_t)p.out & 15) == 0 && ((uintptr_t)p.gate & 7) == 0;
            auto add = [&](auto most) {
                constexpr int R = decltype(most)::value, Q = 8 / R;
                for (int i = (warp - 2) * 32 + lane; i < quads; i += Q * DQ_THREADS) {
                    float x[Q][R][4];
                    uint32_t w[Q][4];
                    auto place = [&](int at) { return (size_t)(m0 + c0 + (at >> 5)) * p.N + n0 + r; };
#pragma unroll
                    for (int j = 0; j < Q; j++)
                        if (i + j * DQ_THREADS < quads) {
                            if (whole) operands4(p.out, p.gate, p.mode, place(i + j * DQ_THREADS), w[j]);
                            else operands(p.out, p.gate, p.mode, place(i + j * DQ_THREADS), 1, p.N - n0 - r, w[j]);
                        }
#pragma unroll
                    for (int j = 0; j < Q; j++)
#pragma unroll
                        for (int k = 0; k < R; k++)
                            if (i + j * DQ_THREADS < quads && k < (int)ranks) {
                                uint32_t at;
                                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(sbase + (uint32_t)((c0 * 32 + i + j * DQ_THREADS) * 16)), "r"(k));
                                asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                                             : "=f"(x[j][k][0]), "=f"(x[j][k][1]), "=f"(x[j][k][2]), "=f"(x[j][k][3]) : "r"(at) : "memory");
                            }
#pragma unroll
                    for (int j = 0; j < Q; j++) {
                        const int at = i + j * DQ_THREADS;
                        if (at >= quads) break;
                        float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int k = 0; k < R; k++)
                            if (k < (int)ranks)
#pragma unroll
                                for (int e = 0; e < 4; e++) v[e] += x[j][k][e];
                        combine(p.mode, w[j], v);
                        if (whole) store4(p.out, p.mode, place(at), v);
                        else store(p.out, p.mode, place(at), 1, p.N - n0 - r, v);
                    }
                }
            };
            if (ranks <= 2) add(std::integral_constant<int, 2>());
            else if (ranks <= 4) add(std::integral_constant<int, 4>());
            else add(std::integral_constant<int, 8>());
        }
        // Nobody leaves while its sums are read. Every value read has been used by now, and nobody in the cluster reads what was stored:
        // no release, which would wait for those stores.
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;\n barrier.cluster.wait.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");      // nobody reads or arrives there any more
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int get_encoder(EncodeTiledFn* out) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        CMLB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        CMLB_REQUIRE(p && q == cudaDriverEntryPointSuccess, "cuTensorMapEncodeTiled is not available in this driver");
        fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    *out = fn;
    return CMLB200_OK;
}

// A call's shape: tiles of 128 weight rows by NX activation rows, the K of a tile shared by `ranks` CTAs
struct Shape { int NX, ranks; bool pair; };

// How many clusters of each size run at once, one CTA an SM: a cluster lies in one GPC, and how many SMs those have is the device's
// own affair. B200: 74 clusters of two, 45, 33, 26, 22, 15, 15 of eight.
template <typename Kern>
const int* clusters_at_once(Kern kern, size_t smem) {
    static int counts[kMaxDevices][9] = {};
    static std::mutex mutex;
    std::lock_guard<std::mutex> lock(mutex);
    int* c = counts[cmlb_device_index()];
    if (c[1]) return c;
    const int sms = cmlb_num_sms();
    for (int ranks = 8; ranks >= 1; ranks--) {                          // (c[1] last)
        int n = 0;
        if (ranks == 1) n = sms;
        else {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(ranks);
            cfg.blockDim = dim3(THREADS);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = ranks;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
        }
        c[ranks] = n;
    }
    return c;
}

// Estimated time (us) of a shape: waves of tiles, each K / 64 / ranks slabs of `expand` us for the weights and 0.14 for every 256
// activation rows, a few us to fill the pipeline and for the epilogue, and for a cluster's sum. Fitted to all shapes of 504 calls (three
// formats, 640 to 32000 weight rows, 1024 to 14336 columns, 33 to 2048 rows of x) before there were pairs and with a sum that took 1 to 2
// us more: 7 % rms then, the shape picked 0.3 % off the best one on average. What the sum takes now (about 1.2 + 0.009 NX + 0.15 ranks)
// would change the pick of one call in twenty, by 1 to 5 % of the estimate, less than its error. 4096x4096, Q4_0, 77 rows: 13.9 us
// with four ranks (32 of the 33 clusters that fit); with the former sum 14.2, 16.0 with three, 27.1 without.
// What it picks above 256 rows, pairs or not, against the best form without pairs (1, 2, 4 or 8 CTAs to a tile; three formats, ten shapes of weights,
// 257 to 2048 rows, 210 calls): 0.86 of its time on average, 0.68 at 32000x4096 (Q4_0, 512 rows: 99.8 and 128 us; 257: 68.2 and 112); more than 3 %
// behind it in nine calls, the worst of short K (NF4 4096x1024, 257 rows: 13.8 and 11.9), where a pair's MMA and expansion do not add up as the estimate has it.
inline double shape_cost(const Shape& s, int M, int N, int KB, const int* at_once, double expand) {
    const int together = s.pair ? 2 : s.ranks, rows = s.pair ? 2 * BN : BN;
    if (!at_once[together] || (s.ranks > 1 && s.NX > B_ROWS)) return 1e30;
    const int tiles = ((M + s.NX - 1) / s.NX) * ((N + rows - 1) / rows);
    const double slab = expand + 0.14 * s.NX / 256;
    const int waves = (tiles + at_once[together] - 1) / at_once[together];
    return waves * (((KB + s.ranks - 1) / s.ranks) * slab + 3.7 + 0.008 * s.NX + (s.ranks > 1 ? 1.5 + 0.014 * s.NX + 0.25 * s.ranks : 0.0));
}
inline Shape pick_shape(int M, int N, int KB, const int* at_once, double expand) {
    Shape best = {16, 1, false};
    double least = 1e300;
    const int tm0 = (M + 511) / 512, tm1 = (M + 255) / 256;
    for (int tm = tm0; tm <= tm1 + min(tm1 + 1, 8); tm++)
        for (int ranks = 1; ranks <= 8; ranks++) {
            if (ranks > 1 && KB < 2 * ranks) continue;
            Shape s = {((M + tm - 1) / tm + 15) / 16 * 16, ranks, false};
            if (s.NX > B_ROWS) {
                if (ranks > 1) continue;
                s.NX = max((s.NX + 31) / 32 * 32, B_ROWS + 32);            // (a pair's MMA has whole 32 columns)
                s.pair = true;
            }
            const double c = shape_cost(s, M, N, KB, at_once, expand);
            if (c < least) { least = c; best = s; }
        }
    return best;
}

template <int TYPE, bool PAIR>
int launch_tiles(const cmlb200_qmat* W, const uint16_t* x, void* y, const uint16_t* gate, int mode, int M, const Shape& shape, int pairs_at_once, cudaStream_t st) {
    using C = Cfg<TYPE, PAIR>;
    const int N = W->rows, K = W->cols;
    GemmArgs a = {};
    a.NX = shape.NX;
    a.tiles_m = (M + a.NX - 1) / a.NX;
    a.tiles = (N + (PAIR ? 2 : 1) * BN - 1) / ((PAIR ? 2 : 1) * BN) * a.tiles_m;
    a.qs = (const uint8_t*)W->qs;
    a.scales = W->scales;
    a.out = y;
    a.gate = (const __nv_bfloat16*)gate;
    a.mode = mode;
    a.M = M;
    a.N = N;
    a.K = K;
    a.nf4_block = W->block;
    a.nf4_shift = W->block == 32 ? 0 : W->block == 64 ? 1 : W->block == 128 ? 2 : W->block == 256 ? 3 : -1;
    EncodeTiledFn enc;
    int rc = get_encoder(&enc);
    if (rc) return rc;
    CUtensorMap xmap;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)min(a.NX, B_ROWS) / (PAIR ? 2 : 1)};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)x, dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CMLB_REQUIRE(cr == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with %d (x must be 16-byte aligned, K*2 a multiple of 16)", (int)cr);
    auto kern = gemm_kernel<TYPE, PAIR>;
    static size_t attr[kMaxDevices] = {};
    const size_t smem = C::total + 1024;
    CMLB_CUDA(cmlb_ensure_smem(kern, smem, attr));
    cudaLaunchConfig_t cfg = {};
    const int ranks = PAIR ? 2 : shape.ranks;
    cfg.gridDim = dim3((unsigned)(PAIR ? 2 * min(a.tiles, pairs_at_once) : ranks > 1 ? a.tiles * ranks : min(a.tiles, cmlb_num_sms())));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = ranks;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    CMLB_CUDA(cudaLaunchKernelEx(&cfg, kern, xmap, a));
    return CMLB200_OK;
}

template <int TYPE>
int launch_gemm(const cmlb200_qmat* W, const uint16_t* x, void* y, const uint16_t* gate, int mode, int M, int splits, cudaStream_t st) {
    const int KB = (W->cols + BK - 1) / BK;
    auto kern = gemm_kernel<TYPE, false>;
    static size_t attr[kMaxDevices] = {};
    const size_t smem = Cfg<TYPE, false>::total + 1024;
    CMLB_CUDA(cmlb_ensure_smem(kern, smem, attr));
    const int* at_once = clusters_at_once(kern, smem);
    Shape s = pick_shape(M, W->rows, KB, at_once, TYPE == CMLB200_Q8_0 ? 0.53 : TYPE == CMLB200_NF4 ? 0.47 : 0.32);
    if (splits > 0) {                                                    // the caller's choice, as far as a cluster and the slabs go
        const int tm = (M + 255) / 256;
        s.NX = ((M + tm - 1) / tm + 15) / 16 * 16;
        s.ranks = 1;
        s.pair = false;
        while (2 * s.ranks <= splits && 2 * s.ranks <= KB && s.ranks < 8) s.ranks *= 2;
    }
    return s.pair ? launch_tiles<TYPE, true>(W, x, y, gate, mode, M, s, at_once[2], st) : launch_tiles<TYPE, false>(W, x, y, gate, mode, M, s, 0, st);
}

int gemm_entry(const cmlb200_qmat* W, const uint16_t* x, void* y, const uint16_t* gate, int mode, int M, int ctas, void* stream) {
    CMLB_REQUIRE(W && W->qs && W->scales && x && y, "cmlb200_gemm_bf16: NULL argument");
    CMLB_REQUIRE(mode >= GEMM_OUT_BF16 && mode <= GEMM_SWIGLU_BF16 && (mode != GEMM_SWIGLU_BF16 || gate), "cmlb200_gemm_bf16_ex: bad output mode %d", mode);
    CMLB_REQUIRE(M >= 1, "cmlb200_gemm_bf16: M=%d must be positive", M);
    CMLB_REQUIRE(W->rows > 0 && W->cols > 0 && W->cols % 32 == 0, "cmlb200_gemm_bf16: cols=%d must be a positive multiple of 32", W->cols);
    CMLB_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)W->qs & 15) == 0 && ((uintptr_t)W->scales & 3) == 0,
                 "cmlb200_gemm_bf16: x and the weight planes must be 16-byte aligned");
    cudaStream_t st = as_stream(stream);
    switch (W->type) {
        case CMLB200_Q8_0: return launch_gemm<CMLB200_Q8_0>(W, x, y, gate, mode, M, ctas, st);
        case CMLB200_Q4_0: return launch_gemm<CMLB200_Q4_0>(W, x, y, gate, mode, M, ctas, st);
        case CMLB200_NF4:
            CMLB_REQUIRE(W->block >= 32 && W->block % 32 == 0 && W->cols % W->block == 0,
                         "cmlb200_gemm_bf16: NF4 block size %d must be a multiple of 32 that divides cols", W->block);
            return launch_gemm<CMLB200_NF4>(W, x, y, gate, mode, M, ctas, st);
        default: CMLB_REQUIRE(false, "cmlb200_gemm_bf16: unsupported weight type %d", W->type);
    }
    return CMLB200_EINVAL;
}

}  // namespace

extern "C" int cmlb200_gemm_bf16(const cmlb200_qmat* W, const uint16_t* d_x_bf16, uint16_t* d_y_bf16, int M, void* stream) {
    return gemm_entry(W, d_x_bf16, d_y_bf16, nullptr, GEMM_OUT_BF16, M, 0, stream);
}

extern "C" int cmlb200_gemm_bf16_ex(const cmlb200_qmat* W, const uint16_t* d_x_bf16, int M, int mode, void* d_out, const uint16_t* d_gate_bf16,
                                    void* stream) {
    return gemm_entry(W, d_x_bf16, d_out, d_gate_bf16, mode, M, 0, stream);
}

extern "C" int cmlb200_gemm_bf16_splitk(const cmlb200_qmat* W, const uint16_t* d_x_bf16, uint16_t* d_y_bf16, int M,
                                        int splits, void* stream) {
    CMLB_REQUIRE(splits >= 1, "cmlb200_gemm_bf16_splitk: splits must be >= 1");
    return gemm_entry(W, d_x_bf16, d_y_bf16, nullptr, GEMM_OUT_BF16, M, splits, stream);
}

extern "C" int cmlb200_gemm_status(int* status, int reset) {
    CMLB_REQUIRE(status, "cmlb200_gemm_status: NULL argument");
    CMLB_CUDA(cudaDeviceSynchronize());
    CMLB_CUDA(cudaMemcpyFromSymbol(status, g_gemm_status, sizeof(int)));
    if (reset) {
        const int zero = 0;
        CMLB_CUDA(cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(int)));
    }
    return CMLB200_OK;
}
