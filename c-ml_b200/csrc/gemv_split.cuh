// Decode GEMV, 1 to 32 rows of x, every block format C-ML reads (Q4_0, Q4_1, Q8_0, Q4_K, Q5_K, Q6_K of
// src/core/gguf_quant.c:66-311 and NF4 of src/core/quantization.c:195-370), on fp16 tensor cores
// (mma.sync m16n8k16, fp32 accumulation) with 32-bit accuracy:
//   * the quants are small integers, which fp16 holds exactly: A = 16 weight rows x 16 quants, made in registers with
//     one or two logic / packed-half operations per register;
//   * x is split into two fp16 numbers, x = hi + lo, after scaling by a power of two that puts the largest value of its
//     256-column unit just below 2^15: 23 bits of every value, and nothing below 2^-39 of the largest is lost;
//   * products and sums of one block are fp32 in the tensor core; block scales are applied to its sums in fp32, the
//     minima of Q4_K / Q5_K by one more small product (sub-block minima times sums of x), those of Q4_1 in fp32.
// Error against 64 bits on N(0,1) inputs: 1.2e-7 to 2e-7 of the result's norm, as the int8-digit kernels have.
//
// Work: item = 16 weight rows x 256 columns; the warps of a CTA share K (a warp takes every W-th 256-column unit), each
// with a ring of its own that cp.async fills, the first items (but NF4's) before the launch waits for its predecessor. Sums of the
// warps meet in shared memory and are added in warp order, so results do not depend on timing.
//
//   gemv_split_kernel   up to 8 rows of x. NT = 0: up to 4 rows, made into hi / lo columns of ONE 8-column product by the
//                       warp itself (columns 2r, 2r+1 = hi, lo of row r); NT = 1: 5 to 8 rows, planes from x_split_kernel.
//                       A warp keeps the B operands of its unit in registers and walks the CTA's row tiles.
//   gemv_split_wide_kernel   9 to 32 rows: B operands are loaded per block and used by T row tiles whose sums stay in registers;
//                       a warp has all columns of x, of short rows half of them.
//
// What bounds it: instructions and the chains between them. A block of 16 x 32 weights at M = 1 takes a thread about 50 (10 to unpack, 6 to
// address and load, 2 products, 8 to apply the scales, the rest the rows of x); logic operations, permutes and packed halves issue every
// second cycle; tensor pipe 44 % busy at M = 32 (mma.sync: 2 cycles a product and SM), DRAM 24 % at M = 1. Sixteen warps (128 registers)
// beat eight with 255 up to 16 rows: 8.2 against 10.4 us at M = 1 (Q4_0 11008x4096), 9.9 against 11.4 at M = 16 (4096x4096); from 17 rows
// on eight are the faster ones, but for short rows. More chains of products (the block's halves apart) cost more additions than they hid: 14.3 against
// 12.9 us at M = 8. The same products by tcgen05.mma, weights put into tensor memory block by block, were no faster: a block's sums have a
// place of their own there and are read back, and every step of that pipeline (a wait, two fences, an arrival, 550 cycles from an
// MMA to who waits for it) costs more than the mma.sync it saves: 34.5 us at M = 32, 17.4 at M = 16 (Q4_0 11008x4096). Times: gemv.cu.
#pragma once
#include "common.cuh"
#include "mma_util.cuh"

namespace {

enum { EPI_STORE = 0, EPI_ACCUM = 1, EPI_SWIGLU = 2 };

// Shared memory of one weight row's 256-column unit: bytes of quants (and headers) as they lie in memory, block scales
// behind them. Row strides are odd multiples of 16 bytes (mod 128), so eight rows hit eight bank groups.
// NF4: of blocks of 64 and more, of blocks of 32; both without the table of codes
constexpr int kNF4Fine = CMLB200_NF4 + 1, kNF4Bare = CMLB200_NF4 + 2, kNF4FineBare = CMLB200_NF4 + 3;
template <int F> constexpr bool kNF4Like = F >= CMLB200_NF4 && F <= kNF4FineBare;
template <int F> constexpr bool kTable = F == CMLB200_NF4 || F == kNF4Fine;
template <int F> struct Lay;
template <> struct Lay<CMLB200_Q4_0> { static constexpr int ROW = 144, CH = 8, SC = 128; };
template <> struct Lay<CMLB200_Q8_0> { static constexpr int ROW = 272, CH = 16, SC = 256; };
template <> struct Lay<CMLB200_NF4> { static constexpr int ROW = 144, CH = 8, SC = 128; };         // blocks of 64 and more
template <> struct Lay<kNF4Fine> { static constexpr int ROW = 176, CH = 8, SC = 128; };            // of 32: eight scales
template <> struct Lay<kNF4Bare> : Lay<CMLB200_NF4> {};
template <> struct Lay<kNF4FineBare> : Lay<kNF4Fine> {};
template <> struct Lay<CMLB200_Q4_1> { static constexpr int ROW = 176, CH = 10, SC = 0; };
template <> struct Lay<CMLB200_Q4_K> { static constexpr int ROW = 144, CH = 9, SC = 0; };
template <> struct Lay<CMLB200_Q5_K> { static constexpr int ROW = 176, CH = 11, SC = 0; };
template <> struct Lay<CMLB200_Q6_K> { static constexpr int ROW = 240, CH = 15, SC = 0; };   // the aligned window around 210 bytes
template <int F> constexpr int kTileBytes = 16 * Lay<F>::ROW;
template <int F> constexpr bool kMins = F == CMLB200_Q4_1 || F == CMLB200_Q4_K || F == CMLB200_Q5_K;     // formats with minima

struct SplitArgs {
    const uint8_t *qs, *qs2;       // weight, second weight (SwiGLU: gate, up)
    const uint8_t *sc, *sc2;       // scales (Q4_0, Q8_0: fp16, NF4: fp32)
    const float* x;                // fp32 rows (NT = 0)
    const __half* nw;              // RMSNorm weight applied to them, or nullptr
    const uint4* planes;           // split rows (NT > 0): [block][NT][hi, lo][lane]
    const float* sums;             // their sums over blocks: [block][8 NT]
    const float* xf;               // power of two that undoes the scaling: [unit][8 NT]
    float* y;
    float eps;
    int N, K, M, tiles, per_cta, stages, epi;
    int lut;                       // NF4: where in shared memory the table of codes lies (whole 16 bytes)
    int extra;                     // 9 rows and more: where in shared memory the address of tensor memory and the scalings go
    int nf4_shift;                 // log2 of how many 32-column blocks one NF4 scale covers, 3 at most
    int nf4_units;                 // units one covers, 1 at least
    bool deep;                     // split_deep's answer: x_split_kernel and the product have to go by the same one
};

// Shared memory through pointers, so that the compiler may order the loads as it likes between the waits
typedef const uint8_t* Shared;
__device__ __forceinline__ uint32_t lds32(Shared p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ uint32_t lds16(Shared p) { return *reinterpret_cast<const uint16_t*>(p); }
__device__ __forceinline__ float ldsf(Shared p) { return *reinterpret_cast<const float*>(p); }
__device__ __forceinline__ void cp_async16_part(uint32_t dst, const void* src, int bytes) {     // the rest is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4_part(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t m, uint32_t o) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(m), "r"(o));
    return d;
}
__device__ __forceinline__ uint32_t hfma2u(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t hadd2u(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

constexpr float kNF4Unit = 16384.0f / 10000.0f;      // what a product of NF4 digits counts

// ---- weights: global memory -> ring ---------------------------------------------------------------------------------
template <int F> __device__ __forceinline__ size_t row_bytes(int nblk) {
    return F == CMLB200_Q8_0 ? (size_t)nblk * 32 : F == CMLB200_Q4_1 ? (size_t)nblk * 20 : F == CMLB200_Q4_K ? (size_t)nblk * 18 :
           F == CMLB200_Q5_K ? (size_t)nblk * 22 : F == CMLB200_Q6_K ? (size_t)nblk / 8 * 210 : (size_t)nblk * 16;
}
// Where a lane's 16-byte pieces of an item lie from its first row on (items whose 16 rows all exist)
template <int F> struct Pieces {
    static constexpr int CH = Lay<F>::CH, COUNT = (16 * CH + 31) / 32;
    uint32_t off[F == CMLB200_Q6_K ? 1 : COUNT];
    __device__ __forceinline__ void init(int nblk, int lane) {
        if constexpr (F != CMLB200_Q6_K) {
#pragma unroll
            for (int i = 0; i < COUNT; i++) {
                const int c = lane + 32 * i;
                off[i] = (uint32_t)(c / CH) * (uint32_t)row_bytes<F>(nblk) + (uint32_t)(c % CH) * 16u;
            }
        }
    }
};
// One item: rows row0 .. row0+15 (rows past N repeat row N-1; never written out), columns of unit `un`.
template <int F>
__device__ __forceinline__ void issue_tile(const SplitArgs& p, const Pieces<F>& pc, int which, int row0, int un, uint32_t dst, int lane) {
    constexpr int ROW = Lay<F>::ROW, CH = Lay<F>::CH;
    const int nblk = p.K / 32, last = p.N - 1;
    const uint8_t *qs = which ? p.qs2 : p.qs, *sc = which ? p.sc2 : p.sc;
    const size_t rb = row_bytes<F>(nblk);
    if (F == CMLB200_Q6_K) {
        const size_t total = rb * p.N;
#pragma unroll
        for (int i = 0; i < (16 * CH + 31) / 32; i++) {
            const int c = lane + 32 * i, r = c / CH, ch = c % CH;
            if (c < 16 * CH) {
                const size_t o = (size_t)min(row0 + r, last) * rb + (size_t)un * 210, at = (o & ~(size_t)15) + 16 * ch;
                const int n = at >= o + 210 ? 0 : (total - at < 16 ? (int)(total - at) : 16);
                cp_async16_part(dst + r * ROW + ch * 16, n ? qs + at : qs, n);
            }
        }
        return;
    }
    if (row0 + 16 <= p.N && (un + 1) * 8 <= nblk) {
        const uint8_t* base = qs + (size_t)row0 * rb + (size_t)un * (CH * 16);
#pragma unroll
        for (int i = 0; i < Pieces<F>::COUNT; i++) {
            const int c = lane + 32 * i;
            if (16 * CH % 32 == 0 || c < 16 * CH) cp_async16(dst + (c / CH) * ROW + (c % CH) * 16, base + pc.off[F == CMLB200_Q6_K ? 0 : i]);
        }
    } else {
        const int left = nblk - un * 8;                                      // blocks of the unit that exist
        const int have = F == CMLB200_Q8_0 ? 2 * left : F == CMLB200_Q4_0 || kNF4Like<F> ? left : CH;
#pragma unroll 1
        for (int c = lane; c < 16 * CH; c += 32) {
            const int r = c / CH, ch = c % CH;
            const uint8_t* src = qs + (size_t)min(row0 + r, last) * rb + (size_t)un * (CH * 16) + ch * 16;
            cp_async16_part(dst + r * ROW + ch * 16, ch < have ? src : qs, ch < have ? 16 : 0);
        }
    }
    if (F == CMLB200_Q4_0 || F == CMLB200_Q8_0) {
        if (lane < 16) cp_async16(dst + lane * ROW + Lay<F>::SC, sc + 2 * ((size_t)min(row0 + lane, last) * nblk + (size_t)un * 8));
    } else if (kNF4Like<F>) {                                          // absmax: one for a few blocks, or for units
        const int ws = 3 - p.nf4_shift, words = 1 << ws, per_row = (nblk >> p.nf4_shift) / p.nf4_units, first = (un << ws) / p.nf4_units;
        for (int c = lane; c < 16 * words; c += 32) {
            const int r = c >> ws, k = c & (words - 1);
            const bool ok = first + k < per_row;
            const uint8_t* src = sc + 4 * ((size_t)min(row0 + r, last) * per_row + first + k);
            cp_async4_part(dst + r * ROW + Lay<F>::SC + 4 * k, ok ? src : sc, ok ? 4 : 0);
        }
    }
}

// ---- weights: ring -> A operands --------------------------------------------------------------------------------------
// A thread (g, t) = (lane / 4, lane % 4) of the product holds rows g and g + 8. Of a 32-column block it takes columns 4t .. 4t+3
// and 16+4t .. 16+4t+3 in the order (0,2) (1,3) (4,6) (5,7) of the eight, of NF4 8t .. 8t+7 as they are; the B operands have the same order,
// and the order of columns inside a product is free. a[0], a[1]: the two m16n8k16 of the block; NF4: two digits of the value.
template <int F> constexpr int kDigits = kNF4Like<F> ? 2 : 1;

// 4-bit formats: word w holds the eight nibbles of one row
__device__ __forceinline__ void nibbles(uint32_t w, uint32_t magic, uint32_t (&h)[4]) {
    const uint32_t v = w >> 8;
    h[0] = and_or(w, 0x000f000fu, magic);
    h[1] = and_or(v, 0x000f000fu, magic);
    h[2] = and_or(w, 0x00f000f0u, magic);
    h[3] = and_or(v, 0x00f000f0u, magic);
}

template <int F>
__device__ __forceinline__ void row_regs(Shared at, int b, int t, uint32_t w0, uint32_t w1, uint32_t off, Shared lut, uint32_t (&h)[kDigits<F>][4]) {
    if constexpr (F == CMLB200_Q4_0 || F == CMLB200_Q4_1 || F == CMLB200_Q4_K) {     // q - 8 from 1024 + q and 1024 + 16 q
        uint32_t n[4];
        nibbles(w0, 0x64006400u, n);
        h[0][0] = hadd2u(n[0], 0xe408e408u);                     // - 1032
        h[0][1] = hadd2u(n[1], 0xe408e408u);
        h[0][2] = hfma2u(n[2], 0x2c002c00u, 0xd480d480u);        // / 16 - 72
        h[0][3] = hfma2u(n[3], 0x2c002c00u, 0xd480d480u);
    } else if constexpr (F == CMLB200_Q8_0) {                   // int8 from 1024 + (q + 128)
        const uint32_t u0 = w0 ^ 0x80808080u, u1 = w1 ^ 0x80808080u;
        h[0][0] = hadd2u(__byte_perm(u0, 0x64646464u, 0x4240), 0xe480e480u);
        h[0][1] = hadd2u(__byte_perm(u0, 0x64646464u, 0x4341), 0xe480e480u);
        h[0][2] = hadd2u(__byte_perm(u1, 0x64646464u, 0x4240), 0xe480e480u);
        h[0][3] = hadd2u(__byte_perm(u1, 0x64646464u, 0x4341), 0xe480e480u);
    } else if constexpr (F == CMLB200_Q5_K) {                   // bit 4 from the block's word of high bits: w1 = bits of columns 0..31
        const uint32_t v = w0 >> 4, b4 = w1 >> (4 * t);          // bits 0-3: columns 4t.., bits 16-19: columns 16+4t..
        // columns 0 and 2 (1 and 3) of the four: bits 0 and 2 (1 and 3) to bit 4 of the two halves, by a multiplication; q - 16 from 1024 + q
        const uint32_t top = b4 >> 16;
        h[0][0] = hadd2u(and_or((b4 & 5u) * 0x00040010u, 0x00100010u, and_or(w0, 0x000f000fu, 0x64006400u)), 0xe410e410u);
        h[0][1] = hadd2u(and_or((b4 & 10u) * 0x00020008u, 0x00100010u, and_or(w0 >> 8, 0x000f000fu, 0x64006400u)), 0xe410e410u);
        h[0][2] = hadd2u(and_or((top & 5u) * 0x00040010u, 0x00100010u, and_or(v, 0x000f000fu, 0x64006400u)), 0xe410e410u);
        h[0][3] = hadd2u(and_or((top & 10u) * 0x00020008u, 0x00100010u, and_or(v >> 8, 0x000f000fu, 0x64006400u)), 0xe410e410u);
    } else if constexpr (F == CMLB200_Q6_K) {                   // q - 32 from 1024 + q
#pragma unroll
        for (int k = 0; k < 2; k++) {
            // a byte's four pairs of high bits: to the places beside the nibbles by a multiplication, two at a time
            const uint32_t q = lds16(at + off + 16 * b + 8 * k + 2 * t), hb = at[off + 128 + 8 * b + 4 * k + t], w = __byte_perm(q, 0, 0x4140);
            h[0][2 * k] = hadd2u(and_or(hb * 0x00010010u, 0x00300030u, and_or(w, 0x000f000fu, 0x64006400u)), 0xe420e420u);              // - 1056
            h[0][2 * k + 1] = hadd2u(and_or(hb * 0x00004004u, 0x00300030u, and_or(w >> 4, 0x000f000fu, 0x64006400u)), 0xe420e420u);
        }
    } else if constexpr (!kTable<F>) {                          // NF4: 10000 times the code = 128 a + b, digits by byte table look-ups
        // a + 128 and b + 128 of the 16 codes (|b| <= 64), four to a word
        constexpr uint32_t A0 = 0x61574a32u, A1 = 0x8079726au, A2 = 0x9a938d86u, A3 = 0xceb8aca2u;
        constexpr uint32_t B0 = 0x937d4e70u, B1 = 0x80714864u, B2 = 0xb39d499cu, B3 = 0x90be7ab7u;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t w = k ? w0 >> 16 : w0;
            const uint32_t s = w & 0x7777u, pick = and_or(w >> 1, 0x4444u, 0x3210u);
            const uint32_t va = __byte_perm(__byte_perm(A0, A1, s), __byte_perm(A2, A3, s), pick);
            const uint32_t vb = __byte_perm(__byte_perm(B0, B1, s), __byte_perm(B2, B3, s), pick);
            // bytes: columns 1, 0, 3, 2. 1024 + (a + 128) -> a * 2^-7, 1024 + (b + 128) -> b * 2^-14
            h[0][2 * k] = hfma2u(__byte_perm(va, 0x64646464u, 0x4041), 0x20002000u, 0xc880c880u);
            h[0][2 * k + 1] = hfma2u(__byte_perm(va, 0x64646464u, 0x4243), 0x20002000u, 0xc880c880u);
            h[1][2 * k] = hfma2u(__byte_perm(vb, 0x64646464u, 0x4041), 0x04000400u, 0xac80ac80u);
            h[1][2 * k + 1] = hfma2u(__byte_perm(vb, 0x64646464u, 0x4243), 0x04000400u, 0xac80ac80u);
        }
    } else {                                                    // a byte's two codes from a table
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint2 v = *reinterpret_cast<const uint2*>(lut + ((k ? w0 >> (8 * k - 7) : w0 << 7) & 0x7f80u));
            h[0][k] = v.x;
            h[1][k] = v.y;
        }
    }
}

// NF4: for every byte the two codes (the high nibble's first) as fp16 numbers a 2^-7, then b 2^-14: 8 bytes, a copy for each lane of half a
// warp, so that lanes with different bytes read different banks. Beside 10 byte permutes and 4 multiplications for 4 codes (ALU: two cycles
// each) it takes 2 shifts, 2 masks and a load: 4096x4096, a launch's products of 4 rows 9,000 cycles before.
constexpr int kLutBytes = 256 * 128;
__device__ __forceinline__ void fill_lut(uint8_t* lut) {
    for (int i = threadIdx.x; i < 512; i += blockDim.x) {
        uint32_t digits[2] = {0u, 0u};
#pragma unroll
        for (int n = 0; n < 2; n++) {
            const int v = __float2int_rn(kNF4[(i >> (n ? 1 : 5)) & 15] * 10000.0f), b = ((v + 64) & 127) - 64, a = (v - b) >> 7;
            digits[0] |= (uint32_t)__half_as_ushort(__float2half_rn((float)a * 0x1p-7f)) << (16 * n);
            digits[1] |= (uint32_t)__half_as_ushort(__float2half_rn((float)b * 0x1p-14f)) << (16 * n);
        }
        const uint4 v = make_uint4(digits[0], digits[1], digits[0], digits[1]);
#pragma unroll
        for (int k = 0; k < 4; k++) *reinterpret_cast<uint4*>(lut + (i >> 1) * 128 + (i & 1) * 64 + 16 * k) = v;
    }
    __syncthreads();
}

// The words of block b that row_regs wants (row at shared address `at`)
template <int F>
__device__ __forceinline__ void row_words(Shared at, int b, int t, uint32_t& w0, uint32_t& w1) {
    if (F == CMLB200_Q4_0 || kNF4Like<F>) w0 = lds32(at + 16 * b + 4 * t);
    else if (F == CMLB200_Q8_0) { w0 = lds32(at + 32 * b + 4 * t); w1 = lds32(at + 32 * b + 16 + 4 * t); }
    else if (F == CMLB200_Q4_1) w0 = lds32(at + 20 * b + 4 + 4 * t);
    else if (F == CMLB200_Q4_K) w0 = lds32(at + 16 + 16 * b + 4 * t);
    else if (F == CMLB200_Q5_K) { w0 = lds32(at + 48 + 16 * b + 4 * t); w1 = lds32(at + 16 + 4 * b); }
}

template <int F>
__device__ __forceinline__ void block_regs(Shared lo, Shared hi, int b, int t, uint32_t off_lo, uint32_t off_hi, Shared lut, uint32_t (&a)[kDigits<F>][2][4]) {
    uint32_t w0 = 0, w1 = 0, v0 = 0, v1 = 0, r[kDigits<F>][4], s[kDigits<F>][4];
    row_words<F>(lo, b, t, w0, w1);
    row_words<F>(hi, b, t, v0, v1);
    row_regs<F>(lo, b, t, w0, w1, off_lo, lut, r);
    row_regs<F>(hi, b, t, v0, v1, off_hi, lut, s);
#pragma unroll
    for (int d = 0; d < kDigits<F>; d++)
#pragma unroll
        for (int k = 0; k < 2; k++) {
            a[d][k][0] = r[d][2 * k];
            a[d][k][1] = s[d][2 * k];
            a[d][k][2] = r[d][2 * k + 1];
            a[d][k][3] = s[d][2 * k + 1];
        }
}

// What a row's header says, decoded once per item
struct Head { float d, m; uint32_t s0, s1, m0, m1, off; };

template <int F>
__device__ __forceinline__ void head_of(const SplitArgs& p, Shared at, int row, int un, Head& h) {
    if (F == CMLB200_Q4_K || F == CMLB200_Q5_K) {
        const uint4 v = *reinterpret_cast<const uint4*>(at);
        h.d = cml_half_to_float((uint16_t)(v.x & 0xffffu));
        h.m = cml_half_to_float((uint16_t)(v.x >> 16));
        h.s0 = v.y & 0x3f3f3f3fu;                                                  // scales of sub-blocks 0-3, 4-7, then minima
        h.s1 = (v.w & 0x0f0f0f0fu) | ((v.y >> 2) & 0x30303030u);
        h.m0 = v.z & 0x3f3f3f3fu;
        h.m1 = ((v.w >> 4) & 0x0f0f0f0fu) | ((v.z >> 2) & 0x30303030u);
    } else if (F == CMLB200_Q6_K) {
        const size_t o = (size_t)min(row, p.N - 1) * ((size_t)p.K / 256 * 210) + (size_t)un * 210;
        h.off = (uint32_t)(o & 15);
        h.d = cml_half_to_float((uint16_t)lds16(at + h.off + 208));
    }
}

// Byte n of w as a float: 2^23 and the byte, less 2^23 (a permute and an addition; a shift, a mask and a conversion take twice the cycles)
__device__ __forceinline__ float byte_of(uint32_t w, int n) { return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440u + (uint32_t)n)) - 8388608.0f; }

// Scale of block b (Q6_K: of its half `k`)
template <int F, bool QUIRK>
__device__ __forceinline__ float scale_of(const SplitArgs& p, Shared at, const Head& h, int b, int k) {
    if (F == CMLB200_Q4_0 || F == CMLB200_Q8_0) {
        const uint16_t s = (uint16_t)lds16(at + Lay<F>::SC + 2 * b);
        return QUIRK ? cml_half_to_float(s) : __half2float(__ushort_as_half(s));
    }
    if (kNF4Like<F>) return ldsf(at + Lay<F>::SC + 4 * (b >> p.nf4_shift)) * kNF4Unit;
    if (F == CMLB200_Q4_1) return cml_half_to_float((uint16_t)lds16(at + 20 * b));
    if (F == CMLB200_Q6_K) return h.d * (float)(int)(int8_t)at[h.off + 192 + 2 * b + k];
    return h.d * byte_of(b < 4 ? h.s0 : h.s1, b & 3);
}

// What block b adds per sum of x: its minimum, and what the centring of its quants took off
template <int F>
__device__ __forceinline__ float offset_of(Shared at, const Head& h, int b, float scale) {
    if (F == CMLB200_Q4_1) return fmaf(8.0f, scale, cml_half_to_float((uint16_t)lds16(at + 20 * b + 2)));
    const float mn = h.m * byte_of(b < 4 ? h.m0 : h.m1, b & 3);
    return fmaf(F == CMLB200_Q5_K ? 16.0f : 8.0f, scale, -mn);
}

// ---- activations --------------------------------------------------------------------------------------------------------
// The power of two that brings values of magnitude up to `most` below 2^15, and its inverse
__device__ __forceinline__ void scaling(float most, float& up, float& down) {
    const int e = (int)(__float_as_uint(most) >> 23);
    const int f = min(268 - e, 253);                            // exponent field of 2^(14 - floor(log2 most))
    up = __uint_as_float((uint32_t)f << 23);
    down = __uint_as_float((uint32_t)(254 - f) << 23);
}
__device__ __forceinline__ float power(uint32_t field) { return __uint_as_float((field & 255u) << 23); }
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Eight values in the order of the product's columns
template <bool CONTIG> __device__ __forceinline__ void split8(const float (&e)[8], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int i = CONTIG ? 2 * k : 4 * (k >> 1) + (k & 1), j = CONTIG ? i + 1 : i + 2;
        split2(e[i], e[j], hi[k], lo[k]);
    }
}

// One output's sums of the warps, in four chains: fewer roundings one upon the other than in a row
template <int COLS> __device__ __forceinline__ float warp_sums(const float* src, int active) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < 16; w++)
        if (w < active) v[w & 3] += src[w * (COLS * 16)];
    return (v[0] + v[1]) + (v[2] + v[3]);
}

// Eight sums of a thread to and from eight columns of tensor memory
__device__ __forceinline__ void tmem_put8(uint32_t at, const float (&v)[4], const float (&w)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 ::"f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]), "r"(at) : "memory");
}
__device__ __forceinline__ void tmem_add8(uint32_t at, float (&v)[4], float (&w)[4]) {
    float r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(at));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 4; k++) { v[k] += r[k]; w[k] += r[4 + k]; }
}

// An output that came out infinite or not a number, once more by plain fp32 multiply-adds: an infinite x is no pair of fp16 numbers
// (inf - inf), and its products have signs. Formats whose former kernels had those results; rows as they are given.
template <int F>
__device__ __noinline__ float plain_dot(const uint8_t* qs, const uint8_t* sc, const float* x, int K, int row, int nf4_shift, int nf4_units) {
    const int nblk = K / 32, per_row = (nblk >> nf4_shift) / nf4_units;
    float sum = 0.f;
    for (int b = 0; b < nblk; b++) {
        const size_t blk = (size_t)row * nblk + b;
        const float s = kNF4Like<F> ? reinterpret_cast<const float*>(sc)[(size_t)row * per_row + (b >> nf4_shift) / nf4_units]
                                         : cml_half_to_float(reinterpret_cast<const uint16_t*>(sc)[blk]);
        float block = 0.f;
        for (int k = 0; k < 32; k++) {
            float w;
            if (F == CMLB200_Q8_0) w = (float)reinterpret_cast<const int8_t*>(qs)[blk * 32 + k];
            else if (F == CMLB200_Q4_0) w = (float)(int)((qs[blk * 16 + (k & 15)] >> (k < 16 ? 0 : 4)) & 15) - 8.0f;
            else w = kNF4[(qs[blk * 16 + (k >> 1)] >> (k & 1 ? 0 : 4)) & 15];
            block = fmaf(w, x[b * 32 + k], block);
        }
        sum = fmaf(block, s, sum);
    }
    return sum;
}
template <int F>
__device__ __forceinline__ float finite_or_plain(float v, const SplitArgs& p, int which, int row, int m) {
    if constexpr (kNF4Like<F> || F == CMLB200_Q8_0 || F == CMLB200_Q4_0)
        if (!(fabsf(v) <= 3.402823466e38f) && !p.nw)
            return plain_dot<F>(which ? p.qs2 : p.qs, which ? p.sc2 : p.sc, p.x + (size_t)m * p.K, p.K, row, p.nf4_shift, p.nf4_units);
    return v;
}

// ---- up to 8 rows of x ------------------------------------------------------------------------------------------------------
constexpr int kWarps = 16;
template <int NT> constexpr int kShares = 32 / NT;      // warps of a CTA with 8 NT columns of x
template <int F, int NT> constexpr int kRing = Lay<F>::ROW > 176 || F == kNF4Fine ? 2 : Lay<F>::ROW == 144 && NT ? 4 : 3;      // items per warp in flight
constexpr int kOwnBytes = 16 + 4 * 8 * 4;                                // NT = 0: a warp's scaling and block sums of its rows, behind the operands
constexpr int kXBytes = 2 * 8 * 4 * 16;                                  // operands of one row and unit: [hi, lo][block][t]

template <int F, int NT, bool QUIRK, int RING>
__global__ void __launch_bounds__(kWarps * 32, 1) gemv_split_kernel(const SplitArgs p) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int ROW = Lay<F>::ROW, TB = kTileBytes<F>, COLS = NT == 0 ? 4 : 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5, g = lane >> 2, t = lane & 3;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // shared memory: rings [W][RING][TB] | NT = 0: operands [W][M][kXBytes], scaling and sums [W][kOwnBytes] | sums [per_cta][W][COLS][16] | squares [W][4]
    Shared rings = smem + warp * (RING * TB);
    const uint32_t ring = smem_u32(rings);
    uint8_t* xs = smem + W * (RING * TB) + warp * (p.M * kXBytes);
    float* own = reinterpret_cast<float*>(smem + W * (RING * TB) + W * (p.M * kXBytes) + warp * kOwnBytes);
    float* part = reinterpret_cast<float*>(smem + W * (RING * TB) + (NT == 0 ? W * (p.M * kXBytes + kOwnBytes) : 0));
    float* squares = part + (size_t)p.per_cta * W * COLS * 16;
    const int units = (p.K + 255) / 256, nblk = p.K / 32, pairs = p.epi == EPI_SWIGLU;
    const int tile0 = blockIdx.x * p.per_cta, mine = min(p.per_cta, p.tiles - tile0);
    const int my_units = warp < units ? (units - warp + W - 1) / W : 0, items = my_units * mine;
    Pieces<F> pc;
    pc.init(nblk, lane);
    int iss = 0, iss_tile = 0, iss_un = warp;
    auto issue = [&](int buf) {
        if (iss < items) {
            const int tile = tile0 + iss_tile;
            issue_tile<F>(p, pc, pairs ? tile & 1 : 0, (pairs ? tile >> 1 : tile) * 16, iss_un, ring + buf * TB, lane);
            iss++;
            if (++iss_tile == mine) { iss_tile = 0; iss_un += W; }
        }
        cp_async_commit();
    };
    // weights do not depend on the launch before, but NF4 ones may: it may have quantized them, or written their scales
    if (kNF4Like<F>) {
        if (kTable<F>) fill_lut(smem + p.lut);
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
#pragma unroll
    for (int i = 0; i < RING; i++) issue(i);
    Shared lut = smem + (kTable<F> ? p.lut + (lane & 15) * 8 : 0);
    if (!kNF4Like<F>) asm volatile("griddepcontrol.wait;" ::: "memory");

    float ss[4] = {0.f, 0.f, 0.f, 0.f};
    int buf = 0;
    for (int u = 0; u < my_units; u++) {
        const int un = warp + u * W;
        uint32_t B[8][NT == 0 ? 4 : 8];                         // NT = 0: hi (even g) or lo (odd g) of row g/2; 1: hi, then lo of row g
        float s32[kMins<F> ? 8 : 1][2];                         // sums of x over the unit's blocks, of the thread's two columns
        float down = 1.f, down1 = 1.f;                          // undo the unit's scaling, of the thread's (two) columns
        if (NT == 0) {
            // one row at a time, eight columns a lane: block lane/4, the columns of thread t = lane%4 of the product
            __syncwarp();
            const int c0 = un * 256 + g * 32 + (kNF4Like<F> ? 8 : 4) * t, c1 = kNF4Like<F> ? c0 + 4 : c0 + 16;
            const bool real = un * 8 + g < nblk;
            float4 xa[4], xc[4];                                // every row is on its way before the first is looked at
#pragma unroll
            for (int m = 0; m < 4; m++) {
                xa[m] = xc[m] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (m < p.M && real) {
                    xa[m] = __ldcg(reinterpret_cast<const float4*>(p.x + (size_t)m * p.K + c0));
                    xc[m] = __ldcg(reinterpret_cast<const float4*>(p.x + (size_t)m * p.K + c1));
                }
            }
            uint2 na = make_uint2(0u, 0u), nc = na;
            if (p.nw && real) {
                na = *reinterpret_cast<const uint2*>(p.nw + c0);
                nc = *reinterpret_cast<const uint2*>(p.nw + c1);
            }
#pragma unroll
            for (int m = 0; m < 4; m++) {
                if (m >= p.M) break;
                float e[8] = {xa[m].x, xa[m].y, xa[m].z, xa[m].w, xc[m].x, xc[m].y, xc[m].z, xc[m].w};
                if (p.nw && real) {
                    const uint32_t h[4] = {na.x, na.y, nc.x, nc.y};
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[k]));
                        ss[m] = fmaf(e[2 * k], e[2 * k], fmaf(e[2 * k + 1], e[2 * k + 1], ss[m]));
                        e[2 * k] *= f.x;
                        e[2 * k + 1] *= f.y;
                    }
                }
                float most = 0.f, up, dn, sum = 0.f;
#pragma unroll
                for (int k = 0; k < 8; k++) most = fmaxf(most, fabsf(e[k]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
                scaling(most, up, dn);
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int k = 0; k < 8; k++) { e[k] *= up; sum += e[k]; }
                split8<kNF4Like<F>>(e, hi, lo);
                uint4* dst = reinterpret_cast<uint4*>(xs + m * kXBytes) + lane;
                dst[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                dst[32] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                if (kMins<F>) {
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    if (t == 0) own[4 + m * 8 + g] = sum;
                }
                if (lane == 0) own[m] = dn;
            }
            __syncwarp();
            const bool there = (g >> 1) < p.M;
#pragma unroll
            for (int b = 0; b < 8; b++) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (there) v = reinterpret_cast<const uint4*>(xs + (g >> 1) * kXBytes)[(g & 1) * 32 + 4 * b + t];
                B[b][0] = v.x; B[b][1] = v.y; B[b][2] = v.z; B[b][3] = v.w;
                if (kMins<F>) s32[kMins<F> ? b : 0][0] = t < p.M ? own[4 + t * 8 + b] : 0.f;
            }
            down = t < p.M ? own[t] : 0.f;
        } else {
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const uint4* src = p.planes + (size_t)(un * 8 + b) * 64 + lane;
                const uint4 h = __ldcg(src), l = __ldcg(src + 32);
                B[b][0] = h.x; B[b][1] = h.y; B[b][2] = h.z; B[b][3] = h.w;
                B[b][NT ? 4 : 0] = l.x; B[b][NT ? 5 : 0] = l.y; B[b][NT ? 6 : 0] = l.z; B[b][NT ? 7 : 0] = l.w;
                if (kMins<F>) {
                    const float2 v = __ldcg(reinterpret_cast<const float2*>(p.sums + (size_t)(un * 8 + b) * 8 + 2 * t));
                    s32[kMins<F> ? b : 0][0] = v.x;
                    s32[kMins<F> ? b : 0][1] = v.y;
                }
            }
            const float2 v = __ldcg(reinterpret_cast<const float2*>(p.xf + (size_t)un * 8 + 2 * t));
            down = v.x;
            down1 = v.y;
        }
        for (int i = 0; i < mine; i++) {
            const int tile = tile0 + i, row0 = (pairs ? tile >> 1 : tile) * 16;
            cp_async_wait<RING - 1>();
            __syncwarp();
            Shared lo = rings + buf * TB + g * ROW, hi = lo + 8 * ROW;
            Head hl, hh;
            head_of<F>(p, lo, row0 + g, un, hl);
            head_of<F>(p, hi, row0 + g + 8, un, hh);
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            // scales and minima that are bytes of a header: the four threads of a row work out those of two blocks each and pass them round
            // (Q4_K 4096x11008: 1 row 12.9 -> 12.0 us, 4 rows 16.5 -> 15.6; Q6_K of five rows and more is faster without, 54.0 and 55.1)
            constexpr bool SPREAD = F == CMLB200_Q4_K || F == CMLB200_Q5_K || (F == CMLB200_Q6_K && NT == 0);
            constexpr int C1 = F == CMLB200_Q6_K ? 1 : 0;       // Q6_K: a scale for each half
            float ps[2][2][C1 + 1], po[2][2];                   // [row][block][half]
            if (SPREAD) {
#pragma unroll
                for (int j = 0; j < 2; j++) {
#pragma unroll
                    for (int k = 0; k <= C1; k++) {
                        ps[0][j][k] = scale_of<F, QUIRK>(p, lo, hl, 2 * t + j, k);
                        ps[1][j][k] = scale_of<F, QUIRK>(p, hi, hh, 2 * t + j, k);
                    }
                    if (kMins<F>) {
                        po[0][j] = offset_of<F>(lo, hl, 2 * t + j, ps[0][j][0]);
                        po[1][j] = offset_of<F>(hi, hh, 2 * t + j, ps[1][j][0]);
                    }
                }
            }
            auto passed = [&](float v, int b) { return __shfl_sync(0xffffffffu, v, b >> 1, 4); };
#pragma unroll
            for (int b = 0; b < 8; b++) {
                uint32_t a[kDigits<F>][2][4];
                block_regs<F>(lo, hi, b, t, hl.off, hh.off, lut, a);
                float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
                for (int d = kDigits<F> - 1; d >= 0; d--) {     // small products first: the tensor core truncates, relative to the sum so far
                    if (NT) {
#pragma unroll
                        for (int k = 0; k < 2; k++) mma_f16(c[k * C1], a[d][k], B[b][NT ? 4 + 2 * k : 0], B[b][NT ? 5 + 2 * k : 0]);
                    }
#pragma unroll
                    for (int k = 0; k < 2; k++) mma_f16(c[k * C1], a[d][k], B[b][2 * k], B[b][2 * k + 1]);
                }
#pragma unroll
                for (int k = 0; k <= C1; k++) {
                    const float sl = SPREAD ? passed(ps[0][b & 1][k], b) : scale_of<F, QUIRK>(p, lo, hl, b, k);
                    const float sh = SPREAD ? passed(ps[1][b & 1][k], b) : scale_of<F, QUIRK>(p, hi, hh, b, k);
                    acc[0] = fmaf(c[k][0], sl, acc[0]);
                    acc[1] = fmaf(c[k][1], sl, acc[1]);
                    acc[2] = fmaf(c[k][2], sh, acc[2]);
                    acc[3] = fmaf(c[k][3], sh, acc[3]);
                    if (kMins<F> && k == 0) {
                        const float ml = SPREAD ? passed(po[0][b & 1], b) : offset_of<F>(lo, hl, b, sl), mh = SPREAD ? passed(po[1][b & 1], b) : offset_of<F>(hi, hh, b, sh);
                        const float x0 = s32[kMins<F> ? b : 0][0], x1 = s32[kMins<F> ? b : 0][1];
                        acc[0] = fmaf(x0, ml, acc[0]);
                        acc[2] = fmaf(x0, mh, acc[2]);
                        if (NT) { acc[1] = fmaf(x1, ml, acc[1]); acc[3] = fmaf(x1, mh, acc[3]); }
                    }
                }
            }
            __syncwarp();                                       // every lane is done with this buffer
            issue(buf);
            if (++buf == RING) buf = 0;
            float* dst = part + ((size_t)i * W + warp) * (COLS * 16);
            if (NT == 0) {
                float v0 = (acc[0] + acc[1]) * down, v1 = (acc[2] + acc[3]) * down;
                dst += t * 16 + g;
                if (u) { v0 += dst[0]; v1 += dst[8]; }
                dst[0] = v0;
                dst[8] = v1;
            } else {
                dst += 2 * t * 16 + g;
                acc[0] *= down; acc[1] *= down1; acc[2] *= down; acc[3] *= down1;
                if (u) { acc[0] += dst[0]; acc[1] += dst[16]; acc[2] += dst[8]; acc[3] += dst[24]; }
                dst[0] = acc[0];
                dst[16] = acc[1];
                dst[8] = acc[2];
                dst[24] = acc[3];
            }
        }
    }
    if (NT == 0 && p.nw) {
#pragma unroll
        for (int m = 0; m < 4; m++) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss[m] += __shfl_xor_sync(0xffffffffu, ss[m], o);
            if (lane == 0) squares[warp * 4 + m] = ss[m];
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    const int active = min(W, units), outs = mine >> pairs;
    for (int idx = threadIdx.x; idx < outs * COLS * 16; idx += blockDim.x) {
        const int r = idx & 15, m = (idx >> 4) & (COLS - 1), o = idx / (COLS * 16);
        const int row = ((pairs ? tile0 >> 1 : tile0) + o) * 16 + r;
        if (m >= p.M || row >= p.N) continue;
        float f = 1.f;
        if (NT == 0 && p.nw) {
            float q = 0.f;
            for (int w = 0; w < active; w++) q += squares[w * 4 + m];
            f = 1.0f / sqrtf(q / (float)p.K + p.eps);
        }
        const float* src = part + (size_t)(o << pairs) * W * (COLS * 16) + m * 16 + r;
        float v = warp_sums<COLS>(src, active);
        v = finite_or_plain<F>(v * f, p, 0, row, m);
        float* out = p.y + (size_t)m * p.N + row;
        if (pairs) {
            const float v2 = finite_or_plain<F>(warp_sums<COLS>(src + W * (COLS * 16), active) * f, p, 1, row, m);
            *out = (v / (1.0f + expf(-v))) * v2;
        } else if (p.epi == EPI_ACCUM) *out += v;
        else *out = v;
    }
}

// ---- 9 to 32 rows of x --------------------------------------------------------------------------------------------------------
// A warp has NT products of eight columns of x and a share of K. CG = 1: all columns of x, sixteen warps up to 16 rows of x, eight with twice
// the registers beyond, so that weights are unpacked once for 32 rows and the chains of a block's products are four. CG = 2: sixteen
// warps, two of them for a share, each with its half of 32 columns; for short rows (few_units). Longer ones of 17 to 32 rows take 29.2 us
// so where eight warps take 27.6 (Q4_0 11008x4096; Q4_K 4096x11008 45.4 and 37.5, Q6_K 32000x4096 135 and 101).
template <int F, int NT, int CG, int T, bool QUIRK, bool DEEP>
__global__ void __launch_bounds__(kShares<NT * CG> * CG * 32, 1) gemv_split_wide_kernel(const SplitArgs p) {
    static_assert(!DEEP || CG == 1, "the place of a warp's sums in tensor memory is that of its share");
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int ROW = Lay<F>::ROW, TB = kTileBytes<F>, OWN = 8 * NT, COLS = OWN * CG, W = kShares<NT * CG>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, share = warp / CG, cg = warp % CG, g = lane >> 2, t = lane & 3;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int stages = p.stages;
    Shared rings = smem + share * (stages * T * TB);
    const uint32_t ring = smem_u32(rings);
    const int units = (p.K + 255) / 256, pairs = p.epi == EPI_SWIGLU, tile0 = blockIdx.x * T;
    const int my_units = share < units ? (units - share + W - 1) / W : 0;
    Pieces<F> pc;
    pc.init(p.K / 32, lane);
    int iss = 0;
    auto issue = [&](int buf) {
        if (iss < my_units) {
#pragma unroll
            for (int i = 0; i < T; i++) {
                if (CG > 1 && i % CG != cg) continue;           // (the warps of a share bring every CG-th tile)
                const int tile = min(tile0 + i, p.tiles - 1);
                issue_tile<F>(p, pc, pairs ? tile & 1 : 0, (pairs ? tile >> 1 : tile) * 16, share + iss * W, ring + (buf * T + i) * TB, lane);
            }
            iss++;
        }
        cp_async_commit();
    };
    auto meet = [&]() {                                         // the warps of a share
        if (CG == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(share + 1), "n"(32 * CG) : "memory");
    };
    if (kNF4Like<F>) {                                          // (as above)
        if (kTable<F>) fill_lut(smem + p.lut);
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    issue(0);
    if (stages > 1) issue(1);
    Shared lut = smem + (kTable<F> ? p.lut + (lane & 15) * 8 : 0);
    uint32_t* const tmem = reinterpret_cast<uint32_t*>(smem + p.extra);
    if (DEEP) {
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");

    float acc[T][NT][4];
#pragma unroll
    for (int i = 0; i < T; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int k = 0; k < 4; k++) acc[i][j][k] = 0.f;
    uint4 nh[NT], nl[NT];                                       // B operands of the next block
    auto fetch = [&](int blk) {
        const uint4* src = p.planes + ((size_t)blk * CG + cg) * (NT * 64) + lane;
#pragma unroll
        for (int j = 0; j < NT; j++) { nh[j] = __ldcg(src + j * 64); nl[j] = __ldcg(src + j * 64 + 32); }
    };
    if (my_units) fetch(share * 8);
    // exponent fields of what undoes the scaling of the warp's columns, unit after unit
    uint8_t* const fields = smem + p.extra + 16 + warp * (OWN * ((units + W - 1) / W));
    constexpr int WORDS = OWN / 4;
    for (int i = lane; i < WORDS * my_units; i += 32) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(p.xf + (size_t)(share + i / WORDS * W) * COLS + OWN * cg + 4 * (i % WORDS)));
        *reinterpret_cast<uint32_t*>(fields + 4 * i) = (__float_as_uint(v.x) >> 23) | (__float_as_uint(v.y) >> 23 << 8) | (__float_as_uint(v.z) >> 23 << 16) |
                                                       (__float_as_uint(v.w) >> 23 << 24);
    }
    __syncwarp();
    auto undoes = [&](int u, int j) { return lds16(fields + OWN * u + 8 * j + 2 * t); };      // the thread's two columns of product j
    // a thread's place in tensor memory: its warp's 32 lanes, as many columns for each of the warps of a quadrant
    const uint32_t totals = DEEP ? *tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * (uint32_t)(1024 / W) : 0u;
    int buf = 0;
    for (int u = 0; u < my_units; u++) {
        const int un = share + u * W;
        if (!DEEP && u) {                                       // the sums follow to the unit's scaling, exactly: by 2^40 at most (x_split_kernel)
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const uint32_t now = undoes(u, j), before = undoes(u - 1, j);
                if (now == before) continue;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const float ratio = power(127u + ((before >> (8 * k)) & 255u) - ((now >> (8 * k)) & 255u));
#pragma unroll
                    for (int i = 0; i < T; i++) { acc[i][j][k] *= ratio; acc[i][j][k + 2] *= ratio; }
                }
            }
        }
        if (stages > 1) cp_async_wait<1>();
        else cp_async_wait<0>();
        meet();
        Shared base = rings + buf * T * TB + g * ROW;
#pragma unroll 1
        for (int b = 0; b < 8; b++) {
            uint4 bh[NT], bl[NT];
#pragma unroll
            for (int j = 0; j < NT; j++) { bh[j] = nh[j]; bl[j] = nl[j]; }
            if (b < 7) fetch(un * 8 + b + 1);
            else if (u + 1 < my_units) fetch((un + W) * 8);
            float2 s32[NT];
            if (kMins<F>) {
#pragma unroll
                for (int j = 0; j < NT; j++) s32[j] = __ldcg(reinterpret_cast<const float2*>(p.sums + (size_t)(un * 8 + b) * COLS + OWN * cg + 8 * j + 2 * t));
            }
#pragma unroll
            for (int i = 0; i < T; i++) {
                Shared lo = base + i * TB, hi = lo + 8 * ROW;
                const int tile = min(tile0 + i, p.tiles - 1), row0 = (pairs ? tile >> 1 : tile) * 16;
                Head hl, hh;
                head_of<F>(p, lo, row0 + g, un, hl);
                head_of<F>(p, hi, row0 + g + 8, un, hh);
                uint32_t a[kDigits<F>][2][4];
                block_regs<F>(lo, hi, b, t, hl.off, hh.off, lut, a);
                constexpr int C1 = F == CMLB200_Q6_K ? 1 : 0;
                float c[C1 + 1][NT][4];
#pragma unroll
                for (int k = 0; k <= C1; k++)
#pragma unroll
                    for (int j = 0; j < NT; j++)
#pragma unroll
                        for (int v = 0; v < 4; v++) c[k][j][v] = 0.f;
#pragma unroll
                for (int d = kDigits<F> - 1; d >= 0; d--) {     // (as above)
#pragma unroll
                    for (int k = 0; k < 2; k++)
#pragma unroll
                        for (int j = 0; j < NT; j++) mma_f16(c[k * C1][j], a[d][k], k ? bl[j].z : bl[j].x, k ? bl[j].w : bl[j].y);
#pragma unroll
                    for (int k = 0; k < 2; k++)
#pragma unroll
                        for (int j = 0; j < NT; j++) mma_f16(c[k * C1][j], a[d][k], k ? bh[j].z : bh[j].x, k ? bh[j].w : bh[j].y);
                }
#pragma unroll
                for (int k = 0; k <= C1; k++) {
                    const float sl = scale_of<F, QUIRK>(p, lo, hl, b, k), sh = scale_of<F, QUIRK>(p, hi, hh, b, k);
                    float ml = 0.f, mh = 0.f;
                    if (kMins<F> && k == 0) { ml = offset_of<F>(lo, hl, b, sl); mh = offset_of<F>(hi, hh, b, sh); }
#pragma unroll
                    for (int j = 0; j < NT; j++) {
                        acc[i][j][0] = fmaf(c[k][j][0], sl, acc[i][j][0]);
                        acc[i][j][1] = fmaf(c[k][j][1], sl, acc[i][j][1]);
                        acc[i][j][2] = fmaf(c[k][j][2], sh, acc[i][j][2]);
                        acc[i][j][3] = fmaf(c[k][j][3], sh, acc[i][j][3]);
                        if (kMins<F> && k == 0) {
                            acc[i][j][0] = fmaf(s32[j].x, ml, acc[i][j][0]);
                            acc[i][j][1] = fmaf(s32[j].y, ml, acc[i][j][1]);
                            acc[i][j][2] = fmaf(s32[j].x, mh, acc[i][j][2]);
                            acc[i][j][3] = fmaf(s32[j].y, mh, acc[i][j][3]);
                        }
                    }
                }
            }
        }
        meet();                                                 // every lane is done with this buffer
        issue(buf);
        if (++buf == stages) buf = 0;
        if (DEEP) {
#pragma unroll
            for (int i = 0; i < T; i++) {
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    const uint32_t undo = undoes(u, j);
#pragma unroll
                    for (int k = 0; k < 4; k++) acc[i][j][k] *= power(undo >> (8 * (k & 1)));
                }
#pragma unroll
                for (int j = 0; j < NT; j += 2) {
                    const uint32_t at = totals + (uint32_t)(4 * NT * i + 4 * j);
                    if (u) tmem_add8(at, acc[i][j], acc[i][j + 1]);
                    if (u + 1 < my_units) tmem_put8(at, acc[i][j], acc[i][j + 1]);
                }
                if (u + 1 < my_units) {
#pragma unroll
                    for (int j = 0; j < NT; j++)
#pragma unroll
                        for (int k = 0; k < 4; k++) acc[i][j][k] = 0.f;
                }
            }
            if (u + 1 < my_units) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
    }
    if (!DEEP && my_units) {
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const uint32_t undo = undoes(my_units - 1, j);
#pragma unroll
            for (int i = 0; i < T; i++)
#pragma unroll
                for (int k = 0; k < 4; k++) acc[i][j][k] *= power(undo >> (8 * (k & 1)));
        }
    }
    if (DEEP) asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cp_async_wait<0>();
    const uint32_t held = DEEP ? *tmem : 0u;
    __syncthreads();                                            // the rings become the place where the warps' sums meet
    if (DEEP && warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(held) : "memory");
    }
    float* part = reinterpret_cast<float*>(smem);               // [T][W][COLS][16]
#pragma unroll
    for (int i = 0; i < T; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) {
            float* dst = part + ((size_t)i * W + share) * (COLS * 16) + (OWN * cg + 8 * j + 2 * t) * 16 + g;
            dst[0] = acc[i][j][0];
            dst[16] = acc[i][j][1];
            dst[8] = acc[i][j][2];
            dst[24] = acc[i][j][3];
        }
    __syncthreads();
    const int active = min(W, units), mine = min(T, p.tiles - tile0), outs = mine >> pairs;
    for (int idx = threadIdx.x; idx < outs * COLS * 16; idx += blockDim.x) {
        const int r = idx & 15, m = (idx >> 4) % COLS, o = idx / (COLS * 16);
        const int row = ((pairs ? tile0 >> 1 : tile0) + o) * 16 + r;
        if (m >= p.M || row >= p.N) continue;
        const float* src = part + (size_t)(o << pairs) * W * (COLS * 16) + m * 16 + r;
        const float v = finite_or_plain<F>(warp_sums<COLS>(src, active), p, 0, row, m);
        float* out = p.y + (size_t)m * p.N + row;
        if (pairs) {
            const float v2 = finite_or_plain<F>(warp_sums<COLS>(src + W * (COLS * 16), active), p, 1, row, m);
            *out = (v / (1.0f + expf(-v))) * v2;
        } else if (p.epi == EPI_ACCUM) *out += v;
        else *out = v;
    }
}

// ---- host side ----------------------------------------------------------------------------------------------------------------------
template <typename Kern>
int launch_split(Kern kern, int grid, int warps, size_t smem, cudaStream_t st, const SplitArgs& p) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CMLB_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
    return CMLB200_OK;
}

template <int F> constexpr size_t kSmemMost = 227 * 1024 - (kTable<F> ? kLutBytes + 16 : 0);      // besides the table
template <int NT> size_t wide_extra(const SplitArgs& p) { return 16 + (size_t)kShares<NT> * 8 * NT * (((p.K + 255) / 256 + kShares<NT> - 1) / kShares<NT>); }

constexpr int kMostTiles = 6;                                            // row tiles of a CTA

// Shared memory of gemv_split_kernel besides NF4's table
template <int F, int NT> constexpr size_t narrow_smem(int ring, int W, int M, int per) {
    return (size_t)W * ring * kTileBytes<F> + (NT == 0 ? (size_t)W * (M * kXBytes + kOwnBytes) : 0) + ((size_t)per * W * (NT == 0 ? 4 : 8) * 16 + W * 4) * sizeof(float);
}

// Warps and row tiles of a CTA: as many tiles as fill the SMs once, or several times where that would be more than six (5 tiles of
// 11008 rows: 8.2 us at M = 1; 3: 11.4, 2: 13.3, for every CTA makes the operands of x again)
struct Narrow { int W, per, rounds; };
inline Narrow narrow_plan(const SplitArgs& p) {
    const int units = (p.K + 255) / 256, sms = cmlb_num_sms();
    const int want = (p.tiles + sms - 1) / sms, rounds = (want + kMostTiles - 1) / kMostTiles;
    const int per = (p.tiles + sms * rounds - 1) / (sms * rounds);
    return {units < kWarps ? units : kWarps, p.epi == EPI_SWIGLU ? (per + 1) & ~1 : per, rounds};
}

template <int F, int NT, bool QUIRK, int RING>
int launch_narrow(SplitArgs& p, int W, cudaStream_t st) {
    size_t smem = narrow_smem<F, NT>(RING, W, p.M, p.per_cta);
    if (kTable<F>) {
        p.lut = (int)((smem + 15) / 16 * 16);
        smem = p.lut + kLutBytes;
    }
    auto kern = gemv_split_kernel<F, NT, QUIRK, RING>;
    static size_t done[kMaxDevices] = {};
    CMLB_CUDA(cmlb_ensure_smem(kern, smem, done));
    return launch_split(kern, (p.tiles + p.per_cta - 1) / p.per_cta, W, smem, st, p);
}

template <int F, int NT, bool QUIRK>
int run_narrow(SplitArgs& p, cudaStream_t st) {
    const Narrow n = narrow_plan(p);
    const int W = n.W, per = p.per_cta = n.per;
    // sixteen warps, four rows, six tiles: where that is too much (NF4, blocks of 64 and more), such calls have rings of two
    // (13824x5120, 4 rows: 25.5 us; without the table, whose place a third item took, 32.4)
    constexpr int ring = kRing<F, NT>;
    constexpr bool fits = narrow_smem<F, NT>(ring, kWarps, 4, kMostTiles) <= kSmemMost<F>;
    static_assert(kMostTiles % 2 == 0 && (fits || narrow_smem<F, NT>(2, kWarps, 4, kMostTiles) <= kSmemMost<F>), "the largest calls do not fit shared memory");
    if constexpr (!fits)
        if (narrow_smem<F, NT>(ring, W, p.M, per) > kSmemMost<F>) return launch_narrow<F, NT, QUIRK, 2>(p, W, st);
    return launch_narrow<F, NT, QUIRK, ring>(p, W, st);
}

template <int F, int NT, int CG, int T, bool QUIRK, bool DEEP>
int run_wide(SplitArgs& p, cudaStream_t st) {
    constexpr size_t stage = (size_t)kShares<NT * CG> * T * kTileBytes<F>, sums = (size_t)T * 32 * 8 * 16 * 4;
    const size_t extra = wide_extra<NT * CG>(p);
    p.stages = (p.K + 255) / 256 > kShares<NT * CG> && 2 * stage + extra <= kSmemMost<F> ? 2 : 1;
    p.extra = (int)(p.stages * stage > sums ? p.stages * stage : sums);
    p.lut = (int)((p.extra + extra + 15) / 16 * 16);
    const size_t smem = kTable<F> ? (size_t)p.lut + kLutBytes : p.extra + extra;
    auto kern = gemv_split_wide_kernel<F, NT, CG, T, QUIRK, DEEP>;
    static size_t done[kMaxDevices] = {};
    CMLB_CUDA(cmlb_ensure_smem(kern, smem, done));
    return launch_split(kern, (p.tiles + T - 1) / T, kShares<NT * CG> * CG, smem, st, p);
}

// Row tiles of a CTA: waves of CTAs, a CTA as long as its tiles and one and a half more
template <int F, int N8> constexpr int kMostWide = kSmemMost<F> / (kShares<N8> * kTileBytes<F>);
template <int F, int N8> int wide_tiles(const SplitArgs& p, double* cost_out) {
    const int sms = cmlb_num_sms(), choice[4] = {1, 2, 3, 5};
    int best = 1;
    double least = 1e30;
    for (int i = 0; i < 4; i++) {
        const int T = choice[i];
        if (T > kMostWide<F, N8> || (p.epi == EPI_SWIGLU && T != 2)) continue;
        if (T > 1 && (size_t)kShares<N8> * T * kTileBytes<F> + wide_extra<N8>(p) > kSmemMost<F>) continue;
        const int ctas = (p.tiles + T - 1) / T;
        const double cost = (double)((ctas + sms - 1) / sms) * (T + 1.5);
        if (cost < least) { least = cost; best = T; }
    }
    *cost_out = least;
    return best;
}

template <int F, int NT, int CG, bool QUIRK, bool DEEP>
int run_wide_t(SplitArgs& p, cudaStream_t st) {
    constexpr int most = kMostWide<F, NT * CG>;
    double cost;
    const int best = wide_tiles<F, NT * CG>(p, &cost);
    if constexpr (most >= 5) if (best == 5) return run_wide<F, NT, CG, 5, QUIRK, DEEP>(p, st);
    if constexpr (most >= 3) if (best == 3) return run_wide<F, NT, CG, 3, QUIRK, DEEP>(p, st);
    if (best == 2) return run_wide<F, NT, CG, 2, QUIRK, DEEP>(p, st);
    return run_wide<F, NT, CG, 1, QUIRK, DEEP>(p, st);
}

// Rows of few units: 17 rows of x and more have sixteen warps with half the columns each: of eight, only as many as there are units would work,
// and the launch is as long as one of those. us, 32 rows, eight warps and sixteen: Q8_0 10000x256 11.5 9.5, Q4_0 17616x1280 27.3 24.7, NF4
// 20000x512 35.0 26.2, 20000x1536 47.8 41.1; three and four units are even, seven and more are for the eight. Q4_K, Q5_K and Q6_K, whose unpacking
// costs most, are for eight from three units on where a CTA has several row tiles (Q6_K 10000x1024 14.1 17.3; Q4_K 2048x768 8.1 7.4).
template <int F> bool few_units(const SplitArgs& p) {
    const int units = (p.K + 255) / 256;
    const bool heavy = F == CMLB200_Q4_K || F == CMLB200_Q5_K || F == CMLB200_Q6_K;
    return units <= 2 || (units <= 6 && (!heavy || p.tiles <= cmlb_num_sms()));
}

template <int F, int NT, bool QUIRK>
int run_wide_d(SplitArgs& p, cudaStream_t st) {
    if constexpr (kNF4Like<F> || F == CMLB200_Q6_K || F == CMLB200_Q8_0)
        if (p.deep) return run_wide_t<F, NT, 1, QUIRK, true>(p, st);
    if constexpr (NT == 4)
        if (few_units<F>(p)) return run_wide_t<F, 2, 2, QUIRK, false>(p, st);
    return run_wide_t<F, NT, 1, QUIRK, false>(p, st);
}

template <int F, bool QUIRK>
int run_split(SplitArgs& p, int nt, cudaStream_t st) {
    switch (nt) {
        case 0: return run_narrow<F, 0, QUIRK>(p, st);
        case 1: return run_narrow<F, 1, QUIRK>(p, st);
        case 2: return run_wide_d<F, 2, QUIRK>(p, st);
        default: return run_wide_d<F, 4, QUIRK>(p, st);
    }
}

}  // namespace
