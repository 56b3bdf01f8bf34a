// Choice of the kernels of gemv_split.cuh and the rows of x as their B operands.
#include "gemv_split.cuh"
#include "call_scratch.cuh"
#include "gemv_paths.cuh"

int cmlb200_split_q4_(void* args, int nt, int quirk, cudaStream_t st);
int cmlb200_split_q8_(void* args, int nt, int quirk, cudaStream_t st);
int cmlb200_split_nf4_(void* args, int nt, cudaStream_t st);
int cmlb200_split_k_(int type, void* args, int nt, cudaStream_t st);

namespace {

// Rows of x as B operands in global memory. One CTA per row of x (rows from M on: zeros); RMSNorm (src/nn/llama.c:71-124) first
// when a weight is given. CONTIG: a thread of the product takes 8 neighbouring columns (NF4). follow: scalings of a row lie no further
// apart than 2^40, so that sums may follow them from unit to unit.
constexpr int kKept = 3;
template <bool CONTIG>
__global__ void __launch_bounds__(512)
x_split_kernel(const float* __restrict__ x, const __half* __restrict__ nw, float eps, int K, int M, int NT, bool follow,
               uint4* __restrict__ planes, float* __restrict__ sums, float* __restrict__ xf) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float red[2][16];
    const int row = blockIdx.x, j = row >> 3, g = row & 7, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int units = (K + 255) / 256, items = units * 32;          // (block, t)
    const float* xr = x + (size_t)row * K;
    auto load = [&](int i, float (&e)[8]) {
        const int at = (i >> 2) * 32;
#pragma unroll
        for (int k = 0; k < 8; k++) e[k] = 0.f;
        if (row >= M || at >= K) return;
        const int c0 = at + (CONTIG ? 8 : 4) * (i & 3), c1 = CONTIG ? c0 + 4 : c0 + 16;
        const float4 u = *reinterpret_cast<const float4*>(xr + c0), v = *reinterpret_cast<const float4*>(xr + c1);
        e[0] = u.x; e[1] = u.y; e[2] = u.z; e[3] = u.w; e[4] = v.x; e[5] = v.y; e[6] = v.z; e[7] = v.w;
    };
    auto weigh = [&](int i, float (&e)[8]) {
        const int at = (i >> 2) * 32;
        if (row >= M || at >= K) return;
        const int c0 = at + (CONTIG ? 8 : 4) * (i & 3), c1 = CONTIG ? c0 + 4 : c0 + 16;
        const uint2 u = *reinterpret_cast<const uint2*>(nw + c0), v = *reinterpret_cast<const uint2*>(nw + c1);
        const uint32_t w[4] = {u.x, u.y, v.x, v.y};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
            e[2 * k] *= f.x;
            e[2 * k + 1] *= f.y;
        }
    };
    float inv = 1.f, least = 0.f, kept[kKept][8];                   // a thread's first items stay in registers
#pragma unroll
    for (int n = 0; n < kKept; n++) load(tid + 512 * n, kept[n]);
    if (nw || follow) {
        float ss = 0.f, most = 0.f;
        auto look = [&](int i, float (&e)[8]) {
            if (nw) {
#pragma unroll
                for (int k = 0; k < 8; k++) ss = fmaf(e[k], e[k], ss);
                weigh(i, e);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) most = fmaxf(most, fabsf(e[k]));
        };
#pragma unroll
        for (int n = 0; n < kKept; n++) look(tid + 512 * n, kept[n]);
        for (int i = tid + 512 * kKept; i < items; i += 512) {
            float e[8];
            load(i, e);
            look(i, e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        }
        if (lane == 0) { red[0][warp] = most; red[1][warp] = ss; }
        __syncthreads();
        most = 0.f, ss = 0.f;
#pragma unroll
        for (int w = 0; w < 16; w++) { most = fmaxf(most, red[0][w]); ss += red[1][w]; }
        if (nw) inv = 1.0f / sqrtf(ss / (float)K + eps);
        if (follow) least = most * inv * 0x1p-40f;
    }
    auto put = [&](int i, float (&e)[8]) {                          // 32 items are a unit, a warp's
        float s = 0.f, most = least, up, down;
        if (nw) {
#pragma unroll
            for (int k = 0; k < 8; k++) e[k] *= inv;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) most = fmaxf(most, fabsf(e[k]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
        scaling(most, up, down);
        if (lane == 0) xf[(size_t)(i >> 5) * (8 * NT) + row] = down;
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int k = 0; k < 8; k++) { e[k] *= up; s += e[k]; }
        split8<CONTIG>(e, hi, lo);
        const int blk = i >> 2, t = i & 3;
        uint4* dst = planes + ((size_t)(blk * NT + j) * 2) * 32 + g * 4 + t;
        dst[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        dst[32] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (t == 0) sums[(size_t)blk * (8 * NT) + row] = s;
    };
#pragma unroll
    for (int n = 0; n < kKept; n++)
        if (tid + 512 * n < items) put(tid + 512 * n, kept[n]);
    for (int i = tid + 512 * kKept; i < items; i += 512) {
        float e[8];
        load(i, e);
        if (nw) weigh(i, e);
        put(i, e);
    }
}

constexpr int kMaxUnits = 512;                               // K < 131072

// One chain through all of a share's blocks rounds at the size of the result each time. For the formats whose former kernels summed
// in shorter chains (1.25 to 1.35e-7 of the result off) chains of more than 16 blocks are cut: a unit's sums to those of the units before
// it, which lie in tensor memory meanwhile, for there are no registers for both. Scalings need not follow one another there.
// K = 11008, 32 rows: NF4 1.57e-7 in one chain, 1.31e-7 so, Q6_K 1.85 and 1.24e-7. It costs 0.5 to 1 us a launch.
bool split_deep(int type, int units, int W) {
    return (type == CMLB200_Q6_K || type == CMLB200_NF4 || type == CMLB200_Q8_0) && units > 2 * W;
}

}  // namespace

// Weights the kernels take: whole 16-byte rows of quants and whole 256-column units of scales, or (NF4) blocks of 32, 64, 128
// or a multiple of 256 columns
bool cmlb200_gemv_split_ok_(const cmlb200_qmat* W, const cmlb200_qmat* W2) {
    if (W2 && !cmlb200_gemv_split_ok_(W2, nullptr)) return false;
    if (W->cols / 256 >= kMaxUnits || ((uintptr_t)W->qs & 15)) return false;
    switch (W->type) {
        case CMLB200_Q4_0:
        case CMLB200_Q8_0: return W->cols % 256 == 0 && !((uintptr_t)W->scales & 15);
        case CMLB200_NF4: return W->cols % 32 == 0 && !((uintptr_t)W->scales & 3) && (W->block == 32 || W->block == 64 || W->block == 128 || W->block % 256 == 0);
        case CMLB200_Q4_1:
        case CMLB200_Q4_K:
        case CMLB200_Q5_K:
        case CMLB200_Q6_K: return W->cols % 256 == 0;
        default: return false;
    }
}

// y[M, rows] (= | += | swiglu) for M <= 32 from fp32 x, RMS-normalised with norm_w first when it is given
int cmlb200_gemv_split_(const cmlb200_qmat* W, const cmlb200_qmat* W2, const float* x, const uint16_t* norm_w, float eps, float* y, int M, int epi,
                        cudaStream_t st) {
    SplitArgs p = {};
    p.qs = (const uint8_t*)W->qs;
    p.sc = (const uint8_t*)W->scales;
    if (W2) { p.qs2 = (const uint8_t*)W2->qs; p.sc2 = (const uint8_t*)W2->scales; }
    p.x = x;
    p.nw = reinterpret_cast<const __half*>(norm_w);
    p.eps = eps;
    p.y = y;
    p.N = W->rows;
    p.K = W->cols;
    p.M = M;
    p.epi = epi;
    p.tiles = (W->rows + 15) / 16 * (epi == EPI_SWIGLU ? 2 : 1);
    p.nf4_shift = W->type != CMLB200_NF4 ? 0 : W->block >= 256 ? 3 : W->block == 128 ? 2 : W->block == 64 ? 1 : 0;
    p.nf4_units = W->type == CMLB200_NF4 && W->block > 256 ? W->block / 256 : 1;
    const int nt = M <= 4 ? 0 : M <= 8 ? 1 : M <= 16 ? 2 : 4;
    CallScratch scratch;                                     // the split rows, the sums of their blocks, their scaling
    if (nt) {
        const size_t blocks = (size_t)((p.K + 255) / 256) * 8, plane_bytes = blocks * nt * 64 * sizeof(uint4), sum_bytes = blocks * 8 * nt * sizeof(float);
        uint8_t* base = nullptr;
        int rc = scratch.get(st, plane_bytes + sum_bytes + sum_bytes / 8, (void**)&base);
        if (rc) return rc;
        uint4* planes = reinterpret_cast<uint4*>(base);
        float* sums = reinterpret_cast<float*>(base + plane_bytes);
        float* xf = reinterpret_cast<float*>(base + plane_bytes + sum_bytes);
        p.planes = planes;
        p.sums = sums;
        p.xf = xf;
        const int shares = nt == 4 ? kWarps / 2 : kWarps, units = (p.K + 255) / 256;
        p.deep = nt > 1 && split_deep(W->type, units, shares);
        const bool follow = nt > 1 && units > shares && !p.deep;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(8 * nt);
        cfg.blockDim = dim3(512);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        CMLB_CUDA(cudaLaunchKernelEx(&cfg, W->type == CMLB200_NF4 ? x_split_kernel<true> : x_split_kernel<false>, x, p.nw, eps, p.K, M, nt, follow, planes, sums, xf));
    }
    const int quirk = (W->flags & CMLB200_QMAT_SUBNORMAL_SCALES) || (W2 && (W2->flags & CMLB200_QMAT_SUBNORMAL_SCALES));
    switch (W->type) {
        case CMLB200_Q4_0: return cmlb200_split_q4_(&p, nt, quirk, st);
        case CMLB200_Q8_0: return cmlb200_split_q8_(&p, nt, quirk, st);
        case CMLB200_NF4: return cmlb200_split_nf4_(&p, nt, st);
        default: return cmlb200_split_k_(W->type, &p, nt, st);
    }
}

// Projections of RMS-normalised rows in one or two launches, for the LLaMA's decode steps beyond what cmlb200_gemv_rmsnorm takes:
// any block format the kernels take, up to 32 rows; epi 2 (SwiGLU) up to 8, where a CTA's row tiles come in pairs at no cost.
extern "C" int cmlb200_gemv_norm_ok_(const cmlb200_qmat* W, const cmlb200_qmat* W2, int M) {
    if (M < 1 || M > (W2 ? 8 : 32) || W->rows <= 0 || W->cols <= 0 || !cmlb200_gemv_split_ok_(W, W2)) return 0;
    return !W2 || (W2->type == W->type && W2->rows == W->rows && W2->cols == W->cols && W2->block == W->block);
}
extern "C" int cmlb200_gemv_norm_(const cmlb200_qmat* W, const cmlb200_qmat* W2, const float* d_x, const uint16_t* d_norm_w, float eps, float* d_y, int M,
                                  void* stream) {
    return cmlb200_gemv_split_(W, W2, d_x, d_norm_w, eps, d_y, M, W2 ? EPI_SWIGLU : EPI_STORE, as_stream(stream));
}
