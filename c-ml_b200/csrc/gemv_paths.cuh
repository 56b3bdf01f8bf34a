// The decode kernels behind cmlb200_gemv and its siblings, one set of entries per source file. W2: the second weight of a SwiGLU
// call, NULL otherwise; a kernel takes a pair only where it takes both of them. epi: EPI_STORE, EPI_ACCUM or EPI_SWIGLU.
#pragma once
#include "common.cuh"

// gemv_dp4a.cu: integer dot products for Q4_0 / Q8_0 at small M, and the choice of the kernel for RMS-normalised rows
int cmlb200_gemv_dp4a_(const cmlb200_qmat* W, const cmlb200_qmat* W2, const float* x, const uint16_t* norm_w, float eps,
                       const uint32_t* xq, float* y, int M, int epi, cudaStream_t st);
size_t cmlb200_xq_bytes_(int M, int K);
int cmlb200_x_digits_(const float* x, int M, int K, uint32_t* xq, cudaStream_t st);

// gemv_mma.cu: the tensor-core decode kernel (mma.sync int8) for up to 4 rows of x per launch
bool cmlb200_gemv_mma_ok_(const cmlb200_qmat* W, const cmlb200_qmat* W2, int epi);
int cmlb200_gemv_mma_rows_(const cmlb200_qmat* W, const cmlb200_qmat* W2, int epi);      // rows of x of a launch; 0: not this weight
int cmlb200_gemv_mma_(const cmlb200_qmat* W, const cmlb200_qmat* W2, const float* x, const uint16_t* norm_w, float eps,
                      const uint32_t* xq, float* y, int M, int epi, cudaStream_t st);

// gemv_mma8.cu: its sibling for 5 to 8 rows of x in one launch (Q4_0, fp32 x)
bool cmlb200_gemv_mma8_ok_(const cmlb200_qmat* W, const cmlb200_qmat* W2, int epi);
int cmlb200_gemv_mma8_(const cmlb200_qmat* W, const cmlb200_qmat* W2, const float* x, const uint16_t* norm_w, float eps, float* y, int M,
                       int epi, cudaStream_t st);

// gemv_split.cu: fp16 tensor cores with x in two fp16 parts, every block format, up to 32 rows of x per launch
bool cmlb200_gemv_split_ok_(const cmlb200_qmat* W, const cmlb200_qmat* W2);
int cmlb200_gemv_split_(const cmlb200_qmat* W, const cmlb200_qmat* W2, const float* x, const uint16_t* norm_w, float eps, float* y, int M, int epi,
                        cudaStream_t st);

// gemv.cu: whether they are the faster ones for so many rows of x
bool cmlb200_gemv_split_faster_(const cmlb200_qmat* W, const cmlb200_qmat* W2, int M, int epi);

// gemv_kquant.cu: Q4_1 / Q4_K / Q5_K / Q6_K weights straight from the GGUF block stream
bool cmlb200_is_kquant_type_(int type);
int cmlb200_gemv_kquant_(const cmlb200_qmat* W, const float* x, float* y, int M, int accumulate, cudaStream_t st);

// gemv_tc.cu: tcgen05 integer tensor-core path over the tile-major copy of the weight
int cmlb200_gemv_tc_(const cmlb200_qmat* W, const float* x, float* y, int M, int accumulate, cudaStream_t st);
