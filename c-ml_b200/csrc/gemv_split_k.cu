// Q4_1, Q4_K, Q5_K and Q6_K weights, straight from the GGUF block stream, through gemv_split.cuh
#include "gemv_split.cuh"

int cmlb200_split_k_(int type, void* args, int nt, cudaStream_t st) {
    SplitArgs& p = *static_cast<SplitArgs*>(args);
    switch (type) {
        case CMLB200_Q4_1: return run_split<CMLB200_Q4_1, false>(p, nt, st);
        case CMLB200_Q4_K: return run_split<CMLB200_Q4_K, false>(p, nt, st);
        case CMLB200_Q5_K: return run_split<CMLB200_Q5_K, false>(p, nt, st);
        default: return run_split<CMLB200_Q6_K, false>(p, nt, st);
    }
}
