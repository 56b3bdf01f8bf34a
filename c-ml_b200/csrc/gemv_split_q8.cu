// Q8_0 weights through gemv_split.cuh
#include "gemv_split.cuh"

int cmlb200_split_q8_(void* args, int nt, int quirk, cudaStream_t st) {
    SplitArgs& p = *static_cast<SplitArgs*>(args);
    return quirk ? run_split<CMLB200_Q8_0, true>(p, nt, st) : run_split<CMLB200_Q8_0, false>(p, nt, st);
}
