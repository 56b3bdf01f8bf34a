// NF4 weights through gemv_split.cuh
#include "gemv_split.cuh"

int cmlb200_split_nf4_(void* args, int nt, cudaStream_t st) {
    SplitArgs& p = *static_cast<SplitArgs*>(args);
    return p.nf4_shift ? run_split<CMLB200_NF4, false>(p, nt, st) : run_split<kNF4Fine, false>(p, nt, st);
}
