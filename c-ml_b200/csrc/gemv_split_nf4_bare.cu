// NF4 weights through gemv_split.cuh, codes by byte permutes
#include "gemv_split.cuh"

int cmlb200_split_nf4_bare_(void* args, int nt, cudaStream_t st) {
    SplitArgs& p = *static_cast<SplitArgs*>(args);
    return p.nf4_shift ? run_split<kNF4Bare, false>(p, nt, st) : run_split<kNF4FineBare, false>(p, nt, st);
}
