// NF4 weights through gemv_split.cuh
#include "gemv_split.cuh"

int cmlb200_split_nf4_(void* args, int nt, cudaStream_t st) { return run_split<CMLB200_NF4, false>(*static_cast<SplitArgs*>(args), nt, st); }
