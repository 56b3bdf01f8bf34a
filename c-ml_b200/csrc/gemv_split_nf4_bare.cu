// NF4 weights through gemv_split.cuh, codes by byte permutes: the calls that the rule of gemv_split_nf4.cu sends here
#include "gemv_split.cuh"

namespace {

template <int F> int run_bare(SplitArgs& p, int nt, cudaStream_t st) {
    switch (nt) {
        case 0: return run_narrow<F, 0, false>(p, st);
        case 1: return run_narrow<F, 1, false>(p, st);
        case 2:
            if constexpr (F == kNF4FineBare) return run_wide_d<F, 2, false>(p, st);
            else return run_wide<F, 2, 1, 2, false, false>(p, st);          // (pairs)
        default: return run_wide_t<F, 2, 2, false, false>(p, st);           // (rows of few units)
    }
}

}  // namespace

int cmlb200_split_nf4_bare_(void* args, int nt, cudaStream_t st) {
    SplitArgs& p = *static_cast<SplitArgs*>(args);
    return p.nf4_shift ? run_bare<kNF4Bare>(p, nt, st) : run_bare<kNF4FineBare>(p, nt, st);
}
