// NF4 weights through gemv_split.cuh
#include "gemv_split.cuh"

int cmlb200_split_nf4_bare_(void* args, int nt, cudaStream_t st);

namespace {

// Where a table of codes costs more than it saves: what it saves is 5 to 20 % of a CTA's work, what it costs is the 0.3 to 0.6 us until it
// is filled and 32 KB. us of 4 to 32 rows, with the table and without:
//   up to 8 rows   where fewer CTAs fit an SM than have work (14336x2048 M = 6 21.3 18.9, SwiGLU 28672x1024 M = 7 41.3 34.6), and at
//                  5 to 8 rows where a CTA has few items (4096x768 M = 6 8.0 7.1, 2048x512 5.7 5.3)
//   9 and more     up to two units of 256 columns from 17 rows on (20000x512 M = 32 26.2 25.0), pairs of up to four, whose CTAs have two row
//                  tiles each (SwiGLU 28672x1024 M = 13 80.5 71.2), and blocks of 32 that five row tiles a CTA, for which there is no room beside
//                  the table, take fewer waves of CTAs (10000x3072 M = 16 29.8 24.2)
template <int TABLE, int BARE>
bool bare_faster(const SplitArgs& p, int nt) {
    const int units = (p.K + 255) / 256;
    if (nt < 2) {
        const Narrow n = narrow_plan(p);
        if (nt && n.per * n.W <= (n.W < 5 ? 12 : 8)) return true;
        if (n.rounds == 1) return false;
        const size_t sm = 228 * 1024, own = (nt ? narrow_smem<TABLE, 1>(kRing<TABLE, 1>, n.W, p.M, n.per) : narrow_smem<TABLE, 0>(kRing<TABLE, 0>, n.W, p.M, n.per)) + 1024;
        const int fit = kWarps / n.W, work = fit < n.rounds ? fit : n.rounds;           // (128 registers a thread)
        return own + kLutBytes <= sm && (int)(sm / (own + kLutBytes)) < work && sm / (own + kLutBytes) < sm / own;
    }
    if (p.epi == EPI_SWIGLU ? units <= 4 : nt == 4 && units <= 2) return true;
    if (TABLE != kNF4Fine || nt != 2) return false;
    double with, without;
    wide_tiles<TABLE, 2>(p, &with);
    wide_tiles<BARE, 2>(p, &without);
    return without < 0.93 * with;
}

}  // namespace

int cmlb200_split_nf4_(void* args, int nt, cudaStream_t st) {
    SplitArgs& p = *static_cast<SplitArgs*>(args);
    if (p.nf4_shift ? bare_faster<CMLB200_NF4, kNF4Bare>(p, nt) : bare_faster<kNF4Fine, kNF4FineBare>(p, nt)) return cmlb200_split_nf4_bare_(args, nt, st);
    return p.nf4_shift ? run_split<CMLB200_NF4, false>(p, nt, st) : run_split<kNF4Fine, false>(p, nt, st);
}
