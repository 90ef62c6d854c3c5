// rys_warp.cu -- host dispatch of the Rys Fock kernel
// (rys_warp.cuh; its instantiations: rys_warp_inst.cu).
#include "rys_warp.h"

#include "fock_kernels.cuh"

namespace fjb {

#define FJB_X(a, b, c, d)                                                         \
    int rys_warp_occ64_##a##b##c##d();                                            \
    int rys_warp_occ32_##a##b##c##d();                                            \
    cudaError_t rys_warp_run64_##a##b##c##d(int, cudaStream_t, const KArgs &);    \
    cudaError_t rys_warp_run32_##a##b##c##d(int, cudaStream_t, const KArgs &);
FJB_RW_CLASSES(FJB_X)
#undef FJB_X

bool rys_warp_available(int la, int lb, int lc, int ld) {
#define FJB_X(a, b, c, d) \
    if (la == a && lb == b && lc == c && ld == d) return true;
    FJB_RW_CLASSES(FJB_X)
#undef FJB_X
    return false;
}

// Against the register kernel: a short program in registers beats the tables'
// round trip; its bodies spill where the boundary (bra e x ket f values of the
// HGP transfer, e and f from the first, smaller shell's l up) grows.  The line
// lies between (sd|sd), 100 values, and (sp|dd), 124.  32-atom cluster of the
// 64-atom workload's shells, classes one after another, ms, register / this
// kernel, FP64: (sp|pd) 5.8 / 13.4, (sp|pp) 5.7 / 10.7, (sp|sf) 4.5 / 9.5,
// (sd|pp) 4.4 / 6.3, (sd|sd) 2.4 / 3.0, (pp|pp) 2.1 / 4.5; then (sp|dd) 3.8 /
// 3.0, (sp|pf) 12.0 / 8.8, (pp|pd) 13.7 / 7.4, (sf|pp) 9.8 / 5.1, (sd|pd) 15.7 /
// 7.3, (sd|sf) 12.1 / 5.5.  In FP32 the two cross a little later -- (sp|dd) 1.9
// / 2.2, (sp|pf) 4.9 / 6.2, (pp|pd) 5.7 / 5.8, (sf|pp) 3.7 / 3.7, (sd|sf) 4.4 /
// 4.4, (sd|pd) 6.5 / 5.7 -- and share the line: 1.6 of 163 ms with every unit
// in FP32.
bool rys_warp_preferred(int la, int lb, int lc, int ld) {
    const auto rows = [](int x, int y) {  // Cartesians of levels x .. x + y
        int n = 0;
        for (int l = x; l <= x + y; ++l) n += (l + 1) * (l + 2) / 2;
        return n;
    };
    return rows(la, lb) * rows(lc, ld) > 100;
}

int rys_warp_blocks_per_sm(int la, int lb, int lc, int ld, bool fp32) {
#define FJB_X(a, b, c, d)                         \
    if (la == a && lb == b && lc == c && ld == d) \
        return fp32 ? rys_warp_occ32_##a##b##c##d() : rys_warp_occ64_##a##b##c##d();
    FJB_RW_CLASSES(FJB_X)
#undef FJB_X
    return 0;
}

cudaError_t rys_warp_launch(int la, int lb, int lc, int ld, bool fp32, int grid, cudaStream_t st, const KArgs &a_) {
#define FJB_X(a, b, c, d)                         \
    if (la == a && lb == b && lc == c && ld == d) \
        return fp32 ? rys_warp_run32_##a##b##c##d(grid, st, a_) : rys_warp_run64_##a##b##c##d(grid, st, a_);
    FJB_RW_CLASSES(FJB_X)
#undef FJB_X
    return cudaErrorInvalidValue;
}

}  // namespace fjb
