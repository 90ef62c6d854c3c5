// rys_warp.cu -- host dispatch of the Rys Fock kernel
// (rys_warp.cuh; its instantiations: rys_warp_inst.cu).
#include "rys_warp.h"

#include "fock_kernels.cuh"

namespace fjb {

bool compiled_available(int la, int lb, int lc, int ld, bool fp32);  // fock_compiled.cu

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
// round trip.  The register kernel's bodies spill where the boundary (bra e x
// ket f values) grows: measured on a 20-atom cluster of the 64-atom workload's
// shells (ms, register / warp kernel, FP64): (sp|sf) 1.46 / 2.85, (sp|pp) 1.77
// / 2.66, (sp|pd) 1.79 / 3.97, (sd|sd) 0.82 / 1.14, (sd|pp) 1.34 / 2.35, (pp|pp)
// 0.62 / 1.43, but (sd|sf) 3.94 / 1.55, (sd|pd) 5.02 / 2.61, (sp|pf) 4.14 / 2.61,
// (sp|dd) 1.54 / 1.13, (pp|pd) 4.28 / 2.58, (sf|pp) 3.02 / 2.75; in FP32 the
// same classes but (sf|pp), whose row in registers is the shorter side, 1.56 / 2.21.
bool rys_warp_preferred(int la, int lb, int lc, int ld, bool fp32) {
    const auto rows = [](int x, int y) {  // Cartesians of levels x .. x + y
        int n = 0;
        for (int l = x; l <= x + y; ++l) n += (l + 1) * (l + 2) / 2;
        return n;
    };
    const int e = rows(la, lb), f = rows(lc, ld);
    return e * f > 100 && !(fp32 && f < e && compiled_available(la, lb, lc, ld, true));
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
