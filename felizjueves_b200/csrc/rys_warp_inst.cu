// rys_warp_inst.cu -- the Rys Fock kernel's instantiations, built
// once per bra class and precision (FJB_RW_PART a class list of rys_warp.h,
// FJB_RW_FP32 0 or 1) so that they compile in parallel.
#include "rys_warp.cuh"
#include "rys_warp.h"

namespace fjb {

#if FJB_RW_FP32
#define FJB_X(a, b, c, d)                                                                    \
    int rys_warp_occ32_##a##b##c##d() { return RysWarpOne<b, a, d, c, float>::occupancy(); } \
    cudaError_t rys_warp_run32_##a##b##c##d(int grid, cudaStream_t st, const KArgs &k) {     \
        return RysWarpOne<b, a, d, c, float>::launch(grid, st, k);                           \
    }
#else
#define FJB_X(a, b, c, d)                                                                     \
    int rys_warp_occ64_##a##b##c##d() { return RysWarpOne<b, a, d, c, double>::occupancy(); } \
    cudaError_t rys_warp_run64_##a##b##c##d(int grid, cudaStream_t st, const KArgs &k) {      \
        return RysWarpOne<b, a, d, c, double>::launch(grid, st, k);                           \
    }
#endif
FJB_RW_PART(FJB_X)
#undef FJB_X

}  // namespace fjb
