// rys_warp.h -- which classes the Rys Fock kernel (rys_warp.cuh) is built
// for, and its host interface (rys_warp.cu).
#pragma once
#include <cuda_runtime.h>

// By bra, one compilation unit each (rys_warp_inst.cu, FJB_RW_PART): every
// class but those of an ss bra and (sp|sp), (sp|sd), which the register kernel
// takes.
#define FJB_RW_SP(X) X(0, 1, 0, 3) X(0, 1, 1, 1) X(0, 1, 1, 2) X(0, 1, 1, 3) X(0, 1, 2, 2) X(0, 1, 2, 3) X(0, 1, 3, 3)
#define FJB_RW_SD(X) \
    X(0, 2, 0, 2) X(0, 2, 0, 3) X(0, 2, 1, 1) X(0, 2, 1, 2) X(0, 2, 1, 3) X(0, 2, 2, 2) X(0, 2, 2, 3) X(0, 2, 3, 3)
#define FJB_RW_SF(X) X(0, 3, 0, 3) X(0, 3, 1, 1) X(0, 3, 1, 2) X(0, 3, 1, 3) X(0, 3, 2, 2) X(0, 3, 2, 3) X(0, 3, 3, 3)
#define FJB_RW_PP(X) X(1, 1, 1, 1) X(1, 1, 1, 2) X(1, 1, 1, 3) X(1, 1, 2, 2) X(1, 1, 2, 3) X(1, 1, 3, 3)
#define FJB_RW_PD(X) X(1, 2, 1, 2) X(1, 2, 1, 3) X(1, 2, 2, 2) X(1, 2, 2, 3) X(1, 2, 3, 3)
#define FJB_RW_DD(X) X(2, 2, 2, 2) X(2, 2, 2, 3) X(2, 2, 3, 3)
#define FJB_RW_PF(X) X(1, 3, 1, 3) X(1, 3, 2, 2) X(1, 3, 2, 3) X(1, 3, 3, 3)
#define FJB_RW_DF(X) X(2, 3, 2, 3) X(2, 3, 3, 3) X(3, 3, 3, 3)
#define FJB_RW_CLASSES(X) \
    FJB_RW_SP(X) FJB_RW_SD(X) FJB_RW_SF(X) FJB_RW_PP(X) FJB_RW_PD(X) FJB_RW_DD(X) FJB_RW_PF(X) FJB_RW_DF(X)

namespace fjb {

struct KArgs;

bool rys_warp_available(int la, int lb, int lc, int ld);
// Whether it is the faster of the class's kernels (rys_warp.cu).
bool rys_warp_preferred(int la, int lb, int lc, int ld);
int rys_warp_blocks_per_sm(int la, int lb, int lc, int ld, bool fp32);
cudaError_t rys_warp_launch(int la, int lb, int lc, int ld, bool fp32, int grid, cudaStream_t st, const KArgs &a);

}  // namespace fjb
