// jrys.h -- the J-engine's records, and its Rys kernel for the record classes
// of high total order (jrys.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "fjb_internal.h"

namespace fjb {

constexpr int kJMaxL = 2 * kMaxL;  // L of one record
constexpr int kNHMax = (kJMaxL + 1) * (kJMaxL + 2) * (kJMaxL + 3) / 6;  // 84

__host__ __device__ constexpr int nh(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }

struct JRec {
    double P[3], PA[3], PB[3];
    double zeta, pre, G;  // pre = c_a c_b (pi/zeta)^{3/2} exp(-alpha beta/zeta |AB|^2)
    int32_t la, lb, ao_a, ao_b;
    int32_t L, pair, dq_off, pad;
};
static_assert(sizeof(JRec) == 128, "JRec is 128 bytes");

// hermite_order's position of (t, u, v): totals ascending, t then u descending
__host__ __device__ constexpr int hc_idx(int t, int u, int v) {
    const int n = t + u + v;
    return (n == 0 ? 0 : nh(n - 1)) + (n - t) * (n - t + 1) / 2 + (n - t - u);
}

// One (bra L, ket L) class of records: the bra records [bra0, bra0 + nbra),
// the kets [ket0, ket0 + nket) in key order (kst, skey, and their D_q in Dq
// at kdq, consecutive).
struct JRysArgs {
    const JRec *recs;
    int bra0, nbra, ket0, nket;
    const double4 *kst;
    const int *kdq;
    const double *skey, *Dq;
    double *Jp;
    double tau, thr32;
    const double *rys_tab;
};

// The classes it is built for: total order above kJSmallL.
constexpr int kJSmallL = 6;
cudaError_t j_rys_launch(int lp, int lq, cudaStream_t st, const JRysArgs &a);

}  // namespace fjb
