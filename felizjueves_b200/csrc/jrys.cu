// jrys.cu -- the J-engine's Rys kernel (record classes of total order 7..12).
//
// J_p += sum_ket sum_q (-1)^|q| R_{p+q} D_q with R written as its n-point
// quadrature, exact at order L = lp + lq for n = L/2 + 1:
//
//   R_{tuv} = sum_r w_r X_t(r) Y_u(r) Z_v(r),  X_0 = 1,
//   X_{t+1} = -2 rho x_r (d_x X_t + t X_{t-1}),   d = P - Q,
//
// (x_r, w_r) the Rys rule at T = rho |d|^2 and (2/sqrt(pi)) sqrt(rho) folded
// into Z: the Boys values of the McMurchie-Davidson recursion replaced by
// their rule.  With d taken as Q - P the sign is (-1)^|p|, applied once to
// the sum.  The contraction is then one axis at a time -- over q_z, q_y, q_x
// -- and needs (lp+1) + (lp+1)(lp+2)/2 intermediates beside the J_p partials,
// where R itself is 120 to 455 values: no table, all indices compile-time.
//
// A CTA per bra record; its warps take the kets GK = 32 / n at a time in key
// order, a lane per (ket, root): the roots of a ket share its scalars' loads
// and the rule's lines (rys_device_at), and a lane's work is one uniform
// stream of FMAs into its own J_p partials, summed over lanes and warps once
// at the end.  The kets' D_q are consecutive in memory; the warp stages them
// through shared memory with coalesced loads.  FP64-pipe and shared-memory
// bound: lp, lq = 3, 4 is 390 FMAs a root for 35 shared loads.  The classes of
// lp = 6 keep 84 J_p partials a lane and spill (32 bytes stored at (6, 1), 400
// at (6, 3), 2,116 at (6, 6)), (5, 5) and (5, 6) a little; the other 13 do not.
#include "jrys.h"

#include "rys_device.cuh"

namespace fjb {

namespace {

constexpr int kJRysWarps = 4;

template <int LP, int LQ, typename R>
__device__ __forceinline__ void j_rys_lane(double T, double rho, double dx, double dy, double dz, int r,
                                           const double *tab, const double *dq, R *jp) {
    constexpr int L = LP + LQ, NR = L / 2 + 1;
    constexpr double kTwoOverSqrtPi = 1.1283791670955126;
    double x, w;
    rys::rule_root<NR>(r, T, tab, &x, &w);
    const double a64 = -2.0 * rho * x;
    const R a = (R)a64, ax = (R)(a64 * dx), ay = (R)(a64 * dy), az = (R)(a64 * dz);
    R X[L + 1], Y[L + 1], Z[L + 1];
    X[0] = (R)1;
    Y[0] = (R)1;
    Z[0] = (R)(kTwoOverSqrtPi * sqrt(rho) * w);
#pragma unroll
    for (int t = 0; t < L; ++t) {
        const R ta = (R)t * a;
        X[t + 1] = t ? ax * X[t] + ta * X[t - 1] : ax * X[t];
        Y[t + 1] = t ? ay * Y[t] + ta * Y[t - 1] : ay * Y[t];
        Z[t + 1] = t ? az * Z[t] + ta * Z[t - 1] : az * Z[t];
    }
#pragma unroll
    for (int qx = 0; qx <= LQ; ++qx) {
        R B[LP + 1][LP + 1];
#pragma unroll
        for (int qy = 0; qx + qy <= LQ; ++qy) {
            R A[LP + 1];
#pragma unroll
            for (int qz = 0; qx + qy + qz <= LQ; ++qz) {
                const R d = (R)dq[hc_idx(qx, qy, qz)];
#pragma unroll
                for (int pz = 0; pz <= LP; ++pz) A[pz] = qz ? A[pz] + Z[pz + qz] * d : Z[pz + qz] * d;
            }
#pragma unroll
            for (int py = 0; py <= LP; ++py)
#pragma unroll
                for (int pz = 0; py + pz <= LP; ++pz)
                    B[py][pz] = qy ? B[py][pz] + Y[py + qy] * A[pz] : Y[py + qy] * A[pz];
        }
#pragma unroll
        for (int px = 0; px <= LP; ++px)
#pragma unroll
            for (int py = 0; px + py <= LP; ++py)
#pragma unroll
                for (int pz = 0; px + py + pz <= LP; ++pz) jp[hc_idx(px, py, pz)] += X[px + qx] * B[py][pz];
    }
}

// thr32 > 0: the kets of a chunk of 32 whose first (largest) bound is below it
// run in FP32, as in j_pq_small_kernel: the products X, Y, Z, D_q and the
// contraction; T, the rule (which holds the Boys values here) and its factors
// and the J_p sums stay FP64.  A step that straddles two chunks may run both.
template <int LP, int LQ>
__global__ void __launch_bounds__(32 * kJRysWarps) j_rys_kernel(const JRysArgs A) {
    constexpr int L = LP + LQ, NR = L / 2 + 1, NP = nh(LP), NQ = nh(LQ), GK = 32 / NR;
    __shared__ double s_dq[kJRysWarps][GK * NQ];
    __shared__ double s_part[kJRysWarps][NP];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int g = lane / NR, r = lane - g * NR;
    double *dq = s_dq[wl];
    for (int bi = blockIdx.x; bi < A.nbra; bi += gridDim.x) {
        const JRec &B = A.recs[A.bra0 + bi];
        const double G = B.G, p = B.zeta, Px = B.P[0], Py = B.P[1], Pz = B.P[2];
        double jp[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) jp[i] = 0.0;
#pragma unroll 1
        for (int k0 = wl * GK; k0 < A.nket; k0 += kJRysWarps * GK) {
            const double first = G * A.skey[A.ket0 + k0];
            if (first < A.tau) break;  // the keys descend
            const int nk = min(GK, A.nket - k0);
            {
                const double *src = A.Dq + A.kdq[A.ket0 + k0];
                for (int i = lane; i < nk * NQ; i += 32) dq[i] = src[i];
            }
            __syncwarp();
            const int k = A.ket0 + k0 + g;
            if (g < nk && !(G * A.skey[k] < A.tau)) {
                const double4 Q = A.kst[k];
                const double q = Q.w, rho = p * q / (p + q);
                const double dx = Q.x - Px, dy = Q.y - Py, dz = Q.z - Pz;
                const double T = rho * (dx * dx + dy * dy + dz * dz);
                if (A.thr32 > 0.0 && G * A.skey[A.ket0 + ((k0 + g) & ~31)] < A.thr32) {
                    float j32[NP];
#pragma unroll
                    for (int i = 0; i < NP; ++i) j32[i] = 0.f;
                    j_rys_lane<LP, LQ, float>(T, rho, dx, dy, dz, r, A.rys_tab, dq + g * NQ, j32);
#pragma unroll
                    for (int i = 0; i < NP; ++i) jp[i] += (double)j32[i];
                } else {
                    j_rys_lane<LP, LQ, double>(T, rho, dx, dy, dz, r, A.rys_tab, dq + g * NQ, jp);
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            double v = jp[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) s_part[wl][i] = v;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < NP; i += 32 * kJRysWarps) {
            double v = s_part[0][i];
#pragma unroll
            for (int w = 1; w < kJRysWarps; ++w) v += s_part[w][i];
            int n = 0;  // |p| of the i-th Hermite index
            while (nh(n) <= i) ++n;
            A.Jp[B.dq_off + i] += (n & 1) ? -v : v;
        }
        __syncthreads();
    }
}

template <int LP, int LQ>
cudaError_t launch_one(cudaStream_t st, const JRysArgs &a) {
    j_rys_kernel<LP, LQ><<<a.nbra, 32 * kJRysWarps, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t j_rys_launch(int lp, int lq, cudaStream_t st, const JRysArgs &a) {
#define FJB_X(p, q) \
    if (lp == p && lq == q) return launch_one<p, q>(st, a);
    FJB_X(1, 6) FJB_X(2, 5) FJB_X(2, 6) FJB_X(3, 4) FJB_X(3, 5) FJB_X(3, 6) FJB_X(4, 3) FJB_X(4, 4) FJB_X(4, 5)
    FJB_X(4, 6) FJB_X(5, 2) FJB_X(5, 3) FJB_X(5, 4) FJB_X(5, 5) FJB_X(5, 6) FJB_X(6, 1) FJB_X(6, 2) FJB_X(6, 3)
    FJB_X(6, 4) FJB_X(6, 5) FJB_X(6, 6)
#undef FJB_X
    return cudaErrorInvalidValue;
}

}  // namespace fjb
