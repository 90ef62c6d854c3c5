// hermite_r.cuh -- the Hermite Coulomb integrals R_{tuv} in registers: the
// McMurchie-Davidson recursion with every index a compile-time constant
// (the J-engine's small classes, the nuclear attraction).
#pragma once
#include <utility>

#include "jrys.h"

namespace fjb {

// hermite_order index -> (t, u, v), constexpr, for the unrolled kernels.
__host__ __device__ constexpr int hc_total(int idx) {
    int n = 0;
    while (nh(n) <= idx) ++n;
    return n;
}
__host__ __device__ constexpr int hc_t(int idx) {
    const int n = hc_total(idx);
    int r = idx - (n == 0 ? 0 : nh(n - 1)), t = n;
    while (r >= n - t + 1) {
        r -= n - t + 1;
        --t;
    }
    return t;
}
__host__ __device__ constexpr int hc_u(int idx) {
    const int n = hc_total(idx);
    int r = idx - (n == 0 ? 0 : nh(n - 1)), t = n;
    while (r >= n - t + 1) {
        r -= n - t + 1;
        --t;
    }
    return n - t - r;
}
__host__ __device__ constexpr int hc_v(int idx) { return hc_total(idx) - hc_t(idx) - hc_u(idx); }
// Compile-time walks of the small classes: every index below is a template
// constant (fold expressions over integer sequences), so R, the signed D_q
// and the J_p partials stay in registers.
// One entry I of the R recursion: [r]^(m) = PQ_d [r-1_d]^(m+1) + (r_d - 1)
// [r-2_d]^(m+1), d the first nonzero axis.
template <int I, typename T>
__device__ __forceinline__ void r_entry(T *R, T X, T Y, T Z) {
    constexpr int t = hc_t(I), u = hc_u(I), v = hc_v(I);
    if constexpr (t > 0) {
        T x = X * R[hc_idx(t - 1, u, v)];
        if constexpr (t >= 2) x += (T)(t - 1) * R[hc_idx(t - 2, u, v)];
        R[I] = x;
    } else if constexpr (u > 0) {
        T x = Y * R[hc_idx(0, u - 1, v)];
        if constexpr (u >= 2) x += (T)(u - 1) * R[hc_idx(0, u - 2, v)];
        R[I] = x;
    } else {
        T x = Z * R[hc_idx(0, 0, v - 1)];
        if constexpr (v >= 2) x += (T)(v - 1) * R[hc_idx(0, 0, v - 2)];
        R[I] = x;
    }
}
template <int I0, typename T, int... K>
__device__ __forceinline__ void r_entries(T *R, T X, T Y, T Z, std::integer_sequence<int, K...>) {
    (r_entry<I0 + K, T>(R, X, Y, Z), ...);
}
// Totals S, S-1, .. 1 of one level (descending: each reads the level above
// at totals S-1 and S-2 before they are rewritten).
template <int S, typename T>
struct RTotals {
    static __device__ __forceinline__ void run(T *R, T X, T Y, T Z) {
        if constexpr (S >= 1) {
            r_entries<nh(S - 1), T>(R, X, Y, Z, std::make_integer_sequence<int, nh(S) - nh(S - 1)>{});
            RTotals<S - 1, T>::run(R, X, Y, Z);
        }
    }
};
// Levels M, M-1, .. 0 of R_{tuv} at total order L.
template <int L, int M, typename T>
struct RLevels {
    static __device__ __forceinline__ void run(T *R, const T *f, T X, T Y, T Z) {
        if constexpr (M >= 0) {
            RTotals<L - M, T>::run(R, X, Y, Z);
            R[0] = f[M];
            RLevels<L, M - 1, T>::run(R, f, X, Y, Z);
        }
    }
};
}  // namespace fjb
