// rys_device.cuh -- what the Rys kernels share: the Cartesian index sets and
// transfer coefficients as compile-time tables, a class's shape, and the
// tabulated rule on the device (the Fock kernel rys_warp.cuh, the J-engine's
// jrys.cu, the three-centre integrals df_eri3.cu).
#pragma once
#include <cuda_runtime.h>

#include "fjb_internal.h"
#include "fock_kernels.cuh"
#include "rys_rule.h"

namespace fjb {

namespace rys {

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int nrange(int lo, int hi) {
    int n = 0;
    for (int l = lo; l <= hi; ++l) n += ncart(l);
    return n;
}
__host__ __device__ constexpr int binom(int n, int k) {
    int r = 1;
    for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
    return r;
}

// The Cartesians of levels LO..HI in cartesians(l) order (x descending, then
// y descending), level by level: the boundary's index order.
// idx[i][j][k] is the position of Cartesian (i, j, k) (-1 outside the set).
template <int LO, int HI>
struct CSet {
    static constexpr int N = nrange(LO, HI);
    int x[N], y[N], z[N];
    int idx[HI + 1][HI + 1][HI + 1];
    __host__ __device__ constexpr CSet() : x(), y(), z(), idx() {
        for (int i = 0; i <= HI; ++i)
            for (int j = 0; j <= HI; ++j)
                for (int k = 0; k <= HI; ++k) idx[i][j][k] = -1;
        int n = 0;
        for (int l = LO; l <= HI; ++l)
            for (int i = l; i >= 0; --i)
                for (int j = l - i; j >= 0; --j) {
                    x[n] = i;
                    y[n] = j;
                    z[n] = l - i - j;
                    idx[i][j][l - i - j] = n;
                    ++n;
                }
    }
};

// HRR coefficients of one side (the second shell's l = LY): for b in
// cartesians(LY) and k <= b componentwise, C(b,k) SEP^(b-k); entry
// off[b] + (k_x (b_y+1) + k_y)(b_z+1) + k_z.
template <int LY>
struct HCoefs {
    static constexpr int NB = ncart(LY);
    int off[NB + 1];
    __host__ __device__ constexpr HCoefs() : off() {
        constexpr CSet<LY, LY> c{};
        off[0] = 0;
        for (int b = 0; b < NB; ++b) off[b + 1] = off[b] + (c.x[b] + 1) * (c.y[b] + 1) * (c.z[b] + 1);
    }
    static constexpr int total() {
        constexpr CSet<LY, LY> c{};
        int n = 0;
        for (int b = 0; b < NB; ++b) n += (c.x[b] + 1) * (c.y[b] + 1) * (c.z[b] + 1);
        return n;
    }
};

// The tables as device constants: every access below has a compile-time
// index once the loops are unrolled, so each folds to an immediate.
template <int LO, int HI>
__device__ constexpr CSet<LO, HI> kCart{};
template <int LY>
__device__ constexpr HCoefs<LY> kHCo{};

template <int LA, int LB, int LC, int LD>
struct Shape {
    static constexpr int E = LA + LB, F = LC + LD;
    static constexpr int NR = (E + F) / 2 + 1;  // Rys roots
    static constexpr int TS = (E + 1) * (F + 1);  // one axis' 2D table
    // the tables as stored: per axis F+1 rows (ket index k), each the E+1
    // values of the bra index padded to whole 16-byte vectors (rp); rows
    // rps apart, an odd number of 16-byte vectors, so that the rows of
    // up to eight different k fall in different banks
    template <typename R>
    __host__ __device__ static constexpr int rp() {
        return ((E + 1) * (int)sizeof(R) + 15) / 16 * 16 / (int)sizeof(R);
    }
    template <typename R>
    __host__ __device__ static constexpr int rps() {
        return ((((E + 1) * (int)sizeof(R) + 15) / 16) | 1) * 16 / (int)sizeof(R);
    }
    template <typename R>
    __host__ __device__ static constexpr int tsp() {
        return (F + 1) * rps<R>();
    }
    // one ket's tables for a chunk of P primitive quartets, padded to an odd
    // number of 16-byte vectors so that different kets' rows do not share
    // banks
    template <typename R>
    __host__ __device__ static constexpr int kstride(int P) {
        return P * NR * 3 * tsp<R>() + (((P * NR * 3 * tsp<R>() * (int)sizeof(R) / 16) & 1) ? 0 : 16 / (int)sizeof(R));
    }
    static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    static constexpr int NAB = NA * NB, NCD = NC * ND;
    static constexpr int NBE = nrange(LA, E), NBF = nrange(LC, F);
    static constexpr int NCB = HCoefs<LB>::total();
};

// Dynamic shared memory of one CTA (doubles) when `minb` CTAs share an SM:
// its share of the SM's 228 KiB less the 1 KiB the hardware reserves per CTA
// and the kernel's static arrays (below 3 KiB).
__host__ __device__ constexpr int rys_smem_budget(int minb) {
    return minb <= 1 ? kSmemBudgetDoubles : (233472 / minb - 1024 - 3072) / 8;
}

// One root of the n-point rule at T (rys_rule, one root's two series) from
// the device table: a power's coefficients of x and of w are one vector load.
template <int N, int DEG, typename R, typename R2>
__device__ __forceinline__ void rule_series(int r, double T, const R *__restrict__ tab, R *x, R *w) {
    if (T < kRysTSwitch) {
        int i = (int)T;
        if (i > kRysNI - 1) i = kRysNI - 1;
        const R u = (R)(2.0 * (T - (double)i) - 1.0);  // kRysWidth = 1
        const R2 *blk = reinterpret_cast<const R2 *>(tab + rys_device_at(DEG, N, i, 0, r));
        R2 c[DEG + 1];
#pragma unroll
        for (int k = 0; k <= DEG; ++k) c[k] = __ldg(blk + k * N);
        R px = c[DEG].x, pw = c[DEG].y;
#pragma unroll
        for (int k = DEG - 1; k >= 0; --k) {
            px = px * u + c[k].x;
            pw = pw * u + c[k].y;
        }
        *x = px;
        *w = pw;
    } else {
        const R *a = tab + rys_device_asym(DEG, N);
        *x = (R)((double)__ldg(a + 2 * r) / T);
        *w = (R)((double)__ldg(a + 2 * r + 1) * (0.5 / sqrt(T)));
    }
}
template <int N>
__device__ __forceinline__ void rule_root(int r, double T, const double *__restrict__ tab, double *x, double *w) {
    rule_series<N, kRysDegD, double, double2>(r, T, tab, x, w);
}
// The same root in FP32 from the FP32 table (the routed path's FP32 tier):
// the interval and its local coordinate from T in FP64, the series in FP32
// (relative error about 1e-7, inside the tier's own).
template <int N>
__device__ __forceinline__ void rule_root_f(int r, double T, const float *__restrict__ tab, float *x, float *w) {
    rule_series<N, kRysDegF, float, float2>(r, T, tab, x, w);
}

// The HRR coefficient `idx` of side LY for separation sep (= A - B or C - D).
template <int LY, typename R>
__device__ __forceinline__ R hrr_coef(int idx, const double *sep) {
    constexpr const HCoefs<LY> &H = kHCo<LY>;
    constexpr const CSet<LY, LY> &c = kCart<LY, LY>;
    int b = 0;
#pragma unroll
    for (int j = 1; j < HCoefs<LY>::NB; ++j)
        if (idx >= H.off[j]) b = j;
    int bx = 0, by = 0, bz = 0;
#pragma unroll
    for (int j = 0; j < HCoefs<LY>::NB; ++j)
        if (j == b) {
            bx = c.x[j];
            by = c.y[j];
            bz = c.z[j];
        }
    const int rem = idx - H.off[b];
    const int kz = rem % (bz + 1), ky = (rem / (bz + 1)) % (by + 1), kx = rem / ((bz + 1) * (by + 1));
    const double v = (double)(binom(bx, kx) * binom(by, ky) * binom(bz, kz)) * ipow(sep[0], bx - kx) *
                     ipow(sep[1], by - ky) * ipow(sep[2], bz - kz);
    return (R)v;
}


// N values of R from a 16-byte aligned shared-memory row, as 16-byte loads.
template <typename R, int N>
__device__ __forceinline__ void ld_row(const R *p, R *out) {
    static_assert(N * sizeof(R) % 16 == 0, "whole 16-byte vectors");
#pragma unroll
    for (int v = 0; v < N * (int)sizeof(R) / 16; ++v) {
        const float4 t = reinterpret_cast<const float4 *>(p)[v];
        memcpy(out + v * (16 / (int)sizeof(R)), &t, 16);
    }
}

// The position of Cartesian index t of cartesians-range LO..HI as (x, y, z),
// for a run-time index (the thread's own f).
template <int LO, int HI>
__device__ __forceinline__ void cart_of(int t, int *x, int *y, int *z) {
    int l = LO;
#pragma unroll
    for (int m = LO; m < HI; ++m)
        if (t >= ncart(m)) {
            t -= ncart(m);
            l = m + 1;
        } else {
            break;
        }
    int i = l;
    while (t > l - i) {
        t -= l - i + 1;
        --i;
    }
    *x = i;
    *y = l - i - t;
    *z = t;
}

}  // namespace rys

}  // namespace fjb
