// rys_warp.cuh -- the Rys Fock kernel.
//
// rys_warp_kernel<LA, LB, LC, LD, R>: a team of threads per work item (a work
// unit -- a bra shell pair and up to 32 of its kets -- or, when the queue is
// short for the grid, a slice of one), the item's computed kets taken GW at a
// time.  The team is one WARP where the bra's row of Cartesians fits a warp
// (to dd: 31): then there is no CTA barrier anywhere, the phases are ordered
// by __syncwarp and the other warps of the SM fill the latencies.  The longer
// bras take a CTA (Shape::tw).
//
// The larger shell of each pair comes first (LA >= LB, LC >= LD; the plan's
// records hold the smaller one first, SB and SK turn them): the boundary then
// spans la <= |e| <= la + lb from the larger l, which is shorter -- 6 e for a
// ds bra where (sd| has 10, 10 for fs instead of 20, 25 for fp instead of 34 --
// and the transfers run over the smaller shell's Cartesians.  32-atom build
// 237 -> 207 ms: (sf|pd) 10.0 -> 6.5, (sf|pp) 8.7 -> 5.1, (pd|pf) 10.1 -> 7.5,
// though the ps and fs rows lose a little to their shorter rounds ((sp|pf) 7.9
// -> 8.7, (sd|sf) 4.7 -> 5.5).  Per group of kets:
//
//   A  tables: a lane per (ket, primitive quartet x root): the Rys rule at T
//      (rys_rule.h) and the three axes' 2D integrals I(i, k), the root's
//      weight and the seed folded into z, into the team's shared memory; CH
//      (quartet, root) entries of each ket a round.
//   B  boundary: a lane per (ket, e), e a bra Cartesian of la <= |e| <= la +
//      lb, holds the whole ket row [e0|f0] for every f with lc <= |f| <= lc +
//      ld in registers: per table entry 3 (lc+ld+1) loads feed the (lc+ld+1)
//      (lc+ld+2)/2 products I_x I_y and one FMA per f.
//   C  ket HRR from those registers (the binomial transfer), the row [e0|cd]
//      to shared memory; the lane's own sum_cd D_cd [e0|cd] stays in one
//      register for the whole item: the bra block J_ab is the bra HRR of
//      that sum, taken once per item.
//   E  digest: a lane per (ket, d) -- and per c modulo CS where lanes are
//      left -- takes the columns [.0|cd], makes their bra HRR in registers
//      and forms J_cd, its shares of K_ad, K_bd (summed over c) and of K_ac,
//      K_bc (summed over d through shared memory); FP64 throughout.
//
// This is the reference's third engine (rys/, eri/fock/kernel_frys.py:194)
// as the VRR of the fused HGP build: the boundary is the same set of values
// the HGP VRR produces, so the HRR and digest are the build's own.  R = double
// is the plain FP64 path; R = float the routed path's FP32 tier (the rule,
// tables, boundary and HRR in FP32; T, the pair scalars, densities and every
// J/K accumulation FP64).
//
// Why this split: with the kets' f in lanes and the bra's e in registers a
// short bra leaves 1.2 FP64 operations per double read from shared memory --
// 15 per 12 for (pp|pf) -- and the phase runs at the shared memory's rate;
// the longer ket side in registers makes it 49 per 15.  A CTA-per-unit kernel
// of that form spent the rest on barriers and on staging one unit at a time:
// 32-atom cluster of the 64-atom workload's shells, ms a class, it / this:
// (pf|df) 16.0 / 5.1, (pf|pf) 13.2 / 4.4, (df|df) 10.2 / 3.1, (df|ff) 9.3 /
// 2.7; 20 atoms: (pd|pf) 8.7 / 2.2, (sd|pf) 8.0 / 1.8, (pp|pf) 8.1 / 2.0,
// (sp|ff) 4.4 / 1.1.
//
// What bounds it: latency and the shared-memory pipe more than FP64.  ncu on
// (sp|pf), (sd|pf) and (pd|df), 14 atoms: FP64 pipe 32, 29 and 24 %, shared/L1
// data pipe 68, 74 and 54 %, issue slots 36, 36 and 26 %; of 6.5, 6.3 and
// 7.5 stall cycles an instruction the long scoreboard has 1.6, 1.1 and 2.6; 12,
// 12 and 10 warps an SM by registers and shared memory.
#pragma once
#include "rys_device.cuh"

namespace fjb {

namespace rysw {

// Below this many items a team, units are cut into slices.  Items of a class
// differ by their kets and degrees, so with few a warp the last ones ran on a
// half-empty chip ((pd|df) at 14 atoms: 3 items a warp, 10 % of 16 % occupancy).
constexpr int kItemsPerWarp = 4;  // a team
constexpr int kGrabs = 64;        // above this many items a team, it takes several at a time
constexpr int kRedSlots = 12;  // FP64 values a lane parks per reduction round

template <int LA, int LB, int LC, int LD, typename R>
struct Shape {
    using S = rys::Shape<LA, LB, LC, LD>;
    static_assert(LA >= LB && LC >= LD, "the larger shell of a pair first");
    // The team of threads that works on an item: a warp where the bra's row
    // fits one, but five kets of an fp bra (25) on a CTA of 128 unless the ket
    // row is the 74 doubles of ff: one ket a warp fills few lanes of a table
    // round ((fp|dd) 4.7 ms / 3.2, FP32 3.9 / 2.5; (fp|fp) 4.4 / 4.4; (fp|ff)
    // 3.1 / 4.3).  fd (46) takes a CTA of 64 in FP64 and of 96, two kets, in
    // FP32 ((fd|fd) 3.1 against 3.6, FP32 2.7 against 2.2); ff (74) one of 96.
    // (32-atom cluster of the 64-atom workload's shells.)
    static constexpr int tw() {
        if (S::NBE == 25) return S::NBF * (int)sizeof(R) > 52 * 8 ? 32 : 128;
        if (S::NBE <= 32) return 32;
        return S::NBE == 46 && sizeof(R) == 8 ? 64 : 96;
    }
    static constexpr int TW = tw();
    static constexpr int kThreads = TW == 32 ? 64 : TW;  // two independent warps, or one team, a CTA
    static constexpr int kTeams = kThreads / TW;
    static constexpr int E = S::E, F = S::F, NR = S::NR;
    static constexpr int NA = S::NA, NB = S::NB, NC = S::NC, ND = S::ND, NAB = S::NAB, NCD = S::NCD;
    static constexpr int NBE = S::NBE, NBF = S::NBF;
    static constexpr int GW = TW / NBE;  // kets a group: a lane per (ket, e)
    static constexpr int TS = (E + 1) * (F + 1);
    static constexpr int STR = (3 * TS) | 1;  // odd: entries start in different banks
    static constexpr int XS = NCD | 1;
    // digest lanes: GX kets x CS residues of c x ND values of d
    static constexpr int cs_of(int gx) {
        const int n = TW / (gx * ND);
        return n < 1 ? 0 : (n > NC ? NC : n);
    }
    static constexpr int cost(int gx) {
        const int cs = cs_of(gx);
        return cs < 1 ? 1 << 20 : ((GW + gx - 1) / gx) * ((NC + cs - 1) / cs);
    }
    static constexpr int pick_gx() {
        int best = 1;
        for (int g = 2; g <= GW; ++g)
            if (cost(g) < cost(best)) best = g;
        return best;
    }
    static constexpr int GX = pick_gx(), CS = cs_of(GX), CPL = (NC + CS - 1) / CS;
    static constexpr int NK = NA + NB;  // K columns a lane owns per c
    static constexpr int BATCH = kRedSlots / NK < 1 ? 1 : (kRedSlots / NK > CPL ? CPL : kRedSlots / NK);
    static constexpr int RED = BATCH * NK * TW;
    // a warp's shared memory, in doubles
    static constexpr int wd(int n) { return (n * (int)sizeof(R) + 7) / 8; }
    static constexpr int XD = wd(GW * NBE * XS);
    // table entries of each ket a round: a lane per entry; the wider teams'
    // tables no larger than the rows they make room for afterwards; in FP32 two
    // entries a lane for the ten kets of a ps bra, whose rounds of three spend
    // their time between phases ((sp|pf) 6.6 ms / 6.2; FP64 8.7 / 9.0)
    static constexpr int ch() {
        const int most = TW / GW, fit = (XD + RED) / wd(GW * STR);
        if (TW == 32) return GW > 8 && sizeof(R) == 4 ? 2 * most : most;
        return fit > most ? most : (fit < 8 ? 8 : fit);
    }
    static constexpr int CH = ch();
    static constexpr int TABD = wd(GW * CH * STR);
    static constexpr int REGION = TABD > XD + RED ? TABD : XD + RED;
    static constexpr int SMD = REGION + NAB + 32 * 4 + 50;  // + D_ab, the kets' degeneracies, separations, indices
    // CTAs an SM: by shared memory, and by the registers of the ket row (16
    // warps leave 128 a thread, 12 leave 168, 8 leave 255).  The FP64 rows of 25
    // to 46 doubles want 12: at 16 the 25 of an fp ket spill through phase A
    // (32-atom build of the 64-atom workload's shells 208.7 ms against 207.3).
    static constexpr int ctas_smem() { return 232448 / (kTeams * SMD * 8 + 1024); }
    static constexpr int warps_regs() {
        const int row = NBF * (int)sizeof(R);
        return row <= 160 ? 16 : (row <= 52 * 8 ? 12 : 8);
    }
    static constexpr int minb() {
        const int r = warps_regs() * 32 / kThreads;
        const int n = ctas_smem() < r ? ctas_smem() : r;
        return n < 1 ? 1 : n;
    }
};

// The powers of a separation that the transfer to a shell of l = LY takes, v(y)
// = sum_{k <= y} C(y, k) SEP^(y-k) x[base + k]: SEP_d^n at [d * (LY + 1) + n].
template <int LY>
__device__ __forceinline__ void sep_powers(const double *sep, double *pw) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        pw[d * (LY + 1)] = 1.0;
#pragma unroll
        for (int n = 1; n <= LY; ++n) pw[d * (LY + 1) + n] = pw[d * (LY + 1) + n - 1] * sep[d];
    }
}

__device__ __forceinline__ void ld_prim(const PrimRec *__restrict__ p, double *o) {
    const double2 *s = reinterpret_cast<const double2 *>(p);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const double2 v = __ldg(s + i);
        o[2 * i] = v.x;
        o[2 * i + 1] = v.y;
    }
}

}  // namespace rysw

template <int LA, int LB, int LC, int LD, typename R>
__global__ void __launch_bounds__((rysw::Shape<LA, LB, LC, LD, R>::kThreads), (rysw::Shape<LA, LB, LC, LD, R>::minb()))
    rys_warp_kernel(const KArgs A) {
    using S = rysw::Shape<LA, LB, LC, LD, R>;
    constexpr int E = S::E, F = S::F, NR = S::NR, GW = S::GW, CH = S::CH, TS = S::TS, STR = S::STR, XS = S::XS;
    constexpr int NA = S::NA, NB = S::NB, NC = S::NC, ND = S::ND, NAB = S::NAB;
    constexpr int TW = S::TW;
    constexpr int NBE = S::NBE, NBF = S::NBF, GX = S::GX, CS = S::CS, CPL = S::CPL, NK = S::NK, BATCH = S::BATCH;
    constexpr const rys::CSet<LA, E> &es = rys::kCart<LA, E>;
    constexpr const rys::CSet<LC, F> &fs = rys::kCart<LC, F>;
    constexpr const rys::CSet<LA, LA> &ca = rys::kCart<LA, LA>;
    constexpr const rys::CSet<LB, LB> &cbs = rys::kCart<LB, LB>;
    constexpr const rys::CSet<LC, LC> &cc = rys::kCart<LC, LC>;
    constexpr const rys::CSet<LD, LD> &cds = rys::kCart<LD, LD>;
    constexpr double kTwoOverSqrtPi = 1.1283791670955126;
    constexpr bool SB = LA > LB, SK = LC > LD;  // the record's shells are the other way round
    constexpr unsigned kAll = 0xffffffffu;

    extern __shared__ __align__(16) double sm[];
    const int lane = threadIdx.x % TW, wl = threadIdx.x / TW;  // place in the team, team in the CTA
    const auto sync = [] {
        if constexpr (TW == 32)
            __syncwarp();
        else
            __syncthreads();
    };
    double *ws = sm + wl * S::SMD;
    R *tab = reinterpret_cast<R *>(ws);
    R *X = reinterpret_cast<R *>(ws);
    double *red = ws + S::XD;
    double *Dab = ws + S::REGION;
    double *s_deg = Dab + NAB;
    double *s_sep = s_deg + 32;  // [3][32]
    int *s_prim = reinterpret_cast<int *>(s_sep + 96);
    int *s_oc = s_prim + 32, *s_od = s_oc + 32, *s_meta = s_od + 32;

    const int n_todo = A.unit_list ? *A.unit_count : A.n_units;
    const int n_teams = gridDim.x * S::kTeams;
    // a queue short for the grid: each unit's groups over several warps
    constexpr int kMaxSlices = (kKetChunk + GW - 1) / GW;
    const int want = rysw::kItemsPerWarp * n_teams;
    int ns = n_todo < want ? (want + n_todo - 1) / max(n_todo, 1) : 1;
    ns = ns > kMaxSlices ? kMaxSlices : ns;
    const int n_items = n_todo * ns;
    const int grab = max(1, n_items / (n_teams * rysw::kGrabs));

    // this lane's bra Cartesian (phases B, C)
    const int gl = lane / NBE, el = lane - gl * NBE;
    int ex = 0, ey = 0, ez = 0;
    rys::cart_of<LA, E>(el, &ex, &ey, &ez);

    // the items, a grab at a time; the next grab's number comes from the
    // counter while this one is worked on
    int left = 0, taken = 0;
    const auto next_item = [&](int64_t it) -> int64_t {
        if (left > 0) return it + 1;
        if (!A.next) return it + (int64_t)n_teams * grab - (grab - 1);
        if constexpr (TW == 32) {
            return (int64_t)(n_teams + __shfl_sync(kAll, taken, 0)) * grab;
        } else {
            if (lane == 0) s_meta[2] = taken;
            sync();
            return (int64_t)(n_teams + s_meta[2]) * grab;  // rewritten only after the next item's barriers
        }
    };
    for (int64_t it = (int64_t)(blockIdx.x * S::kTeams + wl) * grab; it < n_items; it = next_item(it)) {
        if (left == 0) {
            left = grab;
            if (A.next && lane == 0) taken = atomicAdd(A.next, 1);
        }
        --left;
        const int ui = (int)(it / ns), slice = (int)(it - (int64_t)ui * ns);
        const int u = A.unit_list ? A.unit_list[ui] : ui;
        const Unit U = A.units[u];
        const LaunchRec LR = A.launches[U.launch];
        const PairRec bra = A.pairs[LR.bra_pair0 + U.ib];
        const MolCtx M = mol_of(A, U.launch);
        const int n_ao = M.n_ao;
        const int kab = bra.nprim;
        const int oa = SB ? bra.ao_b : bra.ao_a, ob = SB ? bra.ao_a : bra.ao_b;
        const double sab[3] = {SB ? -bra.AB[0] : bra.AB[0], SB ? -bra.AB[1] : bra.AB[1], SB ? -bra.AB[2] : bra.AB[2]};
        int n_list = 0, kcd = 0;
        if (lane < 32) {
            const int ik = U.k0 + lane;
            bool on = false;
            PairRec ket{};
            if (ik < U.k1) {
                ket = A.pairs[LR.ket_pair0 + ik];
                on = !skip6(M.Dsh, M.n_sh, bra.a, bra.b, ket.a, ket.b, bra.G, ket.G, A.tau);
            }
            const unsigned m = __ballot_sync(kAll, on);
            n_list = __popc(m);
            kcd = __shfl_sync(kAll, ket.nprim, 0);  // one degree per ket batch
            if (A.computed && lane == 0 && slice == 0 && n_list)
                atomicAdd(A.computed + U.launch, (unsigned long long)n_list);
            if (on) {
                const int at = __popc(m & ((1u << lane) - 1u));
                s_prim[at] = ket.prim0;
                s_oc[at] = SK ? ket.ao_b : ket.ao_a;
                s_od[at] = SK ? ket.ao_a : ket.ao_b;
                s_deg[at] = (bra.a == bra.b ? 0.5 : 1.0) * (ket.a == ket.b ? 0.5 : 1.0) *
                            ((LR.diag && ik == U.ib) ? 0.5 : 1.0);
#pragma unroll
                for (int d = 0; d < 3; ++d) s_sep[d * 32 + at] = SK ? -ket.AB[d] : ket.AB[d];
            }
            if (TW > 32 && lane == 0) {
                s_meta[0] = n_list;
                s_meta[1] = kcd;
            }
        }
        for (int i = lane; i < NAB; i += TW) Dab[i] = __ldg(M.D + (size_t)(oa + i / NB) * n_ao + ob + i % NB);
        sync();
        if constexpr (TW > 32) {
            n_list = s_meta[0];
            kcd = s_meta[1];
        }
        if (slice * GW >= n_list) {
            sync();  // the lists are read before the next item's
            continue;
        }
        const int KNR = kab * kcd * NR;
        double jsum = 0.0;  // sum over this lane's kets of 2 deg sum_cd D_cd [e0|cd]

        for (int g0 = slice * GW; g0 < n_list; g0 += GW * ns) {
            const int ng = min(GW, n_list - g0);
            R acc[NBF];
#pragma unroll
            for (int f = 0; f < NBF; ++f) acc[f] = (R)0;
#pragma unroll 1
            for (int c0 = 0; c0 < KNR; c0 += CH) {
                // -- A: the tables of CH (primitive quartet, root) entries per ket
#pragma unroll 1
                for (int i0 = lane; i0 < GW * CH; i0 += TW) {
                    const int g = i0 / CH, jl = i0 - g * CH, j = c0 + jl;
                    if (g < ng && j < KNR) {
                        const int t = j / NR, r = j - t * NR, ikcd = t / kab, ikab = t - ikcd * kab;
                        double pb[kPrimWords], pk[kPrimWords];
                        rysw::ld_prim(A.prims + bra.prim0 + ikab, pb);
                        rysw::ld_prim(A.prims + s_prim[g0 + g] + ikcd, pk);
                        // P - A and Q - C of the shells that come first here: the
                        // records hold them for the other ones, A - B away
                        if constexpr (SB) {
#pragma unroll
                            for (int d = 0; d < 3; ++d) pb[3 + d] -= sab[d];
                        }
                        if constexpr (SK) {
#pragma unroll
                            for (int d = 0; d < 3; ++d) pk[3 + d] -= s_sep[d * 32 + g0 + g];
                        }
                        const double p = pb[6], q = pk[6];
                        const double inv = 1.0 / (p + q), rho = p * q * inv;
                        const double qi = q * inv, pi = p * inv;  // rho/p, rho/q
                        const double PQ[3] = {pb[0] - pk[0], pb[1] - pk[1], pb[2] - pk[2]};
                        const double T = rho * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
                        R x, w;
                        if constexpr (sizeof(R) == 4) {
                            rys::rule_root_f<NR>(r, T, A.rys_tab32, &x, &w);
                        } else {
                            rys::rule_root<NR>(r, T, A.rys_tab, &x, &w);
                        }
                        const R seedw = (R)(pb[7] * pk[7] * kTwoOverSqrtPi * sqrt(rho)) * w;
                        const R b00 = (R)(0.5 * inv) * x, b10 = (R)pb[8] * ((R)1 - (R)qi * x),
                                b01 = (R)pk[8] * ((R)1 - (R)pi * x);
                        R *out = tab + (g * CH + jl) * STR;
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const R c00 = (R)pb[3 + d] - (R)(qi * PQ[d]) * x,
                                    c00p = (R)pk[3 + d] + (R)(pi * PQ[d]) * x;
                            R I[E + 1][F + 1];
                            I[0][0] = d == 2 ? seedw : (R)1;
#pragma unroll
                            for (int i = 0; i < E; ++i)
                                I[i + 1][0] = c00 * I[i][0] + (i ? (R)i * b10 * I[i - 1][0] : (R)0);
#pragma unroll
                            for (int k = 0; k < F; ++k)
#pragma unroll
                                for (int i = 0; i <= E; ++i) {
                                    R v = c00p * I[i][k];
                                    if (k) v += (R)k * b01 * I[i][k - 1];
                                    if (i) v += (R)i * b00 * I[i - 1][k];
                                    I[i][k + 1] = v;
                                }
#pragma unroll
                            for (int i = 0; i <= E; ++i)
#pragma unroll
                                for (int k = 0; k <= F; ++k) out[d * TS + i * (F + 1) + k] = I[i][k];
                        }
                    }
                }
                sync();
                // -- B: this lane's ket row over the entries
                if (gl < ng) {
                    const int nj = min(CH, KNR - c0);
                    const R *bx = tab + gl * CH * STR + ex * (F + 1);
                    const R *by = tab + gl * CH * STR + TS + ey * (F + 1);
                    const R *bz = tab + gl * CH * STR + 2 * TS + ez * (F + 1);
#pragma unroll 1
                    for (int jl = 0; jl < nj; ++jl, bx += STR, by += STR, bz += STR) {
                        R ix[F + 1], iy[F + 1], iz[F + 1];
#pragma unroll
                        for (int k = 0; k <= F; ++k) {
                            ix[k] = bx[k];
                            iy[k] = by[k];
                            iz[k] = bz[k];
                        }
#pragma unroll
                        for (int a = 0; a <= F; ++a)
#pragma unroll
                            for (int b = 0; a + b <= F; ++b) {
                                const R pxy = ix[a] * iy[b];
#pragma unroll
                                for (int c = 0; a + b + c <= F; ++c)
                                    if (a + b + c >= LC) acc[fs.idx[a][b][c]] += pxy * iz[c];
                            }
                    }
                }
                sync();
            }

            // -- C: the ket HRR from the row, to X[g][e][cd]; the bra block's share
            if (gl < ng) {
                const int at = g0 + gl;
                const double sep[3] = {s_sep[at], s_sep[32 + at], s_sep[64 + at]};
                double pw[3 * (LD + 1)];
                rysw::sep_powers<LD>(sep, pw);
                const double *dcd = M.D + (size_t)s_oc[at] * n_ao + s_od[at];
                R *xr = X + (gl * NBE + el) * XS;
                double s = 0.0;
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                    R v[NC];
#pragma unroll
                    for (int kx = cds.x[d]; kx >= 0; --kx)
#pragma unroll
                        for (int ky = cds.y[d]; ky >= 0; --ky)
#pragma unroll
                            for (int kz = cds.z[d]; kz >= 0; --kz) {
                                const bool top = kx == cds.x[d] && ky == cds.y[d] && kz == cds.z[d];
                                const R co = (R)((double)(rys::binom(cds.x[d], kx) * rys::binom(cds.y[d], ky) *
                                                          rys::binom(cds.z[d], kz)) *
                                                 pw[cds.x[d] - kx] * pw[(LD + 1) + cds.y[d] - ky] *
                                                 pw[2 * (LD + 1) + cds.z[d] - kz]);
#pragma unroll
                                for (int c = 0; c < NC; ++c) {
                                    const R t = acc[fs.idx[cc.x[c] + kx][cc.y[c] + ky][cc.z[c] + kz]];
                                    v[c] = top ? t : v[c] + co * t;
                                }
                            }
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        xr[c * ND + d] = v[c];
                        s += __ldg(dcd + (size_t)c * n_ao + d) * (double)v[c];
                    }
                }
                jsum += 2.0 * s_deg[at] * s;
            }
            sync();

            // -- E: the digest of the five ket-dependent blocks
            double pw[3 * (LB + 1)];
            rysw::sep_powers<LB>(sab, pw);
            const int gx = lane / (ND * CS), rem = lane - gx * (ND * CS), cs = rem / ND, d = rem - cs * ND;
#pragma unroll 1
            for (int q0 = 0; q0 < ng; q0 += GX) {
                const bool on = gx < GX && q0 + gx < ng;
                const int at = on ? g0 + q0 + gx : g0;
                const int oc = s_oc[at], od = s_od[at];
                const double deg = s_deg[at];
                double dad[NA], dbd[NB], kad[NA], kbd[NB];
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    dad[a] = __ldg(M.D + (size_t)(oa + a) * n_ao + od + d);
                    kad[a] = 0.0;
                }
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    dbd[b] = __ldg(M.D + (size_t)(ob + b) * n_ao + od + d);
                    kbd[b] = 0.0;
                }
                const R *xg = X + (q0 + (on ? gx : 0)) * NBE * XS + d;
#pragma unroll 1
                for (int cb = 0; cb < CPL; cb += BATCH) {
#pragma unroll 1
                    for (int ci = 0; ci < BATCH; ++ci) {
                        const int c = cs + (cb + ci) * CS;
                        double kac[NA], kbc[NB];
#pragma unroll
                        for (int a = 0; a < NA; ++a) kac[a] = 0.0;
#pragma unroll
                        for (int b = 0; b < NB; ++b) kbc[b] = 0.0;
                        if (on && c < NC) {
                            R x[NBE];
#pragma unroll
                            for (int e = 0; e < NBE; ++e) x[e] = xg[e * XS + c * ND];
                            double dac[NA];
#pragma unroll
                            for (int a = 0; a < NA; ++a) dac[a] = __ldg(M.D + (size_t)(oa + a) * n_ao + oc + c);
                            double jcd = 0.0;
#pragma unroll
                            for (int b = 0; b < NB; ++b) {
                                const double dbc = __ldg(M.D + (size_t)(ob + b) * n_ao + oc + c);
                                R y[NA];
#pragma unroll
                                for (int kx = cbs.x[b]; kx >= 0; --kx)
#pragma unroll
                                    for (int ky = cbs.y[b]; ky >= 0; --ky)
#pragma unroll
                                        for (int kz = cbs.z[b]; kz >= 0; --kz) {
                                            const bool top = kx == cbs.x[b] && ky == cbs.y[b] && kz == cbs.z[b];
                                            const R co = (R)((double)(rys::binom(cbs.x[b], kx) *
                                                                      rys::binom(cbs.y[b], ky) *
                                                                      rys::binom(cbs.z[b], kz)) *
                                                             pw[cbs.x[b] - kx] * pw[(LB + 1) + cbs.y[b] - ky] *
                                                             pw[2 * (LB + 1) + cbs.z[b] - kz]);
#pragma unroll
                                            for (int a = 0; a < NA; ++a) {
                                                const R t = x[es.idx[ca.x[a] + kx][ca.y[a] + ky][ca.z[a] + kz]];
                                                y[a] = top ? t : y[a] + co * t;
                                            }
                                        }
#pragma unroll
                                for (int a = 0; a < NA; ++a) {
                                    const double v = (double)y[a];
                                    jcd += Dab[a * NB + b] * v;
                                    kac[a] += dbd[b] * v;
                                    kbc[b] += dad[a] * v;
                                    kad[a] += dbc * v;
                                    kbd[b] += dac[a] * v;
                                }
                            }
                            red_add(M.Jp + (size_t)(oc + c) * n_ao + od + d, 2.0 * deg * jcd);
                        }
#pragma unroll
                        for (int a = 0; a < NA; ++a) red[(ci * NK + a) * TW + lane] = kac[a];
#pragma unroll
                        for (int b = 0; b < NB; ++b) red[(ci * NK + NA + b) * TW + lane] = kbc[b];
                    }
                    sync();
                    // K_ac and K_bc: the sums over d
#pragma unroll 1
                    for (int o = lane; o < GX * CS * BATCH * NK; o += TW) {
                        const int i = o % NK, r1 = o / NK, ci = r1 % BATCH, r2 = r1 / BATCH, c2 = r2 % CS, g2 = r2 / CS;
                        const int c = c2 + (cb + ci) * CS;
                        if (q0 + g2 < ng && c < NC && cb + ci < CPL) {
                            const double *rr = red + (ci * NK + i) * TW + (g2 * CS + c2) * ND;
                            double s = 0.0;
#pragma unroll
                            for (int k = 0; k < ND; ++k) s += rr[k];
                            const int at2 = g0 + q0 + g2;
                            const int row = i < NA ? oa + i : ob + i - NA;
                            red_add(M.Kp + (size_t)row * n_ao + s_oc[at2] + c, s_deg[at2] * s);
                        }
                    }
                    sync();
                }
                if constexpr (CS == 1) {
                    if (on) {
#pragma unroll
                        for (int a = 0; a < NA; ++a)
                            red_add(M.Kp + (size_t)(oa + a) * n_ao + od + d, deg * kad[a]);
#pragma unroll
                        for (int b = 0; b < NB; ++b)
                            red_add(M.Kp + (size_t)(ob + b) * n_ao + od + d, deg * kbd[b]);
                    }
                } else {
                    // the residues of c summed over their lanes (the c = 0 lane's adds)
                    if constexpr (TW > 32) {
#pragma unroll
                        for (int i = 0; i < NK; ++i) red[i * TW + lane] = i < NA ? kad[i < NA ? i : 0] : kbd[i < NA ? 0 : i - NA];
                        sync();
                    }
#pragma unroll
                    for (int i = 0; i < NK; ++i) {
                        const double v = i < NA ? kad[i < NA ? i : 0] : kbd[i < NA ? 0 : i - NA];
                        double s = v;
                        if constexpr (TW == 32) {
#pragma unroll
                            for (int k = 1; k < CS; ++k) s += __shfl_down_sync(kAll, v, k * ND);
                        } else if (on && cs == 0) {
#pragma unroll
                            for (int k = 1; k < CS; ++k) s += red[i * TW + lane + k * ND];
                        }
                        if (on && cs == 0)
                            red_add(M.Kp + (size_t)(i < NA ? oa + i : ob + i - NA) * n_ao + od + d, deg * s);
                    }
                    if constexpr (TW > 32) sync();
                }
            }
            sync();  // X is read before the next group's tables
        }

        // -- the bra block: the bra HRR of the lanes' sums, once per item
        red = ws;  // the region is free here
        red[lane] = gl < GW ? jsum : 0.0;
        sync();
        if (lane < NBE) {
            double s = red[lane];
#pragma unroll
            for (int g = 1; g < GW; ++g) s += red[g * NBE + lane];
            red[TW + lane] = s;
        }
        sync();
        {
            double pw[3 * (LB + 1)];
            rysw::sep_powers<LB>(sab, pw);
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    if (lane != (a * NB + b) % TW) continue;
                    double v = 0.0;
#pragma unroll
                    for (int kx = 0; kx <= cbs.x[b]; ++kx)
#pragma unroll
                        for (int ky = 0; ky <= cbs.y[b]; ++ky)
#pragma unroll
                            for (int kz = 0; kz <= cbs.z[b]; ++kz)
                                v += (double)(rys::binom(cbs.x[b], kx) * rys::binom(cbs.y[b], ky) *
                                              rys::binom(cbs.z[b], kz)) *
                                     pw[cbs.x[b] - kx] * pw[(LB + 1) + cbs.y[b] - ky] *
                                     pw[2 * (LB + 1) + cbs.z[b] - kz] *
                                     red[TW + es.idx[ca.x[a] + kx][ca.y[a] + ky][ca.z[a] + kz]];
                    if (v != 0.0) red_add(M.Jp + (size_t)(oa + a) * n_ao + ob + b, v);
                }
        }
        sync();
        red = ws + S::XD;
    }
}

// One class's kernel: its shared-memory attribute, occupancy and launch.
template <int LA, int LB, int LC, int LD, typename R>
struct RysWarpOne {
    using S = rysw::Shape<LA, LB, LC, LD, R>;
    static constexpr int kSmem = S::kTeams * S::SMD * (int)sizeof(double);
    static void attr() {
        static bool done = false;
        if (done) return;
        cudaFuncSetAttribute(rys_warp_kernel<LA, LB, LC, LD, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        done = true;
    }
    static int occupancy() {  // a constant of the kernel: asked once
        static const int per_sm = [] {
            attr();
            int n = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_warp_kernel<LA, LB, LC, LD, R>, S::kThreads,
                                                          kSmem);
            return n;
        }();
        return per_sm;
    }
    static cudaError_t launch(int grid, cudaStream_t st, const KArgs &a) {
        attr();
        rys_warp_kernel<LA, LB, LC, LD, R><<<grid, S::kThreads, kSmem, st>>>(a);
        return cudaGetLastError();
    }
};

}  // namespace fjb
