// Symmetric DP0 tiles: test and trial are the same DP0 space on one grid, so
// the element pair (i, j) and its transpose (j, i) use the same quadrature
// points with the roles of x and y exchanged.  One sweep over the 36 point
// pairs of (i, j), i < j, gives both entries:
//   single layer      A_ij = A_ji            (the kernel is symmetric in x, y)
//   double layer      A_ij with (y - x).n_j, A_ji with (x - y).n_i
//   adjoint double    the double-layer pair with the two entries exchanged
//   combined field    double layer + eta * the shared single layer
// so r, 1/r and exp(ikr) are evaluated once per point pair for two entries.
// A launch covers the tiles on or above the diagonal (row chunk <= column
// block); inside a diagonal tile only i <= j is processed, and i == j (the
// coincident pair, always adjacent) is zeroed for the singular pass.
// Entry (i, j) is stored by the thread of column j (coalesced); entry (j, i)
// lands in row j (one 8- or 16-byte store per row, merged in L2 with the
// stores of neighbouring rows of the same warp).
#pragma once

#include <type_traits>

#include "dp0.cuh"
#include "orbit_pair.cuh"

namespace bc {

template <int K>
struct SymTraits {
    static constexpr bool slp_part = (K == BEMPPCUDA_LAPLACE_SLP || K == BEMPPCUDA_HELMHOLTZ_SLP ||
                                      K == BEMPPCUDA_MODHELM_SLP || K == BEMPPCUDA_HELMHOLTZ_COMBINED);
    static constexpr bool dlp_part = (K == BEMPPCUDA_LAPLACE_DLP || K == BEMPPCUDA_LAPLACE_ADLP ||
                                      K == BEMPPCUDA_HELMHOLTZ_DLP || K == BEMPPCUDA_HELMHOLTZ_ADLP ||
                                      K == BEMPPCUDA_MODHELM_DLP || K == BEMPPCUDA_MODHELM_ADLP ||
                                      K == BEMPPCUDA_HELMHOLTZ_COMBINED);
    static constexpr bool swap = (K == BEMPPCUDA_LAPLACE_ADLP || K == BEMPPCUDA_HELMHOLTZ_ADLP ||
                                  K == BEMPPCUDA_MODHELM_ADLP);
    static constexpr bool helm = KernelTraits<K>::helm;
    static constexpr bool modhelm = KernelTraits<K>::modhelm;
    static constexpr bool supported = slp_part || dlp_part;
};

// Forms of the FP64 sweep.
//  points: coordinates differenced per point pair, any 6-point rule; a real wavenumber's exp(ikr) factored about the
//    centroid distance by offset class (fastmath.cuh), a complex one or exp(-w r) reduced per point pair.
//  orbit: the two-orbit rule (orbit_pair.cuh), where the amplitudes exp(-Im k r) and exp(-w r) are factored too.
// The orbit form takes fewer FP64 operations in every kernel, but its chains depend on each other more and it
// runs the FP64 pipe at 75 - 80 % against 86 %: with the amplitudes' library exponential gone it is
// 1.25 - 1.6 times faster (n = 16200: combined field k = 4 + 0.4i 28.5 -> 17.5 ms, modified Helmholtz single
// layer 11.2 -> 8.9 ms), without them between 0.92 (Laplace single layer) and 1.05 of the points form (double layer).
constexpr int SYM_POINTS = 0, SYM_POINTS_CK = 3, SYM_ORBIT = 4, SYM_ORBIT_CK = 8;
constexpr bool form_orbit(int form) { return form >= SYM_ORBIT; }
constexpr bool form_ck(int form) { return form == SYM_POINTS_CK || form >= SYM_ORBIT_CK; }
constexpr int form_class(int form) { return form == SYM_POINTS_CK ? 0 : form & 3; }

// The form of a problem: params as in RegParams, radius_sum bounds R_t + R_s (0: unknown).
inline int sym_form(int kernel, const double *params, double radius_sum, bool orbits, const OrbitRule &orbit) {
    const bool laplace = kernel <= BEMPPCUDA_LAPLACE_ADLP;
    const bool modhelm = kernel >= BEMPPCUDA_MODHELM_SLP && kernel <= BEMPPCUDA_MODHELM_ADLP;
    const bool ck = !laplace && !modhelm && params[1] != 0.0;
    if (laplace) return SYM_POINTS;
    const double kmax = ck ? fmax(fabs(params[0]), fabs(params[1])) : fabs(params[0]);
    const int cls = offset_class64(kmax * radius_sum * (orbits ? orbit.rho : 1.0));
    if (!ck && !modhelm) return SYM_POINTS + cls;
    // (the orbit form sums h / Re k: finite above this bound for |k| and 1 / r up to 1e60)
    if (!orbits || fabs(params[0]) < 1e-100) return ck ? SYM_POINTS_CK : SYM_POINTS;
    return (ck ? SYM_ORBIT_CK : SYM_ORBIT) + cls;
}

// Calls f with the form as a compile-time constant, one of those that kernel K has.
template <int K, class F>
static void with_form(int form, F &&f) {
    if constexpr (KernelTraits<K>::helm) {
        switch (form) {
        case SYM_POINTS + 2: f(std::integral_constant<int, SYM_POINTS + 2>()); return;
        case SYM_POINTS + 1: f(std::integral_constant<int, SYM_POINTS + 1>()); return;
        case SYM_POINTS_CK: f(std::integral_constant<int, SYM_POINTS_CK>()); return;
        case SYM_ORBIT_CK: f(std::integral_constant<int, SYM_ORBIT_CK>()); return;
        case SYM_ORBIT_CK + 1: f(std::integral_constant<int, SYM_ORBIT_CK + 1>()); return;
        case SYM_ORBIT_CK + 2: f(std::integral_constant<int, SYM_ORBIT_CK + 2>()); return;
        default: break;
        }
    } else if constexpr (KernelTraits<K>::modhelm) {
        switch (form) {
        case SYM_ORBIT: f(std::integral_constant<int, SYM_ORBIT>()); return;
        case SYM_ORBIT + 1: f(std::integral_constant<int, SYM_ORBIT + 1>()); return;
        case SYM_ORBIT + 2: f(std::integral_constant<int, SYM_ORBIT + 2>()); return;
        default: break;
        }
    }
    f(std::integral_constant<int, SYM_POINTS>());
}

// A test element of the sweep: the orbit form's centroid and vertex offsets, or the six points and the centroid.
union TestElem64s {
    OrbitTest o;
    struct {
        double x[NQ6][3], c[3];
    } p;
};

struct TestBlock64s {
    TestElem64s e[DP0_TCHUNK];
    double n[DP0_TCHUNK][3];
    double ie[DP0_TCHUNK];
    int v[DP0_TCHUNK][3];
};

// FP64.  A complex wavenumber k = kr + i ki has exp(ikr) = exp(i kr r) exp(-ki r) and
// (ikr - 1) / r = -(1/r + ki) + i kr in the double layer; G(x, y) = G(y, x) for complex k too, so the sweep
// is unchanged.  Modified Helmholtz (real, w = p[0]): the Laplace sums with exp(-w r) (single layer) and
// exp(-w r) (1 + w r) (double layers).
//
// The tile is split into three steps shared by the assembly (stores A_ij, A_ji) and the
// matrix-free apply (accumulates A x): staging the test block, loading a thread's trial
// element, and the sweep over the 36 point pairs of one element pair.

// Stage test elements t0 .. t0 + tcount - 1.
template <int FORM>
__device__ __forceinline__ void stage_sym64(const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc,
                                            int64_t t0, int tcount, TestBlock64s &sb) {
    for (int idx = threadIdx.x; idx < tcount; idx += blockDim.x) {
        const int64_t t = prm.tsup[t0 + idx];
        Geom g;
        load_geom(prm.tg, prm.tne, t, prm.tnm ? (double)prm.tnm[t] : 1.0, g);
        if (form_orbit(FORM)) {
            stage_orbit(prm.tg, prm.tne, t, g, oc, sb.e[idx].o);
        } else {
            for (int p = 0; p < NQ6; ++p) to_global(g, rule.x[p], rule.y[p], sb.e[idx].p.x[p]);
#pragma unroll
            for (int d = 0; d < 3; ++d) sb.e[idx].p.c[d] = __ldg(prm.tg + (22 + d) * prm.tne + t);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            sb.n[idx][d] = g.n[d];
            sb.v[idx][d] = __ldg(prm.tel + 3 * t + d);
        }
        sb.ie[idx] = g.ie;
    }
}

// One thread's trial element: vertex ids, and the parked orbit fields, or its geometry and points.
struct SymTrial64 {
    int sv0, sv1, sv2;
    OrbitTrial<DP0_THREADS> o;
    Geom gs;
    double y[NQ6][3], sc[3];
};
constexpr int SYM_PARK = OT_FIELDS * DP0_THREADS;  // doubles of shared memory

template <int FORM>
__device__ __forceinline__ void load_trial_sym64(const RegParams &prm, const QuadRule &rule, int64_t si, double *park,
                                                 SymTrial64 &tr) {
    const int64_t s = prm.ssup[si];
    load_geom(prm.sg, prm.sne, s, prm.snm ? (double)prm.snm[s] : 1.0, tr.gs);
    tr.sv0 = __ldg(prm.sel + 3 * s);
    tr.sv1 = __ldg(prm.sel + 3 * s + 1);
    tr.sv2 = __ldg(prm.sel + 3 * s + 2);
    if (form_orbit(FORM)) {
        tr.o = park_orbit_trial<DP0_THREADS>(prm.sg, prm.sne, s, tr.gs, park);
        orbit_fence();
    } else {
#pragma unroll
        for (int q = 0; q < NQ6; ++q) to_global(tr.gs, rule.x[q], rule.y[q], tr.y[q]);
#pragma unroll
        for (int d = 0; d < 3; ++d) tr.sc[d] = form_class(FORM) > 0 ? __ldg(prm.sg + (22 + d) * prm.sne + s) : 0.0;
    }
}

// The sums of a pair: s single layer, u double layer with the trial normal, v with the test normal
// (weights included, 1 / (4 pi), areas and the factor at r_c left out; u and v as -u_re + i u_im).
struct SymSums {
    double s_re, s_im, u_re, u_im, v_re, v_im;
};

// One test point's terms of the six trial points; yw[q] = (x - y_q) . n_t, xn = (y - x) . n_s.
template <int K, int FORM>
__device__ __forceinline__ void point_sym64(const double r2[6], const double w[6], double wp, double xn,
                                            const double yw[6], double kr, double ki, double krc, double kirc,
                                            SymSums &a) {
    using ST = SymTraits<K>;
    constexpr bool CK = form_ck(FORM) && ST::helm;
    constexpr int CLS = form_class(FORM);
    double pr = 0.0, pi = 0.0, ur = 0.0, ui = 0.0, vr = 0.0, vi = 0.0;
    const double ik = ST::helm && form_orbit(FORM) ? 1.0 / kr : 0.0;
#pragma unroll
    for (int q = 0; q < NQ6; ++q) {
        const double rinv = rsqrt64(r2[q]);
        double f = w[q] * rinv;
        if (!ST::helm) {
            double e = 1.0, e1 = 1.0;  // modified Helmholtz: exp(-w r), exp(-w r) (1 + w r)
            if (ST::modhelm) {
                const double r = r2[q] * rinv;
                e = exp_off64<CLS>(fma(-kr, r, krc));
                e1 = e * fma(kr, r, 1.0);
            }
            if (ST::slp_part) pr = ST::modhelm ? fma(f, e, pr) : pr + f;
            if (ST::dlp_part) {
                const double g3 = ST::modhelm ? f * rinv * rinv * e1 : f * rinv * rinv;
                ur += g3;
                vr = fma(g3, yw[q], vr);
            }
        } else {
            const double r = r2[q] * rinv;
            double sn, cs;
            sincos_off64<CLS>(fma(kr, r, -krc), &sn, &cs);
            if (CK) f *= exp_off64<CLS>(fma(-ki, r, kirc));
            if (ST::slp_part) {
                pr = fma(f, cs, pr);
                pi = fma(f, sn, pi);
            }
            if (ST::dlp_part) {
                // (ikr - 1) e^{ikr} / r^3 is -h1 + i h2 per unit f (dot) / r; the orbit forms carry h / kr
                const double fr = f * rinv, rk = CK ? rinv + ki : rinv;
                double h1, h2;
                if (form_orbit(FORM)) {
                    const double rho = rk * ik;
                    h1 = fma(rho, cs, sn);
                    h2 = fma(-rho, sn, cs);
                } else {
                    h1 = fma(rk, cs, kr * sn);
                    h2 = fma(kr, cs, -rk * sn);
                }
                const double gt = fr * yw[q];
                ur = fma(fr, h1, ur);
                ui = fma(fr, h2, ui);
                vr = fma(gt, h1, vr);
                vi = fma(gt, h2, vi);
            }
        }
    }
    const double wn = wp * xn;
    a.s_re = fma(wp, pr, a.s_re);
    a.s_im = fma(wp, pi, a.s_im);
    a.u_re = fma(wn, ur, a.u_re);
    a.u_im = fma(wn, ui, a.u_im);
    a.v_re = fma(wp, vr, a.v_re);
    a.v_im = fma(wp, vi, a.v_im);
}

// The sums of an element pair in the orbit form (NEAR: differenced coordinates, orbit_r2).
template <int K, int FORM, bool NEAR>
__device__ __forceinline__ void sums_sym64(const OrbitTest &te, const OrbitTrial<DP0_THREADS> &tr, const OrbitPair &p,
                                           const OrbitConsts &oc, double Dn, const double yw[6], double kr, double ki,
                                           SymSums &a) {
    using ST = SymTraits<K>;
    const double w[6] = {oc.w[0], oc.w[0], oc.w[0], oc.w[1], oc.w[1], oc.w[1]};
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        const double e[3] = {te.e[i][0], te.e[i][1], te.e[i][2]};
        double f0[3], f1[3], en = 0.0;
        tr.f(f0, f1);
        const double De = odot(p.D, e), E0 = odot(e, f0), E1 = odot(e, f1);
        const double E[3] = {E0, E1, -(E0 + E1)};
        if (ST::dlp_part) {
            double sn[3];
            tr.n(sn);
            en = odot(e, sn);
        }
#pragma unroll 1
        for (int op = 0; op < 2; ++op) {
            double r2[6];
            orbit_r2<NEAR>(p, tr, oc, op, e, te.ge[op][i], De, E, r2);
            point_sym64<K, FORM>(r2, w, oc.w[op], fma(-oc.g[op], en, Dn), yw, kr, ki, p.krc, p.kirc, a);
        }
    }
}

// A_ij and A_ji of the non-adjacent pair (test element tt of the block, the thread's trial element).
template <int K, int FORM>
__device__ __forceinline__ void pair_sym64(const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc,
                                           const TestBlock64s &sb, int tt, const SymTrial64 &tr, double &a_re,
                                           double &a_im, double &b_re, double &b_im) {
    using ST = SymTraits<K>;
    constexpr bool ORB = form_orbit(FORM), CK = form_ck(FORM) && ST::helm;
    constexpr int CLS = form_class(FORM), FAM = kernel_family<K>();
    const double kr = prm.p[0], ki = CK ? prm.p[1] : 0.0, etar = prm.p[2], etai = prm.p[3];
    const double tn[3] = {sb.n[tt][0], sb.n[tt][1], sb.n[tt][2]};
    // Normal terms: (y - x).n_s is one value per test point since y lies in the plane of the trial element,
    // (x - y).n_t one value per trial point since x lies in the plane of the test element
    double yw[NQ6];
    SymSums a = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double ph_c = 1.0, ph_s = 0.0;
    if constexpr (ORB) {
        const OrbitTest &te = sb.e[tt].o;
        OrbitPair p;
        orbit_pair<FAM, CK, CLS>(te, tr.o, oc, kr, ki, p);
        double Dn = 0.0;
        if (ST::dlp_part) {
            double sn[3], v0[3], v1[3];
            tr.o.n(sn);
            tr.o.f(v0, v1);
            Dn = odot(p.D, sn);
            const double Dt = odot(p.D, tn), f0 = odot(v0, tn), f1 = odot(v1, tn);
            const double f[3] = {f0, f1, -(f0 + f1)};
#pragma unroll
            for (int q = 0; q < NQ6; ++q) yw[q] = -fma(oc.g[q / 3], f[q % 3], Dt);
        }
        if (p.far)
            sums_sym64<K, FORM, false>(te, tr.o, p, oc, Dn, yw, kr, ki, a);
        else
            sums_sym64<K, FORM, true>(te, tr.o, p, oc, Dn, yw, kr, ki, a);
        orbit_phase<FAM, CK, CLS>(p, ph_c, ph_s);
        if (ST::helm && ST::dlp_part) {  // the sums of h / kr
            a.u_re *= kr;
            a.u_im *= kr;
            a.v_re *= kr;
            a.v_im *= kr;
        }
    } else {
        const double(*x)[3] = sb.e[tt].p.x, *c = sb.e[tt].p.c;
        const Geom &gs = tr.gs;
        double krc = 0.0;
        if (CLS > 0) {
            const double D0 = tr.sc[0] - c[0], D1 = tr.sc[1] - c[1], D2 = tr.sc[2] - c[2];
            krc = kr * sqrt(fma(D2, D2, fma(D1, D1, D0 * D0)));
            sincos_cw64(krc, &ph_s, &ph_c);
        }
        if (ST::dlp_part)
#pragma unroll
            for (int q = 0; q < NQ6; ++q)
                yw[q] = fma(c[2] - tr.y[q][2], tn[2], fma(c[1] - tr.y[q][1], tn[1], (c[0] - tr.y[q][0]) * tn[0]));
        for (int p = 0; p < NQ6; ++p) {
            const double x0 = x[p][0], x1 = x[p][1], x2 = x[p][2];
            double xn = 0.0, r2[6];
            if (ST::dlp_part)
                xn = fma(gs.v0[2] - x2, gs.n[2], fma(gs.v0[1] - x1, gs.n[1], (gs.v0[0] - x0) * gs.n[0]));
#pragma unroll
            for (int q = 0; q < NQ6; ++q) {
                const double d0 = tr.y[q][0] - x0, d1 = tr.y[q][1] - x1, d2 = tr.y[q][2] - x2;
                r2[q] = fma(d2, d2, fma(d1, d1, d0 * d0));
            }
            point_sym64<K, FORM>(r2, rule.w, rule.w[p], xn, yw, kr, ki, krc, 0.0, a);
        }
    }
    // kernel values: Laplace DLP -sum f dot / r^2; Helmholtz DLP -u_re + i u_im
    double dr = 0.0, di = 0.0, er = 0.0, ei = 0.0;  // double-layer parts of A_ij, A_ji
    if (ST::dlp_part) {
        dr = -a.u_re;
        di = ST::helm ? a.u_im : 0.0;
        er = -a.v_re;
        ei = ST::helm ? a.v_im : 0.0;
    }
    if (K == BEMPPCUDA_HELMHOLTZ_COMBINED) {
        const double sr = fma(etar, a.s_re, -etai * a.s_im), sim = fma(etar, a.s_im, etai * a.s_re);
        a_re = dr + sr;
        a_im = di + sim;
        b_re = er + sr;
        b_im = ei + sim;
    } else if (ST::slp_part) {
        a_re = b_re = a.s_re;
        a_im = b_im = a.s_im;
    } else if (ST::swap) {
        a_re = er;
        a_im = ei;
        b_re = dr;
        b_im = di;
    } else {
        a_re = dr;
        a_im = di;
        b_re = er;
        b_im = ei;
    }
    const double scale = BC_INV_4PI * sb.ie[tt] * (ORB ? tr.o.ld(OT_IE) : tr.gs.ie);
    ph_c *= scale;
    if (CLS > 0 && ST::helm) {
        ph_s *= scale;
        double t = fma(a_re, ph_c, -a_im * ph_s);
        a_im = fma(a_re, ph_s, a_im * ph_c);
        a_re = t;
        t = fma(b_re, ph_c, -b_im * ph_s);
        b_im = fma(b_re, ph_s, b_im * ph_c);
        b_re = t;
    } else {
        a_re *= ph_c;
        a_im *= ph_c;
        b_re *= ph_c;
        b_im *= ph_c;
    }
}

template <int K, int FORM, bool STRIPE = false>
__device__ __forceinline__ void regular_dp0_fp64_sym_tile(const RegParams &prm, const QuadRule &rule,
                                                        const OrbitConsts &oc, int64_t tile_x, int64_t t0, int rows,
                                                        TestBlock64s &sb, double *park) {
    const int tcount = (int)min((int64_t)rows, prm.ntest - t0);
    stage_sym64<FORM>(prm, rule, oc, t0, tcount, sb);
    __syncthreads();

    const int64_t si = tile_x * DP0_THREADS + threadIdx.x;
    if (si < prm.ntrial && t0 <= si) {
        SymTrial64 tr;
        load_trial_sym64<FORM>(prm, rule, si, park, tr);
#pragma unroll 1
        for (int tt = 0; tt < tcount; ++tt) {
            const int64_t row = t0 + tt;
            if (row > si) break;  // rows increase with tt: the rest of this column lies below the diagonal
            const bool adj = row == si || (prm.grids_identical && shares_vertex(sb.v[tt], tr.sv0, tr.sv1, tr.sv2));
            double a_re = 0.0, a_im = 0.0, b_re = 0.0, b_im = 0.0;  // A_ij, A_ji
            if (!adj) pair_sym64<K, FORM>(prm, rule, oc, sb, tt, tr, a_re, a_im, b_re, b_im);
            store_pair<STRIPE>(prm, row, si, adj, a_re, a_im, b_re, b_im);
        }
    }
    __syncthreads();  // the shared block is reused by the next tile of a persistent loop
}

}  // namespace bc

namespace bc {

// Test block of the packed symmetric sweep, lengths in units of 1/kappa: vertex offsets e_i = kappa (v_i - c_t),
// -g_o^2 |e_i|^2 / 2 per orbit, centroid, normal.
struct TestBlock32q {
    float e[DP0_TCHUNK][3][3];
    float hge[DP0_TCHUNK][2][3];
    double c[DP0_TCHUNK][3];
    float4 n[DP0_TCHUNK];  // unit normal, MIXED_NEAR R
    double ie[DP0_TCHUNK];
    int v[DP0_TCHUNK][3];
    float srad[DP0_THREADS];  // MIXED_NEAR R of each thread's trial element
};

// sin / cos of the point-pair phase offsets of the symmetric sweep (|x| <= 1/2 for phase class
// 2, |x| <= 1 for class 1): the sine by the FP32 minimax polynomial, the cosine by the hardware
// approximation cos.approx.f32 (absolute error below 1e-6 on these ranges; the operator error of
// the sweep measured against FP64 is 1.3e-8 either way).  The cosine moves from the FMA pipe
// to the special-function unit, which this kernel leaves partly idle (its reciprocal and
// reciprocal square root are the other users); the sine stays a polynomial, since both
// functions on that unit saturate it.  Class 0 reduces the argument first (sincos2).
__device__ __forceinline__ float hw_cos(float x) {
    float y;
    asm("cos.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <int PHC>
__device__ __forceinline__ void sincos2_sym(float2 x, float2 *s, float2 *c) {
    if (PHC == 2 || PHC == 1) {
        const float2 x2 = mul2(x, x);
        if (PHC == 2) {
            constexpr float ps[] = BC_SIN_HALF32;
            *s = fma2(mul2(x, x2), fma2(b2(ps[0]), x2, b2(ps[1])), x);
        } else {
            constexpr float ps[] = BC_SIN_SMALL32;
            *s = fma2(mul2(x, x2), fma2(fma2(b2(ps[0]), x2, b2(ps[1])), x2, b2(ps[2])), x);
        }
        *c = f2(hw_cos(x.x), hw_cos(x.y));
    } else {
        sincos2<PHC>(x, s, c);
    }
}

// One thread's trial element, lengths in units of 1/kappa.
struct MixedTrial {
    float f[2][3];  // vertex offsets f_0, f_1 (f_2 = -f_0 - f_1)
    float2 hgf[3];  // -g_q^2 |f_j|^2 / 2 of both orbits
    float n[3], rad;  // normal, MIXED_NEAR R
    double c[3], ie;
    int v[3];
};

template <int K>
__device__ __forceinline__ double mixed_kappa(const RegParams &prm) {
    // units of 1/kappa: Re k (Helmholtz), omega (modified Helmholtz), 1 (Laplace); callers guarantee kappa > 0
    return SymTraits<K>::helm || SymTraits<K>::modhelm ? prm.p[0] : 1.0;
}
// The orbits' offset factors: the first point of an orbit belongs to vertex 2.
__device__ __forceinline__ double mixed_g(const QuadRule &rule, int o) { return 1.0 - 3.0 * rule.x[o * (NQ6 / 2)]; }

template <int K>
__device__ __forceinline__ void load_trial_mixed(const RegParams &prm, const QuadRule &rule, int64_t si, MixedTrial &tr) {
    const double kap = mixed_kappa<K>(prm), g0d = mixed_g(rule, 0), g1d = mixed_g(rule, 1);
    const int64_t s = prm.ssup[si];
    Geom gs;
    load_geom(prm.sg, prm.sne, s, prm.snm ? (double)prm.snm[s] : 1.0, gs);
    double fd[3][3], m2 = 0.0;
    orbit_offsets(gs, fd);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const double ff = odot(fd[j], fd[j]), m = -0.5 * kap * kap * ff;
        m2 = fmax(m2, ff);
        tr.hgf[j] = f2((float)(g0d * g0d * m), (float)(g1d * g1d * m));
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        tr.f[0][d] = (float)(kap * fd[0][d]);
        tr.f[1][d] = (float)(kap * fd[1][d]);
        tr.n[d] = (float)gs.n[d];
        tr.c[d] = __ldg(prm.sg + (22 + d) * prm.sne + s);
        tr.v[d] = __ldg(prm.sel + 3 * s + d);
    }
    tr.rad = (float)(MIXED_NEAR * kap * sqrt(m2));
    tr.ie = gs.ie;
}

// The entries A_ij and A_ji of the test element tt of the block and the trial element, D = kappa (c_s - c_t).  NEAR:
// differenced coordinates and no Newton step: theta = r' - r_c' is as good as r' there.
template <int K, int PHC, bool CK, bool NEAR>
__device__ __forceinline__ void mixed_pair(const RegParams &prm, const QuadRule &rule, const TestBlock32q &sb, int tt,
                                           const MixedTrial &tr, double D0, double D1, double D2, double rc2,
                                           double &a_re, double &a_im, double &b_re, double &b_im) {
    using ST = SymTraits<K>;
    const double kap = mixed_kappa<K>(prm);
    const double betd = CK ? prm.p[1] / prm.p[0] : 0.0;
    const float2 bet2 = b2((float)betd);
    const float go[2] = {(float)mixed_g(rule, 0), (float)mixed_g(rule, 1)};
    const float2 g2 = f2(go[0], go[1]);
    const float(&f)[2][3] = tr.f;
    const float2(&hgf)[3] = tr.hgf;
    const float sn0 = tr.n[0], sn1 = tr.n[1], sn2 = tr.n[2];
    const double ek_r = (K == BEMPPCUDA_HELMHOLTZ_COMBINED) ? kap * prm.p[2] : kap;
    const double ek_i = (K == BEMPPCUDA_HELMHOLTZ_COMBINED) ? kap * prm.p[3] : 0.0;
    const double k2d = kap * kap;
    // weights: w_b for the second test orbit, w_a / w_b applied in FP32 to the first; the trial orbits' at the end
    const double wb = rule.w[NQ6 - 1];
    const float2 rho2 = b2((float)(rule.w[0] / wb));
    const float wqa = rule.wf[0], wqb = rule.wf[NQ6 - 1];
    const auto fdot = [](const float a[3], float b0, float b1, float b2_) {
        return fmaf(a[2], b2_, fmaf(a[1], b1, a[0] * b0));
    };
    const double rc = NEAR ? dist64(rc2) : rc2 * rsqrt64(rc2);
    float ph_s = 0.f, ph_c = 1.f;
    if (ST::helm) phase_reduced32(rc, &ph_s, &ph_c);
    // e^{-beta r_c'} (complex k), e^{-r_c'} (modified Helmholtz)
    const double amp = CK ? exp_neg_reduced(betd * rc) : (ST::modhelm ? exp_neg_reduced(rc) : 1.0);
    const float D0f = (float)D0, D1f = (float)D1, D2f = (float)D2, rcf = (float)rc;
    const float2 rc_2 = b2(rcf), mrc_2 = b2(-rcf), mrc2_2 = b2(-(float)rc2);
    // k (y - x).n_s = Dn - g_p e_i . n_s, one factor per test point; k (x - y).n_t = -Dt - g_q f_j . n_t,
    // one per trial point
    float Dn = 0.f;
    float2 ynt[3];
    if (ST::dlp_part) {
        const float4 tn = sb.n[tt];
        const float mDt = -fmaf(D2f, tn.z, fmaf(D1f, tn.y, D0f * tn.x));
        const float m0 = -fdot(f[0], tn.x, tn.y, tn.z), m1 = -fdot(f[1], tn.x, tn.y, tn.z);
        ynt[0] = fma2(b2(m0), g2, b2(mDt));
        ynt[1] = fma2(b2(m1), g2, b2(mDt));
        ynt[2] = fma2(b2(-(m0 + m1)), g2, b2(mDt));
        Dn = fmaf(D2f, sn2, fmaf(D1f, sn1, D0f * sn0));
    }
    float2 hA[3];  // -A_q / 2
    if (!NEAR) {
        const float a0 = -fdot(f[0], D0f, D1f, D2f), a1 = -fdot(f[1], D0f, D1f, D2f);
        hA[0] = fma2(b2(a0), g2, hgf[0]);
        hA[1] = fma2(b2(a1), g2, hgf[1]);
        hA[2] = fma2(b2(-(a0 + a1)), g2, hgf[2]);
    }
    float E[3][3], De[3], en[3];  // e_i . f_j, D . e_i, e_i . n_s
    if (!NEAR) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float e0 = sb.e[tt][i][0], e1 = sb.e[tt][i][1], e2 = sb.e[tt][i][2];
            De[i] = fmaf(D2f, e2, fmaf(D1f, e1, D0f * e0));
            if (ST::dlp_part) en[i] = fmaf(sn2, e2, fmaf(sn1, e1, sn0 * e0));
            E[i][0] = fdot(f[0], e0, e1, e2);
            E[i][1] = fdot(f[1], e0, e1, e2);
            E[i][2] = -(E[i][0] + E[i][1]);
        }
        De[2] = -(De[0] + De[1]);
        if (ST::dlp_part) en[2] = -(en[0] + en[1]);
#pragma unroll
        for (int j = 0; j < 3; ++j) E[2][j] = -(E[0][j] + E[1][j]);
    }
    float2 s0r = b2(0.f), s0m = b2(0.f), um = b2(0.f), ui = b2(0.f), vm = b2(0.f), vi = b2(0.f);
#pragma unroll (NEAR ? 1 : NQ6)
    for (int p = 0; p < NQ6; ++p) {
        const int i = p % 3, op = p / 3;
        if (p == NQ6 / 2) {  // second orbit: the first orbit's sums times w_a / w_b
            s0r = mul2(s0r, rho2);
            s0m = mul2(s0m, rho2);
            um = mul2(um, rho2);
            ui = mul2(ui, rho2);
            vm = mul2(vm, rho2);
            vi = mul2(vi, rho2);
        }
        const float gp = op == 0 ? go[0] : go[1];
        float x[3];  // NEAR: D - g_p e_i
        float2 hB, gp2, cp2 = b2(0.f);
        if (NEAR) {
            x[0] = fmaf(-gp, sb.e[tt][i][0], D0f);
            x[1] = fmaf(-gp, sb.e[tt][i][1], D1f);
            x[2] = fmaf(-gp, sb.e[tt][i][2], D2f);
            if (ST::dlp_part) cp2 = b2(fdot(x, sn0, sn1, sn2));
        } else {
            hB = b2(fmaf(gp, De[i], sb.hge[tt][op][i]));  // -B_p / 2
            gp2 = f2(gp * go[0], gp * go[1]);
            if (ST::dlp_part) cp2 = b2(fmaf(-gp, en[i], Dn));
        }
        float2 pum = b2(0.f), pui = b2(0.f);  // sums over q of the A_ij double-layer factors, times cp per p
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            float2 hs, mr2;  // -s / 2, -r'^2
            if (NEAR) {
                mr2 = near_mr2(x, f, j, g2);
            } else {
                hs = fma2(b2(E[i][j]), gp2, add2(hA[j], hB));
                mr2 = fma2(hs, b2(2.f), mrc2_2);
            }
            const float2 rinv = f2(rsqrt_approx(-mr2.x), rsqrt_approx(-mr2.y));
            // -theta
            float2 mt = b2(0.f);
            if (ST::helm || ST::modhelm) {
                mt = fma2(mr2, rinv, rc_2);
                if (!NEAR) mt = fma2(fma2(mt, fma2(mt, b2(0.5f), mrc_2), hs), rinv, mt);
            }
            if (!ST::helm) {
                // modified Helmholtz: e^{-theta} per pair (e^{-r_c'} per element pair), the double
                // layers' (1 + r') e^{-theta}
                float2 am = b2(1.f), am1 = b2(1.f);
                if (ST::modhelm) {
                    am = f2(__expf(mt.x), __expf(mt.y));
                    am1 = mul2(am, add2(b2(1.f), mul2(mul2(mr2, rinv), b2(-1.f))));
                }
                if (ST::slp_part) s0r = ST::modhelm ? fma2(rinv, am, s0r) : add2(rinv, s0r);
                if (ST::dlp_part) {
                    float2 fr = mul2(mul2(rinv, rinv), rinv);
                    if (ST::modhelm) fr = mul2(fr, am1);
                    pum = add2(fr, pum);
                    vm = fma2(fr, ynt[j], vm);
                }
            } else {
                float2 ms, cs;  // -sin, cos of theta
                sincos2_sym<PHC>(mt, &ms, &cs);
                if (CK) {
                    const float2 am = f2(__expf(bet2.x * mt.x), __expf(bet2.x * mt.y));
                    cs = mul2(cs, am);
                    ms = mul2(ms, am);
                }
                if (ST::slp_part) {
                    s0r = fma2(rinv, cs, s0r);
                    s0m = fma2(rinv, ms, s0m);
                }
                if (ST::dlp_part) {
                    const float2 fr = mul2(rinv, rinv);
                    const float2 rb = CK ? add2(rinv, bet2) : rinv;  // 1 / r' (+ beta)
                    const float2 mh1 = fma2(mul2(rb, b2(-1.f)), cs, ms);  // -h1
                    const float2 h2 = fma2(rb, ms, cs);
                    const float2 gt = mul2(fr, ynt[j]);
                    pum = fma2(fr, mh1, pum);
                    pui = fma2(fr, h2, pui);
                    vm = fma2(gt, mh1, vm);
                    vi = fma2(gt, h2, vi);
                }
            }
        }
        if (ST::dlp_part) {
            um = fma2(cp2, pum, um);
            if (ST::helm) ui = fma2(cp2, pui, ui);
        }
    }
    // entry = w_b [kappa eta S0 + kappa^2 (-h1 sum + i h2 sum)], rotated by exp(i r_c') and scaled; um and vm
    // hold the -h1 sums (Helmholtz) or the sums of w (d'.n) / r'^3 (real kernels)
    const auto orbits = [&](float2 v) { return (double)fmaf(wqa, v.x, wqb * v.y); };
    double sr = 0.0, sim = 0.0;
    if (ST::slp_part) {
        const double xr = orbits(s0r), xi = ST::helm ? -orbits(s0m) : 0.0;
        sr = fma(ek_r, xr, -ek_i * xi);
        sim = fma(ek_r, xi, ek_i * xr);
    }
    double dr = 0.0, di = 0.0, er = 0.0, ei = 0.0;
    if (ST::dlp_part) {
        const double sg = ST::helm ? k2d : -k2d;
        dr = sg * orbits(um);
        er = sg * orbits(vm);
        if (ST::helm) {
            di = k2d * orbits(ui);
            ei = k2d * orbits(vi);
        }
    }
    if (ST::swap) {
        a_re = er;
        a_im = ei;
        b_re = dr;
        b_im = di;
    } else {
        a_re = sr + dr;
        a_im = sim + di;
        b_re = sr + er;
        b_im = sim + ei;
    }
    const double scale = BC_INV_4PI * sb.ie[tt] * tr.ie * wb * amp;
    const double pc = (double)ph_c, ps = (double)ph_s;
    double rot = a_re * pc - a_im * ps;
    a_im = (a_re * ps + a_im * pc) * scale;
    a_re = rot * scale;
    rot = b_re * pc - b_im * ps;
    b_im = (b_re * ps + b_im * pc) * scale;
    b_re = rot * scale;
}

// A near pair: a function of its own that loads the trial element again, called after the sweep's own evaluation, so
// that the sweep keeps its registers and schedule.  On meshes without such pairs it costs the combined field nothing
// (32768 elements 21.12 -> 21.08 ms), other kernels up to 2 %; branching around the sweep's evaluation 1 - 2 %, inlined or
// collected for after the sweep 2 - 10 %.
template <int K, int PHC, bool CK>
__device__ __noinline__ void mixed_near_pair(const RegParams &prm, const QuadRule &rule, const TestBlock32q &sb, int tt,
                                             int64_t si, double (&ab)[4]) {
    const double kap = mixed_kappa<K>(prm);
    MixedTrial tr;
    load_trial_mixed<K>(prm, rule, si, tr);
    const double D0 = kap * (tr.c[0] - sb.c[tt][0]), D1 = kap * (tr.c[1] - sb.c[tt][1]),
                 D2 = kap * (tr.c[2] - sb.c[tt][2]);
    mixed_pair<K, PHC, CK, true>(prm, rule, sb, tt, tr, D0, D1, D2, fma(D2, D2, fma(D1, D1, D0 * D0)), ab[0], ab[1],
                                 ab[2], ab[3]);
}

// Packed mixed precision in wavenumber-scaled units with the two-orbit rule (orbit.cuh).  The trial points of
// one vertex, one of each orbit, travel together in f32x2 operations, so an orbit's weight is applied to its
// half of the sums at the end of the pair, and the offset products need one dot product per pair of vertices:
//   s = r'^2 - r_c'^2 = A_q + B_p - 2 g_p g_q e_i . f_j,
//   A_q = g_q^2 |f_j|^2 + 2 g_q D . f_j,  B_p = g_p^2 |e_i|^2 - 2 g_p D . e_i.
// 1/r' by rsqrt.approx.  The phase offset theta = r' - r_c' would lose its accuracy in the subtraction (r' is
// good to 1e-7 r', up to 2e-6 at r' = 20); one Newton step on theta^2 + 2 r_c' theta = s from it,
//   theta = t + (s - t (t + 2 r_c')) / (2 r'),  t = r'^2 (1 / r') - r_c',
// restores it to rounding of theta itself, in four packed operations in place of the reciprocal
// 1 / (r' + r_c') of the special-function unit, which with the square root and the cosine bounded the sweep
// beside the FMA pipe.  (The code carries -theta and -s / 2: f32x2 operations have no negation.)
// Per point pair, with g = w (d'.n) / r'^2 and the shared factors h1 = cos / r' + sin, h2 = cos - sin / r', the
// double-layer part of an entry is -g h1 + i g h2 (times kappa^2); the two entries differ only in (d'.n).
//
// Per element pair: the centroid offset D and |D|^2 in FP64 (r_c' for the phase), FP32 copies for the
// point-pair terms; elements whose centroids are farther apart than prm.near_r cannot share a vertex, so the
// vertex test runs only for closer pairs, and of those the near ones difference the coordinates (near_mr2, dp0.cuh);
// the pair phase exp(i r_c') by phase_reduced32.  The FP32 sums of the
// first test orbit are scaled by w_a / w_b when the second begins, and everything is converted to FP64 once,
// times w_b.
// Bound by the FMA pipe: 68 % of its cycles, the special-function unit 49 %, issue 55 %, the first stall its throttle.
// Combined field, 32768 elements, k = 10: 22.02 -> 21.09 ms (against pairs of neighbouring trial points and the
// reciprocal), error 1.4e-8 either way.
// CK: a complex wavenumber k = kr + i ki in units of 1/kr: the amplitude e^{-beta r'} (beta = ki / kr)
// split like the phase, e^{-beta theta} per point pair by __expf and e^{-beta r_c'} per element pair by
// exp_neg_reduced; the double-layer factor (i k r - 1) = -(1 + beta r') + i r' turns 1 / r' into
// 1 / r' + beta in h1 and h2.
template <int K, int PHC, bool STRIPE = false, bool CK = false>
__device__ __forceinline__ void regular_dp0_mixed_sym_tile(const RegParams &prm, const QuadRule &rule,
                                                         int64_t tile_x, int64_t t0, int rows, TestBlock32q &sb) {
    static_assert(!CK || SymTraits<K>::helm, "complex wavenumber: the Helmholtz kernels");
    const double kap = mixed_kappa<K>(prm), g0d = mixed_g(rule, 0), g1d = mixed_g(rule, 1);
    const int tcount = (int)min((int64_t)rows, prm.ntest - t0);
    for (int idx = threadIdx.x; idx < tcount; idx += blockDim.x) {
        const int64_t t = prm.tsup[t0 + idx];
        Geom g;
        load_geom(prm.tg, prm.tne, t, prm.tnm ? (double)prm.tnm[t] : 1.0, g);
        double e[3][3], m2 = 0.0;
        orbit_offsets(g, e);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int d = 0; d < 3; ++d) sb.e[idx][i][d] = (float)(kap * e[i][d]);
            const double ee = odot(e[i], e[i]), m = kap * kap * ee;
            m2 = fmax(m2, ee);
            sb.hge[idx][0][i] = (float)(-0.5 * g0d * g0d * m);
            sb.hge[idx][1][i] = (float)(-0.5 * g1d * g1d * m);
            sb.c[idx][i] = __ldg(prm.tg + (22 + i) * prm.tne + t);
            sb.v[idx][i] = __ldg(prm.tel + 3 * t + i);
        }
        sb.n[idx] = make_float4((float)g.n[0], (float)g.n[1], (float)g.n[2], (float)(MIXED_NEAR * kap * sqrt(m2)));
        sb.ie[idx] = g.ie;
    }
    __syncthreads();

    const int64_t si = tile_x * DP0_THREADS + threadIdx.x;
    if (si < prm.ntrial && t0 <= si) {
        MixedTrial tr;
        load_trial_mixed<K>(prm, rule, si, tr);
        // centroid distances below near_r (scaled) may belong to vertex-sharing pairs
        const double near2 = prm.near_r > 0.0 ? (kap * prm.near_r) * (kap * prm.near_r) : 1e300;
        sb.srad[threadIdx.x] = tr.rad;
        for (int tt = 0; tt < tcount; ++tt) {
            const int64_t row = t0 + tt;
            if (row > si) break;
            const double D0 = kap * (tr.c[0] - sb.c[tt][0]), D1 = kap * (tr.c[1] - sb.c[tt][1]),
                         D2 = kap * (tr.c[2] - sb.c[tt][2]);
            const double rc2 = fma(D2, D2, fma(D1, D1, D0 * D0));
            const bool adj = row == si || (prm.grids_identical && rc2 <= near2 &&
                                           shares_vertex(sb.v[tt], tr.v[0], tr.v[1], tr.v[2]));
            double a_re = 0.0, a_im = 0.0, b_re = 0.0, b_im = 0.0;  // A_ij, A_ji
            if (!adj) {
                mixed_pair<K, PHC, CK, false>(prm, rule, sb, tt, tr, D0, D1, D2, rc2, a_re, a_im, b_re, b_im);
                if (rc2 <= near2) {
                    const float rs = sb.n[tt].w + sb.srad[threadIdx.x];
                    if ((float)rc2 < rs * rs) {  // in place of what the expanded square gave
                        double ab[4];
                        mixed_near_pair<K, PHC, CK>(prm, rule, sb, tt, si, ab);
                        a_re = ab[0];
                        a_im = ab[1];
                        b_re = ab[2];
                        b_im = ab[3];
                    }
                }
            }
            store_pair<STRIPE>(prm, row, si, adj, a_re, a_im, b_re, b_im);
        }
    }
    __syncthreads();
}

}  // namespace bc
