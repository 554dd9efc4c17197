// FP64 sums over the 36 point pairs of two separated elements with the two-orbit rule (orbit.cuh), shared by
// the P1 and RWG sweeps (p1.cuh, rwg.cuh).
//
// With D = c_s - c_t the centroid offset, x_p = c_t + g_p e_i and y_q = c_s + g_q f_j:
//   r^2 = r_c^2 + (g_q^2 |f_j|^2 + 2 g_q D . f_j) + (g_p^2 |e_i|^2 - 2 g_p D . e_i) - 2 g_p g_q e_i . f_j,
// the two brackets once per point and e_i . f_j once per pair of vertices: 2 FP64 operations per point pair
// and 50 per element pair, where differencing the coordinates takes 6.  Points lie within rho R, rho = 0.725, of
// their centroid, so beyond r_c = R_t + R_s (the two elements' own centroid-to-vertex distances) a
// distance is at least 0.27 r_c and the expanded square keeps its accuracy to a few units in the last place
// times (r_c / r)^2; closer pairs, which share no vertex but nearly touch, difference the coordinates.
// The normal terms of the double layers are linear in the same vectors.
//
// Moments with the linear shape functions: lambda_a = d_o + c_o [a = j] over w_o at the points of orbit o
// (c_o = w_o g_o, d_o = w_o (1 - g_o) / 3), so the trial sums T_b = sum_q w_q lambda_b K need the three
// values and the sum of each orbit (12 additions or FMAs per six values and component instead of 18),
// and the test sums likewise.
//
// exp(ikr) = exp(ik r_c) exp(ik (r - r_c)), |r - r_c| <= rho (R_t + R_s): the second factor by the
// polynomials of the offset class (fastmath.cuh); a complex wavenumber's amplitude exp(-Im k r) and modified
// Helmholtz's exp(-w r) split the same way.  The first factor multiplies the pair's block.  Class 0 factors
// nothing.
#pragma once

#include "orbit.cuh"

namespace bc {

// Kernel families.
constexpr int FAM_LAPLACE = 0, FAM_HELM = 1, FAM_MODHELM = 2;
template <int K>
constexpr int kernel_family() {
    return K <= BEMPPCUDA_LAPLACE_ADLP ? FAM_LAPLACE
           : (K >= BEMPPCUDA_MODHELM_SLP && K <= BEMPPCUDA_MODHELM_ADLP) ? FAM_MODHELM
                                                                         : FAM_HELM;
}

struct OrbitConsts {
    double g[2], gg[2], c[2], d[2], w[2], dc[2];  // dc = d / c
};

inline OrbitConsts orbit_consts(const OrbitRule &r) {
    OrbitConsts o;
    for (int k = 0; k < 2; ++k) {
        o.g[k] = r.g[k];
        o.gg[k] = r.g[k] * r.g[k];
        o.w[k] = r.w[k];
        o.c[k] = r.w[k] * r.g[k];
        o.d[k] = r.w[k] * (1.0 - r.g[k]) / 3.0;
        o.dc[k] = o.d[k] / o.c[k];
    }
    return o;
}

__device__ __forceinline__ double odot(const double a[3], const double b[3]) {
    return fma(a[2], b[2], fma(a[1], b[1], a[0] * b[0]));
}

// Vertex offsets e_j = v_j - c of an element from its Jacobian columns.
__device__ __forceinline__ void orbit_offsets(const Geom &g, double e[3][3]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        e[0][d] = -(g.j0[d] + g.j1[d]) / 3.0;
        e[1][d] = e[0][d] + g.j0[d];
        e[2][d] = e[0][d] + g.j1[d];
    }
}

// Pairs with r_c < ORBIT_NEAR (R_t + R_s) difference their coordinates (each element's own R: with the grid's largest, or
// at 1.5, enough ordinary pairs took the branch to cost 4 % in divergence).
constexpr double ORBIT_NEAR = 1.0;

// A test element in shared memory.
struct OrbitTest {
    double c[3];
    double e[3][3];
    double ge[2][3];  // g_o^2 |e_j|^2
    double radius;    // ORBIT_NEAR R
};

__device__ __forceinline__ void stage_orbit(const double *__restrict__ geom, int64_t ne, int64_t t, const Geom &g,
                                            const OrbitConsts &oc, OrbitTest &o) {
    double e[3][3];
    orbit_offsets(g, e);
    double r2 = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        o.c[j] = __ldg(geom + (22 + j) * ne + t);
        const double m = odot(e[j], e[j]);
        r2 = fmax(r2, m);
        o.ge[0][j] = oc.gg[0] * m;
        o.ge[1][j] = oc.gg[1] * m;
#pragma unroll
        for (int d = 0; d < 3; ++d) o.e[j][d] = e[j][d];
    }
    o.radius = ORBIT_NEAR * sqrt(r2);
}

// OrbitTrial::ld is inline assembly that names no memory (a "memory" clobber on every load would hold back the
// scheduling of the sums), so the order of a thread's stores to its column and its loads is stated here: the fence comes
// between the loads of one element and the stores of the next, and between the last store and the first load.
__device__ __forceinline__ void orbit_fence() { asm volatile("" ::: "memory"); }

// A thread's trial element, parked in shared memory (field-major, one column per thread): the sums over the point
// pairs want the registers, and a field is read at most once per test vertex.  Loads are volatile so that they
// stay inside the loop over the test elements (orbit_fence before the first).
constexpr int OT_C = 0, OT_F = 3, OT_FF = 9, OT_N = 12, OT_IE = 15, OT_RAD = 16, OT_FIELDS = 17;

template <int THREADS>
struct OrbitTrial {
    uint32_t at;  // shared-memory address of field 0 of this thread
    __device__ __forceinline__ double ld(int k) const {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at + (uint32_t)(8 * THREADS * k)));
        return v;
    }
    // an integer field (a dof number) stored with __longlong_as_double
    __device__ __forceinline__ int64_t li(int k) const { return __double_as_longlong(ld(k)); }
    __device__ __forceinline__ void f(double f0[3], double f1[3]) const {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            f0[d] = ld(OT_F + d);
            f1[d] = ld(OT_F + 3 + d);
        }
    }
    __device__ __forceinline__ void n(double v[3]) const {
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = ld(OT_N + d);
    }
};

// Centroid, two vertex offsets (f_2 = -f_0 - f_1), |f_j|^2, normal and area of the trial element; `park` is
// [fields][THREADS].
template <int THREADS>
__device__ __forceinline__ OrbitTrial<THREADS> park_orbit_trial(const double *__restrict__ geom, int64_t ne, int64_t s,
                                                                const Geom &g, double *park) {
    orbit_fence();
    double f[3][3];
    orbit_offsets(g, f);
    double *o = park + threadIdx.x;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        o[(OT_C + d) * THREADS] = __ldg(geom + (22 + d) * ne + s);
        o[(OT_F + d) * THREADS] = f[0][d];
        o[(OT_F + 3 + d) * THREADS] = f[1][d];
        o[(OT_FF + d) * THREADS] = odot(f[d], f[d]);
        o[(OT_N + d) * THREADS] = g.n[d];
    }
    o[OT_IE * THREADS] = g.ie;
    o[OT_RAD * THREADS] = ORBIT_NEAR * sqrt(fmax(odot(f[0], f[0]), fmax(odot(f[1], f[1]), odot(f[2], f[2]))));
    return {(uint32_t)__cvta_generic_to_shared(o)};
}

// The pair's centroid offset, distance and the phase / amplitude exponents at r_c (0 in class 0).
struct OrbitPair {
    double D[3], rc2, krc, kirc;
    bool far;
    double A[2][3];  // g_q^2 |f_j|^2 + 2 g_q D . f_j
};

template <int FAM, bool CK, int CLS, class TRIAL>
__device__ __forceinline__ void orbit_pair(const OrbitTest &t, const TRIAL &s, const OrbitConsts &oc,
                                           double kr, double ki, OrbitPair &p) {
#pragma unroll
    for (int d = 0; d < 3; ++d) p.D[d] = s.ld(OT_C + d) - t.c[d];
    p.rc2 = odot(p.D, p.D);
    const double near = t.radius + s.ld(OT_RAD);
    p.far = p.rc2 >= near * near;
    p.krc = p.kirc = 0.0;
    if (CLS > 0 && FAM != FAM_LAPLACE) {
        const double rc = dist64(p.rc2);  // elements of two grids may share a centroid
        p.krc = kr * rc;
        if (CK) p.kirc = ki * rc;
    }
    double f0[3], f1[3];
    s.f(f0, f1);
    const double a0 = odot(p.D, f0), a1 = odot(p.D, f1);
    const double a[3] = {a0, a1, -(a0 + a1)};
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
        for (int j = 0; j < 3; ++j) p.A[o][j] = fma(2.0 * oc.g[o], a[j], oc.gg[o] * s.ld(OT_FF + j));
}

// Squared distances r2[3 oq + j] of the test point (orbit op, vertex offset e) and the six trial points;
// E_j = e . f_j, De = D . e.  NEAR differences the coordinates: a branch per pair around two copies of the sums
// (a branch per test point cost the hypersingular operator 7 % at 8192 elements).
template <bool NEAR, class TRIAL>
__device__ __forceinline__ void orbit_r2(const OrbitPair &p, const TRIAL &s, const OrbitConsts &oc, int op,
                                         const double e[3], double ge, double De, const double E[3], double r2[6]) {
    if constexpr (!NEAR) {
        const double b = p.rc2 + fma(-2.0 * oc.g[op], De, ge);
#pragma unroll
        for (int q = 0; q < 6; ++q)
            r2[q] = fma(-2.0 * oc.g[op] * oc.g[q / 3], E[q % 3], p.A[q / 3][q % 3] + b);
    } else {
        double x[3], f0[3], f1[3];
        s.f(f0, f1);
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = fma(-oc.g[op], e[d], p.D[d]);
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            double m = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double f = q % 3 == 0 ? f0[d] : q % 3 == 1 ? f1[d] : -(f0[d] + f1[d]);
                const double v = fma(oc.g[q / 3], f, x[d]);
                m = fma(v, v, m);
            }
            r2[q] = m;
        }
    }
}

// Kernel value without 1 / (4 pi) and the factor at r_c: G = e^{ikr} / r (GRAD false) or
// H = (ikr - 1) e^{ikr} / r^3 (GRAD true).
template <bool GRAD, int FAM, bool CK, int CLS>
__device__ __forceinline__ void orbit_kernel(double r2, double kr, double ki, const OrbitPair &p, double &re,
                                             double &im) {
    const double rinv = rsqrt64(r2);
    im = 0.0;
    if constexpr (FAM == FAM_LAPLACE) {
        re = GRAD ? -rinv * rinv * rinv : rinv;
    } else if constexpr (FAM == FAM_MODHELM) {
        const double r = r2 * rinv, f = rinv * exp_off64<CLS>(fma(-kr, r, p.krc));
        re = GRAD ? -f * rinv * rinv * fma(kr, r, 1.0) : f;
    } else {
        const double r = r2 * rinv;
        double sn, cs;
        sincos_off64<CLS>(fma(kr, r, -p.krc), &sn, &cs);
        double f = GRAD ? rinv * rinv : rinv;
        if (CK) f *= exp_off64<CLS>(fma(-ki, r, p.kirc));
        if (GRAD) {
            const double rk = CK ? rinv + ki : rinv;
            re = -f * fma(rk, cs, kr * sn);
            im = f * fma(kr, cs, -rk * sn);
        } else {
            re = f * cs;
            im = f * sn;
        }
    }
}

// The factor at r_c that multiplies the pair's block: e^{ik r_c} (CLS > 0).
template <int FAM, bool CK, int CLS>
__device__ __forceinline__ void orbit_phase(const OrbitPair &p, double &c, double &s) {
    c = 1.0;
    s = 0.0;
    if constexpr (CLS > 0 && FAM == FAM_HELM) {
        sincos_cw64(p.krc, &s, &c);
        if (CK) {
            const double a = exp(-p.kirc);
            c *= a;
            s *= a;
        }
    } else if constexpr (CLS > 0 && FAM == FAM_MODHELM) {
        c = exp(-p.krc);
    }
}

// Rows of a block move up by one: the loop over the test vertices writes the last row, and after three steps row
// i holds vertex i (register moves in place of an index that would send the block to memory).
template <int NT, int NS, bool CPLX>
__device__ __forceinline__ void orbit_rotate(double (&re)[NT][NS], double (&im)[NT][NS]) {
#pragma unroll
    for (int i = 0; i + 1 < NT; ++i)
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            re[i][j] = re[i + 1][j];
            if (CPLX) im[i][j] = im[i + 1][j];
        }
#pragma unroll
    for (int j = 0; j < NS; ++j) re[NT - 1][j] = im[NT - 1][j] = 0.0;
}

// Moments L_ij = sum_pq w_p w_q phi_i(p) phi_j(q) K (linear functions, or the constant one with NT / NS = 1).
template <bool GRAD, int FAM, bool CK, int CLS, int NT, int NS, bool NEAR, class TRIAL>
__device__ __forceinline__ void orbit_moments_in(const OrbitTest &t, const TRIAL &s, const OrbitPair &p,
                                              const OrbitConsts &oc, double kr, double ki, double (&lre)[NT][NS],
                                              double (&lim)[NT][NS]) {
    constexpr bool CPLX = FAM == FAM_HELM;
    double bre[NS], bim[NS];  // what every test function gets: sum_p d_p T_j
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        bre[j] = bim[j] = 0.0;
#pragma unroll
        for (int i = 0; i < NT; ++i) lre[i][j] = lim[i][j] = 0.0;
    }
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        const double e[3] = {t.e[i][0], t.e[i][1], t.e[i][2]};
        double f0[3], f1[3];
        s.f(f0, f1);
        const double De = odot(p.D, e), E0 = odot(e, f0), E1 = odot(e, f1);
        const double E[3] = {E0, E1, -(E0 + E1)};
        orbit_rotate<NT, NS, CPLX>(lre, lim);
#pragma unroll 1
        for (int op = 0; op < 2; ++op) {
            double r2[6];
            orbit_r2<NEAR>(p, s, oc, op, e, t.ge[op][i], De, E, r2);
            double tre[3], tim[3], sre[2], sim[2];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                double re, im;
                orbit_kernel<GRAD, FAM, CK, CLS>(r2[q], kr, ki, p, re, im);
                const int o = q / 3, j = q % 3;
                sre[o] = j == 0 ? re : sre[o] + re;
                if (CPLX) sim[o] = j == 0 ? im : sim[o] + im;
                if (NS == 3) {
                    tre[j] = o == 0 ? oc.c[0] * re : fma(oc.c[1], re, tre[j]);
                    if (CPLX) tim[j] = o == 0 ? oc.c[0] * im : fma(oc.c[1], im, tim[j]);
                }
            }
            const double *d = NS == 3 ? oc.d : oc.w;
            const double ore = fma(d[1], sre[1], d[0] * sre[0]), oim = CPLX ? fma(d[1], sim[1], d[0] * sim[0]) : 0.0;
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const double Tr = NS == 3 ? tre[j] + ore : ore, Ti = NS == 3 && CPLX ? tim[j] + oim : oim;
                const double dp = NT == 3 ? oc.d[op] : oc.w[op];
                bre[j] = fma(dp, Tr, bre[j]);
                if (CPLX) bim[j] = fma(dp, Ti, bim[j]);
                if (NT == 3) {
                    lre[NT - 1][j] = fma(oc.c[op], Tr, lre[NT - 1][j]);
                    if (CPLX) lim[NT - 1][j] = fma(oc.c[op], Ti, lim[NT - 1][j]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            lre[i][j] = NT == 3 ? lre[i][j] + bre[j] : bre[j];
            lim[i][j] = !CPLX ? 0.0 : NT == 3 ? lim[i][j] + bim[j] : bim[j];
        }
}

template <bool GRAD, int FAM, bool CK, int CLS, int NT, int NS, class TRIAL>
__device__ __forceinline__ void orbit_moments(const OrbitTest &t, const TRIAL &s, const OrbitPair &p,
                                              const OrbitConsts &oc, double kr, double ki, double (&lre)[NT][NS],
                                              double (&lim)[NT][NS]) {
    if (p.far)
        orbit_moments_in<GRAD, FAM, CK, CLS, NT, NS, false>(t, s, p, oc, kr, ki, lre, lim);
    else
        orbit_moments_in<GRAD, FAM, CK, CLS, NT, NS, true>(t, s, p, oc, kr, ki, lre, lim);
}

// Double-layer moments of H: U_ij with the trial-normal factor (y_q - x_p) . n_s = (D - g_p e_i) . n_s, one
// value per test point (the double layer of the pair), V_ij with (x_p - y_q) . n_t = -(D + g_q f_j) . n_t,
// one value per trial point (its adjoint double layer).
template <bool WITH_U, bool WITH_V, int FAM, bool CK, int CLS, int NT, int NS, bool NEAR, class TRIAL>
__device__ __forceinline__ void orbit_double_in(const OrbitTest &t, const double tn[3], const TRIAL &s,
                                             const OrbitPair &p, const OrbitConsts &oc, double kr,
                                             double ki, double (&ure)[NT][NS], double (&uim)[NT][NS],
                                             double (&vre)[NT][NS], double (&vim)[NT][NS]) {
    constexpr bool CPLX = FAM == FAM_HELM;
    double bur[NS], bui[NS], bvr[NS], bvi[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        bur[j] = bui[j] = bvr[j] = bvi[j] = 0.0;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            if (WITH_U) ure[i][j] = uim[i][j] = 0.0;
            if (WITH_V) vre[i][j] = vim[i][j] = 0.0;
        }
    }
    double sn[3] = {0.0, 0.0, 0.0}, Dn = 0.0;
    if (WITH_U) {
        s.n(sn);
        Dn = odot(p.D, sn);
    }
    double m[6];  // (x - y_q) . n_t times c_o (NS = 3) or w_o
    if (WITH_V) {
        double v0[3], v1[3];
        s.f(v0, v1);
        const double Dt = odot(p.D, tn), f0 = odot(v0, tn), f1 = odot(v1, tn);
        const double f[3] = {f0, f1, -(f0 + f1)};
#pragma unroll
        for (int q = 0; q < 6; ++q)
            m[q] = -(NS == 3 ? oc.c[q / 3] : oc.w[q / 3]) * fma(oc.g[q / 3], f[q % 3], Dt);
    }
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        const double e[3] = {t.e[i][0], t.e[i][1], t.e[i][2]};
        double f0[3], f1[3];
        s.f(f0, f1);
        const double De = odot(p.D, e), E0 = odot(e, f0), E1 = odot(e, f1);
        const double E[3] = {E0, E1, -(E0 + E1)};
        if (WITH_U) orbit_rotate<NT, NS, CPLX>(ure, uim);
        if (WITH_V) orbit_rotate<NT, NS, CPLX>(vre, vim);
        if (WITH_U) s.n(sn);
        const double en = WITH_U ? odot(e, sn) : 0.0;
#pragma unroll 1
        for (int op = 0; op < 2; ++op) {
            double r2[6];
            orbit_r2<NEAR>(p, s, oc, op, e, t.ge[op][i], De, E, r2);
            double tre[3], tim[3], wre[3], wim[3], sre[2], sim[2], xre[2], xim[2];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                double re, im;
                orbit_kernel<true, FAM, CK, CLS>(r2[q], kr, ki, p, re, im);
                const int o = q / 3, j = q % 3;
                if (WITH_U) {
                    sre[o] = j == 0 ? re : sre[o] + re;
                    if (CPLX) sim[o] = j == 0 ? im : sim[o] + im;
                    if (NS == 3) {
                        tre[j] = o == 0 ? oc.c[0] * re : fma(oc.c[1], re, tre[j]);
                        if (CPLX) tim[j] = o == 0 ? oc.c[0] * im : fma(oc.c[1], im, tim[j]);
                    }
                }
                if (WITH_V) {
                    xre[o] = j == 0 ? m[q] * re : fma(m[q], re, xre[o]);
                    if (CPLX) xim[o] = j == 0 ? m[q] * im : fma(m[q], im, xim[o]);
                    if (NS == 3) {
                        wre[j] = o == 0 ? m[q] * re : fma(m[q], re, wre[j]);
                        if (CPLX) wim[j] = o == 0 ? m[q] * im : fma(m[q], im, wim[j]);
                    }
                }
            }
            const double dp = NT == 3 ? oc.d[op] : oc.w[op], cp = oc.c[op];
            if (WITH_U) {
                const double xn = fma(-oc.g[op], en, Dn), dx = dp * xn, cx = cp * xn;
                const double *d = NS == 3 ? oc.d : oc.w;
                const double ore = fma(d[1], sre[1], d[0] * sre[0]);
                const double oim = CPLX ? fma(d[1], sim[1], d[0] * sim[0]) : 0.0;
#pragma unroll
                for (int j = 0; j < NS; ++j) {
                    const double Tr = NS == 3 ? tre[j] + ore : ore, Ti = NS == 3 && CPLX ? tim[j] + oim : oim;
                    bur[j] = fma(dx, Tr, bur[j]);
                    if (CPLX) bui[j] = fma(dx, Ti, bui[j]);
                    if (NT == 3) {
                        ure[NT - 1][j] = fma(cx, Tr, ure[NT - 1][j]);
                        if (CPLX) uim[NT - 1][j] = fma(cx, Ti, uim[NT - 1][j]);
                    }
                }
            }
            if (WITH_V) {
                const double ore = NS == 3 ? fma(oc.dc[1], xre[1], oc.dc[0] * xre[0]) : xre[0] + xre[1];
                const double oim = !CPLX ? 0.0 : NS == 3 ? fma(oc.dc[1], xim[1], oc.dc[0] * xim[0]) : xim[0] + xim[1];
#pragma unroll
                for (int j = 0; j < NS; ++j) {
                    const double Tr = NS == 3 ? wre[j] + ore : ore, Ti = NS == 3 && CPLX ? wim[j] + oim : oim;
                    bvr[j] = fma(dp, Tr, bvr[j]);
                    if (CPLX) bvi[j] = fma(dp, Ti, bvi[j]);
                    if (NT == 3) {
                        vre[NT - 1][j] = fma(cp, Tr, vre[NT - 1][j]);
                        if (CPLX) vim[NT - 1][j] = fma(cp, Ti, vim[NT - 1][j]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            if (WITH_U) {
                ure[i][j] = NT == 3 ? ure[i][j] + bur[j] : bur[j];
                uim[i][j] = !CPLX ? 0.0 : NT == 3 ? uim[i][j] + bui[j] : bui[j];
            }
            if (WITH_V) {
                vre[i][j] = NT == 3 ? vre[i][j] + bvr[j] : bvr[j];
                vim[i][j] = !CPLX ? 0.0 : NT == 3 ? vim[i][j] + bvi[j] : bvi[j];
            }
        }
}

template <bool WITH_U, bool WITH_V, int FAM, bool CK, int CLS, int NT, int NS, class TRIAL>
__device__ __forceinline__ void orbit_double(const OrbitTest &t, const double tn[3], const TRIAL &s,
                                             const OrbitPair &p, const OrbitConsts &oc, double kr, double ki,
                                             double (&ure)[NT][NS], double (&uim)[NT][NS], double (&vre)[NT][NS],
                                             double (&vim)[NT][NS]) {
    if (p.far)
        orbit_double_in<WITH_U, WITH_V, FAM, CK, CLS, NT, NS, false>(t, tn, s, p, oc, kr, ki, ure, uim, vre, vim);
    else
        orbit_double_in<WITH_U, WITH_V, FAM, CK, CLS, NT, NS, true>(t, tn, s, p, oc, kr, ki, ure, uim, vre, vim);
}

}  // namespace bc
