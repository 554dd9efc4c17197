// Touching element pairs with the order-4 Sauter-Schwab rules themselves, where the kernels of singular.cu read
// the rules as flat tables of points (singular_assembler.py:69-448, numba_kernels.py:1471-2147).
//
// Every region map of the three rules (coincident, shared edge, shared vertex; duffy_galerkin.py:25-226)
// places both points at xi times a direction from a shared vertex V0,
//   x = V0 + xi (a1 T1 + a2 T2),  y = V0 + xi (c1 S1 + c2 S2),
// T, S the edges from V0 of the test and trial element, (a, c) functions of eta1..eta3 alone.  So
// y - x = xi delta and r = xi rho with one delta, rho and 1 / rho per (region, eta): the distance and its
// root are formed once for the four Gauss points in xi, and all that depends on xi are the sums
//   Z_m = sum_k w_k xi_k^m e^{ik xi_k rho},
// since shape functions are linear in xi.  With the weight xi^3:
//   G = e^{ikr} / r:              sum xi^3 G = Z2 / rho; times shape functions of degree m in xi: Z_{2+m} / rho
//   H = (ikr - 1) e^{ikr} / r^3:  sum xi^3 H xi^n = (ik rho Z_{n+1} - Z_n) / rho^3
//   double layers                 H (y - x) . n, n = 1 + m, and delta . n_s = -(a1 T1 + a2 T2) . n_s,
//                                 delta . n_t = (c1 S1 + c2 S2) . n_t
//   magnetic field                with p_i the vertex a function vanishes at, relative to V0,
//     (x - y) . ((x - V0 - p_i) x (y - V0 - p_j)) =
//        xi^2 (p_j - p_i) . (beta x alpha) + xi (alpha - beta) . (p_i x p_j),  alpha = a_b T_b, beta = c_b S_b.
// The real families (Laplace) have constant Z_m.  The differences of coordinates carry no cancellation: V0 drops out.
//
// A group of G lanes takes a pair, each lane every G-th (region, eta) of its rule from a table in shared
// memory (written by each block from the four Gauss points); the groups' sums meet in shuffles and the
// entries are finished by the group's lanes.  G = 8 keeps 4 pairs per warp; G = 32 when there are too few
// pairs to fill the GPU.  The flat tables cost a warp 40 bytes per point and lane from L2 (a coincident pair reads
// 61 KB), which bounded those kernels together with the FP64 work this form divides by four.
// Bound by the FP64 pipe (the sine / cosine pair of each point).  Flat tables -> this form: P1 hypersingular, 8192
// elements 0.63 -> 0.26 ms; combined field on DP0, 16200 elements 0.73 -> 0.38 ms; double layer on P1, 10952 elements
// 0.89 -> 0.41 ms; electric field, 2048 elements 0.145 -> 0.075 ms; 24 problems of one batch 1.18 -> 0.65 ms; Laplace on 128 elements 36 -> 9 us.
#pragma once

#include "orbit_pair.cuh"

namespace bc {

constexpr int SD_Q = 4;                     // Gauss points per direction
constexpr int SD_E = SD_Q * SD_Q * SD_Q;    // eta points per region
constexpr int SD_SAME = 6 * SD_E, SD_EDGE = 5 * SD_E, SD_VERT = 2 * SD_E;
constexpr int SD_TAB = SD_SAME + SD_EDGE + SD_VERT;
constexpr int SD_THREADS = 128;

// Gauss points of [0, 1] and wm[m][k] = w_k xi_k^m.
struct DuffyRule {
    double x[SD_Q], w[SD_Q], wm[5][SD_Q], sum[5];
};

inline DuffyRule duffy_rule4() {
    // Gauss-Legendre nodes of order 4 on [-1, 1]: sqrt(3/7 -+ 2/7 sqrt(6/5)), weights (18 +- sqrt 30) / 36
    const double r = 2.0 / 7.0 * sqrt(6.0 / 5.0), n0 = sqrt(3.0 / 7.0 - r), n1 = sqrt(3.0 / 7.0 + r);
    const double w0 = (18.0 + sqrt(30.0)) / 36.0, w1 = (18.0 - sqrt(30.0)) / 36.0;
    DuffyRule d;
    const double n[4] = {n1, n0, -n0, -n1}, w[4] = {w1, w0, w0, w1};
    for (int k = 0; k < SD_Q; ++k) {
        d.x[k] = 0.5 * (1.0 + n[k]);
        d.w[k] = 0.5 * w[k];
    }
    for (int m = 0; m < 5; ++m) {
        d.sum[m] = 0.0;
        for (int k = 0; k < SD_Q; ++k) {
            d.wm[m][k] = (m == 0 ? d.w[k] : d.wm[m - 1][k] * d.x[k]);
            d.sum[m] += d.wm[m][k];
        }
    }
    return d;
}

struct DuffyTable {
    double a1[SD_TAB], a2[SD_TAB], c1[SD_TAB], c2[SD_TAB], w[SD_TAB];
};

// Entry idx of the table: the directions of both points (first and second coordinate on the triangle
// (0, 0), (1, 0), (1, 1), shifted to the reference triangle) and the weight with the region's Jacobian.
__device__ __forceinline__ void duffy_entry(const DuffyRule &d, int idx, DuffyTable &tab) {
    int base = 0, kind = 0;
    if (idx >= SD_SAME + SD_EDGE) {
        base = SD_SAME + SD_EDGE;
        kind = 2;
    } else if (idx >= SD_SAME) {
        base = SD_SAME;
        kind = 1;
    }
    const int region = (idx - base) / SD_E, eta = (idx - base) % SD_E;
    const double e1 = d.x[eta % SD_Q], e2 = d.x[(eta / SD_Q) % SD_Q], e3 = d.x[eta / (SD_Q * SD_Q)];
    double w = d.w[eta % SD_Q] * d.w[(eta / SD_Q) % SD_Q] * d.w[eta / (SD_Q * SD_Q)];
    const double e12 = e1 * e2, e123 = e12 * e3;
    double t1, t2, s1, s2;
    if (kind == 0) {
        w *= e1 * e1 * e2;
        const int r = region / 2;
        if (r == 0) {
            t1 = 1.0, t2 = 1.0 - e1 + e12, s1 = 1.0 - e123, s2 = 1.0 - e1;
        } else if (r == 1) {
            t1 = 1.0, t2 = e1 - e12 + e123, s1 = 1.0 - e12, s2 = e1 - e12;
        } else {
            t1 = 1.0 - e123, t2 = e1 - e123, s1 = 1.0, s2 = e1 - e12;
        }
        if (region & 1) {
            const double u = t1, v = t2;
            t1 = s1, t2 = s2, s1 = u, s2 = v;
        }
    } else if (kind == 1) {
        w *= e1 * e1 * (region == 0 ? 1.0 : e2);
        if (region == 0) {
            t1 = 1.0, t2 = e1 * e3, s1 = 1.0 - e12, s2 = e1 * (1.0 - e2);
        } else if (region == 1) {
            t1 = 1.0, t2 = e1, s1 = 1.0 - e123, s2 = e12 * (1.0 - e3);
        } else if (region == 2) {
            t1 = 1.0 - e12, t2 = e1 * (1.0 - e2), s1 = 1.0, s2 = e123;
        } else if (region == 3) {
            t1 = 1.0 - e123, t2 = e12 * (1.0 - e3), s1 = 1.0, s2 = e1;
        } else {
            t1 = 1.0 - e123, t2 = e1 * (1.0 - e2 * e3), s1 = 1.0, s2 = e12;
        }
    } else {
        w *= e2;
        t1 = 1.0, t2 = e1, s1 = e2, s2 = e2 * e3;
        if (region) {
            const double u = t1, v = t2;
            t1 = s1, t2 = s2, s1 = u, s2 = v;
        }
    }
    tab.a1[idx] = t1 - t2;
    tab.a2[idx] = t2;
    tab.c1[idx] = s1 - s2;
    tab.c2[idx] = s2;
    tab.w[idx] = w;
}

// What a kernel sums over the (region, eta) points of a pair.
constexpr int SD_G = 0;     // linear moments of G (9 values): P1 single layer, hypersingular, electric field
constexpr int SD_DP0 = 1;   // constant functions: single layer, double layer of both orders
constexpr int SD_DL = 2;    // linear moments of a double layer, of both orders of a mirrored pair
constexpr int SD_MAG = 3;   // magnetic field

// True for the point counts and table offsets of the three rules.
__device__ __forceinline__ bool duffy_known(int npts, int64_t toff, int64_t soff) {
    constexpr int64_t n0 = SD_SAME * SD_Q, n1 = SD_EDGE * SD_Q, n2 = SD_VERT * SD_Q;
    if (npts == n0) return toff == 0 && soff == 0;
    const int64_t base = npts == n1 ? n0 : n0 + 6 * n1, count = npts == n1 ? 6 : 3;
    if (npts != n1 && npts != n2) return false;
    const int64_t a = toff - base, b = soff - base;
    return a >= 0 && b >= 0 && a < count * npts && b < count * npts && a % npts == 0 && b % npts == 0;
}

// Vertex order of a pair's element: o[0] is the shared vertex V0 (the shared edge o[0], o[1]).
struct DuffyOrder {
    int o[3];
};
__device__ __forceinline__ DuffyOrder duffy_order(int kind, int64_t offset) {
    constexpr int n0 = SD_SAME * SD_Q, n1 = SD_EDGE * SD_Q, n2 = SD_VERT * SD_Q;
    if (kind == 1) {
        // edge remaps (0,1), (1,0), (1,2), (2,1), (0,2), (2,0)
        const int r = (int)((offset - n0) / n1);
        const int a = r == 0 || r == 4 ? 0 : r == 1 || r == 2 ? 1 : 2, b = r == 1 || r == 5 ? 0 : r == 0 || r == 3 ? 1 : 2;
        return {{a, b, 3 - a - b}};
    }
    if (kind == 2) {
        const int r = (int)((offset - n0 - 6 * n1) / n2);
        return {{r, r == 1 ? 0 : 1, r == 2 ? 0 : 2}};
    }
    return {{0, 1, 2}};
}
__device__ __forceinline__ int duffy_position(const DuffyOrder &o, int v) { return v == o.o[0] ? 0 : v == o.o[1] ? 1 : 2; }

// v_to - v_from of an element.
__device__ __forceinline__ void duffy_edge(const Geom &g, int from, int to, double e[3]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double a = from == 1 ? g.j0[d] : from == 2 ? g.j1[d] : 0.0;
        const double b = to == 1 ? g.j0[d] : to == 2 ? g.j1[d] : 0.0;
        e[d] = b - a;
    }
}

// The sums of one pair over the lane's share of the table.  s: SD_G nine complex moments [u][v] of
// {1, xi a1, xi a2} x {1, xi c1, xi c2}; SD_DP0 (single layer, H delta.n_s, H delta.n_t); SD_DL nine moments
// with n_s and (both) nine with n_t; SD_MAG four sums with c_b a_a, two with a, two with c.
template <int MODE>
constexpr int duffy_sums() {
    return MODE == SD_G ? 9 : MODE == SD_DP0 ? 3 : MODE == SD_DL ? 18 : 8;
}

template <int MODE, int FAM, bool CK, int CLS, bool SL, bool DL>
__device__ __forceinline__ void duffy_pair(const DuffyTable &tab, const DuffyRule &d, int begin, int end, int first,
                                           int step, const double T1[3], const double T2[3], const double S1[3],
                                           const double S2[3], const double tn[3], const double sn[3], bool own_t,
                                           bool both, double kr, double ki, double krc, double kirc,
                                           cplx (&s)[duffy_sums<MODE>()]) {
    constexpr bool CPLX = FAM == FAM_HELM;
    constexpr bool GRAD = MODE == SD_DL || MODE == SD_MAG || (MODE == SD_DP0 && DL);
    // the powers of xi that occur
    constexpr int LO = GRAD ? 1 : 2, HI = MODE == SD_G || MODE == SD_DL ? 4 : MODE == SD_MAG ? 3 : 2;
#pragma unroll
    for (int i = 0; i < duffy_sums<MODE>(); ++i) s[i] = {0.0, 0.0};
    double ns1 = 0.0, ns2 = 0.0, nt1 = 0.0, nt2 = 0.0;
    // (both points of a coincident pair lie in one plane: its normal terms are zero, not the rounding of T . n)
    if ((MODE == SD_DL || (MODE == SD_DP0 && DL)) && begin > 0) {
        ns1 = -odot(T1, sn);
        ns2 = -odot(T2, sn);
        nt1 = odot(S1, tn);
        nt2 = odot(S2, tn);
    }
#pragma unroll 1
    for (int e = begin + first; e < end; e += step) {
        const double a1 = tab.a1[e], a2 = tab.a2[e], c1 = tab.c1[e], c2 = tab.c2[e], w = tab.w[e];
        double rho2 = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double v = fma(c1, S1[i], fma(c2, S2[i], fma(-a1, T1[i], -a2 * T2[i])));
            rho2 = fma(v, v, rho2);
        }
        const double irho = rsqrt64(rho2), rho = rho2 * irho;
        cplx Z[5];
        if constexpr (FAM == FAM_LAPLACE) {
#pragma unroll
            for (int m = LO; m <= HI; ++m) Z[m] = {d.sum[m], 0.0};
        } else {
#pragma unroll
            for (int m = LO; m <= HI; ++m) Z[m] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < SD_Q; ++k) {
                const double r = d.x[k] * rho;
                if constexpr (FAM == FAM_MODHELM) {
                    const double a = exp_off64<CLS>(fma(-kr, r, krc));
#pragma unroll
                    for (int m = LO; m <= HI; ++m) Z[m].re = fma(d.wm[m][k], a, Z[m].re);
                } else {
                    double sv, cv;
                    sincos_off64<CLS>(fma(kr, r, -krc), &sv, &cv);
                    if (CK) {
                        const double a = exp_off64<CLS>(fma(-ki, r, kirc));
                        sv *= a;
                        cv *= a;
                    }
#pragma unroll
                    for (int m = LO; m <= HI; ++m) {
                        Z[m].re = fma(d.wm[m][k], cv, Z[m].re);
                        Z[m].im = fma(d.wm[m][k], sv, Z[m].im);
                    }
                }
            }
        }
        // h(n) = sum xi^{3+n} H without w / rho^3: ik rho Z_{n+1} - Z_n
        const double br = kr * rho, bi = CK ? ki * rho : 0.0, w3 = w * irho * irho * irho;
        const auto h = [&](int n) -> cplx {
            cplx v;
            if constexpr (FAM == FAM_LAPLACE) {
                v = {-Z[n].re, 0.0};
            } else if constexpr (FAM == FAM_MODHELM) {
                v = {-fma(br, Z[n + 1].re, Z[n].re), 0.0};
            } else {
                v = {-fma(br, Z[n + 1].im, Z[n].re), fma(br, Z[n + 1].re, -Z[n].im)};
                if (CK) {
                    v.re = fma(-bi, Z[n + 1].re, v.re);
                    v.im = fma(-bi, Z[n + 1].im, v.im);
                }
            }
            return v;
        };
        const auto add = [&](cplx &t, double f, const cplx &v) {
            t.re = fma(f, v.re, t.re);
            if (CPLX) t.im = fma(f, v.im, t.im);
        };
        if constexpr (MODE == SD_DP0) {
            if (SL) add(s[0], w * irho, Z[2]);
            if (DL) {
                const cplx v = h(1);
                add(s[1], w3 * fma(a1, ns1, a2 * ns2), v);
                add(s[2], w3 * fma(c1, nt1, c2 * nt2), v);
            }
        } else if constexpr (MODE == SD_MAG) {
            const cplx q2 = h(2), q1 = h(1);
            const double wa1 = w3 * a1, wa2 = w3 * a2, wc1 = w3 * c1, wc2 = w3 * c2;
            add(s[0], wa1 * c1, q2);
            add(s[1], wa1 * c2, q2);
            add(s[2], wa2 * c1, q2);
            add(s[3], wa2 * c2, q2);
            add(s[4], wa1, q1);
            add(s[5], wa2, q1);
            add(s[6], wc1, q1);
            add(s[7], wc2, q1);
        } else {
            const auto moments = [&](int at, double f, const cplx &m0, const cplx &m1, const cplx &m2) {
                const double f1 = f * a1, f2 = f * a2;
                add(s[at], f, m0);
                add(s[at + 1], f * c1, m1);
                add(s[at + 2], f * c2, m1);
                add(s[at + 3], f1, m1);
                add(s[at + 4], f1 * c1, m2);
                add(s[at + 5], f1 * c2, m2);
                add(s[at + 6], f2, m1);
                add(s[at + 7], f2 * c1, m2);
                add(s[at + 8], f2 * c2, m2);
            };
            if constexpr (MODE == SD_G) {
                moments(0, w * irho, Z[2], Z[3], Z[4]);
            } else {
                const double ds = w3 * fma(a1, ns1, a2 * ns2), dt = w3 * fma(c1, nt1, c2 * nt2);
                const cplx h1 = h(1), h2 = h(2), h3 = h(3);
                moments(0, own_t ? dt : ds, h1, h2, h3);
                if (both) moments(9, own_t ? ds : dt, h1, h2, h3);
            }
        }
    }
}

// Linear moments of the pair in the elements' own vertex order: position p = 0 has 1 - u1 - u2.
__device__ __forceinline__ cplx duffy_linear(const double2 *m, int pi, int pj) {
    const auto row = [&](int i) -> cplx {
        const double2 m0 = m[3 * i], m1 = m[3 * i + 1], m2 = m[3 * i + 2];
        if (pj == 1) return {m1.x, m1.y};
        if (pj == 2) return {m2.x, m2.y};
        return {m0.x - m1.x - m2.x, m0.y - m1.y - m2.y};
    };
    if (pi > 0) return row(pi);
    const cplx a = row(0), b = row(1), c = row(2);
    return {a.re - b.re - c.re, a.im - b.im - c.im};
}

template <int ASM, int K, int NS>
constexpr int duffy_mode() {
    if (ASM == BEMPPCUDA_ASM_MFIE) return SD_MAG;
    if (ASM != BEMPPCUDA_ASM_SCALAR) return SD_G;
    if (NS == 1) return SD_DP0;
    return K == BEMPPCUDA_LAPLACE_SLP || K == BEMPPCUDA_HELMHOLTZ_SLP || K == BEMPPCUDA_MODHELM_SLP ? SD_G : SD_DL;
}

// What one group needs besides the tables.
struct DuffyTarget {
    const double *g;
    int64_t ne;
    const int32_t *tnm, *snm;
    double p[4];
    bool is_complex;
    void *values, *dense;
    int64_t ld;
    const uint32_t *tl2g, *sl2g;  // null: dof = element, multiplier 1 (DP0 of a batch)
    const double *tmult, *smult;
    double diag_shift;
    bool mirror;  // vertex-adjacent pairs of one space: the pair t < s adds both orders
};

// Pair k by the G lanes of a group (every lane of the warp calls; valid: the group has a pair).
template <int ASM, int K, int N, int CLS, bool CK, int G>
__device__ __forceinline__ void duffy_group(const DuffyTarget &prm, const DuffyTable &tab, const DuffyRule &d,
                                            double2 *scratch, int64_t k, int64_t t, int64_t s, int64_t toff,
                                            int64_t soff, int npts, bool valid) {
    constexpr int MODE = duffy_mode<ASM, K, N>(), FAM = kernel_family<K>(), NV = duffy_sums<MODE>();
    constexpr bool MAXWELL = ASM == BEMPPCUDA_ASM_EFIE || ASM == BEMPPCUDA_ASM_MFIE;
    constexpr bool COMBINED = K == BEMPPCUDA_HELMHOLTZ_COMBINED;
    constexpr bool SL = COMBINED || K == BEMPPCUDA_LAPLACE_SLP || K == BEMPPCUDA_HELMHOLTZ_SLP || K == BEMPPCUDA_MODHELM_SLP;
    constexpr bool AD = K == BEMPPCUDA_LAPLACE_ADLP || K == BEMPPCUDA_HELMHOLTZ_ADLP || K == BEMPPCUDA_MODHELM_ADLP;
    constexpr bool DL = COMBINED || !SL;
    const int lane = threadIdx.x % G;
    const int kind = npts == SD_SAME * SD_Q ? 0 : npts == SD_EDGE * SD_Q ? 1 : 2;
    const bool mirror = prm.mirror && !prm.values && kind == 2;
    if (mirror && t > s) valid = false;
    // the magnetic field of a coincident pair is zero (all its vectors lie in one plane), where the rounding of its sums,
    // each of them large, would be 5e-14 of the matrix
    if (ASM == BEMPPCUDA_ASM_MFIE && kind == 0) valid = false;
    const double kr = prm.p[0], ki = CK ? prm.p[1] : 0.0;
    Geom gt, gs;
    DuffyOrder ot = {}, os = {};
    double T1[3], T2[3], S1[3], S2[3], krc = 0.0, kirc = 0.0;
    cplx sum[NV];
    if (valid) {
        load_geom(prm.g, prm.ne, t, !MAXWELL && prm.tnm ? (double)prm.tnm[t] : 1.0, gt);
        load_geom(prm.g, prm.ne, s, !MAXWELL && prm.snm ? (double)prm.snm[s] : 1.0, gs);
        ot = duffy_order(kind, toff);
        os = duffy_order(kind, soff);
        duffy_edge(gt, ot.o[0], ot.o[1], T1);
        duffy_edge(gt, ot.o[0], ot.o[2], T2);
        duffy_edge(gs, os.o[0], os.o[1], S1);
        duffy_edge(gs, os.o[0], os.o[2], S2);
        if (CLS > 0 && FAM != FAM_LAPLACE) {
            double D[3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
                D[i] = __ldg(prm.g + (22 + i) * prm.ne + s) - __ldg(prm.g + (22 + i) * prm.ne + t);
            const double rc = sqrt(odot(D, D));
            krc = kr * rc;
            if (CK) kirc = ki * rc;
        }
        const int begin = kind == 0 ? 0 : kind == 1 ? SD_SAME : SD_SAME + SD_EDGE;
        const int end = begin + (kind == 0 ? SD_SAME : kind == 1 ? SD_EDGE : SD_VERT);
        duffy_pair<MODE, FAM, CK, CLS, SL, DL>(tab, d, begin, end, lane, G, T1, T2, S1, S2, gt.n, gs.n, AD, mirror, kr,
                                               ki, krc, kirc, sum);
    } else {
#pragma unroll
        for (int i = 0; i < NV; ++i) sum[i] = {0.0, 0.0};
    }
    // the group's totals, in shared memory
#pragma unroll
    for (int i = 0; i < NV; ++i) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            sum[i].re += __shfl_xor_sync(0xffffffffu, sum[i].re, o);
            if (FAM == FAM_HELM) sum[i].im += __shfl_xor_sync(0xffffffffu, sum[i].im, o);
        }
        if (lane == i % G) scratch[i] = make_double2(sum[i].re, sum[i].im);
    }
    __syncwarp();
    if (!valid) return;
    OrbitPair ph;
    ph.krc = krc;
    ph.kirc = kirc;
    double pc, ps;
    orbit_phase<FAM, CK, CLS>(ph, pc, ps);
    // (re, im) of an entry times the phase, added to the matrix or the pair's values
    const auto emit = [&](int i, int j, cplx v, bool reversed) {
        if (FAM == FAM_HELM)
            v = {fma(v.re, pc, -v.im * ps), fma(v.re, ps, v.im * pc)};
        else
            v.re *= pc;
        if (prm.values) {
            const int64_t idx = (k * N + i) * N + j;
            if (prm.is_complex) {
                double *o = reinterpret_cast<double *>(prm.values) + 2 * idx;
                o[0] += v.re;
                o[1] += v.im;
            } else {
                reinterpret_cast<double *>(prm.values)[idx] += v.re;
            }
            return;
        }
        const int64_t te = reversed ? s : t, se = reversed ? t : s;
        double mm = 1.0;
        int64_t row = te, col = se;
        if (prm.tl2g) {
            mm = prm.tmult[te * N + i] * prm.smult[se * N + j];
            if (mm == 0.0) return;
            row = prm.tl2g[te * N + i];
            col = prm.sl2g[se * N + j];
        }
        if (MODE == SD_DP0 && t == s) v.re = fma(prm.diag_shift, 0.5 * gt.ie, v.re);
        if (prm.is_complex) {
            double *o = reinterpret_cast<double *>(prm.dense) + 2 * (row * prm.ld + col);
            atomicAdd(o, v.re * mm);
            atomicAdd(o + 1, v.im * mm);
        } else {
            atomicAdd(reinterpret_cast<double *>(prm.dense) + row * prm.ld + col, v.re * mm);
        }
    };
    if constexpr (MODE == SD_DP0) {
        if (lane > (mirror ? 1 : 0)) return;
        const bool rev = lane == 1;
        const double scale = BC_INV_4PI * gt.ie * gs.ie;
        // double layer of (t, s): H (y - x).n_s, of (s, t): -H (y - x).n_t; adjoint: the other way round
        const double2 z = scratch[0], u = scratch[(rev != AD) ? 2 : 1];
        const double sg = (rev != AD) ? -1.0 : 1.0;
        cplx v = {0.0, 0.0};
        if (COMBINED)
            v = {fma(prm.p[2], z.x, fma(-prm.p[3], z.y, sg * u.x)), fma(prm.p[2], z.y, fma(prm.p[3], z.x, sg * u.y))};
        else if (SL)
            v = {z.x, z.y};
        else
            v = {sg * u.x, sg * u.y};
        emit(0, 0, {scale * v.re, scale * v.im}, rev);
    } else {
        for (int e = lane; e < 9; e += G) {
            const int i = e / 3, j = e - 3 * i;
            cplx v, u = {0.0, 0.0};
            if constexpr (MAXWELL) {
                // p_i: the vertex 2 - i that function i vanishes at, relative to V0
                double p[3], q[3];
                duffy_edge(gt, ot.o[0], 2 - i, p);
                duffy_edge(gs, os.o[0], 2 - j, q);
                if constexpr (ASM == BEMPPCUDA_ASM_EFIE) {
                    // sum G (x - P_i).(y - P_j) and sum G
                    const double f[9] = {odot(p, q), -odot(p, S1), -odot(p, S2), -odot(T1, q), odot(T1, S1),
                                         odot(T1, S2), -odot(T2, q), odot(T2, S1), odot(T2, S2)};
                    v = {0.0, 0.0};
#pragma unroll
                    for (int a = 0; a < 9; ++a) {
                        const double2 z = scratch[a];
                        v.re = fma(f[a], z.x, v.re);
                        v.im = fma(f[a], z.y, v.im);
                    }
                    // -ik E - 4 / (ik) M, 1 / (ik) = (-ki - i kr) / |k|^2
                    const double2 z = scratch[0];
                    const double g4 = 4.0 / fma(kr, kr, ki * ki);
                    v = {fma(ki, v.re, kr * v.im) + g4 * fma(ki, z.x, -kr * z.y),
                         fma(ki, v.im, -kr * v.re) + g4 * fma(ki, z.y, kr * z.x)};
                } else {
                    double pq[3], dp[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const int a = (c + 1) % 3, b = (c + 2) % 3;
                        pq[c] = p[a] * q[b] - p[b] * q[a];
                        dp[c] = q[c] - p[c];
                    }
                    const double *T[2] = {T1, T2}, *S[2] = {S1, S2};
                    v = {0.0, 0.0};
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        const double fa = odot(T[a], pq), fc = -odot(S[a], pq);
                        v.re = fma(fa, scratch[4 + a].x, fma(fc, scratch[6 + a].x, v.re));
                        v.im = fma(fa, scratch[4 + a].y, fma(fc, scratch[6 + a].y, v.im));
#pragma unroll
                        for (int b = 0; b < 2; ++b) {
                            const double f = dp[0] * (S[b][1] * T[a][2] - S[b][2] * T[a][1]) +
                                             dp[1] * (S[b][2] * T[a][0] - S[b][0] * T[a][2]) +
                                             dp[2] * (S[b][0] * T[a][1] - S[b][1] * T[a][0]);
                            v.re = fma(f, scratch[2 * a + b].x, v.re);
                            v.im = fma(f, scratch[2 * a + b].y, v.im);
                        }
                    }
                }
                const double f = BC_INV_4PI * edge_length(prm.g, prm.ne, t, i) * edge_length(prm.g, prm.ne, s, j);
                v = {f * v.re, f * v.im};
                u = v;
            } else {
                const int pi = duffy_position(ot, i), pj = duffy_position(os, j);
                const double scale = BC_INV_4PI * gt.ie * gs.ie;
                v = duffy_linear(scratch, pi, pj);
                if (ASM != BEMPPCUDA_ASM_SCALAR) {
                    double ct[3][3], cs[3][3], a[3], b[3];
                    surface_curls(prm.g, prm.ne, t, gt.n, ct);
                    surface_curls(prm.g, prm.ne, s, gs.n, cs);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        a[c] = i == 0 ? ct[0][c] : i == 1 ? ct[1][c] : ct[2][c];
                        b[c] = j == 0 ? cs[0][c] : j == 1 ? cs[1][c] : cs[2][c];
                    }
                    const double cp = odot(a, b);
                    const double2 z = scratch[0];
                    if (ASM == BEMPPCUDA_ASM_LAPLACE_HYP) {
                        v = {cp * z.x, 0.0};
                    } else {
                        const bool helm = ASM == BEMPPCUDA_ASM_HELM_HYP;
                        const double np = odot(gt.n, gs.n), k2r = (helm ? -(kr * kr - ki * ki) : kr * kr) * np,
                                     k2i = (helm ? -2.0 * kr * ki : 0.0) * np;
                        v = {fma(cp, z.x, fma(k2r, v.re, -k2i * v.im)), fma(cp, z.y, fma(k2r, v.im, k2i * v.re))};
                    }
                    u = v;
                } else if (MODE == SD_DL) {
                    // the reversed pair's block takes the other normal with the other sign
                    if (mirror) u = duffy_linear(scratch + 9, pi, pj);
                    if (AD) v = {-v.re, -v.im};
                    if (!AD) u = {-u.re, -u.im};
                } else {
                    u = v;
                }
                v = {scale * v.re, scale * v.im};
                u = {scale * u.re, scale * u.im};
            }
            emit(i, j, v, false);
            if (mirror) emit(j, i, u, true);
        }
    }
}

}  // namespace bc
