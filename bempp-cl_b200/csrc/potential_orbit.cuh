// FP64 potentials and far fields with the two-orbit six-point rule (orbit.cuh): Laplace, Helmholtz, modified
// Helmholtz and Maxwell potentials, Helmholtz and Maxwell far fields, real and complex wavenumbers.
//
// potential_elements writes one record per source element; potential_orbit evaluates a thread per point
// (PPT points), the four warps of a block sharing 32 PPT points and taking every fourth element of the
// staged tile, so that a few dozen points fill the lanes as well as ten thousand (a block of 128 points left
// half its lanes idle at 64 points).  The grid is (point blocks, element chunks); with more than one chunk
// the block sums are added with FP64 atomics into the zeroed result.
//
// Per (point, element), D = c - x, r_c = |D|; per source y = c + g_o e_j:
//   r^2 = r_c^2 + g_o^2 |e_j|^2 + 2 g_o D . e_j           (two operations per source, two dot products per
//                                                          element; D + g_o e_j squared when r_c < near)
//   exp(ik r) = exp(ik r_c) exp(ik (r - r_c)), |r - r_c| <= rho R: the second factor by the polynomials of
// the offset class without range reduction, the first once per element (complex k: the same for the
// amplitude; class 0 factors nothing and reduces every argument).  `near` = 2.5 R: beyond it r >= 1.7 R and the
// expanded square loses nothing (r_c^2 / r^2 < 2.1).
// Far fields: the phase -k x.y = -k x.c - k g_o x.e_j, the same split.
//
// Maxwell: an RWG function's values on one element are alpha y + beta with complex alpha = sum_i x_i l_i and
// beta = -sum_i x_i l_i P_i, so with gamma = alpha c + beta every source is v = w_o (alpha g_o e_j + gamma),
// its divergence term dv = 2 w_o alpha, and the sums over the six sources reduce to the moments
//   g0 = sum w_o G,  tau_j = sum_o w_o g_o (G_oj - G_o2), j = 0, 1
// of the kernel values (G, and H = G (ikr - 1) / r^2 as h0, sigma_j): the vectors enter once per element,
//   electric potential   ik [gamma g0 + alpha e_j tau'_j + (2 / k^2) alpha h0 (x - c)],
//                        tau'_j = tau_j - (2 / k^2) sigma_j
//   magnetic potential   (x - c) x (alpha e_j sigma_j + gamma h0) - (e_j x gamma) sigma_j
//   far fields           V = gamma g0 + alpha e_j tau_j, W = 2 alpha g0: ik V - x W, ik x x V.
// The kernels they replace evaluated every source's vector terms and a range-reduced sine / cosine pair.
// All of them are bound by the FP64 pipe.  Before -> here: Helmholtz single layer on P1, 8192 elements, 10000 points 1396 ->
// 1232 us; electric potential, 4232 elements, 4999 points 1903 -> 531 us; electric far field, 8192 elements, 3600
// directions 1384 -> 490 us.
#pragma once

#include "potential.cuh"

namespace bc {

// Element record: centroid, e_0, e_1, |e_j|^2, then the sources.
constexpr int PO_SCALAR = 28;   // 12-14 normal, 16-27 coefficients (re, im) of the sources in rule order
constexpr int PO_MAXWELL = 44;  // 12-13 alpha, 14-19 gamma, 20-25 alpha e_0, 26-31 alpha e_1, 32-43 e_j x gamma
constexpr int PO_THREADS = 128;
constexpr int PO_ELEMS = 32;    // elements of a block that writes the records
constexpr int PO_LANES = 32;    // points per thread row of a block
constexpr int PO_TILE = 32;     // elements staged at once

// A thread per element; the records meet in shared memory and leave in whole lines.  Blocks of one warp: a few thousand
// elements in blocks of 128 that stored their records themselves kept half of the SMs and most of a line idle (Laplace
// single layer, 8192 elements, 1500 points 0.0998 -> 0.0975 ms a call, 16200 elements, 1000 points 0.1212 -> 0.1184 ms).
template <bool MAXWELL>
__global__ void __launch_bounds__(PO_ELEMS) potential_elements(PotParams prm, OrbitRule rule) {
    constexpr int ES = MAXWELL ? PO_MAXWELL : PO_SCALAR;
    __shared__ double rec[PO_ELEMS][ES + 1];
    const int64_t e0 = (int64_t)blockIdx.x * PO_ELEMS, ei = min(e0 + threadIdx.x, prm.nsupport - 1);
    const int64_t e = prm.support[ei];
    Geom g;
    load_geom(prm.g, prm.ne, e, prm.nm ? (double)prm.nm[e] : 1.0, g);
    double *o = rec[threadIdx.x];
    double c[3], ev[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        c[d] = __ldg(prm.g + (22 + d) * prm.ne + e);
        ev[0][d] = -(g.j0[d] + g.j1[d]) / 3.0;
        ev[1][d] = ev[0][d] + g.j0[d];
        ev[2][d] = ev[0][d] + g.j1[d];
        o[d] = c[d];
        o[3 + d] = ev[0][d];
        o[6 + d] = ev[1][d];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) o[9 + j] = fma(ev[j][2], ev[j][2], fma(ev[j][1], ev[j][1], ev[j][0] * ev[j][0]));
    const double2 *x = reinterpret_cast<const double2 *>(prm.coeff) + e * prm.nshape;
    if (!MAXWELL) {
#pragma unroll
        for (int d = 0; d < 3; ++d) o[12 + d] = g.n[d];
        o[15] = 0.0;
        double2 mean = x[0], dev[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
        if (prm.nshape == 3) {
            mean = make_double2((x[0].x + x[1].x + x[2].x) / 3.0, (x[0].y + x[1].y + x[2].y) / 3.0);
#pragma unroll
            for (int j = 0; j < 3; ++j) dev[j] = make_double2(x[j].x - mean.x, x[j].y - mean.y);
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const int k = q / 3, j = orbit_vertex(q % 3);
            const double f = g.ie * rule.w[k];
            o[16 + 2 * q] = f * fma(rule.g[k], dev[j].x, mean.x);
            o[17 + 2 * q] = f * fma(rule.g[k], dev[j].y, mean.y);
        }
    } else {
        // local function i vanishes at vertex 2 - i (reference functions (x, y-1), (x-1, y), (x, y))
        double ar = 0.0, ai = 0.0, gr[3] = {0.0, 0.0, 0.0}, gi[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double el = edge_length(prm.g, prm.ne, e, i);
            const double fr = x[i].x * el, fi = x[i].y * el;
            ar += fr;
            ai += fi;
#pragma unroll
            for (int d = 0; d < 3; ++d) {  // gamma = -sum_i f_i (P_i - c)
                gr[d] = fma(-fr, ev[2 - i][d], gr[d]);
                gi[d] = fma(-fi, ev[2 - i][d], gi[d]);
            }
        }
        o[12] = ar;
        o[13] = ai;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            o[14 + 2 * d] = gr[d];
            o[15 + 2 * d] = gi[d];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int a = (d + 1) % 3, b = (d + 2) % 3;
                o[20 + 6 * j + 2 * d] = ar * ev[j][d];
                o[21 + 6 * j + 2 * d] = ai * ev[j][d];
                o[32 + 6 * j + 2 * d] = ev[j][a] * gr[b] - ev[j][b] * gr[a];
                o[33 + 6 * j + 2 * d] = ev[j][a] * gi[b] - ev[j][b] * gi[a];
            }
    }
    __syncthreads();
    const int count = (int)min((int64_t)PO_ELEMS, prm.nsupport - e0) * ES;
    for (int i = threadIdx.x; i < count; i += PO_ELEMS) prm.src[ES * e0 + i] = rec[i / ES][i % ES];
}

__device__ __forceinline__ cplx cfma(cplx a, cplx b, cplx c) {
    return {fma(a.re, b.re, fma(-a.im, b.im, c.re)), fma(a.re, b.im, fma(a.im, b.re, c.im))};
}
__device__ __forceinline__ cplx cmulf(cplx a, cplx b) {
    return {fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re)};
}
__device__ __forceinline__ cplx cdiff(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }

// ASM scalar: K = Laplace / Helmholtz / modified Helmholtz / far-field kernel.  ASM electric / magnetic:
// K = Helmholtz single layer (potential) or far-field single layer.  CLS: offset class (fastmath.cuh).
// CK: complex wavenumber (potentials).
template <int ASM, int K, int CLS, bool CK, int PPT>
__global__ void __launch_bounds__(PO_THREADS) potential_orbit(PotParams prm, OrbitRule rule, int64_t chunk_elems,
                                                              double near2) {
    constexpr bool MAXWELL = ASM != BEMPPCUDA_ASM_SCALAR;
    constexpr bool EL = ASM == BEMPPCUDA_ASM_EFIE;
    constexpr bool FAR = K == BEMPPCUDA_FARFIELD_SLP || K == BEMPPCUDA_FARFIELD_DLP;
    constexpr bool HELM = K == BEMPPCUDA_HELMHOLTZ_SLP || K == BEMPPCUDA_HELMHOLTZ_DLP;
    constexpr bool MH = K == BEMPPCUDA_MODHELM_SLP || K == BEMPPCUDA_MODHELM_DLP;
    constexpr bool DLP = K == BEMPPCUDA_LAPLACE_DLP || K == BEMPPCUDA_HELMHOLTZ_DLP || K == BEMPPCUDA_MODHELM_DLP ||
                         K == BEMPPCUDA_FARFIELD_DLP;
    constexpr int ES = MAXWELL ? PO_MAXWELL : PO_SCALAR;
    constexpr int NA = MAXWELL ? (FAR && EL ? 4 : 3) : 1;  // accumulated complex values per point
    constexpr int GROUPS = PO_THREADS / PO_LANES;
    __shared__ __align__(16) double tile[PO_TILE * ES];
    static_assert(PO_TILE * ES >= (GROUPS - 1) * PO_LANES * NA * 2 * PPT, "the block sum reuses the tile");
    const int lane = threadIdx.x % PO_LANES, group = threadIdx.x / PO_LANES;
    const int64_t ebeg = (int64_t)blockIdx.y * chunk_elems;
    const int64_t eend = min(ebeg + chunk_elems, prm.nsupport);
    const int64_t pbase = (int64_t)blockIdx.x * (PO_LANES * PPT) + lane;
    double x[PPT][3];
    cplx acc[PPT][NA];
    bool unit[PPT];  // far field: |x| <= 1, so the class bounds the phase offsets
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
        const int64_t pj = min(pbase + j * PO_LANES, prm.npoints - 1);
#pragma unroll
        for (int d = 0; d < 3; ++d) x[j][d] = prm.points[3 * pj + d];
        unit[j] = fma(x[j][2], x[j][2], fma(x[j][1], x[j][1], x[j][0] * x[j][0])) <= 1.0001;
#pragma unroll
        for (int a = 0; a < NA; ++a) acc[j][a] = {0.0, 0.0};
    }
    const double k = prm.p[0], ki = CK ? prm.p[1] : 0.0;
    const double g0 = rule.g[0], g1 = rule.g[1];
    const double gg[2] = {g0 * g0, g1 * g1}, g2[2] = {2.0 * g0, 2.0 * g1};
    const double w[2] = {rule.w[0], rule.w[1]}, wg[2] = {rule.w[0] * g0, rule.w[1] * g1};
    // 2 / k^2
    cplx tk = {0.0, 0.0};
    if (MAXWELL && EL && !FAR) {
        if (CK) {
            const double m = fma(k, k, ki * ki), s = 2.0 / (m * m);
            tk = {s * (k * k - ki * ki), -s * (2.0 * k * ki)};
        } else {
            tk = {2.0 / (k * k), 0.0};
        }
    }
    for (int64_t t0 = ebeg; t0 < eend; t0 += PO_TILE) {
        const int te = (int)min((int64_t)PO_TILE, eend - t0);
        __syncthreads();
        for (int s = threadIdx.x; s < te * ES; s += PO_THREADS) tile[s] = prm.src[t0 * ES + s];
        __syncthreads();
#pragma unroll 1
        for (int e = group; e < te; e += GROUPS) {
            const double2 *rec = reinterpret_cast<const double2 *>(tile + e * ES);
            const double2 r0 = rec[0], r1 = rec[1], r2_ = rec[2], r3 = rec[3], r4 = rec[4], r5 = rec[5];
            const double c[3] = {r0.x, r0.y, r1.x}, e0[3] = {r1.y, r2_.x, r2_.y}, e1[3] = {r3.x, r3.y, r4.x};
            const double ee[3] = {r4.y, r5.x, r5.y};
            double q2[PPT][6], ph[PPT], rc_[PPT], D[PPT][3];  // r^2 (near field) or phase offsets (far field)
#pragma unroll
            for (int j = 0; j < PPT; ++j) {
                if (FAR) {
                    ph[j] = -k * fma(x[j][2], c[2], fma(x[j][1], c[1], x[j][0] * c[0]));
                    const double a0 = -k * fma(x[j][2], e0[2], fma(x[j][1], e0[1], x[j][0] * e0[0]));
                    const double a1 = -k * fma(x[j][2], e1[2], fma(x[j][1], e1[1], x[j][0] * e1[0]));
                    const double a[3] = {a0, a1, -(a0 + a1)};
#pragma unroll
                    for (int q = 0; q < 6; ++q) {
                        const double g = rule.g[q / 3], at = a[orbit_vertex(q % 3)];
                        q2[j][q] = CLS == 0 ? fma(g, at, ph[j]) : g * at;
                    }
                } else {
#pragma unroll
                    for (int d = 0; d < 3; ++d) D[j][d] = c[d] - x[j][d];
                    const double rc2 = fma(D[j][2], D[j][2], fma(D[j][1], D[j][1], D[j][0] * D[j][0]));
                    rc_[j] = CLS > 0 ? dist64(rc2) : 0.0;  // a point may sit on a centroid
                    ph[j] = HELM || MH ? k * rc_[j] : 0.0;
                    if (rc2 >= near2) {
                        const double a0 = fma(D[j][2], e0[2], fma(D[j][1], e0[1], D[j][0] * e0[0]));
                        const double a1 = fma(D[j][2], e1[2], fma(D[j][1], e1[1], D[j][0] * e1[0]));
                        const double a[3] = {a0, a1, -(a0 + a1)};
#pragma unroll
                        for (int q = 0; q < 6; ++q) {
                            const int o = q / 3, v = orbit_vertex(q % 3);
                            q2[j][q] = fma(g2[o], a[v], fma(gg[o], ee[v], rc2));
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 6; ++q) {
                            const int v = orbit_vertex(q % 3);
                            double s = 0.0;
#pragma unroll
                            for (int d = 0; d < 3; ++d) {
                                const double ev = v == 0 ? e0[d] : v == 1 ? e1[d] : -(e0[d] + e1[d]);
                                const double t = fma(rule.g[q / 3], ev, D[j][d]);
                                s = fma(t, t, s);
                            }
                            q2[j][q] = s;
                        }
                    }
                }
            }
            if constexpr (!MAXWELL) {
                const double2 *cf = rec + 8;
                cplx s[PPT];
#pragma unroll
                for (int j = 0; j < PPT; ++j) s[j] = {0.0, 0.0};
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const double2 cq = cf[q];
#pragma unroll
                    for (int j = 0; j < PPT; ++j) {
                        if (FAR) {
                            double sn, cs;
                            if (CLS == 0 || unit[j])
                                sincos_off64<CLS>(q2[j][q], &sn, &cs);
                            else
                                sincos_cw64(q2[j][q], &sn, &cs);
                            s[j] = cfma({cs, sn}, {cq.x, cq.y}, s[j]);
                            continue;
                        }
                        const double r2 = q2[j][q], rinv = rsqrt64(r2);
                        double f = DLP ? rinv * rinv * rinv : rinv;
                        if (!HELM) {
                            if (MH) {
                                const double r = r2 * rinv;
                                f *= exp_off64<CLS>(fma(-k, r, ph[j]));
                                if (DLP) f *= fma(k, r, 1.0);
                            }
                            s[j].re = fma(f, cq.x, s[j].re);
                            s[j].im = fma(f, cq.y, s[j].im);
                        } else {
                            const double r = r2 * rinv;
                            double sn, cs;
                            sincos_off64<CLS>(fma(k, r, -ph[j]), &sn, &cs);
                            if (CK) f *= exp_off64<CLS>(-ki * (r - rc_[j]));
                            double wr = f * cq.x, wi = f * cq.y;
                            if (DLP) {  // times (i k r - 1) = -a + i b
                                const double b = k * r, a = CK ? fma(ki, r, 1.0) : 1.0;
                                const double tr = -fma(b, wi, a * wr), ti = fma(b, wr, -a * wi);
                                wr = tr;
                                wi = ti;
                            }
                            s[j] = cfma({cs, sn}, {wr, wi}, s[j]);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < PPT; ++j) {
                    if (DLP) {
                        // a source lies in its element's plane: (y - x) . n = D . n for all six
                        const double2 n0 = rec[6], n1 = rec[7];
                        double dn;
                        if (FAR)
                            dn = -k * fma(x[j][2], n1.x, fma(x[j][1], n0.y, x[j][0] * n0.x));
                        else
                            dn = fma(D[j][2], n1.x, fma(D[j][1], n0.y, D[j][0] * n0.x));
                        if (!FAR && !HELM) dn = -dn;
                        s[j] = FAR ? cplx{-dn * s[j].im, dn * s[j].re} : cplx{dn * s[j].re, dn * s[j].im};
                    }
                    if (CLS > 0 && (HELM || FAR)) {
                        double sn, cs;
                        sincos_cw64(ph[j], &sn, &cs);
                        if (CK) {
                            const double am = exp(-ki * rc_[j]);
                            sn *= am;
                            cs *= am;
                        }
                        acc[j][0] = cfma({cs, sn}, s[j], acc[j][0]);
                    } else {
                        const double am = MH && CLS > 0 ? exp(-ph[j]) : 1.0;
                        acc[j][0].re = fma(am, s[j].re, acc[j][0].re);
                        acc[j][0].im = fma(am, s[j].im, acc[j][0].im);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < PPT; ++j) {
                    // moments of G and of H = G (ikr - 1) / r^2 over the sources (4 pi and the element's phase
                    // left out)
                    cplx m0 = {0.0, 0.0}, t[3], h0 = {0.0, 0.0}, s[3];
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        cplx so = {0.0, 0.0}, ho = {0.0, 0.0};
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            const int q = 3 * o + i, v = orbit_vertex(i);
                            cplx G, H = {0.0, 0.0};
                            if (FAR) {
                                if (CLS == 0 || unit[j])
                                    sincos_off64<CLS>(q2[j][q], &G.im, &G.re);
                                else
                                    sincos_cw64(q2[j][q], &G.im, &G.re);
                            } else {
                                const double r2 = q2[j][q], rinv = rsqrt64(r2), r = r2 * rinv;
                                double sn, cs, f = rinv;
                                sincos_off64<CLS>(fma(k, r, -ph[j]), &sn, &cs);
                                if (CK) f *= exp_off64<CLS>(-ki * (r - rc_[j]));
                                G = {f * cs, f * sn};
                                const double i2 = rinv * rinv, b = k * r;
                                if (CK) {
                                    const double a = fma(ki, r, 1.0);
                                    H = {-fma(b, G.im, a * G.re) * i2, fma(b, G.re, -a * G.im) * i2};
                                } else {
                                    H = {-fma(b, G.im, G.re) * i2, fma(b, G.re, -G.im) * i2};
                                }
                            }
                            if (EL || FAR) {
                                so = {so.re + G.re, so.im + G.im};
                                t[v] = o == 0 ? cplx{wg[0] * G.re, wg[0] * G.im}
                                              : cplx{fma(wg[1], G.re, t[v].re), fma(wg[1], G.im, t[v].im)};
                            }
                            if (!FAR) {
                                ho = {ho.re + H.re, ho.im + H.im};
                                s[v] = o == 0 ? cplx{wg[0] * H.re, wg[0] * H.im}
                                              : cplx{fma(wg[1], H.re, s[v].re), fma(wg[1], H.im, s[v].im)};
                            }
                        }
                        m0 = {fma(w[o], so.re, m0.re), fma(w[o], so.im, m0.im)};
                        h0 = {fma(w[o], ho.re, h0.re), fma(w[o], ho.im, h0.im)};
                    }
                    cplx rot = {1.0, 0.0};
                    if (CLS > 0) sincos_cw64(ph[j], &rot.im, &rot.re);
                    if (CK && CLS > 0) {
                        const double am = exp(-ki * rc_[j]);
                        rot = {am * rot.re, am * rot.im};
                    }
                    const auto vec = [&](int at, int d) -> cplx {
                        const double2 z = rec[at / 2 + d];
                        return {z.x, z.y};
                    };
                    const cplx alpha = vec(12, 0);
                    if (FAR) {
                        const cplx f0 = cmulf(rot, m0), f1 = cmulf(rot, cdiff(t[0], t[2])),
                                   f2 = cmulf(rot, cdiff(t[1], t[2]));
#pragma unroll
                        for (int d = 0; d < 3; ++d)
                            acc[j][d] = cfma(vec(14, d), f0, cfma(vec(20, d), f1, cfma(vec(26, d), f2, acc[j][d])));
                        if (EL) acc[j][NA - 1] = cfma(alpha, f0, acc[j][NA - 1]);
                    } else if (EL) {
                        const cplx s0 = cdiff(s[0], s[2]), s1 = cdiff(s[1], s[2]);
                        cplx f1 = cdiff(t[0], t[2]), f2 = cdiff(t[1], t[2]);
                        const cplx mtk = {-tk.re, -tk.im};
                        cplx hk;  // (2 / k^2) alpha h0
                        if (CK) {
                            f1 = cfma(mtk, s0, f1);
                            f2 = cfma(mtk, s1, f2);
                            hk = cmulf(tk, h0);
                        } else {
                            f1 = {fma(mtk.re, s0.re, f1.re), fma(mtk.re, s0.im, f1.im)};
                            f2 = {fma(mtk.re, s1.re, f2.re), fma(mtk.re, s1.im, f2.im)};
                            hk = {tk.re * h0.re, tk.re * h0.im};
                        }
                        hk = cmulf(alpha, hk);
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const cplx xd = {-D[j][d] * hk.re, -D[j][d] * hk.im};
                            const cplx v = cfma(vec(14, d), m0, cfma(vec(20, d), f1, cfma(vec(26, d), f2, xd)));
                            acc[j][d] = cfma(rot, v, acc[j][d]);
                        }
                    } else {
                        const cplx s0 = cdiff(s[0], s[2]), s1 = cdiff(s[1], s[2]);
                        cplx W[3];
#pragma unroll
                        for (int d = 0; d < 3; ++d)
                            W[d] = cfma(vec(14, d), h0, cfma(vec(20, d), s0, cmulf(vec(26, d), s1)));
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const int a = (d + 1) % 3, b = (d + 2) % 3;
                            const cplx u = cfma(vec(32, d), s0, cmulf(vec(38, d), s1));
                            // (x - c) x W = -D x W
                            const cplx v = {fma(D[j][b], W[a].re, fma(-D[j][a], W[b].re, -u.re)),
                                            fma(D[j][b], W[a].im, fma(-D[j][a], W[b].im, -u.im))};
                            acc[j][d] = cfma(rot, v, acc[j][d]);
                        }
                    }
                }
            }
        }
    }
    // sum over the block's warps
    __syncthreads();
    double2 *part = reinterpret_cast<double2 *>(tile);
    if (group > 0)
#pragma unroll
        for (int j = 0; j < PPT; ++j)
#pragma unroll
            for (int a = 0; a < NA; ++a)
                part[((group - 1) * PPT * NA + j * NA + a) * PO_LANES + lane] = make_double2(acc[j][a].re, acc[j][a].im);
    __syncthreads();
    if (group > 0) return;
#pragma unroll
    for (int j = 0; j < PPT; ++j) {
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int h = 0; h < GROUPS - 1; ++h) {
                const double2 z = part[(h * PPT * NA + j * NA + a) * PO_LANES + lane];
                acc[j][a] = {acc[j][a].re + z.x, acc[j][a].im + z.y};
            }
        const int64_t pj = pbase + j * PO_LANES;
        if (pj >= prm.npoints) break;
        const cplx ik = {-prm.p[1], k};
        cplx u[MAXWELL ? 3 : 1];
        if constexpr (!MAXWELL) {
            u[0] = acc[j][0];
        } else if constexpr (FAR) {
            cplx v[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) v[d] = cmulf(ik, acc[j][d]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int a = (d + 1) % 3, b = (d + 2) % 3;
                if (EL)
                    u[d] = {fma(-2.0 * x[j][d], acc[j][NA - 1].re, v[d].re),
                            fma(-2.0 * x[j][d], acc[j][NA - 1].im, v[d].im)};
                else
                    u[d] = {x[j][a] * v[b].re - x[j][b] * v[a].re, x[j][a] * v[b].im - x[j][b] * v[a].im};
            }
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) u[d] = EL ? cmulf(ik, acc[j][d]) : acc[j][d];
        }
#pragma unroll
        for (int d = 0; d < (MAXWELL ? 3 : 1); ++d) {
            double *out = prm.result + 2 * (d * prm.npoints + pj);
            if (gridDim.y == 1) {
                out[0] = BC_INV_4PI * u[d].re;
                out[1] = BC_INV_4PI * u[d].im;
            } else {
                atomicAdd(out, BC_INV_4PI * u[d].re);
                atomicAdd(out + 1, BC_INV_4PI * u[d].im);
            }
        }
    }
}

}  // namespace bc
