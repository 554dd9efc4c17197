// Regular pairs on P1 / DP1 / P0 spaces in the points form (coordinates differenced per point pair, any 6-point
// rule): the Laplace single layer and hypersingular operators and the Helmholtz single, double and adjoint double
// layers for a real wavenumber.  The orbit form (p1.cuh) takes fewer FP64 operations in each of them, but its sums
// depend on each other more: at 8192 elements, k = 5 it runs the single layer in 3.79 ms against 3.52 here, the
// Laplace single layer in 1.81 against 1.68, the Laplace hypersingular operator in 2.03 against 1.62, and the double
// layers in 6.2 against 5.64 (their skew sweep keeps two complex blocks, the parts they share and the orbit sums).
//
// One thread per trial element, up to 32 test elements staged in shared memory.  Per test point p the trial sums
// T_j(p) = sum_q w_q K psi_j(q) come first, then L_ij += w_p phi_i(p) T_j(p): NS complex FMAs per point pair; the
// hypersingular operator needs only the sum of the kernel values (its test and trial curls are constant).
// exp(ikr) is factored about the centroid distance by offset class (fastmath.cuh).  Symmetric and skew sweeps, the
// deferred transpose and the atomics as in p1.cuh.  Bound by the FP64 pipe (76 - 83 %) from a few thousand elements;
// at 1152, 32 rows per CTA are one working CTA per SM (single layer k = 2: 0.239 -> 0.143 ms with the row blocks
// of lin_row_blocks).
#pragma once

#include "dp0.cuh"

namespace bc {

constexpr int PTS_TCHUNK = 32;

struct TestBlockPoints {
    double x[PTS_TCHUNK][NQ6][3];
    double n[PTS_TCHUNK][3];
    double c[PTS_TCHUNK][3];
    double curl[PTS_TCHUNK][3][3];
    double ie[PTS_TCHUNK];
    double mult[PTS_TCHUNK][3];  // local multipliers of the test functions
    int64_t row[PTS_TCHUNK][3];  // their global dofs
    int v[PTS_TCHUNK][3];
};

template <int ASM, int K, int NT, int NS, int CLS, bool SYM>
__global__ void __launch_bounds__(DP0_THREADS) regular_p1_points(RegParams prm, QuadRule rule) {
    constexpr bool HYP = ASM == BEMPPCUDA_ASM_LAPLACE_HYP;
    constexpr bool HELM = (K == BEMPPCUDA_HELMHOLTZ_SLP || K == BEMPPCUDA_HELMHOLTZ_DLP ||
                           K == BEMPPCUDA_HELMHOLTZ_ADLP);
    constexpr bool DL = K == BEMPPCUDA_HELMHOLTZ_DLP, AD = K == BEMPPCUDA_HELMHOLTZ_ADLP;
    static_assert(HELM || K == BEMPPCUDA_LAPLACE_SLP, "the operators of p1_points_form");
    constexpr bool PH = HELM && CLS > 0;
    static_assert(!SYM || NT == NS, "the symmetric sweep needs one space on both sides");
    constexpr bool SKEW = SYM && (DL || AD);  // the transposed block uses the other element's normal
    __shared__ TestBlockPoints sb;

    // test elements per CTA: ceil(ntest / gridDim.y) <= PTS_TCHUNK (the launch picks the row blocks)
    const int rows = (int)((prm.ntest + gridDim.y - 1) / gridDim.y);
    const int64_t t0 = (int64_t)blockIdx.y * rows;
    if (SYM && t0 >= ((int64_t)blockIdx.x + 1) * DP0_THREADS) return;  // below the diagonal
    const int tcount = (int)min((int64_t)rows, prm.ntest - t0);
    for (int idx = threadIdx.x; idx < tcount; idx += blockDim.x) {
        const int64_t t = prm.tsup[t0 + idx];
        Geom g;
        load_geom(prm.tg, prm.tne, t, prm.tnm ? (double)prm.tnm[t] : 1.0, g);
        for (int p = 0; p < NQ6; ++p) to_global(g, rule.x[p], rule.y[p], sb.x[idx][p]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            sb.n[idx][d] = g.n[d];
            sb.c[idx][d] = __ldg(prm.tg + (22 + d) * prm.tne + t);
            sb.v[idx][d] = __ldg(prm.tel + 3 * t + d);
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            sb.mult[idx][i] = prm.tmult[t * NT + i];
            sb.row[idx][i] = prm.tl2g[t * NT + i];
        }
        if (HYP) {
            double cu[3][3];
            surface_curls(prm.tg, prm.tne, t, g.n, cu);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int d = 0; d < 3; ++d) sb.curl[idx][i][d] = cu[i][d];
        }
        sb.ie[idx] = g.ie;
    }
    __syncthreads();

    const int64_t si = (int64_t)blockIdx.x * DP0_THREADS + threadIdx.x;
    if (si >= prm.ntrial) return;
    const int64_t s = prm.ssup[si];
    Geom gs;
    load_geom(prm.sg, prm.sne, s, prm.snm ? (double)prm.snm[s] : 1.0, gs);
    const int sv0 = __ldg(prm.sel + 3 * s), sv1 = __ldg(prm.sel + 3 * s + 1), sv2 = __ldg(prm.sel + 3 * s + 2);
    double y[NQ6][3];
#pragma unroll
    for (int q = 0; q < NQ6; ++q) to_global(gs, rule.x[q], rule.y[q], y[q]);
    double sc[3] = {0.0, 0.0, 0.0};
    if (PH)
#pragma unroll
        for (int d = 0; d < 3; ++d) sc[d] = __ldg(prm.sg + (22 + d) * prm.sne + s);
    double curl_s[3][3];
    if (HYP) surface_curls(prm.sg, prm.sne, s, gs.n, curl_s);
    // trial / test shape values times the weights (constant operands from the rule)
    const auto psw = [&](int q, int j) -> double { return NS == 1 ? rule.w[q] : rule.sw[q][j]; };
    const double kr = prm.p[0];
    // the trial dofs and multipliers stay in registers for the whole tile
    int64_t scol[NS];
    double smul[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        scol[j] = prm.sl2g[s * NS + j];
        smul[j] = prm.smult[s * NS + j];
    }
    // (y_q - v0_s).n_s, the split of the double-layer normal term about the trial vertex 0
    double ynv[NQ6];
    if (DL && !SKEW)
#pragma unroll
        for (int q = 0; q < NQ6; ++q)
            ynv[q] = fma(y[q][2] - gs.v0[2], gs.n[2], fma(y[q][1] - gs.v0[1], gs.n[1], (y[q][0] - gs.v0[0]) * gs.n[0]));

    for (int tt = 0; tt < tcount; ++tt) {
        if (SYM && t0 + tt >= si) break;  // rows increase with tt
        if (prm.grids_identical && shares_vertex(sb.v[tt], sv0, sv1, sv2)) continue;
        // SKEW: the normal factors by the plane property (a quadrature point lies in its own element's
        // plane): (y_q - x_p).n_s = (v0_s - x_p).n_s, one value per test point (xn below), and
        // (x_p - y_q).n_t = (c_t - y_q).n_t, one value per trial point
        double mdt[SKEW ? NQ6 : 1];
        if (SKEW)
#pragma unroll
            for (int q = 0; q < NQ6; ++q)
                mdt[q % (SKEW ? NQ6 : 1)] =
                    fma(sb.c[tt][2] - y[q][2], sb.n[tt][2],
                        fma(sb.c[tt][1] - y[q][1], sb.n[tt][1], (sb.c[tt][0] - y[q][0]) * sb.n[tt][0]));
        double krc = 0.0, ph_s = 0.0, ph_c = 1.0;
        if (PH) {
            const double D0 = sc[0] - sb.c[tt][0], D1 = sc[1] - sb.c[tt][1], D2 = sc[2] - sb.c[tt][2];
            krc = kr * sqrt(fma(D2, D2, fma(D1, D1, D0 * D0)));
            sincos_cw64(krc, &ph_s, &ph_c);
        }
        double lre[NT][NS], lim[NT][NS];
        double ure[SKEW ? NT : 1][SKEW ? NS : 1], uim[SKEW ? NT : 1][SKEW ? NS : 1];  // SKEW: block of (j, i)
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < NS; ++j) lre[i][j] = lim[i][j] = 0.0;
        if (SKEW)
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int j = 0; j < NS; ++j) ure[i % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)] = uim[i % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)] = 0.0;
        double sre = 0.0;  // HYP: sum_pq w G
        for (int p = 0; p < NQ6; ++p) {
            const double x0 = sb.x[tt][p][0], x1 = sb.x[tt][p][1], x2 = sb.x[tt][p][2];
            double xn = 0.0;
            if (DL || SKEW) xn = fma(gs.v0[2] - x2, gs.n[2], fma(gs.v0[1] - x1, gs.n[1], (gs.v0[0] - x0) * gs.n[0]));
            double tre[NS], tim[NS], vre[SKEW ? NS : 1], vim[SKEW ? NS : 1];
#pragma unroll
            for (int j = 0; j < NS; ++j) tre[j] = tim[j] = 0.0;
            if (SKEW)
#pragma unroll
                for (int j = 0; j < NS; ++j) vre[j % (SKEW ? NS : 1)] = vim[j % (SKEW ? NS : 1)] = 0.0;
#pragma unroll
            for (int q = 0; q < NQ6; ++q) {
                const double d0 = y[q][0] - x0, d1 = y[q][1] - x1, d2 = y[q][2] - x2;
                const double r2 = fma(d2, d2, fma(d1, d1, d0 * d0));
                const double rinv = rsqrt64(r2);
                double kre, kim = 0.0;  // kernel value without 1/(4 pi)
                double k2re = 0.0, k2im = 0.0;  // SKEW: the transposed pair's kernel
                if (!HELM) {
                    kre = rinv;
                } else {
                    const double r = r2 * rinv;
                    double sn, cs;
                    sincos_off64<CLS>(fma(kr, r, -krc), &sn, &cs);
                    if (SKEW) {
                        // double layer of trial normal n: (dot with n) (kre + i kim), whose trial-normal factor xn is
                        // applied per test point, and the same times the test-normal factor of this trial point
                        const double rinv2 = rinv * rinv;
                        kre = -rinv2 * fma(rinv, cs, kr * sn);
                        kim = rinv2 * fma(kr, cs, -rinv * sn);
                        k2re = mdt[q % (SKEW ? NQ6 : 1)] * kre;
                        k2im = mdt[q % (SKEW ? NQ6 : 1)] * kim;
                    } else if (K == BEMPPCUDA_HELMHOLTZ_SLP) {
                        kre = cs * rinv;
                        kim = sn * rinv;
                    } else {
                        // (ikr - 1) e^{ikr} dot / r^3 = g (-h1 + i h2), g = dot / r^2
                        const double dot = DL ? ynv[q] + xn
                                              : -fma(d2, sb.n[tt][2], fma(d1, sb.n[tt][1], d0 * sb.n[tt][0]));
                        const double g = dot * rinv * rinv;
                        kre = -g * fma(rinv, cs, kr * sn);
                        kim = g * fma(kr, cs, -rinv * sn);
                    }
                }
#pragma unroll
                for (int j = 0; j < NS; ++j) {
                    tre[j] = fma(kre, psw(q, j), tre[j]);
                    tim[j] = fma(kim, psw(q, j), tim[j]);
                }
                if (SKEW)
#pragma unroll
                    for (int j = 0; j < NS; ++j) {
                        vre[j % (SKEW ? NS : 1)] = fma(k2re, psw(q, j), vre[j % (SKEW ? NS : 1)]);
                        vim[j % (SKEW ? NS : 1)] = fma(k2im, psw(q, j), vim[j % (SKEW ? NS : 1)]);
                    }
            }
            const double wp = rule.w[p];
            const auto phw = [&](int i) -> double { return NT == 1 ? wp : rule.sw[p][i]; };
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                // SKEW: the sums of h take the trial-normal factor xn of this test point; they form the
                // (i, j) block of the double layer and the transposed block of the adjoint double layer
                const double px = SKEW ? phw(i) * xn : phw(i);
#pragma unroll
                for (int j = 0; j < NS; ++j) {
                    if (!SKEW) {
                        lre[i][j] = fma(phw(i), tre[j], lre[i][j]);
                        lim[i][j] = fma(phw(i), tim[j], lim[i][j]);
                    } else {
                        constexpr int a = SKEW ? NT : 1, b = SKEW ? NS : 1;
                        // (weight, sum) of the (i, j) block and of the transposed pair's block
                        const double w1 = DL ? px : phw(i), w2 = DL ? phw(i) : px;
                        const double s1r = DL ? tre[j] : vre[j % b], s1i = DL ? tim[j] : vim[j % b];
                        const double s2r = DL ? vre[j % b] : tre[j], s2i = DL ? vim[j % b] : tim[j];
                        lre[i][j] = fma(w1, s1r, lre[i][j]);
                        lim[i][j] = fma(w1, s1i, lim[i][j]);
                        ure[i % a][j % b] = fma(w2, s2r, ure[i % a][j % b]);
                        uim[i % a][j % b] = fma(w2, s2i, uim[i % a][j % b]);
                    }
                }
            }
            if (HYP)
#pragma unroll
                for (int j = 0; j < NS; ++j) {
                    sre = fma(wp, tre[j], sre);
                }
        }
        const double scale = BC_INV_4PI * sb.ie[tt] * gs.ie;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const double mt = sb.mult[tt][i];
            if (mt == 0.0) continue;
            const int64_t row = sb.row[tt][i];
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const double ms = smul[j];
                if (ms == 0.0) continue;
                double vr = lre[i][j], vi = lim[i][j];
                if (HYP) {
                    const double cij = sb.curl[tt][i][0] * curl_s[j][0] + sb.curl[tt][i][1] * curl_s[j][1] +
                                       sb.curl[tt][i][2] * curl_s[j][2];
                    vr = cij * sre;
                    vi = 0.0;
                }
                // SKEW: the transposed pair's own block, else the same block
                double wr = SKEW ? ure[i % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)] : vr;
                double wi = SKEW ? uim[i % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)] : vi;
                if (PH) {
                    const double tr = vr * ph_c - vi * ph_s;
                    vi = fma(vr, ph_s, vi * ph_c);
                    vr = tr;
                    if (SKEW) {
                        const double ur = wr * ph_c - wi * ph_s;
                        wi = fma(wr, ph_s, wi * ph_c);
                        wr = ur;
                    } else {
                        wr = vr;
                        wi = vi;
                    }
                }
                const double m = mt * ms * scale;
                const int64_t col = scol[j];
                if (prm.is_complex) {
                    double *o = reinterpret_cast<double *>(prm.result) + 2 * (row * prm.ld + col);
                    atomicAdd(o, vr * m);
                    atomicAdd(o + 1, vi * m);
                    if (SYM && (SKEW || !prm.defer_transpose)) {
                        double *ot = reinterpret_cast<double *>(prm.result) + 2 * (col * prm.ld + row);
                        atomicAdd(ot, wr * m);
                        atomicAdd(ot + 1, wi * m);
                    }
                } else {
                    atomicAdd(reinterpret_cast<double *>(prm.result) + row * prm.ld + col, vr * m);
                    if (SYM && (SKEW || !prm.defer_transpose))
                        atomicAdd(reinterpret_cast<double *>(prm.result) + col * prm.ld + row, wr * m);
                }
            }
        }
    }
}

}  // namespace bc
