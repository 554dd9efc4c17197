// Mixed-precision regular pairs of the single layer, double layer, adjoint
// double layer and hypersingular operators on P1 spaces (6-point rule) for the
// Helmholtz (Re k > 0, real or complex k), Laplace and modified Helmholtz
// kernels: the FP32 counterpart of regular_p1 (p1.cuh) with the geometry of
// the mixed DP0 kernels (dp0.cuh).
//
// Lengths are in units of 1/k.  Per element pair the centroid offset
// D = k (c_s - c_t), r_c' = |D| and exp(i r_c') are FP64; per point pair, with
// the two-orbit rule (orbit.cuh; x_p = c_t + g_p e_i, y_q = c_s + g_q f_j),
//   s = r'^2 - r_c'^2 = A_q + B_p - 2 g_p g_q e_i . f_j
// is formed in FP32, 1/r' by rsqrt.approx, the phase offset theta = r' - r_c'
// by one Newton step on theta^2 + 2 r_c' theta = s (dp0_sym.cuh) and its sine /
// cosine by the fitted FP32 polynomials; near pairs difference the coordinates
// (near_mr2, dp0.cuh) and follow the sweep.  The trial points of one vertex, one
// of each orbit, travel together through packed f32x2 FMAs; the blocks of the
// trial sums T_j(p) = sum_q w_q psi_j(q) K add real and imaginary parts packed.
// Double layers: with h = (i r' - 1) exp(i theta) / r'^3 and d' = k (y - x),
// a quadrature point lies in its own element's plane, so
//   d' . n_s = D . n_s - xo_p . n_s      (one value per test point)
//   d' . n_t = D . n_t + yo_q . n_t      (one value per trial point);
// the double layer (trial normal) sums T_j(p) = sum_q w_q psi_j(q) h and
// multiplies by d'.n_s per test point, the adjoint double layer (test normal,
// kernel -(d . n_t)) sums h (-d'.n_t) per pair.  The 3 x 3 block
// sum_p w_p phi_i(p) T_j(p) is FP32 (36 terms per entry); it is converted to
// FP64 once per element pair, where k / (4 pi) (single layer, hypersingular)
// or k^2 / (4 pi) (double layers), the integration elements, exp(i r_c') and
// (hypersingular) the curl and normal products are applied.  SYM as in
// regular_p1: pairs i < j; single layer and hypersingular add the block at
// (i, j) and, unless deferred to the transpose pass, at (j, i); the double
// layers add at (j, i) the transposed pair's own block, which is the other
// operator's kernel of (i, j) (skew sweep: both normal sums per pair).
// Other kernels, in units of 1/kappa (kappa = Re k, omega, or 1 for Laplace):
// Laplace has no phase (1/r', -1/r'^3 in the double layers); modified
// Helmholtz exp(-r') = exp(-r_c') exp(-theta), the first FP64 per element
// pair, the second __expf per point pair, double-layer factor -(1 + r'); a
// complex wavenumber k = kr + i ki adds exp(-beta r'), beta = ki / kr, split
// the same way beside exp(i r'), the double-layer factor
// (i k r - 1) = -(1 + beta r') + i r', and -k^2 complex in the hypersingular
// operator.  Laplace and modified Helmholtz blocks are real and go to a real
// matrix.
// Maxwell magnetic field on RWG / SNC (ASM_MFIE): with u_i(p) = J_t r_i(p) =
// x_p - P_ti and v_j(q) = y_q - P_sj (P: the vertex each RWG function points
// away from), (x - y) . (u x v) = (P_ti - P_sj) . (u x v), so
//   MFIE_ij = sum_ab det(P_ti - P_sj, J_t^a, J_s^b) N_ab,
//   N_ab = sum_pq w_p w_q H (zeta_a(p) - o_ia)(zeta_b(q) - o_jb),
// zeta = (xi, eta), o_i = (a_i, b_i), H = e^{ikr} (ikr - 1) / r^3: the N are
// shifts of the nine moments of H, which the FP32 core gives as it gives
// the EFIE's moments of G (the double layer's kernel value h without its
// normal factor).  The determinants are FP64 geometry, so pairs of nearly
// coplanar elements, whose triple products nearly vanish, keep the FP32
// moments' relative accuracy (mfie_block_moments).
// Maxwell electric field on RWG / SNC (ASM_EFIE): the nine moments
// M[u][v] = sum_pq w_p w_q G u(p) v(q), u, v in {1, xi, eta}, that the EFIE
// block needs (rwg.cuh) are a fixed linear map of the P1 single-layer block
// (1 = phi_0 + phi_1 + phi_2, xi = phi_1, eta = phi_2), so the FP32 part is
// the single layer's and the FP64 epilogue forms the moments and
// efie_block; the integration elements cancel against the RWG basis.
// Scatter: the FP64 block entries of a warp's 32 pairs (one test element,
// 32 consecutive trial elements) are summed per distinct trial dof in shared
// memory and added to the matrix once per (test dof, trial dof)
// (warp_cols.cuh): ~3.5x fewer FP64 L2 atomics, which bound the double-layer
// sweep (each pair adds two blocks).
// Bound by latency at three CTAs per SM (168 registers; double layer: FMA pipe 55 %
// of its cycles, issue 55 %, first stall the fixed latency).  Double layer, 10952
// elements, k = 6: 6.77 -> 5.67 ms from packing neighbouring trial points to packing
// a vertex's two, with the Newton step of the DP0 sweep; error 3.74e-8 either way.
#pragma once

#include <type_traits>

#include "p1.cuh"
#include "rwg.cuh"
#include "warp_cols.cuh"

namespace bc {

struct TestBlockP1m {
    float e[P1_TCHUNK][3][3];    // vertex offsets kappa (v_i - c_t)
    float hge[P1_TCHUNK][2][3];  // -g_o^2 |e_i|^2 / 2 per orbit
    double c[P1_TCHUNK][3];
    double n[P1_TCHUNK][3];
    double ie[P1_TCHUNK];
    double mult[P1_TCHUNK][3];
    int64_t row[P1_TCHUNK][3];
    int v[P1_TCHUNK][3];
    float rad[P1_TCHUNK];  // MIXED_NEAR R
};

// NT, NS: test / trial functions per element, 3 (P1, DP1, RWG / SNC) or 1 (a P0 space beside a P1 one: its
// constant function takes the rule's weights in place of the P1 shape weights; scalar operators, no
// symmetric sweep).
template <int ASM, int K, int PHC, bool SYM, bool CK = false, int NT = 3, int NS = 3>
__global__ void __launch_bounds__(DP0_THREADS) regular_p1_mixed(RegParams prm, OrbitConsts oc) {
    constexpr bool LAP = K == BEMPPCUDA_LAPLACE_SLP || K == BEMPPCUDA_LAPLACE_DLP || K == BEMPPCUDA_LAPLACE_ADLP;
    constexpr bool MH = K == BEMPPCUDA_MODHELM_SLP || K == BEMPPCUDA_MODHELM_DLP || K == BEMPPCUDA_MODHELM_ADLP;
    constexpr bool REAL = LAP || MH;  // real kernel, real result
    constexpr bool HYP = ASM == BEMPPCUDA_ASM_HELM_HYP || ASM == BEMPPCUDA_ASM_LAPLACE_HYP ||
                         ASM == BEMPPCUDA_ASM_MODHELM_HYP;
    constexpr bool EFIE = ASM == BEMPPCUDA_ASM_EFIE;  // test curl slots hold J_t, multipliers edge lengths
    constexpr bool MFIE = ASM == BEMPPCUDA_ASM_MFIE;  // the same, and v0_t in the third slot
    constexpr bool RWG = EFIE || MFIE;
    constexpr bool DL = K == BEMPPCUDA_HELMHOLTZ_DLP || K == BEMPPCUDA_LAPLACE_DLP || K == BEMPPCUDA_MODHELM_DLP;
    constexpr bool AD = K == BEMPPCUDA_HELMHOLTZ_ADLP || K == BEMPPCUDA_LAPLACE_ADLP || K == BEMPPCUDA_MODHELM_ADLP;
    static_assert(!CK || !REAL, "complex wavenumber: the Helmholtz kernels");
    static_assert((NT == 3 && NS == 3) || (ASM == BEMPPCUDA_ASM_SCALAR && !SYM && (NT == 1 || NS == 1)),
                  "P0 beside P1: scalar operators, per-pair sweep");
    constexpr bool SKEW = SYM && (DL || AD);
    constexpr bool NS_SUM = DL || SKEW;  // sums multiplied by d'.n_s per test point
    constexpr bool NT_SUM = AD || SKEW;  // sums with -d'.n_t per pair
    // the FP32 sums hold the real and imaginary parts of the kernel up to these signs
    constexpr double SGR = DL || AD || MFIE ? -1.0 : 1.0, SGI = -SGR;
    __shared__ TestBlockP1m sb;
    __shared__ double scurl[HYP || RWG ? P1_TCHUNK : 1][3][3];  // curls (HYP) or J_t, v0_t (RWG)
    __shared__ WarpColumns swc[DP0_THREADS / 32];
    // staged block entries per warp: [block row][staging position]; SKEW: the (j, i) blocks too
    __shared__ double2 sst[DP0_THREADS / 32][3][WC_SLOTS];
    __shared__ double2 sst_t[SKEW ? DP0_THREADS / 32 : 1][3][SKEW ? WC_SLOTS : 1];
    // units of 1/kappa: kappa = k (Helmholtz; Re k for a complex wavenumber), omega (modified), 1 (Laplace)
    const double kap = LAP ? 1.0 : prm.p[0];
    // exp(-beta r') beside exp(i r'): beta = Im k / Re k (complex k), 1 (modified: exp(-r') alone)
    const double betd = CK ? prm.p[1] / prm.p[0] : (MH ? 1.0 : 0.0);
    const float bet = (float)betd;

    // test elements per CTA: ceil(ntest / gridDim.y) <= P1_TCHUNK (the launch picks the row blocks)
    const int rows = (int)((prm.ntest + gridDim.y - 1) / gridDim.y);
    const int64_t t0 = (int64_t)blockIdx.y * rows;
    if (SYM && t0 >= ((int64_t)blockIdx.x + 1) * DP0_THREADS) return;  // below the diagonal
    const int tcount = (int)min((int64_t)rows, prm.ntest - t0);
    for (int idx = threadIdx.x; idx < tcount; idx += blockDim.x) {
        const int64_t t = prm.tsup[t0 + idx];
        Geom g;
        load_geom(prm.tg, prm.tne, t, prm.tnm ? (double)prm.tnm[t] : 1.0, g);
        double c[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) c[d] = __ldg(prm.tg + (22 + d) * prm.tne + t);
        double eo[3][3], m2 = 0.0;
        orbit_offsets(g, eo);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
            for (int d = 0; d < 3; ++d) sb.e[idx][i][d] = (float)(kap * eo[i][d]);
            const double ee = odot(eo[i], eo[i]), m = -0.5 * kap * kap * ee;
            m2 = fmax(m2, ee);
            sb.hge[idx][0][i] = (float)(oc.gg[0] * m);
            sb.hge[idx][1][i] = (float)(oc.gg[1] * m);
        }
        sb.rad[idx] = (float)(MIXED_NEAR * kap * sqrt(m2));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            sb.c[idx][d] = c[d];
            sb.n[idx][d] = g.n[d];
            sb.v[idx][d] = __ldg(prm.tel + 3 * t + d);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            sb.mult[idx][i] = i < NT ? prm.tmult[t * NT + i] * (RWG ? edge_length(prm.tg, prm.tne, t, i) : 1.0) : 0.0;
            sb.row[idx][i] = i < NT ? prm.tl2g[t * NT + i] : 0;
        }
        if (RWG) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                scurl[idx][0][d] = g.j0[d];
                scurl[idx][1][d] = g.j1[d];
                scurl[idx][2][d] = g.v0[d];
            }
        }
        if (HYP) {
            double cu[3][3];
            surface_curls(prm.tg, prm.tne, t, g.n, cu);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int d = 0; d < 3; ++d) scurl[idx][i][d] = cu[i][d];
        }
        sb.ie[idx] = g.ie;
    }
    __syncthreads();

    const int64_t si = (int64_t)blockIdx.x * DP0_THREADS + threadIdx.x;
    const bool active = si < prm.ntrial;  // lanes past the last trial element stage nothing
    if (__all_sync(0xffffffffu, !active)) return;
    const int64_t s = prm.ssup[active ? si : prm.ntrial - 1];
    Geom gs;
    load_geom(prm.sg, prm.sne, s, prm.snm ? (double)prm.snm[s] : 1.0, gs);
    const int sv0 = __ldg(prm.sel + 3 * s), sv1 = __ldg(prm.sel + 3 * s + 1), sv2 = __ldg(prm.sel + 3 * s + 2);
    double sc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) sc[d] = __ldg(prm.sg + (22 + d) * prm.sne + s);
    // vertex offsets f_0, f_1 (f_2 = -f_0 - f_1) and -g_q^2 |f_j|^2 / 2 of both orbits
    float f[2][3];
    float2 hgf[3];
    float srad;  // MIXED_NEAR R
    {
        double fd[3][3], m2 = 0.0;
        orbit_offsets(gs, fd);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double ff = odot(fd[j], fd[j]), m = -0.5 * kap * kap * ff;
            m2 = fmax(m2, ff);
            hgf[j] = f2((float)(oc.gg[0] * m), (float)(oc.gg[1] * m));
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            f[0][d] = (float)(kap * fd[0][d]);
            f[1][d] = (float)(kap * fd[1][d]);
        }
        srad = (float)(MIXED_NEAR * kap * sqrt(m2));
    }
    // orbit constants in FP32: offsets g, and w times the linear functions at a point: the own vertex's (c + d) and
    // the other two's (d).  (c and d times the orbit's sum, as in FP64, would cancel: c < 0 in the first orbit.)
    const float go[2] = {(float)oc.g[0], (float)oc.g[1]};
    const float2 g2 = f2(go[0], go[1]);
    const float2 own2 = f2((float)(oc.c[0] + oc.d[0]), (float)(oc.c[1] + oc.d[1])), oth2 = f2((float)oc.d[0], (float)oc.d[1]);
    const float2 w2 = f2((float)oc.w[0], (float)oc.w[1]);
    const float own_[2] = {own2.x, own2.y}, oth_[2] = {oth2.x, oth2.y}, wp_[2] = {w2.x, w2.y};
    const auto fdot = [](const float a[3], float x, float y, float z) { return fmaf(a[2], z, fmaf(a[1], y, a[0] * x)); };
    const float sn0 = (float)gs.n[0], sn1 = (float)gs.n[1], sn2 = (float)gs.n[2];
    double curl_s[3][3];
    if (HYP) surface_curls(prm.sg, prm.sne, s, gs.n, curl_s);
    int64_t scol[3];
    double smul[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        scol[j] = j < NS ? prm.sl2g[s * NS + j] : -1;  // no slot past the element's functions
        smul[j] = j < NS ? prm.smult[s * NS + j] * (RWG ? edge_length(prm.sg, prm.sne, s, j) : 1.0) : 0.0;
    }
    // the warp's columns (distinct trial dofs) and this lane's staging positions
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    WarpColumns &wc = swc[warp];
    int pos[3];
    {
        int dof[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) dof[j] = active && scol[j] >= 0 && scol[j] < INT32_MAX ? (int)scol[j] : -1;
        static_assert(sizeof(sst[0]) >= 2 * WC_TABLE * sizeof(int), "column table scratch");
        wc_build(wc, reinterpret_cast<int *>(&sst[warp][0][0]), dof, pos);
    }
    double2(&st)[3][WC_SLOTS] = sst[warp];
    double2(&st_t)[3][SKEW ? WC_SLOTS : 1] = sst_t[SKEW ? warp : 0];

    // one test element: the blocks of the warp's pairs (has: this lane has one), staged and added per column
    const auto row = [&](int tt, bool has, double D0, double D1, double D2, auto near_) {
        constexpr bool NEAR = decltype(near_)::value;
        if (!has) {
            // no pair: zeros in this lane's staging positions
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    if (pos[j] >= 0) {
                        st[i][pos[j]] = make_double2(0.0, 0.0);
                        if (SKEW) st_t[i][pos[j]] = make_double2(0.0, 0.0);
                    }
        } else {
        const double rc2 = fma(D2, D2, fma(D1, D1, D0 * D0));
        const double rc = sqrt(rc2);
        // the element pair's factor: exp(i r_c'), times exp(-beta r_c') (complex k); exp(-r_c') (modified)
        double ph_s = 0.0, ph_c = 1.0;
        if (!LAP) {
            if (!MH) sincos_cw64(rc, &ph_s, &ph_c);
            if (MH || CK) {
                const double am = exp(-betd * rc);
                ph_c *= am;
                ph_s *= am;
            }
        }
        const float D0f = (float)D0, D1f = (float)D1, D2f = (float)D2;
        const float rcf = (float)rc;
        const float2 rc_2 = b2(rcf), mrc_2 = b2(-rcf), mrc2_2 = b2(-(float)rc2);
        // normal terms: D . n_s; -(d'.n_t) = -(D . n_t) - g_q f_j . n_t per trial point
        const float Dns = NS_SUM ? fmaf(D2f, sn2, fmaf(D1f, sn1, D0f * sn0)) : 0.f;
        float2 cm[3] = {b2(0.f), b2(0.f), b2(0.f)};
        if (NT_SUM) {
            const float tn0 = (float)sb.n[tt][0], tn1 = (float)sb.n[tt][1], tn2 = (float)sb.n[tt][2];
            const float2 mDt = b2(-fmaf(D2f, tn2, fmaf(D1f, tn1, D0f * tn0)));
            const float m0 = -fdot(f[0], tn0, tn1, tn2), m1 = -fdot(f[1], tn0, tn1, tn2);
            cm[0] = fma2(b2(m0), g2, mDt);
            cm[1] = fma2(b2(m1), g2, mDt);
            cm[2] = fma2(b2(-(m0 + m1)), g2, mDt);
        }
        // (re, im) blocks: the block of (i, j): single layer, or its double layer; SKEW: the transposed pair's
        float2 l[NT][NS], u[SKEW ? NT : 1][SKEW ? NS : 1];
        const auto axpy = [](float a, float2 x, float2 y) -> float2 {
            return REAL ? f2(fmaf(a, x.x, y.x), 0.f) : fma2(b2(a), x, y);
        };
#pragma unroll
        for (int a = 0; a < NT; ++a)
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                l[a][j] = b2(0.f);
                if (SKEW) u[a % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)] = b2(0.f);
            }
        float2 hA[3];  // -A_q / 2
        if (!NEAR) {
            const float a0 = -fdot(f[0], D0f, D1f, D2f), a1 = -fdot(f[1], D0f, D1f, D2f);
            hA[0] = fma2(b2(a0), g2, hgf[0]);
            hA[1] = fma2(b2(a1), g2, hgf[1]);
            hA[2] = fma2(b2(-(a0 + a1)), g2, hgf[2]);
        }
        float E[3][3], De[3], en[3] = {0.f, 0.f, 0.f};  // e_i . f_j, D . e_i, e_i . n_s
        if (!NEAR) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float e0 = sb.e[tt][i][0], e1 = sb.e[tt][i][1], e2 = sb.e[tt][i][2];
                De[i] = fmaf(D2f, e2, fmaf(D1f, e1, D0f * e0));
                if (NS_SUM) en[i] = fmaf(sn2, e2, fmaf(sn1, e1, sn0 * e0));
                E[i][0] = fdot(f[0], e0, e1, e2);
                E[i][1] = fdot(f[1], e0, e1, e2);
                E[i][2] = -(E[i][0] + E[i][1]);
            }
            De[2] = -(De[0] + De[1]);
            if (NS_SUM) en[2] = -(en[0] + en[1]);
#pragma unroll
            for (int j = 0; j < 3; ++j) E[2][j] = -(E[0][j] + E[1][j]);
        }
#pragma unroll (NEAR ? 1 : NQ6)
        for (int p = 0; p < NQ6; ++p) {
            const int i = p % 3, op = p / 3;
            const float gp = op == 0 ? go[0] : go[1];
            float x[3];  // NEAR: D - g_p e_i
            float2 hB, gp2;
            if (NEAR) {
                x[0] = fmaf(-gp, sb.e[tt][i][0], D0f);
                x[1] = fmaf(-gp, sb.e[tt][i][1], D1f);
                x[2] = fmaf(-gp, sb.e[tt][i][2], D2f);
            } else {
                hB = b2(fmaf(gp, De[i], sb.hge[tt][op][i]));  // -B_p / 2
                gp2 = f2(gp * go[0], gp * go[1]);
            }
            float2 kr[3], ki[3];
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
                const float2 mrp = mul2(mr2, rinv);  // -r'
                // cs - i ms: exp(i theta) (Helmholtz), times exp(-beta theta) (complex k); exp(-theta)
                // (modified, ms = 0); 1 (Laplace)
                float2 ms = b2(0.f), cs = b2(1.f);
                if (!LAP) {
                    float2 mt = fma2(mr2, rinv, rc_2);  // -theta
                    if (!NEAR) mt = fma2(fma2(mt, fma2(mt, b2(0.5f), mrc_2), hs), rinv, mt);
                    if (!MH) sincos2<PHC>(mt, &ms, &cs);
                    if (MH || CK) {
                        const float2 am = f2(__expf(bet * mt.x), __expf(bet * mt.y));
                        cs = mul2(cs, am);
                        if (CK) ms = mul2(ms, am);
                    }
                }
                ki[j] = b2(0.f);
                if (!DL && !AD && !MFIE) {
                    kr[j] = mul2(rinv, cs);
                    if (!REAL) ki[j] = mul2(rinv, ms);
                } else {
                    // -Re and Im of (ikr - 1) e^{ikr} / r^3 in units of 1/kappa: (a cs + r' sn, r' cs - a sn) / r'^3,
                    // a = 1 + beta r' (a = 1 for real k); modified: (1 + r') e^{-r'} / r'^3
                    const float2 r3 = mul2(rinv, mul2(rinv, rinv));
                    if (LAP) {
                        kr[j] = r3;
                    } else if (MH) {
                        kr[j] = mul2(mul2(r3, cs), fma2(mrp, b2(-1.f), b2(1.f)));
                    } else {
                        const float2 rp = mul2(mrp, b2(-1.f));
                        if (CK) {
                            const float2 a = fma2(b2(bet), rp, b2(1.f));
                            kr[j] = mul2(r3, fma2(mrp, ms, mul2(a, cs)));
                            ki[j] = mul2(r3, fma2(rp, cs, mul2(a, ms)));
                        } else {
                            kr[j] = mul2(r3, fma2(mrp, ms, cs));
                            ki[j] = mul2(r3, fma2(rp, cs, ms));
                        }
                    }
                }
            }
            // the trial sums of each test point: T_j (plain) and V_j (with -(d'.n_t))
            const auto sums = [&](const float2 *k, int j) -> float {
                float2 v;
                if (NS == 3)
                    v = fma2(k[j], own2, mul2(add2(k[(j + 1) % 3], k[(j + 2) % 3]), oth2));
                else
                    v = mul2(add2(add2(k[0], k[1]), k[2]), w2);
                return v.x + v.y;
            };
            float2 T[NS], V[NS];
            if (!AD || SKEW)
#pragma unroll
                for (int j = 0; j < NS; ++j) T[j] = f2(sums(kr, j), REAL ? 0.f : sums(ki, j));
            if (NT_SUM) {
                float2 vr[3], vi[3];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    vr[j] = mul2(kr[j], cm[j]);
                    vi[j] = REAL ? b2(0.f) : mul2(ki[j], cm[j]);
                }
#pragma unroll
                for (int j = 0; j < NS; ++j) V[j] = f2(sums(vr, j), REAL ? 0.f : sums(vi, j));
            }
            // into the blocks: (i, j) double layer -> T times d'.n_s, adjoint -> V; SKEW: the other one at (j, i)
            const float dns = !NS_SUM ? 1.f : NEAR ? fdot(x, sn0, sn1, sn2) : fmaf(-gp, en[i], Dns);
#pragma unroll
            for (int a = 0; a < NT; ++a) {
                const float w = op == 0 ? (NT == 1 ? wp_[0] : a == i ? own_[0] : oth_[0])
                                        : (NT == 1 ? wp_[1] : a == i ? own_[1] : oth_[1]);
                const float wn = NS_SUM ? w * dns : w;
#pragma unroll
                for (int j = 0; j < NS; ++j) {
                    l[a][j] = axpy(DL ? wn : w, AD ? V[j] : T[j], l[a][j]);
                    if (SKEW) {
                        constexpr int A_ = SKEW ? NT : 1, B_ = SKEW ? NS : 1;
                        u[a % A_][j % B_] = axpy(DL ? w : wn, DL ? V[j] : T[j], u[a % A_][j % B_]);
                    }
                }
            }
        }
        float lre[3][3], lim[3][3], ure[3][3], uim[3][3];
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const float2 v = l[i][j];
                lre[i][j] = v.x;
                lim[i][j] = v.y;
                if (SKEW) {
                    const float2 w = u[i % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)];
                    ure[i][j] = w.x;
                    uim[i][j] = w.y;
                }
            }
        // k / (4 pi) or k^2 / (4 pi), |J_t| |J_s| exp(i r_c'), then the hypersingular combination;
        // EFIE: the moments, k (4 pi G = k e^{i theta} / r' in these units) and 1 / (4 pi), no |J|
        double ere[3][3], eim[3][3];
        if (EFIE) {
            double mre[3][3], mim[3][3];
            double rs[3] = {0.0, 0.0, 0.0}, is[3] = {0.0, 0.0, 0.0};  // sums over j (row sums)
            double cs_[3] = {0.0, 0.0, 0.0}, ci_[3] = {0.0, 0.0, 0.0};  // sums over i (column sums)
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const double lr = SGR * kap * (double)lre[i][j], li = SGI * kap * (double)lim[i][j];
                    rs[i] += lr;
                    is[i] += li;
                    cs_[j] += lr;
                    ci_[j] += li;
                }
            mre[0][0] = rs[0] + rs[1] + rs[2];
            mim[0][0] = is[0] + is[1] + is[2];
#pragma unroll
            for (int a = 1; a < 3; ++a) {
                mre[a][0] = rs[a];
                mim[a][0] = is[a];
                mre[0][a] = cs_[a];
                mim[0][a] = ci_[a];
#pragma unroll
                for (int b = 1; b < 3; ++b) {
                    mre[a][b] = SGR * kap * (double)lre[a][b];
                    mim[a][b] = SGI * kap * (double)lim[a][b];
                }
            }
            efie_block<CK>(mre, mim, scurl[tt][0], scurl[tt][1], gs.j0, gs.j1, kap, CK ? prm.p[1] : 0.0, ere, eim);
        } else if (MFIE) {
            // the moments of H = k^3 h (units of 1/k), then the block from the FP64 geometry
            const double k3 = kap * kap * kap;
            double mre[3][3], mim[3][3];
            double rs[3] = {0.0, 0.0, 0.0}, is[3] = {0.0, 0.0, 0.0};
            double cs_[3] = {0.0, 0.0, 0.0}, ci_[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const double lr = SGR * k3 * (double)lre[i][j], li = SGI * k3 * (double)lim[i][j];
                    rs[i] += lr;
                    is[i] += li;
                    cs_[j] += lr;
                    ci_[j] += li;
                    if (i > 0 && j > 0) {
                        mre[i][j] = lr;
                        mim[i][j] = li;
                    }
                }
            mre[0][0] = rs[0] + rs[1] + rs[2];
            mim[0][0] = is[0] + is[1] + is[2];
#pragma unroll
            for (int a = 1; a < 3; ++a) {
                mre[a][0] = rs[a];
                mim[a][0] = is[a];
                mre[0][a] = cs_[a];
                mim[0][a] = ci_[a];
            }
            mfie_block_moments(mre, mim, scurl[tt][2], scurl[tt][0], scurl[tt][1], gs.v0, gs.j0, gs.j1, ere, eim);
        }
        const double scale = RWG ? BC_INV_4PI : (DL || AD ? kap * kap : kap) * BC_INV_4PI * sb.ie[tt] * gs.ie;
        double sre = 0.0, sim = 0.0, cpf = 0.0, cpi = 0.0;
        if (HYP) {
            // S = sum_pq w_p w_q G: the P1 functions add up to 1 on each side
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    sre += SGR * (double)lre[i][j];
                    sim += SGI * (double)lim[i][j];
                }
            // -k^2 (n_t . n_s), complex for a complex wavenumber; +w^2 (n_t . n_s) modified; 0 Laplace
            const double nn = sb.n[tt][0] * gs.n[0] + sb.n[tt][1] * gs.n[1] + sb.n[tt][2] * gs.n[2];
            if (MH) {
                cpf = kap * kap * nn;
            } else if (!LAP) {
                const double ki = CK ? prm.p[1] : 0.0;
                cpf = -(kap * kap - ki * ki) * nn;
                cpi = -2.0 * kap * ki * nn;
            }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const double mt = sb.mult[tt][i];
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const double ms = smul[j];
                if (pos[j] < 0) continue;
                if (mt == 0.0 || ms == 0.0) {
                    st[i][pos[j]] = make_double2(0.0, 0.0);
                    if (SKEW) st_t[i][pos[j]] = make_double2(0.0, 0.0);
                    continue;
                }
                double vr = RWG ? ere[i][j] : SGR * (double)lre[i][j], vi = RWG ? eim[i][j] : SGI * (double)lim[i][j];
                if (HYP) {
                    const double cij = scurl[tt][i][0] * curl_s[j][0] + scurl[tt][i][1] * curl_s[j][1] +
                                       scurl[tt][i][2] * curl_s[j][2];
                    const double lr = vr, li = vi;
                    vr = fma(cij, sre, fma(cpf, lr, -cpi * li));
                    vi = fma(cij, sim, fma(cpf, li, cpi * lr));
                }
                const double tr = vr * ph_c - vi * ph_s;
                vi = fma(vr, ph_s, vi * ph_c);
                vr = tr;
                double wr = vr, wi = vi;  // the (j, i) block: the same, or (SKEW) its own sums
                if (SKEW) {
                    const double ur = SGR * (double)ure[i][j], ui = SGI * (double)uim[i][j];
                    wr = ur * ph_c - ui * ph_s;
                    wi = fma(ur, ph_s, ui * ph_c);
                }
                const double mm = mt * ms * scale;
                st[i][pos[j]] = make_double2(vr * mm, vi * mm);
                if (SKEW) st_t[i][pos[j]] = make_double2(wr * mm, wi * mm);
            }
        }
        }  // pair
        __syncwarp();
        // per (test dof, column): the sum of the column's staged entries, one complex atomic
        // (and, for the symmetric sweep, one at the transposed position)
        const int ncols = wc.ncols;
        double *res = reinterpret_cast<double *>(prm.result);
        // one entry into the matrix: complex (two atomics) or, for the real kernels, real
        const auto add_entry = [](double *m, int64_t ld, int64_t r, int64_t c, double re, double im) {
            if (REAL) {
                atomicAdd(m + r * ld + c, re);
            } else {
                atomicAdd(m + 2 * (r * ld + c), re);
                atomicAdd(m + 2 * (r * ld + c) + 1, im);
            }
        };
        // the rows of a column are summed together: one walk over its staging positions
        for (int c = (int)lane; c < ncols; c += 32) {
            const int b = wc.start[c], e = wc.start[c + 1];
            double ar[NT], ai[NT], br[NT], bi[NT];
#pragma unroll
            for (int i = 0; i < NT; ++i) ar[i] = ai[i] = br[i] = bi[i] = 0.0;
            for (int k = b; k < e; ++k) {
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const double2 v = st[i][k];
                    ar[i] += v.x;
                    if (!REAL) ai[i] += v.y;
                    if (SKEW) {
                        const double2 w = st_t[i][k];
                        br[i] += w.x;
                        if (!REAL) bi[i] += w.y;
                    }
                }
            }
            const int64_t col = wc.col[c];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int64_t row = sb.row[tt][i];
                if (ar[i] != 0.0 || ai[i] != 0.0) {
                    add_entry(res, prm.ld, row, col, ar[i], ai[i]);
                    if (SYM && !SKEW && !prm.defer_transpose) add_entry(res, prm.ld, col, row, ar[i], ai[i]);
                }
                if (SKEW && (br[i] != 0.0 || bi[i] != 0.0)) add_entry(res, prm.ld, col, row, br[i], bi[i]);
            }
        }
        __syncwarp();  // the staging arrays are rewritten by the next test element
    };

    static_assert(P1_TCHUNK <= 32, "a bit per row");
    uint32_t near_rows = 0;  // left for after the sweep, whose registers and schedule stay its own
    for (int tt = 0; tt < tcount; ++tt) {
        const bool done = !active || (SYM && t0 + tt >= si);  // rows increase with tt
        if (__all_sync(0xffffffffu, done)) break;
        bool has = !done && !(prm.grids_identical && shares_vertex(sb.v[tt], sv0, sv1, sv2));
        const double D0 = kap * (sc[0] - sb.c[tt][0]), D1 = kap * (sc[1] - sb.c[tt][1]),
                     D2 = kap * (sc[2] - sb.c[tt][2]);
        const float rs = sb.rad[tt] + srad;
        if (has && (float)fma(D2, D2, fma(D1, D1, D0 * D0)) < rs * rs) {
            near_rows |= 1u << tt;
            has = false;
        }
        row(tt, has, D0, D1, D2, std::false_type());
    }
    for (uint32_t rows_ = __reduce_or_sync(0xffffffffu, near_rows); rows_ != 0; rows_ &= rows_ - 1) {
        const int tt = __ffs(rows_) - 1;
        row(tt, (near_rows >> tt) & 1u, kap * (sc[0] - sb.c[tt][0]), kap * (sc[1] - sb.c[tt][1]),
            kap * (sc[2] - sb.c[tt][2]), std::true_type());
    }
}

}  // namespace bc
