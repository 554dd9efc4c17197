// Regular pairs of scalar operators on linear (P1 / DP1) and mixed P0 / P1
// spaces in the orbit form (two-orbit 6-point rule): the kernels of
// numba_kernels.py:980-1074 (default_scalar_regular_kernel) and the
// hypersingular ones of :1078-1467, for a complex wavenumber, modified
// Helmholtz, the Laplace double layers and the Helmholtz hypersingular
// operator (the others are faster in the points form, p1_points.cuh).
//
// One thread per trial element, up to 32 test elements staged in shared memory
// (as the DP0 tiles); the point sums of an element pair are orbit_moments /
// orbit_double (orbit_pair.cuh): distances from vertex dot products, the phase
// and amplitude split about the centroid distance by offset class, moments
// from orbit sums.  Hypersingular operators reuse the single-layer moments:
// with constant surface curls per element,
//   L_ij = (curl_i . curl_j) S - c (n_t . n_s) M_ij,  S = sum_ij M_ij
// (the P1 shape functions add up to 1), c = k^2 (Helmholtz, complex for a
// complex wavenumber), 0 (Laplace), -w^2 (modified Helmholtz).
// The NT x NS block is added to the matrix with FP64 atomics (l2g, multipliers).
// SYM (the same space on both sides): only pairs i < j (support positions) are
// evaluated and each gives the blocks at (i, j) and (j, i).  Single layer and
// hypersingular: the kernel is symmetric in x and y and so is the curl
// product, so the second block is the transpose of the first; into a zeroed
// result (defer_transpose) only the first is added and the host forms
// A = U + U^T afterwards (the regular diagonal is zero: a pair that reaches
// entry (I, I) shares vertex I and is singular).  Double and adjoint double
// layer: the double layer of the transposed pair (test j, trial i) is the
// adjoint double layer of (i, j), so both blocks share the values of
// H = (ikr - 1) e^{ikr} / r^3 and differ in the normal factor.
// Bound by the FP64 pipe (69 % in the hypersingular sweep, 72 % in the single layer with
// a complex wavenumber; an FMA of three unshared registers issues at 72 % of its peak).  8192 elements, points form before -> orbit form:
// Helmholtz hypersingular k = 5 4.27 -> 4.05 ms, double layer k = 3 + 0.3i
// 11.0 -> 7.4 ms, modified Helmholtz single / double / hypersingular 4.20 ->
// 3.16, 5.51 -> 4.31, 4.56 -> 3.39 ms, Laplace double layer 2.91 -> 2.80 ms.
#pragma once

#include "dp0.cuh"
#include "orbit_pair.cuh"

namespace bc {

constexpr int P1_TCHUNK = 32;

struct TestBlockP1 {
    OrbitTest o[P1_TCHUNK];
    double n[P1_TCHUNK][3];
    double curl[P1_TCHUNK][3][3];
    double ie[P1_TCHUNK];
    double mult[P1_TCHUNK][3];  // local multipliers of the test functions
    int64_t row[P1_TCHUNK][3];  // their global dofs
    int v[P1_TCHUNK][3];
};

// CTAs per SM the P1 kernel is compiled for: 3 (168 registers); 2 for the skew sweeps of the Helmholtz double
// layers (complex wavenumbers), whose two complex blocks would spill.
template <int K, bool SYM>
constexpr int p1_min_blocks() {
    return SYM && (K == BEMPPCUDA_HELMHOLTZ_DLP || K == BEMPPCUDA_HELMHOLTZ_ADLP) ? 2 : 3;
}

// CLS: offset class (fastmath.cuh); CK: complex wavenumber.
template <int ASM, int K, int NT, int NS, int CLS, bool CK, bool SYM>
__global__ void __launch_bounds__(DP0_THREADS, (p1_min_blocks<K, SYM>())) regular_p1(RegParams prm, OrbitConsts oc) {
    constexpr bool HYP = (ASM == BEMPPCUDA_ASM_LAPLACE_HYP || ASM == BEMPPCUDA_ASM_HELM_HYP ||
                          ASM == BEMPPCUDA_ASM_MODHELM_HYP);
    constexpr int FAM = kernel_family<K>();
    constexpr bool DL = (K == BEMPPCUDA_LAPLACE_DLP || K == BEMPPCUDA_HELMHOLTZ_DLP || K == BEMPPCUDA_MODHELM_DLP);
    constexpr bool AD = (K == BEMPPCUDA_LAPLACE_ADLP || K == BEMPPCUDA_HELMHOLTZ_ADLP || K == BEMPPCUDA_MODHELM_ADLP);
    static_assert(!SYM || NT == NS, "the symmetric sweep needs one space on both sides");
    constexpr bool SKEW = SYM && (DL || AD);  // the transposed block uses the other element's normal
    __shared__ TestBlockP1 sb;
    // the trial element's fields, then (hypersingular) its curls, the multipliers and dofs of its functions
    constexpr int CURL = OT_FIELDS, MULT = CURL + (HYP ? 9 : 0), COL = MULT + NS, FIELDS = COL + NS;
    __shared__ double park[FIELDS][DP0_THREADS];

    // test elements per CTA: ceil(ntest / gridDim.y) <= P1_TCHUNK (the launch picks the row blocks)
    const int rows = (int)((prm.ntest + gridDim.y - 1) / gridDim.y);
    const int64_t t0 = (int64_t)blockIdx.y * rows;
    if (SYM && t0 >= ((int64_t)blockIdx.x + 1) * DP0_THREADS) return;  // below the diagonal
    const int tcount = (int)min((int64_t)rows, prm.ntest - t0);
    for (int idx = threadIdx.x; idx < tcount; idx += blockDim.x) {
        const int64_t t = prm.tsup[t0 + idx];
        Geom g;
        load_geom(prm.tg, prm.tne, t, prm.tnm ? (double)prm.tnm[t] : 1.0, g);
        stage_orbit(prm.tg, prm.tne, t, g, oc, sb.o[idx]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            sb.n[idx][d] = g.n[d];
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
    const OrbitTrial<DP0_THREADS> tr = park_orbit_trial<DP0_THREADS>(prm.sg, prm.sne, s, gs, &park[0][0]);
    if (HYP) {
        double cu[3][3];
        surface_curls(prm.sg, prm.sne, s, gs.n, cu);
#pragma unroll
        for (int d = 0; d < 9; ++d) park[(CURL + d) % FIELDS][threadIdx.x] = cu[d / 3][d % 3];
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        park[MULT + j][threadIdx.x] = prm.smult[s * NS + j];
        park[COL + j][threadIdx.x] = __longlong_as_double((int64_t)prm.sl2g[s * NS + j]);
    }
    orbit_fence();
    const double kr = prm.p[0], ki = CK ? prm.p[1] : 0.0;

#pragma unroll 1
    for (int tt = 0; tt < tcount; ++tt) {
        if (SYM && t0 + tt >= si) break;  // rows increase with tt
        if (prm.grids_identical && shares_vertex(sb.v[tt], sv0, sv1, sv2)) continue;
        const OrbitTest &te = sb.o[tt];
        OrbitPair pair;
        orbit_pair<FAM, CK, CLS>(te, tr, oc, kr, ki, pair);
        double lre[NT][NS], lim[NT][NS];  // block of (i, j)
        double ure[SKEW ? NT : 1][SKEW ? NS : 1], uim[SKEW ? NT : 1][SKEW ? NS : 1];  // SKEW: block of (j, i)
        if constexpr (DL || AD) {
            // the double layer takes the trial normal (U), the adjoint double layer the test normal (V); the
            // transposed pair's block is the other of the two
            const double tn[3] = {sb.n[tt][0], sb.n[tt][1], sb.n[tt][2]};
            if constexpr (SKEW && DL)
                orbit_double<true, true, FAM, CK, CLS, NT, NS>(te, tn, tr, pair, oc, kr, ki, lre, lim, ure, uim);
            else if constexpr (SKEW)
                orbit_double<true, true, FAM, CK, CLS, NT, NS>(te, tn, tr, pair, oc, kr, ki, ure, uim, lre, lim);
            else
                orbit_double<DL, AD, FAM, CK, CLS, NT, NS>(te, tn, tr, pair, oc, kr, ki, lre, lim, lre, lim);
        } else {
            orbit_moments<false, FAM, CK, CLS, NT, NS>(te, tr, pair, oc, kr, ki, lre, lim);
        }
        double ph_c, ph_s;
        orbit_phase<FAM, CK, CLS>(pair, ph_c, ph_s);
        const double scale = BC_INV_4PI * sb.ie[tt] * tr.ld(OT_IE);
        ph_c *= scale;
        ph_s *= scale;
        // hypersingular: the sum of the moments, and -k^2 (n_t . n_s), complex for a complex wavenumber;
        // +w^2 (n_t . n_s) modified
        double sre = 0.0, sim = 0.0, cpf = 0.0, cpi = 0.0;
        if (HYP) {
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int j = 0; j < NS; ++j) {
                    sre += lre[i][j];
                    sim += lim[i][j];
                }
            double sn[3];
            tr.n(sn);
            const double nn = odot(sb.n[tt], sn);
            if (ASM == BEMPPCUDA_ASM_HELM_HYP) {
                cpf = -(kr * kr - ki * ki) * nn;
                cpi = -2.0 * kr * ki * nn;
            } else if (ASM == BEMPPCUDA_ASM_MODHELM_HYP) {
                cpf = kr * kr * nn;
            }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const double mt = sb.mult[tt][i];
            if (mt == 0.0) continue;
            const int64_t row = sb.row[tt][i];
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const double ms = tr.ld(MULT + j);
                if (ms == 0.0) continue;
                double vr = lre[i][j], vi = lim[i][j];
                if (HYP) {
                    const double cs[3] = {tr.ld(CURL + 3 * j), tr.ld(CURL + 3 * j + 1), tr.ld(CURL + 3 * j + 2)};
                    const double cij = odot(sb.curl[tt][i], cs);
                    const double lr = vr, li = vi;
                    vr = fma(cij, sre, fma(cpf, lr, CK ? -cpi * li : 0.0));
                    vi = fma(cij, sim, fma(cpf, li, CK ? cpi * lr : 0.0));
                }
                const double m = mt * ms, cm = ph_c * m, sm = ph_s * m;
                const int64_t col = tr.li(COL + j);
                const double ar = FAM == FAM_HELM ? fma(vr, cm, -vi * sm) : vr * cm;
                const double ai = FAM == FAM_HELM ? fma(vr, sm, vi * cm) : 0.0;
                double br = ar, bi = ai;
                if (SKEW) {
                    const double wr = ure[i % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)];
                    const double wi = uim[i % (SKEW ? NT : 1)][j % (SKEW ? NS : 1)];
                    br = FAM == FAM_HELM ? fma(wr, cm, -wi * sm) : wr * cm;
                    bi = FAM == FAM_HELM ? fma(wr, sm, wi * cm) : 0.0;
                }
                if (prm.is_complex) {
                    double *o = reinterpret_cast<double *>(prm.result) + 2 * (row * prm.ld + col);
                    atomicAdd(o, ar);
                    atomicAdd(o + 1, ai);
                    if (SYM && (SKEW || !prm.defer_transpose)) {
                        double *ot = reinterpret_cast<double *>(prm.result) + 2 * (col * prm.ld + row);
                        atomicAdd(ot, br);
                        atomicAdd(ot + 1, bi);
                    }
                } else {
                    atomicAdd(reinterpret_cast<double *>(prm.result) + row * prm.ld + col, ar);
                    if (SYM && (SKEW || !prm.defer_transpose))
                        atomicAdd(reinterpret_cast<double *>(prm.result) + col * prm.ld + row, br);
                }
            }
        }
    }
}

}  // namespace bc
