// Regular pairs of scalar and hypersingular operators on P1 / DP1 / P0 spaces in FP64 (p1.cuh).
#include "p1.cuh"
#include "p1_points.cuh"
#include "regular.cuh"

namespace bc {

template <int ASM, int K, int NT, int NS, bool SYM>
static void launch_p1_class(const RegParams &prm, const OrbitConsts &oc, int cls, dim3 grid, cudaStream_t st) {
    // the offset classes concern exp(ikr) and exp(-w r): one instance for Laplace
    if constexpr (kernel_family<K>() == FAM_LAPLACE) {
        regular_p1<ASM, K, NT, NS, 0, false, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
        return;
    } else if constexpr (kernel_family<K>() == FAM_HELM) {
        if (prm.p[1] != 0.0) {
            if (cls == 2)
                regular_p1<ASM, K, NT, NS, 2, true, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
            else if (cls == 1)
                regular_p1<ASM, K, NT, NS, 1, true, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
            else
                regular_p1<ASM, K, NT, NS, 0, true, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
            return;
        }
    }
    // (the Helmholtz layers with a real wavenumber take the points form)
    if constexpr (kernel_family<K>() == FAM_MODHELM || ASM == BEMPPCUDA_ASM_HELM_HYP) {
        if (cls == 2)
            regular_p1<ASM, K, NT, NS, 2, false, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
        else if (cls == 1)
            regular_p1<ASM, K, NT, NS, 1, false, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
        else
            regular_p1<ASM, K, NT, NS, 0, false, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
    }
}

// single layer and hypersingular: symmetric; double / adjoint double layer: each pair
// also gives the transposed pair's block from the other normal (p1.cuh)
template <int ASM, int K>
static cudaError_t launch_p1(const RegParams &prm, const OrbitConsts &oc, int cls, bool sym, cudaStream_t st) {
    constexpr bool HYP = ASM != BEMPPCUDA_ASM_SCALAR;
    const dim3 grid((unsigned)((prm.ntrial + DP0_THREADS - 1) / DP0_THREADS),
                    lin_row_blocks(prm.ntrial, prm.ntest, sym));
    const int nt = prm.tnshape, ns = prm.snshape;
    if (nt == 3 && ns == 3) {
        if (sym)
            launch_p1_class<ASM, K, 3, 3, true>(prm, oc, cls, grid, st);
        else
            launch_p1_class<ASM, K, 3, 3, false>(prm, oc, cls, grid, st);
    } else if constexpr (!HYP) {
        if (nt == 3)
            launch_p1_class<ASM, K, 3, 1, false>(prm, oc, cls, grid, st);
        else if (ns == 3)
            launch_p1_class<ASM, K, 1, 3, false>(prm, oc, cls, grid, st);
        else if (sym)
            launch_p1_class<ASM, K, 1, 1, true>(prm, oc, cls, grid, st);
        else
            launch_p1_class<ASM, K, 1, 1, false>(prm, oc, cls, grid, st);
    }
    return cudaGetLastError();
}

// The points form (p1_points.cuh): Laplace single layer and hypersingular, Helmholtz layers for a real wavenumber.
template <int ASM, int K, int NT, int NS, bool SYM>
static void launch_points_class(const RegParams &prm, const QuadRule &rule, int cls, dim3 grid, cudaStream_t st) {
    if constexpr (kernel_family<K>() == FAM_HELM) {
        if (cls == 2) {
            regular_p1_points<ASM, K, NT, NS, 2, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
            return;
        }
        if (cls == 1) {
            regular_p1_points<ASM, K, NT, NS, 1, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
            return;
        }
    }
    regular_p1_points<ASM, K, NT, NS, 0, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
}

template <int ASM, int K>
static cudaError_t launch_points(const RegParams &prm, const QuadRule &rule, int cls, bool sym, cudaStream_t st) {
    const dim3 grid((unsigned)((prm.ntrial + DP0_THREADS - 1) / DP0_THREADS),
                    lin_row_blocks(prm.ntrial, prm.ntest, sym));
    const int nt = prm.tnshape, ns = prm.snshape;
    if (nt == 3 && ns == 3) {
        if (sym)
            launch_points_class<ASM, K, 3, 3, true>(prm, rule, cls, grid, st);
        else
            launch_points_class<ASM, K, 3, 3, false>(prm, rule, cls, grid, st);
    } else if constexpr (ASM == BEMPPCUDA_ASM_SCALAR) {
        if (nt == 3)
            launch_points_class<ASM, K, 3, 1, false>(prm, rule, cls, grid, st);
        else if (ns == 3)
            launch_points_class<ASM, K, 1, 3, false>(prm, rule, cls, grid, st);
        else if (sym)
            launch_points_class<ASM, K, 1, 1, true>(prm, rule, cls, grid, st);
        else
            launch_points_class<ASM, K, 1, 1, false>(prm, rule, cls, grid, st);
    }
    return cudaGetLastError();
}

// The operators of the points form; the others need the two-orbit rule.
bool p1_points_form(int assembly, int kernel, const double *params) {
    if (assembly == BEMPPCUDA_ASM_LAPLACE_HYP) return true;
    if (assembly != BEMPPCUDA_ASM_SCALAR) return false;
    if (kernel == BEMPPCUDA_LAPLACE_SLP) return true;
    return params[1] == 0.0 && (kernel == BEMPPCUDA_HELMHOLTZ_SLP || kernel == BEMPPCUDA_HELMHOLTZ_DLP ||
                                kernel == BEMPPCUDA_HELMHOLTZ_ADLP);
}

cudaError_t launch_p1_kernel(int assembly, int kernel, const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc,
                             int cls, bool sym, cudaStream_t st) {
    if (assembly == BEMPPCUDA_ASM_LAPLACE_HYP)
        return launch_points<BEMPPCUDA_ASM_LAPLACE_HYP, BEMPPCUDA_LAPLACE_SLP>(prm, rule, cls, sym, st);
    if (assembly == BEMPPCUDA_ASM_HELM_HYP)
        return launch_p1<BEMPPCUDA_ASM_HELM_HYP, BEMPPCUDA_HELMHOLTZ_SLP>(prm, oc, cls, sym, st);
    if (assembly == BEMPPCUDA_ASM_MODHELM_HYP)
        return launch_p1<BEMPPCUDA_ASM_MODHELM_HYP, BEMPPCUDA_MODHELM_SLP>(prm, oc, cls, sym, st);
    const bool points = p1_points_form(assembly, kernel, prm.p);
    switch (kernel) {
    case BEMPPCUDA_LAPLACE_SLP: return launch_points<0, BEMPPCUDA_LAPLACE_SLP>(prm, rule, cls, sym, st);
    case BEMPPCUDA_LAPLACE_DLP: return launch_p1<0, BEMPPCUDA_LAPLACE_DLP>(prm, oc, cls, sym, st);
    case BEMPPCUDA_LAPLACE_ADLP: return launch_p1<0, BEMPPCUDA_LAPLACE_ADLP>(prm, oc, cls, sym, st);
    case BEMPPCUDA_HELMHOLTZ_SLP:
        return points ? launch_points<0, BEMPPCUDA_HELMHOLTZ_SLP>(prm, rule, cls, sym, st)
                      : launch_p1<0, BEMPPCUDA_HELMHOLTZ_SLP>(prm, oc, cls, sym, st);
    case BEMPPCUDA_HELMHOLTZ_DLP:
        return points ? launch_points<0, BEMPPCUDA_HELMHOLTZ_DLP>(prm, rule, cls, sym, st)
                      : launch_p1<0, BEMPPCUDA_HELMHOLTZ_DLP>(prm, oc, cls, sym, st);
    case BEMPPCUDA_HELMHOLTZ_ADLP:
        return points ? launch_points<0, BEMPPCUDA_HELMHOLTZ_ADLP>(prm, rule, cls, sym, st)
                      : launch_p1<0, BEMPPCUDA_HELMHOLTZ_ADLP>(prm, oc, cls, sym, st);
    case BEMPPCUDA_MODHELM_SLP: return launch_p1<0, BEMPPCUDA_MODHELM_SLP>(prm, oc, cls, sym, st);
    case BEMPPCUDA_MODHELM_DLP: return launch_p1<0, BEMPPCUDA_MODHELM_DLP>(prm, oc, cls, sym, st);
    case BEMPPCUDA_MODHELM_ADLP: return launch_p1<0, BEMPPCUDA_MODHELM_ADLP>(prm, oc, cls, sym, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace bc
