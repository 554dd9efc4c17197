// Regular pairs on P1 / P0 and RWG / SNC spaces in mixed precision (p1_mixed.cuh).
#include "p1_mixed.cuh"
#include "regular.cuh"

namespace bc {

// Mixed-precision single layer, double layers and hypersingular on P1 spaces (p1_mixed.cuh): Helmholtz
// (phase classes, real or complex k), Laplace and modified Helmholtz (no phase classes).
template <int ASM, int K, bool SYM, bool CK>
static void p1_mixed_phase(const RegParams &prm, const OrbitConsts &oc, int phase_class, dim3 grid, cudaStream_t st) {
    if constexpr (K != BEMPPCUDA_HELMHOLTZ_SLP && K != BEMPPCUDA_HELMHOLTZ_DLP && K != BEMPPCUDA_HELMHOLTZ_ADLP) {
        regular_p1_mixed<ASM, K, 0, SYM, false><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
    } else {
        if (phase_class == 2)
            regular_p1_mixed<ASM, K, 2, SYM, CK><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
        else if (phase_class == 1)
            regular_p1_mixed<ASM, K, 1, SYM, CK><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
        else
            regular_p1_mixed<ASM, K, 0, SYM, CK><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
    }
}

// A P0 space beside a P1 one (scalar operators): per-pair sweep, the general phase class.
template <int K, int NT, int NS>
static void p1_mixed_pair(const RegParams &prm, const OrbitConsts &oc, dim3 grid, cudaStream_t st) {
    constexpr bool helm = K == BEMPPCUDA_HELMHOLTZ_SLP || K == BEMPPCUDA_HELMHOLTZ_DLP || K == BEMPPCUDA_HELMHOLTZ_ADLP;
    if constexpr (helm) {
        if (prm.p[1] != 0.0) {
            regular_p1_mixed<BEMPPCUDA_ASM_SCALAR, K, 0, false, true, NT, NS><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
            return;
        }
    }
    regular_p1_mixed<BEMPPCUDA_ASM_SCALAR, K, 0, false, false, NT, NS><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
}

template <int ASM, int K>
static cudaError_t launch_p1_mixed(const RegParams &prm, const OrbitConsts &oc, int phase_class, bool sym,
                                   cudaStream_t st) {
    dim3 grid((unsigned)((prm.ntrial + DP0_THREADS - 1) / DP0_THREADS),
              lin_row_blocks(prm.ntrial, prm.ntest, sym));
    if constexpr (ASM == BEMPPCUDA_ASM_SCALAR) {
        if (prm.tnshape == 3 && prm.snshape == 1) {
            p1_mixed_pair<K, 3, 1>(prm, oc, grid, st);
            return cudaGetLastError();
        }
        if (prm.tnshape == 1 && prm.snshape == 3) {
            p1_mixed_pair<K, 1, 3>(prm, oc, grid, st);
            return cudaGetLastError();
        }
    }
    constexpr bool helm = K == BEMPPCUDA_HELMHOLTZ_SLP || K == BEMPPCUDA_HELMHOLTZ_DLP ||
                          K == BEMPPCUDA_HELMHOLTZ_ADLP;
    const bool ck = helm && prm.p[1] != 0.0;
    if (ck) {
        if constexpr (helm) {
            if (sym)
                p1_mixed_phase<ASM, K, true, true>(prm, oc, phase_class, grid, st);
            else
                p1_mixed_phase<ASM, K, false, true>(prm, oc, phase_class, grid, st);
        }
    } else if (sym) {
        p1_mixed_phase<ASM, K, true, false>(prm, oc, phase_class, grid, st);
    } else {
        p1_mixed_phase<ASM, K, false, false>(prm, oc, phase_class, grid, st);
    }
    return cudaGetLastError();
}

cudaError_t launch_p1_mixed_kernel(int assembly, int kernel, const RegParams &prm, const OrbitConsts &oc,
                                   int phase_class, bool sym, cudaStream_t st) {
    switch (assembly) {
    case BEMPPCUDA_ASM_EFIE:
        return launch_p1_mixed<BEMPPCUDA_ASM_EFIE, BEMPPCUDA_HELMHOLTZ_SLP>(prm, oc, phase_class, sym, st);
    case BEMPPCUDA_ASM_MFIE:
        return launch_p1_mixed<BEMPPCUDA_ASM_MFIE, BEMPPCUDA_HELMHOLTZ_SLP>(prm, oc, phase_class, sym, st);
    case BEMPPCUDA_ASM_HELM_HYP:
        return launch_p1_mixed<BEMPPCUDA_ASM_HELM_HYP, BEMPPCUDA_HELMHOLTZ_SLP>(prm, oc, phase_class, sym, st);
    case BEMPPCUDA_ASM_LAPLACE_HYP:
        return launch_p1_mixed<BEMPPCUDA_ASM_LAPLACE_HYP, BEMPPCUDA_LAPLACE_SLP>(prm, oc, 0, sym, st);
    case BEMPPCUDA_ASM_MODHELM_HYP:
        return launch_p1_mixed<BEMPPCUDA_ASM_MODHELM_HYP, BEMPPCUDA_MODHELM_SLP>(prm, oc, 0, sym, st);
    default: break;
    }
    switch (kernel) {
    case BEMPPCUDA_LAPLACE_SLP: return launch_p1_mixed<0, BEMPPCUDA_LAPLACE_SLP>(prm, oc, 0, sym, st);
    case BEMPPCUDA_LAPLACE_DLP: return launch_p1_mixed<0, BEMPPCUDA_LAPLACE_DLP>(prm, oc, 0, sym, st);
    case BEMPPCUDA_LAPLACE_ADLP: return launch_p1_mixed<0, BEMPPCUDA_LAPLACE_ADLP>(prm, oc, 0, sym, st);
    case BEMPPCUDA_HELMHOLTZ_SLP: return launch_p1_mixed<0, BEMPPCUDA_HELMHOLTZ_SLP>(prm, oc, phase_class, sym, st);
    case BEMPPCUDA_HELMHOLTZ_DLP: return launch_p1_mixed<0, BEMPPCUDA_HELMHOLTZ_DLP>(prm, oc, phase_class, sym, st);
    case BEMPPCUDA_HELMHOLTZ_ADLP: return launch_p1_mixed<0, BEMPPCUDA_HELMHOLTZ_ADLP>(prm, oc, phase_class, sym, st);
    case BEMPPCUDA_MODHELM_SLP: return launch_p1_mixed<0, BEMPPCUDA_MODHELM_SLP>(prm, oc, 0, sym, st);
    case BEMPPCUDA_MODHELM_DLP: return launch_p1_mixed<0, BEMPPCUDA_MODHELM_DLP>(prm, oc, 0, sym, st);
    case BEMPPCUDA_MODHELM_ADLP: return launch_p1_mixed<0, BEMPPCUDA_MODHELM_ADLP>(prm, oc, 0, sym, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace bc
