// Regular pairs of the Maxwell electric and magnetic fields on RWG / SNC spaces in FP64 (rwg.cuh).
#include "regular.cuh"
#include "rwg.cuh"

namespace bc {

template <int ASM, bool SYM>
static void launch_rwg_class(const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc, int cls, dim3 grid,
                             cudaStream_t st) {
    if (prm.p[1] != 0.0) {
        if (cls == 2)
            regular_rwg_orbit<ASM, 2, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
        else if (cls == 1)
            regular_rwg_orbit<ASM, 1, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
        else
            regular_rwg_orbit<ASM, 0, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, oc);
    } else {
        if (cls == 2)
            regular_rwg_points<ASM, 2, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else if (cls == 1)
            regular_rwg_points<ASM, 1, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else
            regular_rwg_points<ASM, 0, SYM><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
    }
}

cudaError_t launch_rwg_kernel(int assembly, const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc, int cls,
                              bool sym, cudaStream_t st) {
    const dim3 grid((unsigned)((prm.ntrial + DP0_THREADS - 1) / DP0_THREADS),
                    lin_row_blocks(prm.ntrial, prm.ntest, sym));
    if (assembly == BEMPPCUDA_ASM_EFIE) {
        if (sym)
            launch_rwg_class<BEMPPCUDA_ASM_EFIE, true>(prm, rule, oc, cls, grid, st);
        else
            launch_rwg_class<BEMPPCUDA_ASM_EFIE, false>(prm, rule, oc, cls, grid, st);
    } else {
        if (sym)
            launch_rwg_class<BEMPPCUDA_ASM_MFIE, true>(prm, rule, oc, cls, grid, st);
        else
            launch_rwg_class<BEMPPCUDA_ASM_MFIE, false>(prm, rule, oc, cls, grid, st);
    }
    return cudaGetLastError();
}

}  // namespace bc
