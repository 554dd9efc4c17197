// Launches of the specialised regular-pair kernels, one translation unit each (regular_dp0.cu, regular_p1.cu,
// regular_p1_mixed.cu, regular_rwg.cu), called by the dispatch in regular.cu.
#pragma once

#include "dp0.cuh"
#include "orbit_pair.cuh"

namespace bc {

// Row blocks of the P1 and Maxwell sweeps: 32 test elements per CTA, halved while that would leave the GPU
// under twelve working CTAs per SM (a symmetric sweep's CTAs below the diagonal exit at once), down to one: four waves of
// the kernels that hold three CTAs per SM, six of those that hold two (the FP64 Maxwell fields with a real wavenumber, the
// skew sweeps of the Helmholtz double layers).  The kernels take their chunk height as ceil(ntest / gridDim.y).  32 rows
// against the halved ones: single layer
// P1, 1152 elements 0.239 and 0.143 ms; electric field, 288 elements 0.094 and 0.075 ms; from 4096 elements on (P1, symmetric) the
// launch has its twelve and keeps 32, one staging per 32 rows.
inline unsigned lin_row_blocks(int64_t ntrial, int64_t ntest, bool sym) {
    const int64_t cols = (ntrial + DP0_THREADS - 1) / DP0_THREADS;
    const int64_t least = 12 * (int64_t)bc_sm_count();
    int rows = 32;
    while (rows > 1 && cols * ((ntest + rows - 1) / rows) / (sym ? 2 : 1) < least) rows /= 2;
    return (unsigned)((ntest + rows - 1) / rows);
}

// DP0 spaces (regular_dp0.cu): rows [row0, row1) of a symmetric sweep (FP64 in the given form, sym_form), or
// the per-pair tiles.
cudaError_t launch_dp0_kernel(int kernel, const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc, int form,
                              int mixed, int phase_class, bool sym, int64_t row0, int64_t row1, cudaStream_t st);

// P1 / DP1 / P0 scalar and hypersingular operators in FP64 (regular_p1.cu): the points form with any 6-point rule
// where p1_points_form says so, else the orbit form with the two-orbit rule.
bool p1_points_form(int assembly, int kernel, const double *params);
cudaError_t launch_p1_kernel(int assembly, int kernel, const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc,
                             int cls, bool sym, cudaStream_t st);

// The same in mixed precision, and the mixed Maxwell fields (regular_p1_mixed.cu).
cudaError_t launch_p1_mixed_kernel(int assembly, int kernel, const RegParams &prm, const OrbitConsts &oc,
                                   int phase_class, bool sym, cudaStream_t st);

// Maxwell electric / magnetic fields in FP64 (regular_rwg.cu): any 6-point rule for a real wavenumber, the two-orbit
// rule for a complex one.
cudaError_t launch_rwg_kernel(int assembly, const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc, int cls,
                              bool sym, cudaStream_t st);

}  // namespace bc
