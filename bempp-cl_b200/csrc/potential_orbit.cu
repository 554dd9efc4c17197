// Launches of the FP64 potential and far-field kernels with the two-orbit rule (potential_orbit.cuh).
#include <algorithm>

#include "potential_chunk.h"
#include "potential_orbit.cuh"

namespace bc {

// Grid (point blocks, element chunks).
static cudaError_t orbit_grid(const PotParams &prm, const void *fn, int points, dim3 *grid, int64_t *chunk_elems) {
    int resident = 0;
    const cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, fn, PO_THREADS, 0);
    if (err != cudaSuccess) return err;
    const int64_t slots = (int64_t)bc_sm_count() * std::max(resident, 1);
    const int64_t pblocks = (prm.npoints + points - 1) / points;
    const int64_t chunk = potential_chunk(prm.nsupport, pblocks, slots);
    *chunk_elems = chunk;
    *grid = dim3((unsigned)pblocks, (unsigned)((prm.nsupport + chunk - 1) / chunk));
    return cudaSuccess;
}

template <int ASM, int K, int CLS, bool CK>
static cudaError_t launch_one(const PotParams &prm, const OrbitRule &rule, double near2, cudaStream_t st) {
    // points per thread: two share the staged coefficients of a scalar source; a Maxwell element's moments
    // fill the registers with one
    constexpr int PPT = ASM == BEMPPCUDA_ASM_SCALAR ? 2 : 1;
    constexpr int KD = ASM == BEMPPCUDA_ASM_SCALAR ? 1 : 3;
    auto fn = potential_orbit<ASM, K, CLS, CK, PPT>;
    dim3 grid;
    int64_t chunk = 0;
    cudaError_t err = orbit_grid(prm, (const void *)fn, PO_LANES * PPT, &grid, &chunk);
    if (err == cudaSuccess && grid.y > 1)
        err = cudaMemsetAsync(prm.result, 0, sizeof(double) * 2 * KD * prm.npoints, st);
    if (err != cudaSuccess) return err;
    fn<<<grid, PO_THREADS, 0, st>>>(prm, rule, chunk, near2);
    return cudaGetLastError();
}

template <int ASM, int K, bool CK = false>
static cudaError_t launch_class(const PotParams &prm, const OrbitRule &rule, int cls, double near2, cudaStream_t st) {
    if (cls == 2) return launch_one<ASM, K, 2, CK>(prm, rule, near2, st);
    if (cls == 1) return launch_one<ASM, K, 1, CK>(prm, rule, near2, st);
    return launch_one<ASM, K, 0, CK>(prm, rule, near2, st);
}

bool potential_orbit_has(int assembly, int kernel) {
    if (assembly == BEMPPCUDA_ASM_EFIE || assembly == BEMPPCUDA_ASM_MFIE)
        return kernel == BEMPPCUDA_HELMHOLTZ_SLP || kernel == BEMPPCUDA_FARFIELD_SLP;
    if (assembly != BEMPPCUDA_ASM_SCALAR) return false;
    return kernel == BEMPPCUDA_LAPLACE_SLP || kernel == BEMPPCUDA_LAPLACE_DLP || kernel == BEMPPCUDA_HELMHOLTZ_SLP ||
           kernel == BEMPPCUDA_HELMHOLTZ_DLP || kernel == BEMPPCUDA_MODHELM_SLP || kernel == BEMPPCUDA_MODHELM_DLP ||
           kernel == BEMPPCUDA_FARFIELD_SLP || kernel == BEMPPCUDA_FARFIELD_DLP;
}

cudaError_t launch_potential_orbit(const PotParams &prm, const OrbitRule &rule, int assembly, int kernel,
                                   double phase_radius, cudaStream_t st) {
    const bool maxwell = assembly != BEMPPCUDA_ASM_SCALAR;
    const unsigned blocks = (unsigned)((prm.nsupport + PO_ELEMS - 1) / PO_ELEMS);
    if (maxwell)
        potential_elements<true><<<blocks, PO_ELEMS, 0, st>>>(prm, rule);
    else
        potential_elements<false><<<blocks, PO_ELEMS, 0, st>>>(prm, rule);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    const bool far = kernel == BEMPPCUDA_FARFIELD_SLP || kernel == BEMPPCUDA_FARFIELD_DLP;
    const bool ck = !far && prm.p[1] != 0.0;
    // offsets |r - r_c| and x.(y - c) are at most rho R; a complex wavenumber's amplitude shares the class
    const double kmax = ck ? fmax(fabs(prm.p[0]), fabs(prm.p[1])) : fabs(prm.p[0]);
    const int cls = offset_class64(kmax * phase_radius * rule.rho);
    const double near = 2.5 * phase_radius, near2 = phase_radius > 0.0 ? near * near : INFINITY;
    constexpr int S = BEMPPCUDA_ASM_SCALAR, E = BEMPPCUDA_ASM_EFIE, M = BEMPPCUDA_ASM_MFIE;
    if (maxwell) {
        if (assembly == E && far) return launch_class<E, BEMPPCUDA_FARFIELD_SLP>(prm, rule, cls, near2, st);
        if (far) return launch_class<M, BEMPPCUDA_FARFIELD_SLP>(prm, rule, cls, near2, st);
        if (assembly == E)
            return ck ? launch_class<E, BEMPPCUDA_HELMHOLTZ_SLP, true>(prm, rule, cls, near2, st)
                      : launch_class<E, BEMPPCUDA_HELMHOLTZ_SLP>(prm, rule, cls, near2, st);
        return ck ? launch_class<M, BEMPPCUDA_HELMHOLTZ_SLP, true>(prm, rule, cls, near2, st)
                  : launch_class<M, BEMPPCUDA_HELMHOLTZ_SLP>(prm, rule, cls, near2, st);
    }
    switch (kernel) {
    case BEMPPCUDA_LAPLACE_SLP: return launch_one<S, BEMPPCUDA_LAPLACE_SLP, 0, false>(prm, rule, near2, st);
    case BEMPPCUDA_LAPLACE_DLP: return launch_one<S, BEMPPCUDA_LAPLACE_DLP, 0, false>(prm, rule, near2, st);
    case BEMPPCUDA_MODHELM_SLP: return launch_class<S, BEMPPCUDA_MODHELM_SLP>(prm, rule, cls, near2, st);
    case BEMPPCUDA_MODHELM_DLP: return launch_class<S, BEMPPCUDA_MODHELM_DLP>(prm, rule, cls, near2, st);
    case BEMPPCUDA_FARFIELD_SLP: return launch_class<S, BEMPPCUDA_FARFIELD_SLP>(prm, rule, cls, near2, st);
    case BEMPPCUDA_FARFIELD_DLP: return launch_class<S, BEMPPCUDA_FARFIELD_DLP>(prm, rule, cls, near2, st);
    case BEMPPCUDA_HELMHOLTZ_SLP:
        return ck ? launch_class<S, BEMPPCUDA_HELMHOLTZ_SLP, true>(prm, rule, cls, near2, st)
                  : launch_class<S, BEMPPCUDA_HELMHOLTZ_SLP>(prm, rule, cls, near2, st);
    default:  // BEMPPCUDA_HELMHOLTZ_DLP
        return ck ? launch_class<S, BEMPPCUDA_HELMHOLTZ_DLP, true>(prm, rule, cls, near2, st)
                  : launch_class<S, BEMPPCUDA_HELMHOLTZ_DLP>(prm, rule, cls, near2, st);
    }
}

}  // namespace bc
