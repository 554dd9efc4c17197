// Launches of the FP64 potential and far-field kernels with the two-orbit rule (potential_orbit.cuh).
#include <algorithm>

#include "potential_orbit.cuh"

namespace bc {

// Grid (point blocks, element chunks).  The chunk count c minimises the work over the slots plus one block's,
//   (pblocks c / slots + 1) (ceil(chunk / 4) + 2)
// in elements per warp (a block's four warps share its chunk; two elements stand for its start and its
// final sum), slots = SMs x resident blocks: blocks start as others end, so the last one's length is what is lost.  With
// whole waves, ceil(pblocks c / slots) (ceil(chunk / 4) + 4), one wave was taken wherever it nearly fitted, and SMs
// with one block fewer idled: 8192 elements, Helmholtz single layer, 3000 points 0.448 -> 0.392 ms, 10000 points 1.321 ->
// 1.231 ms, double layer 1.466 -> 1.439 ms, Laplace 3000 points 0.181 -> 0.163 ms, Maxwell electric far field 7000
// directions 1.018 -> 0.932 ms.  The fewest elements of a chunk are 8, two per warp.
static cudaError_t orbit_grid(const PotParams &prm, const void *fn, int points, dim3 *grid, int64_t *chunk_elems) {
    int resident = 0;
    const cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, fn, PO_THREADS, 0);
    if (err != cudaSuccess) return err;
    const int64_t slots = (int64_t)bc_sm_count() * std::max(resident, 1);
    const int64_t pblocks = (prm.npoints + points - 1) / points;
    int64_t cmax = std::min<int64_t>((prm.nsupport + 7) / 8, 65535);
    cmax = std::max<int64_t>(1, std::min<int64_t>(cmax, 8 * ((slots + pblocks - 1) / pblocks)));
    int64_t best = 0, chunk = prm.nsupport;
    for (int64_t c = 1; c <= cmax; ++c) {
        const int64_t elems = (prm.nsupport + c - 1) / c;
        const int64_t t = (pblocks * c + slots) * ((elems + 3) / 4 + 2);
        if (c == 1 || t < best) {
            best = t;
            chunk = elems;
        }
    }
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
    const unsigned blocks = (unsigned)((prm.nsupport + PO_THREADS - 1) / PO_THREADS);
    if (maxwell)
        potential_elements<true><<<blocks, PO_THREADS, 0, st>>>(prm, rule);
    else
        potential_elements<false><<<blocks, PO_THREADS, 0, st>>>(prm, rule);
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
