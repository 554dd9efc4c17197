// Launches of the touching-pair kernels on the order-4 Sauter-Schwab rules (singular_duffy.cuh).
#include <algorithm>

#include "singular_duffy.cuh"

int bc_singular_launch(const bemppcuda_singular_args *a, cudaStream_t st);

namespace bc {

struct DuffyPairs {
    const uint32_t *te, *se, *toff, *soff, *npts;
    int64_t npairs;
};

template <int ASM, int K, int N, int CLS, bool CK, int G>
__global__ void __launch_bounds__(SD_THREADS) singular_duffy(DuffyTarget prm, DuffyRule d, DuffyPairs list) {
    constexpr int GROUPS = SD_THREADS / G, NV = duffy_sums<duffy_mode<ASM, K, N>()>();
    __shared__ DuffyTable tab;
    __shared__ double2 scratch[GROUPS][NV];
    for (int i = threadIdx.x; i < SD_TAB; i += SD_THREADS) duffy_entry(d, i, tab);
    __syncthreads();
    const int group = threadIdx.x / G;
    for (int64_t base = (int64_t)blockIdx.x * GROUPS; base < list.npairs; base += (int64_t)gridDim.x * GROUPS) {
        const int64_t k = base + group;
        bool valid = k < list.npairs;
        int64_t t = 0, s = 0, toff = 0, soff = 0;
        int npts = 0;
        if (valid) {
            t = list.te[k];
            s = list.se[k];
            toff = list.toff[k];
            soff = list.soff[k];
            npts = (int)list.npts[k];
            valid = t < prm.ne && s < prm.ne && duffy_known(npts, toff, soff);
        }
        __syncwarp();  // the previous pair's sums have been read
        duffy_group<ASM, K, N, CLS, CK, G>(prm, tab, d, scratch[group], k, t, s, toff, soff, npts, valid);
        __syncwarp();
    }
}

// Lanes per pair: 8, or a warp when 8-lane groups would leave the GPU without two blocks per SM (meshes of
// a few hundred elements, where the pass is one pair's latency: 128 elements, Laplace, 35 us with the flat
// tables).
template <int ASM, int K, int N, int CLS, bool CK>
static cudaError_t launch_duffy(const DuffyTarget &prm, const DuffyPairs &list, cudaStream_t st) {
    static const DuffyRule rule = duffy_rule4();
    const int64_t sms = bc_sm_count();
    const bool wide = list.npairs * 8 < 2 * SD_THREADS * sms;
    const int64_t groups = SD_THREADS / (wide ? 32 : 8);
    // at most 16 blocks per SM: each writes the table once
    const unsigned blocks = (unsigned)std::min<int64_t>((list.npairs + groups - 1) / groups, 16 * sms);
    if (wide)
        singular_duffy<ASM, K, N, CLS, CK, 32><<<blocks, SD_THREADS, 0, st>>>(prm, rule, list);
    else
        singular_duffy<ASM, K, N, CLS, CK, 8><<<blocks, SD_THREADS, 0, st>>>(prm, rule, list);
    return cudaGetLastError();
}

template <int ASM, int K, int N>
static cudaError_t launch_duffy_class(const DuffyTarget &prm, const DuffyPairs &list, int cls, cudaStream_t st) {
    if constexpr (kernel_family<K>() == FAM_LAPLACE) {
        return launch_duffy<ASM, K, N, 0, false>(prm, list, st);
    } else {
        if constexpr (kernel_family<K>() == FAM_HELM) {
            if (prm.p[1] != 0.0) {
                if (cls == 2) return launch_duffy<ASM, K, N, 2, true>(prm, list, st);
                if (cls == 1) return launch_duffy<ASM, K, N, 1, true>(prm, list, st);
                return launch_duffy<ASM, K, N, 0, true>(prm, list, st);
            }
        }
        if (cls == 2) return launch_duffy<ASM, K, N, 2, false>(prm, list, st);
        if (cls == 1) return launch_duffy<ASM, K, N, 1, false>(prm, list, st);
        return launch_duffy<ASM, K, N, 0, false>(prm, list, st);
    }
}

}  // namespace bc

using namespace bc;

int bc_singular_duffy_launch(const bemppcuda_singular_args *a, int order, cudaStream_t st) {
    const int nt = a->test.nshape, ns = a->trial.nshape;
    const bool scalar = a->assembly == BEMPPCUDA_ASM_SCALAR;
    const bool combined = a->kernel == BEMPPCUDA_HELMHOLTZ_COMBINED;
    const bool dp0 = scalar && nt == 1 && ns == 1 && (a->kernel <= BEMPPCUDA_MODHELM_ADLP || combined);
    const bool lin = nt == 3 && ns == 3 && (!scalar || a->kernel <= BEMPPCUDA_MODHELM_ADLP);
    // the electric field divides by k
    const bool maxwell = a->assembly == BEMPPCUDA_ASM_EFIE || a->assembly == BEMPPCUDA_ASM_MFIE;
    if (order != SD_Q || !(dp0 || lin) || (maxwell && a->params[0] == 0.0 && a->params[1] == 0.0))
        return bc_singular_launch(a, st);
    if (a->npairs == 0) return BEMPPCUDA_OK;
    DuffyTarget prm;
    prm.g = a->grid.geom;
    prm.ne = a->grid.nelements;
    prm.tnm = a->test.normal_mult;
    prm.snm = a->trial.normal_mult;
    for (int i = 0; i < 4; ++i) prm.p[i] = a->params[i];
    prm.is_complex = a->is_complex != 0;
    prm.values = a->values;
    prm.dense = a->dense;
    prm.ld = a->ld;
    prm.tl2g = a->test.l2g;
    prm.sl2g = a->trial.l2g;
    prm.tmult = a->test.mult;
    prm.smult = a->trial.mult;
    prm.diag_shift = a->diag_shift;
    prm.mirror = a->mirror_weights_offset > 0;
    const DuffyPairs list = {a->test_elements, a->trial_elements, a->test_offsets, a->trial_offsets, a->npoints,
                             a->npairs};
    // the points reach the vertices: offsets from the centroid distance up to R_t + R_s
    const double kmax = fmax(fabs(a->params[0]), a->kernel >= BEMPPCUDA_MODHELM_SLP && a->kernel <= BEMPPCUDA_MODHELM_ADLP
                                                     ? 0.0 : fabs(a->params[1]));
    const int cls = offset_class64(kmax * a->phase_radius);
    cudaError_t err;
#define BC_DUFFY(ASM, K, N) launch_duffy_class<ASM, K, N>(prm, list, cls, st)
    switch (a->assembly) {
    case BEMPPCUDA_ASM_LAPLACE_HYP: err = BC_DUFFY(BEMPPCUDA_ASM_LAPLACE_HYP, BEMPPCUDA_LAPLACE_SLP, 3); break;
    case BEMPPCUDA_ASM_HELM_HYP: err = BC_DUFFY(BEMPPCUDA_ASM_HELM_HYP, BEMPPCUDA_HELMHOLTZ_SLP, 3); break;
    case BEMPPCUDA_ASM_MODHELM_HYP: err = BC_DUFFY(BEMPPCUDA_ASM_MODHELM_HYP, BEMPPCUDA_MODHELM_SLP, 3); break;
    case BEMPPCUDA_ASM_EFIE: err = BC_DUFFY(BEMPPCUDA_ASM_EFIE, BEMPPCUDA_HELMHOLTZ_SLP, 3); break;
    case BEMPPCUDA_ASM_MFIE: err = BC_DUFFY(BEMPPCUDA_ASM_MFIE, BEMPPCUDA_HELMHOLTZ_SLP, 3); break;
    case BEMPPCUDA_ASM_SCALAR:
        switch (a->kernel) {
#define BC_DUFFY_SCALAR(K) case K: err = dp0 ? BC_DUFFY(0, K, 1) : BC_DUFFY(0, K, 3); break;
        BC_DUFFY_SCALAR(BEMPPCUDA_LAPLACE_SLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_LAPLACE_DLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_LAPLACE_ADLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_HELMHOLTZ_SLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_HELMHOLTZ_DLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_HELMHOLTZ_ADLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_MODHELM_SLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_MODHELM_DLP)
        BC_DUFFY_SCALAR(BEMPPCUDA_MODHELM_ADLP)
#undef BC_DUFFY_SCALAR
        default: err = BC_DUFFY(0, BEMPPCUDA_HELMHOLTZ_COMBINED, 1); break;
        }
        break;
    default: return bc_singular_launch(a, st);
    }
#undef BC_DUFFY
    if (err != cudaSuccess) {
        bc_set_error("singular assembly launch failed: %s", cudaGetErrorString(err));
        return BEMPPCUDA_ERR_CUDA;
    }
    return BEMPPCUDA_OK;
}
