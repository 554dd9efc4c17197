// Regular pairs of DP0 spaces: the FP64 and mixed-precision tiles of dp0.cuh and dp0_sym.cuh.
#include "dp0_sym.cuh"
#include "regular.cuh"

namespace bc {

// Symmetric sweeps: blockIdx.x = column block, blockIdx.y = row chunk; chunks
// that start below the block's last column have no pair i <= j and exit
// before touching shared memory.
template <int K, int FORM, bool STRIPE = false>
__global__ void __launch_bounds__(DP0_THREADS) regular_dp0_fp64_sym(RegParams prm, QuadRule rule, OrbitConsts oc,
                                                                    int64_t row0, int64_t row1, int tile_rows) {
    const int64_t t0 = row0 + (int64_t)blockIdx.y * tile_rows;
    if (t0 >= ((int64_t)blockIdx.x + 1) * DP0_THREADS) return;
    __shared__ TestBlock64s sb;
    __shared__ double park[form_orbit(FORM) ? SYM_PARK : 1];
    regular_dp0_fp64_sym_tile<K, FORM, STRIPE>(prm, rule, oc, blockIdx.x, t0,
                                               (int)min((int64_t)tile_rows, row1 - t0), sb, park);
}

// CTAs per SM the mixed symmetric sweep is compiled for (register cap 170 at
// 3): timed at L6, 3 and 4 are equal, 2 is 10 % slower.
#ifndef BC_MSYM_MIN_BLOCKS
#define BC_MSYM_MIN_BLOCKS 3
#endif

template <int K, int PHC, bool STRIPE = false, bool CK = false>
__global__ void __launch_bounds__(DP0_THREADS, BC_MSYM_MIN_BLOCKS)
    regular_dp0_mixed_sym(const __grid_constant__ RegParams prm, const __grid_constant__ QuadRule rule, int64_t row0,
                          int64_t row1, int tile_rows) {
    const int64_t t0 = row0 + (int64_t)blockIdx.y * tile_rows;
    if (t0 >= ((int64_t)blockIdx.x + 1) * DP0_THREADS) return;
    __shared__ TestBlock32q sb;
    regular_dp0_mixed_sym_tile<K, PHC, STRIPE, CK>(prm, rule, blockIdx.x, t0,
                                                   (int)min((int64_t)tile_rows, row1 - t0), sb);
}

// The mixed symmetric sweep in its phase class, real or (Helmholtz) complex wavenumber.
template <int K, bool STRIPE, bool CK>
static void mixed_sym_phase(const RegParams &prm, const QuadRule &rule, int phase_class, int64_t row0, int64_t row1,
                            int tile_rows, dim3 sgrid, cudaStream_t st) {
    if (phase_class == 2)
        regular_dp0_mixed_sym<K, 2, STRIPE, CK><<<sgrid, DP0_THREADS, 0, st>>>(prm, rule, row0, row1, tile_rows);
    else if (phase_class == 1)
        regular_dp0_mixed_sym<K, 1, STRIPE, CK><<<sgrid, DP0_THREADS, 0, st>>>(prm, rule, row0, row1, tile_rows);
    else
        regular_dp0_mixed_sym<K, 0, STRIPE, CK><<<sgrid, DP0_THREADS, 0, st>>>(prm, rule, row0, row1, tile_rows);
}

template <int K, bool STRIPE>
static void launch_mixed_sym(const RegParams &prm, const QuadRule &rule, int phase_class, int64_t row0, int64_t row1,
                             int tile_rows, dim3 sgrid, cudaStream_t st) {
    if constexpr (KernelTraits<K>::helm) {
        if (prm.p[1] != 0.0) {
            mixed_sym_phase<K, STRIPE, true>(prm, rule, phase_class, row0, row1, tile_rows, sgrid, st);
            return;
        }
    }
    mixed_sym_phase<K, STRIPE, false>(prm, rule, phase_class, row0, row1, tile_rows, sgrid, st);
}

// Kernels with a stripe-mode instance (the multi-GPU symmetric stripes): the Helmholtz family, the
// combined field and the Laplace single layer.
template <int K>
constexpr bool stripe_kernel() {
    return K == BEMPPCUDA_HELMHOLTZ_SLP || K == BEMPPCUDA_HELMHOLTZ_DLP || K == BEMPPCUDA_HELMHOLTZ_ADLP ||
           K == BEMPPCUDA_HELMHOLTZ_COMBINED || K == BEMPPCUDA_LAPLACE_SLP;
}

// The symmetric sweep of launch_dp0 in stripe mode (real or complex wavenumber; mixed or FP64).
template <int K>
static cudaError_t launch_dp0_stripe(const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc, int form,
                                     int mixed, int phase_class, int64_t row0, int64_t row1, int tile_rows, dim3 sgrid, cudaStream_t st) {
    if constexpr (stripe_kernel<K>()) {
        if (mixed) {
            launch_mixed_sym<K, true>(prm, rule, phase_class, row0, row1, tile_rows, sgrid, st);
        } else {
            with_form<K>(form, [&](auto f) {
                regular_dp0_fp64_sym<K, decltype(f)::value, true><<<sgrid, DP0_THREADS, 0, st>>>(prm, rule, oc, row0,
                                                                                                row1, tile_rows);
            });
        }
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int K>
static cudaError_t launch_dp0(const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc, int form, int mixed,
                              int phase_class, bool sym, int64_t row0, int64_t row1, cudaStream_t st) {
    dim3 grid((unsigned)((prm.ntrial + DP0_THREADS - 1) / DP0_THREADS), (unsigned)((prm.ntest + DP0_TCHUNK - 1) / DP0_TCHUNK));
    if constexpr (SymTraits<K>::supported) {
        // same DP0 space on both sides; the mixed tiles need Re k > 0 or omega > 0 (scaled units; a
        // complex k adds the amplitude split), the FP64 tiles take any wavenumber (sym_form)
        const bool helm = KernelTraits<K>::helm;
        const bool sweep_ok = helm || KernelTraits<K>::modhelm ? (!mixed || prm.p[0] > 0.0) : true;
        if (sym && sweep_ok) {
            // rows per tile: 32, halved (to 1) while that would leave the GPU under four waves of working CTAs
            // (about half the tiles lie below the diagonal and exit; 3 CTAs per SM)
            int tile_rows = DP0_TCHUNK;
            const int64_t wave = (int64_t)bc_sm_count() * 3;
            while (tile_rows > 1 && (int64_t)grid.x * ((row1 - row0 + tile_rows - 1) / tile_rows) / 2 < 4 * wave)
                tile_rows /= 2;
            const dim3 sgrid(grid.x, (unsigned)((row1 - row0 + tile_rows - 1) / tile_rows));
            if (prm.tresult) return launch_dp0_stripe<K>(prm, rule, oc, form, mixed, phase_class, row0, row1, tile_rows, sgrid, st);
            if (mixed) {
                launch_mixed_sym<K, false>(prm, rule, phase_class, row0, row1, tile_rows, sgrid, st);
                return cudaGetLastError();
            }
            with_form<K>(form, [&](auto f) {
                regular_dp0_fp64_sym<K, decltype(f)::value><<<sgrid, DP0_THREADS, 0, st>>>(prm, rule, oc, row0, row1,
                                                                                          tile_rows);
            });
            return cudaGetLastError();
        }
    }
    const bool ck = prm.p[1] != 0.0 && KernelTraits<K>::helm;
    // the packed path measures lengths in units of 1/k: Helmholtz needs k > 0
    const bool packed = !KernelTraits<K>::helm || prm.p[0] > 0.0;
    if constexpr (!KernelTraits<K>::modhelm) {
        if (mixed && !ck && packed) {
            if (phase_class == 2)
                regular_dp0_mixed2<K, 2><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
            else if (phase_class == 1)
                regular_dp0_mixed2<K, 1><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
            else
                regular_dp0_mixed2<K, 0><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
            return cudaGetLastError();
        }
    }
    if (row0 != 0 || row1 != prm.ntest) return cudaErrorInvalidValue;  // a row range needs the symmetric sweep
    if (mixed) {
        if (ck)
            regular_dp0_mixed<K, true, 0><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else if (phase_class == 2)
            regular_dp0_mixed<K, false, 2><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else if (phase_class == 1)
            regular_dp0_mixed<K, false, 1><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else
            regular_dp0_mixed<K, false, 0><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
    } else {
        if (ck)
            regular_dp0_fp64<K, true, 0><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else if (phase_class == 2)
            regular_dp0_fp64<K, false, 2><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else if (phase_class == 1)
            regular_dp0_fp64<K, false, 1><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
        else
            regular_dp0_fp64<K, false, 0><<<grid, DP0_THREADS, 0, st>>>(prm, rule);
    }
    return cudaGetLastError();
}

cudaError_t launch_dp0_kernel(int kernel, const RegParams &prm, const QuadRule &rule, const OrbitConsts &oc, int form,
                              int mixed, int phase_class, bool sym, int64_t row0, int64_t row1, cudaStream_t st) {
    switch (kernel) {
    case BEMPPCUDA_LAPLACE_SLP: return launch_dp0<BEMPPCUDA_LAPLACE_SLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_LAPLACE_DLP: return launch_dp0<BEMPPCUDA_LAPLACE_DLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_LAPLACE_ADLP: return launch_dp0<BEMPPCUDA_LAPLACE_ADLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_HELMHOLTZ_SLP: return launch_dp0<BEMPPCUDA_HELMHOLTZ_SLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_HELMHOLTZ_DLP: return launch_dp0<BEMPPCUDA_HELMHOLTZ_DLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_HELMHOLTZ_ADLP: return launch_dp0<BEMPPCUDA_HELMHOLTZ_ADLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_MODHELM_SLP: return launch_dp0<BEMPPCUDA_MODHELM_SLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_MODHELM_DLP: return launch_dp0<BEMPPCUDA_MODHELM_DLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_MODHELM_ADLP: return launch_dp0<BEMPPCUDA_MODHELM_ADLP>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    case BEMPPCUDA_HELMHOLTZ_COMBINED: return launch_dp0<BEMPPCUDA_HELMHOLTZ_COMBINED>(prm, rule, oc, form, mixed, phase_class, sym, row0, row1, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace bc
