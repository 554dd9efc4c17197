// Parameters of the potential kernels, and the FP64 kernels with the two-orbit rule (potential_orbit.cu).
#pragma once

#include "orbit.cuh"

namespace bc {

struct PotParams {
    const double *g;
    int64_t ne;
    const uint32_t *support;
    int64_t nsupport;
    const int32_t *nm;
    int nshape;
    int nq;
    const double *coeff;  // complex (ne * nshape)
    double *src;          // workspace SRC_FIELDS * nsrc
    int64_t nsrc;
    const double *points;  // (npoints, 3)
    int64_t npoints;
    double *result;  // complex (kdim, npoints)
    double p[4];
};

// True for the (assembly, kernel) pairs that launch_potential_orbit evaluates.
bool potential_orbit_has(int assembly, int kernel);

// Element records into prm.src and the evaluation (potential_orbit.cuh); phase_radius bounds every source's
// distance from its element centroid (0: unknown).
cudaError_t launch_potential_orbit(const PotParams &prm, const OrbitRule &rule, int assembly, int kernel,
                                   double phase_radius, cudaStream_t st);

}  // namespace bc
