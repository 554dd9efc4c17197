// The six-point triangle rule as two orbits of three points.
//
// The order-4 rule (Strang-Fix / Dunavant) has two orbits of three points of equal weight; the point of
// orbit o that belongs to vertex j has barycentric coordinates alpha_o + g_o at j and alpha_o at the other
// two, alpha_o = (1 - g_o) / 3.  Its offset from the element's centroid c is therefore g_o e_j with
// e_j = v_j - c, and e_0 + e_1 + e_2 = 0: six points need two independent vectors, a dot product with all
// six offsets costs two dot products and a subtraction, and a sum over the points weighted by linear
// functions needs the three values of each orbit and their sum only.
// |y_q - c| <= rho R for every point, R the centroid-to-vertex distance, rho = max_o |g_o| (0.725).
#pragma once

#include <math.h>

#include "common.cuh"

namespace bc {

// Point q of a rule in orbit order: orbit q / 3, vertex 2 - q % 3.
__host__ __device__ constexpr int orbit_vertex(int q) { return 2 - q % 3; }

struct OrbitRule {
    double g[2];
    double w[2];
    double rho;
};

// The orbits of a 6-point rule; false when the rule is not made of them (to 2e-15, the digits of a tabulated rule).
inline bool orbit_rule(const QuadRule &rule, OrbitRule &o) {
    if (rule.nq != 6) return false;
    for (int k = 0; k < 2; ++k) {
        // the first point of the orbit belongs to vertex 2: alpha_o is its coordinate at vertex 1
        o.g[k] = 1.0 - 3.0 * rule.x[3 * k];
        o.w[k] = rule.w[3 * k];
        const double alpha = rule.x[3 * k];
        for (int i = 0; i < 3; ++i) {
            const int q = 3 * k + i, v = orbit_vertex(q);
            const double lx = alpha + (v == 1 ? o.g[k] : 0.0), ly = alpha + (v == 2 ? o.g[k] : 0.0);
            if (!(fabs(rule.x[q] - lx) <= 2e-15) || !(fabs(rule.y[q] - ly) <= 2e-15)) return false;
            if (!(fabs(rule.w[q] - o.w[k]) <= 2e-15 * fabs(o.w[k]))) return false;
        }
    }
    o.rho = fmax(fabs(o.g[0]), fabs(o.g[1]));
    return true;
}

}  // namespace bc
