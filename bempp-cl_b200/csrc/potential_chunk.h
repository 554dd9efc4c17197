// Elements per chunk of the orbit potentials' grid (potential_orbit.cu); host code without CUDA.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <cmath>

namespace bc {

// The chunk count c minimises the work over the slots plus one block's,
//   (pblocks c / slots + 1) (ceil(chunk / 4) + 2)
// in elements per warp (a block's four warps share its chunk; two elements stand for its start and its
// final sum), slots = SMs x resident blocks: blocks start as others end, so the last one's length is what is lost.  With
// whole waves, ceil(pblocks c / slots) (ceil(chunk / 4) + 4), one wave was taken wherever it nearly fitted, and SMs
// with one block fewer idled: 8192 elements, Helmholtz single layer, 3000 points 0.448 -> 0.392 ms, 10000 points 1.321 ->
// 1.231 ms, double layer 1.466 -> 1.439 ms, Laplace 3000 points 0.181 -> 0.163 ms, Maxwell electric far field 7000
// directions 1.018 -> 0.932 ms.  No more than one chunk per eight elements (two per warp), and than eight per slot.
//
// Without the ceilings the least cost lies at c = sqrt(slots n / (8 pblocks)); the search goes from 1 / 1.6 to 1.6
// times that, and from a count to the next one that shortens a warp's share (the counts between cost more).  It
// finds the minimum over all counts (checked over 6000 launches) in 160 looks or fewer, where all of them took
// 4 us of a call at 8192 elements and 64 points and 22 us at 131072.
inline int64_t potential_chunk(int64_t n, int64_t pblocks, int64_t slots) {
    int64_t cmax = std::min<int64_t>((n + 7) / 8, 65535);
    cmax = std::max<int64_t>(1, std::min<int64_t>(cmax, 8 * ((slots + pblocks - 1) / pblocks)));
    const double smooth = std::sqrt((double)slots * (double)n / (8.0 * (double)pblocks));
    const int64_t mid = std::max<int64_t>(1, (int64_t)std::min<double>(smooth, (double)cmax));
    const int64_t last = std::min<int64_t>(cmax, mid + (3 * mid) / 5 + 2);
    int64_t chunk = n, best = 0;
    for (int64_t c = std::max<int64_t>(1, (5 * mid) / 8); c <= last;) {
        const int64_t elems = (n + c - 1) / c, share = (elems + 3) / 4;
        const int64_t t = (pblocks * c + slots) * (share + 2);
        if (best == 0 || t < best) {
            best = t;
            chunk = elems;
        }
        if (share <= 1) break;
        c = std::max<int64_t>(c + 1, (n + 4 * (share - 1) - 1) / (4 * (share - 1)));
    }
    return chunk;
}

}  // namespace bc
