// Pieces of the tally recount shared by tally.cu and population.cu.
#pragma once

#include <climits>

#include "device.cuh"
#include "engine.h"

namespace glz {

// The tallies of label l that a recount rebuilds, zeroed.
__device__ __forceinline__ void clear_tallies(const RecountLaunch &a, int l) {
    a.vs_base[l] = make_int2(0, 0);
    for (int c = 0; c < a.g.ncol; ++c) a.vol_by_colour[(size_t)l * a.g.ncol + c] = 0;
    for (int k = 0; k < 3; ++k) a.vs_delta[k][l] = 0;
    if (a.tracks)
        for (int j = 0; j < a.g.nm; ++j) {
            a.mom_base[(size_t)l * a.g.nm + j] = 0;
            for (int k = 0; k < 3; ++k) a.mom_delta[k][(size_t)l * a.g.nm + j] = 0;
        }
}

// Lower first[label] to site i, through the first lane of each run of equal
// labels in the warp (whose site is the run's lowest); every lane takes part,
// and label 0 has no first site.
__device__ __forceinline__ void first_site(int *first, uint32_t label, int i) {
    const uint32_t before = __shfl_up_sync(0xffffffffu, label, 1);
    if (label != 0 && ((threadIdx.x & 31) == 0 || label != before)) atomicMin(&first[label], i);
}

}  // namespace glz
