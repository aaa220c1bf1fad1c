// How region_group_kernel serves a program: decided on the host, in plain C++ (kernels_region.cu holds the kernels).
#pragma once

#include <cstdint>

#include "../../include/functs_b200.h"

#ifdef __CUDACC__
#define FB_HOST_DEVICE __host__ __device__
#else
#define FB_HOST_DEVICE
#endif

namespace fb {

constexpr int kRegionThreads = 256;
constexpr int kRegionVec = 4;  // elements per thread and pass in the large form
constexpr int kRegionSharedMost = 36 * 1024;  // leaves six CTAs on an SM; below the 48 KB that need no opt-in

enum RegionFetch { kEach, kAhead, kWindow };

// Words of the run behind the first element's pixel that the loads of `elements` elements reach.
FB_HOST_DEVICE inline int region_run_words(int interleave, int elements, int largest_base) { return interleave * (elements - 1) + largest_base + 1; }

struct RegionPlan {
    int fetch;   // RegionFetch
    int shared;  // bytes of dynamic shared memory
};
// The large form of a checked program; rank: the largest of its regions; inter: all regions in one CTA.
// Fetched ahead: float loads of interleaved regions, as many as leave six CTAs on an SM (normalisation of 1440 x 1920: 20.6 us
// without, 18.5 with; one region per CTA gains nothing, 2500 boxes of 80 classes 16.5 us without, 19.3 with).
// One run: rank 1, one tensor, every load at a place below the step, and room for a run as long as the output's (normalisation of
// an image that is in L2, one run / every load fetched ahead for itself: 800 x 1333 8.2 / 10.2 us, 1080 x 1440 10.7 / 12.6; of a new image
// each call, which DRAM bounds, 10.6 / 10.6 and 12.6 / 12.7; 1440 x 1920 17.1 / 17.2 and 18.1 / 19.0).
inline RegionPlan region_plan(const functs_b200_rprogram& P, int rank, bool inter) {
    constexpr int kSlot = kRegionThreads * kRegionVec * 4;
    const int out_bytes = inter ? P.interleave * kSlot : 0;
    int ahead = 0;
    bool floats = inter;
    for (int l = 0; l < P.num_loads; ++l) floats = floats && P.load[l].dtype == 0;
    for (int r = 0; r < P.num_regions; ++r) ahead += P.region[r].num_loads;
    if (!floats || out_bytes + ahead * kSlot > kRegionSharedMost) return {kEach, out_bytes};
    bool window = rank == 1 && ahead > 0 && 2 * out_bytes <= kRegionSharedMost;
    for (int l = 0; window && l < P.num_loads; ++l) {
        const functs_b200_rload& L = P.load[l];
        bool used = false;  // (the run reaches no further than a load that is made)
        for (int r = 0; r < P.num_regions; ++r) used = used || (l >= P.region[r].first_load && l < P.region[r].first_load + P.region[r].num_loads);
        window = used && L.tensor == P.load[0].tensor && L.coef[0] == P.interleave && L.base >= 0 && L.base < P.interleave;
    }
    return window ? RegionPlan{kWindow, 2 * out_bytes} : RegionPlan{kAhead, out_bytes + ahead * kSlot};
}

}  // namespace fb
