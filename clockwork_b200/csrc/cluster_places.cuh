// How many thread-block clusters a GPU holds at a time.
#pragma once

#define CLUSTER_PLACES_MAX 8

// A cluster lies within one group of SMs (GPC), so that the counts are well below SMs / size.  These are what the driver's occupancy
// calculator gave for 148 SMs and an empty kernel with the shared memory of one or of two CTAs to an SM.  They are written down
// and not asked for: which SMs a part's groups lack differs from part to part, and the number of splits of a product, from which
// the order of its sums follows, must not.  A part that holds fewer runs what is left over in a second wave.
static inline int clusters_at_once(int size, int per_sm, int sm_count) {
    constexpr int places[2][CLUSTER_PLACES_MAX + 1] = {{0, 148, 74, 45, 33, 26, 22, 15, 15}, {0, 296, 148, 93, 71, 56, 45, 37, 33}};
    return (int)((long long)places[per_sm - 1][size] * sm_count / 148);
}
