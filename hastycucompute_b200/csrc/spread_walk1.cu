// Walking spreading kernels for 1 transform, the cells on the lanes.
#include "spread_walk.cuh"

namespace hb {

int spread_walk_cc1(const NufftPlan* p, const GridArgs& a, const WalkArgs& w, cudaStream_t s) {
    return launch_spread_walk_w<1>(p, a, w, s);
}

}  // namespace hb
