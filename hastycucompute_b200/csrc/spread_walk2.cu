// Walking spreading kernels for 2 transforms, the cells on the lanes.
#include "spread_walk.cuh"

namespace hb {

int spread_walk_cc2(const NufftPlan* p, const GridArgs& a, const WalkArgs& w, cudaStream_t s) {
    return launch_spread_walk_w<2>(p, a, w, s);
}

}  // namespace hb
