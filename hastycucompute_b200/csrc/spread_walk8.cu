// Walking spreading kernels for 8 transforms per CTA.
#include "spread_walk.cuh"

namespace hb {

int spread_walk_cc8(const NufftPlan* p, const GridArgs& a, const WalkArgs& w, cudaStream_t s) {
    return launch_spread_walk_w<8>(p, a, w, s);
}

}  // namespace hb
