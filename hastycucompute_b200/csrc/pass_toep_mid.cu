// FFT pass instances: fused Toeplitz pass.
#include "toep_ops.cuh"

namespace hb {

HB_INSTANTIATE_PASS(OpToepMid)

}  // namespace hb
