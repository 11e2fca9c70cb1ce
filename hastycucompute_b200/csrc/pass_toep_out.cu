// FFT pass instances: last Toeplitz pass.
#include "toep_ops.cuh"

namespace hb {

HB_INSTANTIATE_PASS(OpToepOutFlat)
HB_INSTANTIATE_PASS(OpToepOutSense)

}  // namespace hb
