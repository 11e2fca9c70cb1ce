// FFT pass instances: plain strided passes (NUFFT axes 0 and 1, Toeplitz kernel build).
#include "ops.cuh"

namespace hb {

HB_INSTANTIATE_PASS(OpStrided)

}  // namespace hb
