// FFT pass instances: middle-axis Toeplitz passes.
#include "toep_ops.cuh"

namespace hb {

HB_INSTANTIATE_PASS(OpStridedPad)
HB_INSTANTIATE_PASS(OpStridedCrop)

}  // namespace hb
