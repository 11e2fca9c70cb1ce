// FFT pass instances: first Toeplitz pass.
#include "toep_ops.cuh"

namespace hb {

HB_INSTANTIATE_PASS(OpToepIn)
HB_INSTANTIATE_PASS(OpToepInSenseT<false>)
HB_INSTANTIATE_PASS(OpToepInSenseT<true>)

}  // namespace hb
