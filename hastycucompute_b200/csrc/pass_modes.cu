// FFT pass instances: mode passes of the NUFFT (axis 2).
#include "modes_ops.cuh"

namespace hb {

HB_INSTANTIATE_PASS(OpModesIn)
HB_INSTANTIATE_PASS(OpModesOut)

}  // namespace hb
