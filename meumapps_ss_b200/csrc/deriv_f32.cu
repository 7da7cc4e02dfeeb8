// axis derivatives and z updates of every supported length, float fields (deriv.cuh)
#include "deriv.cuh"

namespace meu {
template void axis_launch<float>(int, const AxisArgs<float>&, int, const FFT3&, const void*, cudaStream_t);
template void z_div_launch<float>(const ZDivArgs<float>&, int, const FFT3&, cudaStream_t);
}  // namespace meu
