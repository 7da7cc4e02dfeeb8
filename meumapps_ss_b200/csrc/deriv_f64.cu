// axis derivatives and z updates of every supported length, double fields (deriv.cuh)
#include "deriv.cuh"

namespace meu {
template void axis_launch<double>(int, const AxisArgs<double>&, int, const FFT3&, const void*, cudaStream_t);
template void z_div_launch<double>(const ZDivArgs<double>&, int, const FFT3&, cudaStream_t);
}  // namespace meu
