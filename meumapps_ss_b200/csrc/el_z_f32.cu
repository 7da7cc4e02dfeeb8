// elastic z kernels of every supported length, float fields (el_z.cuh)
#include "el_z.cuh"

namespace meu {
template int el_z_blocks<float>(int, int);
template void el_z_launch<float>(const FFT3&, cplx<float>*, cplx<float>*, const ElzCoef&, double*, cudaStream_t);
}  // namespace meu
