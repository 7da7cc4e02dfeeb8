// elastic z kernels of every supported length, double fields (el_z.cuh)
#include "el_z.cuh"

namespace meu {
template int el_z_blocks<double>(int, int);
template void el_z_launch<double>(const FFT3&, cplx<double>*, cplx<double>*, const ElzCoef&, double*, cudaStream_t);
}  // namespace meu
