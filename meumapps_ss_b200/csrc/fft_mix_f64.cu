// transform kernels of the lengths with factors 3, double fields (fft_mix.cuh)
#include "fft_mix.cuh"

namespace meu {
template bool rows_mix<double>(bool, int, int, int64_t, const void*, const void*, const void*, const void*, cudaStream_t);
template bool cols_mix<double, true>(int, int, int, int, int64_t, const PtrList<cplx<double>>&,
                                   const PtrList<cplx<double>>&, const void*, double, cudaStream_t);
template bool cols_mix<double, false>(int, int, int, int, int64_t, const PtrList<cplx<double>>&,
                                   const PtrList<cplx<double>>&, const void*, double, cudaStream_t);
}  // namespace meu
