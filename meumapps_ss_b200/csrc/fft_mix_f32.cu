// transform kernels of the lengths with factors 3, float fields (fft_mix.cuh)
#include "fft_mix.cuh"

namespace meu {
template bool rows_mix<float>(bool, int, int, int64_t, const void*, const void*, const void*, const void*, cudaStream_t);
template bool cols_mix<float, true>(int, int, int, int, int64_t, const PtrList<cplx<float>>&,
                                   const PtrList<cplx<float>>&, const void*, float, cudaStream_t);
template bool cols_mix<float, false>(int, int, int, int, int64_t, const PtrList<cplx<float>>&,
                                   const PtrList<cplx<float>>&, const void*, float, cudaStream_t);
}  // namespace meu
