// driving-force kernels of the KKS step, float fields (kks_point.cuh)
#include "kks_point.cuh"

namespace meu {
template KksPointFn<float> kks_point_kernel<float>(int, int, int);
}  // namespace meu
