// driving-force kernels of the KKS step, double fields (kks_point.cuh)
#include "kks_point.cuh"

namespace meu {
template KksPointFn<double> kks_point_kernel<double>(int, int, int);
}  // namespace meu
