// elastic row kernels, float fields, rows longer than 128 (el_rows.cuh)
#include "el_rows.cuh"

namespace meu {

template <>
bool el_rows_b<float>(const ElRowsArgs<float>& a, const ElRowsCoef<float>& c, bool fp64) {
  return elr::rows_unit<float, elr::LenB>(a, c, fp64);
}
template <>
bool el_ener_b<float>(const ElRowsArgs<float>& a, const ElRowsCoef<float>& c, const float* phi, const DevConst* K, float* el_en,
                       float* elg, const EnerOut<float>& out, int eta2, double* partials) {
  return elr::ener_unit<float, elr::LenB>(a, c, phi, K, el_en, elg, out, eta2, partials);
}

}  // namespace meu
