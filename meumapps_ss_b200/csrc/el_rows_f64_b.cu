// elastic row kernels, double fields, rows longer than 128 (el_rows.cuh)
#include "el_rows.cuh"

namespace meu {

template <>
bool el_rows_b<double>(const ElRowsArgs<double>& a, const ElRowsCoef<double>& c, bool fp64) {
  return elr::rows_unit<double, elr::LenB>(a, c, fp64);
}
template <>
bool el_ener_b<double>(const ElRowsArgs<double>& a, const ElRowsCoef<double>& c, const double* phi, const DevConst* K, double* el_en,
                       double* elg, const EnerOut<double>& out, int eta2, double* partials) {
  return elr::ener_unit<double, elr::LenB>(a, c, phi, K, el_en, elg, out, eta2, partials);
}

}  // namespace meu
