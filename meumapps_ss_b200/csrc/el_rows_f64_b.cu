// elastic row kernels, double fields, longer rows (el_rows.cuh)
#include "el_rows.cuh"

namespace meu {

template <>
bool el_rows_b<double>(const ElRowsArgs<double>& a, const ElRowsCoef<double>& c, bool fp64) {
  (void)fp64;  // FP64 fields have one precision
  switch (a.nx) {
#define MEU_CASE(N)                                                                          \
  case N:                                                                                    \
    if (!c.prop) elr::launch_rows<double, N, double, ElxGen>(a, *c.gen);                \
    else if (sizeof(double) == 4 && fp64) elr::launch_rows<double, N, double, ElxProp>(a, *c.p64); \
    else elr::launch_rows<double, N, double, ElxCoef<double>>(a, *c.pr);                     \
    return true;
    MEU_ROWS_B(MEU_CASE)
#undef MEU_CASE
    default: return false;
  }
}
template <>
bool el_ener_b<double>(const ElRowsArgs<double>& a, const ElRowsCoef<double>& c, const double* phi, const DevConst* K, double* el_en,
                       double* elg, const EnerOut<double>& out, int eta2, double* partials) {
  switch (a.nx) {
#define MEU_CASE(N)                                                                                    \
  case N:                                                                                              \
    if (c.prop) elr::launch_ener<double, N, ElenProp>(a, *c.en, phi, K, el_en, elg, out, eta2, partials); \
    else elr::launch_ener<double, N, ElxGen>(a, *c.gen, phi, K, el_en, elg, out, eta2, partials);      \
    return true;
    MEU_ROWS_B(MEU_CASE)
#undef MEU_CASE
    default: return false;
  }
}

}  // namespace meu
