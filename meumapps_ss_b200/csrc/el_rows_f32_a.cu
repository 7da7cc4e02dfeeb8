// elastic row kernels, float fields, rows of up to 128 (el_rows.cuh)
#include "el_rows.cuh"

namespace meu {

template <>
bool el_rows_a<float>(const ElRowsArgs<float>& a, const ElRowsCoef<float>& c, bool fp64) {
  (void)fp64;  // FP64 fields have one precision
  switch (a.nx) {
#define MEU_CASE(N)                                                                          \
  case N:                                                                                    \
    if (!c.prop) elr::launch_rows<float, N, double, ElxGen>(a, *c.gen);                \
    else if (sizeof(float) == 4 && fp64) elr::launch_rows<float, N, double, ElxProp>(a, *c.p64); \
    else elr::launch_rows<float, N, float, ElxCoef<float>>(a, *c.pr);                     \
    return true;
    MEU_ROWS_A(MEU_CASE)
#undef MEU_CASE
    default: return false;
  }
}
template <>
bool el_ener_a<float>(const ElRowsArgs<float>& a, const ElRowsCoef<float>& c, const float* phi, const DevConst* K, float* el_en,
                       float* elg, const EnerOut<float>& out, int eta2, double* partials) {
  switch (a.nx) {
#define MEU_CASE(N)                                                                                    \
  case N:                                                                                              \
    if (c.prop) elr::launch_ener<float, N, ElenProp>(a, *c.en, phi, K, el_en, elg, out, eta2, partials); \
    else elr::launch_ener<float, N, ElxGen>(a, *c.gen, phi, K, el_en, elg, out, eta2, partials);      \
    return true;
    MEU_ROWS_A(MEU_CASE)
#undef MEU_CASE
    default: return false;
  }
}

}  // namespace meu
