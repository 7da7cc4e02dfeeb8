// kks_point.cuh -- the instantiations of the KKS driving force (k_kks_point), one precision per
// including unit.
#pragma once
#include <utility>

#include "engine.cuh"
#include "step_kernels.cuh"

namespace meu {

// Two phases with one or two solutes: every variant count is compiled in, so that the per-variant
// values live in registers (FP64: up to nine variants without spills) and a voxel's loads are all in
// flight together.  Run-time count / compiled in, us per launch, one solute: 128^3 FP64 one
// variant 84 / 64, two 155 / 80, three 233 / 95, four 326 / 106, six 561 / 172, eight 857 / 233; 96^3
// FP64 twelve 789 / 184, sixteen 1455 / 286; 128^3 FP32 three 227 / 76; two solutes 96^3 FP64 one
// 93 / 90, three 139 / 93, twelve 812 / 225.  Three phases with one solute compile in the
// composition system alone (a variant's phase is known at run time); the rest is general.
template <typename R, int NEL, int... V>
KksPointFn<R> kks_point_two_phases(int nvar, std::integer_sequence<int, V...>) {
  KksPointFn<R> k = nullptr;
  ((nvar == V + 1 ? (void)(k = k_kks_point<R, 2, NEL, V + 1>) : (void)0), ...);
  return k;
}
template <typename R>
KksPointFn<R> kks_point_kernel(int numph, int numel, int nvar) {
  const auto counts = std::make_integer_sequence<int, MEU_MAX_VAR>{};
  if (numph == 2 && numel == 1) return kks_point_two_phases<R, 1>(nvar, counts);
  if (numph == 2 && numel == 2) return kks_point_two_phases<R, 2>(nvar, counts);
  if (numph == 3 && numel == 1) return k_kks_point<R, 3, 1>;
  return k_kks_point<R>;
}

}  // namespace meu
