// fft_mix.cuh -- instantiations of the compile-time transform kernels for the lengths with
// factors 3 (radix plan 3), one precision per including unit.
#pragma once
#include "fft_lines.cuh"

namespace meu {

template <typename R>
bool rows_mix(bool fwd, int L, int nf, int64_t nrows, const void* in, const void* out, const void* tw,
              const void* post, cudaStream_t st) {
  switch (L) {
#define MEU_CASE(N) case N: return rows_launch<R, N, 3>(fwd, nf, nrows, in, out, tw, post, st);
    MEU_CASE(12) MEU_CASE(16) MEU_CASE(18) MEU_CASE(24) MEU_CASE(27) MEU_CASE(36) MEU_CASE(48) MEU_CASE(54)
    MEU_CASE(72) MEU_CASE(81) MEU_CASE(96) MEU_CASE(108) MEU_CASE(144) MEU_CASE(162) MEU_CASE(192) MEU_CASE(216)
#undef MEU_CASE
    default: return false;
  }
}
// columns per block: a multiple of 4 within about 32 KB of tile
template <typename R>
constexpr int col_tile_mix(int L) { return col_tile_s<R>(L) / 4 * 4; }

template <typename R, bool FWD>
bool cols_mix(int L, int nf, int outer, int inner, int64_t ostride, const PtrList<cplx<R>>& in,
              const PtrList<cplx<R>>& out, const void* tw, R scale, cudaStream_t st) {
  switch (L) {
#define MEU_CASE(N) \
  case N: return cols_launch<R, FWD, N, col_tile_mix<R>(N), 3>(nf, outer, inner, ostride, in, out, tw, scale, st);
    MEU_CASE(16) MEU_CASE(24) MEU_CASE(36) MEU_CASE(48) MEU_CASE(54) MEU_CASE(72) MEU_CASE(96) MEU_CASE(108)
    MEU_CASE(144) MEU_CASE(162) MEU_CASE(192) MEU_CASE(216) MEU_CASE(288) MEU_CASE(324) MEU_CASE(384) MEU_CASE(432)
#undef MEU_CASE
    default: return false;
  }
}

}  // namespace meu
