// deriv.cuh -- spectral derivatives along one axis, and the z direction of a semi-implicit
// update, of the KKS step.  Included by deriv_f32.cu / deriv_f64.cu (one precision each).
//
// A derivative along an axis only needs that axis transformed: F^-1 (i b F f) over 3-D spectra
// equals the 1-D transform along the axis, times i b, and back (the other two directions'
// transforms cancel).  So the gradients and kappa-Laplacians of Multi_MEUMAPPS.f:575-615 are
// three passes over the real fields (per variant 5 field reads and 6 writes; the 3-D route moved
// 35 spectra), and so is the flux divergence of :924-943.  Nyquist as in k_space: b zeroed (first
// derivative), a kept (second).  Two real lines travel as one complex line.
//
// k_axis_x: pairs of rows; k_axis_c: columns along y or z of the field read as complex pairs
// (x, x + 1).  The transforms run e^{+} first (decimation in frequency), then e^{-} (decimation
// in time), with -i b between them: nothing is permuted, and the last forward stage, the
// multiplication and the first inverse stage run on one butterfly's registers.
#pragma once
#include "engine.cuh"
#include "fft_stages.cuh"
#include "step_kernels.cuh"

namespace meu {
namespace dv {

constexpr int PV = 4, NT = 128;  // plan 4 ends in a radix of 2 or 3

template <typename R, int L, int ES, int NL, int S, bool FIRST>
__device__ __forceinline__ void stage(cplx<R>* buf, const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  using T = fz::StageOf<L, S, PV>;
#pragma unroll 1
  for (int t = threadIdx.x; t < NL * T::TASKS; t += NT) {
    const int l = t % NL, u = t / NL, j = u % T::M, b = u / T::M;
    C* e = buf + (b * T::SPAN + j) * ES + l;
    C x[T::R];
#pragma unroll
    for (int r = 0; r < T::R; ++r) x[r] = e[r * T::M * ES];
    if (FIRST) {
      Dft<T::R, 1, C>::run(x);
#pragma unroll
      for (int q = 1; q < T::R; ++q) x[q] = cmulc(x[q], tw[j * q * T::TWS]);
    } else {
#pragma unroll
      for (int q = 1; q < T::R; ++q) x[q] = cmul(x[q], tw[j * q * T::TWS]);
      Dft<T::R, -1, C>::run(x);
    }
#pragma unroll
    for (int r = 0; r < T::R; ++r) e[r * T::M * ES] = x[r];
  }
}
template <typename R, int L, int ES, int NL, bool FIRST, int S, int SEND>
__device__ __forceinline__ void stages(cplx<R>* buf, const cplx<R>* tw) {
  if constexpr (FIRST ? S < SEND : S > SEND) {
    stage<R, L, ES, NL, S, FIRST>(buf, tw);
    __syncthreads();
    stages<R, L, ES, NL, FIRST, FIRST ? S + 1 : S - 1, SEND>(buf, tw);
  }
}
// between the transforms: the last stage of the first, times -i b / L (and -a^2 / L into the
// second buffer), the first stage of the second
template <typename R, int L, int ES, int NL, bool LAP>
__device__ __forceinline__ void middle(cplx<R>* buf, cplx<R>* lap) {
  using C = cplx<R>;
  constexpr int NS = fz::rplan(L, PV).ns;
  using T = fz::StageOf<L, NS - 1, PV>;
#pragma unroll 1
  for (int t = threadIdx.x; t < NL * T::TASKS; t += NT) {
    const int l = t % NL, b = t / NL, k0 = fz::rev<L, PV>(b * T::R);  // frequency of q = 0; q steps by L / R
    C* e = buf + b * T::R * ES + l;
    C x[T::R], y[T::R];
#pragma unroll
    for (int q = 0; q < T::R; ++q) x[q] = e[q * ES];
    Dft<T::R, 1, C>::run(x);
#pragma unroll
    for (int q = 0; q < T::R; ++q) {
      const int k = k0 + q * (L / T::R);
      const double a = (double)(k <= L / 2 ? k : k - L) * (6.283185307179586476925286766559 / (double)L);
      const double b1 = 2 * k == L ? 0.0 : a / (double)L;
      const double re = (double)x[q].x, im = (double)x[q].y;
      if (LAP) {
        const double a2 = -a * a / (double)L;
        y[q] = mk((R)(a2 * re), (R)(a2 * im));
      }
      x[q] = mk((R)(b1 * im), (R)(-b1 * re));
    }
    Dft<T::R, -1, C>::run(x);
    if (LAP) Dft<T::R, -1, C>::run(y);
#pragma unroll
    for (int q = 0; q < T::R; ++q) {
      e[q * ES] = x[q];
      if (LAP) (lap + b * T::R * ES + l)[q * ES] = y[q];
    }
  }
}

// out = base + s (acc + D f); lap (+)= g D2 f.  Fields of blockIdx.y at their strides.
template <typename R>
__device__ __forceinline__ R finish(double d, double s, const R* acc, const R* base, int64_t i) {
  if (acc) d += (double)acc[i];
  d *= s;
  if (base) d += (double)base[i];
  return (R)d;
}

// columns along y or z: element e of column (o, c) at o * ostride + e * inner + c (complex pairs)
template <typename R, int L, bool LAP>
__global__ void __launch_bounds__(NT) k_axis_c(const __grid_constant__ AxisArgs<R> A, int inner, int64_t ostride,
                                               const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  constexpr int TM = 128 / (int)sizeof(C), NS = fz::rplan(L, PV).ns;
  using T = fz::StageOf<L, 0, PV>;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;  // element e of column l at e * TM + l
  C* lb = buf + L * TM;
  dep_enter();
  const int tiles = (inner + TM - 1) / TM, o = blockIdx.x / tiles, c0 = (blockIdx.x - o * tiles) * TM;
  const int nc = min(TM, inner - c0), v = blockIdx.y;
  const int64_t at = o * ostride + c0;  // in pairs
  const C* src = (const C*)(A.f + v * A.fs) + at;
#pragma unroll 1
  for (int t = threadIdx.x; t < TM * T::M; t += NT) {
    const int l = t % TM, j = t / TM;
    const C* p = src + (int64_t)j * inner + (l < nc ? l : 0);
    C x[T::R];
#pragma unroll
    for (int q = 0; q < T::R; ++q) x[q] = p[(int64_t)q * T::M * inner];
    Dft<T::R, 1, C>::run(x);
#pragma unroll
    for (int q = 0; q < T::R; ++q) buf[(j + q * T::M) * TM + l] = q ? cmulc(x[q], tw[j * q]) : x[q];
  }
  __syncthreads();
  stages<R, L, TM, TM, true, 1, NS - 1>(buf, tw);
  middle<R, L, TM, TM, LAP>(buf, lb);
  __syncthreads();
  stages<R, L, TM, TM, false, NS - 2, 0>(buf, tw);
  if (LAP) stages<R, L, TM, TM, false, NS - 2, 0>(lb, tw);
  C* out = (C*)(A.out + v * A.os) + at;
  const C* acc = A.acc ? (const C*)(A.acc + v * A.as) + at : nullptr;
  const C* base = A.base ? (const C*)(A.base + v * A.bs) + at : nullptr;
  C* lap = LAP ? (C*)(A.lap + v * A.ls) + at : nullptr;
  const double g = LAP ? A.g[v] : 0.0, s = A.s[v];
#pragma unroll 1
  for (int t = threadIdx.x; t < TM * T::M; t += NT) {
    const int l = t % TM, j = t / TM;
    if (l >= nc) continue;
    C x[T::R];
#pragma unroll
    for (int q = 0; q < T::R; ++q) x[q] = q ? cmul(buf[(j + q * T::M) * TM + l], tw[j * q]) : buf[j * TM + l];
    Dft<T::R, -1, C>::run(x);
#pragma unroll
    for (int q = 0; q < T::R; ++q) {
      const int64_t i = (int64_t)(j + q * T::M) * inner + l;
      double dx = (double)x[q].x, dy = (double)x[q].y;
      if (acc) {
        const C a = acc[i];
        dx += (double)a.x;
        dy += (double)a.y;
      }
      dx *= s;
      dy *= s;
      if (base) {
        const C b = base[i];
        dx += (double)b.x;
        dy += (double)b.y;
      }
      out[i] = mk((R)dx, (R)dy);
    }
    if (LAP) {
#pragma unroll
      for (int q = 0; q < T::R; ++q) x[q] = q ? cmul(lb[(j + q * T::M) * TM + l], tw[j * q]) : lb[j * TM + l];
      Dft<T::R, -1, C>::run(x);
#pragma unroll
      for (int q = 0; q < T::R; ++q) {
        const int64_t i = (int64_t)(j + q * T::M) * inner + l;
        C b = A.lap_add ? lap[i] : mk((R)0, (R)0);
        lap[i] = mk((R)((double)b.x + g * (double)x[q].x), (R)((double)b.y + g * (double)x[q].y));
      }
    }
  }
}

// rows: about 16 KB of lines of two rows
template <typename R, int N>
constexpr int row_lines() {
  constexpr int r = 16 * 1024 / (N * 2 * (int)sizeof(R));
  return r < 1 ? 1 : (r > 16 ? 16 : r);
}
template <typename R, int N, bool LAP>
__global__ void __launch_bounds__(NT) k_axis_x(const __grid_constant__ AxisArgs<R> A, int64_t nrows,
                                               const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  constexpr int NL = row_lines<R, N>(), ES = NL | 1, NS = fz::rplan(N, PV).ns;
  using T = fz::StageOf<N, 0, PV>;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  C* lb = buf + N * ES;
  dep_enter();
  const int v = blockIdx.y;
  const int64_t row0 = (int64_t)blockIdx.x * (2 * NL);
  const int nr = (int)min((int64_t)(2 * NL), nrows - row0);
  const R* src = A.f + v * A.fs + row0 * N;
#pragma unroll 1
  for (int t = threadIdx.x; t < NL * T::M; t += NT) {
    const int j = t % T::M, l = t / T::M;
    // rows past nr (a partial last block) read the block's first row and are never stored
    const R* pa = src + (int64_t)(2 * l < nr ? 2 * l : 0) * N + j;
    const R* pb = 2 * l + 1 < nr ? pa + N : pa;
    C x[T::R];
#pragma unroll
    for (int q = 0; q < T::R; ++q) x[q] = mk(pa[q * T::M], pb[q * T::M]);
    Dft<T::R, 1, C>::run(x);
#pragma unroll
    for (int q = 0; q < T::R; ++q) buf[(j + q * T::M) * ES + l] = q ? cmulc(x[q], tw[j * q]) : x[q];
  }
  __syncthreads();
  stages<R, N, ES, NL, true, 1, NS - 1>(buf, tw);
  middle<R, N, ES, NL, LAP>(buf, lb);
  __syncthreads();
  stages<R, N, ES, NL, false, NS - 2, 0>(buf, tw);
  if (LAP) stages<R, N, ES, NL, false, NS - 2, 0>(lb, tw);
  R* out = A.out + v * A.os + row0 * N;
  const R* acc = A.acc ? A.acc + v * A.as + row0 * N : nullptr;
  const R* base = A.base ? A.base + v * A.bs + row0 * N : nullptr;
  R* lap = LAP ? A.lap + v * A.ls + row0 * N : nullptr;
  const double g = LAP ? A.g[v] : 0.0, s = A.s[v];
#pragma unroll 1
  for (int t = threadIdx.x; t < NL * T::M; t += NT) {
    const int j = t % T::M, l = t / T::M;
    if (2 * l >= nr) continue;
    const int64_t i0 = (int64_t)(2 * l) * N + j;
    const bool two = 2 * l + 1 < nr;
    C x[T::R];
#pragma unroll
    for (int q = 0; q < T::R; ++q) x[q] = q ? cmul(buf[(j + q * T::M) * ES + l], tw[j * q]) : buf[j * ES + l];
    Dft<T::R, -1, C>::run(x);
#pragma unroll
    for (int q = 0; q < T::R; ++q) {
      const int64_t i = i0 + q * T::M;
      out[i] = finish((double)x[q].x, s, acc, base, i);
      if (two) out[i + N] = finish((double)x[q].y, s, acc, base, i + N);
    }
    if (LAP) {
#pragma unroll
      for (int q = 0; q < T::R; ++q) x[q] = q ? cmul(lb[(j + q * T::M) * ES + l], tw[j * q]) : lb[j * ES + l];
      Dft<T::R, -1, C>::run(x);
#pragma unroll
      for (int q = 0; q < T::R; ++q) {
        const int64_t i = i0 + q * T::M;
        lap[i] = (R)((A.lap_add ? (double)lap[i] : 0.0) + g * (double)x[q].x);
        if (two) lap[i + N] = (R)((A.lap_add ? (double)lap[i + N] : 0.0) + g * (double)x[q].y);
      }
    }
  }
}

// z FFT, semi-implicit update, z inverse FFT of one spectrum per blockIdx.y: x / (1 + s k.kappa.k)
// (Multi_MEUMAPPS.f:924-943, :979-987), or with STATE the spectral state's step h <- (h - s x) /
// (1 + s k.kappa.k), which is also what goes back, and the gradient energy of the state it found.
// One read and one write of the spectrum (and of the state) instead of three: 256^3 FP32, four
// variants with their state 0.42 -> 0.22 ms.  Plan 3, in FP32 the radix-8 plan of the separate passes
// where there is one (see FFT3::fast); the last forward stage, the update and the first inverse
// stage run on one butterfly's registers.
constexpr int ZNT = 128;
template <typename R, int L>
constexpr int z_plan() { return sizeof(R) == 4 && L >= 32 && (L & (L - 1)) == 0 ? 0 : 3; }
template <typename R, int L, bool STATE>
__global__ void __launch_bounds__(ZNT) k_z_div(const __grid_constant__ ZDivArgs<R> A, const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  constexpr int ZPV = z_plan<R, L>(), TM = 128 / (int)sizeof(C), NS = fz::rplan(L, ZPV).ns;
  using TL = fz::StageOf<L, NS - 1, ZPV>;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  dep_enter();
  const int64_t inner = A.inner;
  const int c0 = blockIdx.x * TM, nc = min(TM, A.inner - c0), v = blockIdx.y;
  C* sp = A.sp + v * A.stride + c0;
  C* stt = STATE ? A.state + v * A.stride + c0 : nullptr;
  const double* g = A.g[v];
  double en = 0;
  // columns past nc read column 0 and are never stored
  stage_io<C, L, 0, TM, ZNT, ZPV, true>(
      tw, [&](int l, int e) { return sp[e * inner + (l < nc ? l : 0)]; }, [&](int l, int e, C x) { buf[e * TM + l] = x; });
  __syncthreads();
  stages_smem<C, L, TM, TM, ZNT, ZPV, true, 1, NS - 1>(buf, tw);
#pragma unroll 1
  for (int t = threadIdx.x; t < TM * TL::TASKS; t += ZNT) {
    const int l = t % TM, b = t / TM, m = min(c0 + l, A.inner - 1), ky = m / A.nxh, kx = m - ky * A.nxh;
    const int k0 = fz::rev<L, ZPV>(b * TL::R);
    C h[STATE ? TL::R : 1];
    if (STATE) {
#pragma unroll
      for (int q = 0; q < TL::R; ++q) h[q] = stt[(int64_t)(k0 + q * (L / TL::R)) * inner + (l < nc ? l : 0)];
    }
    const double a0 = (double)kx * A.wx, a1 = (double)(ky <= A.ny / 2 ? ky : ky - A.ny) * A.wy;
    const double b0 = 2 * kx == A.nx ? 0.0 : a0, b1 = 2 * ky == A.ny ? 0.0 : a1;
    const double d0 = g[0] * a0 * a0 + g[4] * a1 * a1 + (g[3] + g[1]) * b0 * b1, dz = (g[7] + g[5]) * b1 + (g[2] + g[6]) * b0;
    const double e0 = g[0] * b0 * b0 + g[4] * b1 * b1 + (g[3] + g[1]) * b0 * b1;
    C* e = buf + b * TL::R * TM + l;
    C x[TL::R];
#pragma unroll
    for (int q = 0; q < TL::R; ++q) x[q] = e[q * TM];
    Dft<TL::R, -1, C>::run(x);
    double ek = 0;
#pragma unroll
    for (int q = 0; q < TL::R; ++q) {
      const int kz = k0 + q * (L / TL::R);
      const double a2 = (double)(kz <= L / 2 ? kz : kz - L) * (6.283185307179586476925286766559 / (double)L);
      const double b2 = 2 * kz == L ? 0.0 : a2;
      const double den = 1.0 + A.s[v] * (d0 + g[8] * a2 * a2 + dz * b2);
      if (STATE) {
        const double hr = (double)h[q].x, hi = (double)h[q].y, sc = A.s[v] * A.scale, r = 1.0 / den;
        ek += (e0 + g[8] * b2 * b2 + dz * b2) * (hr * hr + hi * hi);
        x[q] = mk((R)((hr - sc * (double)x[q].x) * r), (R)((hi - sc * (double)x[q].y) * r));
        if (l < nc) stt[(int64_t)kz * inner + l] = x[q];
      } else {
        const double r = A.scale / den;
        x[q] = mk((R)((double)x[q].x * r), (R)((double)x[q].y * r));
      }
    }
    if (STATE && l < nc) en += (kx == 0 || 2 * kx == A.nx ? 0.5 : 1.0) * ek;
    Dft<TL::R, 1, C>::run(x);
#pragma unroll
    for (int q = 0; q < TL::R; ++q) e[q * TM] = x[q];
  }
  __syncthreads();
  stages_smem<C, L, TM, TM, ZNT, ZPV, false, NS - 2, 0>(buf, tw);
  stage_io<C, L, 0, TM, ZNT, ZPV, false>(
      tw, [&](int l, int e) { return buf[e * TM + l]; },
      [&](int l, int e, C x) {
        if (l < nc) sp[e * inner + l] = x;
      });
  if (STATE && A.part) block_reduce_store(en, 0, A.part + (int64_t)v * gridDim.x + blockIdx.x);
}

template <typename R, int L>
void launch_c(const AxisArgs<R>& A, int nf, int outer, int inner, int64_t ostride, const void* tw, cudaStream_t st) {
  using C = cplx<R>;
  constexpr int TM = 128 / (int)sizeof(C);
  const size_t sm = sizeof(C) * (size_t)L * TM * (A.lap ? 2 : 1);
  auto fn = A.lap ? k_axis_c<R, L, true> : k_axis_c<R, L, false>;
  if ((int)sm > smem_optin((const void*)fn)) throw CudaError("derivative tile exceeds shared memory", MEU_ERR_UNSUPPORTED);
  launch_dep(fn, dim3((unsigned)(outer * ((inner + TM - 1) / TM)), nf), NT, sm, st, A, inner, ostride, (const C*)tw);
}
template <typename R, int N>
void launch_x(const AxisArgs<R>& A, int nf, int64_t nrows, const void* tw, cudaStream_t st) {
  using C = cplx<R>;
  constexpr int NL = row_lines<R, N>();
  const size_t sm = sizeof(C) * (size_t)N * (NL | 1) * (A.lap ? 2 : 1);
  auto fn = A.lap ? k_axis_x<R, N, true> : k_axis_x<R, N, false>;
  if ((int)sm > smem_optin((const void*)fn)) throw CudaError("derivative rows exceed shared memory", MEU_ERR_UNSUPPORTED);
  launch_dep(fn, dim3((unsigned)((nrows + 2 * NL - 1) / (2 * NL)), nf), NT, sm, st, A, nrows, (const C*)tw);
}
template <typename R, int L>
void launch_z(const ZDivArgs<R>& A, int nf, const void* tw, cudaStream_t st) {
  using C = cplx<R>;
  constexpr int TM = 128 / (int)sizeof(C);
  const size_t sm = sizeof(C) * (size_t)L * TM;
  auto fn = A.state ? k_z_div<R, L, true> : k_z_div<R, L, false>;
  if ((int)sm > smem_optin((const void*)fn)) throw CudaError("z tile exceeds shared memory", MEU_ERR_UNSUPPORTED);
  launch_dep(fn, dim3((unsigned)((A.inner + TM - 1) / TM), nf), ZNT, sm, st, A, (const C*)tw);
}

}  // namespace dv

#define MEU_AXIS_LENGTHS(X) \
  X(16) X(24) X(32) X(36) X(48) X(54) X(64) X(72) X(96) X(108) X(128) X(144) X(162) X(192) X(216) X(256) X(288) X(324) \
  X(384) X(432) X(512)

template <typename R>
void axis_launch(int axis, const AxisArgs<R>& A, int nf, const FFT3& f, const void* tw_nx, cudaStream_t st) {
  const int L = axis == 0 ? f.nx : axis == 1 ? f.ny : f.nz;
  switch (L) {
#define MEU_CASE(N)                                                                                              \
  case N:                                                                                                        \
    if (axis == 0) dv::launch_x<R, N>(A, nf, (int64_t)f.ny * f.nz, tw_nx, st);                                   \
    else if (axis == 1) dv::launch_c<R, N>(A, nf, f.nz, f.nx / 2, (int64_t)f.ny * (f.nx / 2), f.py.tw, st);      \
    else dv::launch_c<R, N>(A, nf, 1, f.ny * (f.nx / 2), 0, f.pz.tw, st);                                        \
    break;
    MEU_AXIS_LENGTHS(MEU_CASE)
#undef MEU_CASE
    default: throw CudaError("internal: derivative along an unsupported length", MEU_ERR_UNSUPPORTED);
  }
  MEU_CHECK_LAUNCH();
}
template <typename R>
void z_div_launch(const ZDivArgs<R>& A, int nf, const FFT3& f, cudaStream_t st) {
  switch (f.nz) {
#define MEU_CASE(N) case N: dv::launch_z<R, N>(A, nf, f.pz.tw, st); break;
    MEU_AXIS_LENGTHS(MEU_CASE)
#undef MEU_CASE
    default: throw CudaError("internal: z division of an unsupported length", MEU_ERR_UNSUPPORTED);
  }
  MEU_CHECK_LAUNCH();
}

}  // namespace meu
