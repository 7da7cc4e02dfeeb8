// fft_lines.cuh -- the compile-time x, y and z transform kernels of the generic path and
// their launch helpers, templated on length and radix plan.  fft.cu instantiates the power-of-two
// lengths (radix plans 0 and 2), fft_mix_f32.cu / fft_mix_f64.cu the lengths with factors 3.
#pragma once
#include <type_traits>

#include "fft.cuh"
#include "fft_stages.cuh"
#include "fused.cuh"

namespace meu {

// ----------------------------------------------- compile-time specialisations
// The same transforms with the length, radix plan and line count as template
// constants (stage_io of fft_stages.cuh on the radix plans of fused.cuh): index
// arithmetic folds to shifts and constant multiplies, and the digit reversal is
// computed instead of read from the table.  Powers of two 32..512 take them on radix plans
// 0 and 2, the lengths of fft_mix.cuh on plan 3 (108 x 144 x 96 FP64, six fields: y 59 -> 35 us,
// x 59 -> 40 us against the run-time plan, whose stages are bound by integer division and by
// two to four more shared-memory passes); other lengths keep the run-time plan of fft.cu.
constexpr int rows_per_block_c(int L) { return 2048 / L < 1 ? 1 : (2048 / L > 64 ? 64 : 2048 / L); }

// Rows interleaved in shared memory: element e of row r at e * ES + r with the odd
// stride ES = NR + 1, so that runs of consecutive e and runs of consecutive r both
// spread over the banks.  The global-facing stage walks consecutive elements of a
// row (JFAST); the stage next to the split step permutes between digit-reversed
// positions and natural frequency order (HOLD), so the split reads and writes
// consecutive frequencies, in shared and in global memory alike.
template <typename R, int L, int PV>
__global__ void __launch_bounds__(256) k_rows_r2c_s(PtrList<const R> in, PtrList<cplx<R>> out, int64_t nrows,
                                                    const cplx<R>* __restrict__ tw, const cplx<R>* __restrict__ post) {
  using C = cplx<R>;
  constexpr int NR = rows_per_block_c(L), ES = NR + 1, NXH = L + 1, NP = L / 2 + 1;
  constexpr int NS = fz::rplan(L, PV).ns;
  static_assert(NS >= 2, "first and last stage must differ");
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  dep_enter();
  const int64_t row0 = (int64_t)blockIdx.x * NR;
  const int nr = (int)min((int64_t)NR, nrows - row0);
  const C* src = (const C*)(in.p[blockIdx.y] + row0 * (2 * L));
  C* dst = out.p[blockIdx.y] + row0 * NXH;
  // a row of 2L reals is L complex pairs (rows past nr read row 0, never stored)
  stage_io<C, L, 0, NR, 256, PV, true, true>(
      tw, [&](int r, int e) { return src[(int64_t)(r < nr ? r : 0) * L + e]; },
      [&](int r, int e, C v) { buf[e * ES + r] = v; });
  __syncthreads();
  stages_smem<C, L, NR, ES, 256, PV, true, 1, NS - 1>(buf, tw);
  // last stage: position e holds frequency rev(e); store it at its frequency
  stage_io<C, L, NS - 1, NR, 256, PV, true, false, true>(
      tw, [&](int r, int e) { return buf[e * ES + r]; },
      [&](int r, int e, C v) { buf[fz::rev<L, PV>(e) * ES + r] = v; });
  __syncthreads();
  // split: X[k] = E + W^k O with E = (Z[k] + conj Z[L-k])/2, O = -i (Z[k] - conj Z[L-k])/2
  for (int i = threadIdx.x; i < NR * NP; i += 256) {
    const int r = i / NP, k = i - r * NP;
    if (r >= nr) continue;
    const int km = k == 0 ? 0 : L - k;
    const C zk = buf[k * ES + r], zm = buf[km * ES + r];
    C* drow = dst + (int64_t)r * NXH;
    {
      C e = cscale(cadd(zk, cconj(zm)), (R)0.5);
      C o = cscale(csub(zk, cconj(zm)), (R)0.5);
      o = mk(o.y, -o.x);
      drow[k] = cadd(e, Tw<C>::mul(o, post, k, NXH));
    }
    if (k != L - k) {
      C e = cscale(cadd(zm, cconj(zk)), (R)0.5);
      C o = cscale(csub(zm, cconj(zk)), (R)0.5);
      o = mk(o.y, -o.x);
      drow[L - k] = cadd(e, Tw<C>::mul(o, post, L - k, NXH));
    }
  }
}

template <typename R, int L, int PV>
__global__ void __launch_bounds__(256) k_rows_c2r_s(PtrList<const cplx<R>> in, PtrList<R> out, int64_t nrows,
                                                    const cplx<R>* __restrict__ tw, const cplx<R>* __restrict__ post) {
  using C = cplx<R>;
  constexpr int NR = rows_per_block_c(L), ES = NR + 1, NXH = L + 1, NP = L / 2 + 1;
  constexpr int NS = fz::rplan(L, PV).ns;
  static_assert(NS >= 2, "first and last stage must differ");
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  dep_enter();
  const int64_t row0 = (int64_t)blockIdx.x * NR;
  const int nr = (int)min((int64_t)NR, nrows - row0);
  const C* src = in.p[blockIdx.y] + row0 * NXH;
  C* dst = (C*)(out.p[blockIdx.y] + row0 * (2 * L));
  // Z[k] = (X[k] + conj X[L-k]) + i (X[k] - conj X[L-k]) W^-k, in natural order
  for (int i = threadIdx.x; i < NR * NP; i += 256) {
    const int r = i / NP, k = i - r * NP;
    if (r >= nr) continue;
    const C* srow = src + (int64_t)r * NXH;
    C xk = srow[k], xm = srow[L - k];
    if (k == 0) { xk.y = 0; xm.y = 0; }
    {
      C ex = cadd(xk, cconj(xm));
      C ox = Tw<C>::mulc(csub(xk, cconj(xm)), post, k, NXH);
      buf[k * ES + r] = cadd(ex, mk(-ox.y, ox.x));
    }
    if (k != 0 && k != L - k) {
      C ex = cadd(xm, cconj(xk));
      C ox = Tw<C>::mulc(csub(xm, cconj(xk)), post, L - k, NXH);
      buf[(L - k) * ES + r] = cadd(ex, mk(-ox.y, ox.x));
    }
  }
  __syncthreads();
  // first DIT stage: position e takes frequency rev(e)
  stage_io<C, L, NS - 1, NR, 256, PV, false, false, true>(
      tw, [&](int r, int e) { return buf[fz::rev<L, PV>(e) * ES + r]; },
      [&](int r, int e, C v) { buf[e * ES + r] = v; });
  __syncthreads();
  stages_smem<C, L, NR, ES, 256, PV, false, NS - 2, 0>(buf, tw);
  stage_io<C, L, 0, NR, 256, PV, false, true>(
      tw, [&](int r, int e) { return buf[e * ES + r]; },
      [&](int r, int e, C v) {
        if (r < nr) dst[(int64_t)r * L + e] = v;
      });
}

// TM columns of length L per block; element l of column (o, c) at o*ostride + l*inner + c.
// The first stage reads its butterflies straight from global memory and the last
// writes straight to global memory (digit reversal and forward scale folded into
// the addressing); only the stages between them go through shared memory.
template <typename R, bool FWD, int L, int TM, int PV>
__global__ void __launch_bounds__(256) k_cols_s(PtrList<cplx<R>> in, PtrList<cplx<R>> out, int inner, int64_t ostride,
                                                const cplx<R>* __restrict__ tw, R scale) {
  using C = cplx<R>;
  constexpr int NS = fz::rplan(L, PV).ns;
  static_assert(NS >= 2, "first and last stage must differ");
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  dep_enter();
  const int tiles = (inner + TM - 1) / TM;
  const int o = blockIdx.x / tiles, t = blockIdx.x - o * tiles;
  const int c0 = t * TM, nc = min(TM, inner - c0);
  const C* src = in.p[blockIdx.y] + (int64_t)o * ostride + c0;
  C* dst = out.p[blockIdx.y] + (int64_t)o * ostride + c0;
  // lines past nc (a partial last tile) read column 0 and are never stored
  auto gld = [&](int l, int e) {
    const int c = l < nc ? l : 0;
    return src[(int64_t)(FWD ? e : fz::rev<L, PV>(e)) * inner + c];
  };
  auto sst = [&](int l, int e, C v) { buf[e * TM + l] = v; };
  auto sld = [&](int l, int e) { return buf[e * TM + l]; };
  auto gst = [&](int l, int e, C v) {
    if (l < nc) dst[(int64_t)(FWD ? fz::rev<L, PV>(e) : e) * inner + l] = FWD ? cscale(v, scale) : v;
  };
  if constexpr (FWD) {
    stage_io<C, L, 0, TM, 256, PV, true>(tw, gld, sst);
    __syncthreads();
    stages_smem<C, L, TM, TM, 256, PV, true, 1, NS - 1>(buf, tw);
    stage_io<C, L, NS - 1, TM, 256, PV, true>(tw, sld, gst);
  } else {
    stage_io<C, L, NS - 1, TM, 256, PV, false>(tw, gld, sst);
    __syncthreads();
    stages_smem<C, L, TM, TM, 256, PV, false, NS - 2, 0>(buf, tw);
    stage_io<C, L, 0, TM, 256, PV, false>(tw, sld, gst);
  }
}

// Raise a kernel's dynamic shared-memory limit to the opt-in maximum once
// (227 KB per block on sm_100 minus the kernel's static shared memory).
template <typename R>
inline void set_smem(const void* fn, size_t bytes) {
  // always: without the opt-in, dynamic plus static shared memory must stay within 48 KB
  if ((int)bytes > smem_optin(fn)) throw CudaError("transform tile exceeds shared memory", 103);
}

// columns per block of the specialised column kernels: about 32 KB of tile
template <typename R>
constexpr int col_tile_s(int L) {
  const int t = 32768 / (L * 2 * (int)sizeof(R));
  return t < 4 ? 4 : (t > 16 ? 16 : t);
}

// launches for one (length, plan)
template <typename R, int LL, int PV>
bool rows_launch(bool fwd, int nf, int64_t nrows, const void* in, const void* out, const void* tw, const void* post,
                 cudaStream_t st) {
  using C = cplx<R>;
  constexpr int NR = rows_per_block_c(LL);
  const size_t sm = (size_t)(NR + 1) * LL * sizeof(C);
  const dim3 g((unsigned)((nrows + NR - 1) / NR), nf);
  if (fwd) {
    set_smem<R>((const void*)k_rows_r2c_s<R, LL, PV>, sm);
    launch_dep(k_rows_r2c_s<R, LL, PV>, g, 256, sm, st, *(const PtrList<const R>*)in, *(const PtrList<C>*)out, nrows,
               (const C*)tw, (const C*)post);
  } else {
    set_smem<R>((const void*)k_rows_c2r_s<R, LL, PV>, sm);
    launch_dep(k_rows_c2r_s<R, LL, PV>, g, 256, sm, st, *(const PtrList<const C>*)in, *(const PtrList<R>*)out, nrows,
               (const C*)tw, (const C*)post);
  }
  return true;
}
template <typename R, bool FWD, int LL, int TM, int PV>
bool cols_launch(int nf, int outer, int inner, int64_t ostride, const PtrList<cplx<R>>& in,
                 const PtrList<cplx<R>>& out, const void* tw, R scale, cudaStream_t st) {
  using C = cplx<R>;
  const size_t sm = (size_t)LL * TM * sizeof(C);
  set_smem<R>((const void*)k_cols_s<R, FWD, LL, TM, PV>, sm);
  const dim3 g((unsigned)(outer * ((inner + TM - 1) / TM)), nf);
  launch_dep(k_cols_s<R, FWD, LL, TM, PV>, g, 256, sm, st, in, out, inner, ostride, (const C*)tw, scale);
  return true;
}
// lengths with factors 3 (radix plan 3); false when L has no such kernel
template <typename R>
bool rows_mix(bool fwd, int L, int nf, int64_t nrows, const void* in, const void* out, const void* tw,
              const void* post, cudaStream_t st);
template <typename R, bool FWD>
bool cols_mix(int L, int nf, int outer, int inner, int64_t ostride, const PtrList<cplx<R>>& in,
              const PtrList<cplx<R>>& out, const void* tw, R scale, cudaStream_t st);

}  // namespace meu
