// el_rows.cuh -- the x direction of the elastic problem in one pass per iteration.  The state
// of the fixed point between iterations is the six strain spectra after their z and y inverse
// passes ("row spectra": rows of nx/2 + 1 along kx).  k_el_rows runs, for a block of rows, the
// x C2R transform, the polarisation of every voxel (ModElastic.f:248-327) and the x R2C
// transform back into the same rows; k_el_ener runs the x C2R transform and elener
// (ModElastic.f:540-687).  The real strain and polarisation never reach global memory: per cell
// an iteration moves 6 spectra in, V reals in, 6 spectra out.  Included by the units
// el_rows_*.cu, which instantiate the lengths.
//
// Two rows of one component travel as one complex line of the full length nx (row + i next
// row), so the split steps of a half-length transform and their twiddles are additions here.
// (Two components as one line would do the same with half the registers, but rounding would
// carry a component into one that is exactly zero, and the convergence test compares ratios.)
// The inverse runs its stages in decimation in frequency and the forward in decimation in time,
// so the voxels between them sit in digit-reversed order, which pointwise work does not mind,
// and nothing is permuted; the last inverse stage, the polarisation and the first forward stage
// run on one butterfly's registers of all six components.
#pragma once
#include <type_traits>

#include "engine.cuh"
#include "fft_stages.cuh"
#include "step_kernels.cuh"

namespace meu {
namespace elr {

constexpr int PV = 4;

// Tile, threads and resident blocks per SM it is compiled for.  What bounds it is issue and the
// latency of a block's phases, so small blocks that overlap one another win where the voxel work
// is in the field precision:
//  FP32, proportional: 16 KB of lines, 128 threads, six blocks (256^3, 4 variants, per launch:
//   0.38 ms; 24 KB x 256 x 3 0.41, 48 KB x 384 x 2 0.43);
//  FP64: 24 KB, 128 threads, four blocks (KKS 128^3 0.111 ms, 24 KB x 256 x 2 0.138; 108 x 144 x 96
//   70 us, 48 KB x 256 x 2 74 us);
//  FP32 with general moduli (FP64 voxel work): 48 KB, 256 threads, two blocks.  Against 24 KB x 128 x 4
//   small grids and many variants gain and large ones lose (KKS 64^3, one variant 16.8 us, 20.9 with the
//   latter; Landau 64^3, 12 variants 23.4, 29.6; 128 x 128 x 64, 12 variants 73, 80; four 50.8, 46.7).
template <typename R, bool GEN>
struct Cfg {
  static constexpr int KB = sizeof(R) == 8 ? 24 : GEN ? 48 : 16;
  static constexpr int NT = sizeof(R) == 8 || !GEN ? 128 : 256;
  static constexpr int BLOCKS = sizeof(R) == 8 ? 4 : GEN ? 2 : 6;
};
template <typename COEF>
constexpr bool is_gen() { return std::is_same<COEF, ElxGen>::value; }

// rows per block (even)
template <typename R, int N, bool GEN>
constexpr int rows() {
  constexpr int r = Cfg<R, GEN>::KB * 1024 / (3 * N * 2 * (int)sizeof(R)) / 2 * 2;
  return r < 2 ? 2 : (r > 16 ? 16 : r);
}
template <typename R, int N, bool GEN>
struct Geo {
  using C = cplx<R>;
  static constexpr int NT = Cfg<R, GEN>::NT;
  static constexpr int NR = rows<R, N, GEN>(), NL = 3 * NR, ES = NL | 1;  // odd: consecutive elements spread over the banks
  static constexpr int PS = N + 16 / (int)sizeof(R);                 // row stride of the order parameters
  static constexpr size_t line_bytes = sizeof(cplx<R>) * (size_t)N * ES;
};

// One stage over the block's lines (line l = 6 i + m: component m of the row pair 2i, 2i + 1),
// element e of line l at buf[e * ES + l].  INV: DIF with e^{+}; else DIT with e^{-}.
template <typename R, int N, typename G, int S, bool INV>
__device__ __forceinline__ void stage(cplx<R>* buf, const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  using T = fz::StageOf<N, S, PV>;
#pragma unroll 1
  for (int t = threadIdx.x; t < G::NL * T::TASKS; t += G::NT) {
    const int l = t % G::NL, u = t / G::NL, j = u % T::M, b = u / T::M;
    C* e = buf + (b * T::SPAN + j) * G::ES + l;
    C x[T::R];
#pragma unroll
    for (int r = 0; r < T::R; ++r) x[r] = e[r * T::M * G::ES];
    if (INV) {
      Dft<T::R, 1, C>::run(x);
      if (T::M > 1) {
#pragma unroll
        for (int q = 1; q < T::R; ++q) x[q] = cmulc(x[q], tw[j * q * T::TWS]);
      }
    } else {
      if (T::M > 1) {
#pragma unroll
        for (int q = 1; q < T::R; ++q) x[q] = cmul(x[q], tw[j * q * T::TWS]);
      }
      Dft<T::R, -1, C>::run(x);
    }
#pragma unroll
    for (int r = 0; r < T::R; ++r) e[r * T::M * G::ES] = x[r];
  }
}
template <typename R, int N, typename G, bool INV, int S, int SEND>
__device__ __forceinline__ void stages(cplx<R>* buf, const cplx<R>* tw) {
  if constexpr (INV ? S < SEND : S >= SEND) {
    stage<R, N, G, S, INV>(buf, tw);
    __syncthreads();
    stages<R, N, G, INV, INV ? S + 1 : S - 1, SEND>(buf, tw);
  }
}
// the first inverse stage from the spectral rows: Z = X_2i + i X_2i+1, the upper half from the
// Hermitian symmetry (c2r: the imaginary parts of k = 0 and k = N/2 are not read)
template <typename R, int N, typename G>
__device__ __forceinline__ void head(cplx<R>* buf, const cplx<R>* __restrict__ sp, int64_t nk, int64_t row0, int nr,
                                     const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  using T = fz::StageOf<N, 0, PV>;
  constexpr int NXH = N / 2 + 1;
#pragma unroll 1
  for (int t = threadIdx.x; t < G::NL * T::M; t += G::NT) {
    const int j = t % T::M, l = t / T::M, m = l % 6, r = l / 6 * 2;
    // rows past nr (a partial last block) read row0 and are never stored
    const C* a = sp + m * nk + (row0 + (r < nr ? r : 0)) * NXH;
    const int nb = r + 1 < nr ? NXH : 0;
    C x[T::R];
#pragma unroll
    for (int q = 0; q < T::R; ++q) {
      const int k = j + q * T::M;
      // which half k is in is known per q, except in the middle of an odd radix
      const bool up = T::R % 2 == 0 ? q >= T::R / 2 : 2 * k > N;
      const C* c = up ? a + (N - k) : a + k;
      const C xa = c[0], xb = c[nb];
      R ya = up ? -xa.y : xa.y, yb = up ? -xb.y : xb.y;
      if ((q == 0 && j == 0) || 2 * k == N) ya = yb = 0;
      x[q] = mk(xa.x - yb, ya + xb.x);
    }
    Dft<T::R, 1, C>::run(x);
    C* e = buf + j * G::ES + l;
#pragma unroll
    for (int q = 0; q < T::R; ++q) {
      if (T::M > 1 && q > 0) x[q] = cmulc(x[q], tw[j * q * T::TWS]);
      e[q * T::M * G::ES] = x[q];
    }
  }
}

// the block's rows of V fields (n3 apart) into dst, 16-byte copies; row r of field v at
// dst + (v * NR + r) * PS
template <typename R, int N, typename G>
__device__ __forceinline__ void prefetch(R* dst, const R* __restrict__ src, int V, int64_t n3, int64_t row0, int nr) {
  using C = cplx<R>;
  constexpr int PER = N % (16 / (int)sizeof(R)) == 0 ? 16 / (int)sizeof(R) : 2, CPR = N / PER;
  const R* s0 = src + row0 * N;
  for (int v = 0; v < V; ++v)
    for (int i = threadIdx.x; i < nr * CPR; i += G::NT) {
      const int r = i / CPR, n = (i - r * CPR) * PER;
      if constexpr (PER == 2) fz::cp_async_c((C*)(dst + (v * G::NR + r) * G::PS + n), (const C*)(s0 + v * n3 + r * N + n));
      else fz::cp_async16(dst + (v * G::NR + r) * G::PS + n, s0 + v * n3 + r * N + n);
    }
}

// fn(v) for every variant, unrolled (coefficients at fixed parameter addresses) up to four; UN at a
// time beyond (4 where the order parameters come from global memory: their loads overlap)
template <int UN, typename FN>
__device__ __forceinline__ void each_variant(int V, FN&& fn) {
  if (V <= 4) {
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (v < V) fn(v);
  } else {
#pragma unroll UN
    for (int v = 0; v < V; ++v) fn(v);
  }
}

// mixed compliance of a voxel: sum over phases of S_n times the sum of its order parameters,
// plus (1 - sum) S_1 (eldis: only below 1); returns the sum
template <typename R>
__device__ __forceinline__ double gen_mix(const ElxGen& E, const R* pp, int64_t vs, double* Cm, bool below_one) {
  double psum = 0;
#pragma unroll
  for (int i = 0; i < 36; ++i) Cm[i] = 0;
#pragma unroll
  for (int n = 1; n < MEU_MAX_PH; ++n) {
    if (n >= E.numph) break;
    double ps = 0;
    for (int v = E.lo[n]; v < E.hi[n]; ++v) ps += (double)pp[v * vs];
    psum += ps;
#pragma unroll
    for (int i = 0; i < 36; ++i)
      if (ortho_nz(i)) Cm[i] += ps * E.s[n][i];
  }
  const double w = below_one && !(psum < 1.0) ? 0.0 : 1.0 - psum;
#pragma unroll
  for (int i = 0; i < 36; ++i)
    if (ortho_nz(i)) Cm[i] += w * E.s[0][i];
  return psum;
}

// polarisation of two voxels (h = 0, 1) from their engineering strains g[m][h], in place,
// proportional moduli (C(x) = C_1 / s(x); k_el_x_prop's formula) in the precision W.  Order
// parameter v of voxel h at pp[v * vs + h * hs].
template <int UN, typename W, typename R, typename S>
__device__ __forceinline__ void polarise(const ElxCoef<W>& E, W cfac, R (*g)[2], const R* pp, S vs, int hs, int* err) {
  W e0[2][6] = {}, psum[2] = {0, 0}, sc[2] = {0, 0};
  each_variant<UN>(E.nvar, [&](int v) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const W q = (W)pp[v * vs + h * hs];
      psum[h] += E.inc[v] * q;
      sc[h] += E.av[v] * q;
#pragma unroll
      for (int m = 0; m < 6; ++m) e0[h][m] += q * E.ep[v][m];
    }
  });
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (psum[h] < (W)1) sc[h] += (W)1 - psum[h];
    if (!(sc[h] != (W)0)) set_err(err, MEU_ERR_C_SINGULAR);
    const W r = (W)1 / sc[h];
    W gam[6], d[6], a0[6], a1[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      gam[m] = (W)g[m][h] + E.ebar[m];
      d[m] = e0[h][m] - cfac * gam[m];
    }
    if (E.ortho) {
      mv6<true>(E.c0, gam, a0);
      mv6<true>(E.c1, d, a1);
    } else {
      mv6<false>(E.c0, gam, a0);
      mv6<false>(E.c1, d, a1);
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) g[i][h] = (R)(cfac * a0[i] + r * a1[i]);
  }
}
// the same for general moduli with decoupled normal and shear parts (k_el_x<R, true>): the
// mixed compliance inverted as a 3x3 block and three shears, FP64
template <int UN, typename W, typename R, typename S>
__device__ __forceinline__ void polarise(const ElxGen& E, W cfac, R (*g)[2], const R* pp, S vs, int hs, int* err) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double Cm[36], e0[6] = {0, 0, 0, 0, 0, 0};
    gen_mix(E, pp + h * hs, vs, Cm, true);
    each_variant<UN>(E.nvar, [&](int v) {
      const double q = (double)pp[v * vs + h * hs];
#pragma unroll
      for (int m = 0; m < 6; ++m) e0[m] += q * E.ep[v][m];
    });
    set_err(err, invert6_ortho(Cm, MEU_ERR_C_SINGULAR));
    double gam[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) gam[m] = (double)g[m][h] + E.ebar[m];
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      double a = 0;
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        if (!ortho_nz(r + m * 6)) continue;
        const double c = Cm[r + m * 6];
        a += cfac * (E.c0[r + m * 6] - c) * gam[m] + c * e0[m];
      }
      g[r][h] = (R)a;
    }
  }
}

// sp: the six row spectra (contiguous, nk apart), in place; E: ElxCoef<W> or ElxGen.  Dynamic
// shared memory: the lines, then with STAGE the block's order parameters (cp.async, in flight during
// the inverse transform); else they are read from global memory where they are used.
template <typename R, int N, typename W, typename COEF, bool STAGE>
__global__ void __launch_bounds__((Cfg<R, is_gen<COEF>()>::NT), (Cfg<R, is_gen<COEF>()>::BLOCKS))
    k_el_rows(cplx<R>* sp, int64_t nk, const R* pphi, int64_t n3, int64_t nrows,
              const cplx<R>* __restrict__ tw, const __grid_constant__ COEF E, const double* cfac_p, int* err) {
  using C = cplx<R>;
  using G = Geo<R, N, is_gen<COEF>()>;
  constexpr int NR = G::NR, NS = fz::rplan(N, PV).ns, NXH = N / 2 + 1, NT = G::NT;
  using TL = fz::StageOf<N, NS - 1, PV>;
  static_assert(NS >= 2 && TL::M == 1, "two stages or more");
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  R* pbuf = (R*)(smraw + (G::line_bytes + 15) / 16 * 16);
  const int64_t row0 = (int64_t)blockIdx.x * NR;
  const int nr = (int)min((int64_t)NR, nrows - row0);
  dep_enter();
  if constexpr (STAGE) {
    prefetch<R, N, G>(pbuf, pphi, E.nvar, n3, row0, nr);
    fz::cp_async_commit();
  }
  const W cfac = cfac_p ? (W)*cfac_p : (W)1;
  head<R, N, G>(buf, sp, nk, row0, nr, tw);
  __syncthreads();
  stages<R, N, G, true, 1, NS - 1>(buf, tw);
  if constexpr (STAGE) {
    fz::cp_async_wait_all();
    __syncthreads();
  }
  // last inverse stage, polarisation, first forward stage on the registers of one butterfly
#pragma unroll 1
  for (int t = threadIdx.x; t < NR / 2 * TL::TASKS; t += G::NT) {
    const int i = t % (NR / 2), b = t / (NR / 2);
    C* e = buf + b * TL::R * G::ES + 6 * i;
    C x[6][TL::R];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
#pragma unroll
      for (int q = 0; q < TL::R; ++q) x[m][q] = e[q * G::ES + m];
      Dft<TL::R, 1, C>::run(x[m]);
    }
    const int n0 = fz::rev<N, PV>(b * TL::R);  // voxel of q = 0; q steps by N / R
#pragma unroll
    for (int q = 0; q < TL::R; ++q) {
      R g[6][2];
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        g[m][0] = x[m][q].x;
        g[m][1] = x[m][q].y;
      }
      // a row past nr takes the block's first row (it is not stored)
      const int r0 = 2 * i < nr ? 2 * i : 0, r1 = 2 * i + 1 < nr ? 2 * i + 1 : r0;
      const int n = n0 + q * (N / TL::R);
      if constexpr (STAGE) polarise<STAGE ? 1 : 4, W>(E, cfac, g, pbuf + r0 * G::PS + n, NR * G::PS, (r1 - r0) * G::PS, err);
      else polarise<STAGE ? 1 : 4, W>(E, cfac, g, pphi + (row0 + r0) * N + n, n3, (r1 - r0) * N, err);
#pragma unroll
      for (int m = 0; m < 6; ++m) x[m][q] = mk(g[m][0], g[m][1]);
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      Dft<TL::R, -1, C>::run(x[m]);
#pragma unroll
      for (int q = 0; q < TL::R; ++q) e[q * G::ES + m] = x[m][q];
    }
  }
  __syncthreads();
  stages<R, N, G, false, NS - 2, 0>(buf, tw);
  // Z(k) in natural order: X_2i = (Z(k) + conj Z(-k)) / 2, X_2i+1 = -i (Z(k) - conj Z(-k)) / 2
  const int lane = threadIdx.x & 31;
  for (int l = threadIdx.x >> 5; l < G::NL; l += NT / 32) {
    const int m = l % 6, r = l / 6 * 2;
    if (r >= nr) continue;
    const C* z = buf + l;
    C* d = sp + m * nk + (row0 + r) * NXH;
    C* d1 = r + 1 < nr ? d + NXH : nullptr;
    auto put = [&](int k, const C zk, const C zm) {
      d[k] = mk((R)0.5 * (zk.x + zm.x), (R)0.5 * (zk.y - zm.y));
      if (d1) d1[k] = mk((R)0.5 * (zk.y + zm.y), (R)0.5 * (zm.x - zk.x));
    };
    for (int k = lane; k < N / 2; k += 32) put(k, z[k * G::ES], z[(k == 0 ? 0 : N - k) * G::ES]);
    if (lane == 0) put(N / 2, z[N / 2 * G::ES], z[N / 2 * G::ES]);
  }
}

// elener of one voxel (FP64): stress, energy density and each variant's driving force
struct EnerVox {
  double sig[6], mat, psum;
};
// proportional moduli (k_elener_prop): sigma = C_1 eps / s
template <int UN, typename R, typename S>
__device__ __forceinline__ void ener_stress(const ElenProp& E, const DevConst&, const double* gam, const R* pp,
                                            S vs, EnerVox& o, int* err) {
  double te[6] = {0, 0, 0, 0, 0, 0}, ps = 0, sc = 0, eps[6], em[6];
  each_variant<UN>(E.nvar, [&](int v) {
    const double q = (double)pp[v * vs];
    ps += q;
    sc += E.av[v] * q;
#pragma unroll
    for (int m = 0; m < 6; ++m) te[m] += q * E.tp[v][m];
  });
#pragma unroll
  for (int m = 0; m < 6; ++m)
    eps[m] = (m < 3) ? (E.emean[m] + gam[m] - te[m]) : (2.0 * E.emean[m] + gam[m] - 2.0 * te[m]);
  sc += 1.0 - ps;
  if (!(sc != 0.0)) set_err(err, MEU_ERR_C_ELENER_SINGULAR);
  const double r = 1.0 / sc;
  if (E.ortho) mv6<true>(E.c1, eps, o.sig);
  else mv6<false>(E.c1, eps, o.sig);
#pragma unroll
  for (int i = 0; i < 6; ++i) o.sig[i] *= r;
  if (E.ortho) mv6<true>(E.s1, o.sig, em);
  else mv6<false>(E.s1, o.sig, em);
  double mat = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i) mat += o.sig[i] * em[i];
  o.mat = 0.5 * mat;
  o.psum = ps;
}
__device__ __forceinline__ double ener_ppt(const ElenProp& E, const DevConst&, int v, const EnerVox& o) {
  return E.av[v] * o.mat;
}
__device__ __forceinline__ bool ener_use(const ElenProp& E, const DevConst&, int v) { return E.use[v] != 0; }
__device__ __forceinline__ const double* ener_tp(const ElenProp& E, const DevConst&, int v) { return E.tp[v]; }

// general moduli with decoupled normal and shear parts (k_elener<R, true>)
template <int UN, typename R, typename S>
__device__ __forceinline__ void ener_stress(const ElxGen& E, const DevConst& K, const double* gam, const R* pp,
                                            S vs, EnerVox& o, int* err) {
  double te[6] = {0, 0, 0, 0, 0, 0}, Cm[36], eps[6];
  each_variant<UN>(E.nvar, [&](int v) {
    const double q = (double)pp[v * vs];
#pragma unroll
    for (int m = 0; m < 6; ++m) te[m] += q * E.ep[v][m];  // engineering shear
  });
#pragma unroll
  for (int m = 0; m < 6; ++m) eps[m] = (m < 3 ? 1.0 : 2.0) * K.p.e_mean[m] + gam[m] - te[m];
  const double ps = gen_mix(E, pp, vs, Cm, false);
  set_err(err, invert6_ortho(Cm, MEU_ERR_C_ELENER_SINGULAR));
  mv6<true>(Cm, eps, o.sig);
  double em[6], mat = 0;
  mv6<true>(E.s[0], o.sig, em);
#pragma unroll
  for (int i = 0; i < 6; ++i) mat += o.sig[i] * em[i];
  o.mat = 0.5 * mat;
  o.psum = ps;
}
__device__ __forceinline__ double ener_ppt(const ElxGen& E, const DevConst&, int v, const EnerVox& o) {
  double em[6], a = 0;
  mv6<true>(E.s[E.phase[v]], o.sig, em);
#pragma unroll
  for (int i = 0; i < 6; ++i) a += o.sig[i] * em[i];
  return 0.5 * a;
}
__device__ __forceinline__ bool ener_use(const ElxGen&, const DevConst& K, int v) { return K.use_var[v] != 0; }
__device__ __forceinline__ const double* ener_tp(const ElxGen&, const DevConst& K, int v) { return K.p.trans_ppt[v]; }

// Row blocks of the final strain: x C2R, then elener with the voxels in row order (the last
// inverse stage stores every voxel at its own place, after a barrier, so that global memory is
// read and written in rows; with STAGE order parameters and P by cp.async during the transform);
// the driving force as EnerOut says.  Grid-stride over row blocks: at most PSTRIDE
// blocks, each one partial of the energy sum.
template <typename R, int N, typename COEF, bool STAGE>
__global__ void __launch_bounds__((Cfg<R, is_gen<COEF>()>::NT), (Cfg<R, is_gen<COEF>()>::BLOCKS))
    k_el_ener(const cplx<R>* __restrict__ sp, int64_t nk, const R* __restrict__ phi, const R* __restrict__ pphi,
              int64_t n3, int64_t nrows, const cplx<R>* __restrict__ tw, const DevConst* __restrict__ Kp,
              const __grid_constant__ COEF E, R* __restrict__ el_en, R* __restrict__ elg,
              const __grid_constant__ EnerOut<R> out, int eta2, double* partials, int* err) {
  using C = cplx<R>;
  using G = Geo<R, N, is_gen<COEF>()>;
  constexpr int NR = G::NR, NS = fz::rplan(N, PV).ns, NT = G::NT, VS = NR * G::PS;
  using VT = std::conditional_t<STAGE, int, int64_t>;
  constexpr int UN = STAGE ? 1 : 4;
  using TL = fz::StageOf<N, NS - 1, PV>;
  constexpr int IT = (G::NL * TL::TASKS + NT - 1) / NT;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  R* pb = (R*)(smraw + (G::line_bytes + 15) / 16 * 16);
  R* fb = pb + E.nvar * VS;
  const DevConst& K = *Kp;
  double esum = 0;
#pragma unroll 1
  for (int64_t row0 = (int64_t)blockIdx.x * NR; row0 < nrows; row0 += (int64_t)gridDim.x * NR) {
    const int nr = (int)min((int64_t)NR, nrows - row0);
    if constexpr (STAGE) {
      prefetch<R, N, G>(pb, pphi, E.nvar, n3, row0, nr);
      prefetch<R, N, G>(fb, phi, E.nvar, n3, row0, nr);
      fz::cp_async_commit();
    }
    head<R, N, G>(buf, sp, nk, row0, nr, tw);
    __syncthreads();
    stages<R, N, G, true, 1, NS - 1>(buf, tw);
    {
      C x[IT][TL::R];
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int t = threadIdx.x + it * NT, l = t % G::NL, b = t / G::NL;
        if (t < G::NL * TL::TASKS) {
#pragma unroll
          for (int q = 0; q < TL::R; ++q) x[it][q] = buf[(b * TL::R + q) * G::ES + l];
          Dft<TL::R, 1, C>::run(x[it]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int t = threadIdx.x + it * NT, l = t % G::NL, b = t / G::NL;
        if (t < G::NL * TL::TASKS) {
          const int n0 = fz::rev<N, PV>(b * TL::R);
#pragma unroll
          for (int q = 0; q < TL::R; ++q) buf[(n0 + q * (N / TL::R)) * G::ES + l] = x[it][q];
        }
      }
    }
    if constexpr (STAGE) fz::cp_async_wait_all();
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < nr * N; i += G::NT) {
      const int r = i / N, n = i - r * N;
      const int64_t id = (row0 + r) * N + n;
      const R* e = (const R*)(buf + n * G::ES + r / 2 * 6) + (r & 1);
      const R *pv = STAGE ? pb + r * G::PS + n : pphi + id, *fv = STAGE ? fb + r * G::PS + n : phi + id;
      const VT vs = STAGE ? (VT)VS : (VT)n3;
      double gam[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) gam[m] = (double)e[2 * m];
      EnerVox o;
      ener_stress<UN>(E, K, gam, pv, vs, o, err);
      double en = (1.0 - o.psum) * o.mat, s2 = 0, cv = 0;
      if (out.mode == 3) {
        cv = K.c_mean[0] + (double)out.c[id];
        each_variant<UN>(E.nvar, [&](int v) { s2 += (double)fv[v * vs] * (double)fv[v * vs]; });
      }
      each_variant<UN>(E.nvar, [&](int v) {
        const double f = (double)fv[v * vs];
        double eg = 0;
        if (ener_use(E, K, v)) {
          const double elp = ener_ppt(E, K, v, o);
          en += elp * (double)pv[v * vs];
          const double* t = ener_tp(E, K, v);
          const double g = o.sig[0] * t[0] + o.sig[1] * t[1] + o.sig[2] * t[2] +
                           2.0 * (o.sig[3] * t[3] + o.sig[4] * t[4] + o.sig[5] * t[5]);
          const double pr = eta2 ? 2.0 * f : 30.0 * f * f * (f * f - 2.0 * f + 1.0);
          eg = pr * (o.mat - elp) - g * pr;
        } else if (out.mode < 2) {
          return;
        }
        R* d = elg + v * n3 + id;
        if (out.mode == 2) {
          const double nz = out.noise ? out.dt * (double)out.noise[v * n3 + id] : 0.0;
          const R t = *d + (R)eg;  // the force in the fields' precision, as mode 0 leaves it
          *d = (R)(f - out.dtl * (double)t + nz);
        } else if (out.mode == 0) {
          *d += (R)eg;
        } else if (out.mode == 3) {
          const meu_params& p = K.p;
          const double e2 = f * f;
          *d = (R)(p.lan_b * (p.lan_c2 - cv) * f - p.lan_c * e2 * f + p.lan_d * e2 * e2 * f +
                   4.0 * p.cross_w * f * (s2 - e2) + eg);
        } else {
          *d = (R)eg;
        }
      });
      el_en[id] = (R)en;
      esum += en;
    }
    __syncthreads();
  }
  block_reduce_store(esum, 0, partials + Q_ELEN * PSTRIDE + blockIdx.x);
}

// Order parameters come through shared memory while that leaves two blocks per SM, for elener (which
// stages P and the order parameters, and reads them row by row otherwise) also more than half of
// the blocks that the lines alone would; else straight from global memory, so that any number of
// variants runs on every length.  Staged / direct, us per launch: k_el_rows KKS 64^3 FP64 3
// variants 20.9 / 23.5, 12 36.4 / 31.0; 1024 x 32 x 16 FP32 4 variants 32 / 37, 8 49 / 35, FP64 3 82 / 73;
// 512 x 32 x 32 FP64 10 variants 135 / 82.  k_el_ener: KKS 64^3 FP64 12 169 / 68; 128^3 FP64 3
// 167 / 196; 512 x 32 x 32 FP64 2 61 / 76, 10 232 / 196; 128 x 128 x 64 FP32 16 234 / 172.  With three
// blocks left of four either wins (FP64 64^3 6 variants 46.9 / 36.4, 128^3 6 271 / 266).
template <typename R, bool GEN>
bool stage_pars(size_t lines, size_t pars, bool ener) {
  auto blocks = [](size_t sm) { return std::min(Cfg<R, GEN>::BLOCKS, (int)((228 * 1024) / (sm + 1024))); };
  const int b = blocks(lines + pars);
  return b >= 2 && (!ener || 2 * b > blocks(lines));
}
template <typename R, int N, typename W, typename COEF>
void launch_rows(const ElRowsArgs<R>& a, const COEF& E) {
  using G = Geo<R, N, is_gen<COEF>()>;
  const size_t lines = (G::line_bytes + 15) / 16 * 16, pars = sizeof(R) * (size_t)E.nvar * G::NR * G::PS;
  const bool stage = stage_pars<R, is_gen<COEF>()>(lines, pars, false);
  const size_t sm = lines + (stage ? pars : 0);
  auto fn = stage ? k_el_rows<R, N, W, COEF, true> : k_el_rows<R, N, W, COEF, false>;
  if ((int)sm > smem_optin((const void*)fn)) throw CudaError("fused elastic rows exceed shared memory", MEU_ERR_UNSUPPORTED);
  launch_dep(fn, dim3((unsigned)((a.nrows + G::NR - 1) / G::NR)), G::NT, sm, a.st, a.sp, a.nk, a.pphi, a.n3, a.nrows,
             (const cplx<R>*)a.tw, E, a.cfac, a.err);
}
template <typename R, int N, typename COEF>
void launch_ener(const ElRowsArgs<R>& a, const COEF& E, const R* phi, const DevConst* K, R* el_en, R* elg,
                 const EnerOut<R>& out, int eta2, double* partials) {
  using G = Geo<R, N, is_gen<COEF>()>;
  const size_t lines = (G::line_bytes + 15) / 16 * 16, pars = sizeof(R) * (size_t)(2 * E.nvar) * G::NR * G::PS;
  const bool stage = stage_pars<R, is_gen<COEF>()>(lines, pars, true);
  const size_t sm = lines + (stage ? pars : 0);
  auto fn = stage ? k_el_ener<R, N, COEF, true> : k_el_ener<R, N, COEF, false>;
  if ((int)sm > smem_optin((const void*)fn))
    throw CudaError("elastic energy rows exceed shared memory", MEU_ERR_UNSUPPORTED);
  const unsigned blocks = (unsigned)std::min<int64_t>((a.nrows + G::NR - 1) / G::NR, PSTRIDE);
  fn<<<blocks, G::NT, sm, a.st>>>(a.sp, a.nk, phi, a.pphi, a.n3, a.nrows, (const cplx<R>*)a.tw, K, E, el_en, elg,
                                         out, eta2, partials, a.err);
}

// lengths of the two units of a precision (el_rows_*_a.cu: up to 128, el_rows_*_b.cu: longer)
template <int... N>
struct Lengths {};
using LenA = Lengths<16, 24, 32, 36, 48, 54, 64, 72, 96, 108, 128>;
using LenB = Lengths<144, 162, 192, 216, 256, 288, 324, 384, 432, 512, 1024>;
// fn(N as an integral constant) for N = nx; false when the unit has no kernels of that length
template <int... N, typename FN>
bool with_length(Lengths<N...>, int nx, FN&& fn) {
  return ((nx == N && (fn(std::integral_constant<int, N>{}), true)) || ...);
}
// FP32 fields with proportional moduli form the polarisation in FP64, but for rows of 64 to 1024 in
// powers of two, which take it in the field precision after a step's first iteration.  It is a
// difference of stresses, so FP32 leaves 2^-24 times the larger ones in it: strains against FP64 at 48 x 12 x 16 4.4 units of 2^-24 from FP64, 5.0 from
// FP32; under a mean strain of 0.3 53 and 103.  FP64 / FP32, us per launch: 48^3 one variant
// 15.0 / 14.2, 96^3 two 35.6 / 32.6, 108 x 144 x 96 three 54.4 / 49.2.
template <typename R, int N>
constexpr bool field_polarisation() {
  return sizeof(R) == 8 || (N >= 64 && (N & (N - 1)) == 0);
}
template <typename R, typename LEN>
bool rows_unit(const ElRowsArgs<R>& a, const ElRowsCoef<R>& c, bool fp64) {
  return with_length(LEN{}, a.nx, [&](auto n) {
    constexpr int N = decltype(n)::value;
    if (!c.prop) return launch_rows<R, N, double, ElxGen>(a, *c.gen);
    if constexpr (field_polarisation<R, N>()) {
      if (sizeof(R) == 8 || !fp64) return launch_rows<R, N, R, ElxCoef<R>>(a, *c.pr);
    }
    if constexpr (sizeof(R) == 4) launch_rows<R, N, double, ElxProp>(a, *c.p64);
  });
}
template <typename R, typename LEN>
bool ener_unit(const ElRowsArgs<R>& a, const ElRowsCoef<R>& c, const R* phi, const DevConst* K, R* el_en, R* elg,
               const EnerOut<R>& out, int eta2, double* partials) {
  return with_length(LEN{}, a.nx, [&](auto n) {
    constexpr int N = decltype(n)::value;
    if (c.prop) launch_ener<R, N, ElenProp>(a, *c.en, phi, K, el_en, elg, out, eta2, partials);
    else launch_ener<R, N, ElxGen>(a, *c.gen, phi, K, el_en, elg, out, eta2, partials);
  });
}

}  // namespace elr

}  // namespace meu
