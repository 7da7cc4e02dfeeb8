// el_z.cuh -- the z direction of one elastic fixed-point iteration in one kernel: z FFT of
// the six polarisation spectra, Green operator u^ = Q(k)^-1 (kf . x^) with the convergence
// sums, strain gamma^(u^), z inverse FFT (ModElastic.f:329-430).  Included by el_z_f32.cu /
// el_z_f64.cu, which instantiate every supported length for one precision.
//
// A block holds TM columns (consecutive (ky, kx)) of all six components in shared memory:
// the first DIF stage reads global memory, the k-space work goes through the tile at the
// positions the forward stages leave (kz digit-reversed, so nothing is permuted), the last
// DIT stage writes global memory.  Per k it moves 6 + 3 complex in and 6 + 3 out; the three
// separate passes (z forward, k-space kernel, z inverse) move 42, and all of them ran at
// 4.1-5.3 TB/s, so the bytes were the cost.
#pragma once
#include "engine.cuh"
#include "fft_stages.cuh"
#include "step_kernels.cuh"

namespace meu {
namespace elz {

constexpr int PV = 3;

// Columns and threads per block.  What bounds it is latency: a block is a chain of load,
// transform, k-space and store phases, and only other warps and blocks fill the waits.
//  FP32: 16 columns, so a row of one component fills a 128-byte line (256^3, per launch:
//   16 columns x 512 threads 0.40 ms, 8 x 256 with two blocks per SM 0.44, 4 x 128 with
//   four 0.61); 8 where 16 pass 200 KB.
//  FP64: 8 columns x 256 threads while two blocks fit with room to spare (108 x 144 x 96:
//   56 us, 4 x 192 60 us), else 4 x 192 with three (128^3: 87 us, 8 x 256 94 us).
// Against the three kernels it replaced: 256^3 FP32 0.575 -> 0.40 ms, 128^3 FP64 129 -> 87 us.
template <typename R, int L>
constexpr int cols() {
  if (sizeof(R) == 4) return 6 * 16 * 8 * L <= 200 * 1024 ? 16 : 8;
  return 6 * 8 * 16 * L < 96 * 1024 ? 8 : 4;
}
template <typename R, int L>
constexpr int threads() { return sizeof(R) == 4 ? 512 : (cols<R, L>() == 8 ? 256 : 192); }
template <typename R, int L>
constexpr size_t smem_bytes() { return sizeof(cplx<R>) * (size_t)L * 6 * cols<R, L>(); }
// resident blocks per SM it is compiled for, as many as the tile leaves room for
template <typename R, int L>
constexpr int min_blocks() {
  constexpr int fit = (int)((228 * 1024) / (smem_bytes<R, L>() + L * 12 + 2048));
  constexpr int cap = sizeof(R) == 4 ? 1 : (cols<R, L>() == 8 ? 2 : 3);
  return fit < 1 ? 1 : (fit < cap ? fit : cap);
}

// The tile: element e (position along z) of component m, column c.  Rows of 6 TM complex; when
// a row's TM columns of one component fill half the banks (64 bytes), odd rows hold the
// components pairwise swapped, so that two rows read together do not meet in a bank.
template <typename C, int TM>
struct Tile {
  static constexpr int ES = 6 * TM;
  static constexpr bool SWAP = TM * (int)sizeof(C) == 64;
  static __device__ __forceinline__ int at(int m, int c, int e) {
    return e * ES + (SWAP ? (m ^ (e & 1)) : m) * TM + c;
  }
};

// One radix stage of the six components.  A task is one butterfly position (column c, j, b) of
// a group of NM components, which share its twiddles and addresses; the components are split
// into as many groups as give every thread a task.  Global side (GIN: stage input, GOUT: stage
// output): element e of column c of component m at g + m * ms + e * es + c, columns past nc
// read as column 0 and not stored.
template <typename C, int L, int S, int TM, int NT, bool FWD, bool GIN, bool GOUT>
__device__ __forceinline__ void stage6(const C* __restrict__ tw, C* buf, C* g, int64_t es, int64_t ms, int nc) {
  using T = fz::StageOf<L, S, PV>;
  using A = Tile<C, TM>;
  constexpr int PER = TM * T::TASKS;  // tasks of one group
  // FP64 keeps one component per task (its radix-16 butterflies leave no registers to share)
  constexpr int G = sizeof(C) == 16 ? 6 : PER >= NT ? 1 : (2 * PER >= NT ? 2 : 3), NM = 6 / G;
  // held in registers across the group where they fit (double radix 12 and 16 reload them)
  constexpr bool HOLD = sizeof(C) == 8 || T::R <= 9;
#pragma unroll 1
  for (int t = threadIdx.x; t < PER * G; t += NT) {
    const int c = t % TM, v = t / TM, gr = v % G, u = v / G, j = u % T::M, b = u / T::M;
    const int e0 = b * T::SPAN + j;
    C* gp = g + (int64_t)(gr * NM) * ms + e0 * es + (c < nc ? c : 0);
    C w[T::R];
    if (HOLD && T::M > 1) {
#pragma unroll
      for (int q = 1; q < T::R; ++q) w[q] = tw[j * q * T::TWS];
    }
#pragma unroll 1
    for (int m = 0; m < NM; ++m) {
      // element r of the butterfly in the tile: rows r * M apart, of the parity of e0 + r * M
      C* s0 = buf + A::at(gr * NM + m, c, e0);
      C* s1 = A::SWAP ? buf + e0 * A::ES + ((gr * NM + m) ^ (~e0 & 1)) * TM + c : s0;
      C x[T::R];
#pragma unroll
      for (int r = 0; r < T::R; ++r)
        x[r] = GIN ? gp[r * (T::M * es)] : (((r * T::M) & 1) ? s1 : s0)[r * T::M * A::ES];
      if (FWD) {
        Dft<T::R, -1, C>::run(x);
        if (T::M > 1) {
#pragma unroll
          for (int q = 1; q < T::R; ++q) x[q] = cmul(x[q], HOLD ? w[q] : tw[j * q * T::TWS]);
        }
      } else {
        if (T::M > 1) {
#pragma unroll
          for (int q = 1; q < T::R; ++q) x[q] = cmulc(x[q], HOLD ? w[q] : tw[j * q * T::TWS]);
        }
        Dft<T::R, 1, C>::run(x);
      }
      if (GOUT) {
        if (c < nc) {
#pragma unroll
          for (int q = 0; q < T::R; ++q) gp[q * (T::M * es)] = x[q];
        }
      } else {
#pragma unroll
        for (int q = 0; q < T::R; ++q) (((q * T::M) & 1) ? s1 : s0)[q * T::M * A::ES] = x[q];
      }
      gp += ms;
    }
  }
}
// stages S, S+1, .. SEND-1 (FWD) or S, S-1, .. SEND+1 in shared memory, a barrier after each
template <typename C, int L, int TM, int NT, bool FWD, int S, int SEND>
__device__ __forceinline__ void stages6(C* buf, const C* tw) {
  if constexpr (FWD ? (S < SEND) : (S > SEND)) {
    stage6<C, L, S, TM, NT, FWD, false, false>(tw, buf, nullptr, 0, 0, TM);
    __syncthreads();
    stages6<C, L, TM, NT, FWD, FWD ? S + 1 : S - 1, SEND>(buf, tw);
  }
}

template <typename R, int L>
__global__ void __launch_bounds__((threads<R, L>()), (min_blocks<R, L>()))
    k_el_z(cplx<R>* sp, cplx<R>* uk, int64_t nk, const cplx<R>* __restrict__ tw,
           const __grid_constant__ ElzCoef E, double* part) {
  using C = cplx<R>;
  constexpr int TM = cols<R, L>(), NT = threads<R, L>(), NS = fz::rplan(L, PV).ns;
  using A = Tile<C, TM>;
  static_assert(NS >= 2, "first and last stage must differ");
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  __shared__ double az[L];
  __shared__ int kzt[L];
  __shared__ double cax[TM], cbx[TM], cay[TM], cby[TM], cw[TM];
  const int c0 = blockIdx.x * TM, nc = min(TM, E.inner - c0), tid = threadIdx.x;
  for (int p = tid; p < L; p += NT) {
    const int kz = fz::rev<L, PV>(p);
    kzt[p] = kz;
    az[p] = (double)(kz <= L / 2 ? kz : kz - L) * (6.283185307179586476925286766559 / (double)L);
  }
  if (tid < TM) {
    const int m = min(c0 + tid, E.inner - 1), ky = m / E.nxh, kx = m - ky * E.nxh;
    const double ax = (double)kx * E.wx, ay = (double)(ky <= E.ny / 2 ? ky : ky - E.ny) * E.wy;
    cax[tid] = ax;
    cay[tid] = ay;
    cbx[tid] = 2 * kx == E.nx ? 0.0 : ax;
    cby[tid] = 2 * ky == E.ny ? 0.0 : ay;
    cw[tid] = (kx == 0 || 2 * kx == E.nx) ? 1.0 : 2.0;
  }
  const int64_t inner = E.inner;
  C* src = sp + c0;
  dep_enter();
  stage6<C, L, 0, TM, NT, true, true, false>(tw, buf, src, inner, nk, nc);
  __syncthreads();
  stages6<C, L, TM, NT, true, 1, NS>(buf, tw);
  // ---- k-space: every point of the tile, the previous u^ of the next point in flight
  double er[6] = {0, 0, 0, 0, 0, 0};
  C uo[3] = {};
  auto fetch = [&](int i, C* o) {
    const int p = i / TM, c = i - p * TM;
    if (i < L * TM && c < nc) {
      const C* s = uk + (int64_t)kzt[p] * inner + c0 + c;
#pragma unroll
      for (int d = 0; d < 3; ++d) o[d] = s[d * nk];
    }
  };
  fetch(tid, uo);
#pragma unroll 1
  for (int i = tid; i < L * TM; i += NT) {
    C un[3] = {};
    fetch(i + NT, un);
    const int p = i / TM, c = i - p * TM, kz = kzt[p];
    C* e = buf + p * A::ES + c;
    const int sw = A::SWAP ? p & 1 : 0;
    const double ax = cax[c], ay = cay[c], a2 = az[p];
    const double bx = cbx[c], by = cby[c], bz = 2 * kz == L ? 0.0 : a2;
    double xr[6], xi[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const C v = e[(m ^ sw) * TM];
      xr[m] = (double)v.x * E.scale;
      xi[m] = (double)v.y * E.scale;
    }
    // R = kf . x (Voigt 1..6 -> x1 x2 x3 x4 x5 x6), times the power of two Q was scaled by
    const double tr1 = xr[0] * bx + xr[5] * by + xr[4] * bz, ti1 = xi[0] * bx + xi[5] * by + xi[4] * bz;
    const double tr2 = xr[5] * bx + xr[1] * by + xr[3] * bz, ti2 = xi[5] * bx + xi[1] * by + xi[3] * bz;
    const double tr3 = xr[4] * bx + xr[3] * by + xr[2] * bz, ti3 = xi[4] * bx + xi[3] * by + xi[2] * bz;
    double ur[3] = {0, 0, 0}, ui[3] = {0, 0, 0};
    if (p != 0 || c0 + c != 0) {
      const double Kv[6] = {ax * ax, ay * ay, a2 * a2, by * bz, bx * bz, bx * by};
      double q[6];
      if (E.ortho) {
#pragma unroll
        for (int m = 0; m < 3; ++m) q[m] = E.q[m][0] * Kv[0] + E.q[m][1] * Kv[1] + E.q[m][2] * Kv[2];
#pragma unroll
        for (int m = 3; m < 6; ++m) q[m] = E.q[m][m] * Kv[m];
      } else {
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          double acc = 0;
#pragma unroll
          for (int n = 0; n < 6; ++n) acc += E.q[m][n] * Kv[n];
          q[m] = acc;
        }
      }
      // adjugate of the symmetric [[q0, q5, q4], [q5, q1, q3], [q4, q3, q2]]
      const double i00 = q[1] * q[2] - q[3] * q[3], i01 = q[4] * q[3] - q[2] * q[5], i02 = q[5] * q[3] - q[1] * q[4];
      const double i11 = q[0] * q[2] - q[4] * q[4], i12 = q[5] * q[4] - q[0] * q[3], i22 = q[0] * q[1] - q[5] * q[5];
      const double rd = E.qs / (q[0] * i00 + q[5] * i01 + q[4] * i02);
      const double Rr[3] = {-ti1 * rd, -ti2 * rd, -ti3 * rd}, Ri[3] = {tr1 * rd, tr2 * rd, tr3 * rd};
      ur[0] = i00 * Rr[0] + i01 * Rr[1] + i02 * Rr[2];
      ui[0] = i00 * Ri[0] + i01 * Ri[1] + i02 * Ri[2];
      ur[1] = i01 * Rr[0] + i11 * Rr[1] + i12 * Rr[2];
      ui[1] = i01 * Ri[0] + i11 * Ri[1] + i12 * Ri[2];
      ur[2] = i02 * Rr[0] + i12 * Rr[1] + i22 * Rr[2];
      ui[2] = i02 * Ri[0] + i12 * Ri[1] + i22 * Ri[2];
    }
    // gamma = i (b (x) u) symmetrised, engineering Voigt order 11,22,33,23,13,12
    e[(0 ^ sw) * TM] = mk((R)(-bx * ui[0]), (R)(bx * ur[0]));
    e[(1 ^ sw) * TM] = mk((R)(-by * ui[1]), (R)(by * ur[1]));
    e[(2 ^ sw) * TM] = mk((R)(-bz * ui[2]), (R)(bz * ur[2]));
    e[(3 ^ sw) * TM] = mk((R)(-(by * ui[2] + bz * ui[1])), (R)(by * ur[2] + bz * ur[1]));
    e[(4 ^ sw) * TM] = mk((R)(-(bx * ui[2] + bz * ui[0])), (R)(bx * ur[2] + bz * ur[0]));
    e[(5 ^ sw) * TM] = mk((R)(-(bx * ui[1] + by * ui[0])), (R)(bx * ur[1] + by * ur[0]));
    if (c < nc) {
      const double w = cw[c];
      C* d = uk + (int64_t)kz * inner + c0 + c;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double orr = (double)uo[k].x, oi = (double)uo[k].y, dr = ur[k] - orr, di = ui[k] - oi;
        er[2 * k] += w * (dr * dr + di * di);
        er[2 * k + 1] += w * (orr * orr + oi * oi);
        d[k * nk] = mk((R)ur[k], (R)ui[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) uo[k] = un[k];
  }
  __syncthreads();
  stages6<C, L, TM, NT, false, NS - 1, 0>(buf, tw);
  stage6<C, L, 0, TM, NT, false, false, true>(tw, buf, src, inner, nk, nc);
  // block partials of the six sums
  __shared__ double red[NT / 32][6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const double v = warp_sum(er[q]);
    if ((tid & 31) == 0) red[tid >> 5][q] = v;
  }
  __syncthreads();
  if (tid < 6) {
    double v = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) v += red[w][tid];
    part[(int64_t)tid * gridDim.x + blockIdx.x] = v;
  }
}

template <typename R, int L>
void launch(cplx<R>* sp, cplx<R>* uk, int64_t nk, const void* tw, const ElzCoef& E, double* part, cudaStream_t st) {
  constexpr size_t sm = smem_bytes<R, L>();
  const int blocks = (E.inner + cols<R, L>() - 1) / cols<R, L>();
  if ((int)sm > smem_optin((const void*)k_el_z<R, L>)) throw CudaError("elastic z tile exceeds shared memory", MEU_ERR_UNSUPPORTED);
  launch_dep(k_el_z<R, L>, dim3(blocks), threads<R, L>(), sm, st, sp, uk, nk, (const cplx<R>*)tw, E, part);
}

}  // namespace elz

// lengths with a compile-time kernel (the mixed plan, two or three stages)
#define MEU_MIX_LENGTHS(X) \
  X(16) X(24) X(32) X(36) X(48) X(54) X(64) X(72) X(96) X(108) X(128) X(144) X(162) X(192) X(216) X(256) X(288) X(324) \
  X(384) X(432) X(512)

template <typename R>
int el_z_blocks(int nz, int inner) {
  switch (nz) {
#define MEU_CASE(L) case L: return (inner + elz::cols<R, L>() - 1) / elz::cols<R, L>();
    MEU_MIX_LENGTHS(MEU_CASE)
#undef MEU_CASE
    default: return 0;
  }
}
template <typename R>
void el_z_launch(const FFT3& f, cplx<R>* sp, cplx<R>* uk, const ElzCoef& E, double* part, cudaStream_t st) {
  switch (f.nz) {
#define MEU_CASE(L) case L: elz::launch<R, L>(sp, uk, f.nk(), f.pz.tw, E, part, st); break;
    MEU_MIX_LENGTHS(MEU_CASE)
#undef MEU_CASE
    default: throw CudaError("internal: elastic z kernel for an unsupported length", MEU_ERR_UNSUPPORTED);
  }
}

}  // namespace meu
