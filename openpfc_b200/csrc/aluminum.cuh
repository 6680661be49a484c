// aluminum.cuh -- fused x pass of the Aluminum model with a moving temperature
// gradient: C2R of psi, psi_MF and P*psi, nonlinearity, R2C.
//
// The temperature depends on x and the time only, so the three coefficients it
// enters (one exp and four divisions in FP64) are computed once per x position
// and CTA, into shared memory, instead of once per cell: a CTA's W rows share
// them.  Where shared memory allows, the rows of the three fields are loaded
// together, one wait on memory instead of three.
#pragma once
#include "kernels.cuh"

namespace opfc {

// coefficients of N at position x and time t (Aluminum.hpp:270-307; al as
// XLaunch::al): q2N v + q3 v^2 - kern q beside the constant terms
template <typename Real> struct AlCoef {
  Real q2, q3, kern;
};
template <typename Real> __device__ __forceinline__ AlCoef<Real> aluminum_coef(const double *al, double t, double x) {
  const double dist = x + al[3] - (x > al[4] ? al[2] : 0.0);
  const double Tv = al[5] * (dist - al[6] - al[7] * t);
  AlCoef<Real> c;
  c.q2 = (Real)(al[10] * Tv / al[8]);
  c.q3 = (Real)(al[12] * (al[9] + Tv) / al[8] + al[11]);
  c.kern = (Real)(-(1.0 - exp(-Tv / al[8])));
  return c;
}
template <typename Real>
__device__ __forceinline__ Real aluminum_nl(const double *al, const AlCoef<Real> &c, Real u, Real v, Real q) {
  return (Real)al[13] * u * u + (Real)al[14] * u * u * u + c.q2 * v + c.q3 * v * v + (Real)al[15] * v * v * v -
         c.kern * q - (Real)al[16] * u;
}

// shared memory: twiddles, the coefficients of the N0 positions, 3 or 1 row tiles
template <typename Real, int M> struct AlCfg {
  using C = typename Cx<Real>::T;
  static constexpr int W = Width<Real>::W;
  static constexpr size_t TILE = sizeof(C) * (size_t)(M + 1) * (W + 1);
  static constexpr size_t FIX = sizeof(C) * 2 * M + sizeof(AlCoef<Real>) * 2 * M;
  static constexpr int NB = FIX + 3 * TILE <= 113 * 1024 ? 3 : 1;  // two CTAs per SM
  static constexpr size_t SMEM = FIX + NB * TILE;
};

template <typename Real, int M>
__global__ void __launch_bounds__(Width<Real>::W *(M / Plan<M>::E)) al_x_kernel(const __grid_constant__ XArgs<Real> a, const double *mean_dev) {
  using C = typename Cx<Real>::T;
  using Cfg = AlCfg<Real, M>;
  constexpr int W = Cfg::W, E = Plan<M>::E, T = M / E, NT = W * T, ld = W + 1, N0 = 2 * M, NB = Cfg::NB;
  extern __shared__ __align__(16) unsigned char smraw[];
  C *tw = reinterpret_cast<C *>(smraw);
  C *tile = tw + N0;
  AlCoef<Real> *coef = reinterpret_cast<AlCoef<Real> *>(tile + (size_t)NB * (M + 1) * ld);
  const int tid = threadIdx.x, c = tid % W, j = tid / W;
  const int row0 = blockIdx.x * W;
  const void *src[3] = {a.in0, a.in1, a.in2};
  for (int i = tid; i < N0; i += NT) tw[i] = reinterpret_cast<const C *>(a.tw)[i];
  if constexpr (NB == 3) {
#pragma unroll
    for (int f = 0; f < 3; ++f)
      x_load_rows<C, M, W, NT>(reinterpret_cast<const C *>(src[f]), a.nyq_off, row0, a.rows,
                               tile + (size_t)f * (M + 1) * ld, tid);
  }
  const double t = *a.time, mean0 = *mean_dev;
  for (int i = tid; i < N0; i += NT) coef[i] = aluminum_coef<Real>(a.al, t, a.al[0] + i * a.al[1]);
  C fld[3][E];
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    C *buf = tile + (size_t)(NB == 3 ? f : 0) * (M + 1) * ld;
    if constexpr (NB == 1)
      x_load_rows<C, M, W, NT>(reinterpret_cast<const C *>(src[f]), a.nyq_off, row0, a.rows, buf, tid);
    if (NB == 1 || f == 0) __syncthreads();
    x_pre<C, M, W, E>(buf, tw, c, j, fld[f]);
    __syncthreads();
    fft_line<C, M, +1, N0>(fld[f], buf, ld, c, j, tw);
    // the mean of P*psi is P_F(0) times that of psi
    const double mean = f == 2 ? a.al[17] * mean0 : mean0;
#pragma unroll
    for (int m = 0; m < E; ++m)
      fld[f][m] = mk<C>(to_real_plus_mean(fld[f][m].x, a.scale, mean), to_real_plus_mean(fld[f][m].y, a.scale, mean));
  }
  C v[E];
  bool bad = false;
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int i0 = 2 * (j + T * m);
    const Real nx = aluminum_nl<Real>(a.al, coef[i0], fld[0][m].x, fld[1][m].x, fld[2][m].x);
    const Real ny = aluminum_nl<Real>(a.al, coef[i0 + 1], fld[0][m].y, fld[1][m].y, fld[2][m].y);
    bad |= !(isfinite(nx) && isfinite(ny));
    v[m] = mk<C>(nx, ny);
  }
  if (bad && a.flag) atomicOr(a.flag, 1u);
  fft_line<C, M, -1, N0>(v, tile, ld, c, j, tw);
#pragma unroll
  for (int m = 0; m < E; ++m) tile[(j + T * m) * ld + c] = v[m];
  __syncthreads();
  x_post_store<C, M, W, NT>(tile, tw, reinterpret_cast<C *>(a.out), a.nyq_off, row0, a.rows, tid);
}

template <typename Real, int M> static int launch_al_x_m(const XLaunch &L, const double *mean_dev, cudaStream_t s) {
  using Cfg = AlCfg<Real, M>;
  constexpr int NT = Cfg::W * (M / Plan<M>::E);
  static int setup[kDevCache];
  kernel_setup(al_x_kernel<Real, M>, NT, Cfg::SMEM, setup);
  al_x_kernel<Real, M><<<(L.rows + Cfg::W - 1) / Cfg::W, NT, Cfg::SMEM, s>>>(x_args<Real>(L), mean_dev);
  return (int)cudaGetLastError();
}

template <typename Real> int launch_al_x(const XLaunch &L, const double *mean_dev, cudaStream_t s) {
  switch (L.M) {
#define OPFC_CASE(n) \
  case n: return launch_al_x_m<Real, n>(L, mean_dev, s);
    OPFC_SIZES(OPFC_CASE)
    OPFC_CASE(1)
#undef OPFC_CASE
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace opfc
