// ens_plane.cuh -- y inverse, fused x pass and y forward of an ensemble, one
// member's kz plane per CTA (plane.cuh): one launch and one read and write of the
// spectra in place of three.  Used where that was measured to win (plane_pays in
// ensemble.cu: 64 cubes of 64 FP32 248 to 214 us a step).
//
// Members' planes are at most 65 x 128 modes, so every one fits.  Blocks have
// 288 threads: 36 lines of a 64-point column (33 are needed), 72 of an 80- or
// 96-point one.  Planes are walked in members sorted by plane size, longest
// first, so that the CTAs that run together run the same length's code.
#pragma once
#include "ensemble.cuh"
#include "plane.cuh"

namespace opfc {

constexpr int kEnsPlaneThreads = 288;

template <typename Real> __global__ void __launch_bounds__(kEnsPlaneThreads, 2) ens_plane_kernel(const EnsArgs a) {
  using C = typename Cx<Real>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int k = ens_find(a.prefix, a.count, blockIdx.x);
  const EnsInst *in = a.inst + a.order[k];
  const int M = in->M, n1 = in->n1, n0 = 2 * M;
  C *twy = reinterpret_cast<C *>(smraw);
  C *twx = twy + n1;
  C *plane = twx + n0;
  const C *tw = reinterpret_cast<const C *>(a.tw);
  for (int i = threadIdx.x; i < n1; i += blockDim.x) twy[i] = tw[in->tw1 + i];
  for (int i = threadIdx.x; i < n0; i += blockDim.x) twx[i] = tw[in->tw0 + i];
  __syncthreads();
  const int z = blockIdx.x - a.prefix[k];
  C *main = reinterpret_cast<C *>(a.work) + in->off_c + (long long)z * M * n1;
  C *nyq = reinterpret_cast<C *>(a.work) + in->off_c + (long long)M * n1 * in->n2 + (long long)z * n1;
  PlaneArgs p;
  p.n1 = n1;
  p.scale = 1.0 / ((double)n0 * n1 * in->n2);
  p.mean_dev = &in->mean;
  bool bad = false;
#define OPFC_ENS_PLANE_Y(X) X(16) X(32) X(48) X(64) X(80) X(96) X(128)
#define OPFC_ENS_PLANE_X(X) X(16) X(24) X(32) X(40) X(48) X(64)
#define OPFC_CASE(n) \
  case n: plane_y_in<C, n>(main, nyq, plane, twy, M); break;
  switch (n1) { OPFC_ENS_PLANE_Y(OPFC_CASE) }
#undef OPFC_CASE
  __syncthreads();
#define OPFC_CASE(n) \
  case n: plane_x<Real, n, MK_PLAIN>(p, plane, 0, twx, nullptr, bad); break;
  switch (M) { OPFC_ENS_PLANE_X(OPFC_CASE) }
#undef OPFC_CASE
  __syncthreads();
#define OPFC_CASE(n) \
  case n: plane_y_out<C, n>(main, nyq, plane, twy, M); break;
  switch (n1) { OPFC_ENS_PLANE_Y(OPFC_CASE) }
#undef OPFC_CASE
  if (bad && a.flag) atomicOr(a.flag, 1u);
}

template <typename Real> int ens_launch_plane(int planes, size_t smem, const EnsArgs &a, cudaStream_t s) {
  static int setup[kDevCache];
  kernel_setup(ens_plane_kernel<Real>, kEnsPlaneThreads, (size_t)kMaxDynSmem, setup);
  ens_plane_kernel<Real><<<planes, kEnsPlaneThreads, smem, s>>>(a);
  return (int)cudaGetLastError();
}

}  // namespace opfc
