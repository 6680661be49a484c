// plane.h -- host side of the plane kernel (plane.cuh): y inverse, fused x pass
// and y forward of one kz plane in shared memory.
#pragma once
#include <stddef.h>

#include "launch.h"

namespace opfc {

// the plain model's reverse step as a plane_kernel "model": fields psi, a, w ->
// lambda = a + 3 psi^2 w
constexpr int kPlaneAdjoint = 16;

// real fields of a step, one shared-memory plane each
constexpr int plane_fields(int model) {
  return model == MK_TUNGSTEN ? 2 : model == MK_ALUMINUM_G || model == kPlaneAdjoint ? 3 : 1;
}

struct PlaneArgs {
  const void *in[3];  // F_z^-1 of psi (or of the filtered density), psi_MF, P*psi
  void *out;          // F_xy of N, same layout (may be in[0])
  const void *rin;    // launch_plane_fft: real rows
  void *rout;
  const void *tw_x, *tw_y;
  int M, n1, n2;
  long long nyq_off;
  double scale, mean;
  const double *mean_dev;  // launch_plane: the mean density
  double c[5];
  double al[18];  // as XLaunch
  const double *time;
  unsigned int *flag;
};

// threads the kernel is compiled for (FP64 lines hold up to 24 complex values a
// thread: 384 threads leave 168 registers each)
template <typename Real> constexpr int kPlaneThreads = sizeof(Real) == 8 ? 384 : 512;

// threads that own one line of length N (N / Plan<N>::E of fft_core.cuh)
constexpr int plane_line_threads(int N) {
  return N == 24 ? 1 : N == 40 ? 2 : N == 48 || N == 80 || N == 96 ? 4 : N / 8;
}
constexpr bool plane_len_ok(int N) {
  return N == 16 || N == 24 || N == 32 || N == 40 || N == 48 || N == 64 || N == 80 || N == 96 || N == 128 ||
         N == 256 || N == 512;
}
constexpr size_t plane_smem(int M, int n1, int rsz, int model) {
  return (size_t)2 * rsz * (n1 + 2 * (size_t)M + (size_t)plane_fields(model) * (M + 1) * n1) +
         (model == MK_ALUMINUM_G ? (size_t)3 * rsz * 2 * M : 0);  // temperature coefficients per x position
}
constexpr bool plane_fits(int M, int n1, int rsz, int model) {
  return plane_len_ok(M) && plane_len_ok(n1) && plane_smem(M, n1, rsz, model) <= 232448;
}
// Block size: the phase with more line threads (M + 1 columns of n1, or n1 rows
// of M) is cut into the fewest equal turns of at most the compiled size.
inline int plane_threads(int M, int n1, int rsz) {
  const int most = rsz == 8 ? 384 : 512;
  auto want = [&](int lines, int N) {
    const int t = plane_line_threads(N), cap = most / t;
    const int turns = (lines + cap - 1) / cap;
    return (lines + turns - 1) / turns * t;
  };
  const int y = want(M + 1, n1), x = want(n1, M), b = y > x ? y : x;
  return (b + 31) / 32 * 32;
}

// plane_kernel on every kz plane (plane_f32.cu / plane_f64.cu); cudaError_t as int
template <typename Real> int launch_plane(int model, const PlaneArgs &a, cudaStream_t s);
// dir < 0: rin -> x R2C, y forward -> out; dir > 0: in[0] -> y inverse, x C2R -> rout
template <typename Real> int launch_plane_fft(int dir, const PlaneArgs &a, cudaStream_t s);

// Fused x pass of MK_ALUMINUM_G, mean density from device memory (aluminum_f32.cu / aluminum_f64.cu)
template <typename Real> int launch_al_x(const XLaunch &L, const double *mean_dev, cudaStream_t s);

// z transform of a whole spectrum, split layout -> reference layout (dir < 0)
// or back (dir > 0)
struct ZRefArgs {
  const void *in;
  void *out;
  const void *tw;
  int M, n1, n2;
  long long nyq_off;
};
template <typename Real> int launch_z_ref(int dir, const ZRefArgs &a, cudaStream_t s);

// z part of the plain model's reverse step (split layout): with lambda_hat and
// N_hat the forward z transforms of lam and nxy,
//   partials += Re sum w conj(lambda_hat) (tar psi_hat + tbr N_hat)
//   out_a = F_z^-1[ta lambda_hat] (may be lam), out_b = F_z^-1[tb lambda_hat]
// (w = 1 on the kx = 0 and kx = M planes, else 2).  At most `npartials` blocks.
struct ZAdjArgs {
  const void *lam, *nxy, *psi_hat;
  void *out_a, *out_b;
  const void *ta, *tb, *tar, *tbr, *tw;
  int M, n1, n2;
  long long nyq_off;
  double *partials;
  int npartials;
};
template <typename Real> int launch_z_adj(const ZAdjArgs &a, cudaStream_t s);

}  // namespace opfc
