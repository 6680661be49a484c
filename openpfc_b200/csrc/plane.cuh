// plane.cuh -- y inverse, fused x pass and y forward of one kz plane in one CTA.
//
// The step's three passes between the z updates (y inverse, x: C2R -> N -> R2C,
// y forward) touch each kz plane on its own.  Where a plane of (M+1) x N1 modes
// (one per real field) fits in shared memory, one CTA carries it through all
// three: the spectrum is read and written once instead of three times and one
// launch takes the place of three.
//
// Layout: plane[ky][kx], pitch P = M + 1 (odd, M is even), so the threads of a
// warp that hold neighbouring columns (y phases) or neighbouring rows (x phase)
// of one position hit different banks, and the Nyquist mode of a row sits where
// the C2R pairing looks for it.  Lines exchange in place; T = N / E threads own
// a line as in fft_core.cuh.  The y inverse reads its first stage from HBM into
// registers and the y forward writes its last stage from registers.
//
// Bound by latency (a plane's phases are a serial chain of loads, exchanges and
// barriers in one CTA), so it pays where the three launches it replaces were
// short.  A step of 64^3 FP32 went from 16.8 to 11.3 us, of 160x80x96 from 43 to
// 30 us, of 192x96x80 FP64 from 66 to 50 us (direct-load z update on both sides).
//
// The block is as many lines wide as the longer phase needs in equal turns
// (plane_threads); lines past the end run their barriers idle.
#pragma once
#include "aluminum.cuh"
#include "plane.h"

namespace opfc {

// Stockham stages on one line at line[p * ps]; `ok` is false for a line past
// the end (it takes part in the barriers only).
template <typename C, int N, int E, int DIR, int TWS, int Ns, int R, int... Rest>
__device__ __forceinline__ void plane_stages(C (&v)[E], C *line, int ps, int j, const C *tw, bool ok) {
  constexpr int T = N / E;
  constexpr int B = E / R;
  constexpr bool last = sizeof...(Rest) == 0;
#pragma unroll
  for (int t = 0; t < B; ++t) {
    C x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = v[t + r * B];
    const int b = j + t * T;
    const int k = (Ns > 1) ? (b % Ns) : 0;
    if constexpr (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) x[r] = twmul<DIR>(x[r], tw[k * r * (TWS / (Ns * R))]);
    }
    Dft<R, DIR, C>::run(x);
    if constexpr (last) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[t + r * B] = x[r];
    } else if (ok) {
      const int base = (b / Ns) * Ns * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) line[(base + r * Ns) * ps] = x[r];
    }
  }
  if constexpr (!last) {
    __syncthreads();
    if (ok) {
#pragma unroll
      for (int m = 0; m < E; ++m) v[m] = line[(j + T * m) * ps];
    }
    __syncthreads();
    plane_stages<C, N, E, DIR, TWS, Ns * R, Rest...>(v, line, ps, j, tw, ok);
  }
}

template <typename C, int N, int DIR, int TWS, int... Rs>
__device__ __forceinline__ void plane_fft(Radices<Rs...>, C (&v)[Plan<N>::E], C *line, int ps, int j, const C *tw,
                                          bool ok) {
  plane_stages<C, N, Plan<N>::E, DIR, TWS, 1, Rs...>(v, line, ps, j, tw, ok);
}

// y inverse of one field: HBM -> plane
template <typename C, int N>
__device__ __forceinline__ void plane_y_in(const C *in, const C *nyq, C *plane, const C *tw, int M) {
  constexpr int E = Plan<N>::E, T = N / E;
  const int P = M + 1, wc = blockDim.x / T;
  const int c = threadIdx.x % wc, j = threadIdx.x / wc;
  for (int c0 = 0; c0 <= M; c0 += wc) {
    const int kx = c0 + c;
    const bool ok = kx <= M && j < T;
    C v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int ky = j + T * m;
      v[m] = ok ? (kx < M ? in[(long long)ky * M + kx] : nyq[ky]) : mk<C>(0, 0);
    }
    plane_fft<C, N, +1, N>(typename Plan<N>::R{}, v, plane + kx, P, j, tw, ok);
    if (ok) {
#pragma unroll
      for (int m = 0; m < E; ++m) plane[(j + T * m) * P + kx] = v[m];
    }
  }
}

// y forward: plane -> HBM
template <typename C, int N>
__device__ __forceinline__ void plane_y_out(C *out, C *nyq, C *plane, const C *tw, int M) {
  constexpr int E = Plan<N>::E, T = N / E;
  const int P = M + 1, wc = blockDim.x / T;
  const int c = threadIdx.x % wc, j = threadIdx.x / wc;
  for (int c0 = 0; c0 <= M; c0 += wc) {
    const int kx = c0 + c;
    const bool ok = kx <= M && j < T;
    C v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = ok ? plane[(j + T * m) * P + kx] : mk<C>(0, 0);
    __syncthreads();  // the line is read before its first exchange overwrites it
    plane_fft<C, N, -1, N>(typename Plan<N>::R{}, v, plane + kx, P, j, tw, ok);
    if (ok) {
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const int ky = j + T * m;
        if (kx < M)
          out[(long long)ky * M + kx] = v[m];
        else
          nyq[ky] = v[m];
      }
    }
  }
}

// C2R of row `row` into registers: v[m] = field at z positions j + T m, scaled, + mean
template <typename Real, typename C, int M>
__device__ __forceinline__ void plane_x_inverse(C (&v)[Plan<M>::E], C *row, const C *tw, int j, bool ok, double scale,
                                                double mean) {
  constexpr int E = Plan<M>::E, T = M / E;
#pragma unroll
  for (int m = 0; m < E; ++m) {
    const int k = j + T * m;
    C X = mk<C>(0, 0), Y = mk<C>(0, 0);
    if (ok) {
      X = row[k];
      Y = row[M - k];
    }
    if (k == 0) {
      X.y = 0;
      Y.y = 0;
    }
    const C s = mk<C>(X.x + Y.x, X.y - Y.y);
    const C d = mk<C>(X.x - Y.x, X.y + Y.y);
    const C e = twmul<+1>(d, tw[k]);
    v[m] = mk<C>(s.x - e.y, s.y + e.x);
  }
  __syncthreads();
  plane_fft<C, M, +1, 2 * M>(typename Plan<M>::R{}, v, row, 1, j, tw, ok);
#pragma unroll
  for (int m = 0; m < E; ++m)
    v[m] = mk<C>(to_real_plus_mean(v[m].x, scale, mean), to_real_plus_mean(v[m].y, scale, mean));
}

// R2C of one row held in registers; the spectrum (modes 0..M) replaces the row
template <typename Real, typename C, int M>
__device__ __forceinline__ void plane_x_forward(C (&v)[Plan<M>::E], C *row, const C *tw, int j, bool ok) {
  constexpr int E = Plan<M>::E, T = M / E;
  plane_fft<C, M, -1, 2 * M>(typename Plan<M>::R{}, v, row, 1, j, tw, ok);
  if (ok) {
#pragma unroll
    for (int m = 0; m < E; ++m) row[j + T * m] = v[m];
  }
  __syncthreads();
  // post-processing in place, modes k and M - k together
  // (X[M-k] = conj(s + i e) / 2 with the s and e of X[k] = (s - i e) / 2)
  if (ok) {
    for (int k = j; k <= M / 2; k += T) {
      const C Z = row[k];
      if (k == 0) {
        row[0] = mk<C>(Z.x + Z.y, Real(0));
        row[M] = mk<C>(Z.x - Z.y, Real(0));
      } else {
        const C Y = row[M - k];
        const C s = mk<C>(Z.x + Y.x, Z.y - Y.y);
        const C d = mk<C>(Z.x - Y.x, Z.y + Y.y);
        const C e = twmul<-1>(d, tw[k]);
        row[k] = mk<C>(Real(0.5) * (s.x + e.y), Real(0.5) * (s.y - e.x));
        row[M - k] = mk<C>(Real(0.5) * (s.x - e.y), Real(-0.5) * (s.y + e.x));
      }
    }
  }
}

// C2R, nonlinearity and R2C of the plane's rows; the result replaces the rows of
// the last field's plane.  The earlier fields' real values wait in their own rows.
template <typename Real, int M, int MODEL>
__device__ __forceinline__ void plane_x(const PlaneArgs &a, typename Cx<Real>::T *planes, size_t psz,
                                        const typename Cx<Real>::T *tw, const AlCoef<Real> *coef, bool &bad) {
  using C = typename Cx<Real>::T;
  constexpr int E = Plan<M>::E, T = M / E, P = M + 1;
  constexpr int NF = plane_fields(MODEL);
  const int wc = blockDim.x / T;
  const int c = threadIdx.x % wc, j = threadIdx.x / wc;
  const double mean = *a.mean_dev;
  const Real c0 = (Real)a.c[0], c1 = (Real)a.c[1], c2 = (Real)a.c[2], c3 = (Real)a.c[3], c4 = (Real)a.c[4];
  for (int r0 = 0; r0 < a.n1; r0 += wc) {
    const bool ok = r0 + c < a.n1 && j < T;
    const int off = (r0 + c) * P;
    C v[E];
#pragma unroll 1
    for (int f = 0; f + 1 < NF; ++f) {
      C *row = planes + f * psz + off;
      plane_x_inverse<Real, C, M>(v, row, tw, j, ok, a.scale, MODEL == kPlaneAdjoint && f > 0 ? 0.0 : mean);
      if (ok) {
#pragma unroll
        for (int m = 0; m < E; ++m) row[j + T * m] = v[m];  // read back by this thread only
      }
    }
    C *row = planes + (NF - 1) * psz + off;
    // MK_ALUMINUM_G: the last field is P*psi, whose mean is P_F(0) times psi's
    plane_x_inverse<Real, C, M>(v, row, tw, j, ok, a.scale,
                                MODEL == MK_ALUMINUM_G ? a.al[17] * mean : MODEL == kPlaneAdjoint ? 0.0 : mean);
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const Real x = v[m].x, y = v[m].y;
      Real nx, ny;
      if constexpr (MODEL == MK_PLAIN) {
        nx = x * x * x;
        ny = y * y * y;
      } else if constexpr (MODEL == MK_FILTERED) {
        // N = p2 v^2/2 + p3 v^3/3 + p4 v^4/4 of the filtered density
        nx = x * x * (c0 + c1 * x + c2 * x * x);
        ny = y * y * (c0 + c1 * y + c2 * y * y);
      } else if constexpr (MODEL == MK_TUNGSTEN) {
        // N = p3b u^2 + p4b u^3 + q3b v^2 + q4b v^3 - stabP u
        const C u = ok ? planes[off + j + T * m] : mk<C>(0, 0);
        nx = c0 * u.x * u.x + c1 * u.x * u.x * u.x + c2 * x * x + c3 * x * x * x - c4 * u.x;
        ny = c0 * u.y * u.y + c1 * u.y * u.y * u.y + c2 * y * y + c3 * y * y * y - c4 * u.y;
      } else if constexpr (MODEL == kPlaneAdjoint) {
        const C u = ok ? planes[off + j + T * m] : mk<C>(0, 0);
        const C g = ok ? planes[psz + off + j + T * m] : mk<C>(0, 0);
        nx = g.x + Real(3) * u.x * u.x * x;
        ny = g.y + Real(3) * u.y * u.y * y;
      } else {
        const C u = ok ? planes[off + j + T * m] : mk<C>(0, 0);
        const C w = ok ? planes[psz + off + j + T * m] : mk<C>(0, 0);
        const int i0 = 2 * (j + T * m);
        nx = aluminum_nl<Real>(a.al, coef[i0], u.x, w.x, x);
        ny = aluminum_nl<Real>(a.al, coef[i0 + 1], u.y, w.y, y);
      }
      // (the flag reports the steps' nonlinearity, not a gradient's values)
      if constexpr (MODEL != kPlaneAdjoint) bad |= ok && !(isfinite(nx) && isfinite(ny));
      v[m] = mk<C>(nx, ny);
    }
    plane_x_forward<Real, C, M>(v, row, tw, j, ok);
  }
}

// R2C of the plane's rows, which hold the real values (x[2p], x[2p+1]) at p < M
template <typename Real, int M>
__device__ __forceinline__ void plane_rows_r2c(typename Cx<Real>::T *plane, int n1, const typename Cx<Real>::T *tw) {
  using C = typename Cx<Real>::T;
  constexpr int E = Plan<M>::E, T = M / E, P = M + 1;
  const int wc = blockDim.x / T;
  const int c = threadIdx.x % wc, j = threadIdx.x / wc;
  for (int r0 = 0; r0 < n1; r0 += wc) {
    const bool ok = r0 + c < n1 && j < T;
    C *row = plane + (r0 + c) * P;
    C v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = ok ? row[j + T * m] : mk<C>(0, 0);
    __syncthreads();
    plane_x_forward<Real, C, M>(v, row, tw, j, ok);
  }
}

// C2R of the plane's rows in place (real values at p < M)
template <typename Real, int M>
__device__ __forceinline__ void plane_rows_c2r(typename Cx<Real>::T *plane, int n1, const typename Cx<Real>::T *tw,
                                               double scale, double mean) {
  using C = typename Cx<Real>::T;
  constexpr int E = Plan<M>::E, T = M / E, P = M + 1;
  const int wc = blockDim.x / T;
  const int c = threadIdx.x % wc, j = threadIdx.x / wc;
  for (int r0 = 0; r0 < n1; r0 += wc) {
    const bool ok = r0 + c < n1 && j < T;
    C *row = plane + (r0 + c) * P;
    C v[E];
    plane_x_inverse<Real, C, M>(v, row, tw, j, ok, scale, mean);
    if (ok) {
#pragma unroll
      for (int m = 0; m < E; ++m) row[j + T * m] = v[m];
    }
  }
}

#define OPFC_PLANE_POW2(X) X(16) X(32) X(64) X(128) X(256) X(512)
#define OPFC_PLANE_MIXED(X) X(24) X(40) X(48) X(80) X(96)

// switch over the supported lengths (CASE(n) per length)
#define OPFC_PLANE_SWITCH(len, CASE)        \
  switch (len) {                            \
    OPFC_PLANE_POW2(CASE)                   \
    default:                                \
      if constexpr (MIXED) {                \
        switch (len) { OPFC_PLANE_MIXED(CASE) } \
      }                                     \
  }

// MIXED: a length that is no power of two occurs (up to 24 values per thread,
// one CTA per SM); the other kernels hold 8 values per thread and are compiled
// for two CTAs per SM (FP32).
template <typename Real, bool MIXED> constexpr int kPlaneCtas = (MIXED || sizeof(Real) == 8) ? 1 : 2;

template <typename Real, int MODEL, bool MIXED>
__global__ void __launch_bounds__(kPlaneThreads<Real>, kPlaneCtas<Real, MIXED>)
    plane_kernel(const __grid_constant__ PlaneArgs a) {
  using C = typename Cx<Real>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int M = a.M, n1 = a.n1, n0 = 2 * M;
  C *twy = reinterpret_cast<C *>(smraw);
  C *twx = twy + n1;
  C *planes = twx + n0;
  constexpr int NF = plane_fields(MODEL);
  const size_t psz = (size_t)(M + 1) * n1;
  for (int i = threadIdx.x; i < n1; i += blockDim.x) twy[i] = reinterpret_cast<const C *>(a.tw_y)[i];
  for (int i = threadIdx.x; i < n0; i += blockDim.x) twx[i] = reinterpret_cast<const C *>(a.tw_x)[i];
  __syncthreads();
  const long long main0 = (long long)blockIdx.x * M * n1, nyq0 = a.nyq_off + (long long)blockIdx.x * n1;
  bool bad = false;
  AlCoef<Real> *coef = nullptr;  // MK_ALUMINUM_G: per x position (visible after the y phase's barrier)
  if constexpr (MODEL == MK_ALUMINUM_G) {
    coef = reinterpret_cast<AlCoef<Real> *>(planes + NF * psz);
    const double t = *a.time;
    for (int i = threadIdx.x; i < n0; i += blockDim.x) coef[i] = aluminum_coef<Real>(a.al, t, a.al[0] + i * a.al[1]);
  }
#pragma unroll 1
  for (int f = 0; f < NF; ++f) {
    const C *in = reinterpret_cast<const C *>(a.in[f]);
#define OPFC_CASE(n) \
  case n: plane_y_in<C, n>(in + main0, in + nyq0, planes + f * psz, twy, M); break;
    OPFC_PLANE_SWITCH(n1, OPFC_CASE)
#undef OPFC_CASE
  }
  __syncthreads();
#define OPFC_CASE(n) \
  case n: plane_x<Real, n, MODEL>(a, planes, psz, twx, coef, bad); break;
  OPFC_PLANE_SWITCH(M, OPFC_CASE)
#undef OPFC_CASE
  __syncthreads();
  C *out = reinterpret_cast<C *>(a.out);
#define OPFC_CASE(n) \
  case n: plane_y_out<C, n>(out + main0, out + nyq0, planes + (NF - 1) * psz, twy, M); break;
  OPFC_PLANE_SWITCH(n1, OPFC_CASE)
#undef OPFC_CASE
  if (bad && a.flag) atomicOr(a.flag, 1u);
}

// The transform's own passes on one kz plane: x R2C and y forward (DIR < 0), or
// y inverse and x C2R (DIR > 0); a.rin / a.rout are the real rows.
template <typename Real, int DIR, bool MIXED>
__global__ void __launch_bounds__(kPlaneThreads<Real>, kPlaneCtas<Real, MIXED>)
    plane_fft_kernel(const __grid_constant__ PlaneArgs a) {
  using C = typename Cx<Real>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int M = a.M, n1 = a.n1, n0 = 2 * M, P = M + 1;
  C *twy = reinterpret_cast<C *>(smraw);
  C *twx = twy + n1;
  C *plane = twx + n0;
  for (int i = threadIdx.x; i < n1; i += blockDim.x) twy[i] = reinterpret_cast<const C *>(a.tw_y)[i];
  for (int i = threadIdx.x; i < n0; i += blockDim.x) twx[i] = reinterpret_cast<const C *>(a.tw_x)[i];
  const long long main0 = (long long)blockIdx.x * M * n1, nyq0 = a.nyq_off + (long long)blockIdx.x * n1;
  if constexpr (DIR < 0) {
    const C *rin = reinterpret_cast<const C *>(a.rin) + main0;
    for (int i = threadIdx.x; i < M * n1; i += blockDim.x) {
      const int r = i / M;
      plane[r * P + (i - r * M)] = rin[i];
    }
    __syncthreads();
#define OPFC_CASE(n) \
  case n: plane_rows_r2c<Real, n>(plane, n1, twx); break;
    OPFC_PLANE_SWITCH(M, OPFC_CASE)
#undef OPFC_CASE
    __syncthreads();
    C *out = reinterpret_cast<C *>(a.out);
#define OPFC_CASE(n) \
  case n: plane_y_out<C, n>(out + main0, out + nyq0, plane, twy, M); break;
    OPFC_PLANE_SWITCH(n1, OPFC_CASE)
#undef OPFC_CASE
  } else {
    __syncthreads();
    const C *in = reinterpret_cast<const C *>(a.in[0]);
#define OPFC_CASE(n) \
  case n: plane_y_in<C, n>(in + main0, in + nyq0, plane, twy, M); break;
    OPFC_PLANE_SWITCH(n1, OPFC_CASE)
#undef OPFC_CASE
    __syncthreads();
#define OPFC_CASE(n) \
  case n: plane_rows_c2r<Real, n>(plane, n1, twx, a.scale, a.mean); break;
    OPFC_PLANE_SWITCH(M, OPFC_CASE)
#undef OPFC_CASE
    __syncthreads();
    C *rout = reinterpret_cast<C *>(a.rout) + main0;
    for (int i = threadIdx.x; i < M * n1; i += blockDim.x) {
      const int r = i / M;
      rout[i] = plane[r * P + (i - r * M)];
    }
  }
}

template <typename Real, int MODEL, bool MIXED> static int launch_plane_t(const PlaneArgs &a, cudaStream_t s) {
  auto k = plane_kernel<Real, MODEL, MIXED>;
  const size_t smem = plane_smem(a.M, a.n1, (int)sizeof(Real), MODEL);
  // the attribute belongs to (kernel, device); set for the largest size once
  static int setup[kDevCache];
  kernel_setup(k, kPlaneThreads<Real>, (size_t)kMaxDynSmem, setup);
  k<<<a.n2, plane_threads(a.M, a.n1, (int)sizeof(Real)), smem, s>>>(a);
  return (int)cudaGetLastError();
}

template <typename Real> int launch_plane(int model, const PlaneArgs &a, cudaStream_t s) {
  if (!plane_fits(a.M, a.n1, (int)sizeof(Real), model)) return (int)cudaErrorInvalidValue;
  const bool mixed = (a.M & (a.M - 1)) || (a.n1 & (a.n1 - 1));
#define OPFC_CASE(m) \
  case m: return mixed ? launch_plane_t<Real, m, true>(a, s) : launch_plane_t<Real, m, false>(a, s);
  switch (model) {
    OPFC_CASE(MK_PLAIN) OPFC_CASE(MK_FILTERED) OPFC_CASE(MK_TUNGSTEN) OPFC_CASE(MK_ALUMINUM_G) OPFC_CASE(kPlaneAdjoint)
  }
#undef OPFC_CASE
  return (int)cudaErrorInvalidValue;
}

template <typename Real, int DIR, bool MIXED> static int launch_plane_fft_t(const PlaneArgs &a, cudaStream_t s) {
  auto k = plane_fft_kernel<Real, DIR, MIXED>;
  static int setup[kDevCache];
  kernel_setup(k, kPlaneThreads<Real>, (size_t)kMaxDynSmem, setup);
  k<<<a.n2, plane_threads(a.M, a.n1, (int)sizeof(Real)), plane_smem(a.M, a.n1, (int)sizeof(Real), MK_PLAIN), s>>>(a);
  return (int)cudaGetLastError();
}

template <typename Real> int launch_plane_fft(int dir, const PlaneArgs &a, cudaStream_t s) {
  if (!plane_fits(a.M, a.n1, (int)sizeof(Real), MK_PLAIN)) return (int)cudaErrorInvalidValue;
  const bool mixed = (a.M & (a.M - 1)) || (a.n1 & (a.n1 - 1));
  if (dir < 0) return mixed ? launch_plane_fft_t<Real, -1, true>(a, s) : launch_plane_fft_t<Real, -1, false>(a, s);
  return mixed ? launch_plane_fft_t<Real, +1, true>(a, s) : launch_plane_fft_t<Real, +1, false>(a, s);
}

// ---------------------------------------------------------------------------
// z transform between the split layout and the reference layout ((M+1) values a
// row).  A column is q = kx + (M+1) ky, so W neighbouring columns are W
// neighbouring values of every reference plane; on the split side the run breaks
// once a row.  The transform pass does the layout change, which otherwise is a
// read and a write of the whole spectrum on its own (256^3 FP64 forward and
// backward: 543 us with that and the real field's copies, 387 us without).
// ---------------------------------------------------------------------------
template <typename Real, int N, int DIR>
__global__ void __launch_bounds__(Width<Real>::W *(N / Plan<N>::E)) z_ref_kernel(const __grid_constant__ ZRefArgs a) {
  using C = typename Cx<Real>::T;
  constexpr int W = Width<Real>::W, E = Plan<N>::E, T = N / E, NT = W * T, ld = W + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  C *tw = reinterpret_cast<C *>(smraw);
  C *sm = tw + N;
  const int c = threadIdx.x % W, j = threadIdx.x / W;
  for (int i = threadIdx.x; i < N; i += NT) tw[i] = reinterpret_cast<const C *>(a.tw)[i];
  const int H = a.M + 1, cols = H * a.n1;
  const int q = blockIdx.x * W + c;
  const bool ok = q < cols;
  const int ky = q / H, kx = q - ky * H;
  const bool nyq = kx == a.M;
  const long long split0 = nyq ? a.nyq_off + ky : (long long)ky * a.M + kx;
  const long long split_s = nyq ? a.n1 : (long long)a.M * a.n1;
  const long long in0 = DIR < 0 ? split0 : q, in_s = DIR < 0 ? split_s : cols;
  const long long out0 = DIR < 0 ? q : split0, out_s = DIR < 0 ? cols : split_s;
  const C *in = reinterpret_cast<const C *>(a.in);
  C *out = reinterpret_cast<C *>(a.out);
  C v[E];
#pragma unroll
  for (int m = 0; m < E; ++m) v[m] = ok ? in[in0 + (j + T * m) * in_s] : mk<C>(0, 0);
  __syncthreads();
  fft_line<C, N, DIR, N>(v, sm, ld, c, j, tw);
  if (ok) {
#pragma unroll
    for (int m = 0; m < E; ++m) out[out0 + (j + T * m) * out_s] = v[m];
  }
}

template <typename Real, int N> static int launch_z_ref_n(int dir, const ZRefArgs &a, cudaStream_t s) {
  using C = typename Cx<Real>::T;
  constexpr int W = Width<Real>::W, NT = W * (N / Plan<N>::E);
  const size_t smem = sizeof(C) * ((size_t)N + (size_t)N * (W + 1));
  static int setup[2][kDevCache];
  const int blocks = ((a.M + 1) * a.n1 + W - 1) / W;
  if (dir < 0) {
    kernel_setup(z_ref_kernel<Real, N, -1>, NT, smem, setup[0]);
    z_ref_kernel<Real, N, -1><<<blocks, NT, smem, s>>>(a);
  } else {
    kernel_setup(z_ref_kernel<Real, N, +1>, NT, smem, setup[1]);
    z_ref_kernel<Real, N, +1><<<blocks, NT, smem, s>>>(a);
  }
  return (int)cudaGetLastError();
}

template <typename Real> int launch_z_ref(int dir, const ZRefArgs &a, cudaStream_t s) {
  switch (a.n2) {
#define OPFC_CASE(n) \
  case n: return launch_z_ref_n<Real, n>(dir, a, s);
    OPFC_SIZES(OPFC_CASE)
    OPFC_CASE(1)
#undef OPFC_CASE
  }
  return (int)cudaErrorInvalidValue;
}

// z part of the plain model's reverse step: two forward and two inverse
// transforms and the mode products in one pass (see ZAdjArgs).  With the plane
// kernel on (psi, a, w) a reverse step is two launches instead of nineteen; the
// gradient of 40 steps at 128^3 FP32 went from 28.7 to 6.3 ms with it.
template <typename Real, int N>
__global__ void __launch_bounds__(Width<Real>::W *(N / Plan<N>::E)) z_adj_kernel(const __grid_constant__ ZAdjArgs a) {
  using C = typename Cx<Real>::T;
  constexpr int W = Width<Real>::W, E = Plan<N>::E, T = N / E, NT = W * T, ld = W + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  C *tw = reinterpret_cast<C *>(smraw);
  C *sm = tw + N;
  const int c = threadIdx.x % W, j = threadIdx.x / W;
  for (int i = threadIdx.x; i < N; i += NT) tw[i] = reinterpret_cast<const C *>(a.tw)[i];
  const int ti = (a.M + W - 1) / W, mains = ti * a.n1, tiles = mains + (a.n1 + W - 1) / W;
  const C *lam = reinterpret_cast<const C *>(a.lam), *nxy = reinterpret_cast<const C *>(a.nxy);
  const C *psi = reinterpret_cast<const C *>(a.psi_hat);
  C *oa = reinterpret_cast<C *>(a.out_a), *ob = reinterpret_cast<C *>(a.out_b);
  const Real *ta = reinterpret_cast<const Real *>(a.ta), *tb = reinterpret_cast<const Real *>(a.tb);
  const Real *tar = reinterpret_cast<const Real *>(a.tar), *tbr = reinterpret_cast<const Real *>(a.tbr);
  double s = 0;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    const bool nyq = t >= mains;
    const int cg = (nyq ? t - mains : t % ti) * W + c;
    const bool ok = cg < (nyq ? a.n1 : a.M);
    const long long base = nyq ? a.nyq_off + cg : (long long)(t / ti) * a.M + cg;
    const long long fs = nyq ? a.n1 : (long long)a.M * a.n1;
    const double wgt = nyq || cg == 0 ? 1.0 : 2.0;
    C l[E], q[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
      l[m] = ok ? lam[base + (j + T * m) * fs] : mk<C>(0, 0);
      q[m] = ok ? nxy[base + (j + T * m) * fs] : mk<C>(0, 0);
    }
    __syncthreads();  // tw; the previous tile's last reads of sm
    fft_line<C, N, -1, N>(l, sm, ld, c, j, tw);
    fft_line<C, N, -1, N>(q, sm, ld, c, j, tw);
#pragma unroll
    for (int m = 0; m < E; ++m) {
      if (ok) {
        const long long i = base + (j + T * m) * fs;
        const C p = psi[i];
        const double ar = tar[i], br = tbr[i];
        s += wgt * ((double)l[m].x * (ar * p.x + br * q[m].x) + (double)l[m].y * (ar * p.y + br * q[m].y));
        const Real la = ta[i], lb = tb[i];
        q[m] = mk<C>(lb * l[m].x, lb * l[m].y);
        l[m] = mk<C>(la * l[m].x, la * l[m].y);
      }
    }
    fft_line<C, N, +1, N>(l, sm, ld, c, j, tw);
    fft_line<C, N, +1, N>(q, sm, ld, c, j, tw);
    if (ok) {
#pragma unroll
      for (int m = 0; m < E; ++m) {
        oa[base + (j + T * m) * fs] = l[m];
        ob[base + (j + T * m) * fs] = q[m];
      }
    }
  }
  // block sum in a fixed order (sm holds NT doubles: NT <= N W)
  double *red = reinterpret_cast<double *>(sm);
  __syncthreads();
  red[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double r = 0;
    for (int i = threadIdx.x; i < NT; i += 32) r += red[i];
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) r += __shfl_xor_sync(0xffffffffu, r, h);
    if (threadIdx.x == 0) a.partials[blockIdx.x] += r;
  }
}

template <typename Real, int N> static int launch_z_adj_n(const ZAdjArgs &a, cudaStream_t s) {
  using C = typename Cx<Real>::T;
  constexpr int W = Width<Real>::W, NT = W * (N / Plan<N>::E);
  const size_t smem = sizeof(C) * ((size_t)N + (size_t)N * (W + 1));
  static int setup[kDevCache];
  kernel_setup(z_adj_kernel<Real, N>, NT, smem, setup);
  const int tiles = (a.M + W - 1) / W * a.n1 + (a.n1 + W - 1) / W;
  z_adj_kernel<Real, N><<<tiles < a.npartials ? tiles : a.npartials, NT, smem, s>>>(a);
  return (int)cudaGetLastError();
}

// lengths whose block has a whole warp for the final sum
template <typename Real> int launch_z_adj(const ZAdjArgs &a, cudaStream_t s) {
  switch (a.n2) {
#define OPFC_CASE(n) \
  case n: return launch_z_adj_n<Real, n>(a, s);
    OPFC_CASE(32) OPFC_CASE(48) OPFC_CASE(64) OPFC_CASE(80) OPFC_CASE(96) OPFC_CASE(128) OPFC_CASE(256)
    OPFC_CASE(512) OPFC_CASE(1024)
#undef OPFC_CASE
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace opfc
