// Broken-line helix fits on B200, one thread per tuple, FP64 as in the
// reference, for 3-hit tuples, 4-hit tuples and 5-hit tuples fitted on
// their first four hits (fit5as4).  Reference: plugin-PixelTriplets/
// BrokenLineFitOnGPU.h:25-182 (kernelBLFastFit/kernelBLFit), BrokenLine.h:46-504,
// choleskyInversion.h:22-161, TrajectoryStateSoA.h:30-47.
//
// Products are accumulated over the inner index in ascending order, starting
// from the first term, and the kernels are compiled without FMA contraction,
// so results agree with the serial build to the last bit except where the
// device and host transcendental functions (atan2, sin, cos, log, asinhf)
// round differently.
#include <atomic>

#include "device_utils.cuh"
#include "pixgpu_internal.cuh"

namespace pixgpu {

namespace {

// Block sizes and blocks per SM of the fits, measured on 1M 4-hit broken-line
// tuples and 200k 4-hit Riemann tuples:
// - broken line: 256 threads, two blocks (128 registers) 246 us; 320 threads
//   (96 registers, spills) 252 us; 512 threads, one block 291 us, 128 threads,
//   four blocks 310 us; without the phases' barriers 285 us.
// - Riemann (its matrices live in local memory, so registers matter less
//   than warps): 128 threads, four blocks 371 us; three blocks (168
//   registers) 440 us, two (255 registers) 500 us; barriers between its
//   phases cost more than they saved (478 us at 384 threads).
constexpr uint32_t kFitBlock = 256;
constexpr uint32_t kRiemannBlock = 128;

#include "fit_linalg.cuh"
#include "k_fit_riemann.cuh"

__device__ __forceinline__ double multScatt(double length, double B, double R, double slope) {
  double pt2 = fmin(20., B * R);
  pt2 *= pt2;
  constexpr double XXI_0 = 0.06 / 16.;
  constexpr double fact = 0.7 * ((13.6 / 1000.) * (13.6 / 1000.));
  return fact / (pt2 * (1. + sqr(slope))) * (fabs(length) * XXI_0) * sqr(1. + 0.038 * log(fabs(length) * XXI_0));
}

__device__ __forceinline__ M<2, 2> rotationMatrix(double slope) {
  M<2, 2> r;
  r(0, 0) = 1. / sqrt(1. + sqr(slope));
  r(0, 1) = slope * r(0, 0);
  r(1, 0) = -r(0, 1);
  r(1, 1) = r(0, 0);
  return r;
}

__device__ __forceinline__ double cross2D(double ax, double ay, double bx, double by) { return ax * by - ay * bx; }

// kNoDca: row and column 1 of cov are zero (their terms are left out)
template <bool kNoDca>
__device__ __forceinline__ void translateKarimaki(double* par, M<3, 3>& cov, double x0, double y0) {
  double s0, c0;
  s0 = sin(par[0]);
  c0 = cos(par[0]);
  double DP = x0 * c0 + y0 * s0;
  double DO = x0 * s0 - y0 * c0 + par[1];
  double uu = 1 + par[2] * par[1];
  double C = -par[2] * y0 + uu * c0;
  double BB = par[2] * x0 + uu * s0;
  double A = 2. * DO + par[2] * (sqr(DO) + sqr(DP));
  double U = sqrt(1. + par[2] * A);
  double xi = 1. / (sqr(BB) + sqr(C));
  double v = 1. + par[2] * DO;
  double lambda = (0.5 * A) / (U * sqr(1. + U));
  double mu = 1. / (U * (1. + U)) + par[2] * lambda;
  double zeta = sqr(DO) + sqr(DP);
  // J = (J0; J1; 0 0 1)
  const double J0[3] = {xi * uu * v, -xi * sqr(par[2]) * DP, xi * DP};
  const double J1[3] = {2. * mu * uu * DP, 2. * mu * v, mu * zeta - lambda * A};
  par[0] = atan2(BB, C);
  par[1] = A / (1 + U);
  M<3, 3> t;  // J cov
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (kNoDca && k == 1) continue;
    t(0, k) = kNoDca ? J0[0] * cov(0, k) + J0[2] * cov(2, k)
                     : J0[0] * cov(0, k) + J0[1] * cov(1, k) + J0[2] * cov(2, k);
    t(1, k) = kNoDca ? J1[0] * cov(0, k) + J1[2] * cov(2, k)
                     : J1[0] * cov(0, k) + J1[1] * cov(1, k) + J1[2] * cov(2, k);
    t(2, k) = cov(2, k);
  }
  const double nil = kNoDca ? 0. : 0. * (cov(0, 0) + cov(0, 1) + cov(0, 2) + cov(1, 1) + cov(1, 2));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    cov(i, 0) = kNoDca ? t(i, 0) * J0[0] + t(i, 2) * J0[2] : t(i, 0) * J0[0] + t(i, 1) * J0[1] + t(i, 2) * J0[2];
    cov(i, 1) = kNoDca ? t(i, 0) * J1[0] + t(i, 2) * J1[2] : t(i, 0) * J1[0] + t(i, 1) * J1[1] + t(i, 2) * J1[2];
    cov(i, 2) = kNoDca ? t(i, 2) : t(i, 2) + nil;  // J's zeros times a non-finite element
  }
}

// The symmetric band matrix of the hits' weights and the kinks at the inner
// hits, kink by kink: the kink at i couples hits i - 1, i and i + 1.  The
// terms of an element are added in ascending order of their kink's distance
// from it, as the reference's element-wise sums add them (first the weight,
// then the kinks at i - 1, i and i + 1 of a diagonal element; first the kink
// at i, then at i + 1 of an element next to it).
template <int N>
__device__ __forceinline__ M<N, N> matrixCu(const double* w, const double* S, const double* VarBeta) {
  constexpr int n = N;
  M<N, N> C;
#pragma unroll
  for (int k = 0; k < N * N; ++k) C.a[k] = 0;
  // per kink: d0, d1 the lengths on its two sides, ratio (d0 + d1) / (d1 d0)
  double d0[N], d1[N], ratio[N];
#pragma unroll
  for (int k = 1; k < n - 1; ++k) {
    d0[k] = S[k] - S[k - 1];
    d1[k] = S[k + 1] - S[k];
    ratio[k] = (S[k + 1] - S[k - 1]) / (d1[k] * d0[k]);
  }
#pragma unroll
  for (int i = 0; i < n; ++i) {
    C(i, i) = w[i];
    if (i > 1) C(i, i) += 1. / (VarBeta[i - 1] * sqr(d1[i - 1]));
    if (i > 0 && i < n - 1) C(i, i) += (1. / VarBeta[i]) * sqr(ratio[i]);
    if (i < n - 2) C(i, i) += 1. / (VarBeta[i + 1] * sqr(d0[i + 1]));
    if (i > 0 && i < n - 1) C(i, i + 1) = 1. / (VarBeta[i] * d1[i]) * -ratio[i];
    if (i < n - 2) {
      const double t = 1. / (VarBeta[i + 1] * d0[i + 1]) * -ratio[i + 1];
      C(i, i + 1) = i > 0 ? C(i, i + 1) + t : t;
      C(i, i + 2) = 1. / (VarBeta[i + 1] * d1[i + 1] * d0[i + 1]);
    }
  }
#pragma unroll
  for (int j = 0; j < n; ++j)
#pragma unroll
    for (int i = j + 1; i < n; ++i) C(i, j) = C(j, i);
  return C;
}

// hits: x,y,z of hit i at H[3*i+k]; ge: 6 floats per hit
template <int N>
__device__ void blFit(const double* H3, const float* ge, double B, FitOut& out) {
  constexpr int n = N;
  auto H = [&](int r, int c) { return H3[3 * c + r]; };
  double ff[4];
  {
    double ax = H(0, n / 2) - H(0, 0), ay = H(1, n / 2) - H(1, 0);
    double bx = H(0, n - 1) - H(0, n / 2), by = H(1, n - 1) - H(1, n / 2);
    double cx = H(0, 0) - H(0, n - 1), cy = H(1, 0) - H(1, n - 1);
    double tmp = 0.5 / cross2D(cx, cy, ax, ay);
    double csq = cx * cx + cy * cy, asq = ax * ax + ay * ay, bsq = bx * bx + by * by;
    ff[0] = H(0, 0) - (ay * csq + cy * asq) * tmp;
    ff[1] = H(1, 0) + (ax * csq + cx * asq) * tmp;
    ff[2] = sqrt(asq * bsq * csq) / (2. * fabs(cross2D(bx, by, ax, ay)));
    double dx = H(0, 0) - ff[0], dy = H(1, 0) - ff[1];
    double ex = H(0, n - 1) - ff[0], ey = H(1, n - 1) - ff[1];
    ff[3] = ff[2] * atan2(cross2D(dx, dy, ex, ey), dx * ex + dy * ey) / (H(2, n - 1) - H(2, 0));
  }
  // Bound by instruction issue and latency (FP64 with its divisions, square
  // roots and transcendental functions, which the compiler does not merge
  // across their slow-path branches): quantities that the reference's three
  // functions each form are formed once and kept (the slope and its rotation,
  // the scattering variance of each step, the hits' radii), and products with
  // the Jacobians' constant zeros and ones are left out.  Every value keeps
  // its bits.  5137 -> about 4500 instructions per 4-hit tuple.
  int q;
  double radii[2][N], rad[N], s[N], S[N], Z[N], VarBeta[N], ms01, slope;
  M<2, 2> R;
  {
    double dx = H(0, 1) - H(0, 0), dy = H(1, 1) - H(1, 0);
    double ex = H(0, n - 1) - H(0, n - 2), ey = H(1, n - 1) - H(1, n - 2);
    q = cross2D(dx, dy, ex, ey) > 0 ? -1 : 1;
    slope = -q / ff[3];
    R = rotationMatrix(slope);
#pragma unroll
    for (int i = 0; i < n; ++i) {
      radii[0][i] = H(0, i) - ff[0] * 1.0;
      radii[1][i] = H(1, i) - ff[1] * 1.0;
      rad[i] = sqrt(radii[0][i] * radii[0][i] + radii[1][i] * radii[1][i]);
    }
    double nrm = sqrt(ff[0] * ff[0] + ff[1] * ff[1]);
    double e0 = (-ff[2] * ff[0]) / nrm, e1 = (-ff[2] * ff[1]) / nrm;
#pragma unroll
    for (int i = 0; i < n; ++i)
      s[i] = q * ff[2] * atan2(cross2D(radii[0][i], radii[1][i], e0, e1), radii[0][i] * e0 + radii[1][i] * e1);
    PG_FIT_PHASE();
#pragma unroll
    for (int i = 0; i < n; ++i) {
      double p0 = s[i], p1 = H(2, i);
      S[i] = R(0, 0) * p0 + R(0, 1) * p1;
      Z[i] = R(1, 0) * p0 + R(1, 1) * p1;
    }
    VarBeta[0] = VarBeta[n - 1] = 0;
    double ms = ms01 = multScatt(S[1] - S[0], B, ff[2], slope);
#pragma unroll
    for (int i = 1; i < n - 1; ++i) {
      const double next = multScatt(S[i + 1] - S[i], B, ff[2], slope);
      VarBeta[i] = next + ms;
      ms = next;
    }
  }
  PG_FIT_PHASE();
  // ---- line fit
  double lpar[2];
  M<2, 2> lcov;
  double lchi2;
  {
    double w[N];
#pragma unroll
    for (int i = 0; i < n; ++i) {
      // element (1, 1) of R J V (R J)^T, J = (ry, -rx, 0; 0, 0, 1) / r
      const float* g = ge + 6 * i;
      const double gxx = g[0], gxy = g[1], gyy = g[2], gxz = g[3], gyz = g[4], gzz = g[5];
      const double tmp = 1. / rad[i];
      const double jx = radii[1][i] * tmp, jy = -radii[0][i] * tmp;
      const double a0 = R(1, 0) * jx, a1 = R(1, 0) * jy, a2 = R(1, 1);
      const double b0 = a0 * gxx + a1 * gxy + a2 * gxz;
      const double b1 = a0 * gxy + a1 * gyy + a2 * gyz;
      const double b2 = a0 * gxz + a1 * gyz + a2 * gzz;
      // J's zeros are left out; zero times an infinite or NaN term is NaN
      w[i] = 1. / ((b0 * jx + b1 * jy) * R(1, 0) + b2 * R(1, 1) + 0. * (b0 + b1 + b2));
    }
    double r_u[N];
#pragma unroll
    for (int i = 0; i < n; ++i) r_u[i] = w[i] * Z[i];
    PG_FIT_PHASE();
    M<N, N> I;
    invert(matrixCu<N>(w, S, VarBeta), I);
    double u[N];
#pragma unroll
    for (int i = 0; i < n; ++i) {
      double acc = I(i, 0) * r_u[0];
#pragma unroll
      for (int k = 1; k < n; ++k) acc += I(i, k) * r_u[k];
      u[i] = acc;
    }
    lpar[0] = (u[1] - u[0]) / (S[1] - S[0]);
    lpar[1] = u[0];
    double idiff = 1. / (S[1] - S[0]);
    lcov(0, 0) = (I(0, 0) - 2 * I(0, 1) + I(1, 1)) * sqr(idiff) + ms01;
    lcov(0, 1) = (I(0, 1) - I(0, 0)) * idiff;
    lcov(1, 0) = (I(0, 1) - I(0, 0)) * idiff;
    lcov(1, 1) = I(0, 0);
    lpar[1] += -lpar[0] * S[0];
    {  // (1, 0; -S0, 1)
      const double j = -S[0];
      const double t10 = j * lcov(0, 0) + lcov(1, 0), t11 = j * lcov(0, 1) + lcov(1, 1);
      lcov(0, 1) = lcov(0, 0) * j + lcov(0, 1);
      lcov(1, 0) = t10;
      lcov(1, 1) = t10 * j + t11;
    }
    double t = R(0, 0) - lpar[0] * R(0, 1);
    {  // (j0, 0; j1, j2)
      const double j2 = 1. / t;
      const double j0 = j2 * j2;
      const double j1 = lpar[1] * R(0, 1) * j0;
      lpar[1] = lpar[1] * j2;
      lpar[0] = (R(0, 1) + lpar[0] * R(0, 0)) * j2;
      const double t00 = j0 * lcov(0, 0), t01 = j0 * lcov(0, 1);
      const double t10 = j1 * lcov(0, 0) + j2 * lcov(1, 0), t11 = j1 * lcov(0, 1) + j2 * lcov(1, 1);
      lcov(0, 0) = t00 * j0;
      lcov(0, 1) = t00 * j1 + t01 * j2;
      lcov(1, 0) = t10 * j0;
      lcov(1, 1) = t10 * j1 + t11 * j2;
    }
    lchi2 = 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      lchi2 += w[i] * sqr(Z[i] - u[i]);
      if (i > 0 && i < n - 1)
        lchi2 += sqr(u[i - 1] / (S[i] - S[i - 1]) - u[i] * (S[i + 1] - S[i - 1]) / ((S[i + 1] - S[i]) * (S[i] - S[i - 1])) +
                     u[i + 1] / (S[i + 1] - S[i])) /
                 VarBeta[i];
    }
  }
  PG_FIT_PHASE();
  // ---- circle fit
  double cpar[3];
  M<3, 3> ccov;
  float cchi2;
  {
#pragma unroll
    for (int i = 0; i < n; ++i) VarBeta[i] *= 1. + sqr(slope);
#pragma unroll
    for (int i = 0; i < n; ++i) Z[i] = rad[i] - ff[2];
    double w[N];
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float* g = ge + 6 * i;
      // element (1, 1) of the rotated covariance
      const double gxx = g[0], gxy = g[1], gyy = g[2];
      const M<2, 2> RR = rotationMatrix(-radii[0][i] / radii[1][i]);
      const double t0 = RR(1, 0) * gxx + RR(1, 1) * gxy, t1 = RR(1, 0) * gxy + RR(1, 1) * gyy;
      w[i] = 1. / (t0 * RR(1, 0) + t1 * RR(1, 1));
    }
    double r_u[N + 1];
    r_u[n] = 0;
#pragma unroll
    for (int i = 0; i < n; ++i) r_u[i] = w[i] * Z[i];
    PG_FIT_PHASE();
    M<N + 1, N + 1> C;
    {
      M<N, N> cu = matrixCu<N>(w, s, VarBeta);
#pragma unroll
      for (int j = 0; j < n; ++j)
#pragma unroll
        for (int i = 0; i < n; ++i) C(i, j) = cu(i, j);
    }
    C(n, n) = 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      C(i, n) = 0;
      if (i > 0 && i < n - 1)
        C(i, n) += -(s[i + 1] - s[i - 1]) * (s[i + 1] - s[i - 1]) / (2. * VarBeta[i] * (s[i + 1] - s[i]) * (s[i] - s[i - 1]));
      if (i > 1) C(i, n) += (s[i] - s[i - 2]) / (2. * VarBeta[i - 1] * (s[i] - s[i - 1]));
      if (i < n - 2) C(i, n) += (s[i + 2] - s[i]) / (2. * VarBeta[i + 1] * (s[i + 1] - s[i]));
      C(n, i) = C(i, n);
      if (i > 0 && i < n - 1) C(n, n) += sqr(s[i + 1] - s[i - 1]) / (4. * VarBeta[i]);
    }
    PG_FIT_PHASE();
    M<N + 1, N + 1> I;
    invert(C, I);
    double u[N + 1];
#pragma unroll
    for (int i = 0; i < n + 1; ++i) {
      double acc = I(i, 0) * r_u[0];
#pragma unroll
      for (int k = 1; k < n + 1; ++k) acc += I(i, k) * r_u[k];
      u[i] = acc;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      radii[0][c] /= rad[c];
      radii[1][c] /= rad[c];
    }
    double dx = H(0, 0) + (-Z[0] + u[0]) * radii[0][0], dy = H(1, 0) + (-Z[0] + u[0]) * radii[1][0];
    double ex = H(0, 1) + (-Z[1] + u[1]) * radii[0][1], ey = H(1, 1) + (-Z[1] + u[1]) * radii[1][1];
    double emdx = ex - dx, emdy = ey - dy;
    cpar[0] = atan2(emdy, emdx);
    cpar[1] = -q * (ff[2] - sqrt(sqr(ff[2]) - 0.25 * (emdx * emdx + emdy * emdy)));
    cpar[2] = q * (1. / ff[2] + u[n]);
    double tmp1 = emdx * emdx + emdy * emdy;
    // The Jacobian (a0 a1 0; 0 0 0; 0 0 q) of (phi, dca, k) by the two offsets
    // and the curvature correction: the reference's elements of dca have the
    // integer factor q / 2, which is zero (BrokenLine.h, the circle fit's jacobian).
    const double a0 = (radii[1][0] * emdx - emdy * radii[0][0]) / tmp1;
    const double a1 = (radii[1][1] * emdx - emdy * radii[0][1]) / tmp1;
    const double t00 = a0 * I(0, 0) + a1 * I(1, 0), t01 = a0 * I(0, 1) + a1 * I(1, 1);
    const double t02 = a0 * I(0, n) + a1 * I(1, n);
    const double t20 = q * I(n, 0), t21 = q * I(n, 1), t22 = q * I(n, n);
    ccov(0, 0) = t00 * a0 + t01 * a1;
    ccov(0, 2) = t02 * q;
    ccov(2, 0) = t20 * a0 + t21 * a1;
    // the zeros' terms are left out here too
    ccov(2, 2) = t22 * q + 0. * (I(0, 0) + I(0, 1) + I(1, 1) + I(0, n) + I(1, n));
    PG_FIT_PHASE();
    translateKarimaki<true>(cpar, ccov, 0.5 * emdx, 0.5 * emdy);
    ccov(0, 0) += (1 + sqr(slope)) * ms01;
    PG_FIT_PHASE();
    translateKarimaki<false>(cpar, ccov, dx, dy);
    cchi2 = 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      cchi2 += w[i] * sqr(Z[i] - u[i]);
      if (i > 0 && i < n - 1)
        cchi2 += sqr(u[i - 1] / (s[i] - s[i - 1]) - u[i] * (s[i + 1] - s[i - 1]) / ((s[i + 1] - s[i]) * (s[i] - s[i - 1])) +
                     u[i + 1] / (s[i + 1] - s[i]) + (s[i + 1] - s[i - 1]) * u[n] / 2) /
                 VarBeta[i];
    }
  }
  float b = 1.f / float(B);
  out.state[0] = float(cpar[0]);
  out.state[1] = float(cpar[1]);
  out.state[2] = float(cpar[2]) * b;
  out.state[3] = float(lpar[0]);
  out.state[4] = float(lpar[1]);
  out.cov[0] = float(ccov(0, 0));
  out.cov[1] = float(ccov(0, 1));
  out.cov[2] = b * float(ccov(0, 2));
  out.cov[3] = out.cov[4] = 0;
  out.cov[5] = float(ccov(1, 1));
  out.cov[6] = b * float(ccov(1, 2));
  out.cov[7] = out.cov[8] = 0;
  out.cov[9] = b * b * float(ccov(2, 2));
  out.cov[10] = out.cov[11] = 0;
  out.cov[12] = float(lcov(0, 0));
  out.cov[13] = float(lcov(0, 1));
  out.cov[14] = float(lcov(1, 1));
  out.pt = float(B) / float(fabs(cpar[2]));
  out.eta = asinhf(float(lpar[0]));
  out.chi2 = float((double(cchi2) + lchi2) / (2 * N - 5));
}

#include "k_fit_mixed.cuh"

// zero the fit results of every stored tuple (the reference's TrackSoA is value-initialised)
// Tuples that no fit writes get zero fit results: those kept out of the
// multiplicity bins (duplicates), and every tuple of an event whose bins
// overflowed (the fits then cover an order-dependent subset).
__global__ void kFitZero(Workspace ws) {
  const uint32_t e = blockIdx.y;
  const uint32_t nt = ws.ev[e].nTuples;
  const bool all = (ws.ev[e].flags & (kFlagFitBinOverflow | kFlagTmOverflow)) != 0;
  const uint32_t* toff = ws.tupleOff + size_t(e) * (ws.cap.tuples + 1);
  const uint8_t* q = ws.quality + size_t(e) * ws.cap.tuples;
  const size_t tb = size_t(e) * ws.cap.tuples;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
    if (!all && toff[t + 1] - toff[t] >= 3 && q[t] != 1) continue;  // 1: duplicate
    for (int k = 0; k < 5; ++k) ws.state[tb * 5 + size_t(t) * 5 + k] = 0.f;
    for (int k = 0; k < 15; ++k) ws.cov[tb * 15 + size_t(t) * 15 + k] = 0.f;
    ws.pt[tb + t] = 0.f;
    ws.eta[tb + t] = 0.f;
    ws.chi2[tb + t] = 0.f;
  }
}

// the fits a chain can run (pg_config riemann_fit, mixed_fit)
enum FitMode { kFitBrokenLine, kFitRiemann, kFitBrokenLineMixed, kFitRiemannMixed };

// the tuples of multiplicity bin nh of every event of the batch, as one flat
// range over the events (uneven events share the whole grid): pre[e] is the
// exclusive prefix of the per-event bin sizes, built by each block
__device__ __forceinline__ uint32_t fitBinPrefix(const Workspace& ws, uint32_t nh, uint32_t nEvents, uint32_t* pre,
                                                 uint32_t* scanSh) {
  uint32_t carry = 0;
  for (uint32_t e0 = 0; e0 < nEvents; e0 += blockDim.x) {
    const uint32_t e = e0 + threadIdx.x;
    const uint32_t v = e < nEvents ? min(ws.tmOff[size_t(e) * 16 + nh], ws.cap.multiplicity) : 0u;
    uint32_t tot;
    const uint32_t x = blockExclusiveScan(v, scanSh, &tot);
    if (e < nEvents) pre[e] = carry + x;
    carry += tot;
  }
  if (threadIdx.x == 0) pre[nEvents] = carry;
  __syncthreads();
  return pre[nEvents];
}

// one thread per tuple of the multiplicity bin nh, flat items [g0, g0 +
// blockDim.x) of total; fits the first N hits
template <int N, int kMode>
__device__ __forceinline__ void fitTile(const DeviceES& es, const Workspace& ws, uint32_t nh, uint32_t nEvents,
                                        const uint32_t* pre, uint32_t g0, uint32_t total) {
  extern __shared__ double tile[];  // the threads' inputs (ChainTile)
  const double B = double(float(0.0114256972711507));
  // the block fits in step (PG_FIT_PHASE): threads past the end repeat the last item
  const bool live = g0 + threadIdx.x < total;
  const uint32_t g = min(g0 + threadIdx.x, total - 1);
  // the event of flat item g: the last e with pre[e] <= g (empty events skipped)
  uint32_t lo = 0, hi = nEvents;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (pre[mid] <= g)
      lo = mid;
    else
      hi = mid;
  }
  const uint32_t e = lo, k = g - pre[lo];
  const uint32_t start = ws.tmOff[size_t(e) * 16 + 8 + nh];
  const uint32_t* bins = ws.tmBins + size_t(e) * ws.cap.tuples;
  const uint32_t* toff = ws.tupleOff + size_t(e) * (ws.cap.tuples + 1);
  const uint32_t* th = ws.tupleHits + size_t(e) * ws.cap.tupleHits();
  const size_t hb = size_t(e) * ws.cap.hits;
  const size_t tb = size_t(e) * ws.cap.tuples;
  uint32_t tkid = bins[start + k];
  const uint32_t* hid = th + toff[tkid];
  // only this thread's, whichever N the block's other warps are at: the Riemann
  // fits have no barrier, and a warp ahead of the others fills its next tile
  // while they still read theirs
  double* H = tile + ChainTile::hits(threadIdx.x);
  float* ge = reinterpret_cast<float*>(tile) + ChainTile::ge(threadIdx.x, blockDim.x);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    uint32_t hit = hid[i];
    const PfFrame& f = es.det[ws.detInd[hb + hit]].frame;
    float cxx = ws.xerr[hb + hit], cxy = 0, cyy = ws.yerr[hb + hit];
    float* gl = ge + 6 * i;
    gl[0] = f.R11 * (f.R11 * cxx + f.R21 * cxy) + f.R21 * (f.R11 * cxy + f.R21 * cyy);
    gl[1] = f.R11 * (f.R12 * cxx + f.R22 * cxy) + f.R21 * (f.R12 * cxy + f.R22 * cyy);
    gl[2] = f.R12 * (f.R12 * cxx + f.R22 * cxy) + f.R22 * (f.R12 * cxy + f.R22 * cyy);
    gl[3] = f.R11 * (f.R13 * cxx + f.R23 * cxy) + f.R21 * (f.R13 * cxy + f.R23 * cyy);
    gl[4] = f.R12 * (f.R13 * cxx + f.R23 * cxy) + f.R22 * (f.R13 * cxy + f.R23 * cyy);
    gl[5] = f.R13 * (f.R13 * cxx + f.R23 * cxy) + f.R23 * (f.R13 * cxy + f.R23 * cyy);
    H[3 * i + 0] = ws.xg[hb + hit];
    H[3 * i + 1] = ws.yg[hb + hit];
    H[3 * i + 2] = ws.zg[hb + hit];
  }
  FitOut o;
  if constexpr (kMode == kFitRiemann) {
    rfFit<N, double>(H, ge, B, o);
  } else if constexpr (kMode == kFitRiemannMixed) {
    rfFit<N, float>(H, ge, B, o);
  } else if constexpr (kMode == kFitBrokenLineMixed) {
    // the mixed fit takes single-precision hits relative to the first one
    // and the first hit in double precision (k_fit_mixed.cuh)
    float Hf[3 * N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      Hf[3 * i + 0] = float(H[3 * i + 0] - H[0]);
      Hf[3 * i + 1] = float(H[3 * i + 1] - H[1]);
      Hf[3 * i + 2] = float(H[3 * i + 2]);
    }
    blFitMixed<N>(Hf, ge, H[0], H[1], float(B), B, o);
  } else {
    blFit<N>(H, ge, B, o);
  }
  if (!live) return;
#pragma unroll
  for (int j = 0; j < 5; ++j) ws.state[tb * 5 + size_t(tkid) * 5 + j] = o.state[j];
#pragma unroll
  for (int j = 0; j < 15; ++j) ws.cov[tb * 15 + size_t(tkid) * 15 + j] = o.cov[j];
  ws.pt[tb + tkid] = o.pt;
  ws.eta[tb + tkid] = o.eta;
  ws.chi2[tb + tkid] = o.chi2;
}

// The three multiplicity bins (3-hit tuples, 4-hit tuples, 5-hit tuples
// fitted on their first 4 hits) in one launch of as many blocks as the SMs
// hold, which take the batch's tuples in tiles of a block, the dearer bins
// first.  The number of tuples is not known on the host, and a grid sized for
// the usual event left the SMs to one block each on a heavy one (two PU180
// events: 222 blocks, 374 us), while a larger grid costs a light one its idle blocks.
template <int kMode>
__device__ __forceinline__ void fitBins(const DeviceES& es, const Workspace& ws, uint32_t nEvents) {
  __shared__ uint32_t pre[3][kFlatMaxEvents + 1], scanSh[33];
  uint32_t total[3], tiles[3];
#pragma unroll
  for (uint32_t b = 0; b < 3; ++b) {
    total[b] = fitBinPrefix(ws, 3 + b, nEvents, pre[b], scanSh);
    tiles[b] = (total[b] + blockDim.x - 1) / blockDim.x;
  }
  for (uint32_t t = blockIdx.x; t < tiles[0] + tiles[1] + tiles[2]; t += gridDim.x) {
    if (t < tiles[2] + tiles[1]) {
      const uint32_t b = t < tiles[2] ? 2u : 1u, k = b == 2 ? t : t - tiles[2];
      fitTile<4, kMode>(es, ws, 3 + b, nEvents, pre[b], k * blockDim.x, b == 2 ? total[2] : total[1]);
    } else {
      fitTile<3, kMode>(es, ws, 3, nEvents, pre[0], (t - tiles[2] - tiles[1]) * blockDim.x, total[0]);
    }
  }
}

__global__ void __launch_bounds__(kFitBlock, 2) kBLFit(DeviceES es, Workspace ws, uint32_t nEvents) {
  fitBins<kFitBrokenLine>(es, ws, nEvents);
}

// the same bins through the Riemann fit (useRiemannFit,
// CAHitNtupletGeneratorOnGPU.cc:116-120; RiemannFitOnGPU.cc:3-110)
__global__ void __launch_bounds__(kRiemannBlock, 4) kRiemannFit(DeviceES es, Workspace ws, uint32_t nEvents) {
  fitBins<kFitRiemann>(es, ws, nEvents);
}

// the mixed-precision variants of both fits inside the chain (pg_config
// mixed_fit): a precision choice beside the reference's FP64 fits, whose
// effect on the chain's quality codes and vertices is measured against them
__global__ void __launch_bounds__(kFitBlock, 2) kBLFitMixed(DeviceES es, Workspace ws, uint32_t nEvents) {
  fitBins<kFitBrokenLineMixed>(es, ws, nEvents);
}
__global__ void __launch_bounds__(kRiemannBlock, 4) kRiemannFitMixed(DeviceES es, Workspace ws, uint32_t nEvents) {
  fitBins<kFitRiemannMixed>(es, ws, nEvents);
}

template <int kBytes>
__device__ __forceinline__ void copyAsync(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src),
               "n"(kBytes)
               : "memory");
}

// A warp's 32 tuples of W elements each, contiguous in global memory, into
// shared memory at stride S (m: elements that exist).  A lane's elements
// repeat their place in a tuple every kPeriod steps, kPeriod * 32 / W tuples
// further, so only that many places are computed.  All copies of a thread
// are in flight at once.
template <int W, int S, typename T>
__device__ __forceinline__ void copyTuples(T* dst, const T* src, uint32_t m) {
  constexpr int kPeriod = W % 3 == 0 ? (W % 9 == 0 ? 9 : 3) : W;  // W = 9, 12, 18, 24
  static_assert(kPeriod * 32 % W == 0 && W % kPeriod == 0, "tuple width");
  const uint32_t lane = laneId();
#pragma unroll
  for (int j = 0; j < kPeriod; ++j) {
    const uint32_t k = uint32_t(j) * 32 + lane, at = k / W * S + k % W;
#pragma unroll
    for (int r = 0; r < W / kPeriod; ++r)
      if (k + r * (kPeriod * 32) < m) copyAsync<sizeof(T)>(dst + at + r * (kPeriod * 32 / W * S), src + k + r * (kPeriod * 32));
  }
}

// Standalone fits of n tuples given in global memory (fit workload and
// tests).  Each warp copies its 32 tuples into shared memory and its results
// out of it contiguously, where a lane's own accesses would touch a sector
// each (1M 4-hit tuples: 288 -> 246 us; with the shared quantities and the
// block size, 378 us before).  Every thread fits (PG_FIT_PHASE), those past the end the last tuple.
template <int N, typename Fit>
__device__ __forceinline__ void fitTuples(uint32_t n, const double* hits, const float* hge, float* state, float* cov,
                                          float* pt, float* eta, float* chi2, Fit&& fit) {
  using Tile = FitTile<N>;
  extern __shared__ double fitSm[];
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  double* hs = reinterpret_cast<double*>(reinterpret_cast<char*>(fitSm) + warp * 32 * Tile::kBytes);
  float* gs = reinterpret_cast<float*>(hs + 32 * Tile::kHitStride);
  float* ss = reinterpret_cast<float*>(hs);  // results, once the fits are done
  float* cs = ss + 32 * 5;
  for (uint32_t t0 = blockIdx.x * blockDim.x; t0 < n; t0 += gridDim.x * blockDim.x) {
    const uint32_t w0 = min(t0 + warp * 32, n - 1), m = min(32u, n - w0);
    copyTuples<Tile::kHits, Tile::kHitStride>(hs, hits + size_t(w0) * Tile::kHits, m * Tile::kHits);
    copyTuples<Tile::kGe, Tile::kGeStride>(gs, hge + size_t(w0) * Tile::kGe, m * Tile::kGe);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    const uint32_t i = min(lane, m - 1);
    FitOut o;
    fit(hs + i * Tile::kHitStride, gs + i * Tile::kGeStride, o);
    if (t0 + warp * 32 >= n) continue;  // a whole warp past the end (its tuple is another warp's)
    __syncwarp();
    if (lane < m) {
#pragma unroll
      for (int j = 0; j < 5; ++j) ss[lane * 5 + j] = o.state[j];
#pragma unroll
      for (int j = 0; j < 15; ++j) cs[lane * 15 + j] = o.cov[j];
      pt[w0 + lane] = o.pt;
      eta[w0 + lane] = o.eta;
      chi2[w0 + lane] = o.chi2;
    }
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < 5; ++k)
      if (k * 32 + lane < m * 5) state[size_t(w0) * 5 + k * 32 + lane] = ss[k * 32 + lane];
#pragma unroll
    for (uint32_t k = 0; k < 15; ++k)
      if (k * 32 + lane < m * 15) cov[size_t(w0) * 15 + k * 32 + lane] = cs[k * 32 + lane];
    __syncwarp();
  }
}

template <int N>
__global__ void __launch_bounds__(kFitBlock, 2) kBLFitDirect(uint32_t n, const double* hits, const float* hge, double B,
                                                             float* state, float* cov, float* pt, float* eta,
                                                             float* chi2) {
  fitTuples<N>(n, hits, hge, state, cov, pt, eta, chi2,
               [&](const double* H, const float* ge, FitOut& o) { blFit<N>(H, ge, B, o); });
}

template <int N>
__global__ void __launch_bounds__(kFitBlock, 2) kBLFitDirectMixed(uint32_t n, const double* hits, const float* hge,
                                                                  double B, float* state, float* cov, float* pt,
                                                                  float* eta, float* chi2) {
  const float Bf = float(B);
  fitTuples<N>(n, hits, hge, state, cov, pt, eta, chi2, [&](const double* h, const float* ge, FitOut& o) {
    const double x0 = h[0], y0 = h[1];
    float H[3 * N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      H[3 * i + 0] = float(h[3 * i + 0] - x0);
      H[3 * i + 1] = float(h[3 * i + 1] - y0);
      H[3 * i + 2] = float(h[3 * i + 2]);
    }
    blFitMixed<N>(H, ge, x0, y0, Bf, B, o);
  });
}

template <int N, typename S>
__global__ void __launch_bounds__(kRiemannBlock, 4) kRiemannFitDirect(uint32_t n, const double* hits, const float* hge,
                                                                      double B, float* state, float* cov, float* pt,
                                                                      float* eta, float* chi2) {
  fitTuples<N>(n, hits, hge, state, cov, pt, eta, chi2,
               [&](const double* H, const float* ge, FitOut& o) { rfFit<N, S>(H, ge, B, o); });
}

}  // namespace

// launches a fit kernel whose blocks hold their inputs in dynamic shared
// memory (up to 53 KB, above the default limit: opted in once per kernel and device)
template <typename... KArgs, typename... Args>
static cudaError_t launchFit(void (*k)(KArgs...), std::atomic<uint64_t>& configured, uint32_t most, uint32_t grid,
                             uint32_t block, uint32_t tupleBytes, cudaStream_t stream, Args... args) {
  int dev = 0;
  cudaGetDevice(&dev);
  const uint64_t bit = uint64_t(1) << (dev & 63);
  if (!(configured.load() & bit)) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most * tupleBytes));
    if (e != cudaSuccess) return e;
    configured.fetch_or(bit);
  }
  k<<<grid, block, size_t(block) * tupleBytes, stream>>>(args...);
  return cudaGetLastError();
}

cudaError_t runFits(const DeviceES& es, Workspace& ws, uint32_t nEvents, cudaStream_t stream, bool riemann) {
  const uint32_t gx = nEvents >= 32 ? 8 : (nEvents >= 8 ? 32 : 148);
  dim3 g(gx, nEvents);
  PG_PROBED("kFitZero", stream, kFitZero<<<dim3(tunedGrid(ws, kTuneFitZero, g.x), nEvents), 256, 0, stream>>>(ws));
  // one wave of blocks of 512 threads per SM; a few events' tuples (a PU50 event
  // has 10.6k) go in tiles of 64, over all SMs.  The launch table does not scale
  // this grid: it follows from the SMs alone.
  // Otherwise tiles of 128: the hits' gathers make the block wait, and two more
  // blocks per SM fill that better than one wide block in step (64 PU50 events:
  // 174 us with 256, 167 us with 128).
  const uint32_t most = riemann ? kRiemannBlock : kFitBlock;
  const uint32_t fb = nEvents <= 4 ? 64u : 128u, fg = 148 * (512 / fb);
  static std::atomic<uint64_t> configured[4];
  cudaError_t le = cudaSuccess;
  auto launch = [&](int which, auto kernel) {
    le = launchFit(kernel, configured[which], most, fg, fb, ChainTile::kBytes, stream, es, ws, nEvents);
  };
  if (riemann && ws.ca.mixedFit)
    PG_PROBED("kRiemannFitMixed", stream, launch(0, kRiemannFitMixed));
  else if (riemann)
    PG_PROBED("kRiemannFit", stream, launch(1, kRiemannFit));
  else if (ws.ca.mixedFit)
    PG_PROBED("kBLFitMixed", stream, launch(2, kBLFitMixed));
  else
    PG_PROBED("kBLFit", stream, launch(3, kBLFit));
  return le;
}

// block size of a standalone fit of n tuples: the largest (a block's warps
// share their instruction fetches) that still gives each of the 148 SMs a block
// (6007 3-hit tuples: 14.3 us in 47 blocks of 128, 13.3 us in 188 of 32)
static uint32_t directBlock(uint32_t n, uint32_t most) {
  uint32_t b = most;
  while (b > 32 && (n + b - 1) / b < 148) b /= 2;
  return b;
}

template <int N, typename... KArgs>
static cudaError_t launchDirect(void (*k)(KArgs...), const char* name, std::atomic<uint64_t>& configured, uint32_t most,
                                uint32_t n, const double* hits, const float* ge, double B, float* state, float* cov,
                                float* pt, float* eta, float* chi2, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const uint32_t fb = directBlock(n, most);
  cudaError_t e = cudaSuccess;
  PG_PROBED(name, stream,
            e = launchFit(k, configured, most, min((n - 1) / fb + 1, 148u * 16u), fb, FitTile<N>::kBytes, stream, n,
                          hits, ge, B, state, cov, pt, eta, chi2));
  return e;
}

cudaError_t fitDirect(int N, uint32_t n, const double* hits, const float* ge, double B, float* state, float* cov,
                      float* pt, float* eta, float* chi2, cudaStream_t stream) {
  static std::atomic<uint64_t> configured[2];
  return N == 3 ? launchDirect<3>(kBLFitDirect<3>, "kBLFitDirect", configured[0], kFitBlock, n, hits, ge, B, state, cov,
                                  pt, eta, chi2, stream)
                : launchDirect<4>(kBLFitDirect<4>, "kBLFitDirect", configured[1], kFitBlock, n, hits, ge, B, state, cov,
                                  pt, eta, chi2, stream);
}

cudaError_t fitDirectMixed(int N, uint32_t n, const double* hits, const float* ge, double B, float* state, float* cov,
                           float* pt, float* eta, float* chi2, cudaStream_t stream) {
  static std::atomic<uint64_t> configured[2];
  return N == 3 ? launchDirect<3>(kBLFitDirectMixed<3>, "kBLFitDirectMixed", configured[0], kFitBlock, n, hits, ge, B,
                                  state, cov, pt, eta, chi2, stream)
                : launchDirect<4>(kBLFitDirectMixed<4>, "kBLFitDirectMixed", configured[1], kFitBlock, n, hits, ge, B,
                                  state, cov, pt, eta, chi2, stream);
}

cudaError_t fitDirectRiemann(int N, uint32_t n, const double* hits, const float* ge, double B, float* state,
                             float* cov, float* pt, float* eta, float* chi2, bool mixed, cudaStream_t stream) {
  static std::atomic<uint64_t> configured[4];
  auto launch = [&](auto tile, auto kernel, const char* name, int which) {
    return launchDirect<decltype(tile)::kHits / 3>(kernel, name, configured[which], kRiemannBlock, n, hits, ge, B, state,
                                                   cov, pt, eta, chi2, stream);
  };
  if (N == 3)
    return mixed ? launch(FitTile<3>{}, kRiemannFitDirect<3, float>, "kRiemannFitDirectMixed", 0)
                 : launch(FitTile<3>{}, kRiemannFitDirect<3, double>, "kRiemannFitDirect", 1);
  return mixed ? launch(FitTile<4>{}, kRiemannFitDirect<4, float>, "kRiemannFitDirectMixed", 2)
               : launch(FitTile<4>{}, kRiemannFitDirect<4, double>, "kRiemannFitDirect", 3);
}

}  // namespace pixgpu
