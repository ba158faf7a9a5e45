// Broken-line helix fit in FP64, N hits by one thread (reference:
// plugin-PixelTriplets/BrokenLine.h:46-504).  Included inside the anonymous
// namespace of k_fit.cu after fit_linalg.cuh; like it, it can be compiled for
// the host.
#pragma once

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
      // (the zero times an infinite or NaN element is NaN)
      const double t00 = j0 * lcov(0, 0), t01 = j0 * lcov(0, 1) + 0. * lcov(1, 1);
      const double t10 = j1 * lcov(0, 0) + j2 * lcov(1, 0), t11 = j1 * lcov(0, 1) + j2 * lcov(1, 1);
      lcov(0, 0) = t00 * j0 + 0. * t01;
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
    // integer factor q / 2, which is zero (BrokenLine.h, the circle fit's
    // jacobian), over a square root: they are NaN, and so is the covariance,
    // where the chord is no shorter than the circle's diameter.
    const double nil = sqr(2 * ff[2]) - tmp1 > 0. ? 0. : NAN;
    const double a0 = (radii[1][0] * emdx - emdy * radii[0][0]) / tmp1;
    const double a1 = (radii[1][1] * emdx - emdy * radii[0][1]) / tmp1;
    const double t00 = a0 * I(0, 0) + a1 * I(1, 0), t01 = a0 * I(0, 1) + a1 * I(1, 1);
    const double t02 = a0 * I(0, n) + a1 * I(1, n);
    const double t20 = q * I(n, 0), t21 = q * I(n, 1), t22 = q * I(n, n);
    ccov(0, 0) = t00 * a0 + t01 * a1 + nil;
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
