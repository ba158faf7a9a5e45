// Test infrastructure: the device helix-fit code of the B200 library
// (pixeltrack-standalone_b200/csrc/fit_linalg.cuh, k_fit_broken_line.cuh,
// k_fit_mixed.cuh, k_fit_riemann.cuh)
// compiled by the host compiler, so that tests without a GPU can compare the
// kernel's arithmetic with the oracle operation by operation.  The device
// and host builds differ only in their transcendental functions.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>

#define __device__
#define __forceinline__ inline
using std::acos;
using std::atan;
using std::atan2;
using std::cos;
using std::fabs;
using std::fmin;
using std::hypot;
using std::log;
using std::sin;
using std::sqrt;

namespace {
#include "fit_linalg.cuh"
#include "k_fit_riemann.cuh"
#include "k_fit_broken_line.cuh"
#include "k_fit_mixed.cuh"

template <int N>
struct BrokenLine {
  static void fit(const double* H, const float* ge, double B, FitOut& o) { blFit<N>(H, ge, B, o); }
};
template <int N>
struct BrokenLineMixed {  // with the hits relative to the first one, as the kernels pass them
  static void fit(const double* h, const float* ge, double B, FitOut& o) {
    float H[3 * N];
    for (int i = 0; i < N; ++i) {
      H[3 * i + 0] = float(h[3 * i + 0] - h[0]);
      H[3 * i + 1] = float(h[3 * i + 1] - h[1]);
      H[3 * i + 2] = float(h[3 * i + 2]);
    }
    blFitMixed<N>(H, ge, h[0], h[1], float(B), B, o);
  }
};
template <int N, typename S>
struct Riemann {
  static void fit(const double* H, const float* ge, double B, FitOut& o) { rfFit<N, S>(H, ge, B, o); }
};

template <int N, typename Fit>
void fitAll(uint32_t n, const double* hits, const float* ge, double B, float* state, float* cov, float* pt, float* eta,
            float* chi2) {
  for (uint32_t t = 0; t < n; ++t) {
    FitOut o;
    Fit::fit(hits + size_t(t) * 3 * N, ge + size_t(t) * 6 * N, B, o);
    std::memcpy(state + size_t(t) * 5, o.state, sizeof o.state);
    std::memcpy(cov + size_t(t) * 15, o.cov, sizeof o.cov);
    pt[t] = o.pt;
    eta[t] = o.eta;
    chi2[t] = o.chi2;
  }
}
}  // namespace

template <template <int> class Fit>
static int fitN(int N, uint32_t n, const double* hits, const float* ge, double B, float* state, float* cov, float* pt,
                float* eta, float* chi2) {
  if (N == 3)
    fitAll<3, Fit<3>>(n, hits, ge, B, state, cov, pt, eta, chi2);
  else if (N == 4)
    fitAll<4, Fit<4>>(n, hits, ge, B, state, cov, pt, eta, chi2);
  else
    return -1;
  return 0;
}
template <int N>
using RiemannF64 = Riemann<N, double>;
template <int N>
using RiemannMixed = Riemann<N, float>;

extern "C" int hf_fit_riemann(int N, int mixed, uint32_t n, const double* hits, const float* ge, double B, float* state,
                              float* cov, float* pt, float* eta, float* chi2) {
  return mixed ? fitN<RiemannMixed>(N, n, hits, ge, B, state, cov, pt, eta, chi2)
               : fitN<RiemannF64>(N, n, hits, ge, B, state, cov, pt, eta, chi2);
}

extern "C" int hf_fit_broken_line(int N, int mixed, uint32_t n, const double* hits, const float* ge, double B,
                                  float* state, float* cov, float* pt, float* eta, float* chi2) {
  return mixed ? fitN<BrokenLineMixed>(N, n, hits, ge, B, state, cov, pt, eta, chi2)
               : fitN<BrokenLine>(N, n, hits, ge, B, state, cov, pt, eta, chi2);
}

// Byte range [out[0], out[1]) of the hits and [out[2], out[3]) of the covariances
// of an N-hit tuple that thread `thread` of `threads` holds in the chain fits'
// shared memory; returns the bytes of the block's shared memory.
extern "C" uint32_t hf_chain_tile(int N, uint32_t thread, uint32_t threads, uint32_t* out) {
  out[0] = ChainTile::hits(thread) * 8;
  out[1] = out[0] + 3 * N * 8;
  out[2] = ChainTile::ge(thread, threads) * 4;
  out[3] = out[2] + 6 * N * 4;
  return threads * ChainTile::kBytes;
}
