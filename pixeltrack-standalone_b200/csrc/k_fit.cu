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
#include "k_fit_broken_line.cuh"
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
  // One wave of blocks, 512 threads on each of the 148 SMs of a B200.  Tiles of
  // 128: the hits' gathers make the block wait, and two more blocks per SM fill
  // that better than one wide block in step (64 PU50 events: 174 us with 256, 167
  // us with 128; the grid before, sized for such events, took 159 us there but
  // 1035 instead of 480 us on 12 uneven ones).  A few events' tuples (a PU50 event
  // has 10.6k) go in tiles of 64, over all SMs: one event 0.2 % faster, 2 to 8
  // events the same with either, 16 events and three batches in flight 1.6 %
  // slower.  The launch table does not scale this grid: half or a quarter of it
  // is 1.5 and 4 % slower at 8 events alone, 2 and 6 % at 64 (1 % faster there
  // with three batches in flight), twice of it changes nothing.
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
