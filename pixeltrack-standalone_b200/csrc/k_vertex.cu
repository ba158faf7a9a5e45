// Pixel vertexing on B200: a cluster of CTAs per event runs loadTracks and
// the neighbour searches of clusterTracksByDensity, its first CTA the rest:
// fitVertices(50), splitVertices(9), fitVertices(5000) and sortByPt2, with the
// PixelVertexProducerCUDA configuration (minT=2, eps=0.07, errmax=0.01,
// chi2max=9, ptMin=0.5).
// Reference: plugin-PixelVertexFinding/gpuVertexFinderImpl.h:10-43,
// gpuClusterTracksByDensity.h:20-207, gpuFitVertices.h:15-98,
// gpuSplitVertices.h:15-125, gpuSortByPt2.h:15-55,
// PixelVertexProducerCUDA.cc:16-26.
//
// All float sums run sequentially per vertex in ascending track order (the
// serial order), histogram bins are scanned in the serial storage order
// (descending track index inside a bin) and new split vertices are numbered
// by a prefix over the parent vertex index.
#include <atomic>

#include <cooperative_groups.h>

#include "device_utils.cuh"
#include "pixgpu_internal.cuh"

namespace pixgpu {

namespace {

// the per-event scratch stride is at least the reference's 2 x 458752 words
// (pixgpu_internal.cuh referenceCaps; larger capacities only widen it)
static_assert(kVtxScratchAWords <= 2 * size_t(PF_MAX_DOUBLETS_PARAM) &&
                  kVtxScratchBWords <= 2 * size_t(PF_MAX_DOUBLETS_PARAM),
              "vertex scratch exceeds the per-event scratchA/scratchB stride");
constexpr int kVtxThreads = 1024;
// events with at most this many vertex tracks keep every per-track array in
// shared memory (40 bytes per track: 220 KB, about the vertex tracks of a
// PU 250 event); larger ones use the global scratch
constexpr uint32_t kSmemTracks = 5500;
constexpr size_t kTrackBytes = 9 * 4 + 2 + 2;
constexpr size_t kVtxSmemBytes = kSmemTracks * kTrackBytes;
// with the kernel's static shared memory (about 9.4 KB) within the 227 KB of a block
static_assert(kVtxSmemBytes + 10 * 1024 <= 227 * 1024, "vertex shared memory");
constexpr uint32_t kVtxCtas = 8;  // CTAs per event in a small batch

struct VtxScratch {
  float *zt, *ezt2, *ptt2, *zz;
  uint32_t* itrk;    // tuple index of each vertex track
  uint8_t *izt, *newV;
  int32_t *iv, *nn, *root;
  uint32_t* list;    // tracks grouped by vertex
  uint16_t* hbins;   // z-histogram content
};

__device__ __forceinline__ VtxScratch carve(char* p, uint32_t cap) {
  VtxScratch s;
  s.zt = reinterpret_cast<float*>(p);
  s.ezt2 = s.zt + cap;
  s.ptt2 = s.ezt2 + cap;
  s.zz = s.ptt2 + cap;
  s.iv = reinterpret_cast<int32_t*>(s.zz + cap);
  s.nn = s.iv + cap;
  s.root = s.nn + cap;
  s.list = reinterpret_cast<uint32_t*>(s.root + cap);
  s.itrk = s.list + cap;
  s.hbins = reinterpret_cast<uint16_t*>(s.itrk + cap);
  s.izt = reinterpret_cast<uint8_t*>(s.hbins + cap);
  s.newV = s.izt + cap;
  return s;
}

__device__ __forceinline__ VtxScratch scratchOf(const Workspace& ws, uint32_t e) {
  // carve per-event scratch out of scratchA/scratchB (cap.scratch words each;
  // kVtxScratchAWords and kVtxScratchBWords of them are used)
  uint32_t* a = ws.scratchA + size_t(e) * ws.cap.scratch;
  uint32_t* b = ws.scratchB + size_t(e) * ws.cap.scratch;
  VtxScratch s;
  s.zt = reinterpret_cast<float*>(a);
  s.ezt2 = reinterpret_cast<float*>(a + kMaxVtxTracks);
  s.ptt2 = reinterpret_cast<float*>(a + 2 * kMaxVtxTracks);
  s.zz = reinterpret_cast<float*>(a + 3 * kMaxVtxTracks);
  s.iv = reinterpret_cast<int32_t*>(a + 4 * kMaxVtxTracks);
  s.nn = reinterpret_cast<int32_t*>(a + 5 * kMaxVtxTracks);
  s.root = reinterpret_cast<int32_t*>(a + 6 * kMaxVtxTracks);
  s.list = a + 7 * kMaxVtxTracks;
  s.itrk = a + 8 * kMaxVtxTracks;
  static_assert(9 * size_t(kMaxVtxTracks) == kVtxScratchAWords, "scratch A layout");
  s.hbins = reinterpret_cast<uint16_t*>(b);
  s.izt = reinterpret_cast<uint8_t*>(b + kMaxVtxTracks / 2);
  s.newV = reinterpret_cast<uint8_t*>(b + kMaxVtxTracks / 2) + kMaxVtxTracks;
  static_assert(size_t(kMaxVtxTracks) / 2 + 2 * size_t(kMaxVtxTracks) / 4 == kVtxScratchBWords, "scratch B layout");
  return s;
}

// Groups n items by key in item order (a stable counting sort): off[0..nb]
// receives the groups' starts, place(i, pos) every item with a key < nb.
// Each of W warps walks a contiguous part of the items twice, first counting
// its keys in its own row of tab (nb entries), then, after the rows' prefix
// sums, placing them; lanes of the same key are ranked among themselves (a
// ballot per key bit: a match instruction costs more than the ten ballots of
// the largest key).  So a warp walks n / W items, where letting each warp own a range
// of keys made every warp walk all of them (1087 tracks: 21k of the kernel's
// 113k cycles for the z histogram and 12k for each grouping by vertex).
// Called by the whole block; ends with a barrier.
template <typename Key, typename Place>
__device__ __forceinline__ void orderedFill(uint32_t n, uint32_t nb, uint16_t* tab, uint32_t W, uint32_t* off,
                                            uint32_t* scanSh, Key&& key, Place&& place) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t k = threadIdx.x; k < nb * W; k += blockDim.x) tab[k] = 0;
  __syncthreads();
  const uint32_t part = (n + W * 32 - 1) / (W * 32) * 32;
  const uint32_t i0 = warp < W ? min(n, warp * part) : n, i1 = min(n, i0 + part);
  uint16_t* row = tab + warp * nb;
  const uint32_t bits = 32 - __clz(nb | 1);
  auto sameKey = [&](uint32_t b) {
    uint32_t m = __ballot_sync(0xffffffffu, b < nb);
    for (uint32_t k = 0; k < bits; ++k) {
      const bool one = (b >> k) & 1u;
      const uint32_t with = __ballot_sync(0xffffffffu, one);
      m &= one ? with : ~with;
    }
    return m;  // meaningless for lanes without a key below nb
  };
  for (uint32_t ib = i0; ib < i1; ib += 32) {
    const uint32_t i = ib + lane, b = i < i1 ? key(i) : 0xffffffffu;
    const uint32_t peers = sameKey(b);
    if (b < nb && (peers & lanemaskLt()) == 0) row[b] = uint16_t(row[b] + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 <= nb; b0 += blockDim.x) {
    const uint32_t b = b0 + threadIdx.x;
    uint32_t run = 0;
    if (b < nb) {
#pragma unroll 8
      for (uint32_t w = 0; w < W; ++w) {
        const uint32_t t = tab[w * nb + b];
        tab[w * nb + b] = uint16_t(run);
        run += t;
      }
    }
    uint32_t tot;
    const uint32_t pre = blockExclusiveScan(run, scanSh, &tot);
    if (b <= nb) off[b] = carry + pre;
    carry += tot;
  }
  __syncthreads();
  for (uint32_t ib = i0; ib < i1; ib += 32) {
    const uint32_t i = ib + lane, b = i < i1 ? key(i) : 0xffffffffu;
    const uint32_t peers = sameKey(b);
    if (b < nb) {
      const uint32_t at = row[b];
      place(i, off[b] + at + __popc(peers & lanemaskLt()));
      __syncwarp(peers);
      if ((peers & lanemaskLt()) == 0) row[b] = uint16_t(at + __popc(peers));
    }
    __syncwarp();
  }
  __syncthreads();
}

// group tracks by vertex id (ascending track order inside each vertex);
// tab: tabBytes of shared memory
__device__ void groupByVertex(const VtxScratch& s, uint32_t nt, uint32_t nv, uint32_t* vOff, uint32_t* scanSh,
                              uint16_t* tab, uint32_t tabBytes) {
  const uint32_t W = min(blockDim.x >> 5, tabBytes / 2 / max(nv, 1u));
  orderedFill(nt, nv, tab, W, vOff, scanSh, [&](uint32_t i) { return uint32_t(s.iv[i]); },
              [&](uint32_t i, uint32_t pos) { s.list[pos] = i; });
}

// Float sums that must follow the serial order (ascending track order inside
// a vertex) are formed by a warp: the lanes evaluate 32 consecutive terms at
// once, and K sums are formed together, lane k < K adding the 32 terms of the
// k-th in order.  Terms of tracks that the serial loop skips are +0.0, which
// leaves a sum unchanged (a sum that starts at +0.0 never becomes -0.0 under
// round-to-nearest).  The terms go through shared memory, so that the K
// chains of additions run side by side in K lanes: 40 instructions for all of
// them, where shuffling each term to every lane took 64 for each sum.  Bound
// by instruction issue on the event's one CTA.
constexpr uint32_t kSumStride = 36;  // floats between the sums' terms: 16-byte rows in different banks
constexpr uint32_t kSumWords = 4 * kSumStride;  // a warp's buffer
template <int K>
__device__ __forceinline__ void orderedSums(float* buf, const float (&term)[K], float& sum) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < K; ++k) buf[k * kSumStride + lane] = term[k];
  __syncwarp();
  if (lane < K) {
    const float4* row = reinterpret_cast<const float4*>(buf + lane * kSumStride);
    float4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = row[j];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      sum += v[j].x;
      sum += v[j].y;
      sum += v[j].z;
      sum += v[j].w;
    }
  }
  __syncwarp();
}

// fitVertices: weighted z, chi2 outlier rejection (iv = 9999), ndof and weight;
// one warp per vertex
__device__ void fitVertices(const VtxScratch& s, uint32_t nt, uint32_t nv, float chi2Max, float* zv, float* wv,
                            float* chi2, int32_t* ndof, uint32_t* vOff, uint32_t* scanSh, float* sumBuf, uint16_t* tab,
                            uint32_t tabBytes) {
  groupByVertex(s, nt, nv, vOff, scanSh, tab, tabBytes);
  const uint32_t lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (uint32_t v = threadIdx.x >> 5; v < nv; v += nw) {
    const uint32_t b = vOff[v], n = vOff[v + 1] - b;
    float zw = 0;  // lane 0: the sum of z, lane 1: of the weights
    for (uint32_t k0 = 0; k0 < n; k0 += 32) {
      const uint32_t k = k0 + lane;
      float t[2] = {0.f, 0.f};
      if (k < n) {
        const uint32_t i = s.list[b + k];
        const float wi = 1.f / s.ezt2[i];
        t[0] = s.zt[i] * wi;
        t[1] = wi;
      }
      orderedSums(sumBuf, t, zw);
    }
    float z = __shfl_sync(0xffffffffu, zw, 0), w = __shfl_sync(0xffffffffu, zw, 1);
    z /= w;
    int32_t nd = -1;
    float c2s = 0;
    for (uint32_t k0 = 0; k0 < n; k0 += 32) {
      const uint32_t k = k0 + lane;
      float t[1] = {0.f};
      bool acc = false;
      if (k < n) {
        const uint32_t i = s.list[b + k];
        float c2 = z - s.zt[i];
        c2 *= c2 / s.ezt2[i];
        if (c2 > chi2Max) {
          s.iv[i] = 9999;
        } else {
          acc = true;
          t[0] = c2;
        }
      }
      nd += __popc(__ballot_sync(0xffffffffu, acc));
      orderedSums(sumBuf, t, c2s);
    }
    c2s = __shfl_sync(0xffffffffu, c2s, 0);
    if (nd > 0) w *= float(nd) / c2s;
    if (lane == 0) {
      zv[v] = z;
      wv[v] = w;
      chi2[v] = c2s;
      ndof[v] = nd;
    }
  }
  __syncthreads();
}

// lanes that share a track in the neighbour searches, and reductions over
// them (called by whole warps)
constexpr uint32_t kNbrLanes = 8;
template <typename T, typename Op>
__device__ __forceinline__ T groupReduce(T v, Op&& op) {
#pragma unroll
  for (uint32_t o = 1; o < kNbrLanes; o <<= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ uint32_t groupSum(uint32_t v) {
  return groupReduce(v, [](uint32_t a, uint32_t b) { return a + b; });
}
__device__ __forceinline__ int32_t groupMax(int32_t v) {
  return groupReduce(v, [](int32_t a, int32_t b) { return max(a, b); });
}
__device__ __forceinline__ int32_t groupMin(int32_t v) {
  return groupReduce(v, [](int32_t a, int32_t b) { return min(a, b); });
}
__device__ __forceinline__ unsigned long long groupMin(unsigned long long v) {
  return groupReduce(v, [](unsigned long long a, unsigned long long b) { return b < a ? b : a; });
}

// order-preserving map of a float to unsigned (negative values reversed)
__device__ __forceinline__ uint32_t orderedBits(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The bins a track's candidates lie in: its own and the two next to it.
__device__ __forceinline__ void candidateRange(const VtxScratch& s, const uint32_t* hoff, uint32_t i, uint32_t& pb,
                                               uint32_t& pe) {
  const int b0 = max(0, int(s.izt[i]) - 1), b1 = min(255, int(s.izt[i]) + 1);
  pb = hoff[b0];
  pe = hoff[b1 + 1];
}

// DBSCAN (gpuClusterTracksDBSCAN.h:16-227), first step, divided among the
// CTAs as the neighbour counts are: every core track is linked (iv) to its
// core neighbour of lowest z below its own, first in bin order among equal z;
// a track whose candidates include a NaN is done by its first lane literally.
__device__ void linkCores(const VtxScratch& s, uint32_t nt, const uint32_t* hoff, float eps, int32_t minT,
                          uint32_t gFirst, uint32_t gStride, int32_t* iv) {
  const uint32_t sub = threadIdx.x / kNbrLanes % (32 / kNbrLanes), gl = threadIdx.x % kNbrLanes;
  const float* zP = s.zz;
  const int32_t* nP = s.root;
  for (uint32_t p0 = gFirst; p0 < nt; p0 += gStride) {
    const uint32_t pi = p0 + sub;
    const bool core = pi < nt && nP[pi] >= minT;
    uint32_t pb = 0, pe = 0, i = 0, bestPos = 0xffffffffu;
    float zi = 0.f;
    if (core) {
      i = s.hbins[pi];
      candidateRange(s, hoff, i, pb, pe);
      zi = zP[pi];
    }
    float bestZ = zi;
    int32_t nan = isnan(zi) ? 1 : 0;
    for (uint32_t p = pb + gl; p < pe; p += kNbrLanes) {
      const float zj = zP[p];
      if (isnan(zj)) nan = 1;
      if (zj < bestZ && nP[p] >= minT && !(fabsf(zi - zj) > eps)) {
        bestZ = zj;
        bestPos = p;
      }
    }
    nan = groupMax(nan);
    const unsigned long long best = groupMin(
        bestPos == 0xffffffffu ? ~0ull : (uint64_t(orderedBits(bestZ)) << 32) | bestPos);
    if (nan) {
      if (gl == 0) {  // the serial loop as written
        float mz = zi;
        for (uint32_t p = pb; p < pe; ++p) {
          if (zP[p] >= mz || nP[p] < minT || fabsf(zi - zP[p]) > eps) continue;
          mz = zP[p];
          iv[i] = int32_t(s.hbins[p]);
        }
      }
    } else if (gl == 0 && best != ~0ull) {
      iv[i] = int32_t(s.hbins[uint32_t(best & 0xffffffffu)]);
    }
  }
}

// The rest of DBSCAN and the iterative clustering
// (gpuClusterTracksIterative.h:16-201) after the neighbour counts:
// iv[i] left pointing at track i's root (the numbering that follows is the
// one of the density clusterer).  One block; kNbrLanes lanes per track for the
// neighbour loops, whose serial order is reproduced by (key, position)
// reductions; a track whose candidates include a NaN is done by its first lane
// literally.
__device__ void clusterCoresAndEdges(const VtxScratch& s, uint32_t nt, const uint32_t* hoff, int algo, float eps,
                                     float chi2max, int32_t minT, int* sFlag) {
  const uint32_t sub = threadIdx.x / kNbrLanes % (32 / kNbrLanes), gl = threadIdx.x % kNbrLanes;
  const uint32_t gFirst = threadIdx.x / 32 * (32 / kNbrLanes), gStride = blockDim.x / kNbrLanes;
  auto range = [&](uint32_t i, uint32_t& pb, uint32_t& pe) { candidateRange(s, hoff, i, pb, pe); };
  auto percolate = [&]() {
    for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
      int32_t m = s.iv[i];
      while (m != s.iv[m]) m = s.iv[m];
      s.root[i] = m;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) s.iv[i] = s.root[i];
    __syncthreads();
  };
  // z, its error and the neighbour count in histogram order; the counts' place
  // (root) is free for the percolation once the cores are linked
  const float* zP = s.zz;
  const float* eP = reinterpret_cast<const float*>(s.list);
  const int32_t* nP = s.root;
  if (algo == 1) {
    percolate();
  } else {
    // connected components of the compatible core tracks: every label
    // becomes the lowest track index of its component, the fixed point of the
    // reference's alternating min-propagation and percolation
    for (uint32_t it = 0; it <= nt + 1; ++it) {
      if (threadIdx.x == 0) *sFlag = 0;
      __syncthreads();
      for (uint32_t p0 = gFirst; p0 < nt; p0 += gStride) {
        const uint32_t pi = p0 + sub, i = pi < nt ? s.hbins[pi] : 0u;
        const bool core = pi < nt && nP[pi] >= minT;
        uint32_t pb = 0, pe = 0;
        float zi = 0.f, ei = 0.f;
        int32_t m = 0;
        if (core) {
          range(i, pb, pe);
          zi = zP[pi];
          ei = eP[pi];
          m = s.iv[i];
        }
        for (uint32_t p = pb + gl; p < pe; p += kNbrLanes) {
          if (p == pi || nP[p] < minT) continue;
          const float dist = fabsf(zi - zP[p]);
          if (dist > eps || dist * dist > chi2max * (ei + eP[p])) continue;
          m = min(m, s.iv[s.hbins[p]]);
        }
        m = groupMin(m);
        if (gl == 0 && core && m < s.iv[i]) {
          atomicMin(&s.iv[i], m);
          *sFlag = 1;
        }
      }
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
        const int32_t l = s.iv[i], ll = s.iv[l];
        if (ll < l) {
          atomicMin(&s.iv[i], ll);
          *sFlag = 1;
        }
      }
      __syncthreads();
      const int more = *sFlag;
      __syncthreads();
      if (!more) break;
    }
  }
  // edge rule: a non-core track joins its closest chi2-compatible core
  // neighbour (last in bin order among equal distances)
  for (uint32_t p0 = gFirst; p0 < nt; p0 += gStride) {
    const uint32_t pi = p0 + sub, i = pi < nt ? s.hbins[pi] : 0u;
    const bool edge = pi < nt && s.nn[i] < minT;
    uint32_t pb = 0, pe = 0;
    float zi = 0.f, ei = 0.f;
    if (edge) {
      range(i, pb, pe);
      zi = zP[pi];
      ei = eP[pi];
    }
    unsigned long long best = ~0ull;
    int32_t nan = 0;
    for (uint32_t p = pb + gl; p < pe; p += kNbrLanes) {
      if (s.nn[s.hbins[p]] < minT) continue;
      const float dist = fabsf(zi - zP[p]), reach = chi2max * (ei + eP[p]);
      if (isnan(dist) || isnan(reach)) nan = 1;
      if (dist > eps || dist * dist > reach) continue;
      const unsigned long long key = (uint64_t(__float_as_uint(dist)) << 32) | uint64_t(0xffffffffu - p);
      best = key < best ? key : best;
    }
    nan = groupMax(nan);
    best = groupMin(best);
    if (!edge || gl != 0) continue;  // (no reduction follows in this step)
    if (nan) {
      s.root[i] = s.iv[i];
      float mdist = eps;
      for (uint32_t p = pb; p < pe; ++p) {
        const uint32_t j = s.hbins[p];
        if (s.nn[j] < minT) continue;
        const float dist = fabsf(zi - s.zt[j]);
        if (dist > mdist || dist * dist > chi2max * (ei + s.ezt2[j])) continue;
        mdist = dist;
        s.root[i] = s.iv[j];
      }
      continue;
    }
    s.root[i] = best != ~0ull ? s.iv[s.hbins[0xffffffffu - uint32_t(best & 0xffffffffu)]] : s.iv[i];
  }
  __syncthreads();
  // edge tracks take their core's root; the others keep theirs
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x)
    if (s.nn[i] < minT) s.iv[i] = s.root[i];
  __syncthreads();
}

// Launched as a cluster of P CTAs per event (pairs for large batches).  With
// P > 1 and the per-track arrays in shared memory, every CTA builds the track
// arrays and the z histogram, the two neighbour searches are divided among the
// CTAs by track, each result written into every CTA's shared memory, and rank
// 0 alone continues from there.
__global__ void __launch_bounds__(kVtxThreads) kVertices(Workspace ws, int algo) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const uint32_t rank = cl.block_rank(), P = cl.num_blocks();
  extern __shared__ __align__(16) char vsm[];
  __shared__ uint32_t scanSh[33];
  __shared__ uint32_t hoff[257];
  __shared__ uint32_t vOff[kMaxVtx + 1], vCur[kMaxVtx + 1];
  __shared__ uint32_t sNt, sFound, sGuard, sNv;
  __shared__ uint32_t sCtaCnt;  // tracks this CTA selected
  __shared__ int sFlag;
  const uint32_t e = blockIdx.y;
  const uint32_t lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  EventCounters* c = ws.ev + e;
  const uint32_t nTuples = c->nTuples;
  const uint32_t* toff = ws.tupleOff + size_t(e) * (ws.cap.tuples + 1);
  const uint8_t* q = ws.quality + size_t(e) * ws.cap.tuples;
  const float* pt = ws.pt + size_t(e) * ws.cap.tuples;
  const float* st = ws.state + size_t(e) * ws.cap.tuples * 5;
  const float* cov = ws.cov + size_t(e) * ws.cap.tuples * 15;
  int16_t* idv = ws.idv + size_t(e) * ws.cap.tuples;
  float* zv = ws.zv + size_t(e) * kMaxVtx;
  float* wv = ws.wv + size_t(e) * kMaxVtx;
  float* vchi2 = ws.vchi2 + size_t(e) * kMaxVtx;
  float* ptv2 = ws.ptv2 + size_t(e) * kMaxVtx;
  int32_t* ndof = ws.ndof + size_t(e) * kMaxVtx;
  uint16_t* sortInd = ws.sortInd + size_t(e) * kMaxVtx;

  // ---- loadTracks: the serial loop stops at the first empty tuple
  if (threadIdx.x == 0) {
    uint32_t g = nTuples;
    const uint32_t bins = ws.cap.tuples;
    if (nTuples == bins && toff[bins] == toff[bins - 1]) g = bins - 1;
    sGuard = g;
  }
  __syncthreads();
  const uint32_t guard = sGuard;
  // the selection of tuple t, its four loads issued together
  auto selected = [&](uint32_t t) {
    const uint32_t nh = toff[t + 1] - toff[t];
    const uint8_t qt = q[t];
    const float ptt = pt[t];
    return (nh >= 4) & (qt == 2) & !(ptt < 0.5f);
  };
  // The cluster's CTAs split the tuples: CTA r takes [g0, g1).  Inside it each
  // warp takes a contiguous range, 32 consecutive tuples per step (coalesced
  // loads, four steps in flight).  Block scans over the warps' counts and the
  // CTAs' counts place every run, and a second walk writes the selected tracks
  // in ascending order (into every CTA's shared memory, or the global
  // scratch).  The selection of each step is kept as a bit when the range has
  // at most 64 steps, else evaluated again.
  const uint32_t g0 = uint32_t(uint64_t(guard) * rank / P), g1 = uint32_t(uint64_t(guard) * (rank + 1) / P);
  for (uint32_t t = g0 + threadIdx.x; t < g1; t += blockDim.x) idv[t] = -1;
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t R = (g1 - g0 + nw * 32 - 1) / (nw * 32) * 32;
  const uint32_t w0 = min(g1, g0 + warp * R), w1 = min(g1, w0 + R);
  const uint32_t steps = (w1 - w0 + 31) / 32;
  const bool keepBits = steps <= 64;
  uint32_t cnt = 0;
  uint64_t bits = 0;
  for (uint32_t k = 0; k < steps; k += 4) {
    bool sel[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
      const uint32_t t = w0 + (k + u) * 32 + lane;
      sel[u] = k + u < steps && t < w1 && selected(t);
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
      if (sel[u] && keepBits) bits |= uint64_t(1) << (k + u);
      cnt += __popc(__ballot_sync(0xffffffffu, sel[u]));
    }
  }
  uint32_t ctaTotal;
  const uint32_t first = __shfl_sync(0xffffffffu, blockExclusiveScan(lane == 0 ? cnt : 0u, scanSh, &ctaTotal), 0);
  if (threadIdx.x == 0) sCtaCnt = ctaTotal;
  // every CTA has started and holds its count (and every tuple's idv is
  // cleared): the counts are read across the cluster
  cl.sync();
  uint32_t base = 0, total = 0;
  for (uint32_t r = 0; r < P; ++r) {
    const uint32_t n = *cl.map_shared_rank(&sCtaCnt, r);
    base += r < rank ? n : 0u;
    total += n;
  }
  if (threadIdx.x == 0) {
    sNt = min(total, kMaxVtxTracks);
    // beyond ZVertexSoA::MAXTRACKS the reference writes past its arrays
    if (total > kMaxVtxTracks && rank == 0) atomicOr(&c->flags, kFlagVtxOverflow);
  }
  __syncthreads();
  // The count decides where the per-track arrays live: in the shared memory
  // of every CTA, or once in the global scratch.  The neighbour searches are
  // split among the cluster's CTAs (not the iterative clusterer's); their results go
  // to every CTA's shared memory, or once to the global scratch.
  const bool smemPath = sNt <= kSmemTracks;
  const VtxScratch s = smemPath ? carve(vsm, kSmemTracks) : scratchOf(ws, e);
  const bool split = P > 1 && algo != 2;
  const bool remote = split && smemPath;       // results written into every CTA
  const bool active = split || rank == 0;      // CTAs that take part in the searches
  const bool writer = smemPath || rank == 0;   // CTAs that build their own track arrays
  // the searches' tracks: kNbrLanes lanes each, 32 / kNbrLanes tracks per warp
  const uint32_t sub = lane / kNbrLanes, gl = lane % kNbrLanes;
  const uint32_t gFirst = ((split ? rank * nw : 0u) + (threadIdx.x >> 5)) * (32 / kNbrLanes);
  const uint32_t gStride = (split ? P * nw : nw) * (32 / kNbrLanes);
  // every CTA places its selected tracks; in the shared-memory path each
  // track goes to every CTA that works on it (all with the split, else rank 0)
  const uint32_t nDst = smemPath ? (split ? P : 1u) : 1u;
  {
    uint32_t pos = base + first;
    for (uint32_t k = 0; k < steps; k += 4) {
      bool sel[4];
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t t = w0 + (k + u) * 32 + lane;
        sel[u] = keepBits ? ((bits >> (k + u)) & 1u) != 0 : (k + u < steps && t < w1 && selected(t));
      }
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t t = w0 + (k + u) * 32 + lane;
        const uint32_t m = __ballot_sync(0xffffffffu, sel[u]);
        const uint32_t it = pos + __popc(m & lanemaskLt());
        if (sel[u] && it < kMaxVtxTracks) {
          const float z = st[size_t(t) * 5 + 4], ez = cov[size_t(t) * 15 + 14], p2 = pt[t] * pt[t];
          for (uint32_t d = 0; d < nDst; ++d) {
            VtxScratch sd = s;
            if (smemPath) sd = carve(reinterpret_cast<char*>(cl.map_shared_rank(vsm, split ? d : 0u)), kSmemTracks);
            sd.itrk[it] = t;
            sd.zt[it] = z;
            sd.ezt2[it] = ez;
            sd.ptt2[it] = p2;
          }
        }
        pos += __popc(m);
      }
    }
  }
  // every track array is complete
  cl.sync();
  const uint32_t nt = sNt;
  const float eps = 0.07f, errmax = 0.01f, chi2max = 9.f;
  const float er2mx = errmax * errmax;

  if (active) {
  // ---- clusterTracksByDensity: z histogram (256 bins of 1 mm)
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
    int iz = int(double(s.zt[i]) * 10.);
    iz = min(max(iz, -128), 127);
    if (writer) {
      s.izt[i] = uint8_t(iz + 128);
      s.iv[i] = int32_t(i);
      s.nn[i] = 0;
    }
  }
  __syncthreads();
  // The serial fill stores each bin in descending track order: the items are
  // the tracks from the last one down.  In the global-scratch path every CTA
  // needs the bins' starts, and rank 0 writes their content; a CTA cannot
  // read another's izt before the cluster barrier, so each forms its own.
  static_assert(kVtxThreads / 32 * 256 * 2 <= kSmemTracks * 4, "the histogram's table in root");
  orderedFill(nt, 256, smemPath ? reinterpret_cast<uint16_t*>(s.root) : reinterpret_cast<uint16_t*>(vsm), nw, hoff,
              scanSh,
              [&](uint32_t r) { return uint32_t(min(max(int(double(s.zt[nt - 1 - r]) * 10.), -128), 127) + 128); },
              [&](uint32_t r, uint32_t pos) {
                if (writer) s.hbins[pos] = uint16_t(nt - 1 - r);
              });
  if (writer) {
    // z and its error of every track in histogram order, so that the
    // neighbour searches read their candidates contiguously (zz and list are
    // free until the fits)
    float* zP = s.zz;
    float* eP = reinterpret_cast<float*>(s.list);
    for (uint32_t p = threadIdx.x; p < nt; p += blockDim.x) {
      const uint32_t j = s.hbins[p];
      zP[p] = s.zt[j];
      eP[p] = s.ezt2[j];
    }
  }
  }
  // every CTA of the cluster has cleared its own neighbour counts before any
  // CTA writes counts into the others' shared memory; the global scratch's
  // histogram is complete
  cl.sync();
  // candidates in histogram order: z, its error and (below) the neighbour count
  const float* zP = s.zz;
  const float* eP = reinterpret_cast<const float*>(s.list);
  int32_t* nP = s.root;  // free until the percolation
  if (active) {
  // neighbour counts: kNbrLanes lanes per track (taken in histogram order)
  // share the entries of the track's three bins.  Each count is kept by track
  // (nn) and by histogram position (nP).  A track has a few tens of
  // candidates: a warp per track left most of its instructions in the
  // reductions (1087 tracks: 8k and, for the closest denser neighbour below,
  // 17k of the kernel's 113k cycles).
  for (uint32_t p0 = gFirst; p0 < nt; p0 += gStride) {
    const uint32_t pi = p0 + sub;
    uint32_t cnt = 0, i = 0;
    if (pi < nt) {
      i = s.hbins[pi];
      const float zi = zP[pi], ei = eP[pi];
      if (!(ei > er2mx)) {
        const int b0 = max(0, int(s.izt[i]) - 1), b1 = min(255, int(s.izt[i]) + 1);
        const uint32_t pb = hoff[b0], pe = hoff[b1 + 1];
        for (uint32_t p = pb + gl; p < pe; p += kNbrLanes) {
          const float dist = fabsf(zi - zP[p]);
          // a track is not its own neighbour: its histogram position is pi
          cnt += (p != pi && !(dist > eps) && (algo == 1 || !(dist * dist > chi2max * (ei + eP[p])))) ? 1u : 0u;
        }
      }
    }
    cnt = groupSum(cnt);
    if (pi < nt) {
      if (remote) {
        for (uint32_t r = gl; r < P; r += kNbrLanes) {
          cl.map_shared_rank(s.nn, r)[i] = int32_t(cnt);
          cl.map_shared_rank(nP, r)[pi] = int32_t(cnt);
        }
      } else if (gl == 0) {
        s.nn[i] = int32_t(cnt);
        nP[pi] = int32_t(cnt);
      }
    }
  }
  }
  // every CTA holds every neighbour count
  cl.sync();
  // only rank 0 goes on after the searches: their results go there
  int32_t* const ivOut = remote ? cl.map_shared_rank(s.iv, 0) : s.iv;
  if (active && algo == 1) linkCores(s, nt, hoff, eps, 2, gFirst, gStride, ivOut);
  if (active && algo == 0) {
  // Closest denser neighbour.  The serial loop (mdist starts at eps; a
  // candidate is taken when denser, not farther than mdist and
  // chi2-compatible) ends on the last candidate of minimal distance among the
  // qualifying ones: each lane runs it over its candidates, and the lanes'
  // results are combined as the minimum of (distance, reversed position).  A
  // track with a denser candidate at a NaN distance runs the serial loop.
  for (uint32_t p0 = gFirst; p0 < nt; p0 += gStride) {
    const uint32_t pi = p0 + sub;
    uint32_t i = 0;
    // per lane, in ascending position: the closest so far (the last of equal
    // distances) and whether a NaN distance was met
    float bestDist = eps;
    uint32_t bestPos = 0xffffffffu;
    int32_t nan = 0;
    uint32_t pb = 0, pe = 0;
    float zi = 0.f, ei = 0.f;
    int32_t ni = 0;
    auto denser = [&](uint32_t p) {
      const int32_t nj = nP[p];
      return !(nj < ni) && !(nj == ni && zP[p] >= zi);
    };
    auto near = [&](float dist, uint32_t p) { return !(dist * dist > chi2max * (ei + eP[p])); };
    if (pi < nt) {
      i = s.hbins[pi];
      const int b0 = max(0, int(s.izt[i]) - 1), b1 = min(255, int(s.izt[i]) + 1);
      pb = hoff[b0];
      pe = hoff[b1 + 1];
      zi = zP[pi];
      ei = eP[pi];
      ni = nP[pi];
      for (uint32_t p = pb + gl; p < pe; p += kNbrLanes) {
        const float dist = fabsf(zi - zP[p]);
        if (!denser(p)) continue;
        if (isnan(dist)) nan = 1;
        if (dist <= bestDist && near(dist, p)) {
          bestDist = dist;
          bestPos = p;
        }
      }
    }
    nan = groupMax(nan);
    const unsigned long long bestKey =
        groupMin(bestPos == 0xffffffffu
                     ? ~0ull
                     : (uint64_t(__float_as_uint(bestDist)) << 32) | uint64_t(0xffffffffu - bestPos));
    int32_t best = int32_t(i);
    if (pi < nt) {
      if (nan) {
        // the serial loop as written
        float mdist = eps;
        for (uint32_t p = pb; p < pe; ++p) {
          const float dist = fabsf(zi - zP[p]);
          if (!denser(p) || dist > mdist || !near(dist, p)) continue;
          mdist = dist;
          best = int32_t(s.hbins[p]);
        }
      } else if (bestKey != ~0ull)
        best = int32_t(s.hbins[0xffffffffu - uint32_t(bestKey & 0xffffffffu)]);
      if (gl == 0) ivOut[i] = best;
    }
  }
  }
  // rank 0 holds every track's link and goes on alone; no CTA reads another
  // CTA's shared memory after this point
  cl.sync();
  if (rank != 0) return;
  if (algo != 0) clusterCoresAndEdges(s, nt, hoff, algo, eps, chi2max, 2, &sFlag);
  // percolate to the seed
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
    int32_t m = s.iv[i];
    while (m != s.iv[m]) m = s.iv[m];
    s.root[i] = m;
  }
  __syncthreads();
  // number the seeds with nn >= minT in ascending track order
  {
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < nt; i0 += blockDim.x) {
      uint32_t i = i0 + threadIdx.x;
      uint32_t seed = (i < nt && s.root[i] == int32_t(i) && s.nn[i] >= 2) ? 1u : 0u;
      uint32_t tot;
      uint32_t pre = blockExclusiveScan(seed, scanSh, &tot);
      if (seed) s.iv[i] = int32_t(carry + pre);  // rank of the seed
      carry += tot;
    }
    if (threadIdx.x == 0) sFound = carry;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) {
    int32_t r = s.root[i];
    // seeds hold their rank in iv[r]; noise seeds end as 9997 (= -(-9998) - 1)
    s.zz[i] = 0;
    s.newV[i] = 0;
    int32_t v = (s.nn[r] >= 2) ? s.iv[r] : 9997;
    s.root[i] = v;  // staged: iv of a seed is still read by other threads in this loop
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) s.iv[i] = s.root[i];
  __syncthreads();
  uint32_t found = sFound;
  if (found >= kMaxVtx) {
    if (threadIdx.x == 0) atomicOr(&c->flags, kFlagVtxOverflow);
    found = kMaxVtx - 1;
  }

  // the grouping's table and the warps' sum buffers (used in turn): the place of
  // nn and root, free from here on, or the dynamic shared memory that the
  // global-scratch path leaves unused
  static_assert(kVtxThreads / 32 * kSumWords <= kSmemTracks && 5 * kSmemTracks % 4 == 0, "sum buffers in nn, aligned");
  static_assert(2 * kSmemTracks * 4 / 2 / kMaxVtx >= 1, "a table row for every vertex in nn and root");
  char* const spare = smemPath ? reinterpret_cast<char*>(s.nn) : vsm;
  float* const sumBuf = reinterpret_cast<float*>(spare) + (threadIdx.x >> 5) * kSumWords;
  uint16_t* const tab = reinterpret_cast<uint16_t*>(spare);
  const uint32_t tabBytes = smemPath ? 2 * kSmemTracks * 4 : uint32_t(kVtxSmemBytes);

  // ---- fitVertices(50)
  fitVertices(s, nt, found, 50.f, zv, wv, vchi2, ndof, vOff, scanSh, sumBuf, tab, tabBytes);

  // ---- splitVertices(9): tracks of each vertex are the list built by the fit
  //      minus the ones rejected there (iv = 9999)
  if (threadIdx.x == 0) sNv = found;
  __syncthreads();
  for (uint32_t kv = threadIdx.x >> 5; kv < found; kv += nw) {
    if (lane == 0) vCur[kv] = 0;  // split flag
    if (ndof[kv] < 4) continue;
    if (vchi2[kv] < 9.f * float(ndof[kv])) continue;
    if (ndof[kv] >= 512) {
      if (lane == 0) atomicOr(&c->flags, kFlagVtxOverflow);
      continue;
    }
    const uint32_t b = vOff[kv], n = vOff[kv + 1] - b;
    for (uint32_t k = lane; k < n; k += 32) {
      const uint32_t i = s.list[b + k];
      if (s.iv[i] != int32_t(kv)) continue;
      s.zz[i] = s.zt[i] - zv[kv];
      s.newV[i] = s.zz[i] < 0 ? 0 : 1;
    }
    __syncwarp();
    float znew[2], wnew[2];
    int maxiter = 20;
    bool more = true;
    while (more) {
      more = false;
      float sums = 0;  // lanes 0..3: z and weight of the first half, of the second
      for (uint32_t k0 = 0; k0 < n; k0 += 32) {
        const uint32_t k = k0 + lane;
        float t[4] = {0.f, 0.f, 0.f, 0.f};
        if (k < n) {
          const uint32_t i = s.list[b + k];
          if (s.iv[i] == int32_t(kv)) {
            const float ww = 1.f / s.ezt2[i];
            const float p = s.zz[i] * ww;
            const bool second = s.newV[i] != 0;
            t[0] = second ? 0.f : p;
            t[1] = second ? 0.f : ww;
            t[2] = second ? p : 0.f;
            t[3] = second ? ww : 0.f;
          }
        }
        orderedSums(sumBuf, t, sums);
      }
      znew[0] = __shfl_sync(0xffffffffu, sums, 0);
      wnew[0] = __shfl_sync(0xffffffffu, sums, 1);
      znew[1] = __shfl_sync(0xffffffffu, sums, 2);
      wnew[1] = __shfl_sync(0xffffffffu, sums, 3);
      znew[0] /= wnew[0];
      znew[1] /= wnew[1];
      bool changed = false;
      for (uint32_t k = lane; k < n; k += 32) {
        const uint32_t i = s.list[b + k];
        if (s.iv[i] != int32_t(kv)) continue;
        const float d0 = fabsf(s.zz[i] - znew[0]);
        const float d1 = fabsf(s.zz[i] - znew[1]);
        const uint8_t newer = d0 < d1 ? 0 : 1;
        changed |= newer != s.newV[i];
        s.newV[i] = newer;
      }
      more = __any_sync(0xffffffffu, changed);
      __syncwarp();
      --maxiter;
      if (maxiter <= 0) more = false;
    }
    if (0 == wnew[0] || 0 == wnew[1]) continue;
    const float dist2 = (znew[0] - znew[1]) * (znew[0] - znew[1]);
    const float chi2Dist = dist2 / (1.f / wnew[0] + 1.f / wnew[1]);
    if (chi2Dist < 4) continue;
    if (lane == 0) vCur[kv] = 1;
  }
  __syncthreads();
  // new vertex numbers in ascending order of the vertex that was split
  {
    uint32_t carry = 0;
    for (uint32_t k0 = 0; k0 < found; k0 += blockDim.x) {
      uint32_t kv = k0 + threadIdx.x;
      uint32_t f = kv < found ? vCur[kv] : 0u;
      uint32_t tot;
      uint32_t pre = blockExclusiveScan(f, scanSh, &tot);
      if (kv < found) vCur[kv] = f ? (found + carry + pre + 1) : 0u;  // 0: no split, else igv+1
      carry += tot;
    }
    if (threadIdx.x == 0) sNv = found + carry;
  }
  __syncthreads();
  // tracks of the split-off halves to their new vertices (warp per vertex)
  for (uint32_t kv = threadIdx.x >> 5; kv < found; kv += nw) {
    if (vCur[kv] == 0) continue;
    const uint32_t igv = vCur[kv] - 1;
    const uint32_t b = vOff[kv], n = vOff[kv + 1] - b;
    for (uint32_t k = lane; k < n; k += 32) {
      const uint32_t i = s.list[b + k];
      if (s.iv[i] == int32_t(kv) && s.newV[i] == 1) s.iv[i] = int32_t(igv);
    }
  }
  __syncthreads();
  uint32_t nv = sNv;
  if (nv >= kMaxVtx) {
    if (threadIdx.x == 0) atomicOr(&c->flags, kFlagVtxOverflow);
    nv = kMaxVtx - 1;
  }

  // ---- fitVertices(5000)
  fitVertices(s, nt, nv, 5000.f, zv, wv, vchi2, ndof, vOff, scanSh, sumBuf, tab, tabBytes);

  // ---- sortByPt2
  if (threadIdx.x == 0) c->nVertices = nv;
  if (nv < 1) return;
  for (uint32_t i = threadIdx.x; i < nt; i += blockDim.x) idv[s.itrk[i]] = int16_t(s.iv[i]);
  // the fit above left every vertex's accepted tracks in vOff/list order
  for (uint32_t v = threadIdx.x >> 5; v < nv; v += nw) {
    const uint32_t b = vOff[v], n = vOff[v + 1] - b;
    float p2 = 0;
    for (uint32_t k0 = 0; k0 < n; k0 += 32) {
      const uint32_t k = k0 + lane;
      float t[1] = {0.f};
      if (k < n) {
        const uint32_t i = s.list[b + k];
        if (s.iv[i] <= 9990) t[0] = s.ptt2[i];
      }
      orderedSums(sumBuf, t, p2);
    }
    if (lane == 0) ptv2[v] = p2;
  }
  __syncthreads();
  if (nv == 1) {
    if (threadIdx.x == 0) sortInd[0] = 0;
    return;
  }
  for (uint32_t v = threadIdx.x; v < nv; v += blockDim.x) {
    float p = ptv2[v];
    uint32_t r = 0;
    for (uint32_t u = 0; u < nv; ++u) {
      float o = ptv2[u];
      r += (o < p || (o == p && u < v)) ? 1u : 0u;
    }
    sortInd[r] = uint16_t(v);
  }
  if (threadIdx.x == 0) c->nVtxTracks = nt;
}

}  // namespace

cudaError_t runVertices(Workspace& ws, uint32_t nEvents, cudaStream_t stream, int algo) {
  // opt in to the large shared-memory carve-out, once per device
  static std::atomic<uint64_t> configured{0};
  int dev = 0;
  cudaGetDevice(&dev);
  const uint64_t bit = uint64_t(1) << (dev & 63);
  if (!(configured.load() & bit)) {
    cudaError_t e = cudaFuncSetAttribute(kVertices, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kVtxSmemBytes));
    if (e != cudaSuccess) return e;
    configured.fetch_or(bit);
  }
  // small batches: a cluster of kVtxCtas CTAs per event, as many as the SMs
  // hold (a CTA's shared memory takes one whole), shortens the event's
  // latency (8 instead of 4: 93k -> 52k cycles for walking the 318k tuples of a
  // PU200 event); large batches: pairs of CTAs (measured at 64 PU50 events:
  // 0.52 -> 0.39 ms per batch and +2 % throughput with three batches in
  // flight).  Four CTAs from 17 to 32 events: 24 uneven PU20-200 events 2 % faster
  // than in pairs; 17, 24 and 32 PU50 events, 24 PU20 ones and 24 dense ones with
  // and without DBSCAN within 0.4 % either way.  The iterative clusterer does its
  // searches on one CTA; there the others share the loading only.
  const uint32_t P = nEvents <= kClusterMaxEvents ? kVtxCtas : (nEvents <= 2 * kClusterMaxEvents ? 4u : 2u);
  cudaError_t le = cudaSuccess;
  PG_PROBED("kVertices", stream,
            le = launchClustered(kVertices, P, nEvents, kVtxThreads, kVtxSmemBytes, stream, ws, algo));
  if (le != cudaSuccess) return le;
  return cudaGetLastError();
}

}  // namespace pixgpu
