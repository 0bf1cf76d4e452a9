// gh.cu -- batched Greiner-Hormann clipping of polygon pairs on sm_100a.
//
// Reference path: ghcuda (GH-CUDA/ghcuda.cpp:385-425) clips one pair at a time:
// calculateIntersections on the GPU (gppolyclip_mDIV512.cu:1298-1715: CMBR edge filter,
// counts, host scans, neighbour map, intersections, per-edge alpha sort, initial labels),
// then the CPU phases of GH-CUDA/lib/polyclip.h (labelIntersections :335-735,
// createResult :743-783, cleanUpResult :791-807).  Here every phase of every pair of a
// batch runs on the device:
//
//   G0 setup        thread/pair: the swap rule (ghcuda.cpp:64-91: the polygon with more
//                   vertices is P), MBRs, common MBR (ghcuda.cpp:94-125), disjoint check
//   G1 edge filter  warp/pair: P and Q edges whose box touches the common MBR
//                   (gppolyclip_mDIV512.cu:382-415), compacted in edge order
//   G2/G3 records   warp per 32-edge-pair chunk of each pair's filtered P x Q grid: box
//                   test (:345-371) and classification from both sides (:95-169);
//                   records = P-side hits, appended as they are found, the P/Q totals
//                   decide validity (:1461).  Pairs with large grids: a uniform grid over
//                   the common MBR, a warp per eight P edges.  (The record export counts
//                   first and writes in (pair, P edge, Q edge) order.)
//   G4 ring layout  per edge: 1 source vertex + inserted vertices; one device scan per
//                   side gives every vertex its slot (replaces the host scans :1431-1434)
//   G5 ring fill    thread, warp or block per edge by its insertions: inserted vertices
//                   ordered by exact parameter (ties: later insertion first, as
//                   polygon.h:101-113 inserts in the loop order of polyclip.h:202-205)
//                   instead of the reference GPU's 1e-7-quantised radix sort (:290-305, :1034)
//   G6 links        thread/record: neighbour links as polyclip.h:215-267 makes them; a
//                   source vertex linked by several records keeps the last one
//   G7 label+trace  thread, warp, block or grid per pair by its size: initial labels, chains,
//                   special cases, entry/exit, split pairs, crossing candidates, tracing and
//                   clean-up
//   G8 compaction   per-pair output regions -> one contiguous result
//
// Layout in HBM: the input layers stay interleaved FP64 (16 B per vertex).  Records are
// structure-of-arrays (P edge, Q edge, alpha, beta, type, pair).  Each pair owns a ring
// region per side holding its merged vertex ring followed by room for the vertices the
// labelling may add (one temporary vertex, one duplicate per split vertex): x, y, next,
// prev, neighbour (pair-local slot on the other side), flags, label, entry/exit.
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>
#include <vector>
#include "common.cuh"
#include "engine.cuh"
#include "prims.cuh"

namespace gcmfgh {

__device__ __noinline__ int classify_exact_open(double2 P1, double2 P2, double2 Q1, double2 Q2, double2* ab, bool* qhit) {
  double a2, b2;
  *qhit = classify_exact(Q1.x, Q1.y, Q2.x, Q2.y, P1.x, P1.y, P2.x, P2.y, a2, b2) != 0;
  return classify_exact(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y, ab->x, ab->y);
}

namespace {

constexpr int kThreads = 256;
constexpr int kWarpsPerBlock = kThreads / 32;
constexpr int kChunk = 32;             // edge pairs per warp work unit (one per lane; 64 and 128 measured slower)
constexpr int64_t kFirstRecordCap = 1 << 22;   // records held by a fused count + emit without a hint
constexpr int kFilterTile = 4;         // lanes per small pair in the edge filter
constexpr int64_t kFilterTileMax = 64; // ring size up to which the narrow tiles take a pair

inline unsigned blocks_for_warps(int64_t warps) {
  return (unsigned)((warps + kWarpsPerBlock - 1) / kWarpsPerBlock);
}
inline unsigned blocks_for(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }


// ---------------------------------------------------------------- pair setup
struct PairDev {
  int64_t* pS;      // first vertex (index into P's layer)
  int64_t* qS;
  int32_t* nP;      // ring size (closing vertex excluded)
  int32_t* nQ;
  int8_t* pSide;    // 0: P is the base polygon, 1: P is the overlay polygon
  double* cmbr;     // [4 K]
  int32_t* status;  // 0 ok, 1 invalid, 2 disjoint, 3 trace error
};

__device__ __forceinline__ const double2* layer_xy(const LayerDev& Lb, const LayerDev& Lo, int side) {
  return reinterpret_cast<const double2*>(side == 0 ? Lb.xy : Lo.xy);
}

__global__ void setup_kernel(LayerDev Lb, LayerDev Lo, const int32_t* __restrict__ pid,
                             const int32_t* __restrict__ qid, int64_t K, const double* __restrict__ mb,
                             const double* __restrict__ mo, PairDev D, int32_t* __restrict__ swapped,
                             int no_swap) {
  int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k >= K) return;
  int b = pid[k], o = qid[k];
  int nb = Lb.vnum[b] - 1, no = Lo.vnum[o] - 1;
  bool sw = !no_swap && nb < no;        // ghcuda.cpp:66: swap when |P| < |Q|
  int64_t sb = Lb.vps[b] - Lb.vnum[b], so = Lo.vps[o] - Lo.vnum[o];
  double4 MB = reinterpret_cast<const double4*>(mb)[b];
  double4 MO = reinterpret_cast<const double4*>(mo)[o];
  double4 MP = sw ? MO : MB, MQ = sw ? MB : MO;
  D.pS[k] = sw ? so : sb; D.qS[k] = sw ? sb : so;
  D.nP[k] = sw ? no : nb; D.nQ[k] = sw ? nb : no;
  D.pSide[k] = sw ? 1 : 0;
  swapped[k] = sw ? 1 : 0;
  int st = 0;
  if (MP.x > MQ.z || MP.z < MQ.x || MP.y > MQ.w || MP.w < MQ.y) st = 2;   // ghcuda.cpp:109-116
  if (D.nP[k] < 1 || D.nQ[k] < 1) st = 2;
  D.status[k] = st;
  reinterpret_cast<double4*>(D.cmbr)[k] = make_double4(fmax(MP.x, MQ.x), fmax(MP.y, MQ.y),
                                                       fmin(MP.z, MQ.z), fmin(MP.w, MQ.w));
}

// ---------------------------------------------------------------- G1 edge filter
// W lanes per pair (W = 32: a warp).  Two passes split the pairs by ring size: narrow
// tiles for small pairs (they also zero the counts of pairs with nothing to test), whole
// warps for the rest.
// A pair of a join's clip set whose candidate has the join's common-MBR edge lists (the
// same boxes, the same test) takes them from there: the join tests every stored edge
// including the zero-length one from the stored closing vertex back to the first
// (GPU_Join.h:576-577), which the clip's open ring does not have, so that entry (the last,
// index n) is dropped; and both rings must be closed (stored closing vertex equal to the
// first), so that the join's last real edge is the clip's.
__device__ __forceinline__ bool ring_closed(const double2* v, int n) {
  const double2 a = __ldg(v), b = __ldg(v + n);
  return a.x == b.x && a.y == b.y;
}

// member `me` of `of` takes its part of a pair's lists from the join; false: the join has none
template <int kMode>
__device__ __forceinline__ bool join_lists(const LayerDev& Lb, const LayerDev& Lo, const PairDev& D, int64_t w, int pside,
                                           const JoinEdges& je, int32_t* cP, int32_t* cQ, const int64_t* offP,
                                           const int64_t* offQ, int32_t* LP, int32_t* LQ, int me, int of) {
  if (!je.cand) return false;
  const int64_t cd = je.cand[w];
  if (!je.flag[cd] || !ring_closed(layer_xy(Lb, Lo, pside) + D.pS[w], D.nP[w]) ||
      !ring_closed(layer_xy(Lb, Lo, 1 - pside) + D.qS[w], D.nQ[w]))
    return false;
  for (int side = 0; side < 2; ++side) {
    const bool base = (side == 0 ? pside : 1 - pside) == 0;
    const int n = side == 0 ? D.nP[w] : D.nQ[w];
    const int E = (base ? je.bE : je.oE)[cd];
    const int32_t* src = base ? je.bList + je.bOff[cd] : je.oList + je.oOff[cd];
    const int cnt = E - ((E > 0 && src[E - 1] == n) ? 1 : 0);
    if (kMode == 0) {
      if (me == 0) (side == 0 ? cP : cQ)[w] = cnt;
    } else {
      int32_t* dst = side == 0 ? LP + offP[w] : LQ + offQ[w];
      for (int j = me; j < cnt; j += of) dst[j] = src[j];
    }
  }
  return true;
}

template <int kMode, int W>
__global__ void __launch_bounds__(kThreads, 6)
edge_filter_kernel(LayerDev Lb, LayerDev Lo, PairDev D, int64_t K, int32_t* __restrict__ cP,
                   int32_t* __restrict__ cQ, const int64_t* __restrict__ offP,
                   const int64_t* __restrict__ offQ, int32_t* __restrict__ LP, int32_t* __restrict__ LQ,
                   int64_t lo, int64_t hi, JoinEdges je, LongPairs longs) {
  constexpr unsigned kBits = (W == 32) ? 0xffffffffu : ((1u << (W & 31)) - 1u);
  const int64_t w = ((int64_t)blockIdx.x * kThreads + threadIdx.x) / W;
  const int tl = (int)(threadIdx.x & (W - 1));
  const int tbase = (int)(lane_id() & ~(unsigned)(W - 1));
  const unsigned tmask = kBits << tbase;
  if (w >= K) return;
  if (D.status[w] != 0) { if (kMode == 0 && W != 32 && tl == 0) { cP[w] = 0; cQ[w] = 0; } return; }
  {
    const int64_t size = (int64_t)D.nP[w] + D.nQ[w];
    if (size <= lo || size > hi) {                   // another pass takes this pair
      if (kMode == 0 && W == 32 && size > hi && longs.ids && tl == 0) longs.add(w);
      return;
    }
  }
  const int pside = D.pSide[w];
  if (join_lists<kMode>(Lb, Lo, D, w, pside, je, cP, cQ, offP, offQ, LP, LQ, tl, W)) return;
  double4 c = reinterpret_cast<const double4*>(D.cmbr)[w];
  for (int side = 0; side < 2; ++side) {
    const double2* v = layer_xy(Lb, Lo, side == 0 ? pside : 1 - pside) + (side == 0 ? D.pS[w] : D.qS[w]);
    const int n = side == 0 ? D.nP[w] : D.nQ[w];
    int cnt = 0;
    int64_t pos = 0;
    int32_t* list = nullptr;
    if (kMode == 1) { pos = side == 0 ? offP[w] : offQ[w]; list = side == 0 ? LP : LQ; }
    // whole warps take kUnroll groups of W edges per step: every group's loads are issued
    // before the first ballot
    constexpr int kUnroll = (W == 32) ? 4 : 1;
    for (int k0 = 0; k0 < n; k0 += W * kUnroll) {
      bool hit[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = k0 + u * W + tl;
        hit[u] = false;
        if (k < n) {
          double2 a = __ldg(v + k), b = __ldg(v + (k + 1 < n ? k + 1 : 0));
          hit[u] = edge_touches_box(a.x, a.y, b.x, b.y, c.x, c.y, c.z, c.w);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        unsigned m = __ballot_sync(tmask, hit[u]);
        if (W != 32) m = (m >> tbase) & kBits;
        if (kMode == 1 && hit[u]) list[pos + cnt + __popc(m & ((1u << tl) - 1u))] = k0 + u * W + tl;
        cnt += __popc(m);
      }
    }
    if (kMode == 0 && tl == 0) { if (side == 0) cP[w] = cnt; else cQ[w] = cnt; }
  }
}

// A block per pair: the listed pairs (too long for a warp), or, with n given, the first n pairs
// of a batch that has no more pairs than blocks.
constexpr int kFilterLongThreads = 512;
constexpr int kFilterLongRounds = 4;
constexpr int kFilterLongBlocks = 2 * kSms;

template <int kMode>
__global__ void __launch_bounds__(kFilterLongThreads)
edge_filter_long_kernel(LayerDev Lb, LayerDev Lo, PairDev D, int32_t* __restrict__ cP, int32_t* __restrict__ cQ,
                        const int64_t* __restrict__ offP, const int64_t* __restrict__ offQ, int32_t* __restrict__ LP,
                        int32_t* __restrict__ LQ, JoinEdges je, LongPairs longs, int n) {
  __shared__ int cnt[kFilterLongRounds * (kFilterLongThreads / 32) + 1];
  const unsigned total = longs.ids ? *longs.n : (unsigned)n;
  for (unsigned j = blockIdx.x; j < total; j += gridDim.x) {
    const int64_t w = longs.ids ? longs.ids[j] : (int64_t)j;
    if (D.status[w] != 0) {
      if (kMode == 0 && threadIdx.x == 0) { cP[w] = 0; cQ[w] = 0; }
      continue;
    }
    const int pside = D.pSide[w];
    if (join_lists<kMode>(Lb, Lo, D, w, pside, je, cP, cQ, offP, offQ, LP, LQ, (int)threadIdx.x, kFilterLongThreads)) continue;
    const double4 c = reinterpret_cast<const double4*>(D.cmbr)[w];
    for (int side = 0; side < 2; ++side) {
      const double2* v = layer_xy(Lb, Lo, side == 0 ? pside : 1 - pside) + (side == 0 ? D.pS[w] : D.qS[w]);
      const int m = side == 0 ? D.nP[w] : D.nQ[w];
      auto touches = [&](int k) {
        const double2 a = __ldg(v + k), b = __ldg(v + (k + 1 < m ? k + 1 : 0));
        return edge_touches_box(a.x, a.y, b.x, b.y, c.x, c.y, c.z, c.w);
      };
      if (kMode == 0) {
        int mine = 0;
#pragma unroll 4
        for (int k = threadIdx.x; k < m; k += kFilterLongThreads) mine += touches(k) ? 1 : 0;
        mine = warp_sum(mine);
        __syncthreads();
        if (lane_id() == 0) cnt[threadIdx.x >> 5] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
          int sum = 0;
          for (int i = 0; i < kFilterLongThreads / 32; ++i) sum += cnt[i];
          (side == 0 ? cP : cQ)[w] = sum;
        }
      } else {
        int32_t* dst = side == 0 ? LP + offP[w] : LQ + offQ[w];
        block_list<kFilterLongThreads, kFilterLongRounds>(m, cnt, touches, [&](int k, int before) { dst[before] = k; });
      }
    }
  }
}

// Pairs whose filtered edge grid exceeds ClipParams::bin_grid edge pairs are not
// enumerated pair by pair: their edges are binned on a uniform grid (bin_* kernels).

// edge -> pair: a warp per pair fills the entries of its cnt[k] edges starting at off[k]
__global__ void range_owner_kernel(const int64_t* __restrict__ off, const int32_t* __restrict__ cnt, int64_t K,
                                   int32_t* __restrict__ owner) {
  const int64_t k = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  if (k >= K) return;
  const int64_t o = off[k];
  const int n = cnt[k];
  for (int j = lane_id(); j < n; j += 32) owner[o + j] = (int32_t)k;
}

// chunk -> pair: a warp per pair fills its chunks' entries
__global__ void chunk_pair_kernel(const int64_t* __restrict__ chunkOff, const int64_t* __restrict__ nchunk, int64_t K,
                                  int32_t* __restrict__ chunkPair) {
  const int64_t k = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  if (k >= K) return;
  const int64_t o = chunkOff[k], n = nchunk[k];
  for (int64_t j = lane_id(); j < n; j += 32) chunkPair[o + j] = (int32_t)k;
}

__global__ void chunk_count_kernel(const int32_t* __restrict__ cP, const int32_t* __restrict__ cQ,
                                   int64_t K, int64_t* __restrict__ nchunk, int64_t* __restrict__ bigList,
                                   unsigned long long* __restrict__ nBig, int64_t binGrid) {
  int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k >= K) return;
  int64_t W = (int64_t)cP[k] * cQ[k];
  if (W > binGrid) {
    nchunk[k] = 0;
    bigList[atomicAdd(nBig, 1ull)] = k;
  } else {
    nchunk[k] = (W + kChunk - 1) / kChunk;
  }
}

// ---------------------------------------------------------------- G2/G3 count + emit
struct Records {
  int32_t* p;       // pair-local P edge
  int32_t* q;       // pair-local Q edge
  double* a;        // alpha (on P)
  double* b;        // beta (on Q)
  int8_t* t;        // intersection type 1..8
  int32_t* k;       // pair
};

// Occupancy over registers: the count pass at most 64 registers (4 blocks per SM; count
// stage 1.29 -> 0.81 ms), the emit pass 40 (6 blocks; 0.55 -> 0.39 ms).  The
// exact-predicate instances keep 128 registers (their expansions would spill).
template <int kMode, int kExact>
__global__ void __launch_bounds__(kThreads, kExact ? 2 : (kMode == 1 ? 6 : 4))
intersect_kernel(LayerDev Lb, LayerDev Lo, PairDev D, int64_t K, const int64_t* __restrict__ chunkOff,
                 int64_t nChunks, const int32_t* __restrict__ cP, const int32_t* __restrict__ cQ,
                 const int64_t* __restrict__ offP, const int64_t* __restrict__ offQ,
                 const int32_t* __restrict__ LP, const int32_t* __restrict__ LQ, double eps,
                 int32_t* __restrict__ chunkRec, int32_t* __restrict__ chunkQ,
                 const int64_t* __restrict__ chunkRecOff, const int64_t* __restrict__ recOff, Records R,
                 const int32_t* __restrict__ chunkPair) {
  int64_t c = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  if (c >= nChunks) return;
  const int64_t k = chunkPair[c];                  // the pair this chunk belongs to
  const int nq = cQ[k];
  const int64_t W = (int64_t)cP[k] * nq;
  const int64_t t0 = (c - chunkOff[k]) * kChunk;
  const int pside = D.pSide[k];
  const double2* pv = layer_xy(Lb, Lo, pside) + D.pS[k];
  const double2* qv = layer_xy(Lb, Lo, 1 - pside) + D.qS[k];
  const int np_ = D.nP[k], nq_ = D.nQ[k];
  const int32_t* lp = LP + offP[k];
  const int32_t* lq = LQ + offQ[k];
  int recs = 0, qhits = 0;
  int64_t pos = (kMode == 1) ? recOff[k] + chunkRecOff[c] - chunkRecOff[chunkOff[k]] : 0;
  for (int it = 0; it < kChunk / 32; ++it) {
    int64_t t = t0 + it * 32 + lane_id();
    int tp = 0, tq = 0;
    int pe = 0, qe = 0;
    double alpha = 0, beta = 0;
    if (t < W) {
      if (W <= INT32_MAX) {                         // 32-bit division when it suffices
        const int tt = (int)t, r = tt / nq;
        pe = lp[r];
        qe = lq[tt - r * nq];
      } else {
        pe = lp[t / nq];
        qe = lq[t % nq];
      }
      double2 P1 = __ldg(pv + pe), P2 = __ldg(pv + (pe + 1 < np_ ? pe + 1 : 0));
      double2 Q1 = __ldg(qv + qe), Q2 = __ldg(qv + (qe + 1 < nq_ ? qe + 1 : 0));
      if (edge_boxes_touch(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y)) {
        if (kMode == 0 && !kExact) {
          bool qhit;
          tp = classify_edges_both(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y, eps, alpha, beta, qhit);
          tq = qhit ? 1 : 0;
        } else {
          tp = classify_mode(kExact, P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y, eps, alpha, beta);
          if (kMode == 0) {
            double a2, b2;
            tq = classify_mode(kExact, Q1.x, Q1.y, Q2.x, Q2.y, P1.x, P1.y, P2.x, P2.y, eps, a2, b2);
          }
        }
      }
    }
    unsigned m = __ballot_sync(0xffffffffu, tp != 0);
    if (kMode == 0) {
      recs += __popc(m);
      qhits += __popc(__ballot_sync(0xffffffffu, tq != 0));
    } else if (tp != 0) {
      int64_t r = pos + __popc(m & lanemask_lt());
      R.p[r] = pe; R.q[r] = qe; R.a[r] = alpha; R.b[r] = beta; R.t[r] = (int8_t)tp; R.k[r] = (int32_t)k;
    }
    pos += __popc(m);
  }
  if (kMode == 0 && lane_id() == 0) { chunkRec[c] = recs; chunkQ[c] = qhits; }
}

// Count and emit in one pass over the chunks.  Each warp classifies its chunk's edge pairs
// from both sides as the count pass does and stages its P-side records in shared memory;
// the block then takes one range of a global counter and copies its records there.  The
// records end up in block order, which nothing downstream depends on (the ring fill orders
// a ring's insertions by parameter and other edge; a link keeps the largest other edge).
// Per pair, the P-side records and the Q-side hits are added into pairRec / pairQ (skipped
// when pairRec is null: a re-run after an overflow).  Records at or past cap are counted
// and not written; the host then re-runs with arrays of the counted size.
struct FusedRecords {
  unsigned long long* total;   // records taken so far (all blocks)
  int64_t cap;                 // records the arrays hold
  int32_t* pairRec;            // per pair: P-side records
  int32_t* pairQ;              // per pair: Q-side hits
};

template <int kExact, int kWarpAppend>
__global__ void __launch_bounds__(kThreads, kExact ? 3 : 4)   // (the open cases' function takes 80 registers)
intersect_fused_kernel(LayerDev Lb, LayerDev Lo, PairDev D, const int64_t* __restrict__ chunkOff, int64_t nChunks,
                       const int32_t* __restrict__ cP, const int32_t* __restrict__ cQ,
                       const int64_t* __restrict__ offP, const int64_t* __restrict__ offQ,
                       const int32_t* __restrict__ LP, const int32_t* __restrict__ LQ, double eps, Records R,
                       const int32_t* __restrict__ chunkPair, FusedRecords F) {
  constexpr int kWarps = kThreads / 32;
  constexpr int kStage = kWarps * kChunk;           // at most one record per edge pair
  __shared__ double sA[kStage], sB[kStage];
  __shared__ int32_t sP[kStage], sQ[kStage];
  __shared__ int8_t sT[kStage];
  __shared__ int sOff[kWarps + 1];
  __shared__ int32_t sK[kWarps];
  __shared__ unsigned long long sBase;
  const int wib = (int)(threadIdx.x >> 5);
  const int64_t c = (int64_t)blockIdx.x * kWarps + wib;
  int recs = 0, qhits = 0;
  int64_t k = -1;
  if (c < nChunks) {
    k = chunkPair[c];
    const int nq = cQ[k];
    const int64_t W = (int64_t)cP[k] * nq;
    const int64_t t0 = (c - chunkOff[k]) * kChunk;
    const int pside = D.pSide[k];
    const double2* pv = layer_xy(Lb, Lo, pside) + D.pS[k];
    const double2* qv = layer_xy(Lb, Lo, 1 - pside) + D.qS[k];
    const int np_ = D.nP[k], nq_ = D.nQ[k];
    const int32_t* lp = LP + offP[k];
    const int32_t* lq = LQ + offQ[k];
    for (int it = 0; it < kChunk / 32; ++it) {
      const int64_t t = t0 + it * 32 + lane_id();
      int tp = 0, tq = 0, pe = 0, qe = 0;
      double alpha = 0, beta = 0;
      if (t < W) {
        if (W <= INT32_MAX) {
          const int tt = (int)t, r = tt / nq;
          pe = lp[r];
          qe = lq[tt - r * nq];
        } else {
          pe = lp[t / nq];
          qe = lq[t % nq];
        }
        double2 P1 = __ldg(pv + pe), P2 = __ldg(pv + (pe + 1 < np_ ? pe + 1 : 0));
        double2 Q1 = __ldg(qv + qe), Q2 = __ldg(qv + (qe + 1 < nq_ ? qe + 1 : 0));
        if (edge_boxes_touch(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y)) {
          if (!kExact) {
            bool qhit;
            tp = classify_edges_both(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y, eps, alpha, beta, qhit);
            tq = qhit ? 1 : 0;
          } else {
            bool qhit;
            tp = classify_exact_both(P1, P2, Q1, Q2, alpha, beta, qhit);
            tq = qhit ? 1 : 0;
          }
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, tp != 0);
      if (tp != 0) {
        const int i = wib * kChunk + recs + __popc(m & lanemask_lt());
        sP[i] = pe; sQ[i] = qe; sA[i] = alpha; sB[i] = beta; sT[i] = (int8_t)tp;
      }
      recs += __popc(m);
      qhits += __popc(__ballot_sync(0xffffffffu, tq != 0));
    }
  }
  if (lane_id() == 0 && k >= 0 && F.pairRec) {
    if (recs) atomicAdd(&F.pairRec[k], recs);
    if (qhits) atomicAdd(&F.pairQ[k], qhits);
  }
  if (kWarpAppend) {                                // each warp takes its own range
    unsigned long long b = 0;
    if (lane_id() == 0 && recs) b = atomicAdd(F.total, (unsigned long long)recs);
    const int64_t base = (int64_t)__shfl_sync(0xffffffffu, b, 0);
    __syncwarp();
    for (int j = lane_id(); j < recs; j += 32) {
      const int i = wib * kChunk + j;
      const int64_t r = base + j;
      if (r < F.cap) { R.p[r] = sP[i]; R.q[r] = sQ[i]; R.a[r] = sA[i]; R.b[r] = sB[i]; R.t[r] = sT[i]; R.k[r] = (int32_t)k; }
    }
    return;
  }
  if (lane_id() == 0) { sOff[wib] = recs; sK[wib] = (int32_t)k; }
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int w = 0; w < kWarps; ++w) { const int n = sOff[w]; sOff[w] = run; run += n; }
    sOff[kWarps] = run;
    sBase = run ? atomicAdd(F.total, (unsigned long long)run) : 0ull;
  }
  __syncthreads();
  const int n = sOff[kWarps];
  const int64_t base = (int64_t)sBase;
  for (int j = threadIdx.x; j < n; j += kThreads) {
    int w = 0;
    while (w + 1 < kWarps && sOff[w + 1] <= j) ++w;
    const int i = w * kChunk + (j - sOff[w]);
    const int64_t r = base + j;
    if (r < F.cap) { R.p[r] = sP[i]; R.q[r] = sQ[i]; R.a[r] = sA[i]; R.b[r] = sB[i]; R.t[r] = sT[i]; R.k[r] = sK[w]; }
  }
}

// per pair: record count (chunked + binned), validity
__global__ void pair_records_kernel(const int64_t* __restrict__ chunkOff, const int64_t* __restrict__ nchunk,
                                    const int64_t* __restrict__ recScan, const int64_t* __restrict__ qScan,
                                    const int32_t* __restrict__ chunkRec, const int32_t* __restrict__ chunkQ,
                                    const int64_t* __restrict__ binRec, const int64_t* __restrict__ binQ,
                                    int64_t K, int64_t* __restrict__ nrec64, int32_t* __restrict__ nrec,
                                    int64_t* __restrict__ count1, PairDev D,
                                    const int32_t* __restrict__ pairRec, const int32_t* __restrict__ pairQ) {
  int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k >= K) return;
  int64_t c0 = chunkOff[k], n = nchunk[k];
  int64_t r = binRec[k], q = binQ[k];
  if (pairRec) {                                   // the fused pass counted per pair
    r += pairRec[k];
    q += pairQ[k];
  } else if (n > 0) {
    r += recScan[c0 + n - 1] + chunkRec[c0 + n - 1] - recScan[c0];
    q += qScan[c0 + n - 1] + chunkQ[c0 + n - 1] - qScan[c0];
  }
  nrec64[k] = r;
  nrec[k] = (int32_t)r;
  count1[k] = r;
  if (D.status[k] == 0 && r != q) D.status[k] = 1;   // gppolyclip_mDIV512.cu:1461
}

// ---------------------------------------------------------------- G2/G3 binned
// Pairs whose filtered edge grid exceeds ClipParams::bin_grid edge pairs are not
// enumerated edge pair by edge pair.  Each gets a uniform grid over its common MBR
// (about one Q edge per cell); its Q edges are listed in every cell their box covers;
// each P edge visits the cells its box covers and tests a Q edge only in the cell holding
// the lower-left corner of the two boxes' overlap, so every edge pair whose boxes touch
// is tested exactly once (cell indices are monotone in the coordinate).  All binned pairs
// go through the same launches: their P and Q edges are numbered consecutively (pair by
// pair) and each edge finds its pair through an owner table.
struct BinGrid { double x0, y0, cw, ch; int gx, gy; float M; };   // M: range of the FP32 copies

__device__ __forceinline__ int cell_1d(double v, double c0, double cs, int g) {
  double t = (v - c0) / cs;
  if (!(t > 0)) return 0;             // also NaN
  if (t >= (double)g) return g - 1;
  return (int)t;
}

// The binned pairs, i = 0..B-1 (pair k = list[i]).
struct BinSet {
  const int64_t* list;
  int32_t* cp; int32_t* cq;           // filtered edges per side
  int64_t* pBase; int64_t* qBase;     // first binned P / Q edge of pair i
  int32_t* ownP; int32_t* ownQ;       // binned edge -> i
  double* ext;                        // per pair: sums of the Q edges' box widths, heights
  BinGrid* grid;
  int64_t* cellBase;                  // first cell of pair i (cells of all pairs in one array)
  int32_t* ncell;
};

__global__ void bin_sizes_kernel(BinSet S, int n, const int32_t* __restrict__ cP, const int32_t* __restrict__ cQ) {
  int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const int64_t k = S.list[i];
  S.cp[i] = cP[k];
  S.cq[i] = cQ[k];
}

// the pair-local Q (P) edge of binned edge j
__device__ __forceinline__ int binned_q(const BinSet& S, int64_t j, int i, const int64_t* offQ, const int32_t* LQ) {
  return LQ[offQ[S.list[i]] + (j - S.qBase[i])];
}
__device__ __forceinline__ int binned_p(const BinSet& S, int64_t j, int i, const int64_t* offP, const int32_t* LP) {
  return LP[offP[S.list[i]] + (j - S.pBase[i])];
}

// Sums of the Q edges' box widths and heights per pair (they size the cells).  Edges of
// one pair are consecutive, so a warp reduces each run of equal owners and one lane per
// run adds it.
__global__ void bin_extent_kernel(LayerDev Lb, LayerDev Lo, PairDev D, BinSet S, int64_t nq,
                                  const int64_t* __restrict__ offQ, const int32_t* __restrict__ LQ) {
  const int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  int i = -1;
  double w = 0, h = 0;
  if (j < nq) {
    i = S.ownQ[j];
    const int64_t k = S.list[i];
    const double2* qv = layer_xy(Lb, Lo, 1 - D.pSide[k]) + D.qS[k];
    const int n = D.nQ[k];
    const int q = binned_q(S, j, i, offQ, LQ);
    const double2 a = __ldg(qv + q), b = __ldg(qv + (q + 1 < n ? q + 1 : 0));
    w = fabs(b.x - a.x);
    h = fabs(b.y - a.y);
  }
  const int lane = (int)lane_id();
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {          // segmented inclusive scan over equal owners
    const double uw = __shfl_up_sync(0xffffffffu, w, d), uh = __shfl_up_sync(0xffffffffu, h, d);
    const int ui = __shfl_up_sync(0xffffffffu, i, d);
    if (lane >= d && ui == i) { w += uw; h += uh; }
  }
  const int ni = __shfl_down_sync(0xffffffffu, i, 1);
  if (i >= 0 && (lane == 31 || ni != i)) {
    atomicAdd(S.ext + 2 * i, w);
    atomicAdd(S.ext + 2 * i + 1, h);
  }
}

// Grid of each binned pair: about one Q edge per cell, but never cells smaller than half the
// Q edges' mean box (long edges would otherwise be listed in many cells); at most 4096 cells
// per axis.  (Count + emit of the 400,000 x 200,000-vertex pair: 22.4 ms with cells of the
// mean box, 18.6 ms with half, 17.2 ms with a quarter; degenerate batch 10.4, 10.5, 10.8 ms.)
__global__ void bin_grid_kernel(PairDev D, BinSet S, int n) {
  int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const double4 c = reinterpret_cast<const double4*>(D.cmbr)[S.list[i]];
  const double w = c.z - c.x, h = c.w - c.y;
  const double target = (double)max(1, S.cq[i]);
  const double mw = S.ext[2 * i] / target, mh = S.ext[2 * i + 1] / target;
  double gx = 1, gy = 1;
  if (w > 0 && h > 0) {
    gx = ceil(sqrt(target * w / h));
    gx = fmin(fmax(gx, 1.0), 4096.0);
    gy = ceil(target / gx);
    if (mw > 0) gx = fmin(gx, ceil(2.0 * w / mw));
    if (mh > 0) gy = fmin(gy, ceil(2.0 * h / mh));
    gx = fmin(fmax(gx, 1.0), 4096.0);
    gy = fmin(fmax(gy, 1.0), 4096.0);
  } else if (w > 0) {
    gx = fmin(target, 4096.0);
  } else if (h > 0) {
    gy = fmin(target, 4096.0);
  }
  // The FP32 copies' range M.  What the side test's margins leave beside its error bound
  // (2^-45 M^2, bin_f32_rejects) is above what products rounded at FP32's smallest step
  // (2^-149) can lose for M >= 2^-50, and no product overflows up to 2^60.  Other ranges get no
  // copies (a negative M): their edges all go to FP64.
  const double range = 2.0 * fmax(fmax(w, h), 0.0);
  const float M = range >= 0x1p-50 && range <= 0x1p60 ? __double2float_ru(range) : -1.f;
  BinGrid G{c.x, c.y, w > 0 ? w / gx : 1.0, h > 0 ? h / gy : 1.0, (int)gx, (int)gy, M};
  S.grid[i] = G;
  S.ncell[i] = G.gx * G.gy;
}

// A Q edge is listed in every cell its box covers.  Within a cell the listings stand in four
// classes, by whether the cell is in the first column and the first row of the edge's box:
//   0 first column only, 1 both, 2 first row only, 3 neither
// so that a P edge's visits meet each Q edge once, in the cell of their overlap's lower
// left corner, without testing for it: from the corner cell of its own box it takes all
// classes, from the other cells of the first row those of first-column cells (0, 1), from the
// other cells of the first column those of first-row cells (1, 2), elsewhere class 1.
__device__ __forceinline__ int bin_class(bool firstCol, bool firstRow) {
  return firstCol ? (firstRow ? 1 : 0) : (firstRow ? 2 : 3);
}

// The FP32 copy of an edge relative to the grid's corner (four NaNs when it leaves the
// range M, or M is negative: no FP32 test then rejects it).  Each value is within M * 2^-24 of the exact one.
__device__ __forceinline__ float4 bin_edge_f32(double2 a, double2 b, const BinGrid& G) {
  const float4 r = make_float4(__double2float_rn(a.x - G.x0), __double2float_rn(a.y - G.y0),
                               __double2float_rn(b.x - G.x0), __double2float_rn(b.y - G.y0));
  const float m = fmaxf(fmaxf(fabsf(r.x), fabsf(r.y)), fmaxf(fabsf(r.z), fabsf(r.w)));
  const float nan = __int_as_float(0x7fffffff);
  return m <= G.M ? r : make_float4(nan, nan, nan, nan);
}

// kMode 0: count the listings per cell and class; kMode 1: list every Q edge in the cells its
// box covers, with its FP32 copy when cellBox is given
template <int kMode>
__global__ void bin_cells_kernel(LayerDev Lb, LayerDev Lo, PairDev D, BinSet S, int64_t nq,
                                 const int64_t* __restrict__ offQ, const int32_t* __restrict__ LQ,
                                 int32_t* __restrict__ cellCnt, const int64_t* __restrict__ cellOff,
                                 int32_t* __restrict__ cursor, int32_t* __restrict__ cellList,
                                 float4* __restrict__ cellBox) {
  const int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (j >= nq) return;
  const int i = S.ownQ[j];
  const int64_t k = S.list[i];
  const double2* qv = layer_xy(Lb, Lo, 1 - D.pSide[k]) + D.qS[k];
  const int n = D.nQ[k];
  const int q = binned_q(S, j, i, offQ, LQ);
  const double2 a = __ldg(qv + q), b = __ldg(qv + (q + 1 < n ? q + 1 : 0));
  const BinGrid G = S.grid[i];
  const int64_t cb = S.cellBase[i];
  const int x0 = cell_1d(fmin(a.x, b.x), G.x0, G.cw, G.gx), x1 = cell_1d(fmax(a.x, b.x), G.x0, G.cw, G.gx);
  const int y0 = cell_1d(fmin(a.y, b.y), G.y0, G.ch, G.gy), y1 = cell_1d(fmax(a.y, b.y), G.y0, G.ch, G.gy);
  const float4 box = (kMode == 1 && cellBox) ? bin_edge_f32(a, b, G) : make_float4(0.f, 0.f, 0.f, 0.f);
  for (int y = y0; y <= y1; ++y)
    for (int x = x0; x <= x1; ++x) {
      const int64_t c = 4 * (cb + (int64_t)y * G.gx + x) + bin_class(x == x0, y == y0);
      if (kMode == 0) atomicAdd(&cellCnt[c], 1);
      else {
        const int64_t at = cellOff[c] + atomicAdd(&cursor[c], 1);
        cellList[at] = q;
        if (cellBox) cellBox[at] = box;
      }
    }
}

// The record export's two passes over the binned pairs, a thread per P edge.  kMode 0: per
// binned P edge, its records (P side) into recCnt, and the pair's Q-side count into binQ;
// kMode 1: write the records of each P edge at its offset, the pair's recOff plus the edge's
// place in the pair (in cell order: nothing downstream depends on that).
template <int kMode, int kExact>
__global__ void __launch_bounds__(kThreads, kExact ? 2 : 4)
bin_pairs_kernel(LayerDev Lb, LayerDev Lo, PairDev D, BinSet S, int64_t np,
                 const int64_t* __restrict__ offP, const int32_t* __restrict__ LP,
                 const int64_t* __restrict__ cellOff, const int32_t* __restrict__ cellList, double eps,
                 int32_t* __restrict__ recCnt, int64_t* __restrict__ binQ,
                 const int64_t* __restrict__ recPos, const int64_t* __restrict__ recOff, Records R) {
  const int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (j >= np) return;
  const int i = S.ownP[j];
  const int64_t k = S.list[i];
  const int pside = D.pSide[k];
  const double2* pv = layer_xy(Lb, Lo, pside) + D.pS[k];
  const double2* qv = layer_xy(Lb, Lo, 1 - pside) + D.qS[k];
  const int np_ = D.nP[k], nq = D.nQ[k];
  const int p = binned_p(S, j, i, offP, LP);
  const double2 P1 = __ldg(pv + p), P2 = __ldg(pv + (p + 1 < np_ ? p + 1 : 0));
  const double pminx = fmin(P1.x, P2.x), pmaxx = fmax(P1.x, P2.x);
  const double pminy = fmin(P1.y, P2.y), pmaxy = fmax(P1.y, P2.y);
  const BinGrid G = S.grid[i];
  const int64_t cb = S.cellBase[i];
  const int x0 = cell_1d(pminx, G.x0, G.cw, G.gx), x1 = cell_1d(pmaxx, G.x0, G.cw, G.gx);
  const int y0 = cell_1d(pminy, G.y0, G.ch, G.gy), y1 = cell_1d(pmaxy, G.y0, G.ch, G.gy);
  int recs = 0, qhits = 0;
  const int64_t base = (kMode == 0) ? 0 : recOff[k] + recPos[j] - recPos[S.pBase[i]];
  for (int y = y0; y <= y1; ++y)
    for (int x = x0; x <= x1; ++x) {
      const int64_t c = 4 * (cb + (int64_t)y * G.gx + x);
      const int64_t e1 = cellOff[c + (y == y0 ? (x == x0 ? 4 : 2) : (x == x0 ? 3 : 2))];
      for (int64_t e = cellOff[c + (y == y0 ? 0 : 1)]; e < e1; ++e) {
        const int q = cellList[e];
        const double2 Q1 = __ldg(qv + q), Q2 = __ldg(qv + (q + 1 < nq ? q + 1 : 0));
        if (!edge_boxes_touch(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y)) continue;
        double alpha = 0, beta = 0;
        const int tp = classify_mode(kExact, P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y, eps, alpha, beta);
        if (kMode == 0) {
          double a2, b2;
          if (classify_mode(kExact, Q1.x, Q1.y, Q2.x, Q2.y, P1.x, P1.y, P2.x, P2.y, eps, a2, b2)) ++qhits;
          if (tp) ++recs;
        } else if (tp) {
          const int64_t r = base + recs++;
          R.p[r] = p; R.q[r] = q; R.a[r] = alpha; R.b[r] = beta; R.t[r] = (int8_t)tp; R.k[r] = (int32_t)k;
        }
      }
    }
  if (kMode == 0) {
    recCnt[j] = recs;
    if (qhits) atomicAdd(reinterpret_cast<unsigned long long*>(binQ + k), (unsigned long long)qhits);
  }
}

// Whether two edges that meet may be rejected on their FP32 copies: true only when the exact
// boxes are apart, or (exact predicates) both ends of one edge lie strictly on one side
// of the other, the sign tests having room for the copies' and the arithmetic's rounding.
// With d = M 2^-24 the copies' error, A and B the 1-norms of the two differences that an
// area is the cross product of (each at most 4 M), the area's error is below
// 2 d (A + B) + 4 d min(A, B) + 8 d^2 + 4 2^-24 A B < 24 d (A + B + d); 32 is used.  The rest,
// 8 d (A + B + d) >= 2^-45 M^2, covers underflow for the M that have copies (bin_grid_kernel).
template <int kExact>
__device__ __forceinline__ bool bin_f32_rejects(float4 p, float4 q, float M) {
  const float slop = M * 2.3841858e-7f;                                  // 2^-22
  if (fminf(q.x, q.z) > fmaxf(p.x, p.z) + slop || fmaxf(q.x, q.z) < fminf(p.x, p.z) - slop) return true;
  if (fminf(q.y, q.w) > fmaxf(p.y, p.w) + slop || fmaxf(q.y, q.w) < fminf(p.y, p.w) - slop) return true;
  if (!kExact) return false;
  const float d = M * 1.9073486e-6f;                                     // 32 * 2^-24 M
  const float px = p.z - p.x, py = p.w - p.y, qx = q.z - q.x, qy = q.w - q.y;
  // An edge of no length is collinear with everything (classify_exact's second branch goes
  // by projections alone); copies that differ show that the ends do.
  if ((px == 0.f && py == 0.f) || (qx == 0.f && qy == 0.f)) return false;
  const float ax = q.x - p.x, ay = q.y - p.y;                            // P1 -> Q1
  const float bx = q.z - p.x, by = q.w - p.y;                            // P1 -> Q2
  const float cx = q.x - p.z, cy = q.y - p.w;                            // P2 -> Q1
  const float A = fabsf(px) + fabsf(py) + M * 5.9604645e-8f, B = fabsf(qx) + fabsf(qy) + M * 5.9604645e-8f;
  const float s1 = px * ay - py * ax, s2 = px * by - py * bx;            // Q1, Q2 beside P
  const float e1 = d * (A + fabsf(ax) + fabsf(ay)), e2 = d * (A + fabsf(bx) + fabsf(by));
  if ((s1 > e1 && s2 > e2) || (s1 < -e1 && s2 < -e2)) return true;
  const float t1 = qx * ay - qy * ax, t2 = qx * cy - qy * cx;            // P1, P2 beside Q (sign of both flipped)
  const float f1 = d * (B + fabsf(ax) + fabsf(ay)), f2 = d * (B + fabsf(cx) + fabsf(cy));
  return (t1 > f1 && t2 > f2) || (t1 < -f1 && t2 < -f2);
}

// Count and emit of the binned pairs in one pass, a warp per kBinEdges consecutive P edges.
// The listings of a P edge's cells are taken as one run, 32 at a time (the cells' shares
// by a scan, so that many small cells fill the lanes as well as one large one), tested on
// their FP32 copies with coalesced loads, and the few that pass are queued in shared
// memory until 32 of them can be classified in FP64 by a full warp.  The records go to a
// range of the global counter taken per classified group, as in intersect_fused_kernel.
// Bound by instruction issue.  A thread per P edge enumerating its listings in FP64, once to
// count and once to emit, took 271 ms for the 400,000 x 200,000-vertex pair (2.9e7
// records) and 31.3 ms for the degenerate batch of 10,007 pairs (2.3e7), this 14.1 and 9.2 ms.
// (3 blocks per SM at 80 registers: 22.4 ms against 27.2 ms for 2 at 128, cells of the mean box.)
// kBoxes 0: there are no copies (kMaxBoxes), every listing is classified.
constexpr int kBinEdges = 8;

// Listings up to which the FP32 copies are made: 16 bytes each beside the 4 of the listing, 8.6 GB
// here.  A ring of n edges with about sqrt(n) of them as long as the ring has up to 2 n sqrt(n)
// listings, which with copies would not fit the GPU from 3e6 edges on.
constexpr int64_t kMaxBoxes = 1ll << 29;

template <int kExact, int kBoxes>
__global__ void __launch_bounds__(kThreads, 3)
bin_append_kernel(LayerDev Lb, LayerDev Lo, PairDev D, BinSet S, int64_t np,
                  const int64_t* __restrict__ offP, const int32_t* __restrict__ LP,
                  const int64_t* __restrict__ cellOff, const int32_t* __restrict__ cellList,
                  const float4* __restrict__ cellBox, double eps, Records R, FusedRecords F,
                  unsigned long long* __restrict__ binRec, unsigned long long* __restrict__ binQ) {
  __shared__ int2 queue[kWarpsPerBlock][64];
  int2* const wq = queue[threadIdx.x >> 5];
  const int lane = (int)lane_id();
  const int64_t j0 = (((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5) * kBinEdges;
  const int64_t j1 = min(j0 + kBinEdges, np);
  int cur = -1, queued = 0, np_ = 0, nq = 0;
  int64_t k = 0;
  unsigned recs = 0, qhits = 0;
  const double2* pv = nullptr;
  const double2* qv = nullptr;
  BinGrid G{};
  int64_t cb = 0;
  // classifies the queue's last n entries
  auto classify = [&](int n) {
    int tp = 0, pe = 0, qe = 0;
    bool tq = false;
    double alpha = 0, beta = 0;
    __syncwarp();
    if (lane < n) {
      const int2 pq = wq[queued - n + lane];
      pe = pq.x;
      qe = pq.y;
      const double2 P1 = __ldg(pv + pe), P2 = __ldg(pv + (pe + 1 < np_ ? pe + 1 : 0));
      const double2 Q1 = __ldg(qv + qe), Q2 = __ldg(qv + (qe + 1 < nq ? qe + 1 : 0));
      if (edge_boxes_touch(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y)) {
        if (kExact) tp = classify_exact_both(P1, P2, Q1, Q2, alpha, beta, tq);
        else tp = classify_edges_both(P1.x, P1.y, P2.x, P2.y, Q1.x, Q1.y, Q2.x, Q2.y, eps, alpha, beta, tq);
      }
    }
    __syncwarp();
    queued -= n;
    const unsigned m = __ballot_sync(0xffffffffu, tp != 0);
    recs += __popc(m);
    qhits += __popc(__ballot_sync(0xffffffffu, tq));
    if (m) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(F.total, (unsigned long long)__popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      const int64_t r = (int64_t)base + __popc(m & lanemask_lt());
      if (tp != 0 && r < F.cap) {
        R.p[r] = pe; R.q[r] = qe; R.a[r] = alpha; R.b[r] = beta; R.t[r] = (int8_t)tp; R.k[r] = (int32_t)k;
      }
    }
  };
  auto finish_pair = [&]() {
    if (queued) classify(queued);
    if (lane == 0 && binRec) {
      if (recs) atomicAdd(binRec + k, (unsigned long long)recs);
      if (qhits) atomicAdd(binQ + k, (unsigned long long)qhits);
    }
    recs = qhits = 0;
  };
  for (int64_t j = j0; j < j1; ++j) {
    const int i = S.ownP[j];
    if (i != cur) {
      if (cur >= 0) finish_pair();
      cur = i;
      k = S.list[i];
      const int pside = D.pSide[k];
      pv = layer_xy(Lb, Lo, pside) + D.pS[k];
      qv = layer_xy(Lb, Lo, 1 - pside) + D.qS[k];
      np_ = D.nP[k];
      nq = D.nQ[k];
      G = S.grid[i];
      cb = S.cellBase[i];
    }
    const int p = binned_p(S, j, i, offP, LP);
    const double2 P1 = __ldg(pv + p), P2 = __ldg(pv + (p + 1 < np_ ? p + 1 : 0));
    const float4 pf = bin_edge_f32(P1, P2, G);
    const int x0 = cell_1d(fmin(P1.x, P2.x), G.x0, G.cw, G.gx), x1 = cell_1d(fmax(P1.x, P2.x), G.x0, G.cw, G.gx);
    const int y0 = cell_1d(fmin(P1.y, P2.y), G.y0, G.ch, G.gy), y1 = cell_1d(fmax(P1.y, P2.y), G.y0, G.ch, G.gy);
    const int wx = x1 - x0 + 1, cells = wx * (y1 - y0 + 1);
    for (int c0 = 0; c0 < cells; c0 += 32) {
      int64_t from = 0;
      int len = 0;
      if (c0 + lane < cells) {
        const int cy = (c0 + lane) / wx, cx = (c0 + lane) - cy * wx;
        const int64_t c = 4 * (cb + (int64_t)(y0 + cy) * G.gx + x0 + cx);
        from = cellOff[c + (cy == 0 ? 0 : 1)];
        len = (int)(cellOff[c + (cy == 0 ? (cx == 0 ? 4 : 2) : (cx == 0 ? 3 : 2))] - from);
      }
      const int incl = warp_incl_scan(len);
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      from -= incl - len;                                // listing of flat index t: from + t
      for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        int lo = 0;                                      // the cell: shares whose scan is <= t
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
          const int v = __shfl_sync(0xffffffffu, incl, lo + w - 1);
          if (v <= t) lo += w;
        }
        const int64_t e = __shfl_sync(0xffffffffu, from, lo & 31) + t;
        bool keep = false;
        if (t < total) keep = !kBoxes || !bin_f32_rejects<kExact>(pf, __ldg(cellBox + e), G.M);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) wq[queued + __popc(m & lanemask_lt())] = make_int2(p, cellList[e]);
        queued += __popc(m);
        if (queued >= 32) classify(32);
      }
    }
  }
  if (cur >= 0) finish_pair();
}

// per binned pair: its records (the P edges' counts summed through their scan)
__global__ void bin_rec_total_kernel(BinSet S, int n, const int64_t* __restrict__ recPos,
                                     int64_t* __restrict__ binRec) {
  int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const int64_t b = S.pBase[i];
  binRec[S.list[i]] = recPos[b + S.cp[i]] - recPos[b];
}

// ---------------------------------------------------------------- G4 ring layout
// Per record: insertion counts per edge, and the winning (last) record for each source
// vertex that records link (P: types 2,4,5,6,8; Q: types 3,4,5,7,8).
// "Last record wins" in the reference's loop order (P edge outer, Q edge inner) is the
// record with the largest other-side edge, so the winner is the maximum of
// (other edge, record index): independent of the order records were emitted in.
constexpr int kLinkKeyShift = 33;             // record indices below 2^33
__device__ __forceinline__ unsigned long long link_key(int other, int64_t r) {
  return (((unsigned long long)other << kLinkKeyShift) | (unsigned long long)r) + 1ull;
}

__global__ void record_count_kernel(Records R, int64_t nR, const int64_t* __restrict__ eoffP,
                                    const int64_t* __restrict__ eoffQ, const int32_t* __restrict__ status,
                                    int32_t* __restrict__ insP, int32_t* __restrict__ insQ,
                                    int64_t* __restrict__ srcLinkP, int64_t* __restrict__ srcLinkQ) {
  int64_t r = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (r >= nR) return;
  int k = R.k[r];
  if (status[k] != 0) return;
  int t = R.t[r];
  int64_t eP = eoffP[k] + R.p[r], eQ = eoffQ[k] + R.q[r];
  if (t == 1 || t == 3 || t == 5 || t == 7) atomicAdd(&insP[eP], 1);
  if (t == 1 || t == 2 || t == 5 || t == 6) atomicAdd(&insQ[eQ], 1);
  if (t == 2 || t == 4 || t == 5 || t == 6 || t == 8)
    atomicMax(reinterpret_cast<unsigned long long*>(&srcLinkP[eP]), link_key(R.q[r], r));
  if (t == 3 || t == 4 || t == 5 || t == 7 || t == 8)
    atomicMax(reinterpret_cast<unsigned long long*>(&srcLinkQ[eQ]), link_key(R.p[r], r));
}

// slot of each edge's source vertex in the concatenated merged rings: the exclusive scan
// of (1 + insertions) over the edges, i.e. the edge index plus the scan of the insertions
// (both sides in one launch, as in pair_ring_kernel: blockIdx.y)
__global__ void edge_slots_kernel(const int64_t* __restrict__ insP, int64_t nEP, int64_t* __restrict__ vposP,
                                  const int64_t* __restrict__ insQ, int64_t nEQ, int64_t* __restrict__ vposQ) {
  int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (blockIdx.y == 0) { if (e < nEP) vposP[e] = e + insP[e]; }
  else if (e < nEQ) vposQ[e] = e + insQ[e];
}

// The merged rings of one side live in one buffer of n slots, column by column:
//   xy (double2) | nx pv nb (int32) | tn tl to ls (int32) | it lb ee fl (byte)
// 48 bytes per slot.  A ring is then the buffer, n and its first slot: a thread that
// walks a pair keeps three words per ring instead of a pointer per column, and each
// column stays dense for the scans over one field.
//   nx, pv, nb  next, previous, neighbour (slot on the other ring, -1 none)
//   tn tl to ls scratch of the trace and the clean-up
//   it          intersection flag (cleared when visited by the trace)
//   lb, ee      IntersectionLabel, EntryExitLabel
//   fl          bit0 split candidate, bit1 crossing candidate
#define GCMFGH_RING_COLUMNS(IDX)                                                                   \
  __device__ __forceinline__ double2& xy(int64_t i) const { return reinterpret_cast<double2*>(b)[IDX]; } \
  __device__ __forceinline__ double& x(int64_t i) const { return xy(i).x; }                         \
  __device__ __forceinline__ double& y(int64_t i) const { return xy(i).y; }                         \
  __device__ __forceinline__ int32_t& nx(int64_t i) const { return reinterpret_cast<int32_t*>(b + 16 * n)[IDX]; } \
  __device__ __forceinline__ int32_t& pv(int64_t i) const { return reinterpret_cast<int32_t*>(b + 20 * n)[IDX]; } \
  __device__ __forceinline__ int32_t& nb(int64_t i) const { return reinterpret_cast<int32_t*>(b + 24 * n)[IDX]; } \
  __device__ __forceinline__ int32_t& tn(int64_t i) const { return reinterpret_cast<int32_t*>(b + 28 * n)[IDX]; } \
  __device__ __forceinline__ int32_t& tl(int64_t i) const { return reinterpret_cast<int32_t*>(b + 32 * n)[IDX]; } \
  __device__ __forceinline__ int32_t& to(int64_t i) const { return reinterpret_cast<int32_t*>(b + 36 * n)[IDX]; } \
  __device__ __forceinline__ int32_t& ls(int64_t i) const { return reinterpret_cast<int32_t*>(b + 40 * n)[IDX]; } \
  __device__ __forceinline__ uint8_t& it(int64_t i) const { return reinterpret_cast<uint8_t*>(b + 44 * n)[IDX]; } \
  __device__ __forceinline__ int8_t& lb(int64_t i) const { return reinterpret_cast<int8_t*>(b + 45 * n)[IDX]; } \
  __device__ __forceinline__ int8_t& ee(int64_t i) const { return reinterpret_cast<int8_t*>(b + 46 * n)[IDX]; } \
  __device__ __forceinline__ uint8_t& fl(int64_t i) const { return reinterpret_cast<uint8_t*>(b + 47 * n)[IDX]; }

constexpr int64_t kRingSlotBytes = 48;

// Kernels that take a RingSet by value keep its column pointers in the parameter space,
// so the side-wide kernels (fill, links, export, grid path) index columns directly.
struct RingSet {
  char* b;          // column buffer
  int64_t n;        // slots per column (a multiple of 16, so every column stays aligned)
  int exact;        // orientation signs exact (ClipParams::exact)
  double2* cxy; int32_t* cnx; int32_t* cpv; int32_t* cnb;
  uint8_t* cit; int8_t* clb; int8_t* cee; uint8_t* cfl;
  void set(char* buf, int64_t slots) {
    b = buf; n = slots;
    cxy = reinterpret_cast<double2*>(b);
    cnx = reinterpret_cast<int32_t*>(b + 16 * n); cpv = reinterpret_cast<int32_t*>(b + 20 * n);
    cnb = reinterpret_cast<int32_t*>(b + 24 * n); cit = reinterpret_cast<uint8_t*>(b + 44 * n);
    clb = reinterpret_cast<int8_t*>(b + 45 * n); cee = reinterpret_cast<int8_t*>(b + 46 * n);
    cfl = reinterpret_cast<uint8_t*>(b + 47 * n);
  }
  __device__ __forceinline__ double& x(int64_t i) const { return cxy[i].x; }
  __device__ __forceinline__ double& y(int64_t i) const { return cxy[i].y; }
  __device__ __forceinline__ int32_t& nx(int64_t i) const { return cnx[i]; }
  __device__ __forceinline__ int32_t& pv(int64_t i) const { return cpv[i]; }
  __device__ __forceinline__ int32_t& nb(int64_t i) const { return cnb[i]; }
  __device__ __forceinline__ uint8_t& it(int64_t i) const { return cit[i]; }
  __device__ __forceinline__ int8_t& lb(int64_t i) const { return clb[i]; }
  __device__ __forceinline__ int8_t& ee(int64_t i) const { return cee[i]; }
  __device__ __forceinline__ uint8_t& fl(int64_t i) const { return cfl[i]; }
};

// per pair: ring size, region offset (ring + room for added vertices)
struct RingSide {
  const int64_t* eoff; const int64_t* vpos; const int32_t* n;
  int64_t nE;
  const int64_t* insTot;
  int32_t* m; int64_t* regSize;
};
__global__ void pair_ring_kernel(RingSide sideP, RingSide sideQ, const int32_t* __restrict__ nrec,
                                 const int32_t* __restrict__ status, int64_t K,
                                 unsigned long long* __restrict__ ringTot) {
  const RingSide& S = blockIdx.y == 0 ? sideP : sideQ;
  const int64_t* eoff = S.eoff;
  const int64_t* vpos = S.vpos;
  const int32_t* n = S.n;
  const int64_t nE = S.nE;
  const int64_t* insTot = S.insTot;
  int32_t* m = S.m;
  int64_t* regSize = S.regSize;
  int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  unsigned long long mm = 0;
  if (k < K) {
    const int64_t vtot = nE + *insTot;                      // slots of the side's merged rings
    int64_t e0 = eoff[k], e1 = e0 + (status[k] == 2 ? 0 : n[k]);
    int64_t v0 = e0 < nE ? vpos[e0] : vtot, v1 = e1 < nE ? vpos[e1] : vtot;
    mm = status[k] == 0 ? (unsigned long long)(v1 - v0) : 0ull;
    m[k] = (int)mm;
    regSize[k] = status[k] == 0 ? (int64_t)mm + 2 + 2 * (int64_t)nrec[k] : 0;
  }
  mm = warp_sum(mm);                                        // merged-ring vertices, all pairs
  if (lane_id() == 0 && mm) atomicAdd(ringTot, mm);
}

// ---------------------------------------------------------------- G5 ring fill
// Thread per edge: the edge's source vertex, then its inserted vertices sorted by
// (parameter ascending, other edge descending).  side 0 fills P rings, side 1 Q rings.
// An edge of the smaller polygon can cross thousands of edges of a large one: edges with
// more than kLightEdge insertions are listed for mid_fill_kernel (a warp each), those with more than
// kMidEdge for heavy_fill_kernel (a block each).
constexpr int kLightEdge = 8;
constexpr int kMidEdge = 256;

struct EdgeFill {
  int64_t k, base;
  int s0, mm, np_;
  const double2* pvx;
  const double2* qvx;
};

template <int kSide>
__device__ __forceinline__ void write_inserted(const EdgeFill& f, const Records& R, int64_t r, int i,
                                               RingSet& S, int64_t* slotOfRec) {
  int t = R.t[r];
  double X, Y;
  if (t == 1) {
    // I = (1-alpha) P1 + alpha P2 (gppolyclip_mDIV512.cu:1029, polyclip.h:220)
    int pe = R.p[r];
    double a = R.a[r];
    double2 P1 = __ldg(f.pvx + pe), P2 = __ldg(f.pvx + (pe + 1 < f.np_ ? pe + 1 : 0));
    X = (1.0 - a) * P1.x + a * P2.x;
    Y = (1.0 - a) * P1.y + a * P2.y;
  } else if (kSide == 0) {          // types 3, 5, 7: a copy of Q1 on P
    double2 Q1 = __ldg(f.qvx + R.q[r]);
    X = Q1.x; Y = Q1.y;
  } else {                          // types 2, 5, 6: a copy of P1 on Q
    double2 P1 = __ldg(f.pvx + R.p[r]);
    X = P1.x; Y = P1.y;
  }
  int sl = f.s0 + 1 + i;
  int64_t gs = f.base + sl;
  S.x(gs) = X; S.y(gs) = Y;
  S.nx(gs) = (sl + 1) % f.mm; S.pv(gs) = (sl + f.mm - 1) % f.mm; S.nb(gs) = -1;
  S.it(gs) = 0; S.lb(gs) = L_NONE; S.ee(gs) = E_NEITHER; S.fl(gs) = 0;
  slotOfRec[r] = sl;
}

template <int kSide>
__device__ __forceinline__ bool edge_fill_info(const LayerDev& Lb, const LayerDev& Lo, const PairDev& D,
                                               const int64_t* eoff, const int32_t* edgePair, const int64_t* vpos,
                                               const int64_t* regOff, const int32_t* m, int64_t e, EdgeFill& f) {
  const int64_t k = edgePair[e];
  if (D.status[k] != 0) return false;
  const int n = kSide == 0 ? D.nP[k] : D.nQ[k];
  if ((int)(e - eoff[k]) >= n) return false;
  const int pside = D.pSide[k];
  f.k = k;
  f.mm = m[k];
  f.base = regOff[k];
  f.s0 = (int)(vpos[e] - vpos[eoff[k]]);
  f.pvx = layer_xy(Lb, Lo, pside) + D.pS[k];
  f.qvx = layer_xy(Lb, Lo, 1 - pside) + D.qS[k];
  f.np_ = D.nP[k];
  return true;
}

// At most 64 registers (4 blocks per SM): the kernel is latency-bound and the extra
// occupancy outweighs a few spilled values (measured 1.35 -> 1.03 ms for the fill stage).
template <int kSide>
__global__ void __launch_bounds__(kThreads, 4) ring_fill_kernel(LayerDev Lb, LayerDev Lo, PairDev D, Records R,
                                 const int64_t* __restrict__ eoff, int64_t nE, const int32_t* __restrict__ edgePair,
                                 const int64_t* __restrict__ vpos, const int64_t* __restrict__ regOff,
                                 const int32_t* __restrict__ m, RingSet S, int64_t* __restrict__ slotOfRec,
                                 const int64_t* __restrict__ insCursorBase, int32_t* __restrict__ insCursor,
                                 const int64_t* __restrict__ insList, int64_t* __restrict__ heavy,
                                 unsigned long long* __restrict__ nHeavy) {
  // heavy: the mid edges from the front (nHeavy[1]), the heavy ones from the back (nHeavy[0])
  int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (e >= nE) return;
  EdgeFill f;
  if (!edge_fill_info<kSide>(Lb, Lo, D, eoff, edgePair, vpos, regOff, m, e, f)) return;
  const int le = (int)(e - eoff[f.k]);
  const double2 A = __ldg((kSide == 0 ? f.pvx : f.qvx) + le);
  const int64_t g = f.base + f.s0;
  S.x(g) = A.x; S.y(g) = A.y;
  S.nx(g) = (f.s0 + 1) % f.mm; S.pv(g) = (f.s0 + f.mm - 1) % f.mm; S.nb(g) = -1;
  S.it(g) = 0; S.lb(g) = L_NONE; S.ee(g) = E_NEITHER; S.fl(g) = 0;
  // inserted records of this edge, gathered by record_scatter_kernel into insList
  const int64_t l0 = insCursorBase[e];
  const int cnt = insCursor[e];
  if (cnt > kLightEdge) {
    if (cnt > kMidEdge) heavy[nE - 1 - (int64_t)atomicAdd(nHeavy, 1ull)] = e;
    else heavy[atomicAdd(nHeavy + 1, 1ull)] = e;
    return;
  }
  // insertion sort of the (few) records by (parameter asc, other edge desc)
  int64_t* lst = const_cast<int64_t*>(insList) + l0;
  for (int i = 1; i < cnt; ++i) {
    int64_t r = lst[i];
    double key = kSide == 0 ? R.a[r] : R.b[r];
    int oth = kSide == 0 ? R.q[r] : R.p[r];
    int j = i - 1;
    while (j >= 0) {
      int64_t rj = lst[j];
      double kj = kSide == 0 ? R.a[rj] : R.b[rj];
      int oj = kSide == 0 ? R.q[rj] : R.p[rj];
      bool after = (kj > key) || (kj == key && oj < oth);
      if (!after) break;
      lst[j + 1] = rj;
      --j;
    }
    lst[j + 1] = r;
  }
  for (int i = 0; i < cnt; ++i) write_inserted<kSide>(f, R, lst[i], i, S, slotOfRec);
}

// Sort key of an insertion's parameter: both zeros are one parameter (a crossing's parameter
// rounds to -0.0 or +0.0 by the other edge's direction), as ring_fill_kernel compares them.
__device__ __forceinline__ uint64_t param_key(double v) { return ordered_key(v + 0.0); }

// A warp per mid edge: the records' (parameter bits, ~other edge) sorted in the warp's part of
// shared memory, up to 32 by counting each record's predecessors with shuffles, more with
// a bitonic network; then the vertices are written in order.  A block per edge beyond 32
// insertions (512 threads over 64 elements, a barrier per step) took 2.8 of the fill's 4.0 ms on
// 2,500 degenerate pairs, and most of 16 ms on the large pair, whose edges all have 70 to 140.
// The bound of kMidEdge is its shared memory, 14 bytes an element for every warp: with 512 (28
// KB a block, all of an SM's at 8 blocks) four contexts on alternate steps of the batched join
// took 5.66 ms a step, with 256 5.53, the L1 that their other kernels use being left to them;
// 10,007 degenerate pairs 31.3 -> 29.4 ms, the large pair 48.7 -> 47.0.  With 128 the step takes 5.52,
// the large pair 49.8 ms.
constexpr int kMidThreads = 128;

template <int kSide>
__global__ void __launch_bounds__(kMidThreads)
mid_fill_kernel(LayerDev Lb, LayerDev Lo, PairDev D, Records R, const int64_t* __restrict__ eoff,
                const int32_t* __restrict__ edgePair,
                const int64_t* __restrict__ vpos, const int64_t* __restrict__ regOff,
                const int32_t* __restrict__ m, RingSet S, int64_t* __restrict__ slotOfRec,
                const int64_t* __restrict__ insCursorBase, const int32_t* __restrict__ insCursor,
                const int64_t* __restrict__ insList, const int64_t* __restrict__ mid,
                const unsigned long long* __restrict__ nMid) {
  __shared__ uint64_t skey[kMidThreads / 32][kMidEdge];
  __shared__ uint32_t stie[kMidThreads / 32][kMidEdge];
  __shared__ uint16_t sidx[kMidThreads / 32][kMidEdge];
  const int lane = (int)lane_id(), warp = (int)(threadIdx.x >> 5);
  uint64_t* key = skey[warp];
  uint32_t* tie = stie[warp];
  uint16_t* idx = sidx[warp];
  const unsigned long long n = *nMid;
  for (unsigned long long h = (unsigned long long)blockIdx.x * (kMidThreads / 32) + warp; h < n;
       h += (unsigned long long)gridDim.x * (kMidThreads / 32)) {
    const int64_t e = mid[h];
    EdgeFill f;
    edge_fill_info<kSide>(Lb, Lo, D, eoff, edgePair, vpos, regOff, m, e, f);
    const int64_t l0 = insCursorBase[e];
    const int cnt = insCursor[e];
    if (cnt <= 32) {
      int64_t r = 0;
      uint64_t k = ~0ull;
      uint32_t t = ~0u;
      if (lane < cnt) {
        r = insList[l0 + lane];
        k = param_key(kSide == 0 ? R.a[r] : R.b[r]);
        t = 0xffffffffu - (uint32_t)(kSide == 0 ? R.q[r] : R.p[r]);
      }
      int rank = 0;
      for (int j = 0; j < cnt; ++j) {
        const uint64_t kj = __shfl_sync(0xffffffffu, k, j);
        const uint32_t tj = __shfl_sync(0xffffffffu, t, j);
        rank += (kj < k || (kj == k && tj < t)) ? 1 : 0;
      }
      if (lane < cnt) write_inserted<kSide>(f, R, r, rank, S, slotOfRec);
      continue;
    }
    int npad = 64;
    while (npad < cnt) npad <<= 1;
    for (int i = lane; i < npad; i += 32) {
      key[i] = ~0ull;
      tie[i] = 0xffffffffu;
      idx[i] = (uint16_t)i;
      if (i < cnt) {
        const int64_t r = insList[l0 + i];
        key[i] = param_key(kSide == 0 ? R.a[r] : R.b[r]);
        tie[i] = 0xffffffffu - (uint32_t)(kSide == 0 ? R.q[r] : R.p[r]);
      }
    }
    __syncwarp();
    for (int size = 2; size <= npad; size <<= 1)
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = lane; i < (npad >> 1); i += 32) {
          const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
          const uint64_t ka = key[lo], kb = key[hi];
          const uint32_t ta = tie[lo], tb = tie[hi];
          if (((ka > kb) || (ka == kb && ta > tb)) == ((lo & size) == 0)) {
            key[lo] = kb; key[hi] = ka;
            tie[lo] = tb; tie[hi] = ta;
            const uint16_t x = idx[lo];
            idx[lo] = idx[hi];
            idx[hi] = x;
          }
        }
        __syncwarp();
      }
    for (int i = lane; i < cnt; i += 32) write_inserted<kSide>(f, R, insList[l0 + idx[i]], i, S, slotOfRec);
    __syncwarp();
  }
}

// Block per heavy edge: bitonic sort of (parameter bits, ~other edge, list position) --
// ascending parameter, descending other edge -- in shared memory up to kHeavySmem
// elements, in a global scratch segment beyond; then the vertices are written in order.
constexpr int kHeavyThreads = 512;
constexpr int kHeavySmem = 4096;

__device__ void bitonic_sort(uint64_t* key, uint32_t* tie, uint32_t* idx, int npad) {
  for (int size = 2; size <= npad; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < (npad >> 1); i += blockDim.x) {
        int lo = 2 * i - (i & (stride - 1));
        int hi = lo + stride;
        bool up = (lo & size) == 0;
        uint64_t ka = key[lo], kb = key[hi];
        uint32_t ta = tie[lo], tb = tie[hi];
        bool gt = (ka > kb) || (ka == kb && ta > tb);
        if (gt == up) {
          key[lo] = kb; key[hi] = ka;
          tie[lo] = tb; tie[hi] = ta;
          uint32_t x = idx[lo]; idx[lo] = idx[hi]; idx[hi] = x;
        }
      }
      __syncthreads();
    }
  }
}

template <int kSide>
__global__ void __launch_bounds__(kHeavyThreads)
heavy_fill_kernel(LayerDev Lb, LayerDev Lo, PairDev D, Records R, const int64_t* __restrict__ eoff,
                  const int32_t* __restrict__ edgePair,
                  const int64_t* __restrict__ vpos, const int64_t* __restrict__ regOff,
                  const int32_t* __restrict__ m, RingSet S, int64_t* __restrict__ slotOfRec,
                  const int64_t* __restrict__ insCursorBase, const int32_t* __restrict__ insCursor,
                  const int64_t* __restrict__ insList, const int64_t* __restrict__ heavy, int64_t nE,
                  const unsigned long long* __restrict__ nHeavy, uint64_t* gkey, uint32_t* gtie, uint32_t* gidx) {
  extern __shared__ unsigned char smem[];
  uint64_t* skey = reinterpret_cast<uint64_t*>(smem);
  uint32_t* stie = reinterpret_cast<uint32_t*>(skey + kHeavySmem);
  uint32_t* sidx = stie + kHeavySmem;
  __shared__ EdgeFill f;
  const unsigned long long nh = *nHeavy;
  for (unsigned long long h = blockIdx.x; h < nh; h += gridDim.x) {
    const int64_t e = heavy[nE - 1 - (int64_t)h];
    if (threadIdx.x == 0) edge_fill_info<kSide>(Lb, Lo, D, eoff, edgePair, vpos, regOff, m, e, f);
    __syncthreads();
    const int64_t l0 = insCursorBase[e];
    const int cnt = insCursor[e];
    int npad = 1;
    while (npad < cnt) npad <<= 1;
    uint64_t* key = skey;
    uint32_t* tie = stie;
    uint32_t* idx = sidx;
    if (npad > kHeavySmem) { key = gkey + 2 * l0; tie = gtie + 2 * l0; idx = gidx + 2 * l0; }
    for (int i = threadIdx.x; i < npad; i += blockDim.x) {
      if (i < cnt) {
        int64_t r = insList[l0 + i];
        key[i] = param_key(kSide == 0 ? R.a[r] : R.b[r]);
        tie[i] = 0xffffffffu - (uint32_t)(kSide == 0 ? R.q[r] : R.p[r]);
        idx[i] = (uint32_t)i;
      } else {
        key[i] = ~0ull; tie[i] = 0xffffffffu; idx[i] = 0xffffffffu;
      }
    }
    __syncthreads();
    bitonic_sort(key, tie, idx, npad);
    for (int i = threadIdx.x; i < cnt; i += blockDim.x)
      write_inserted<kSide>(f, R, insList[l0 + idx[i]], i, S, slotOfRec);
    __syncthreads();
  }
}

// records inserting on an edge -> that edge's list (order fixed later by ring_fill)
__global__ void record_scatter_kernel(Records R, int64_t nR, const int64_t* __restrict__ eoffP,
                                      const int64_t* __restrict__ eoffQ, const int32_t* __restrict__ status,
                                      const int64_t* __restrict__ baseP, int32_t* __restrict__ curP,
                                      int64_t* __restrict__ listP, const int64_t* __restrict__ baseQ,
                                      int32_t* __restrict__ curQ, int64_t* __restrict__ listQ) {
  int64_t r = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (r >= nR) return;
  int k = R.k[r];
  if (status[k] != 0) return;
  int t = R.t[r];
  int64_t eP = eoffP[k] + R.p[r], eQ = eoffQ[k] + R.q[r];
  if (t == 1 || t == 3 || t == 5 || t == 7) listP[baseP[eP] + atomicAdd(&curP[eP], 1)] = r;
  if (t == 1 || t == 2 || t == 5 || t == 6) listQ[baseQ[eQ] + atomicAdd(&curQ[eQ], 1)] = r;
}

// ---------------------------------------------------------------- G6 links
__device__ __forceinline__ void set_link(RingSet& S, int64_t base, int slot, int target) {
  S.nb(base + slot) = target;
  S.it(base + slot) = 1;
}

__global__ void link_kernel(Records R, int64_t nR, const int32_t* __restrict__ status,
                            const int64_t* __restrict__ eoffP, const int64_t* __restrict__ eoffQ,
                            const int64_t* __restrict__ vposP, const int64_t* __restrict__ vposQ,
                            const int64_t* __restrict__ regP, const int64_t* __restrict__ regQ,
                            const int64_t* __restrict__ slotP, const int64_t* __restrict__ slotQ,
                            const int64_t* __restrict__ srcLinkP, const int64_t* __restrict__ srcLinkQ,
                            RingSet SP, RingSet SQ) {
  int64_t r = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (r >= nR) return;
  int k = R.k[r];
  if (status[k] != 0) return;
  int t = R.t[r];
  int64_t eP = eoffP[k] + R.p[r], eQ = eoffQ[k] + R.q[r];
  const int srcP = (int)(vposP[eP] - vposP[eoffP[k]]);
  const int srcQ = (int)(vposQ[eQ] - vposQ[eoffQ[k]]);
  const int64_t bP = regP[k], bQ = regQ[k];
  const bool winP = (unsigned long long)srcLinkP[eP] == link_key(R.q[r], r);
  const bool winQ = (unsigned long long)srcLinkQ[eQ] == link_key(R.p[r], r);
  switch (t) {
    case 1: {
      int sp = (int)slotP[r], sq = (int)slotQ[r];
      set_link(SP, bP, sp, sq); set_link(SQ, bQ, sq, sp);
      break;
    }
    case 2: case 6: {
      int sq = (int)slotQ[r];
      set_link(SQ, bQ, sq, srcP);
      SP.it(bP + srcP) = 1;
      if (winP) SP.nb(bP + srcP) = sq;
      break;
    }
    case 3: case 7: {
      int sp = (int)slotP[r];
      set_link(SP, bP, sp, srcQ);
      SQ.it(bQ + srcQ) = 1;
      if (winQ) SQ.nb(bQ + srcQ) = sp;
      break;
    }
    case 4: case 8: {
      SP.it(bP + srcP) = 1; SQ.it(bQ + srcQ) = 1;
      if (winP) SP.nb(bP + srcP) = srcQ;
      if (winQ) SQ.nb(bQ + srcQ) = srcP;
      break;
    }
    case 5: {
      int sp = (int)slotP[r], sq = (int)slotQ[r];
      set_link(SQ, bQ, sq, srcP);
      SP.it(bP + srcP) = 1;
      if (winP) SP.nb(bP + srcP) = sq;
      set_link(SP, bP, sp, srcQ);
      SQ.it(bQ + srcQ) = 1;
      if (winQ) SQ.nb(bQ + srcQ) = sp;
      break;
    }
  }
}

// ---------------------------------------------------------------- ring export
// The reference's calculateIntersections (gppolyclip_mDIV512.cu:1298-1640) returns the
// merged rings with an integer parameter key per vertex: (int)(1e7 * alpha) where the
// vertex carries an intersection, -100 at plain vertices (:926).  Inserted vertices get
// the key of their one record (:997-1053).  The source vertex of an edge gets the key of
// its degenerate records (P: types 2/4/6/8, Q: types 3/4/7/8).  The P side is written by
// the P edge's loop over ascending Q edges, so the largest Q edge wins.  The Q side is
// written by concurrent P-edge threads (a race in the reference); here the largest P edge
// wins.  Keys are packed as (other edge + 1) << 32 | key and combined with atomicMax.
// Per pair it also counts the records that insert a vertex on each ring.
__device__ __forceinline__ uint32_t alpha_key(double a) {
  return (uint32_t)(int32_t)(10000000.0 * a);      // (int)pow(10, EPSILON_POSITIONS)*alpha
}

__global__ void export_key_kernel(Records R, int64_t nR, const int32_t* __restrict__ status,
                                  const int64_t* __restrict__ eoffP, const int64_t* __restrict__ eoffQ,
                                  const int64_t* __restrict__ vposP, const int64_t* __restrict__ vposQ,
                                  const int64_t* __restrict__ regP, const int64_t* __restrict__ regQ,
                                  const int64_t* __restrict__ slotP, const int64_t* __restrict__ slotQ,
                                  unsigned long long* __restrict__ keyP, unsigned long long* __restrict__ keyQ,
                                  int32_t* __restrict__ cntP, int32_t* __restrict__ cntQ) {
  int64_t r = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (r >= nR) return;
  const int k = R.k[r];
  const int t = R.t[r];
  const bool insOnP = t == 1 || t == 3 || t == 5 || t == 7;
  const bool insOnQ = t == 1 || t == 2 || t == 5 || t == 6;
  if (insOnP) atomicAdd(&cntP[k], 1);
  if (insOnQ) atomicAdd(&cntQ[k], 1);
  if (status[k] != 0) return;
  const int64_t eP = eoffP[k] + R.p[r], eQ = eoffQ[k] + R.q[r];
  const uint32_t kp = alpha_key(R.a[r]), kq = alpha_key(R.b[r]);
  if (insOnP) {
    keyP[regP[k] + slotP[r]] = (1ull << 32) | kp;
  } else {
    const int64_t src = vposP[eP] - vposP[eoffP[k]];
    atomicMax(&keyP[regP[k] + src], ((unsigned long long)(R.q[r] + 1) << 32) | kp);
  }
  if (insOnQ) {
    keyQ[regQ[k] + slotQ[r]] = (1ull << 32) | kq;
  } else {
    const int64_t src = vposQ[eQ] - vposQ[eoffQ[k]];
    atomicMax(&keyQ[regQ[k] + src], ((unsigned long long)(R.p[r] + 1) << 32) | kq);
  }
}

__device__ __forceinline__ int32_t unpack_key(unsigned long long v) {
  return v == 0 ? -100 : (int32_t)(uint32_t)v;
}

// oracle() of gppolyclip_mDIV512.cu:195-215: Q's position relative to the chain
// (P1, P2, P3), or which of P1 / P3 it is linked to
__device__ int export_rel(int exact, int pMN, int pPN, int qId, const RingSet& SQ, int64_t bQ,
                          const RingSet& SP, int64_t bP, int p1, int p2, int p3) {
  if (pMN != -100 && pMN == qId) return R_IS_P_M;
  if (pPN != -100 && pPN == qId) return R_IS_P_P;
  const double qx = SQ.x(bQ + qId), qy = SQ.y(bQ + qId);
  const double x1 = SP.x(bP + p1), y1 = SP.y(bP + p1), x2 = SP.x(bP + p2), y2 = SP.y(bP + p2);
  const double x3 = SP.x(bP + p3), y3 = SP.y(bP + p3);
  const int s1 = orient_sign(exact, qx, qy, x1, y1, x2, y2);
  const int s2 = orient_sign(exact, qx, qy, x2, y2, x3, y3);
  const int s3 = orient_sign(exact, x1, y1, x2, y2, x3, y3);
  if (s3 > 0) return (s1 > 0 && s2 > 0) ? R_LEFT : R_RIGHT;
  return (s1 < 0 && s2 < 0) ? R_RIGHT : R_LEFT;
}

// getInitialLabel of gppolyclip_mDIV512.cu:237-252, including its -102 for combinations
// that name no label
__device__ int32_t export_label(int m, int p) {
  auto is = [&](int a, int b) { return (m == a && p == b) || (m == b && p == a); };
  if (is(R_LEFT, R_RIGHT)) return L_CROSSING;
  if ((m == R_LEFT && p == R_LEFT) || (m == R_RIGHT && p == R_RIGHT)) return L_BOUNCING;
  if (is(R_IS_P_P, R_RIGHT)) return L_LEFT_ON;
  if (is(R_IS_P_P, R_LEFT)) return L_RIGHT_ON;
  if (is(R_IS_P_P, R_IS_P_M)) return L_ON_ON;
  if (is(R_IS_P_M, R_RIGHT)) return L_ON_LEFT;
  if (is(R_IS_P_M, R_LEFT)) return L_ON_RIGHT;
  return -102;
}

// Block per pair: the merged rings in ring order (slot order before any labelling), their
// keys and 1-based neighbours; then the initial labels of gpuCalculateInitLabel
// (gppolyclip_mDIV512.cu:1171-1223), computed at the P vertices that carry a key and
// copied to their Q neighbours.  Output arrays are indexed like the ring regions.
__global__ void export_ring_kernel(int64_t K, const int32_t* __restrict__ status, const int32_t* __restrict__ mP,
                                   const int32_t* __restrict__ mQ, const int64_t* __restrict__ regP,
                                   const int64_t* __restrict__ regQ, RingSet SP, RingSet SQ,
                                   const unsigned long long* __restrict__ keyP,
                                   const unsigned long long* __restrict__ keyQ, double* __restrict__ xyP,
                                   double* __restrict__ xyQ, int32_t* __restrict__ alP, int32_t* __restrict__ alQ,
                                   int32_t* __restrict__ lbP, int32_t* __restrict__ lbQ, int32_t* __restrict__ nbP,
                                   int32_t* __restrict__ nbQ) {
  const int64_t k = blockIdx.x;
  if (k >= K || status[k] != 0) return;
  const int np = mP[k], nq = mQ[k];
  const int64_t bP = regP[k], bQ = regQ[k];
  for (int s = threadIdx.x; s < np; s += blockDim.x) {
    const int64_t g = bP + s;
    xyP[2 * g] = SP.x(g); xyP[2 * g + 1] = SP.y(g);
    alP[g] = unpack_key(keyP[g]);
    lbP[g] = -100;
    nbP[g] = SP.nb(g) + 1;
  }
  for (int s = threadIdx.x; s < nq; s += blockDim.x) {
    const int64_t g = bQ + s;
    xyQ[2 * g] = SQ.x(g); xyQ[2 * g + 1] = SQ.y(g);
    alQ[g] = unpack_key(keyQ[g]);
    lbQ[g] = -100;
    nbQ[g] = SQ.nb(g) + 1;
  }
  __syncthreads();
  for (int s = threadIdx.x; s < np; s += blockDim.x) {
    if (keyP[bP + s] == 0) continue;
    const int nId = SP.nb(bP + s);
    if (nId < 0 || nId >= nq) continue;
    const int pm = s > 0 ? s - 1 : np - 1, pp = s + 1 < np ? s + 1 : 0;
    const int pMN = keyP[bP + pm] != 0 ? SP.nb(bP + pm) : -100;
    const int pPN = keyP[bP + pp] != 0 ? SP.nb(bP + pp) : -100;
    const int qm = nId > 0 ? nId - 1 : nq - 1, qp = nId + 1 < nq ? nId + 1 : 0;
    const int a = export_rel(SP.exact, pMN, pPN, qm, SQ, bQ, SP, bP, pm, s, pp);
    const int b = export_rel(SP.exact, pMN, pPN, qp, SQ, bQ, SP, bP, pm, s, pp);
    const int32_t L = export_label(a, b);
    lbP[bP + s] = L;
    lbQ[bQ + nId] = L;
  }
}

// ---------------------------------------------------------------- G7 label + trace
struct Ring {
  char* b; int64_t n;   // the side's column buffer (RingSet)
  int64_t o;            // first slot of this ring
  int m;        // slots in the merged ring
  int used;     // slots in use (ring + added vertices)
  int cap;      // region capacity
  int exact;    // orientation signs exact
  GCMFGH_RING_COLUMNS(o + i)
};

__device__ __forceinline__ Ring ring_of(const RingSet& S, int64_t base, int m, int cap) {
  Ring r;
  r.b = S.b; r.n = S.n; r.o = base;
  r.m = m; r.used = m; r.cap = cap; r.exact = S.exact;
  return r;
}

__device__ int add_vertex(Ring& R, double X, double Y) {
  if (R.used >= R.cap) return -1;
  int v = R.used++;
  R.x(v) = X; R.y(v) = Y; R.nx(v) = v; R.pv(v) = v; R.nb(v) = -1;
  R.it(v) = 0; R.lb(v) = L_NONE; R.ee(v) = E_NEITHER; R.fl(v) = 0;
  return v;
}

__device__ __forceinline__ void insert_after(Ring& R, int v, int after) {
  int c = R.nx(after);
  R.nx(R.pv(c)) = v; R.pv(v) = R.pv(c); R.nx(v) = c; R.pv(c) = v;
}

// polygon.h:427-448 (winding parity) over the ring reached from slot 0, skipping `skip`
template <int EX>
__device__ bool point_in_ring(const Ring& R, double Rx, double Ry, int skip) {
  int w = 0;
  int one = 0;
  int guard = R.used + 2;
  do {
    int two = R.nx(one);
    if (two == skip) two = R.nx(two);
    double P0x = R.x(one), P0y = R.y(one), P1x = R.x(two), P1y = R.y(two);
    if ((P0y < Ry) != (P1y < Ry)) {
      if (P0x >= Rx) {
        if (P1x > Rx) w = w + 2 * (P1y > P0y) - 1;
        else if ((orient_sign(EX, P0x, P0y, P1x, P1y, Rx, Ry) > 0) == (P1y > P0y)) w = w + 2 * (P1y > P0y) - 1;
      } else if (P1x > Rx) {
        if ((orient_sign(EX, P0x, P0y, P1x, P1y, Rx, Ry) > 0) == (P1y > P0y)) w = w + 2 * (P1y > P0y) - 1;
      }
    }
    one = two;
  } while (one != 0 && --guard > 0);
  return (w % 2) != 0;
}

// relative position of Q w.r.t. the chain (P1, P2, P3): polyclip.h:297-326
template <int EX>
__device__ int rel_position(const Ring& P, const Ring& Q, int qv, int p1, int p2, int p3) {
  if (P.it(p1) && P.nb(p1) == qv) return R_IS_P_M;
  if (P.it(p3) && P.nb(p3) == qv) return R_IS_P_P;
  const int ex = EX;
  int s1 = orient_sign(ex, Q.x(qv), Q.y(qv), P.x(p1), P.y(p1), P.x(p2), P.y(p2));
  int s2 = orient_sign(ex, Q.x(qv), Q.y(qv), P.x(p2), P.y(p2), P.x(p3), P.y(p3));
  int s3 = orient_sign(ex, P.x(p1), P.y(p1), P.x(p2), P.y(p2), P.x(p3), P.y(p3));
  if (s3 > 0) return (s1 > 0 && s2 > 0) ? R_LEFT : R_RIGHT;
  return (s1 < 0 && s2 < 0) ? R_RIGHT : R_LEFT;
}

// gppolyclip_mDIV512.cu:237-252
__device__ __forceinline__ int8_t initial_label(int m, int p) {
  auto is = [&](int a, int b) { return (m == a && p == b) || (m == b && p == a); };
  if (is(R_LEFT, R_RIGHT)) return L_CROSSING;
  if ((m == R_LEFT && p == R_LEFT) || (m == R_RIGHT && p == R_RIGHT)) return L_BOUNCING;
  if (is(R_IS_P_P, R_RIGHT)) return L_LEFT_ON;
  if (is(R_IS_P_P, R_LEFT)) return L_RIGHT_ON;
  if (is(R_IS_P_P, R_IS_P_M)) return L_ON_ON;
  if (is(R_IS_P_M, R_RIGHT)) return L_ON_LEFT;
  if (is(R_IS_P_M, R_LEFT)) return L_ON_RIGHT;
  return L_NONE;
}

struct OutRegion {
  double* xy;        // vertex region of the pair (2 doubles per vertex)
  int32_t* csz;      // component sizes of the pair
  int64_t vcap;
  int ccap;
  int64_t nv;
  int nc;
  bool overflow;
  __device__ void begin() { if (nc < ccap) csz[nc] = 0; else overflow = true; }
  __device__ void push(double X, double Y) {
    if (overflow) return;
    if (nv >= vcap) { overflow = true; return; }
    xy[2 * nv] = X; xy[2 * nv + 1] = Y; ++nv; ++csz[nc];
  }
  __device__ void end() { if (!overflow) ++nc; }
};

// first non-intersection vertex in ring order from slot 0, else the first vertex whose
// edge to the next vertex is not collinear with the other polygon (polygon.h:480-512)
__device__ int first_non_intersection(const Ring& A, const Ring& B, bool& midpoint) {
  midpoint = false;
  int v = 0, guard = A.used + 1;
  do { if (!A.it(v)) return v; v = A.nx(v); } while (v != 0 && --guard > 0);
  v = 0; guard = A.used + 1;
  do {
    int nb = A.nb(v), nx = A.nx(v);
    if (nb >= 0 && A.nb(nx) != B.pv(nb) && A.nb(nx) != B.nx(nb)) { midpoint = true; return v; }
    v = A.nx(v);
  } while (v != 0 && --guard > 0);
  return -1;
}

__device__ void push_ring(OutRegion& O, const Ring& A) {
  O.begin();
  int v = 0, guard = A.used + 1;
  do { O.push(A.x(v), A.y(v)); v = A.nx(v); } while (v != 0 && --guard > 0);
  O.end();
}

// Per-pair state of the labelling and tracing phases.
struct PairCtx {
  Ring R[2];
  OutRegion O;
  bool uni;
  double eps_clean;
  int* err;
  int32_t* status;
  bool noInter[2];
  bool ident[2];
};

__device__ __forceinline__ int8_t toggled(int8_t st) {
  return (st == E_ENTRY) ? E_EXIT : (st == E_EXIT ? E_ENTRY : st);
}

__device__ __forceinline__ void fail(PairCtx& c, int code) {
  raise_error(c.err, code);
  *c.status = 3;
}

// ================================================================ sequential phases
// One thread walks the pair exactly as polyclip.h does.  Used whole when the links are not
// one-to-one, and for the parts the warp version leaves to one lane (chain anomalies,
// split vertices, tracing through added vertices).

// step 1: initial labels (computed on P, copied to the neighbour on Q)
template <int EX>
__device__ void seq_step1(PairCtx& c) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  for (int s = 0; s < P.m; ++s) {
    if (!P.it(s)) continue;
    int nb = P.nb(s);
    if (nb < 0) continue;
    int pm = P.pv(s), pp = P.nx(s);
    int a = rel_position<EX>(P, Q, Q.pv(nb), pm, s, pp);
    int b = rel_position<EX>(P, Q, Q.nx(nb), pm, s, pp);
    int8_t L = initial_label(a, b);
    if (L != L_NONE) { P.lb(s) = L; Q.lb(nb) = L; }
  }
}

// What one member's long loops call as they go on: a grid's barrier counts it as progress.
struct NoBeat { __device__ __forceinline__ void operator()(int) const {} };

// step 2: intersection chains (polyclip.h:405-451).  n >= 0: the chain starts are among the n
// slots listed in P.ls, in order
template <class B = NoBeat>
__device__ void seq_step2(PairCtx& c, int n = -1, B beat = B()) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  const int count = n < 0 ? P.m : n;
  for (int i = 0; i < count; ++i) {
    const int s = n < 0 ? i : P.ls(i);
    beat(i);
    if (!P.it(s) || (P.lb(s) != L_LEFT_ON && P.lb(s) != L_RIGHT_ON)) continue;
    int x = P.lb(s) == L_LEFT_ON ? R_LEFT : R_RIGHT;
    int X = s, I = s, guard = P.m + 1;
    do {
      beat(guard);
      P.lb(I) = L_NONE;
      if (P.nb(I) >= 0) Q.lb(P.nb(I)) = L_NONE;
      I = P.nx(I);
    } while (P.lb(I) == L_ON_ON && --guard > 0);
    int y = P.lb(I) == L_ON_LEFT ? R_LEFT : R_RIGHT;
    int8_t ct = (x != y) ? L_DELAYED_CROSSING : L_DELAYED_BOUNCING;
    P.lb(X) = ct; P.lb(I) = ct;
    if (P.nb(X) >= 0) Q.lb(P.nb(X)) = ct;
    if (P.nb(I) >= 0) Q.lb(P.nb(I)) = ct;
  }
}

// step 3.5: components without crossings (polyclip.h:474-541)
template <int EX>
__device__ void seq_step35(PairCtx& c) {
  for (int sd = 0; sd < 2; ++sd) {
    Ring& A = c.R[sd];
    bool none = true, allOn = true;
    for (int v = 0; v < A.m; ++v) {
      int8_t l = A.lb(v);
      if (l != L_ON_ON) allOn = false;
      if (A.it(v)) {
        if (l == L_CROSSING || l == L_DELAYED_CROSSING) none = false;
        if (c.uni && (l == L_BOUNCING || l == L_DELAYED_BOUNCING)) none = false;
      }
    }
    c.noInter[sd] = none;
    c.ident[sd] = none && allOn;
  }
  for (int sd = 0; sd < 2; ++sd) {
    if (!c.noInter[sd] || c.ident[sd]) continue;
    Ring& A = c.R[sd];
    Ring& B = c.R[1 - sd];
    bool mid;
    int v = first_non_intersection(A, B, mid);
    if (v < 0) continue;
    double px = A.x(v), py = A.y(v);
    if (mid) { int n = A.nx(v); px = 0.5 * (A.x(v) + A.x(n)); py = 0.5 * (A.y(v) + A.y(n)); }
    bool inside = point_in_ring<EX>(B, px, py, -1);
    if (inside ^ c.uni) push_ring(c.O, A);
  }
  if (c.ident[0] && c.ident[1]) push_ring(c.O, c.R[0]);
}

// step 4: entry/exit flags (polyclip.h:549-655)
template <int EX>
__device__ bool seq_step4(PairCtx& c) {
  for (int sd = 0; sd < 2; ++sd) {
    if (c.noInter[sd]) continue;
    Ring& A = c.R[sd];
    Ring& B = c.R[1 - sd];
    bool mid;
    int V = first_non_intersection(A, B, mid);
    if (V < 0) continue;
    if (mid) {
      int n = A.nx(V);
      int T = add_vertex(A, 0.5 * (A.x(V) + A.x(n)), 0.5 * (A.y(V) + A.y(n)));
      if (T < 0) { fail(c, DEV_CAPACITY); return false; }
      insert_after(A, T, V);
      V = T;
    }
    // the Q pass sees P's temporary vertex; P's pass cannot see Q's (not yet added)
    int8_t st = point_in_ring<EX>(B, A.x(V), A.y(V), -1) ? E_EXIT : E_ENTRY;
    bool first = true;
    int I = A.nx(V), guard = A.used + 1;
    while (I != V && --guard > 0) {
      if (A.it(I)) {
        int8_t l = A.lb(I);
        if (l == L_CROSSING) { A.ee(I) = st; st = toggled(st); }
        if (A.lb(I) == L_BOUNCING && ((st == E_EXIT) ^ c.uni)) A.fl(I) |= 1;
        if (A.lb(I) == L_DELAYED_CROSSING) {
          A.ee(I) = st;
          if (first) { if ((st == E_EXIT) ^ c.uni) A.lb(I) = L_CROSSING; first = false; }
          else {
            if ((st == E_ENTRY) ^ c.uni) A.lb(I) = L_CROSSING;
            first = true;
            st = toggled(st);
          }
        }
        if (A.lb(I) == L_DELAYED_BOUNCING) {
          A.ee(I) = st;
          if (first) { if ((st == E_EXIT) ^ c.uni) A.fl(I) |= 2; first = false; }
          else { if ((st == E_ENTRY) ^ c.uni) A.fl(I) |= 2; first = true; }
          st = toggled(st);
        }
      }
      I = A.nx(I);
    }
  }
  return true;
}

// step 5: split vertex pairs (polyclip.h:661-714).  n >= 0: the candidates of P are the n
// slots listed in P.ls, in order
template <int EX, class B = NoBeat>
__device__ bool seq_step5(PairCtx& c, int n = -1, B beat = B()) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  const int pm0 = n < 0 ? P.used : n;
  for (int i = 0; i < pm0; ++i) {
    const int ip = n < 0 ? i : P.ls(i);
    beat(i);
    if (!(P.fl(ip) & 1)) continue;
    int iq = P.nb(ip);
    if (iq < 0 || !(Q.fl(iq) & 1)) continue;
    int vp = add_vertex(P, P.x(ip), P.y(ip));
    int vq = add_vertex(Q, Q.x(iq), Q.y(iq));
    if (vp < 0 || vq < 0) { fail(c, DEV_CAPACITY); return false; }
    bool same;
    if (EX) {
      same = orient_exact_call(P.x(P.pv(ip)), P.y(P.pv(ip)), P.x(ip), P.y(ip), P.x(P.nx(ip)), P.y(P.nx(ip))) *
             orient_exact_call(Q.x(Q.pv(iq)), Q.y(Q.pv(iq)), Q.x(iq), Q.y(iq), Q.x(Q.nx(iq)), Q.y(Q.nx(iq))) > 0;
    } else {
      double sP = area2(P.x(P.pv(ip)), P.y(P.pv(ip)), P.x(ip), P.y(ip), P.x(P.nx(ip)), P.y(P.nx(ip)));
      double sQ = area2(Q.x(Q.pv(iq)), Q.y(Q.pv(iq)), Q.x(iq), Q.y(iq), Q.x(Q.nx(iq)), Q.y(Q.nx(iq)));
      same = sP * sQ > 0;
    }
    if (same) {
      P.nb(ip) = vq; Q.nb(vq) = ip; P.it(ip) = 1; Q.it(vq) = 1;
      Q.nb(iq) = vp; P.nb(vp) = iq; Q.it(iq) = 1; P.it(vp) = 1;
    } else {
      P.nb(vp) = vq; Q.nb(vq) = vp; P.it(vp) = 1; Q.it(vq) = 1;
    }
    insert_after(P, vp, ip);
    insert_after(Q, vq, iq);
    int8_t e1 = c.uni ? E_ENTRY : E_EXIT, e2 = c.uni ? E_EXIT : E_ENTRY;
    P.ee(ip) = e1; P.ee(vp) = e2; Q.ee(iq) = e1; Q.ee(vq) = e2;
    P.lb(ip) = L_CROSSING; P.lb(vp) = L_CROSSING; Q.lb(iq) = L_CROSSING; Q.lb(vq) = L_CROSSING;
  }
  return true;
}

// step 6: crossing candidates (polyclip.h:723-734)
__device__ void seq_step6(PairCtx& c) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  for (int ip = 0; ip < P.m; ++ip) {
    if (!(P.fl(ip) & 2)) continue;
    int iq = P.nb(ip);
    if (iq >= 0 && (Q.fl(iq) & 2)) { P.lb(ip) = L_CROSSING; Q.lb(iq) = L_CROSSING; }
  }
}

// A walk that never closes repeats itself: the piece that starts at V of a ring is the same
// each time within one component.  Brent's cycle detection (1980) over the pieces' starts
// ends such a pair after a few rounds of its cycle instead of the whole step budget; the
// pair's status is the same (3, no output).
struct WalkRepeat {
  int v = -1, side = -1, steps = 0, power = 1;
  __device__ __forceinline__ bool seen(int V, int s) {
    if (V == v && s == side) return true;
    if (++steps == power) { v = V; side = s; steps = 0; power <<= 1; }
    return false;
  }
};

// tracing (polyclip.h:743-783): starts at unvisited CROSSING vertices of P in ring order
// from slot 0; visited vertices are marked by clearing their intersection flag.
__device__ bool seq_trace(PairCtx& c) {
  Ring& P = c.R[0];
  OutRegion& O = c.O;
  long long budget = 4ll * (c.R[0].used + c.R[1].used) + 16;
  int I = 0;
  bool have = P.it(I) && P.lb(I) == L_CROSSING;
  if (!have) {
    int guard = P.used + 1;
    do { I = P.nx(I); } while (!(P.it(I) && P.lb(I) == L_CROSSING) && I != 0 && --guard > 0);
    have = I != 0 && guard > 0;
  }
  while (have) {
    O.begin();
    int side = 0, V = I;
    P.it(V) = 0;
    WalkRepeat again;
    do {
      Ring& C = c.R[side];
      int8_t st = toggled(C.ee(V));
      int left = C.used + 1;                           // once round the ring finds every stop
      if (again.seen(V, side)) { fail(c, DEV_TRACE); return false; }
      do {
        if (--budget < 0 || --left < 0) { fail(c, DEV_TRACE); return false; }
        V = ((st == E_EXIT) ^ c.uni) ? C.nx(V) : C.pv(V);
        C.it(V) = 0;
        O.push(C.x(V), C.y(V));
      } while (!(C.ee(V) == st) && !(side == 0 && V == I));
      if (!(side == 0 && V == I)) {
        int nb = C.nb(V);
        if (nb < 0) { fail(c, DEV_TRACE); return false; }
        V = nb;
        side = 1 - side;
        c.R[side].it(V) = 0;
      }
    } while (!(side == 0 && V == I));
    O.end();
    int guard = P.used + 1;
    do { I = P.nx(I); } while (!(P.it(I) && P.lb(I) == L_CROSSING) && I != 0 && --guard > 0);
    have = I != 0 && guard > 0;
  }
  if (O.overflow) { fail(c, DEV_CAPACITY); return false; }
  return true;
}

// clean-up of one component (polyclip.h:791-807): drop the first vertex while it is
// collinear with its ring neighbours, then one forward pass that removes every vertex
// collinear with the last kept vertex and its original successor.  Reads n vertices at
// src and returns how many are kept; kWrite: writes them to dst (which may be src itself,
// or anything before it).
template <bool kWrite>
__device__ int seq_cleanup_component(const double2* src, double2* dst, int n, double eps) {
  if (n == 0) return 0;
  const double2 last = src[n - 1];
  int r = 0;
  while (r < n) {
    const double2 v = src[r], nx = src[(r + 1 < n) ? r + 1 : r];
    double a = area2(last.x, last.y, v.x, v.y, nx.x, nx.y);
    if (r == n - 1) a = 0.0;              // ring of the last vertex alone: A(v,v,v)
    if (fabs(a) < eps) ++r; else break;
  }
  if (r >= n) return 0;
  double2 k = src[r];
  const double2 first = k;
  int kept = 1;
  if (kWrite) dst[0] = k;
  for (int j = r + 1; j < n; ++j) {
    const double2 v = src[j], nx = (j + 1 < n) ? src[j + 1] : first;
    if (fabs(area2(k.x, k.y, v.x, v.y, nx.x, nx.y)) < eps) continue;
    if (kWrite) dst[kept] = v;
    ++kept;
    k = v;
  }
  return kept;
}

__device__ void seq_cleanup(PairCtx& c, int32_t* outNC, int64_t* outNV) {
  OutRegion& O = c.O;
  int64_t vin = 0, vout = 0;
  int nc = 0;
  for (int k = 0; k < O.nc; ++k) {
    const int n = O.csz[k];
    double2* xy = reinterpret_cast<double2*>(O.xy);
    int kept = seq_cleanup_component<true>(xy + vin, xy + vout, n, c.eps_clean);
    vin += n;
    if (kept == 0) continue;
    O.csz[nc++] = kept;
    vout += kept;
  }
  *outNC = nc;
  *outNV = vout;
}

// the whole pair from `step` on (1: everything, 2: after the initial labels)
template <int EX>
__device__ void seq_pair_from(PairCtx& c, int step, int32_t* outNC, int64_t* outNV) {
  if (step <= 1) seq_step1<EX>(c);
  seq_step2(c);
  seq_step35<EX>(c);
  if (!seq_step4<EX>(c) || !seq_step5<EX>(c)) return;
  seq_step6(c);
  if (!seq_trace(c)) return;
  seq_cleanup(c, outNC, outNV);
}

// ================================================================ warp phases
constexpr unsigned kFull = 0xffffffffu;

// winding increment of edge (P0,P1) for point R: polygon.h:433-444
__device__ __forceinline__ int wind(double P0x, double P0y, double P1x, double P1y, double Rx, double Ry,
                                    int ex) {
  if ((P0y < Ry) == (P1y < Ry)) return 0;
  int d = 2 * (P1y > P0y) - 1;
  if (P0x >= Rx) {
    if (P1x > Rx) return d;
    return ((orient_sign(ex, P0x, P0y, P1x, P1y, Rx, Ry) > 0) == (P1y > P0y)) ? d : 0;
  }
  if (P1x > Rx) return ((orient_sign(ex, P0x, P0y, P1x, P1y, Rx, Ry) > 0) == (P1y > P0y)) ? d : 0;
  return 0;
}

// How a piece of a ring changes the state of the entry/exit pass, (d, t) = (parity of the
// chain ends met, parity of the status changes): d' = d ^ a, t' = t ^ b ^ (c & d), as bits
// a | b << 1 | c << 2.  Pieces compose, so the pass is a scan over any split of the ring.
__device__ __forceinline__ unsigned flow_then(unsigned f, unsigned g) {
  const unsigned fa = f & 1u, gc = (g >> 2) & 1u;
  return ((f ^ g) & 7u) ^ ((gc & fa) << 1);
}
__device__ __forceinline__ unsigned flow_of(int8_t label) {
  return label == L_CROSSING ? 2u : label == L_DELAYED_BOUNCING ? 3u : label == L_DELAYED_CROSSING ? 5u : 0u;
}
__device__ __forceinline__ unsigned warp_flow_scan(unsigned x) {   // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if ((int)lane_id() >= o) x = flow_then(y, x);
  }
  return x;
}

// ---- cooperative groups for the parallel labelling and tracing of one pair.  The same
// code runs with a warp per pair (WarpGroup) or, for pairs with long rings, a whole block
// (BlockGroup) or the whole grid (GridGroup) per pair; every member executes every group
// call (uniform control flow).  kItems: ring slots a member takes between two scans.
struct WarpGroup {
  __device__ __forceinline__ void beat(int) const {}
  static constexpr bool kBlock = false;
  static constexpr bool kGrid = false;
  static constexpr bool kSolo = false;
  static constexpr int kItems = 4;
  // exclusive scan of flows in member order, and their composition
  __device__ __forceinline__ unsigned flow_excl(unsigned x, unsigned& total) const {
    const unsigned v = warp_flow_scan(x), e = __shfl_up_sync(kFull, v, 1);
    total = __shfl_sync(kFull, v, 31);
    return lane_id() == 0 ? 0u : e;
  }
  __device__ __forceinline__ int rank() const { return (int)lane_id(); }
  __device__ __forceinline__ int size() const { return 32; }
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ bool all(bool v) const { return __all_sync(kFull, v); }
  __device__ __forceinline__ bool any(bool v) const { return __any_sync(kFull, v); }
  __device__ __forceinline__ int sum(int v) const { return warp_sum(v); }
  template <class T>
  __device__ __forceinline__ T bcast0(T v) const { return __shfl_sync(kFull, v, 0); }
  // smallest member index whose flag is set, -1 if none
  __device__ __forceinline__ int first(bool hit) const {
    unsigned m = __ballot_sync(kFull, hit);
    return m ? __ffs(m) - 1 : -1;
  }
  __device__ __forceinline__ int incl_scan(int v, int& total) const {
    int x = warp_incl_scan(v);
    total = __shfl_sync(kFull, x, 31);
    return x;
  }
  // f(s, hit, hits before s) for every s in [0, n); returns the number of hits
  template <class P, class F>
  __device__ __forceinline__ int list(int n, P pred, F f) const {
    int carry = 0;
    for (int b = 0; b < n; b += 32) {
      const int s = b + rank();
      const bool hit = s < n && pred(s);
      const unsigned m = __ballot_sync(kFull, hit);
      if (s < n) f(s, hit, carry + __popc(m & lanemask_lt()));
      carry += __popc(m);
    }
    return carry;
  }
};

// One thread per pair: every collective is the identity, nothing synchronises.
struct SoloGroup {
  __device__ __forceinline__ void beat(int) const {}
  static constexpr bool kGrid = false;
  static constexpr bool kSolo = true;
  static constexpr int kItems = 1;
  __device__ __forceinline__ unsigned flow_excl(unsigned x, unsigned& total) const { total = x; return 0u; }
  __device__ __forceinline__ int rank() const { return 0; }
  __device__ __forceinline__ int size() const { return 1; }
  __device__ __forceinline__ void sync() const {}
  __device__ __forceinline__ bool all(bool v) const { return v; }
  __device__ __forceinline__ bool any(bool v) const { return v; }
  __device__ __forceinline__ int sum(int v) const { return v; }
  template <class T>
  __device__ __forceinline__ T bcast0(T v) const { return v; }
  __device__ __forceinline__ int first(bool hit) const { return hit ? 0 : -1; }
  __device__ __forceinline__ int incl_scan(int v, int& total) const { total = v; return v; }
};

// Block-wide versions over shared scratch (kBlockLabelThreads / 32 warps); each call
// begins with a barrier so the scratch of the previous call is free.
constexpr int kBlockLabelThreads = 512;
constexpr int kBlockLabelWarps = kBlockLabelThreads / 32;
// Dynamic shared memory of the block labelling kernel: the trace's loop table of pairs with
// up to 8,192 segments of P, 12 bytes each.  (At 122 to 128 registers one block fits an SM.)
constexpr int kBlockLoopTableBytes = 96 * 1024;
constexpr int kBlockListRounds = 8;   // elements per thread between two barriers of list()
constexpr int kBlockScratch = kBlockLabelWarps + 1 + (kBlockListRounds * kBlockLabelWarps + 2) / 2;
struct BlockGroup {
  __device__ __forceinline__ void beat(int) const {}
  static constexpr bool kBlock = true;
  static constexpr bool kGrid = false;
  static constexpr bool kSolo = false;
  static constexpr int kItems = 16;
  long long* sm;        // kBlockScratch entries
  uint32_t* loops;      // shared memory for the trace's loop table
  int loopsCap;         // segments that fit
  __device__ __forceinline__ int rank() const { return (int)threadIdx.x; }
  __device__ __forceinline__ int size() const { return kBlockLabelThreads; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  __device__ __forceinline__ bool all(bool v) const { return __syncthreads_and(v) != 0; }
  __device__ __forceinline__ bool any(bool v) const { return __syncthreads_or(v) != 0; }
  __device__ __forceinline__ int sum(int v) const {
    v = warp_sum(v);
    __syncthreads();
    if (lane_id() == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    long long t = 0;
    for (int w = 0; w < kBlockLabelThreads / 32; ++w) t += sm[w];
    return (int)t;
  }
  template <class T>
  __device__ __forceinline__ T bcast0(T v) const {
    static_assert(sizeof(T) <= sizeof(long long), "bcast0: scalar types only");
    __syncthreads();
    if (threadIdx.x == 0) { long long x = 0; memcpy(&x, &v, sizeof(T)); sm[kBlockLabelThreads / 32] = x; }
    __syncthreads();
    long long x = sm[kBlockLabelThreads / 32];
    T r;
    memcpy(&r, &x, sizeof(T));
    return r;
  }
  __device__ __forceinline__ int first(bool hit) const {
    unsigned m = __ballot_sync(kFull, hit);
    __syncthreads();
    if (lane_id() == 0) sm[threadIdx.x >> 5] = m ? (long long)((threadIdx.x & ~31u) + __ffs(m) - 1) : -1;
    __syncthreads();
    for (int w = 0; w < kBlockLabelThreads / 32; ++w)
      if (sm[w] >= 0) return (int)sm[w];
    return -1;
  }
  __device__ __forceinline__ int incl_scan(int v, int& total) const {
    int x = warp_incl_scan(v);
    __syncthreads();
    if (lane_id() == 31) sm[threadIdx.x >> 5] = x;
    __syncthreads();
    long long before = 0, all = 0;
    const int me = (int)(threadIdx.x >> 5);
    for (int w = 0; w < kBlockLabelThreads / 32; ++w) { if (w < me) before += sm[w]; all += sm[w]; }
    total = (int)all;
    return (int)(before + x);
  }
  __device__ __forceinline__ unsigned flow_excl(unsigned x, unsigned& total) const {
    const unsigned v = warp_flow_scan(x), e = __shfl_up_sync(kFull, v, 1);
    __syncthreads();
    if (lane_id() == 31) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned before = 0, all = 0;
    const int me = (int)(threadIdx.x >> 5);
    for (int w = 0; w < kBlockLabelWarps; ++w) { if (w == me) before = all; all = flow_then(all, (unsigned)sm[w]); }
    total = all;
    return flow_then(before, lane_id() == 0 ? 0u : e);
  }
  // One step of list(): the hits of this block's kBlockListRounds * kBlockLabelThreads elements
  // from b on.  m: this thread's ballots, at[r]: hits of the step before round r of its warp.
  template <class P>
  __device__ __forceinline__ int list_step(int b, int n, P pred, unsigned* m, int*& at) const {
    int* cnt = reinterpret_cast<int*>(sm + kBlockLabelWarps + 1);   // [round][warp], then the total
    const int warp = (int)(threadIdx.x >> 5), lane = (int)lane_id();
    constexpr int kCounts = kBlockListRounds * kBlockLabelWarps, kPer = kCounts / 32;
#pragma unroll
    for (int r = 0; r < kBlockListRounds; ++r) {
      const int s = b + r * kBlockLabelThreads + (int)threadIdx.x;
      m[r] = __ballot_sync(kFull, s < n && pred(s));
    }
    __syncthreads();
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < kBlockListRounds; ++r) cnt[r * kBlockLabelWarps + warp] = __popc(m[r]);
    }
    __syncthreads();
    if (warp == 0) {
      int v[kPer], t = 0;
#pragma unroll
      for (int j = 0; j < kPer; ++j) { v[j] = cnt[lane * kPer + j]; t += v[j]; }
      const int incl = warp_incl_scan(t);
      int run = incl - t;
#pragma unroll
      for (int j = 0; j < kPer; ++j) { cnt[lane * kPer + j] = run; run += v[j]; }
      if (lane == 31) cnt[kCounts] = incl;
    }
    __syncthreads();
    at = cnt + warp;
    return cnt[kCounts];
  }
  // As WarpGroup's: each thread takes kBlockListRounds elements per step, so that the
  // barriers and the scan of the warps' counts are paid once per 4,096 elements.
  template <class P, class F>
  __device__ __forceinline__ int list(int n, P pred, F f) const {
    int carry = 0;
    for (int b = 0; b < n; b += kBlockListRounds * kBlockLabelThreads) {
      unsigned m[kBlockListRounds];
      int* at;
      const int total = list_step(b, n, pred, m, at);
#pragma unroll
      for (int r = 0; r < kBlockListRounds; ++r) {
        const int s = b + r * kBlockLabelThreads + (int)threadIdx.x;
        if (s < n) f(s, ((m[r] >> lane_id()) & 1u) != 0, carry + at[r * kBlockLabelWarps] + __popc(m[r] & lanemask_lt()));
      }
      carry += total;
    }
    return carry;
  }
};

// The whole grid on one pair (a cooperative launch: all blocks are resident).  The blocks meet
// at a counting barrier.  Its wait is bounded by progress: it gives up only when, for
// ClipParams::grid_wait polls, no block has arrived and no member that works alone (a chain, a
// long loop, the split vertices) has called beat().  A wait that gave up ends the kernel: the
// error is raised, and every block leaves at the barrier where it learns of it, before it uses what
// it would have waited for.
constexpr int kGridBlocksMax = 512;
struct GridScratch {
  unsigned arrive;
  unsigned beats;
  int dead;
  unsigned long long slot[3];                            // reductions, in turn
  unsigned long long blk[2][kGridBlocksMax];             // blocks' parts of a scan, in turn
};

struct GridGroup {
  static constexpr bool kBlock = false;
  static constexpr bool kGrid = true;
  static constexpr bool kSolo = false;
  static constexpr int kItems = 16;
  BlockGroup blk;
  GridScratch* gs;
  int* err;
  long long wait;
  int* gone;                                             // shared: the block leaves
  mutable unsigned epoch = 0, reds = 0, scans = 0;
  __device__ __forceinline__ GridGroup(const BlockGroup& b, GridScratch* g, int* e, long long w, int* left)
      : blk(b), gs(g), err(e), wait(w), gone(left) {}
  __device__ __forceinline__ int rank() const { return (int)(blockIdx.x * kBlockLabelThreads + threadIdx.x); }
  __device__ __forceinline__ int size() const { return (int)(gridDim.x * kBlockLabelThreads); }
  // progress of a member's long loop, by its step count
  __device__ __forceinline__ void beat(int step) const { if ((step & 1023) == 1023) atomicAdd(&gs->beats, 1u); }
  __device__ void sync() const {
    ++epoch;
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned target = epoch * gridDim.x;
      __threadfence();
      atomicAdd(&gs->arrive, 1u);
      volatile GridScratch* v = gs;
      unsigned seen = v->arrive + v->beats;
      for (long long polls = 0; (int)(v->arrive - target) < 0 && !v->dead;) {
        if (++polls <= wait) continue;
        const unsigned now = v->arrive + v->beats;
        if (now == seen) { v->dead = 1; raise_error(err, DEV_TIMEOUT); break; }
        seen = now;
        polls = 0;
      }
      __threadfence();
      *gone = v->dead;
    }
    __syncthreads();
    if (*gone) asm volatile("exit;");
  }
  // combine one value per block: add(slot, value) by each block's first thread
  template <class A>
  __device__ __forceinline__ unsigned long long reduce(A add) const {
    unsigned long long* s = &gs->slot[reds % 3];
    if (rank() == 0) *reinterpret_cast<volatile unsigned long long*>(&gs->slot[(reds + 1) % 3]) = 0ull;
    ++reds;
    if (threadIdx.x == 0) add(s);
    sync();
    return *reinterpret_cast<volatile unsigned long long*>(s);
  }
  __device__ __forceinline__ bool any(bool v) const {
    const int b = __syncthreads_or(v);
    return reduce([&](unsigned long long* s) { if (b) atomicOr(s, 1ull); }) != 0;
  }
  __device__ __forceinline__ bool all(bool v) const { return !any(!v); }
  __device__ __forceinline__ int sum(int v) const {
    const int b = blk.sum(v);
    return (int)reduce([&](unsigned long long* s) { if (b) atomicAdd(s, (unsigned long long)(long long)b); });
  }
  template <class T>
  __device__ __forceinline__ T bcast0(T v) const {
    static_assert(sizeof(T) <= sizeof(long long), "bcast0: scalar types only");
    unsigned long long x = 0;
    memcpy(&x, &v, sizeof(T));
    x = reduce([&](unsigned long long* s) { if (blockIdx.x == 0) atomicExch(s, x); });
    T r;
    memcpy(&r, &x, sizeof(T));
    return r;
  }
  __device__ __forceinline__ int first(bool hit) const {
    const int f = blk.first(hit);
    const unsigned long long top = 1ull << 40;
    const unsigned long long m = reduce([&](unsigned long long* s) {
      if (f >= 0) atomicMax(s, top - (unsigned long long)(blockIdx.x * kBlockLabelThreads + f));
    });
    return m ? (int)(top - m) : -1;
  }
  // parts of all blocks after a barrier: op folds them in block order; before: those of earlier blocks
  template <class T, class O>
  __device__ __forceinline__ T block_parts(T mine, T none, O op, T& before) const {
    unsigned long long* parts = gs->blk[scans++ & 1];
    if (threadIdx.x == 0) *reinterpret_cast<volatile unsigned long long*>(&parts[blockIdx.x]) = (unsigned long long)mine;
    sync();
    T all = none;
    before = none;
    for (unsigned b0 = 0; b0 < gridDim.x; b0 += 32) {    // every warp folds them by itself
      const unsigned b = b0 + lane_id();
      T v = b < gridDim.x ? (T)*reinterpret_cast<volatile unsigned long long*>(&parts[b]) : none;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(kFull, v, o);
        if ((int)lane_id() >= o) v = op(u, v);
      }
      if (blockIdx.x > b0 && blockIdx.x <= b0 + 32) before = op(all, __shfl_sync(kFull, v, (int)(blockIdx.x - b0) - 1));
      all = op(all, __shfl_sync(kFull, v, 31));
    }
    return all;
  }
  __device__ __forceinline__ int incl_scan(int v, int& total) const {
    int mine, before;
    const int x = blk.incl_scan(v, mine);
    total = block_parts<int>(mine, 0, [](int a, int b) { return a + b; }, before);
    return before + x;
  }
  __device__ __forceinline__ unsigned flow_excl(unsigned x, unsigned& total) const {
    unsigned mine, before;
    const unsigned e = blk.flow_excl(x, mine);
    total = block_parts<unsigned>(mine, 0u, [](unsigned a, unsigned b) { return flow_then(a, b); }, before);
    return flow_then(before, e);
  }
  template <class P, class F>
  __device__ __forceinline__ int list(int n, P pred, F f) const {
    constexpr int kStep = kBlockListRounds * kBlockLabelThreads;
    int carry = 0;
    for (int64_t b0 = 0; b0 < n; b0 += (int64_t)kStep * gridDim.x) {
      const int b = (int)min(b0 + (int64_t)blockIdx.x * kStep, (int64_t)n);   // this block's elements
      unsigned m[kBlockListRounds];
      int* at;
      int before;
      const int mine = blk.list_step(b, n, pred, m, at);
      const int total = block_parts<int>(mine, 0, [](int x, int y) { return x + y; }, before);
#pragma unroll
      for (int r = 0; r < kBlockListRounds; ++r) {
        const int s = b + r * kBlockLabelThreads + (int)threadIdx.x;
        if (s < n)
          f(s, ((m[r] >> lane_id()) & 1u) != 0, carry + before + at[r * kBlockLabelWarps] + __popc(m[r] & lanemask_lt()));
      }
      carry += total;
    }
    return carry;
  }
};

// polygon.h:427-448 over ring B in slot order; `after`/`T`: a temporary vertex T inserted
// after slot `after` (or -1)
template <int EX, class G>
__device__ bool grp_point_in_ring(const G& g, const Ring& B, double Rx, double Ry, int after, int T) {
  int w = 0;
  for (int s = g.rank(); s < B.m; s += g.size()) {
    int n = (s + 1 < B.m) ? s + 1 : 0;
    if (s == after) {
      w += wind(B.x(s), B.y(s), B.x(T), B.y(T), Rx, Ry, EX);
      w += wind(B.x(T), B.y(T), B.x(n), B.y(n), Rx, Ry, EX);
    } else {
      w += wind(B.x(s), B.y(s), B.x(n), B.y(n), Rx, Ry, EX);
    }
  }
  w = g.sum(w);
  return (w % 2) != 0;
}

// first slot s >= from (slot order, s < n) where pred(s); n if none
template <class G, class F>
__device__ int grp_find_first(const G& g, int from, int n, F pred) {
  for (int b = from; b < n; b += g.size()) {
    int s = b + g.rank();
    int f = g.first(s < n && pred(s));
    if (f >= 0) return b + f;
  }
  return n;
}

template <class G>
__device__ bool grp_links_one_to_one(const G& g, const Ring& P, const Ring& Q) {
  bool ok = true;
  for (int s = g.rank(); s < P.m; s += g.size())
    if (P.it(s)) { int nb = P.nb(s); if (nb < 0 || nb >= Q.m || Q.nb(nb) != s) ok = false; }
  for (int s = g.rank(); s < Q.m; s += g.size())
    if (Q.it(s)) { int nb = Q.nb(s); if (nb < 0 || nb >= P.m || P.nb(nb) != s) ok = false; }
  return g.all(ok);
}

template <int EX, class G>
__device__ void grp_step1(const G& g, PairCtx& c) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  for (int s = g.rank(); s < P.m; s += g.size()) {
    if (!P.it(s)) continue;
    int nb = P.nb(s);
    int pm = (s > 0) ? s - 1 : P.m - 1, pp = (s + 1 < P.m) ? s + 1 : 0;
    int a = rel_position<EX>(P, Q, (nb > 0) ? nb - 1 : Q.m - 1, pm, s, pp);
    int b = rel_position<EX>(P, Q, (nb + 1 < Q.m) ? nb + 1 : 0, pm, s, pp);
    int8_t L = initial_label(a, b);
    if (L != L_NONE) { P.lb(s) = L; Q.lb(nb) = L; }
  }
  g.sync();
}

// Step 1 for links that are not one-to-one: of the P vertices linked to one Q vertex the
// last one with a label gives it to that vertex, as in the sequential loop.
template <int EX, class G>
__device__ void grp_step1_shared(const G& g, PairCtx& c) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  for (int s = g.rank(); s < Q.m; s += g.size()) Q.tn(s) = -1;
  g.sync();
  for (int s = g.rank(); s < P.m; s += g.size()) {
    const int nb = P.it(s) ? P.nb(s) : -1;
    if (nb < 0) continue;
    const int pm = (s > 0) ? s - 1 : P.m - 1, pp = (s + 1 < P.m) ? s + 1 : 0;
    const int8_t L = initial_label(rel_position<EX>(P, Q, (nb > 0) ? nb - 1 : Q.m - 1, pm, s, pp),
                                   rel_position<EX>(P, Q, (nb + 1 < Q.m) ? nb + 1 : 0, pm, s, pp));
    if (L != L_NONE) { P.lb(s) = L; atomicMax(&Q.tn(nb), s); }
  }
  g.sync();
  for (int s = g.rank(); s < P.m; s += g.size()) {
    const int nb = P.it(s) ? P.nb(s) : -1;
    if (nb >= 0 && P.lb(s) != L_NONE && Q.tn(nb) == s) Q.lb(nb) = P.lb(s);
  }
  g.sync();
}

// Chains run from a LEFT_ON/RIGHT_ON vertex over ON_ON vertices to an ON_LEFT/ON_RIGHT
// vertex.  When every chain ends so, chains are disjoint and can be resolved in parallel
// with the sequential result; otherwise returns false and nothing is changed.
template <class G>
__device__ bool grp_step2(const G& g, PairCtx& c) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  const int m = P.m;
  bool ok = true;
  for (int s = g.rank(); s < m; s += g.size()) {
    if (!P.it(s) || (P.lb(s) != L_LEFT_ON && P.lb(s) != L_RIGHT_ON)) continue;
    int I = (s + 1 < m) ? s + 1 : 0, guard = m;
    while (P.lb(I) == L_ON_ON && --guard > 0) { g.beat(guard); I = (I + 1 < m) ? I + 1 : 0; }
    if ((P.lb(I) != L_ON_LEFT && P.lb(I) != L_ON_RIGHT) || !P.it(I)) ok = false;
  }
  if (!g.all(ok)) return false;
  for (int s = g.rank(); s < m; s += g.size()) {
    int8_t l0 = P.lb(s);
    if (!P.it(s) || (l0 != L_LEFT_ON && l0 != L_RIGHT_ON)) continue;
    int x = l0 == L_LEFT_ON ? R_LEFT : R_RIGHT;
    int I = (s + 1 < m) ? s + 1 : 0;
    Q.lb(P.nb(s)) = L_NONE;
    while (P.lb(I) == L_ON_ON) {
      g.beat(I);
      P.lb(I) = L_NONE;
      Q.lb(P.nb(I)) = L_NONE;
      I = (I + 1 < m) ? I + 1 : 0;
    }
    int y = P.lb(I) == L_ON_LEFT ? R_LEFT : R_RIGHT;
    int8_t ct = (x != y) ? L_DELAYED_CROSSING : L_DELAYED_BOUNCING;
    P.lb(s) = ct; P.lb(I) = ct;
    Q.lb(P.nb(s)) = ct; Q.lb(P.nb(I)) = ct;
  }
  g.sync();
  return true;
}

// copies ring A (slot order, no added vertices) as one output component
template <class G>
__device__ void grp_push_ring(const G& g, OutRegion& O, const Ring& A) {
  // (the size is written by one member only: no begin(), whose zero another could write later)
  if (O.nc >= O.ccap || O.nv + A.m > O.vcap) { O.overflow = true; return; }
  for (int s = g.rank(); s < A.m; s += g.size()) { O.xy[2 * (O.nv + s)] = A.x(s); O.xy[2 * (O.nv + s) + 1] = A.y(s); }
  if (g.rank() == 0) O.csz[O.nc] = A.m;
  O.nv += A.m;
  O.end();
  g.sync();
}

// first non-intersection slot (slot order = ring order before any insertion), else the
// first vertex whose edge to the next one is not collinear with the other polygon
// (polygon.h:480-512); returns -1 if none
template <class G>
__device__ int grp_first_non_intersection(const G& g, const Ring& A, const Ring& B, bool& mid) {
  mid = false;
  int v = grp_find_first(g, 0, A.m, [&](int s) { return !A.it(s); });
  if (v < A.m) return v;
  // B's own links: B may already hold its temporary vertex when A is Q
  v = grp_find_first(g, 0, A.m, [&](int s) {
    int nb = A.nb(s), nx = A.nx(s);
    return nb >= 0 && A.nb(nx) != B.pv(nb) && A.nb(nx) != B.nx(nb);
  });
  if (v < A.m) { mid = true; return v; }
  return -1;
}

template <int EX, class G>
__device__ void grp_step35(const G& g, PairCtx& c) {
  for (int sd = 0; sd < 2; ++sd) {
    Ring& A = c.R[sd];
    bool none = true, allOn = true;
    for (int v = g.rank(); v < A.m; v += g.size()) {
      int8_t l = A.lb(v);
      if (l != L_ON_ON) allOn = false;
      if (A.it(v)) {
        if (l == L_CROSSING || l == L_DELAYED_CROSSING) none = false;
        if (c.uni && (l == L_BOUNCING || l == L_DELAYED_BOUNCING)) none = false;
      }
    }
    none = g.all(none);
    allOn = g.all(allOn);
    c.noInter[sd] = none;
    c.ident[sd] = none && allOn;
  }
  for (int sd = 0; sd < 2; ++sd) {
    if (!c.noInter[sd] || c.ident[sd]) continue;
    Ring& A = c.R[sd];
    Ring& B = c.R[1 - sd];
    bool mid;
    int v = grp_first_non_intersection(g, A, B, mid);
    if (v < 0) continue;
    double px = A.x(v), py = A.y(v);
    if (mid) { int n = (v + 1 < A.m) ? v + 1 : 0; px = 0.5 * (A.x(v) + A.x(n)); py = 0.5 * (A.y(v) + A.y(n)); }
    bool inside = grp_point_in_ring<EX>(g, B, px, py, -1, -1);
    if (inside ^ c.uni) grp_push_ring(g, c.O, A);
  }
  if (c.ident[0] && c.ident[1]) grp_push_ring(g, c.O, c.R[0]);
}

// Entry/exit flags as a scan over the ring from the start vertex: the status at a vertex is
// the start status toggled once per earlier CROSSING, DELAYED_BOUNCING and second-of-a-chain
// DELAYED_CROSSING; "first chain vertex" alternates over the DELAYED vertices met
// (polyclip.h:582-653).  Each member takes kItems consecutive slots per step and one scan
// composes their effects (flow_then).
template <int EX, class G>
__device__ bool grp_step4(const G& g, PairCtx& c, int tempAfter[2], int tempSlot[2]) {
  for (int sd = 0; sd < 2; ++sd) {
    tempAfter[sd] = -1;
    tempSlot[sd] = -1;
  }
  for (int sd = 0; sd < 2; ++sd) {
    if (c.noInter[sd]) continue;
    Ring& A = c.R[sd];
    Ring& B = c.R[1 - sd];
    bool mid;
    int V0 = grp_first_non_intersection(g, A, B, mid);
    if (V0 < 0) continue;
    double qx = A.x(V0), qy = A.y(V0);
    if (mid) {
      int T = -1;
      if (g.rank() == 0) {
        T = add_vertex(A, 0.5 * (A.x(V0) + A.x((V0 + 1 < A.m) ? V0 + 1 : 0)),
                       0.5 * (A.y(V0) + A.y((V0 + 1 < A.m) ? V0 + 1 : 0)));
        if (T >= 0) insert_after(A, T, V0);
      }
      T = g.bcast0(T);
      A.used = g.bcast0(A.used);
      g.sync();
      if (T < 0) { if (g.rank() == 0) fail(c, DEV_CAPACITY); return false; }
      tempAfter[sd] = V0;
      tempSlot[sd] = T;
      qx = A.x(T);
      qy = A.y(T);
    }
    // the Q pass tests against P's ring including P's temporary vertex
    int8_t st0 = (sd == 1 ? grp_point_in_ring<EX>(g, B, qx, qy, tempAfter[0], tempSlot[0])
                          : grp_point_in_ring<EX>(g, B, qx, qy, -1, -1)) ? E_EXIT : E_ENTRY;
    unsigned d = 0, t = 0;                               // the state before this step's slots
    const int m = A.m;
    constexpr int kI = G::kItems;
    for (int b = 0; b < m; b += g.size() * kI) {
      const int j0 = b + g.rank() * kI;
      auto slot = [&](int j) { const int s = V0 + 1 + j; return s >= m ? s - m : s; };
      int8_t L[kI];
      unsigned mine = 0, all;
#pragma unroll
      for (int i = 0; i < kI; ++i) {
        L[i] = L_NONE;
        if (j0 + i < m && A.it(slot(j0 + i))) L[i] = A.lb(slot(j0 + i));
      }
#pragma unroll
      for (int i = 0; i < kI; ++i) mine = flow_then(mine, flow_of(L[i]));
      const unsigned e = g.flow_excl(mine, all);
      unsigned td = d ^ (e & 1u), tt = t ^ ((e >> 1) & 1u) ^ ((e >> 2) & d);
#pragma unroll
      for (int i = 0; i < kI; ++i) {
        if (L[i] == L_NONE) continue;
        const int s = slot(j0 + i);
        const bool first = td == 0;
        int8_t st = tt ? toggled(st0) : st0;
        if (L[i] == L_CROSSING) A.ee(s) = st;
        else if (L[i] == L_BOUNCING) { if ((st == E_EXIT) ^ c.uni) A.fl(s) |= 1; }
        else if (L[i] == L_DELAYED_CROSSING) {
          A.ee(s) = st;
          if (first) { if ((st == E_EXIT) ^ c.uni) A.lb(s) = L_CROSSING; }
          else if ((st == E_ENTRY) ^ c.uni) A.lb(s) = L_CROSSING;
        } else if (L[i] == L_DELAYED_BOUNCING) {
          A.ee(s) = st;
          if (first) { if ((st == E_EXIT) ^ c.uni) A.fl(s) |= 2; }
          else if ((st == E_ENTRY) ^ c.uni) A.fl(s) |= 2;
        }
        const unsigned f = flow_of(L[i]);
        tt ^= ((f >> 1) & 1u) ^ ((f >> 2) & td);
        td ^= f & 1u;
      }
      t ^= ((all >> 1) & 1u) ^ ((all >> 2) & d);
      d ^= all & 1u;
    }
    g.sync();
  }
  return true;
}

template <class G>
__device__ bool grp_any_split(const G& g, const Ring& P, const Ring& Q) {
  bool any = false;
  for (int s = g.rank(); s < P.m; s += g.size())
    if (P.fl(s) & 1) { int nb = P.nb(s); if (nb >= 0 && (Q.fl(nb) & 1)) any = true; }
  return g.any(any);
}

template <class G>
__device__ void grp_step6(const G& g, PairCtx& c) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  for (int ip = g.rank(); ip < P.m; ip += g.size()) {
    if (!(P.fl(ip) & 2)) continue;
    int iq = P.nb(ip);
    if (iq >= 0 && (Q.fl(iq) & 2)) { P.lb(ip) = L_CROSSING; Q.lb(iq) = L_CROSSING; }
  }
  g.sync();
}

// Run-table tracing for one-thread pairs.  With entry/exit flags alternating along both
// rings (checked here), every run of the sequential walk goes from a flagged vertex to the
// adjacent flagged vertex in its direction, and the next run starts at that vertex's
// neighbour.  Phase 1 gives each flagged vertex, by its slot, its run (tl: the length, signed
// by direction; tn: the next run's start); phase 2 follows the runs in the order of the
// sequential walk and assigns each its output offset (to), marking visited vertices in the
// rings' intersection flags; phase 3 copies the runs.  Returns 0 when done, 1 when the
// flags do not alternate (the caller then runs the general walk), -1 on a capacity or trace
// error.
__device__ int grp_trace_runs_slots(const SoloGroup& g, PairCtx& c) {
  int nF[2];
  bool mismatch = false;     // a flagged vertex that is not a crossing, or the reverse
  for (int sd = 0; sd < 2; ++sd) {
    Ring& A = c.R[sd];
    int carry = 0;
    for (int b = 0; b < A.m; b += g.size()) {
      const int s = b + g.rank();
      const int f = (s < A.m && (A.ee(s) == E_ENTRY || A.ee(s) == E_EXIT)) ? 1 : 0;
      if (s < A.m && (f != 0) != (A.it(s) && A.lb(s) == L_CROSSING)) mismatch = true;
      int tot;
      const int incl = g.incl_scan(f, tot);
      if (f) A.ls(carry + incl - 1) = s;
      carry += tot;
    }
    nF[sd] = carry;
  }
  if (g.any(mismatch)) return 1;
  if (nF[0] == 0 && nF[1] == 0) return 0;
  bool bad = nF[0] < 2 || nF[1] < 2;
  bool longRun = false;
  for (int sd = 0; sd < 2 && !bad; ++sd) {
    Ring& A = c.R[sd];
    const Ring& B = c.R[1 - sd];
    const int n = nF[sd], m = A.m;
    for (int i = g.rank(); i < n; i += g.size()) {
      const int s = A.ls(i);
      const int8_t e = A.ee(s);
      if (!A.it(s) || A.lb(s) != L_CROSSING) { bad = true; continue; }
      if (A.ee(A.ls((i + 1 < n) ? i + 1 : 0)) == e) { bad = true; continue; }   // alternation
      const int nb = A.nb(s);
      if (nb < 0 || nb >= B.m || B.ee(nb) != toggled(e)) { bad = true; continue; }
      const int8_t st = toggled(e);
      const int dir = ((st == E_EXIT) ^ c.uni) ? 1 : -1;
      const int W = A.ls((i + dir + n) % n);
      int L = dir > 0 ? W - s : s - W;
      if (L <= 0) L += m;
      const int nbW = A.nb(W);
      if (nbW < 0 || nbW >= B.m) { bad = true; continue; }
      A.tl(s) = dir * L;
      A.tn(s) = nbW;
      A.to(s) = -1;
      if (L > 32) longRun = true;
    }
  }
  if (g.any(bad)) return 1;
  const bool anyLong = g.any(longRun);
  // ---- phase 2: the walk over the run table, one member
  OutRegion& O = c.O;
  int status = 0;
  int64_t nv = O.nv;
  int nc = O.nc;
  if (g.rank() == 0) {
    Ring& P = c.R[0];
    const int64_t nv0 = O.nv;
    long long budget = (long long)nF[0] + nF[1] + 4;
    for (int i = 0; i < nF[0] && status == 0; ++i) {
      const int I = P.ls(i);
      if (!P.it(I)) continue;
      if (nc >= O.ccap) { status = -1; fail(c, DEV_CAPACITY); break; }
      P.it(I) = 0;
      int side = 0, V = I;
      int64_t csz = 0;
      for (;;) {
        Ring& C = c.R[side];
        const int t = C.tl(V), L = t < 0 ? -t : t, m = C.m;
        int W = V + t % m;
        W = (W % m + m) % m;
        C.to(V) = (int32_t)(nv - nv0);
        nv += L;
        csz += L;
        C.it(W) = 0;
        if (side == 0 && W == I) break;
        const int V2 = C.tn(V);
        side ^= 1;
        if (side == 0 && V2 == I) break;
        c.R[side].it(V2) = 0;
        V = V2;
        if (--budget < 0) { status = -1; fail(c, DEV_TRACE); break; }
      }
      if (status == 0) {
        if (nv > O.vcap) { status = -1; fail(c, DEV_CAPACITY); break; }
        O.csz[nc++] = (int32_t)csz;
      }
    }
  }
  status = g.bcast0(status);
  if (status != 0) return -1;
  const int64_t nv0 = O.nv;
  O.nv = g.bcast0((long long)nv);
  O.nc = g.bcast0(nc);
  // ---- phase 3: copy every run to its place; short runs one member each, long runs by
  // the whole group (no barrier between runs: runs write disjoint ranges)
  constexpr int kShortRun = 32;      // the run-length threshold of phase 1's longRun
  for (int sd = 0; sd < 2; ++sd) {
    const Ring& A = c.R[sd];
    const int m = A.m;
    for (int i = g.rank(); i < nF[sd]; i += g.size()) {
      const int s = A.ls(i);
      const int off = A.to(s);
      if (off < 0) continue;
      const int t = A.tl(s), L = t < 0 ? -t : t, dir = t < 0 ? -1 : 1;
      if (anyLong && L > kShortRun) continue;
      double* dst = O.xy + 2 * (nv0 + off);
      int w = s;
      for (int j = 0; j < L; ++j) {
        w += dir;
        if (w >= m) w -= m;
        if (w < 0) w += m;
        dst[2 * j] = A.x(w);
        dst[2 * j + 1] = A.y(w);
      }
    }
    for (int i = 0; anyLong && i < nF[sd]; ++i) {
      const int s = A.ls(i);
      const int off = A.to(s);
      const int t = A.tl(s), L = t < 0 ? -t : t;
      if (off < 0 || L <= kShortRun) continue;
      const int dir = t < 0 ? -1 : 1;
      double* dst = O.xy + 2 * (nv0 + off);
      for (int j = g.rank(); j < L; j += g.size()) {
        int w = s + dir * (j + 1);
        w %= m;
        if (w < 0) w += m;
        dst[2 * j] = A.x(w);
        dst[2 * j + 1] = A.y(w);
      }
    }
  }
  g.sync();
  return 0;
}

// Copies one run per lane (L vertices of ring A from slot s0 on, exclusive, in direction
// dir) to dst: short runs by their lane, long ones by the whole warp one after another.
// Every lane of the warp calls it; lanes without a run pass L = 0.
__device__ __forceinline__ void warp_copy_runs(const Ring& A, int s0, int L, int dir, double2* dst) {
  constexpr int kShortRun = 16;
  const int m = A.m;
  if (L <= kShortRun) {
    int w = s0;
    for (int j = 0; j < L; ++j) {
      w += dir;
      if (w >= m) w -= m;
      if (w < 0) w += m;
      dst[j] = A.xy(w);
    }
  }
  unsigned longs = __ballot_sync(kFull, L > kShortRun);
  while (longs) {
    const int src = __ffs(longs) - 1;
    longs &= longs - 1;
    const int bs = __shfl_sync(kFull, s0, src), bL = __shfl_sync(kFull, L, src), bd = __shfl_sync(kFull, dir, src);
    double2* d = reinterpret_cast<double2*>(__shfl_sync(kFull, (unsigned long long)dst, src));
    for (int j = (int)lane_id(); j < bL; j += 32) {
      int w = bs + bd * (j + 1);                       // |j + 1| <= m: one wrap at most
      if (w >= m) w -= m;
      if (w < 0) w += m;
      d[j] = A.xy(w);
    }
  }
}

// The loop table of one pair.  A P segment t has two ends, 0 its first and 1 its last vertex.
// link(t, e): the P segment and the end of it that a walk leaving t at end e gets to over the
// Q segment there, as 2 * segment + end; w(t, e): the vertices of t and of that Q segment.
// Bit 31 of w(t, 1) is set when neither end is a crossing.
constexpr unsigned kNoCrossing = 0x80000000u;
struct LoopsGlobal {
  const int32_t *l0, *l1, *w0, *w1;
  __device__ __forceinline__ int link(int t, int e) const { return (e ? l1 : l0)[t]; }
  __device__ __forceinline__ unsigned raw(int t) const { return (unsigned)w1[t]; }
  __device__ __forceinline__ int w(int t, int e) const { return e ? (int)(raw(t) & ~kNoCrossing) : w0[t]; }
};
struct LoopsShared {                                     // 12 bytes per segment, fewer than 2^15 segments
  uint32_t* p;
  int n;
  __device__ __forceinline__ int link(int t, int e) const { return (int)((p[t] >> (16 * e)) & 0xffffu); }
  __device__ __forceinline__ unsigned raw(int t) const { return p[2 * n + t]; }
  __device__ __forceinline__ int w(int t, int e) const { return e ? (int)(raw(t) & ~kNoCrossing) : (int)p[n + t]; }
};

// The loops' nodes (long loops of the grid path): every kNodeEvery-th segment and the segments
// that the bounded search left open, in this order; link and w lead from node to node.
constexpr int kNodeEvery = 256;
struct LoopsNodes {
  const int32_t *l0, *l1, *w0, *w1;
  int open;                                              // the first of the open segments
  __device__ __forceinline__ int link(int i, int e) const { return (e ? l1 : l0)[i]; }
  __device__ __forceinline__ unsigned raw(int i) const { return i < open ? kNoCrossing : 0u; }
  __device__ __forceinline__ int w(int i, int e) const { return (e ? w1 : w0)[i]; }
};

// The size of t's loop when t is its smallest segment with a crossing, else 0 (-1: the walk
// did not close within guard steps).  The walk goes both ways at once and stops at the
// first smaller segment: over a loop of L segments the searches take O(L log L) steps in
// all, whatever its order, and the smallest segment's own takes L / 2.
template <class T, class B = NoBeat>
__device__ __forceinline__ int loop_size(const T& tab, int t, int guard, B beat = B()) {
  if (tab.raw(t) & kNoCrossing) return 0;
  int f = tab.link(t, 1), b = tab.link(t, 0);            // where the two walks arrive
  int sz = tab.w(t, 1);
  while ((f >> 1) != t) {
    beat(guard >> 1);
    const int ft = f >> 1, bt = b >> 1, fo = 1 - (f & 1), bi = b & 1;
    if ((ft < t && !(tab.raw(ft) & kNoCrossing)) || (bt < t && !(tab.raw(bt) & kNoCrossing))) return 0;
    sz += tab.w(ft, fo);
    if (ft == bt) break;
    sz += tab.w(bt, bi);
    f = tab.link(ft, fo);
    if ((f >> 1) == bt) break;
    b = tab.link(bt, 1 - bi);
    if ((guard -= 2) < 0) return -1;
  }
  return sz;
}

// Output offsets of the segments of t's loop (size vertices from base on), walked from t
// entered at end `in`; from both ends of the range.  A segment entered at its last vertex
// has ~offset.
template <class T>
__device__ __forceinline__ void loop_offsets(const T& tab, int t, int in, int base, int size, int32_t* off) {
  off[t] = in ? ~base : base;
  int of = base + tab.w(t, 1 - in), ob = base + size;
  int f = tab.link(t, 1 - in), b = tab.link(t, in);
  while (of < ob) {
    const int ft = f >> 1, fi = f & 1;
    off[ft] = fi ? ~of : of;
    of += tab.w(ft, 1 - fi);
    if (of >= ob) break;
    const int bt = b >> 1, be = b & 1;                   // the walk leaves bt at end be
    ob -= tab.w(bt, be);
    off[bt] = be ? ob : ~ob;
    f = tab.link(ft, 1 - fi);
    b = tab.link(bt, 1 - be);
  }
}

// Tracing by loops.  The walk of polyclip.h:743-783 starts at crossings of P, leaves a vertex
// that starts a piece (a forward vertex: entry, or exit for a union) in ring order and stops
// at the next flagged vertex of the other kind, leaves one of the other kind against ring
// order, and goes on at a stop's neighbour.  Wherever a ring's flags change from forward to
// backward there is a segment: forward walks stop at its last vertex, backward walks at
// its first, and no other flagged vertex is ever stopped at.  The neighbours link the segments of
// P and Q into loops.  Where every stop has a flagged neighbour, the links are the same in
// both directions, and every crossing of P ends a segment (all checked here), the loops
// are disjoint and the walk emits them in the order of their smallest crossing of P, each
// from that crossing on.  So instead of walking them one after another (a chain of dependent
// loads over all pieces of the pair, with the rest of the group waiting), every segment finds
// out whether it is its loop's smallest, the loops' sizes are scanned, and all loops are
// walked at once for the offsets of their segments.  Trace of 10,007 degenerate pairs (2.3e7
// crossings): 10.5 s of blocks' time as one walk per pair, 0.8 s so (a step costs two shared
// loads where the loop table fits shared memory).
// Returns 0 when done, 1 when the conditions do not hold (the caller then runs the general
// walk), -1 on a capacity error.
template <class G>
__device__ int grp_trace_loops(const G& g, PairCtx& c) {
  Ring& P = c.R[0];
  Ring& Q = c.R[1];
  const bool uni = c.uni;
  const int mP = P.m, mQ = Q.m;
  auto fwd_at = [uni](const Ring& A, int s) { return (A.ee(s) == E_ENTRY) != uni; };
  auto cross_at = [](const Ring& A, int s) { return A.it(s) && A.lb(s) == L_CROSSING; };
  bool bad = false, crossing = false, beside = false;
  int nF[2], nS[2];
  bool wrapFirst = false;
  for (int sd = 0; sd < 2; ++sd) {
    Ring& A = c.R[sd];
    // ls: the flagged slots in ring order
    nF[sd] = g.list(
        A.m,
        [&](int s) {
          const bool flagged = A.ee(s) != E_NEITHER;
          if (sd == 0 && cross_at(A, s)) { crossing = true; if (!flagged) bad = true; }
          return flagged;
        },
        [&](int s, bool hit, int before) { if (hit) A.ls(before) = s; });
    g.sync();
    const int n = nF[sd];
    // Segment numbers by the place of the first vertex, except that P's segment around
    // slot 0 is the first one when its smaller end is a crossing (the walk starts there).
    // tn: segment -> place of its first vertex in ls; to: flagged slot -> its segment
    if (sd == 0) wrapFirst = n > 1 && !fwd_at(A, A.ls(0)) && fwd_at(A, A.ls(n - 1)) && cross_at(A, A.ls(0));
    nS[sd] = g.list(n, [&](int f) { return fwd_at(A, A.ls(f)) && !fwd_at(A, A.ls(f + 1 < n ? f + 1 : 0)); },
                    [&](int f, bool hit, int before) {
                      const int s = A.ls(f);
                      const bool fw = fwd_at(A, s);
                      if (hit) A.tn(before) = f;
                      else if (sd == 0 && cross_at(A, s) && (fw || !fwd_at(A, A.ls(f > 0 ? f - 1 : n - 1)))) beside = true;
                      A.to(s) = (hit || fw) ? before : before - 1;   // -1 and the count stand for the wrapped one
                    });
    g.sync();
  }
  if (g.any(bad)) return 1;
  if (!g.any(crossing)) return 0;                        // nothing to start from
  const int n = nS[0], nQ = nS[1], nFP = nF[0], nFQ = nF[1];
  if (n == 0 || n > nQ) return 1;
  // scratch: at most half of a ring's vertices start segments, so a column holds two arrays
  int32_t* bP = &P.tn(0);
  int32_t* lead = &P.tn(mP >> 1);
  int32_t* bQ = &Q.tn(0);
  int32_t* eV = &Q.tn(mQ >> 1);                          // where a segment is entered, if not at its end
  int32_t* off = &P.to(0);                               // (when the slot map is done with)
  const LoopsGlobal glob{&P.tl(0), &P.tl(mP >> 1), &Q.tl(0), &Q.tl(mQ >> 1)};
  bool shared = false;
  LoopsShared shrd{nullptr, n};
  if constexpr (G::kBlock) { shared = n <= g.loopsCap; shrd.p = g.loops; }
  auto link = [&](int t, int e) { return shared ? shrd.link(t, e) : glob.link(t, e); };
  auto place = [&](int t) { return bP[wrapFirst ? (t > 0 ? t - 1 : n - 1) : t]; };
  auto end_p = [&](int t, int e) { const int f = place(t) + e; return P.ls(f < nFP ? f : 0); };
  auto end_q = [&](int j, int e) { const int f = bQ[j] + e; return Q.ls(f < nFQ ? f : 0); };
  auto seg_p = [&](int p) {
    int t = P.to(p);
    t = t < 0 ? n - 1 : (t >= n ? 0 : t);
    return wrapFirst ? (t + 1 < n ? t + 1 : 0) : t;
  };
  auto seg_q = [&](int q) { const int j = Q.to(q); return j < 0 ? nQ - 1 : (j >= nQ ? 0 : j); };
  auto dist = [](int from, int to, int m) { const int d = to - from; return d > 0 ? d : d + m; };
  bool odd = false;                                      // some segment is entered beside its end
  for (int t = g.rank(); t < n; t += g.size()) {
    const int v0 = end_p(t, 0), v1 = end_p(t, 1);
    const int lp = dist(v0, v1, mP);
    int lk[2] = {0, 0};
    unsigned w[2] = {0, 0};
    for (int e = 0; e < 2; ++e) {
      const int q = P.nb(e ? v1 : v0);
      if (q < 0 || q >= mQ || Q.ee(q) == E_NEITHER) { bad = true; break; }
      const int qe = fwd_at(Q, q) ? 0 : 1, j = seg_q(q); // entered at end qe, left at the other
      const int W = end_q(j, 1 - qe), p2 = Q.nb(W);
      if (p2 < 0 || p2 >= mP || P.ee(p2) == E_NEITHER) { bad = true; break; }
      const int t2 = seg_p(p2), pe = fwd_at(P, p2) ? 0 : 1;
      if (q != end_q(j, qe) || p2 != end_p(t2, pe)) odd = true;
      lk[e] = 2 * t2 + pe;
      w[e] = (unsigned)(lp + (qe ? dist(W, q, mQ) : dist(q, W, mQ)));
    }
    if (!cross_at(P, v0) && !cross_at(P, v1)) w[1] |= kNoCrossing;
    if (shared) {
      shrd.p[t] = (uint32_t)lk[0] | ((uint32_t)lk[1] << 16);
      shrd.p[n + t] = w[0];
      shrd.p[2 * n + t] = w[1];
    } else {
      const_cast<int32_t*>(glob.l0)[t] = lk[0];
      const_cast<int32_t*>(glob.l1)[t] = lk[1];
      const_cast<int32_t*>(glob.w0)[t] = (int32_t)w[0];
      const_cast<int32_t*>(glob.w1)[t] = (int32_t)w[1];
    }
  }
  g.sync();
  if (g.any(bad)) return 1;
  odd = g.any(odd);
  bool lop = false;                                      // links that differ by direction
  for (int t = g.rank(); t < n; t += g.size())
    for (int e = 0; e < 2; ++e) {
      const int l = link(t, e);
      if (link(l >> 1, l & 1) != 2 * t + e) lop = true;
    }
  if (g.any(lop || beside)) {
    // The walk may run into a loop that it did not start on, and never close.  Take the walk
    // that entered t at end e as a state: every state has one successor, so beyond the
    // tails the states form cycles, and walks that close go round one of them.  A crossing
    // of P that no cycle passes is therefore met by no closed walk; it will start one that
    // does not close, and the pair fails.  Otherwise the general walk decides.
    int32_t* deg[2] = {eV, lead};                        // predecessors of the state
    int32_t* way[2] = {&P.nx(0), &P.nx(mP >> 1)};        // the cycle's way into the segment, from its entry to its end
    for (int t = g.rank(); t < n; t += g.size())
      for (int e = 0; e < 2; ++e) { deg[e][t] = 0; way[e][t] = 0; }
    g.sync();
    for (int t = g.rank(); t < n; t += g.size())
      for (int e = 0; e < 2; ++e) { const int l = link(t, e); atomicAdd(&deg[l & 1][l >> 1], 1); }
    g.sync();
    for (int t = g.rank(); t < n; t += g.size())
      for (int e = 0; e < 2; ++e) if (deg[e][t] == 0) way[e][t] = -1;
    g.sync();
    for (int t = g.rank(); t < n; t += g.size())         // peel the tails from their first states on
      for (int e = 0; e < 2; ++e) {
        if (way[e][t] != -1) continue;
        int l = link(t, 1 - e), steps = 0;
        while (atomicSub(&deg[l & 1][l >> 1], 1) == 1) { g.beat(++steps); l = link(l >> 1, 1 - (l & 1)); }
      }
    g.sync();
    auto way_in = [&](int s, int t, int e) { return e ? dist(end_p(t, 0), s, mP) : dist(s, end_p(t, 1), mP); };
    for (int t = g.rank(); t < n; t += g.size())
      for (int e = 0; e < 2; ++e) {
        if (deg[e][t] <= 0) continue;
        const int q = P.nb(end_p(t, 1 - e)), l = link(t, 1 - e);
        way[l & 1][l >> 1] = way_in(Q.nb(end_q(seg_q(q), fwd_at(Q, q) ? 1 : 0)), l >> 1, l & 1);
      }
    g.sync();
    bool never = false;
    for (int f = g.rank(); f < nFP; f += g.size()) {
      const int s = P.ls(f);
      if (!cross_at(P, s)) continue;
      const int t = seg_p(s), e = fwd_at(P, s) ? 0 : 1;
      const bool passed = s == end_p(t, e) ? deg[0][t] > 0 || deg[1][t] > 0 : deg[e][t] > 0 && way[e][t] >= way_in(s, t, e);
      if (!passed) never = true;
    }
    never = g.any(never);
    for (int s = g.rank(); s < mP; s += g.size()) P.nx(s) = s + 1 < mP ? s + 1 : 0;
    g.sync();
    if (!never) return 1;
    if (g.rank() == 0) fail(c, DEV_TRACE);
    return -1;
  }
  // the end at which the walk enters its first segment: the smaller one that is a crossing
  auto start_end = [&](int t) { return ((t == 0 && wrapFirst) || !cross_at(P, end_p(t, 0))) ? 1 : 0; };
  // the pieces of one step: along P from `entry` to t's other end, along Q to where it is left
  struct Step { int sp, lp, sq, lq, dq, left; };
  auto step_of = [&](int t, int in, int entry, int left) {
    Step r;
    const int v = end_p(t, 1 - in);
    r.sp = entry;
    r.lp = in ? dist(v, entry, mP) : dist(entry, v, mP);
    r.sq = P.nb(v);
    const bool fq = fwd_at(Q, r.sq);
    r.left = left < 0 ? end_q(seg_q(r.sq), fq ? 1 : 0) : left;
    r.dq = fq ? 1 : -1;
    r.lq = fq ? dist(r.sq, r.left, mQ) : dist(r.left, r.sq, mQ);
    return r;
  };
  // ---- the loops' smallest segments and sizes
  // The grid bounds the search: a loop of 50,000 segments would keep one thread walking for
  // 18 ms, twice.  Segments that are smallest within kNodeEvery steps both ways stay open and
  // are nodes, with every kNodeEvery-th segment; all nodes walk to their neighbours, and
  // the open ones are decided over the nodes.
  int nOpen = 0;
  const int nEvery = (n + kNodeEvery - 1) / kNodeEvery;
  int32_t* node = &Q.to(0);                              // segment -> its node, -1 none (the slot map is done with)
  int32_t* nodeT = &Q.nx(0);
  int32_t* nodeOff = &Q.pv(0);
  const LoopsNodes nodes{&P.nx(0), &P.nx(mP >> 1), &P.pv(0), &P.pv(mP >> 1), nEvery};
  const bool bounded = G::kGrid && !odd;
  auto beat = [&g](int step) { g.beat(step); };
  for (int t = g.rank(); t < n; t += g.size()) {
    int sz = shared ? loop_size(shrd, t, n + 2) : loop_size(glob, t, bounded ? 2 * kNodeEvery : n + 2, beat);
    if (sz < 0 && !bounded) { bad = true; sz = 0; }
    if (odd && sz > 0) {                                 // the pieces depend on the direction: walk them
      const int in0 = start_end(t), I = end_p(t, in0);
      int u = t, in = in0, v = I, steps = 0;
      sz = 0;
      do {
        beat(++steps);
        const Step r = step_of(u, in, v, -1);
        sz += r.lp + r.lq;
        v = Q.nb(r.left);
        const int l = link(u, 1 - in);
        u = l >> 1;
        in = l & 1;
      } while (u != t);
      if (v != I) bad = true;                            // closes elsewhere than at its start
    }
    off[t] = sz;
  }
  g.sync();
  if (g.any(bad)) return 1;
  if constexpr (G::kGrid) {
    if (bounded) {
      nOpen = g.list(n, [&](int t) { return off[t] < 0; },
                     [&](int t, bool hit, int before) {
                       node[t] = hit ? nEvery + before : (t % kNodeEvery == 0 ? t / kNodeEvery : -1);
                       if (hit) { nodeT[nEvery + before] = t; off[t] = 0; }
                     });
      g.sync();
    }
    if (nOpen > 0) {
      for (int i = g.rank(); i < nEvery + nOpen; i += g.size()) {
        const int t = i < nEvery ? i * kNodeEvery : nodeT[i];
        if (i < nEvery) nodeT[i] = t;
        nodeOff[i] = INT_MIN;
        if (node[t] != i) continue;                      // an open one
        for (int e = 0; e < 2; ++e) {
          int u = t, out = e, l, to, sum = 0, left = n + 1;
          do {
            beat(left);
            sum += glob.w(u, out);
            l = glob.link(u, out);
            u = l >> 1;
            out = 1 - (l & 1);
            to = node[u];
          } while (to < 0 && --left > 0);
          if (to < 0) { bad = true; to = i; }
          const_cast<int32_t*>(e ? nodes.l1 : nodes.l0)[i] = 2 * to + (l & 1);
          const_cast<int32_t*>(e ? nodes.w1 : nodes.w0)[i] = sum;
        }
      }
      g.sync();
      for (int i = nEvery + g.rank(); i < nEvery + nOpen; i += g.size()) {
        const int sz = loop_size(nodes, i, nEvery + nOpen + 2);
        if (sz < 0) bad = true;
        off[nodeT[i]] = sz;
      }
      g.sync();
    }
    if (g.any(bad)) { if (g.rank() == 0) fail(c, DEV_TRACE); return -1; }
  }
  OutRegion& O = c.O;
  int32_t* csz = O.csz + O.nc;
  const int room = O.ccap - O.nc;
  const int nl = g.list(n, [&](int t) { return off[t] > 0; },
                        [&](int t, bool hit, int before) {
                          if (hit) {
                            lead[before] = t;
                            if (before < room) csz[before] = off[t];
                          }
                          off[t] = INT_MIN;              // stays so in loops without a crossing
                        });
  if (nl > room) { if (g.rank() == 0) fail(c, DEV_CAPACITY); return -1; }
  g.sync();
  long long total = 0;
  for (int b = 0; b < nl; b += g.size()) {
    const int k = b + g.rank();
    const int v = k < nl ? csz[k] : 0;
    int tot;
    const int incl = g.incl_scan(v, tot);
    if (k < nl) off[lead[k]] = (int32_t)total + incl - v;
    total += tot;
  }
  if (O.nv + total > O.vcap) { if (g.rank() == 0) fail(c, DEV_CAPACITY); return -1; }
  g.sync();
  // ---- offsets of the segments
  for (int k = g.rank(); k < nl; k += g.size()) {
    const int t0 = lead[k], base = off[t0], in0 = start_end(t0);
    if (odd) {
      int u = t0, in = in0, v = end_p(t0, in0), o = base, steps = 0;
      do {
        beat(++steps);
        const Step r = step_of(u, in, v, -1);
        off[u] = in ? ~o : o;
        eV[u] = v;
        o += r.lp + r.lq;
        v = Q.nb(r.left);
        const int l = link(u, 1 - in);
        u = l >> 1;
        in = l & 1;
      } while (u != t0);
    } else if (shared) {
      loop_offsets(shrd, t0, in0, base, csz[k], off);
    } else if (nOpen > 0 && node[t0] >= nEvery) {
      loop_offsets(nodes, node[t0], in0, base, csz[k], nodeOff);
    } else {
      loop_offsets(glob, t0, in0, base, csz[k], off);
    }
  }
  g.sync();
  if constexpr (G::kGrid) {
    if (nOpen > 0) {                                     // from each node on to the next one
      for (int i = g.rank(); i < nEvery + nOpen; i += g.size()) {
        int o = nodeOff[i];
        if (o == INT_MIN) continue;
        int in = o < 0 ? 1 : 0, u = nodeT[i], steps = 0;
        if (in) o = ~o;
        do {
          beat(++steps);
          off[u] = in ? ~o : o;
          o += glob.w(u, 1 - in);
          const int l = glob.link(u, 1 - in);
          u = l >> 1;
          in = l & 1;
        } while (node[u] < 0);
      }
      g.sync();
    }
  }
  // ---- copy the pieces
  double2* out = reinterpret_cast<double2*>(O.xy) + O.nv;
  for (int b = 0; b < n; b += g.size()) {
    const int t = b + g.rank();
    Step r{0, 0, 0, 0, 1, 0};
    int op = t < n ? off[t] : INT_MIN, dp = 1;
    if (op != INT_MIN) {
      const int in = op < 0 ? 1 : 0, l = link(t, 1 - in);
      if (in) { op = ~op; dp = -1; }
      // the next segment's entry is the neighbour of the vertex at which Q is left
      r = step_of(t, in, odd ? eV[t] : end_p(t, in), P.nb(odd ? eV[l >> 1] : end_p(l >> 1, l & 1)));
    } else {
      op = 0;
    }
    warp_copy_runs(P, r.sp, r.lp, dp, out + op);
    warp_copy_runs(Q, r.sq, r.lq, r.dq, out + op + r.lp);
  }
  O.nv += total;
  O.nc += nl;
  g.sync();
  return 0;
}

// Tracing when neither ring has added vertices (rings in slot order): each run from V to
// the next vertex with the target entry/exit flag (or back at the start) is found with a
// group ballot and copied with coalesced stores.
template <class G>
__device__ bool grp_trace(const G& g, PairCtx& c) {
  Ring& P = c.R[0];
  OutRegion& O = c.O;
  long long budget = 4ll * (c.R[0].used + c.R[1].used) + 16;
  int from = 0;
  for (;;) {
    int I = grp_find_first(g, from, P.m, [&](int s) { return P.it(s) && P.lb(s) == L_CROSSING; });
    if (I >= P.m) break;
    O.begin();
    if (O.overflow) { if (g.rank() == 0) fail(c, DEV_CAPACITY); return false; }
    int side = 0, V = I;
    if (g.rank() == 0) P.it(V) = 0;
    g.sync();
    WalkRepeat again;
    do {
      Ring& C = c.R[side];
      const int m = C.m;
      if (again.seen(V, side)) { if (g.rank() == 0) fail(c, DEV_TRACE); return false; }
      int8_t st = toggled(C.ee(V));
      const int dir = ((st == E_EXIT) ^ c.uni) ? 1 : -1;
      int L = -1;
      for (int j0 = 1; j0 <= m && L < 0; j0 += g.size()) {
        int j = j0 + g.rank();
        bool hit = false;
        if (j <= m) {
          int w = V + dir * (j % m);
          w = (w % m + m) % m;
          hit = (C.ee(w) == st) || (side == 0 && w == I);
        }
        int f = g.first(hit);
        if (f >= 0) L = j0 + f;
      }
      if (L < 0) { if (g.rank() == 0) fail(c, DEV_TRACE); return false; }
      budget -= L;
      if (budget < 0) { if (g.rank() == 0) fail(c, DEV_TRACE); return false; }
      if (O.nv + L > O.vcap) { if (g.rank() == 0) fail(c, DEV_CAPACITY); return false; }
      for (int j0 = 1; j0 <= L; j0 += g.size()) {
        int j = j0 + g.rank();
        if (j <= L) {
          int w = V + dir * (j % m);
          w = (w % m + m) % m;
          C.it(w) = 0;
          O.xy[2 * (O.nv + j - 1)] = C.x(w);
          O.xy[2 * (O.nv + j - 1) + 1] = C.y(w);
        }
      }
      O.nv += L;
      if (g.rank() == 0) O.csz[O.nc] += L;
      int W = V + dir * (L % m);
      V = (W % m + m) % m;
      g.sync();
      if (!(side == 0 && V == I)) {
        int nb = C.nb(V);
        if (nb < 0) { if (g.rank() == 0) fail(c, DEV_TRACE); return false; }
        V = nb;
        side = 1 - side;
        if (g.rank() == 0) c.R[side].it(V) = 0;
        g.sync();
      }
    } while (!(side == 0 && V == I));
    O.end();
    from = I + 1;
  }
  return true;
}

// Vertices were added to the rings (linked in after their place, kept in slots past the
// merged ring): puts both rings back into slot order, so that they are traced like rings
// without added vertices.  Coordinates go through the free end of the pair's output region,
// the rest through scratch columns.
template <class G>
__device__ bool grp_linearize(const G& g, PairCtx& c) {
  for (int sd = 0; sd < 2; ++sd) {                       // to: new slot of each vertex
    Ring& A = c.R[sd];
    int added = 0;
    for (int b = 0; b < A.m; b += g.size()) {
      const int s = b + g.rank();
      int k = 0;
      if (s < A.m)
        for (int v = A.nx(s); v >= A.m && k <= A.used - A.m; v = A.nx(v)) ++k;
      int tot;
      const int at = s + added + g.incl_scan(k, tot) - k;
      if (s < A.m) {
        A.to(s) = at;
        int v = A.nx(s);
        for (int i = 1; i <= k; ++i) { A.to(v) = at + i; v = A.nx(v); }
      }
      added += tot;
    }
    if (A.m + added != A.used) return false;             // not reached from its place: left to the links
  }
  if (c.O.nv + max(c.R[0].used, c.R[1].used) > c.O.vcap) return false;
  g.sync();
  double2* stage = reinterpret_cast<double2*>(c.O.xy) + c.O.nv;
  for (int sd = 0; sd < 2; ++sd) {
    Ring& A = c.R[sd];
    const Ring& B = c.R[1 - sd];
    for (int s = g.rank(); s < A.used; s += g.size()) {
      const int at = A.to(s), nb = A.nb(s);
      stage[at] = A.xy(s);
      A.tn(at) = nb >= 0 && nb < B.used ? B.to(nb) : nb;
      A.tl(at) = (int)A.it(s) | ((int)(uint8_t)A.lb(s) << 8) | ((int)(uint8_t)A.ee(s) << 16);
    }
    g.sync();
    for (int s = g.rank(); s < A.used; s += g.size()) {
      A.xy(s) = stage[s];
      A.nb(s) = A.tn(s);
      const int v = A.tl(s);
      A.it(s) = (uint8_t)v;
      A.lb(s) = (int8_t)(v >> 8);
      A.ee(s) = (int8_t)(v >> 16);
      A.nx(s) = s + 1 < A.used ? s + 1 : 0;
      A.pv(s) = s > 0 ? s - 1 : A.used - 1;
    }
    g.sync();
  }
  c.R[0].m = c.R[0].used;
  c.R[1].m = c.R[1].used;
  return true;
}

// The clean-up of a long component by one warp: the lanes take consecutive parts of the
// forward pass, each assuming that the vertex before its part is kept.  Where that was
// wrong the part is gone over again from the vertex that was kept, until nothing changes
// (lane 0's part is right from the start, so at most 32 times; parts agree after one
// or two).  Returns how many vertices are kept; writes them to dst when it is given.
template <class G>
__device__ int warp_cleanup_component(const G& g, const double2* src, double2* dst, int n, double eps) {
  const int lane = (int)lane_id();
  auto area_is_small = [eps](double2 a, double2 b, double2 c) { return fabs(area2(a.x, a.y, b.x, b.y, c.x, c.y)) < eps; };
  const double2 last = src[n - 1];
  int r = 0;
  while (r < n && (r == n - 1 ? 0.0 < eps : area_is_small(last, src[r], src[r + 1]))) g.beat(++r);
  if (r >= n) return 0;
  const int len = n - 1 - r, per = (len + 31) / 32;
  const int a = r + 1 + min(lane * per, len), b = r + 1 + min((lane + 1) * per, len);
  const double2 first = src[r];
  // decisions of one part from a kept vertex on
  auto pass = [&](int prev, double2* out, int& kept) {
    kept = 0;
    double2 k = src[prev];
    for (int j = a; j < b; ++j) {
      const double2 v = src[j], nx = j + 1 < n ? src[j + 1] : first;
      if (area_is_small(k, v, nx)) continue;
      if (out) out[kept] = v;
      ++kept;
      k = v;
      prev = j;
    }
    return prev;                                         // the last kept vertex so far
  };
  int from = a - 1, kept = 0;                            // (a - 1 >= r)
  int end = pass(from, nullptr, kept);
  for (int round = 0; round < 32; ++round) {
    if (lane == 0 && per > 1023) g.beat(1023);          // (once a round: a beat per vertex took 0.5 of the large pair's 48 ms)
    int before = __shfl_up_sync(kFull, end, 1);
    if (lane == 0) before = r;
    const bool wrong = before != from;
    if (!__any_sync(kFull, wrong)) break;
    if (wrong) { from = before; end = pass(from, nullptr, kept); }
  }
  const int incl = warp_incl_scan(kept), total = __shfl_sync(kFull, incl, 31) + 1;
  if (dst) {
    if (lane == 0) dst[0] = first;
    int again;
    pass(from, dst + 1 + incl - kept, again);
  }
  return total;
}

// Clean-up (polyclip.h:791-807).  One-thread pairs take their components one after another
// with the sequential pass.  Wider groups first count what each component keeps -- a warp
// takes 32 components, short ones a lane each, long ones all lanes together -- and leave
// the result in place when nothing is removed; else the kept vertices go, in order, to the
// free part of the pair's output region behind the traced ones (*where: its offset there).
// sequential(): one member's clean-up, component after component.
template <class G, class S>
__device__ void grp_cleanup(const G& g, PairCtx& c, int32_t* outNC, int64_t* outNV, int64_t* where, S sequential) {
  OutRegion& O = c.O;
  if constexpr (G::kSolo) {
    double2* xy = reinterpret_cast<double2*>(O.xy);
    int64_t vin = 0, vout = 0;
    int kc = 0;
    for (int k = 0; k < O.nc; ++k) {
      const int n = O.csz[k];
      double2* v = xy + vin;
      bool any = n == 0;
      double2 p = v[n > 0 ? n - 1 : 0], q = v[0];
      for (int j = 0; j < n && !any; ++j) {
        const double2 nx = v[j + 1 < n ? j + 1 : 0];
        any = fabs(area2(p.x, p.y, q.x, q.y, nx.x, nx.y)) < c.eps_clean;
        p = q;
        q = nx;
      }
      int kept = n;
      if (any) kept = seq_cleanup_component<true>(v, xy + vout, n, c.eps_clean);
      else if (vout != vin) for (int j = 0; j < n; ++j) xy[vout + j] = v[j];
      vin += n;
      if (kept == 0) continue;
      if (kc != k || any) O.csz[kc] = kept;
      ++kc;
      vout += kept;
    }
    *outNC = kc;
    *outNV = vout;
  } else {
    constexpr int kShortComp = 32;
    const int nc = O.nc, lane = (int)lane_id();
    if (nc == 0 || 2 * O.nv > O.vcap) {                  // (the region has room for twice a well-formed trace)
      if (g.rank() == 0) sequential();
      g.sync();
      return;
    }
    const double2* xy = reinterpret_cast<const double2*>(O.xy);
    double2* out = reinterpret_cast<double2*>(O.xy) + O.nv;
    int32_t* start = &c.R[0].tn(0);                      // the trace's scratch is free now
    int32_t* keptA = &c.R[0].ls(0);
    int32_t* dstA = &c.R[0].tl(0);
    int carry = 0;
    for (int b = 0; b < nc; b += g.size()) {
      const int k = b + g.rank();
      const int v = (k < nc) ? O.csz[k] : 0;
      int tot;
      const int incl = g.incl_scan(v, tot);
      if (k < nc) start[k] = carry + incl - v;
      carry += tot;
    }
    g.sync();
    bool removed = false;
    for (int b = 0; b < nc; b += g.size()) {
      const int k = b + g.rank();
      const int n = k < nc ? O.csz[k] : 0, s0 = k < nc ? start[k] : 0;
      int kept = n;
      if (n > 0 && n <= kShortComp) {
        const double2* v = xy + s0;
        double2 p = v[n - 1], q = v[0];
        bool any = false;
        for (int j = 0; j < n; ++j) {
          const double2 nx = v[j + 1 < n ? j + 1 : 0];
          if (fabs(area2(p.x, p.y, q.x, q.y, nx.x, nx.y)) < c.eps_clean) { any = true; break; }
          p = q;
          q = nx;
        }
        if (any) kept = seq_cleanup_component<false>(v, nullptr, n, c.eps_clean);
      }
      unsigned longs = __ballot_sync(kFull, n > kShortComp);
      while (longs) {
        const int src = __ffs(longs) - 1;
        longs &= longs - 1;
        const int ln = __shfl_sync(kFull, n, src);
        const double2* v = xy + __shfl_sync(kFull, s0, src);
        bool any = false;
        for (int j0 = 0; j0 < ln && !any; j0 += 128) {
          bool small = false;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = j0 + u * 32 + lane;
            if (j >= ln) continue;
            const double2 p = v[j > 0 ? j - 1 : ln - 1], q = v[j], nx = v[j + 1 < ln ? j + 1 : 0];
            if (fabs(area2(p.x, p.y, q.x, q.y, nx.x, nx.y)) < c.eps_clean) small = true;
          }
          any = __any_sync(kFull, small) != 0;
        }
        const int lk = any ? warp_cleanup_component(g, v, nullptr, ln, c.eps_clean) : ln;
        if (lane == src) kept = lk;
      }
      if (k < nc) {
        keptA[k] = kept;
        if (kept != n) removed = true;
      }
    }
    g.sync();
    if (!g.any(removed)) {
      if (g.rank() == 0) { *outNC = nc; *outNV = O.nv; }
      return;
    }
    int total = 0;
    for (int b = 0; b < nc; b += g.size()) {
      const int k = b + g.rank();
      const int v = (k < nc) ? keptA[k] : 0;
      int tot;
      const int incl = g.incl_scan(v, tot);
      if (k < nc) dstA[k] = total + incl - v;
      total += tot;
    }
    g.sync();
    for (int b = 0; b < nc; b += g.size()) {
      const int k = b + g.rank();
      const int n = k < nc ? O.csz[k] : 0, s0 = k < nc ? start[k] : 0, kept = k < nc ? keptA[k] : 0;
      const int d0 = k < nc ? dstA[k] : 0;
      if (n <= kShortComp && kept > 0) {
        if (kept == n) for (int j = 0; j < n; ++j) out[d0 + j] = xy[s0 + j];
        else seq_cleanup_component<true>(xy + s0, out + d0, n, c.eps_clean);
      }
      unsigned longs = __ballot_sync(kFull, n > kShortComp && kept > 0);
      while (longs) {
        const int src = __ffs(longs) - 1;
        longs &= longs - 1;
        const int ln = __shfl_sync(kFull, n, src), lk = __shfl_sync(kFull, kept, src);
        const double2* v = xy + __shfl_sync(kFull, s0, src);
        double2* d = out + __shfl_sync(kFull, d0, src);
        if (lk == ln) for (int j = lane; j < ln; j += 32) d[j] = v[j];
        else warp_cleanup_component(g, v, d, ln, c.eps_clean);
      }
    }
    g.sync();
    // sizes of the components that are left
    const int left = g.list(nc, [&](int k) { return keptA[k] > 0; },
                            [&](int k, bool hit, int before) { if (hit) dstA[before] = keptA[k]; });
    g.sync();
    for (int k = g.rank(); k < left; k += g.size()) O.csz[k] = dstA[k];
    if (g.rank() == 0) { *outNC = left; *outNV = total; *where += O.nv; }
    g.sync();
  }
}

// Pulls a pair's ring arrays into L1 in one burst, one request per 128-byte line, so the
// labelling phases (each of which touches some of the arrays first) do not pay a DRAM
// round trip each.
__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

template <class G>
__device__ void prefetch_ring(const G& g, const Ring& R) {
  for (int s = g.rank() * 8; s < R.m; s += g.size() * 8) {
    prefetch_l1(&R.xy(s));
    if ((s & 31) == 0) { prefetch_l1(&R.nx(s)); prefetch_l1(&R.pv(s)); prefetch_l1(&R.nb(s)); }
    if ((s & 127) == 0) { prefetch_l1(&R.it(s)); prefetch_l1(&R.lb(s)); prefetch_l1(&R.ee(s)); prefetch_l1(&R.fl(s)); }
  }
}

// What a grid leaves of a pair to one thread: 1 the trace and the clean-up, 2 the clean-up
// (rings of m slots, `used` with the added vertices; components and vertices already out).
struct BigSeq { int from, mP, mQ, usedP, usedQ, nc; int64_t nv; };

// Arguments of the labelling kernels (one struct so the warp and block kernels agree).
struct LabelArgs {
  PairDev D;
  int64_t K;
  const int32_t* mP; const int32_t* mQ;
  const int64_t* regP; const int64_t* regQ;
  const int64_t* regSizeP; const int64_t* regSizeQ;
  RingSet SP, SQ;
  double* outXY; int64_t* outVOff; const int64_t* outVCap;
  int32_t* outCsz; const int64_t* outCOff; const int32_t* outCCap;
  int32_t* outNC; int64_t* outNV;
  ClipParams prm;
  int* err;
  const unsigned long long* midCount;
  unsigned long long* midNext; // work-stealing cursor of the block kernel
  int blockLoopCap;           // segments the block kernel's shared loop table holds (0: none)
  // The one-thread, warp and block pairs in size order, largest first (label_order_kernel):
  // the one-thread kernel takes order[0, nTile), the warp kernel order[nTile, nTile + nWarp),
  // the block kernel the *midCount entries after those.
  const uint32_t* order;
  int64_t nTile, nWarp;
  BigSeq* seq = nullptr;      // grid kernel: set when a pair is left to the sequential phases
};

// One pair labelled and traced by group g.  The group phases give the sequential result
// whenever neighbour links are one-to-one (then labels written through a link never
// collide) and chains are well formed; otherwise member 0 runs the sequential phases from
// the first one that could differ.
template <int EX, class G>
__device__ void label_trace_pair(const G& g, const LabelArgs& a, int64_t k) {
  const bool lead = g.rank() == 0;
  int32_t* outNC = a.outNC + k;
  int64_t* outNV = a.outNV + k;
  PairCtx c;
  c.R[0] = ring_of(a.SP, a.regP[k], a.mP[k], (int)a.regSizeP[k]);
  c.R[1] = ring_of(a.SQ, a.regQ[k], a.mQ[k], (int)a.regSizeQ[k]);
  c.O.xy = a.outXY + 2 * a.outVOff[k]; c.O.csz = a.outCsz + a.outCOff[k];
  c.O.vcap = a.outVCap[k]; c.O.ccap = a.outCCap[k];
  c.O.nv = 0; c.O.nc = 0; c.O.overflow = false;
  c.uni = a.prm.union_mode != 0;
  c.eps_clean = a.prm.eps_clean;
  c.err = a.err;
  c.status = a.D.status + k;
  c.noInter[0] = c.noInter[1] = c.ident[0] = c.ident[1] = false;
  if constexpr (!G::kGrid) {
    prefetch_ring(g, c.R[0]);
    prefetch_ring(g, c.R[1]);
  }
  // what a grid leaves to a kernel of one thread
  auto leave = [&](int from) {
    if (lead) *a.seq = BigSeq{from, c.R[0].m, c.R[1].m, c.R[0].used, c.R[1].used, c.O.nc, c.O.nv};
  };
  const bool oneToOne = grp_links_one_to_one(g, c.R[0], c.R[1]);
  if constexpr (G::kSolo) {
    if (!oneToOne) { seq_pair_from<EX>(c, 1, outNC, outNV); return; }
    grp_step1<EX>(g, c);
    if (!grp_step2(g, c)) { seq_pair_from<EX>(c, 2, outNC, outNV); return; }
  } else {
    // Links that are not one-to-one and malformed chains leave only the chains' resolution
    // (over the listed chain starts) and, for the former, the trace to one member.
    if (oneToOne) grp_step1<EX>(g, c);
    else grp_step1_shared<EX>(g, c);
    if (!oneToOne || !grp_step2(g, c)) {
      Ring& P = c.R[0];
      const int n = g.list(P.m, [&](int s) { return P.it(s) && (P.lb(s) == L_LEFT_ON || P.lb(s) == L_RIGHT_ON); },
                           [&](int s, bool hit, int before) { if (hit) P.ls(before) = s; });
      g.sync();
      if (lead) seq_step2(c, n, [&g](int step) { g.beat(step); });
      g.sync();
    }
  }
  grp_step35<EX>(g, c);
  int tempAfter[2], tempSlot[2];
  if (!grp_step4<EX>(g, c, tempAfter, tempSlot)) return;
  if (grp_any_split(g, c.R[0], c.R[1])) {
    bool ok = true;
    int n = -1;
    if constexpr (!G::kSolo) {
      Ring& P = c.R[0];
      n = g.list(P.used, [&](int s) { return (P.fl(s) & 1) != 0; }, [&](int s, bool hit, int before) { if (hit) P.ls(before) = s; });
      g.sync();
    }
    if (lead) ok = seq_step5<EX>(c, n, [&g](int step) { g.beat(step); });
    ok = g.bcast0((int)ok);
    c.R[0].used = g.bcast0(c.R[0].used);
    c.R[1].used = g.bcast0(c.R[1].used);
    g.sync();
    if (!ok) return;
  }
  grp_step6(g, c);
  bool added = c.R[0].used != c.R[0].m || c.R[1].used != c.R[1].m;
  if constexpr (!G::kSolo) {
    if (added && oneToOne) added = !grp_linearize(g, c);
  }
  if (added || !oneToOne) {
    // trace through the next/prev links on one member
    if constexpr (G::kGrid) { leave(1); return; }
    int ok = 1;
    if (lead) ok = seq_trace(c) ? 1 : 0;
    ok = g.bcast0(ok);
    c.O.nv = g.bcast0((long long)c.O.nv);
    c.O.nc = g.bcast0(c.O.nc);
    c.O.overflow = g.bcast0((int)c.O.overflow) != 0;
    g.sync();
    if (!ok) return;
  } else {
    int r;
    if constexpr (G::kSolo) r = grp_trace_runs_slots(g, c);
    else r = grp_trace_loops(g, c);
    if (r < 0) return;
    if (r > 0) {
      if constexpr (G::kGrid) { leave(1); return; }
      else if (!grp_trace(g, c)) return;
    }
  }
  if (c.O.overflow) {
    if (lead) fail(c, DEV_CAPACITY);
    return;
  }
  grp_cleanup(g, c, outNC, outNV, a.outVOff + k, [&]() {
    if constexpr (G::kGrid) leave(2);
    else seq_cleanup(c, outNC, outNV);
  });
}

// Two register budgets for the warp and one-thread kernels.  kWide (batches of at least
// ClipParams::wide_label_min pairs): 6 blocks of 128 (at most 80 registers) here and 12 blocks (40
// registers) for the tiles below -- both kernels wait on dependent loads, and on a full
// GPU the occupancy pays for the spills (label stage 2.59 -> 2.11 ms from the tile kernel,
// -0.07 ms from this one; with the column-buffer rings, 12 tile blocks measured 2.00 ms
// against 2.08 ms for 16).  Small batches (serving) leave most SMs idle, so there the
// kernels keep 4 blocks and spill nothing.  Exact-predicate instances always keep 4
// blocks: their expansion arithmetic would spill.
template <int EX, int kWide>
__global__ void __launch_bounds__(128, (kWide && !EX) ? 6 : 4)
label_trace_kernel(LabelArgs a) {
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= a.nWarp) return;
  WarpGroup g;
  label_trace_pair<EX>(g, a, (int64_t)a.order[a.nTile + w]);
}

// Pairs whose merged rings have at most ClipParams::tile_label_max slots: one thread per pair
// (SoloGroup, measured slightly faster than 2-lane tiles on the batched workload), the
// pairs in size order so that the 32 pairs of a warp take about as long as each other.
template <int EX, int kWide>
__global__ void __launch_bounds__(128, (kWide && !EX) ? 12 : 4)
label_trace_tile_kernel(LabelArgs a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nTile) return;
  SoloGroup g;
  label_trace_pair<EX>(g, a, (int64_t)a.order[i]);
}

// sizes in the labelling order, and the scanned offsets back to pair order
__global__ void permute_sizes_kernel(const uint32_t* __restrict__ order, int64_t K, const int64_t* __restrict__ sP,
                                     const int64_t* __restrict__ sQ, int64_t* __restrict__ oP, int64_t* __restrict__ oQ) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K) return;
  const uint32_t k = order[i];
  oP[i] = sP[k];
  oQ[i] = sQ[k];
}

__global__ void unpermute_offsets_kernel(const uint32_t* __restrict__ order, int64_t K,
                                         const int64_t* __restrict__ offP, const int64_t* __restrict__ offQ,
                                         int64_t* __restrict__ regP, int64_t* __restrict__ regQ) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K) return;
  const uint32_t k = order[i];
  regP[k] = offP[i];
  regQ[k] = offQ[i];
}

// Sort keys of the pairs by labelling class and size, for one 8-bit radix pass: one-thread
// pairs 0..84, warp pairs 85..169, block pairs 170..254 (85 size buckets each, largest
// first; the block class on a log scale, so that its largest pairs start first and do not
// trail the stage), the rest 255.  Class counts: cnt[2] one-thread, cnt[3] warp, cnt[0] block,
// cnt[4] grid.
__global__ void label_order_kernel(const int32_t* __restrict__ mP, const int32_t* __restrict__ mQ,
                                   const int32_t* __restrict__ status, int64_t K, int64_t tileMax, int64_t midMin,
                                   int64_t bigMin, uint64_t* __restrict__ key, uint32_t* __restrict__ val,
                                   unsigned long long* __restrict__ cnt) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  const int64_t slots = (int64_t)mP[k] + mQ[k];
  const int64_t tl = tileMax < midMin ? tileMax : midMin;
  uint64_t kk = 255;
  if (status[k] == 0 && slots <= midMin) {
    if (slots <= tl) {
      kk = 84 - (uint64_t)((slots * 85) / (tl + 1));
      atomicAdd(cnt + 2, 1ull);
    } else {
      kk = 169 - (uint64_t)(((slots - tl) * 85) / (midMin - tl + 1));
      atomicAdd(cnt + 3, 1ull);
    }
  } else if (status[k] == 0 && slots <= bigMin) {
    const double r = log2((double)slots / (double)midMin) / log2((double)bigMin / (double)midMin);
    const int b = (int)fmin(84.0, fmax(0.0, 85.0 * r));
    kk = 254 - (uint64_t)b;
    atomicAdd(cnt, 1ull);
  } else if (status[k] == 0) {
    atomicAdd(cnt + 4, 1ull);
  }
  key[k] = kk;
  val[k] = (uint32_t)k;
}

// Pairs with mid_label_min < slots <= big_label_min: persistent blocks take pairs from the
// list through an atomic cursor (work stealing), one block of kBlockLabelThreads per pair.
template <int EX>
__global__ void __launch_bounds__(kBlockLabelThreads)
label_trace_block_kernel(LabelArgs a) {
  __shared__ long long sm[kBlockScratch];
  __shared__ long long next;
  extern __shared__ uint32_t loopTable[];
  BlockGroup g{sm, loopTable, a.blockLoopCap};
  const unsigned long long n = *a.midCount;
  for (;;) {
    if (threadIdx.x == 0) next = (long long)atomicAdd(a.midNext, 1ull);
    __syncthreads();
    const long long i = next;
    __syncthreads();
    if (i >= (long long)n) return;
    label_trace_pair<EX>(g, a, (int64_t)a.order[a.nTile + a.nWarp + i]);
    __syncthreads();
  }
}


// ================================================================ grid path for huge pairs
// Pairs whose merged rings exceed ClipParams::big_label_min slots are labelled and traced
// by the whole GPU, one after another in one cooperative launch: the same phases with the
// grid as the group.  A kernel per phase with host reads between them, the loops found by
// pointer jumping over all runs, took 182 ms for the 400,000 x 200,000-vertex pair (5.8e7
// slots, 2.9e7 crossings).
__global__ void big_label_list_kernel(const int32_t* __restrict__ mP, const int32_t* __restrict__ mQ,
                                      const int32_t* __restrict__ status, int64_t K, int64_t minSlots,
                                      int64_t* __restrict__ list, unsigned long long* __restrict__ n) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K || status[k] != 0) return;
  if ((int64_t)mP[k] + mQ[k] > minSlots) list[atomicAdd(n, 1ull)] = k;
}

template <int EX>
__global__ void __launch_bounds__(kBlockLabelThreads)
label_trace_grid_kernel(LabelArgs a, const int64_t* __restrict__ list, int n, GridScratch* gs, BigSeq* seq) {
  __shared__ long long sm[kBlockScratch];
  __shared__ int gone;
  const GridGroup g(BlockGroup{sm, nullptr, 0}, gs, a.err, a.prm.grid_wait, &gone);
  for (int i = 0; i < n; ++i) {
    a.seq = seq + i;
    label_trace_pair<EX>(g, a, list[i]);
    g.sync();
  }
}

// the pairs that the grid left to the sequential phases, a thread each
template <int EX>
__global__ void big_seq_kernel(LabelArgs a, const int64_t* __restrict__ list, const BigSeq* __restrict__ seq,
                               const GridScratch* __restrict__ gs) {
  const BigSeq q = seq[blockIdx.x];
  if (q.from == 0 || gs->dead) return;                   // (a grid that gave up leaves rings half done)
  const int64_t k = list[blockIdx.x];
  PairCtx c;
  c.R[0] = ring_of(a.SP, a.regP[k], q.mP, (int)a.regSizeP[k]);
  c.R[1] = ring_of(a.SQ, a.regQ[k], q.mQ, (int)a.regSizeQ[k]);
  c.R[0].used = q.usedP;
  c.R[1].used = q.usedQ;
  c.O.xy = a.outXY + 2 * a.outVOff[k]; c.O.csz = a.outCsz + a.outCOff[k];
  c.O.vcap = a.outVCap[k]; c.O.ccap = a.outCCap[k];
  c.O.nv = q.nv; c.O.nc = q.nc; c.O.overflow = false;
  c.uni = a.prm.union_mode != 0;
  c.eps_clean = a.prm.eps_clean;
  c.err = a.err;
  c.status = a.D.status + k;
  c.noInter[0] = c.noInter[1] = c.ident[0] = c.ident[1] = false;
  if (q.from == 2 || seq_trace(c)) seq_cleanup(c, a.outNC + k, a.outNV + k);
}

// ---------------------------------------------------------------- G8 compaction
__global__ void out_sizes_kernel(const int32_t* __restrict__ mP, const int32_t* __restrict__ mQ,
                                 const int32_t* __restrict__ nrec, const int32_t* __restrict__ status,
                                 int64_t K, int64_t* __restrict__ vcap, int32_t* __restrict__ ccap) {
  int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (k >= K) return;
  if (status[k] != 0) { vcap[k] = 0; ccap[k] = 0; return; }
  int64_t ext = (int64_t)mP[k] + mQ[k] + 4 * ((int64_t)nrec[k] + 1);
  vcap[k] = 2 * ext + 16;
  ccap[k] = mP[k] + 2 * nrec[k] + 8;
}

// A warp copies a pair's result; results of more than kCopyPiece vertices are listed in pieces
// of that size for out_compact_pieces_kernel (one warp on the 5.4e6 vertices of the large
// pair took 31 ms).
constexpr int kCopyPiece = 4096;
struct CopyPieces { int2* at; unsigned* n; };

__global__ void __launch_bounds__(kThreads, 8)   // 32 registers: compact 0.33 -> 0.20 ms
out_compact_kernel(int64_t K, const double2* __restrict__ xy, const int64_t* __restrict__ vOff,
                   const int32_t* __restrict__ csz, const int64_t* __restrict__ cOff,
                   const int32_t* __restrict__ nc, const int64_t* __restrict__ nv,
                   const int64_t* __restrict__ fVOff, const int64_t* __restrict__ fCOff,
                   double2* __restrict__ oxy, int32_t* __restrict__ ocsz, CopyPieces pieces) {
  int64_t w = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  if (w >= K) return;
  const double2* s = xy + vOff[w];
  double2* d = oxy + fVOff[w];
  const int64_t n = nv[w];
  const int comps = nc[w];
  if (n > kCopyPiece) {
    // the pieces of the vertices, then those of the component sizes (as negative numbers)
    const int pv = (int)((n + kCopyPiece - 1) / kCopyPiece), pc = (comps + kCopyPiece - 1) / kCopyPiece;
    unsigned at = 0;
    if (lane_id() == 0) at = atomicAdd(pieces.n, (unsigned)(pv + pc));
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int i = lane_id(); i < pv + pc; i += 32) pieces.at[at + i] = make_int2((int)w, i < pv ? i : ~(i - pv));
    return;
  }
  for (int64_t i = lane_id(); i < n; i += 32) d[i] = s[i];
  for (int i = lane_id(); i < comps; i += 32) ocsz[fCOff[w] + i] = csz[cOff[w] + i];
}

__global__ void __launch_bounds__(kThreads)
out_compact_pieces_kernel(CopyPieces pieces, const double2* __restrict__ xy, const int64_t* __restrict__ vOff,
                          const int32_t* __restrict__ csz, const int64_t* __restrict__ cOff,
                          const int32_t* __restrict__ nc, const int64_t* __restrict__ nv,
                          const int64_t* __restrict__ fVOff, const int64_t* __restrict__ fCOff,
                          double2* __restrict__ oxy, int32_t* __restrict__ ocsz) {
  const unsigned n = *pieces.n;
  for (unsigned p = blockIdx.x; p < n; p += gridDim.x) {
    const int2 pc = pieces.at[p];
    const int64_t w = pc.x;
    if (pc.y >= 0) {
      const int64_t a = (int64_t)pc.y * kCopyPiece, b = min(a + kCopyPiece, nv[w]);
      const double2* s = xy + vOff[w];
      double2* d = oxy + fVOff[w];
#pragma unroll 4
      for (int64_t i = a + threadIdx.x; i < b; i += kThreads) d[i] = s[i];
    } else {
      const int a = ~pc.y * kCopyPiece, b = min(a + kCopyPiece, nc[w]);
      for (int i = a + (int)threadIdx.x; i < b; i += kThreads) ocsz[fCOff[w] + i] = csz[cOff[w] + i];
    }
  }
}

}  // namespace

int run_clip(const LayerDev& Lb, const LayerDev& Lo, const int32_t* d_pid, const int32_t* d_qid,
             int64_t K, const ClipParams& prm, Arena& A, ClipDev& C, int* d_err, int64_t* hs,
             cudaStream_t s, Marks* mk, cudaStream_t aux, RingExport* ex, cudaStream_t aux2,
             const double* mbrB, const double* mbrO, const JoinEdges* je) {
  Marks dummy;
  if (!mk) mk = &dummy;
  C = ClipDev();
  const JoinEdges jed = je ? *je : JoinEdges{};
  mk->mark("clip:start", s);
  C.n_pairs = K;
  if (K <= 0) return ST_OK;
  auto sync = [&]() { return cudaStreamSynchronize(s) == cudaSuccess; };
  // layer MBRs (same definition as the join's)
  const double* mb = mbrB;
  const double* mo = mbrO;
  if (!mb) {
    double* m = A.take_n<double>(4 * Lb.n);
    if (!m) return ST_OUT_OF_MEMORY;
    layer_mbrs(Lb, m, s);
    mb = m;
  }
  if (!mo) {
    double* m = A.take_n<double>(4 * Lo.n);
    if (!m) return ST_OUT_OF_MEMORY;
    layer_mbrs(Lo, m, s);
    mo = m;
  }
  // ---- G0 setup
  PairDev D;
  D.pS = A.take_n<int64_t>(K); D.qS = A.take_n<int64_t>(K);
  D.nP = A.take_n<int32_t>(K); D.nQ = A.take_n<int32_t>(K);
  D.pSide = A.take_n<int8_t>(K); D.cmbr = A.take_n<double>(4 * K);
  C.status = D.status = A.take_n<int32_t>(K);
  C.swapped = A.take_n<int32_t>(K);
  C.count1 = A.take_n<int64_t>(K);
  int32_t* cP = A.take_n<int32_t>(K);
  int32_t* cQ = A.take_n<int32_t>(K);
  int64_t* offP = A.take_n<int64_t>(K);
  int64_t* offQ = A.take_n<int64_t>(K);
  int64_t* nchunk = A.take_n<int64_t>(K);
  int64_t* chunkOff = A.take_n<int64_t>(K);
  int64_t* eoffP = A.take_n<int64_t>(K);
  int64_t* eoffQ = A.take_n<int64_t>(K);
  // totals and counters, cleared at once: 0-15 totals, 16 binned pairs, 20-27 labelling
  // classes, 28-31 heavy and mid edges, 32 long pairs of the edge filter
  int64_t* tot = A.take_n<int64_t>(40);
  void* stK = A.take(scan_temp_bytes(K));
  if (!D.pS || !D.qS || !D.nP || !D.nQ || !D.pSide || !D.cmbr || !D.status || !C.swapped || !C.count1 ||
      !cP || !cQ || !offP || !offQ || !nchunk || !chunkOff || !eoffP || !eoffQ || !tot || !stK)
    return ST_OUT_OF_MEMORY;
  cudaMemsetAsync(tot, 0, 40 * sizeof(int64_t), s);
  { setup_kernel<<<blocks_for(K), kThreads, 0, s>>>(Lb, Lo, d_pid, d_qid, K, mb, mo, D, C.swapped, prm.no_swap); note_launch(); }
  // The narrow-tile and whole-warp passes of the edge filter take disjoint pairs (by size):
  // with an auxiliary stream the warp pass runs beside the tile pass.
  cudaEvent_t fev[2] = {nullptr, nullptr};
  const bool two = aux && cudaEventCreateWithFlags(&fev[0], cudaEventDisableTiming) == cudaSuccess &&
                   cudaEventCreateWithFlags(&fev[1], cudaEventDisableTiming) == cudaSuccess;
  struct EvGuard { cudaEvent_t* e; ~EvGuard() { for (int i = 0; i < 2; ++i) if (e[i]) cudaEventDestroy(e[i]); } } fguard{fev};
  cudaStream_t sw = two ? aux : s;
  auto fork_aux = [&]() { if (two) { cudaEventRecord(fev[0], s); cudaStreamWaitEvent(aux, fev[0], 0); } };
  auto join_aux = [&]() { if (two) { cudaEventRecord(fev[1], aux); cudaStreamWaitEvent(s, fev[1], 0); } };
  // ---- G1 edge filter: narrow tiles, warps, and blocks for the pairs too long for a warp
  // (left out where the join or the layers' sizes rule such pairs out); a batch of fewer
  // pairs than blocks takes a block per pair throughout
  const bool fewPairs = K <= kFilterLongBlocks;
  const bool longPairs = !fewPairs && jed.max_ring > kLongRing &&
                         !(Lb.nverts > 0 && Lo.nverts > 0 && Lb.nverts + Lo.nverts <= kLongRing);
  LongPairs lpF;
  if (longPairs) {
    lpF.ids = A.take_n<int32_t>(K);
    lpF.n = reinterpret_cast<unsigned*>(tot + 32);
    if (!lpF.ids) return ST_OUT_OF_MEMORY;
  }
  auto edge_filter = [&](auto mode, int32_t* lp, int32_t* lq) {
    constexpr int kMode = decltype(mode)::value;
    if (fewPairs) {
      edge_filter_long_kernel<kMode><<<(unsigned)K, kFilterLongThreads, 0, s>>>(Lb, Lo, D, cP, cQ, offP, offQ, lp, lq, jed,
                                                                              LongPairs{}, (int)K);
      note_launch();
      return;
    }
    fork_aux();
    { edge_filter_kernel<kMode, kFilterTile><<<(unsigned)((K * kFilterTile + kThreads - 1) / kThreads), kThreads, 0, s>>>(
          Lb, Lo, D, K, cP, cQ, offP, offQ, lp, lq, -1, kFilterTileMax, jed, LongPairs{}); note_launch(); }
    { edge_filter_kernel<kMode, 32><<<blocks_for_warps(K), kThreads, 0, sw>>>(
          Lb, Lo, D, K, cP, cQ, offP, offQ, lp, lq, kFilterTileMax, longPairs ? kLongRing : INT64_MAX, jed, lpF); note_launch(); }
    if (longPairs)
      { edge_filter_long_kernel<kMode><<<kFilterLongBlocks, kFilterLongThreads, 0, sw>>>(Lb, Lo, D, cP, cQ, offP, offQ, lp,
                                                                                       lq, jed, lpF, 0); note_launch(); }
    join_aux();
  };
  edge_filter(std::integral_constant<int, 0>{}, nullptr, nullptr);
  exclusive_scan_i32(cP, offP, K, tot + 0, stK, d_err, s);
  exclusive_scan_i32(cQ, offQ, K, tot + 1, stK, d_err, s);
  exclusive_scan_i32(D.nP, eoffP, K, tot + 2, stK, d_err, s);
  exclusive_scan_i32(D.nQ, eoffQ, K, tot + 3, stK, d_err, s);
  int64_t* bigList = A.take_n<int64_t>(K);
  unsigned long long* nBig = reinterpret_cast<unsigned long long*>(tot + 16);
  if (!bigList) return ST_OUT_OF_MEMORY;
  { chunk_count_kernel<<<blocks_for(K), kThreads, 0, s>>>(cP, cQ, K, nchunk, bigList, nBig, prm.bin_grid); note_launch(); }
  exclusive_scan_i64(nchunk, chunkOff, K, tot + 4, stK, d_err, s);
  mk->mark("clip:setup+filter", s);
  cudaMemcpyAsync(hs, tot, 5 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(hs + 5, nBig, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  if (!sync()) return ST_CUDA_ERROR;
  const int64_t nLP = hs[0], nLQ = hs[1], nEP = hs[2], nEQ = hs[3], nCh = hs[4];
  const int nBigPairs = (int)hs[5];
  int32_t* LP = A.take_n<int32_t>(nLP);
  int32_t* LQ = A.take_n<int32_t>(nLQ);
  // Count + emit in one pass (intersect_fused_kernel) unless the records are exported:
  // the export keeps them in (pair, P edge, Q edge) order.
  const bool fused = prm.fused_emit && !ex;
  int32_t* chunkPair = A.take_n<int32_t>(nCh);
  int32_t* chunkRec = nullptr;
  int32_t* chunkQ = nullptr;
  int64_t* recScan = nullptr;
  int64_t* qScan = nullptr;
  void* stC = nullptr;
  int32_t* pairRec = nullptr;
  int32_t* pairQ = nullptr;
  if (!fused) {
    chunkRec = A.take_n<int32_t>(nCh);
    chunkQ = A.take_n<int32_t>(nCh);
    recScan = A.take_n<int64_t>(nCh);
    qScan = A.take_n<int64_t>(nCh);
    stC = A.take(scan_temp_bytes(std::max<int64_t>(nCh, 1)));
    if (!chunkRec || !chunkQ || !recScan || !qScan || !stC) return ST_OUT_OF_MEMORY;
  }
  // per-pair counts, cleared at once: binned records and Q hits, and the fused pass's
  int64_t* binRec = A.take_n<int64_t>(3 * K);
  if (!LP || !LQ || !chunkPair || !binRec) return ST_OUT_OF_MEMORY;
  int64_t* binQ = binRec + K;
  if (fused) {
    pairRec = reinterpret_cast<int32_t*>(binRec + 2 * K);
    pairQ = pairRec + K;
  }
  if (nCh > 0) { chunk_pair_kernel<<<blocks_for_warps(K), kThreads, 0, s>>>(chunkOff, nchunk, K, chunkPair); note_launch(); }
  cudaMemsetAsync(binRec, 0, 3 * K * sizeof(int64_t), s);
  edge_filter(std::integral_constant<int, 1>{}, LP, LQ);
  // The binned pairs (below) go to the auxiliary stream when there is one: fork here, before
  // the chunked count is queued on s, so that the two run side by side.
  cudaStream_t sb = s;
  cudaEvent_t bev[2] = {nullptr, nullptr};
  struct BinEvGuard { cudaEvent_t* e; ~BinEvGuard() { for (int i = 0; i < 2; ++i) if (e[i]) cudaEventDestroy(e[i]); } } bguard{bev};
  if (nBigPairs > 0 && aux && cudaEventCreateWithFlags(&bev[0], cudaEventDisableTiming) == cudaSuccess &&
      cudaEventCreateWithFlags(&bev[1], cudaEventDisableTiming) == cudaSuccess) {
    cudaEventRecord(bev[0], s);
    cudaStreamWaitEvent(aux, bev[0], 0);
    sb = aux;
  }
  // ---- G2 count: chunked pairs
  Records R{};
  unsigned long long* recTot = reinterpret_cast<unsigned long long*>(tot + 15);
  int64_t recCap = 0;
  auto take_records = [&](int64_t n) {
    n = std::max<int64_t>(n, 1);
    R.p = A.take_n<int32_t>(n); R.q = A.take_n<int32_t>(n);
    R.a = A.take_n<double>(n); R.b = A.take_n<double>(n);
    R.t = A.take_n<int8_t>(n); R.k = A.take_n<int32_t>(n);
    return R.p && R.q && R.a && R.b && R.t && R.k;
  };
  auto launch_fused = [&](bool countPairs) {
    if (nCh == 0) return;
    const FusedRecords F{recTot, recCap, countPairs ? pairRec : nullptr, pairQ};
    auto kern = prm.exact ? (prm.fused_emit == 2 ? intersect_fused_kernel<1, 1> : intersect_fused_kernel<1, 0>)
                          : (prm.fused_emit == 2 ? intersect_fused_kernel<0, 1> : intersect_fused_kernel<0, 0>);
    kern<<<blocks_for_warps(nCh), kThreads, 0, s>>>(Lb, Lo, D, chunkOff, nCh, cP, cQ, offP, offQ, LP, LQ, prm.eps, R,
                                                    chunkPair, F);
    note_launch();
  };
  if (fused) {
    // Capacity: the last clip's record count with room to spare, else a first guess,
    // never more than one record per chunked edge pair when nothing is binned.  A clip
    // that counts more records runs the pass again with arrays of the counted size.
    recCap = prm.rec_hint > 0 ? prm.rec_hint + prm.rec_hint / 4 + 4096 : kFirstRecordCap;
    if (nBigPairs == 0) recCap = std::min(recCap, std::max<int64_t>(nCh * kChunk, 1));
    if (!take_records(recCap)) return ST_OUT_OF_MEMORY;
    launch_fused(true);
  } else if (nCh > 0) {
    { (prm.exact ? intersect_kernel<0, 1> : intersect_kernel<0, 0>)<<<blocks_for_warps(nCh), kThreads, 0, s>>>(
        Lb, Lo, D, K, chunkOff, nCh, cP, cQ, offP, offQ, LP, LQ, prm.eps, chunkRec, chunkQ, nullptr, nullptr, R, chunkPair); note_launch(); }
    exclusive_scan_i32(chunkRec, recScan, nCh, nullptr, stC, d_err, s);
    exclusive_scan_i32(chunkQ, qScan, nCh, nullptr, stC, d_err, s);
  }
  // ---- G2 count: binned pairs, all in the same launches.  With an auxiliary stream they
  // run there, beside the chunked count; s waits for them before the per-pair totals.
  auto syncb = [&]() { return cudaStreamSynchronize(sb) == cudaSuccess; };
  BinSet BS{};
  int64_t nBinP = 0, nBinQ = 0;
  int64_t* cellOff = nullptr;
  int32_t* cellList = nullptr;
  float4* cellBox = nullptr;
  int64_t* binRecPos = nullptr;
  // the binned pairs' records, beside the chunked ones (one counter for both)
  auto launch_binned = [&](cudaStream_t st, bool countPairs) {
    if (nBinP == 0) return;
    const FusedRecords F{recTot, recCap, nullptr, nullptr};
    auto u64 = [](int64_t* p) { return reinterpret_cast<unsigned long long*>(p); };
    auto kern = cellBox ? (prm.exact ? bin_append_kernel<1, 1> : bin_append_kernel<0, 1>)
                        : (prm.exact ? bin_append_kernel<1, 0> : bin_append_kernel<0, 0>);
    kern<<<blocks_for_warps((nBinP + kBinEdges - 1) / kBinEdges),
                                                               kThreads, 0, st>>>(
        Lb, Lo, D, BS, nBinP, offP, LP, cellOff, cellList, cellBox, prm.eps, R, F, countPairs ? u64(binRec) : nullptr,
        u64(binQ));
    note_launch();
  };
  if (nBigPairs > 0) {
    const int B = nBigPairs;
    BS.list = bigList;
    BS.cp = A.take_n<int32_t>(B); BS.cq = A.take_n<int32_t>(B);
    BS.pBase = A.take_n<int64_t>(B); BS.qBase = A.take_n<int64_t>(B);
    BS.ext = A.take_n<double>(2 * B); BS.grid = A.take_n<BinGrid>(B);
    BS.cellBase = A.take_n<int64_t>(B); BS.ncell = A.take_n<int32_t>(B);
    int64_t* d_t = A.take_n<int64_t>(4);
    void* stB = A.take(scan_temp_bytes(B));
    if (!BS.cp || !BS.cq || !BS.pBase || !BS.qBase || !BS.ext || !BS.grid || !BS.cellBase || !BS.ncell || !d_t ||
        !stB)
      return ST_OUT_OF_MEMORY;
    { bin_sizes_kernel<<<blocks_for(B), kThreads, 0, sb>>>(BS, B, cP, cQ); note_launch(); }
    exclusive_scan_i32(BS.cp, BS.pBase, B, d_t + 0, stB, d_err, sb);
    exclusive_scan_i32(BS.cq, BS.qBase, B, d_t + 1, stB, d_err, sb);
    cudaMemsetAsync(BS.ext, 0, 2 * (size_t)B * sizeof(double), sb);
    cudaMemcpyAsync(hs + 40, d_t, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, sb);
    if (!syncb()) return ST_CUDA_ERROR;
    nBinP = hs[40];
    nBinQ = hs[41];
    BS.ownP = A.take_n<int32_t>(nBinP);
    BS.ownQ = A.take_n<int32_t>(nBinQ);
    if (!BS.ownP || !BS.ownQ) return ST_OUT_OF_MEMORY;
    { range_owner_kernel<<<blocks_for_warps(B), kThreads, 0, sb>>>(BS.pBase, BS.cp, B, BS.ownP); note_launch(); }
    { range_owner_kernel<<<blocks_for_warps(B), kThreads, 0, sb>>>(BS.qBase, BS.cq, B, BS.ownQ); note_launch(); }
    if (nBinQ > 0)
      { bin_extent_kernel<<<blocks_for(nBinQ), kThreads, 0, sb>>>(Lb, Lo, D, BS, nBinQ, offQ, LQ); note_launch(); }
    { bin_grid_kernel<<<blocks_for(B), kThreads, 0, sb>>>(D, BS, B); note_launch(); }
    exclusive_scan_i32(BS.ncell, BS.cellBase, B, d_t + 2, stB, d_err, sb);
    cudaMemcpyAsync(hs + 42, d_t + 2, sizeof(int64_t), cudaMemcpyDeviceToHost, sb);
    if (!syncb()) return ST_CUDA_ERROR;
    const int64_t nCells = hs[42];
    const int64_t nCls = 4 * nCells;                // four listing classes per cell
    int32_t* cellCnt = A.take_n<int32_t>(nCls + 1);
    cellOff = A.take_n<int64_t>(nCls + 1);
    void* stCell = A.take(scan_temp_bytes(nCls + 1));
    if (!cellCnt || !cellOff || !stCell) return ST_OUT_OF_MEMORY;
    cudaMemsetAsync(cellCnt, 0, (nCls + 1) * sizeof(int32_t), sb);
    if (nBinQ > 0)
      { bin_cells_kernel<0><<<blocks_for(nBinQ), kThreads, 0, sb>>>(Lb, Lo, D, BS, nBinQ, offQ, LQ, cellCnt, nullptr,
                                                                   nullptr, nullptr, nullptr); note_launch(); }
    exclusive_scan_i32(cellCnt, cellOff, nCls + 1, d_t + 3, stCell, d_err, sb);
    cudaMemcpyAsync(hs + 43, d_t + 3, sizeof(int64_t), cudaMemcpyDeviceToHost, sb);
    cudaMemsetAsync(cellCnt, 0, nCls * sizeof(int32_t), sb);        // the listing cursors
    if (!syncb()) return ST_CUDA_ERROR;
    cellList = A.take_n<int32_t>(hs[43]);
    const bool boxes = fused && hs[43] <= kMaxBoxes;
    if (boxes) cellBox = A.take_n<float4>(hs[43]);
    if (!cellList || (boxes && !cellBox)) return ST_OUT_OF_MEMORY;
    if (nBinQ > 0)
      { bin_cells_kernel<1><<<blocks_for(nBinQ), kThreads, 0, sb>>>(Lb, Lo, D, BS, nBinQ, offQ, LQ, nullptr, cellOff,
                                                                   cellCnt, cellList, cellBox); note_launch(); }
    if (fused) {
      launch_binned(sb, true);
    } else {
      int32_t* binRecCnt = A.take_n<int32_t>(nBinP + 1);
      binRecPos = A.take_n<int64_t>(nBinP + 1);
      void* stP = A.take(scan_temp_bytes(nBinP + 1));
      if (!binRecCnt || !binRecPos || !stP) return ST_OUT_OF_MEMORY;
      cudaMemsetAsync(binRecCnt + nBinP, 0, sizeof(int32_t), sb);   // so the scan's last entry is the total
      if (nBinP > 0)
        { (prm.exact ? bin_pairs_kernel<0, 1> : bin_pairs_kernel<0, 0>)<<<blocks_for(nBinP), kThreads, 0, sb>>>(
              Lb, Lo, D, BS, nBinP, offP, LP, cellOff, cellList, prm.eps, binRecCnt, binQ, nullptr, nullptr, R); note_launch(); }
      exclusive_scan_i32(binRecCnt, binRecPos, nBinP + 1, nullptr, stP, d_err, sb);
      { bin_rec_total_kernel<<<blocks_for(B), kThreads, 0, sb>>>(BS, B, binRecPos, binRec); note_launch(); }
    }
  }
  if (sb != s) {
    cudaEventRecord(bev[1], sb);
    cudaStreamWaitEvent(s, bev[1], 0);
  }
  int64_t* nrec64 = A.take_n<int64_t>(K);
  int64_t* recOff = A.take_n<int64_t>(K);
  int32_t* nrec = A.take_n<int32_t>(K);
  if (!nrec64 || !recOff || !nrec) return ST_OUT_OF_MEMORY;
  { pair_records_kernel<<<blocks_for(K), kThreads, 0, s>>>(chunkOff, nchunk, recScan, qScan, chunkRec, chunkQ,
                                                         binRec, binQ, K, nrec64, nrec, C.count1, D,
                                                         pairRec, pairQ); note_launch(); }
  int64_t nR = 0;
  if (fused) {
    mk->mark("clip:count+emit", s);
    cudaMemcpyAsync(hs, recTot, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (!sync()) return ST_CUDA_ERROR;
    nR = hs[0];
    if (nR >= (1ll << kLinkKeyShift)) return ST_OUT_OF_MEMORY;
    if (nR > recCap) {                              // the arrays were short: again, at the counted size
      recCap = nR;
      if (!take_records(recCap)) return ST_OUT_OF_MEMORY;
      cudaMemsetAsync(recTot, 0, sizeof(unsigned long long), s);
      launch_fused(false);
      launch_binned(s, false);
    }
  } else {
    exclusive_scan_i64(nrec64, recOff, K, tot + 5, stK, d_err, s);
    mk->mark("clip:count", s);
    cudaMemcpyAsync(hs, tot + 5, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (!sync()) return ST_CUDA_ERROR;
    nR = hs[0];
    if (nR >= (1ll << kLinkKeyShift)) return ST_OUT_OF_MEMORY;
    // ---- G3 emit
    if (!take_records(nR)) return ST_OUT_OF_MEMORY;
    if (sb != s && nBigPairs > 0) {                 // the binned pairs' emit beside the chunked one
      cudaEventRecord(bev[0], s);
      cudaStreamWaitEvent(sb, bev[0], 0);
    }
    if (nCh > 0)
      { (prm.exact ? intersect_kernel<1, 1> : intersect_kernel<1, 0>)<<<blocks_for_warps(nCh), kThreads, 0, s>>>(
          Lb, Lo, D, K, chunkOff, nCh, cP, cQ, offP, offQ, LP, LQ, prm.eps, nullptr, nullptr, recScan, recOff, R,
          chunkPair); note_launch(); }
    if (nBinP > 0)
      { (prm.exact ? bin_pairs_kernel<1, 1> : bin_pairs_kernel<1, 0>)<<<blocks_for(nBinP), kThreads, 0, sb>>>(
          Lb, Lo, D, BS, nBinP, offP, LP, cellOff, cellList, prm.eps, nullptr, nullptr, binRecPos, recOff, R);
        note_launch(); }
    if (sb != s && nBigPairs > 0) {
      cudaEventRecord(bev[1], sb);
      cudaStreamWaitEvent(s, bev[1], 0);
    }
    mk->mark("clip:emit", s);
  }
  if (ex && ex->records_only) {
    ex->n_records = nR;
    ex->rec_p = R.p; ex->rec_q = R.q; ex->rec_a = R.a; ex->rec_b = R.b; ex->rec_t = R.t; ex->rec_k = R.k;
    C.n_records = nR;
    return ST_OK;
  }
  // ---- G4 ring layout
  // per edge, cleared at once: links of the source vertices, insertion counts and cursors
  int64_t* srcLinkP = A.take_n<int64_t>(2 * (nEP + nEQ));
  int64_t* vposP = A.take_n<int64_t>(nEP);
  int64_t* vposQ = A.take_n<int64_t>(nEQ);
  int64_t* insBaseP = A.take_n<int64_t>(nEP);
  int64_t* insBaseQ = A.take_n<int64_t>(nEQ);
  int64_t* slotP = A.take_n<int64_t>(nR);
  int64_t* slotQ = A.take_n<int64_t>(nR);
  void* stE = A.take(scan_temp_bytes(std::max<int64_t>(std::max(nEP, nEQ), 1)));
  if (!srcLinkP || !vposP || !vposQ || !insBaseP || !insBaseQ || !slotP || !slotQ || !stE) return ST_OUT_OF_MEMORY;
  int64_t* srcLinkQ = srcLinkP + nEP;
  int32_t* insP = reinterpret_cast<int32_t*>(srcLinkQ + nEQ);
  int32_t* insQ = insP + nEP;
  int32_t* curP = insQ + nEQ;
  int32_t* curQ = curP + nEP;
  cudaMemsetAsync(srcLinkP, 0, 2 * (nEP + nEQ) * sizeof(int64_t), s);
  if (nR > 0)
    { record_count_kernel<<<blocks_for(nR), kThreads, 0, s>>>(R, nR, eoffP, eoffQ, D.status, insP, insQ,
                                                            srcLinkP, srcLinkQ); note_launch(); }
  exclusive_scan_i32(insP, insBaseP, nEP, tot + 9, stE, d_err, s);
  exclusive_scan_i32(insQ, insBaseQ, nEQ, tot + 10, stE, d_err, s);
  { edge_slots_kernel<<<dim3(blocks_for(std::max<int64_t>(std::max(nEP, nEQ), 1)), 2), kThreads, 0, s>>>(
        insBaseP, nEP, vposP, insBaseQ, nEQ, vposQ); note_launch(); }
  // Sizes: the record export reads the exact ones back; the clip takes bounds instead
  // and saves the two host round trips (a record inserts at most one vertex per side).
  const bool exactSizes = ex != nullptr;
  int64_t nInsP = nR, nInsQ = nR;
  if (exactSizes) {
    cudaMemcpyAsync(hs + 2, tot + 9, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (!sync()) return ST_CUDA_ERROR;
    nInsP = hs[2];
    nInsQ = hs[3];
  }
  int64_t* insListP = A.take_n<int64_t>(nInsP);
  int64_t* insListQ = A.take_n<int64_t>(nInsQ);
  int32_t* mP = A.take_n<int32_t>(K);
  int32_t* mQ = A.take_n<int32_t>(K);
  int64_t* regSizeP = A.take_n<int64_t>(K);
  int64_t* regSizeQ = A.take_n<int64_t>(K);
  int64_t* regP = A.take_n<int64_t>(K);
  int64_t* regQ = A.take_n<int64_t>(K);
  if (!insListP || !insListQ || !mP || !mQ || !regSizeP || !regSizeQ || !regP || !regQ) return ST_OUT_OF_MEMORY;
  if (nR > 0)
    { record_scatter_kernel<<<blocks_for(nR), kThreads, 0, s>>>(R, nR, eoffP, eoffQ, D.status, insBaseP, curP,
                                                              insListP, insBaseQ, curQ, insListQ); note_launch(); }
  unsigned long long* ringTot = reinterpret_cast<unsigned long long*>(tot + 6);
  { pair_ring_kernel<<<dim3(blocks_for(K), 2), kThreads, 0, s>>>(RingSide{eoffP, vposP, D.nP, nEP, tot + 9, mP, regSizeP},
                                                              RingSide{eoffQ, vposQ, D.nQ, nEQ, tot + 10, mQ, regSizeQ},
                                                              nrec, D.status, K, ringTot); note_launch(); }
  // The one-thread and warp labelling kernels take their pairs in size order (largest
  // first, label_order_kernel), and the ring regions are laid out in that order, so that
  // the pairs labelled side by side have neighbouring regions.  The record export keeps
  // the regions in pair order.
  const int64_t midMin = std::min(prm.mid_label_min, prm.big_label_min);
  unsigned long long* mcnt = reinterpret_cast<unsigned long long*>(tot + 20);
  uint32_t* oval = A.take_n<uint32_t>(K);
  if (!oval) return ST_OUT_OF_MEMORY;
  if (!ex) {
    uint64_t* okey = A.take_n<uint64_t>(K);
    uint64_t* okeyAlt = A.take_n<uint64_t>(K);
    uint32_t* ovalAlt = A.take_n<uint32_t>(K);
    void* otmp = A.take(radix_temp_bytes(K));
    int64_t* sortedP = A.take_n<int64_t>(K);
    int64_t* sortedQ = A.take_n<int64_t>(K);
    int64_t* offSP = A.take_n<int64_t>(K);
    int64_t* offSQ = A.take_n<int64_t>(K);
    if (!okey || !okeyAlt || !ovalAlt || !otmp || !sortedP || !sortedQ || !offSP || !offSQ) return ST_OUT_OF_MEMORY;
    { label_order_kernel<<<blocks_for(K), kThreads, 0, s>>>(mP, mQ, D.status, K, std::max<int64_t>(prm.tile_label_max, 0),
                                                           midMin, prm.big_label_min, okey, oval, mcnt); note_launch(); }
    if (K == 1) {                                     // one pair: nothing to order, its regions come first
      cudaMemsetAsync(regP, 0, sizeof(int64_t), s);
      cudaMemsetAsync(regQ, 0, sizeof(int64_t), s);
    } else {
      radix_sort_pairs(okey, oval, okeyAlt, ovalAlt, K, 8, otmp, d_err, s);
      { permute_sizes_kernel<<<blocks_for(K), kThreads, 0, s>>>(oval, K, regSizeP, regSizeQ, sortedP, sortedQ); note_launch(); }
      exclusive_scan_i64(sortedP, offSP, K, tot + 11, stK, d_err, s);
      exclusive_scan_i64(sortedQ, offSQ, K, tot + 12, stK, d_err, s);
      { unpermute_offsets_kernel<<<blocks_for(K), kThreads, 0, s>>>(oval, K, offSP, offSQ, regP, regQ); note_launch(); }
    }
  } else {
    exclusive_scan_i64(regSizeP, regP, K, tot + 11, stK, d_err, s);
    exclusive_scan_i64(regSizeQ, regQ, K, tot + 12, stK, d_err, s);
  }
  // region slots: merged rings (edges + insertions) + 2 + 2 records per valid pair
  int64_t regTotP = nEP + nInsP + 2 * K + 2 * nR, regTotQ = nEQ + nInsQ + 2 * K + 2 * nR;
  if (exactSizes) {
    cudaMemcpyAsync(hs, tot + 11, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(hs + 2, tot + 6, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (!sync()) return ST_CUDA_ERROR;
    regTotP = hs[0];
    regTotQ = hs[1];
    C.n_ring_vertices = hs[2];
  }
  C.n_records = nR;
  auto take_ring = [&](int64_t n, RingSet& S) {
    const int64_t slots = (std::max<int64_t>(n, 1) + 15) & ~int64_t(15);
    char* buf = static_cast<char*>(A.take((size_t)(kRingSlotBytes * slots)));
    S.set(buf, slots);
    return buf != nullptr;
  };
  RingSet SP, SQ;
  if (!take_ring(regTotP, SP) || !take_ring(regTotQ, SQ)) return ST_OUT_OF_MEMORY;
  SP.exact = SQ.exact = prm.exact;
  mk->mark("clip:layout", s);
  // ---- G5 ring fill (light edges per thread, heavy edges per block).  The P and Q rings
  // are independent, and each side's latency-bound fill leaves room on the GPU for the
  // other, so the Q side runs on the auxiliary stream when there is one.
  {
    const size_t smem = (size_t)kHeavySmem * (sizeof(uint64_t) + 2 * sizeof(uint32_t));
    cudaFuncSetAttribute(heavy_fill_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(heavy_fill_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int dev = 0, nsm = kSms;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    unsigned long long* nHeavy = reinterpret_cast<unsigned long long*>(tot + 28);     // [heavy, mid] of P, of Q
    const unsigned midBlocks = 8 * (unsigned)nsm;
    cudaStream_t sq = s;
    cudaEvent_t fork = nullptr, join = nullptr;
    if (aux && cudaEventCreateWithFlags(&fork, cudaEventDisableTiming) == cudaSuccess &&
        cudaEventCreateWithFlags(&join, cudaEventDisableTiming) == cudaSuccess) {
      cudaEventRecord(fork, s);
      cudaStreamWaitEvent(aux, fork, 0);
      sq = aux;
    }
    int st = ST_OK;
    for (int side = 0; side < 2 && st == ST_OK; ++side) {
      cudaStream_t ss = side == 0 ? s : sq;
      const int64_t nE = side == 0 ? nEP : nEQ, nIns = side == 0 ? nInsP : nInsQ;
      int64_t* heavy = A.take_n<int64_t>(nE);
      uint64_t* gkey = A.take_n<uint64_t>(2 * nIns);
      uint32_t* gtie = A.take_n<uint32_t>(2 * nIns);
      uint32_t* gidx = A.take_n<uint32_t>(2 * nIns);
      int32_t* edgePair = A.take_n<int32_t>(nE);                    // edge -> pair
      if (!heavy || !gkey || !gtie || !gidx || !edgePair) { st = ST_OUT_OF_MEMORY; break; }
      if (nE == 0) continue;
      if (side == 0) {
        { range_owner_kernel<<<blocks_for_warps(K), kThreads, 0, ss>>>(eoffP, D.nP, K, edgePair); note_launch(); }
        { ring_fill_kernel<0><<<blocks_for(nEP), kThreads, 0, ss>>>(Lb, Lo, D, R, eoffP, nEP, edgePair, vposP, regP, mP,
                                                                  SP, slotP, insBaseP, curP, insListP, heavy,
                                                                  nHeavy); note_launch(); }
        { mid_fill_kernel<0><<<midBlocks, kMidThreads, 0, ss>>>(Lb, Lo, D, R, eoffP, edgePair, vposP, regP, mP, SP, slotP,
                                                              insBaseP, curP, insListP, heavy, nHeavy + 1); note_launch(); }
        { heavy_fill_kernel<0><<<2 * nsm, kHeavyThreads, smem, ss>>>(Lb, Lo, D, R, eoffP, edgePair, vposP, regP, mP, SP,
                                                                     slotP, insBaseP, curP, insListP, heavy, nEP, nHeavy,
                                                                     gkey, gtie, gidx); note_launch(); }
      } else {
        { range_owner_kernel<<<blocks_for_warps(K), kThreads, 0, ss>>>(eoffQ, D.nQ, K, edgePair); note_launch(); }
        { ring_fill_kernel<1><<<blocks_for(nEQ), kThreads, 0, ss>>>(Lb, Lo, D, R, eoffQ, nEQ, edgePair, vposQ, regQ, mQ,
                                                                  SQ, slotQ, insBaseQ, curQ, insListQ, heavy,
                                                                  nHeavy + 2); note_launch(); }
        { mid_fill_kernel<1><<<midBlocks, kMidThreads, 0, ss>>>(Lb, Lo, D, R, eoffQ, edgePair, vposQ, regQ, mQ, SQ, slotQ,
                                                              insBaseQ, curQ, insListQ, heavy, nHeavy + 2 + 1); note_launch(); }
        { heavy_fill_kernel<1><<<2 * nsm, kHeavyThreads, smem, ss>>>(Lb, Lo, D, R, eoffQ, edgePair, vposQ, regQ, mQ, SQ,
                                                                     slotQ, insBaseQ, curQ, insListQ, heavy, nEQ, nHeavy + 2,
                                                                     gkey, gtie, gidx); note_launch(); }
      }
    }
    if (sq != s) {
      cudaEventRecord(join, sq);
      cudaStreamWaitEvent(s, join, 0);
    }
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    if (st != ST_OK) return st;
  }
  // ---- G6 links
  if (nR > 0)
    { link_kernel<<<blocks_for(nR), kThreads, 0, s>>>(R, nR, D.status, eoffP, eoffQ, vposP, vposQ, regP, regQ,
                                                    slotP, slotQ, srcLinkP, srcLinkQ, SP, SQ); note_launch(); }
  // ---- export of the merged rings instead of labelling (calculateIntersections)
  if (ex) {
    unsigned long long* keyP = A.take_n<unsigned long long>(std::max<int64_t>(regTotP, 1));
    unsigned long long* keyQ = A.take_n<unsigned long long>(std::max<int64_t>(regTotQ, 1));
    int32_t* cnt = A.take_n<int32_t>(2 * K);
    double* xyP = A.take_n<double>(2 * std::max<int64_t>(regTotP, 1));
    double* xyQ = A.take_n<double>(2 * std::max<int64_t>(regTotQ, 1));
    int32_t* iP = A.take_n<int32_t>(3 * std::max<int64_t>(regTotP, 1));
    int32_t* iQ = A.take_n<int32_t>(3 * std::max<int64_t>(regTotQ, 1));
    if (!keyP || !keyQ || !cnt || !xyP || !xyQ || !iP || !iQ) return ST_OUT_OF_MEMORY;
    cudaMemsetAsync(keyP, 0, std::max<int64_t>(regTotP, 1) * sizeof(unsigned long long), s);
    cudaMemsetAsync(keyQ, 0, std::max<int64_t>(regTotQ, 1) * sizeof(unsigned long long), s);
    cudaMemsetAsync(cnt, 0, 2 * K * sizeof(int32_t), s);
    if (nR > 0)
      { export_key_kernel<<<blocks_for(nR), kThreads, 0, s>>>(R, nR, D.status, eoffP, eoffQ, vposP, vposQ, regP,
                                                              regQ, slotP, slotQ, keyP, keyQ, cnt, cnt + K); note_launch(); }
    const int64_t rP = std::max<int64_t>(regTotP, 1), rQ = std::max<int64_t>(regTotQ, 1);
    { export_ring_kernel<<<(unsigned)K, kThreads, 0, s>>>(K, D.status, mP, mQ, regP, regQ, SP, SQ, keyP, keyQ, xyP,
                                                         xyQ, iP, iQ, iP + rP, iQ + rQ, iP + 2 * rP,
                                                         iQ + 2 * rQ); note_launch(); }
    // pair 0: status, record counts per ring, edges, merged sizes, region offsets
    int32_t h32[6];
    int64_t h64[2];
    cudaMemcpyAsync(h32 + 0, D.status, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h32 + 1, cnt, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h32 + 2, cnt + K, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h32 + 3, D.nP, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h32 + 4, D.nQ, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h32 + 5, mP, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h64 + 0, regP, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h64 + 1, regQ, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (!sync()) return ST_CUDA_ERROR;
    ex->status = h32[0];
    ex->edges_p = h32[3];
    ex->edges_q = h32[4];
    ex->n_p = (int64_t)h32[3] + h32[1];
    ex->n_q = (int64_t)h32[4] + h32[2];
    if (ex->status == 0) {
      if (h32[5] != ex->n_p) return ST_DEVICE_ERROR;   // the ring layout disagrees with the records
      const int64_t np = ex->n_p, nq = ex->n_q, oP = h64[0], oQ = h64[1];
      ex->xy_p.resize(2 * np); ex->xy_q.resize(2 * nq);
      ex->alpha_p.resize(np); ex->label_p.resize(np); ex->nb_p.resize(np);
      ex->alpha_q.resize(nq); ex->label_q.resize(nq); ex->nb_q.resize(nq);
      cudaMemcpyAsync(ex->xy_p.data(), xyP + 2 * oP, 2 * np * sizeof(double), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(ex->xy_q.data(), xyQ + 2 * oQ, 2 * nq * sizeof(double), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(ex->alpha_p.data(), iP + oP, np * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(ex->label_p.data(), iP + rP + oP, np * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(ex->nb_p.data(), iP + 2 * rP + oP, np * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(ex->alpha_q.data(), iQ + oQ, nq * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(ex->label_q.data(), iQ + rQ + oQ, nq * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(ex->nb_q.data(), iQ + 2 * rQ + oQ, nq * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
      if (!sync()) return ST_CUDA_ERROR;
    }
    return ST_OK;
  }
  // ---- G7 label + trace into per-pair output regions
  int64_t* vcap = A.take_n<int64_t>(K);
  int32_t* ccap = A.take_n<int32_t>(K);
  int64_t* vOff = A.take_n<int64_t>(K);
  int64_t* cOff = A.take_n<int64_t>(K);
  int32_t* nc = A.take_n<int32_t>(K);
  int64_t* nv = A.take_n<int64_t>(K);
  if (!vcap || !ccap || !vOff || !cOff || !nc || !nv) return ST_OUT_OF_MEMORY;
  { out_sizes_kernel<<<blocks_for(K), kThreads, 0, s>>>(mP, mQ, nrec, D.status, K, vcap, ccap); note_launch(); }
  exclusive_scan_i64(vcap, vOff, K, tot + 13, stK, d_err, s);
  exclusive_scan_i32(ccap, cOff, K, tot + 14, stK, d_err, s);
  // the pairs of the one-thread, warp and block kernels, in order, and their counts came
  // with the ring layout; the counts are read with the output sizes
  cudaMemcpyAsync(hs, tot + 13, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(hs + 2, mcnt, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(hs + 3, mcnt + 2, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(hs + 6, tot + 6, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  if (!sync()) return ST_CUDA_ERROR;
  C.n_ring_vertices = hs[6];
  double* oxy = A.take_n<double>(2 * hs[0]);
  int32_t* ocsz = A.take_n<int32_t>(hs[1]);
  const int64_t nMid = hs[2], nTile = hs[3], nWarp = hs[4], nGrid = hs[5];
  if (!oxy || !ocsz) return ST_OUT_OF_MEMORY;
  mk->mark("clip:fill+link", s);
  {
    cudaMemsetAsync(nc, 0, K * sizeof(int32_t), s);
    cudaMemsetAsync(nv, 0, K * sizeof(int64_t), s);
    int dev = 0, nsm = kSms;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    LabelArgs la{D, K, mP, mQ, regP, regQ, regSizeP, regSizeQ, SP, SQ, oxy, vOff, vcap, ocsz, cOff, ccap, nc, nv,
                 prm, d_err, mcnt, mcnt + 1, 0, oval,
                 nTile, nWarp};
    // long pairs: a block each, on the auxiliary stream when there is one, so they start
    // first and overlap the warp-per-pair kernel instead of trailing it
    cudaStream_t ls = s;
    cudaEvent_t fork = nullptr, join = nullptr;
    if (aux && cudaEventCreateWithFlags(&fork, cudaEventDisableTiming) == cudaSuccess &&
        cudaEventCreateWithFlags(&join, cudaEventDisableTiming) == cudaSuccess) {
      cudaEventRecord(fork, s);
      cudaStreamWaitEvent(aux, fork, 0);
      ls = aux;
    }
    if (nMid > 0) {
      // The loop table goes to shared memory only when block pairs make up at least a
      // quarter of the batch: otherwise the one-thread and warp kernels beside this one
      // need the SMs' L1 more (batched workload: label stage 2.02 -> 2.52 ms with it).
      const int smem = (4 * nMid >= K) ? kBlockLoopTableBytes : 0;
      auto kern = prm.exact ? label_trace_block_kernel<1> : label_trace_block_kernel<0>;
      if (smem) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      la.blockLoopCap = smem / 12;
      kern<<<(unsigned)std::min<int64_t>(2 * nsm, nMid), kBlockLabelThreads, smem, ls>>>(la);
      note_launch();
    }
    const bool wide = K >= prm.wide_label_min;
    // the warp-per-pair pairs on the third stream, beside the one-thread pairs on s
    cudaStream_t ws = s;
    cudaEvent_t wfork = nullptr, wjoin = nullptr;
    if (aux2 && cudaEventCreateWithFlags(&wfork, cudaEventDisableTiming) == cudaSuccess &&
        cudaEventCreateWithFlags(&wjoin, cudaEventDisableTiming) == cudaSuccess) {
      cudaEventRecord(wfork, s);
      cudaStreamWaitEvent(aux2, wfork, 0);
      ws = aux2;
    }
    if (nWarp > 0)
      { (prm.exact ? label_trace_kernel<1, 0>
                   : (wide ? label_trace_kernel<0, 1> : label_trace_kernel<0, 0>))<<<(unsigned)((nWarp + 3) / 4), 128, 0, ws>>>(la); note_launch(); }
    if (nTile > 0)
      { (prm.exact ? label_trace_tile_kernel<1, 0>
                   : (wide ? label_trace_tile_kernel<0, 1> : label_trace_tile_kernel<0, 0>))<<<(unsigned)((nTile + 127) / 128), 128, 0, s>>>(la); note_launch(); }
    if (ws != s) {
      cudaEventRecord(wjoin, ws);
      cudaStreamWaitEvent(s, wjoin, 0);
    }
    if (wfork) cudaEventDestroy(wfork);
    if (wjoin) cudaEventDestroy(wjoin);
    if (ls != s) {
      cudaEventRecord(join, ls);
      cudaStreamWaitEvent(s, join, 0);
    }
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    // huge pairs: the grid path
    if (nGrid > 0) {
      int64_t* blist = A.take_n<int64_t>(K);
      unsigned long long* nbl = A.take_n<unsigned long long>(1);
      GridScratch* gs = A.take_n<GridScratch>(1);
      BigSeq* seq = A.take_n<BigSeq>(nGrid);
      if (!blist || !nbl || !gs || !seq) return ST_OUT_OF_MEMORY;
      cudaMemsetAsync(nbl, 0, sizeof(unsigned long long), s);
      cudaMemsetAsync(gs, 0, sizeof(GridScratch), s);
      cudaMemsetAsync(seq, 0, nGrid * sizeof(BigSeq), s);
      { big_label_list_kernel<<<blocks_for(K), kThreads, 0, s>>>(mP, mQ, D.status, K, prm.big_label_min, blist, nbl); note_launch(); }
      const void* kern = prm.exact ? (const void*)label_trace_grid_kernel<1> : (const void*)label_trace_grid_kernel<0>;
      int per = 0, n = (int)nGrid;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kBlockLabelThreads, 0) != cudaSuccess || per < 1)
        return ST_CUDA_ERROR;
      void* args[] = {&la, &blist, &n, &gs, &seq};
      if (cudaLaunchCooperativeKernel(kern, dim3((unsigned)std::min(per * nsm, kGridBlocksMax)), dim3(kBlockLabelThreads),
                                      args, 0, s) != cudaSuccess)
        return ST_CUDA_ERROR;
      note_launch();
      { (prm.exact ? big_seq_kernel<1> : big_seq_kernel<0>)<<<(unsigned)nGrid, 1, 0, s>>>(la, blist, seq, gs); note_launch(); }
    }
  }
  mk->mark("clip:label+trace", s);
  // ---- G8 compaction
  C.ncomp = nc;
  C.comp_off = A.take_n<int64_t>(K);
  int64_t* fVOff = A.take_n<int64_t>(K);
  if (!C.comp_off || !fVOff) return ST_OUT_OF_MEMORY;
  exclusive_scan_i32(nc, C.comp_off, K, tot + 0, stK, d_err, s);
  exclusive_scan_i64(nv, fVOff, K, tot + 1, stK, d_err, s);
  cudaMemcpyAsync(hs, tot, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  if (!sync()) return ST_CUDA_ERROR;
  C.n_components = hs[0];
  C.n_vertices = hs[1];
  C.xy = A.take_n<double>(2 * C.n_vertices);
  C.comp_size = A.take_n<int32_t>(C.n_components);
  if (!C.xy || !C.comp_size) return ST_OUT_OF_MEMORY;
  // at most one piece per kCopyPiece vertices of a listed pair and one more, and as many for
  // its components (each has a vertex)
  const int64_t maxPieces = C.n_vertices > kCopyPiece ? 4 * (C.n_vertices / kCopyPiece) + 4 : 0;
  CopyPieces pieces{nullptr, nullptr};
  if (maxPieces > 0) {
    pieces = CopyPieces{A.take_n<int2>(maxPieces), A.take_n<unsigned>(1)};
    if (!pieces.at || !pieces.n) return ST_OUT_OF_MEMORY;
    cudaMemsetAsync(pieces.n, 0, sizeof(unsigned), s);
  }
  const double2* oxy2 = reinterpret_cast<const double2*>(oxy);
  double2* cxy2 = reinterpret_cast<double2*>(C.xy);
  { out_compact_kernel<<<blocks_for_warps(K), kThreads, 0, s>>>(K, oxy2, vOff, ocsz, cOff, nc, nv, fVOff, C.comp_off, cxy2,
                                                              C.comp_size, pieces); note_launch(); }
  if (maxPieces > 0)
    { out_compact_pieces_kernel<<<(unsigned)std::min<int64_t>(maxPieces, 8 * kSms), kThreads, 0, s>>>(
          pieces, oxy2, vOff, ocsz, cOff, nc, nv, fVOff, C.comp_off, cxy2, C.comp_size); note_launch(); }
  C.vert_off = fVOff;
  mk->mark("clip:compact", s);
  return ST_OK;
}

}  // namespace gcmfgh
