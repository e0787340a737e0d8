// Borůvka rounds on the GPU (template bodies; instantiated per metric).
//
// Round structure (the reference runs steps 2-5 on the CPU with two
// synchronous copies per round, mst.cuh:118-181; here nothing leaves the
// device but two counters):
//   1. BVH purity of the current components; every row gets the lightest edge
//      to another component it already knows (from its k-NN list, or last
//      round's answer) and a lower bound of every edge it does not know; the
//      components' best known weights are seeded from those edges;
//   2. rows that can still matter search: not the settled ones (their known
//      edge is provably their lightest), not those whose bound exceeds their
//      component's best, not those of components that sit the round out (see
//      Participation). The rows left are packed into row tiles of their own,
//      and the pass finds, per row, its minimum edge to another component;
//   3. per component, the minimum edge under the order (weight, u, v) with
//      ORIGINAL indices: an atomicMin over (weight bits << 32 | u), then an
//      atomicMin over v among the points that hold that (weight, u). Any
//      point's best edge ties toward the lower other endpoint, which is also
//      the lower edge under (u, v) for that point, so the component minimum
//      is the minimum over its points (as in the reference's CPU loop);
//   4. hooking: each component points at the component across its edge; a
//      pair that chose the same edge keeps the lower label as root and adds
//      the edge once. With one strict total order on edges the chosen edges
//      form a forest plus those 2-cycles, so this is cycle free;
//   5. pointer jumping to the roots, relabel, count components and edges.
#pragma once

#include <algorithm>
#include <typeinfo>
#include <mutex>
#include <tuple>
#include <map>
#include <random>
#include <type_traits>

#include "profiling.cuh"
#include "mst.cuh"
#include "passes.cuh"
#include "screen.cuh"

namespace cuhc {
// Sets the calling thread's screened pipeline shape for a scope.
struct ScreenShapeScope {
  ScreenShape previous;
  explicit ScreenShapeScope(ScreenShape shape) : previous(currentScreenShape()) {
    setScreenShape(shape);
  }
  ~ScreenShapeScope() { setScreenShape(previous); }
};

// Pipeline-shape tuner of the screened k-NN pass (defined below).
template <class Metric>
ScreenShape tunedScreenShape(SpatialIndex &index, const Metric &m, int k, float *scratch,
                             cudaStream_t s);

// Whether the index's data suits the metric's tensor-core screen (callers
// check useScreen too): coordinate extents for every screened metric, and for
// cosine the range of the points' squared norms.
template <class Metric> inline bool screenDataOk(SpatialIndex &index) {
  if (!index.extentsWithin(kScreenMaxExtent))
    return false;
  if constexpr (std::is_same<Metric, CosineMetric>::value)
    return index.normsWithin(kCosineNormLow, kCosineNormHigh);
  return true;
}

namespace boruvka_detail {

inline int blocks(long long work, int threads = 256) { return (int)((work + threads - 1) / threads); }

// Which components search in a round. Borůvka's cut argument holds for every
// component on its own, so a component may sit a round out: the edges that the
// others choose are in the tree whatever it does, and whoever joins it spares
// its rows their search. The largest component of an instance sits out (its
// edges are found from the other side, by fewer rows), and so does every
// component of more than twice the instance's mean size: at most half of the
// components can be that large, so at least half choose an edge and the rounds
// stay logarithmic. Components under kSitOutMin rows (8 row tiles) always
// search; their rows cost less than a round. A component that is alone in its
// instance is done. Arrays are indexed by the instance's root node.
constexpr int kSitOutMin = 1024;

struct Participation {
  const int *size = nullptr;                   // points per component root
  const unsigned long long *largest = nullptr; // size << 32 | label, of sizes >= kSitOutMin
  const int *roots = nullptr;                  // components (of real points)
  const int *points = nullptr;                 // points
  const int *rootOfTile = nullptr;             // null: one instance, root node 0
  bool everyone = false;                       // no component sits out

  __device__ __forceinline__ int instanceOf(int pos) const {
    return rootOfTile ? rootOfTile[pos / kTile] : 0;
  }
  __device__ __forceinline__ bool sitsOut(int c) const {
    if (everyone)
      return false;
    const int inst = instanceOf(c), count = roots[inst];
    if (count <= 1)
      return true;
    const int s = size[c];
    return s >= kSitOutMin && ((int)(uint32_t)largest[inst] == c ||
                               (long long)s * count > 2LL * points[inst]);
  }
};

// Every point a component of its own; padding slots have size 0. One thread
// per position; the points of an instance are counted warp by warp (a warp's
// positions lie in one tile).
static __global__ void initComponents(const int *__restrict__ order, int n,
                                      const int *__restrict__ rootOfTile, int *__restrict__ comp,
                                      int *__restrict__ size, int *__restrict__ points,
                                      int *__restrict__ roots) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool real = i < n && order[i] >= 0;
  if (i < n) {
    comp[i] = i;
    size[i] = real;
  }
  const unsigned bits = __ballot_sync(0xffffffffu, real);
  if ((threadIdx.x & 31) == 0 && bits) {
    const int inst = rootOfTile ? rootOfTile[i / kTile] : 0;
    atomicAdd(&points[inst], __popc(bits));
    atomicAdd(&roots[inst], __popc(bits));
  }
}

// Clears the round's per-component results and counters[1..2], and finds each
// instance's largest component (`largest` was zeroed by the last round).
static __global__ void startRound(const int *__restrict__ comp, const int *__restrict__ size,
                                  const int *__restrict__ rootOfTile, int n,
                                  unsigned int *__restrict__ compBest,
                                  unsigned long long *__restrict__ compKey,
                                  unsigned int *__restrict__ compV,
                                  unsigned long long *__restrict__ largest,
                                  int *__restrict__ counters) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  compBest[i] = 0x7f800000u;
  compKey[i] = kEmptyKey;
  compV[i] = 0xffffffffu;
  if (i == 0)
    counters[1] = counters[2] = 0;
  if (comp[i] == i && size[i] >= kSitOutMin)
    atomicMax(&largest[rootOfTile ? rootOfTile[i / kTile] : 0],
              ((unsigned long long)(unsigned int)size[i] << 32) | (unsigned int)i);
}

constexpr float kNoSearch = -1.0f;

// What a row already knows at a round's start. Its lightest known edge to
// another component (key order: weight, original index): last round's answer
// if that still leaves, and with k-NN lists the list's members of other
// components. A member at distance v weighs w = v (single linkage) or
// max(core_i, core_j, v) (mutual reachability, alpha 1), the bits that the
// pass computes (fmaxf is exact). Every point outside the list lies at the
// k-th distance or beyond, hence weighs at least kth = the k-th distance (it
// is at least core_i). So the known edge is the row's answer when it weighs
// less than kth, or exactly kth with no point outside the list tying it, or
// when the list holds every point; such a row is settled. bound[i] <- the
// least weight an unknown edge can have, kNoSearch for rows that need no
// search (settled, of a component sitting out, padding). The known edge goes
// to nearest (the answer unless the pass finds better) and to seed (the pass's
// starting key), and its weight into the component's best.
template <bool kMutual>
static __global__ void seedRows(KnnLists knn, const float *__restrict__ core,
                                const int *__restrict__ order, const int *__restrict__ rank,
                                const int *__restrict__ comp, Participation who,
                                unsigned long long *__restrict__ seed,
                                unsigned long long *__restrict__ nearest,
                                unsigned int *__restrict__ compBest, float *__restrict__ bound,
                                int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int c = comp[i];
  if (order[i] < 0 || who.sitsOut(c)) {
    seed[i] = nearest[i] = kEmptyKey;
    bound[i] = kNoSearch;
    return;
  }
  const float ci = kMutual ? core[i] : 0.0f;
  unsigned long long best = nearest[i];
  if (best != kEmptyKey && comp[rank[keyIndex(best)]] == c)
    best = kEmptyKey;
  float least = ci;
  bool settled = false;
  if (knn.pos) {
    for (int e = 0; e < knn.k; ++e) {
      const float v = knn.val[knnSlot(i, e, knn.k)];
      // +inf: the list holds every point; heavier entries cannot win.
      if (!(v < INFINITY) || (best != kEmptyKey && v > keyWeight(best)))
        break;
      const int j = knn.pos[knnSlot(i, e, knn.k)];
      if (comp[j] == c)
        continue;
      const unsigned long long key =
          packKey(kMutual ? fmaxf(fmaxf(ci, core[j]), v) : v, (uint32_t)order[j]);
      best = key < best ? key : best;
    }
    least = knn.val[knnSlot(i, knn.k - 1, knn.k)];
    const float w = best == kEmptyKey ? INFINITY : keyWeight(best);
    settled = !(least < INFINITY) || w < least || (w == least && knn.tie[i] == 0);
  }
  if (best != kEmptyKey) {
    const unsigned int bits = (unsigned int)(best >> 32);
    if (bits < __ldcg(&compBest[c]))
      atomicMin(&compBest[c], bits);
  }
  nearest[i] = best;
  seed[i] = best;
  bound[i] = settled ? kNoSearch : least;
}

// flag[i] <- whether row i searches: it may know too little (bound >= 0), and
// an edge it does not know could still be its component's lightest or tie it.
// Also the screened pass's per-tile metadata of the round (packed, may be
// null): [orig, comp, value] x 128 slots per tile; slots past n hold -1, 0, 0.
static __global__ void chooseRows(const float *__restrict__ bound,
                                  const unsigned int *__restrict__ compBest,
                                  const int *__restrict__ order, const int *__restrict__ comp,
                                  const float *__restrict__ value, int n, int numTiles,
                                  unsigned char *__restrict__ flag, int *__restrict__ packed) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= numTiles * kTile)
    return;
  const bool real = pos < n;
  if (real && flag) {
    const float b = bound[pos];
    flag[pos] = b >= 0.0f && b <= bitsFloat(compBest[comp[pos]]);
  }
  if (packed) {
    int *tile = packed + (size_t)(pos / kTile) * 3 * kTile + pos % kTile;
    tile[0] = real ? order[pos] : -1;
    tile[kTile] = real ? comp[pos] : 0;
    tile[2 * kTile] = real && value ? __float_as_int(value[pos]) : 0;
  }
}

// Learned radius: rows of components that sit the round out are not proposed
// (radius -1); counts the others, rows that need no search themselves included.
static __global__ void proposeRows(const int *__restrict__ order, const int *__restrict__ comp,
                                   Participation who, int n, float *__restrict__ radius,
                                   unsigned long long *__restrict__ proposed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool takes = i < n && order[i] >= 0;
  if (takes && who.sitsOut(comp[i])) {
    radius[i] = -1.0f;
    takes = false;
  }
  const unsigned bits = __ballot_sync(0xffffffffu, takes);
  if ((threadIdx.x & 31) == 0 && bits)
    atomicAdd(proposed, (unsigned long long)__popc(bits));
}

static __global__ void componentKeyPass1(const unsigned long long *__restrict__ nearest,
                                  const int *__restrict__ order, const int *__restrict__ comp,
                                  unsigned long long *__restrict__ compKey, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const unsigned long long key = nearest[i];
  if (key == kEmptyKey)
    return;
  const uint32_t oi = (uint32_t)order[i], oj = keyIndex(key);
  const unsigned long long k1 = (key & 0xffffffff00000000ull) | (oi < oj ? oi : oj);
  atomicMin(&compKey[comp[i]], k1);
}

static __global__ void componentKeyPass2(const unsigned long long *__restrict__ nearest,
                                  const int *__restrict__ order, const int *__restrict__ comp,
                                  const unsigned long long *__restrict__ compKey,
                                  unsigned int *__restrict__ compV, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const unsigned long long key = nearest[i];
  if (key == kEmptyKey)
    return;
  const uint32_t oi = (uint32_t)order[i], oj = keyIndex(key);
  const unsigned long long k1 = (key & 0xffffffff00000000ull) | (oi < oj ? oi : oj);
  if (k1 == compKey[comp[i]])
    atomicMin(&compV[comp[i]], oi < oj ? oj : oi);
}

// One thread per position that is a component root (comp[r] == r).
static __global__ void hookComponents(const int *__restrict__ comp, const int *__restrict__ rank,
                               const unsigned long long *__restrict__ compKey,
                               const unsigned int *__restrict__ compV, int *__restrict__ parent,
                               int *__restrict__ edgeU, int *__restrict__ edgeV,
                               float *__restrict__ edgeW, int *__restrict__ counters,
                               int edgeCapacity, int n, unsigned long long *__restrict__ largest,
                               int *__restrict__ roots, int numNodes) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < numNodes) { // counted anew by finishRoots and the next startRound
    largest[r] = 0;
    roots[r] = 0;
  }
  if (r >= n || comp[r] != r)
    return;
  const unsigned long long k1 = compKey[r];
  if (k1 == kEmptyKey) {
    parent[r] = r;
    return;
  }
  const int u = (int)keyIndex(k1), v = (int)compV[r];
  const int cu = comp[rank[u]], cv = comp[rank[v]];
  const int t = cu == r ? cv : cu;
  const bool mutual = compKey[t] == k1 && compV[t] == (unsigned int)v;
  bool add = true;
  if (mutual && r > t) {
    add = false; // the lower label adds the shared edge
  }
  parent[r] = (mutual && r < t) ? r : t;
  if (add) {
    const int slot = atomicAdd(&counters[0], 1);
    if (slot >= edgeCapacity)
      return; // more edges than a tree has: the host reports the error
    edgeU[slot] = u;
    edgeV[slot] = v;
    edgeW[slot] = keyWeight(k1);
  }
}

// Follows each root's parent chain up to kHops steps and points the root at
// its end. Other threads shorten the chain meanwhile, which only skips
// ancestors, so L launches reach at least kHops^L steps up.
constexpr int kHops = 16;

static __global__ void jumpParents(const int *__restrict__ comp, int *parent, int n) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n || comp[r] != r)
    return;
  volatile int *up = parent;
  int at = up[r];
  for (int h = 0; h < kHops; ++h) {
    const int next = up[at];
    if (next == at)
      break;
    at = next;
  }
  up[r] = at;
}

// Counts the new components (counters[1]; per instance, padding slots left
// out, roots) and adds the absorbed components' sizes to their roots'.
static __global__ void finishRoots(const int *__restrict__ comp, const int *__restrict__ parent,
                                   const int *__restrict__ order,
                                   const int *__restrict__ rootOfTile, int *__restrict__ size,
                                   int *__restrict__ roots, int *__restrict__ counters, int n) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const bool old = r < n && comp[r] == r;
  const int up = old ? parent[r] : -1;
  const bool root = old && up == r, real = root && order[r] >= 0;
  const unsigned allBits = __ballot_sync(0xffffffffu, root);
  const unsigned bits = __ballot_sync(0xffffffffu, real);
  if ((threadIdx.x & 31) == 0) {
    if (allBits)
      atomicAdd(&counters[1], __popc(allBits));
    if (bits)
      atomicAdd(&roots[rootOfTile ? rootOfTile[r / kTile] : 0], __popc(bits));
  }
  if (old && !root) {
    atomicAdd(&size[up], size[r]);
    if (parent[up] != up)
      atomicAdd(&counters[2], 1); // not fully jumped (would be a bug)
  }
}

static __global__ void relabel(int *__restrict__ comp, const int *__restrict__ parent, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    comp[i] = parent[comp[i]];
}

} // namespace boruvka_detail

template <class Metric, class Weight>
int boruvkaMst(SpatialIndex &index, const Metric &metric, const Weight &weight, bool prune,
               DeviceEdges &edges, PassStats *stats, cudaStream_t stream, RadiusLog *radiusLog,
               const KnnLists *knn) {
  using namespace boruvka_detail;
  const int n = index.n;
  StatusChain st;
  edges.count = 0;
  CUHC_TRY(st, edges.u.allocate(std::max(n - 1, 1), stream));
  CUHC_TRY(st, edges.v.allocate(std::max(n - 1, 1), stream));
  CUHC_TRY(st, edges.w.allocate(std::max(n - 1, 1), stream));
  if (n < 2 || !st.ok())
    return st.code;

  const int numNodes = index.topo.numNodes;
  const int *rootOfTile = index.numInstances > 1 ? index.rootOfTile.get() : nullptr;
  DeviceBuffer<int> comp, parent, counters, size, instanceRoots, instancePoints;
  DeviceBuffer<unsigned long long> nearest, compKey, tiles, seed, largest;
  DeviceBuffer<unsigned int> compBest, compV;
  DeviceBuffer<float> bound;
  DeviceBuffer<unsigned char> flag;
  CUHC_TRY(st, comp.allocate(paddedToTiles(n), stream));
  CUHC_TRY(st, parent.allocate(n, stream));
  // Edges so far, roots, unjumped parents, the passes' error word.
  CUHC_TRY(st, counters.allocate(4, stream));
  CUHC_TRY(st, size.allocate(n, stream));
  CUHC_TRY(st, instanceRoots.allocate(numNodes, stream));
  CUHC_TRY(st, instancePoints.allocate(numNodes, stream));
  CUHC_TRY(st, largest.allocate(numNodes, stream));
  CUHC_TRY(st, nearest.allocate(n, stream));
  CUHC_TRY(st, seed.allocate(n, stream));
  CUHC_TRY(st, bound.allocate(n, stream));
  CUHC_TRY(st, flag.allocate(n, stream));
  CUHC_TRY(st, compKey.allocate(n, stream));
  CUHC_TRY(st, tiles.allocate(1, stream));
  CUHC_TRY(st, compBest.allocate(n, stream));
  CUHC_TRY(st, compV.allocate(n, stream));
  if (!st.ok())
    return st.code;
  CUHC_TRY(st, cudaMemsetAsync(instanceRoots.get(), 0, instanceRoots.bytes(), stream));
  CUHC_TRY(st, cudaMemsetAsync(instancePoints.get(), 0, instancePoints.bytes(), stream));
  CUHC_TRY(st, cudaMemsetAsync(largest.get(), 0, largest.bytes(), stream));
  CUHC_TRY(st, cudaMemsetAsync(nearest.get(), 0xff, n * sizeof(unsigned long long), stream));
  CUHC_TRY(st, cudaMemsetAsync(counters.get(), 0, 4 * sizeof(int), stream));
  CUHC_TRY(st, cudaMemsetAsync(tiles.get(), 0, sizeof(unsigned long long), stream));
  initComponents<<<blocks(n), 256, 0, stream>>>(index.order.get(), n, rootOfTile, comp.get(),
                                                size.get(), instancePoints.get(),
                                                instanceRoots.get());
  noteLaunch();
  CUHC_TRY(st, cudaGetLastError());

  PassParams p{};
  p.tiled = index.tiled.get();
  p.n = n;
  p.d = index.d;
  p.numChunks = index.numChunks;
  p.numTiles = index.numTiles;
  p.order = index.order.get();
  p.component = comp.get();
  p.nodeLeft = index.nodeLeft.get();
  p.nodeRight = index.nodeRight.get();
  p.nodeFirstTile = index.nodeFirstTile.get();
  p.leafOfTile = index.leafOfTile.get();
  p.nodePure = index.nodePure.get();
  p.nodeLow = index.nodeLow.get();
  p.nodeHigh = index.nodeHigh.get();
  p.nodeMinValue = index.hasMinValues ? index.nodeMinValue.get() : nullptr;
  p.prune = prune;
  p.nearest = nearest.get();
  p.compBest = compBest.get();
  p.tilesComputed = tiles.get();
  p.error = counters.get() + 3;
  p.screenStats = screenCounters();
  p.screenAudit = screenAuditWords();
  p.rootOfTile = rootOfTile;

  const bool screened = useScreen<Metric>(index.d, 0) && screenDataOk<Metric>(index);
  DeviceBuffer<int> packed;
  if (screened)
    CUHC_TRY(st, packed.allocate((size_t)index.numTiles * 3 * kTile, stream));
  int numComponents = n, totalEdges = 0, rounds = 0;
  unsigned long long tilesSoFar = 0;
  int hostCounters[4];
  // Each instance of a batch ends as one component; padding slots stay
  // components of their own.
  const int finalComponents = index.numInstances + index.numPads;
  auto jumpsFor = [](int components) {
    int launches = 1;
    for (long long reach = kHops; reach < components; reach *= kHops)
      ++launches;
    return launches;
  };
  // Radius proposal (single linkage, one instance, 16 features, a model
  // loaded) or training-row logging: per-round features of every position.
  const RadiusModel model = currentRadiusModel();
  const bool plainWeight = std::is_same<Weight, PlainWeight>::value;
  const bool useRadius = plainWeight && !radiusLog && model.params && index.d == kRadiusDims &&
                         index.numInstances == 1;
  const bool logRows = plainWeight && radiusLog && index.d == kRadiusDims &&
                       index.numInstances == 1;
  // Lists give edges whose weight is known without the distance formula:
  // plain weights, and mutual reachability with alpha 1.
  KnnLists lists;
  bool listsUsable = plainWeight;
  if constexpr (std::is_same<Weight, MutualReachWeight>::value)
    listsUsable = weight.alpha == 1.0f;
  if (knn && listsUsable && !logRows)
    lists = *knn;
  Participation who;
  who.size = size.get();
  who.largest = largest.get();
  who.roots = instanceRoots.get();
  who.points = instancePoints.get();
  who.rootOfTile = rootOfTile;
  // The rows that search are a scattered few in most rounds. Packed into row
  // tiles of their own they need a fraction of the blocks, and few row tiles
  // can be split over the columns (blockWork); but a packed row tile spans
  // many tiles' worth of space, so its box excludes less. Packing pays where
  // boxes exclude little anyway, which the list pass has just measured: the
  // share of tile pairs it computed. Rounds' passes in ms, in place against
  // packed: share 1.00 (300,000 x 32 normal) 11.1 / 0.3; 0.93 (50,001 x 50
  // blobs, HDBSCAN) 41.7 / 29.4; 0.79 (batch, 32 features) 15.5 / 12.9; 0.47
  // (batch, 8 features) 2.5 / 3.4; 0.48 (500,000 x 16) 61.7 / 58.4; 0.25
  // (100,000 x 8, HDBSCAN) 1.02 / 1.22; 0.08 (1,000,000 x 8, HDBSCAN) 15.1 /
  // 12.9; 0.04 (batch, 2 features) 3.1 / 9.6.
  const bool packRows = lists.pos && lists.tilesSearched > 0.5 * index.fullTilePairs() &&
                        index.reserveRows(st);
  // Sitting out saves rows and may cost a round. Rows are worth less than a
  // round where nothing knows their answers (no lists: nearly every other row
  // searches) and where all row tiles start at once anyway (in place, at most
  // two blocks an SM: the pass lasts as long as its slowest tile). Whole calls in
  // ms, with components sitting out and without: HDBSCAN alpha 1.5 20,000 x 48
  // quantised 22.6 / 18.1, manhattan 20,000 x 48 blobs 23.1 / 19.8; batch of 256
  // 167 / 196, 500,000 x 16 138 / 148, HDBSCAN 1,000,000 x 8 173 / 189. Training
  // rows want every row's answer, every round.
  who.everyone = logRows || !lists.pos || !(packRows || index.orderMatters());
  DeviceBuffer<float> features, prediction, radius, targets;
  DeviceBuffer<int> compSize;
  DeviceBuffer<unsigned long long> certified;
  if (useRadius || logRows) {
    CUHC_TRY(st, features.allocate((size_t)n * kRadiusFeatures, stream));
    CUHC_TRY(st, compSize.allocate(n, stream));
    CUHC_TRY(st, prediction.allocate(n, stream));
    CUHC_TRY(st, radius.allocate(n, stream));
    CUHC_TRY(st, targets.allocate(n, stream));
    // Certified rows, [mark, capped, fallback], proposed rows.
    CUHC_TRY(st, certified.allocate(5, stream));
    CUHC_TRY(st, cudaMemsetAsync(certified.get(), 0, 5 * sizeof(unsigned long long), stream));
  }
  auto enqueueFeatures = [&](int round) {
    StatusChain fs;
    CUHC_TRY(fs, cudaMemsetAsync(compSize.get(), 0, n * sizeof(int), stream));
    radius_detail::componentSizes<<<blocks(n), 256, 0, stream>>>(comp.get(), index.order.get(), n,
                                                                 compSize.get());
    noteLaunch();
    radius_detail::radiusFeatures<<<blocks(n), 256, 0, stream>>>(
        index.tiled.get(), n, index.d, index.kc, index.tileFloats(), index.order.get(),
        index.nodeLow.get(), index.nodeHigh.get(), comp.get(), compSize.get(), nearest.get(),
        round, features.get());
    noteLaunch();
    CUHC_TRY(fs, cudaGetLastError());
    return fs.code;
  };
  std::mt19937_64 logRng(radiusLog ? radiusLog->seed : 0);

  // One round, enqueued on the stream with no host work: counters[0] counts
  // every edge so far (edges are written at absolute slots), counters[1..2]
  // this round's roots and unjumped parents.
  auto enqueueRound = [&](bool first, int jumps, bool timed) {
    StatusChain rs;
    CUHC_TRY(rs, index.updatePurity(comp.get()));
    startRound<<<blocks(n), 256, 0, stream>>>(comp.get(), size.get(), rootOfTile, n,
                                              compBest.get(), compKey.get(), compV.get(),
                                              largest.get(), counters.get());
    noteLaunch();
    if (useRadius || logRows)
      CUHC_TRY(rs, enqueueFeatures(rounds));
    seedRows<!std::is_same<Weight, PlainWeight>::value><<<blocks(n), 256, 0, stream>>>(
        lists, weight.value, index.order.get(), index.rank.get(), comp.get(), who, seed.get(),
        nearest.get(), compBest.get(), bound.get(), n);
    noteLaunch();
    p.seedKey = logRows ? nullptr : seed.get();
    // A first round without lists searches every row; so do training rows.
    const bool chosen = !logRows && (lists.pos || !first), someRows = chosen && packRows;
    if (chosen || screened) {
      chooseRows<<<blocks(index.numTiles * kTile), 256, 0, stream>>>(
          bound.get(), compBest.get(), index.order.get(), comp.get(), weight.value, n,
          index.numTiles, chosen ? flag.get() : nullptr, screened ? packed.get() : nullptr);
      noteLaunch();
      p.packedMeta = screened ? packed.get() : nullptr;
    }
    CUHC_TRY(rs, cudaGetLastError());
    p.singletons = first;
    p.radius = nullptr;
    p.active = chosen ? flag.get() : nullptr;
    // Heaviest row tiles first: by the last full pass's work (boxes before any).
    if (someRows) {
      bool ordered = false;
      CUHC_TRY(rs, index.selectRows(flag.get(), comp.get(),
                                    index.hasMinValues ? weight.value : nullptr, &ordered));
      p.rowPos = index.rowPos.get();
      p.rowTiles = index.rowTiles.get();
      p.rowTiled = index.rowTiled.get();
      p.rowBoxLow = index.rowBoxLow.get();
      p.rowBoxHigh = index.rowBoxHigh.get();
      p.rowMinValue = index.rowMinValue.get();
      p.rowPure = index.rowPure.get();
      p.tileOrder = ordered ? index.tileOrder.get() : nullptr;
      p.tileWork = nullptr;
    } else if (index.orderMatters()) {
      CUHC_TRY(rs, index.orderTiles(!index.tileWorkValid, true));
      p.tileOrder = index.tileOrder.get();
      p.tileWork = index.tileWork.get();
    }
    if (useRadius) {
      CUHC_TRY(rs, mlpForward(model.params, features.get(), n, prediction.get(), stream));
      radius_detail::radiusFromPrediction<<<blocks(n), 256, 0, stream>>>(
          prediction.get(), index.order.get(), n, model.offset, radius.get());
      noteLaunch();
      proposeRows<<<blocks(n), 256, 0, stream>>>(index.order.get(), comp.get(), who, n,
                                                 radius.get(), certified.get() + 4);
      noteLaunch();
      p.radius = radius.get();
      radius_detail::radiusTileStep<<<1, 1, 0, stream>>>(tiles.get(), 0, certified.get() + 1);
      noteLaunch();
    }
    {
      PassTimer timer(timed ? (screened ? kTimerScreenPass : kTimerNearestPass) : -1, stream);
      if (screened)
        CUHC_TRY(rs, (launchScreen<Metric, Weight, false>(p, metric, weight, index.kc, stream)));
      else
        CUHC_TRY(rs, (launchPass<Metric, Weight, false>(p, metric, weight, index.kc, stream)));
      if (useRadius) {
        // Certify by component; the rest search again with no cap while
        // certified rows sit out. compBest already holds real edge weights
        // (seeds from the last round, and what rows published during the
        // pass); every row's final best goes in too, so it ends at most the
        // lightest edge found, which is what certification compares with.
        radius_detail::radiusTileStep<<<1, 1, 0, stream>>>(tiles.get(), 1, certified.get() + 1);
        noteLaunch();
        radius_detail::componentMinFound<<<blocks(n), 256, 0, stream>>>(
            nearest.get(), index.order.get(), comp.get(), n, compBest.get());
        noteLaunch();
        radius_detail::certifyRows<<<blocks(n), 256, 0, stream>>>(
            nearest.get(), index.order.get(), comp.get(), compBest.get(), n, radius.get(),
            certified.get());
        noteLaunch();
        if (screened)
          CUHC_TRY(rs, (launchScreen<Metric, Weight, false>(p, metric, weight, index.kc, stream)));
        else
          CUHC_TRY(rs, (launchPass<Metric, Weight, false>(p, metric, weight, index.kc, stream)));
        radius_detail::radiusTileStep<<<1, 1, 0, stream>>>(tiles.get(), 2, certified.get() + 1);
        noteLaunch();
        p.radius = nullptr;
      }
      if (timer.start) {
        unsigned long long tilesNow = 0;
        cudaMemcpyAsync(&tilesNow, tiles.get(), sizeof(tilesNow), cudaMemcpyDeviceToHost, stream);
        timer.finish(tilesNow - tilesSoFar);
        tilesSoFar = tilesNow;
      }
    }
    if (logRows) {
      radius_detail::radiusTargets<<<blocks(n), 256, 0, stream>>>(nearest.get(), index.order.get(),
                                                                  n, targets.get());
      noteLaunch();
      std::vector<float> hf((size_t)n * kRadiusFeatures), ht(n);
      CUHC_TRY(rs, cudaMemcpyAsync(hf.data(), features.get(), hf.size() * sizeof(float),
                                   cudaMemcpyDeviceToHost, stream));
      CUHC_TRY(rs, cudaMemcpyAsync(ht.data(), targets.get(), ht.size() * sizeof(float),
                                   cudaMemcpyDeviceToHost, stream));
      CUHC_TRY(rs, cudaStreamSynchronize(stream));
      std::vector<int> rows;
      for (int i = 0; i < n; ++i)
        if (std::isfinite(ht[i]))
          rows.push_back(i);
      std::shuffle(rows.begin(), rows.end(), logRng);
      rows.resize(std::min<size_t>(rows.size(), (size_t)radiusLog->maxRowsPerRound));
      for (const int i : rows) {
        radiusLog->features.insert(radiusLog->features.end(), hf.begin() + (size_t)i * kRadiusFeatures,
                                   hf.begin() + (size_t)(i + 1) * kRadiusFeatures);
        radiusLog->targets.push_back(ht[i]);
      }
    }
    if (!someRows)
      index.tileWorkValid = true;
    componentKeyPass1<<<blocks(n), 256, 0, stream>>>(nearest.get(), index.order.get(), comp.get(),
                                                     compKey.get(), n); noteLaunch();
    componentKeyPass2<<<blocks(n), 256, 0, stream>>>(nearest.get(), index.order.get(), comp.get(),
                                                     compKey.get(), compV.get(), n); noteLaunch();
    hookComponents<<<blocks(n), 256, 0, stream>>>(
        comp.get(), index.rank.get(), compKey.get(), compV.get(), parent.get(), edges.u.get(),
        edges.v.get(), edges.w.get(), counters.get(), n - 1, n, largest.get(),
        instanceRoots.get(), numNodes); noteLaunch();
    for (int jmp = 0; jmp < jumps; ++jmp) {
      jumpParents<<<blocks(n), 256, 0, stream>>>(comp.get(), parent.get(), n);
      noteLaunch();
    }
    finishRoots<<<blocks(n), 256, 0, stream>>>(comp.get(), parent.get(), index.order.get(),
                                               rootOfTile, size.get(), instanceRoots.get(),
                                               counters.get(), n);
    noteLaunch();
    relabel<<<blocks(n), 256, 0, stream>>>(comp.get(), parent.get(), n); noteLaunch();
    CUHC_TRY(rs, cudaGetLastError());
    return rs.code;
  };
  // Batches replay rounds after the first as one captured CUDA graph (the
  // round's launches and memsets with the largest jump count, extra jumps
  // being no-ops); timing needs events between launches and runs eagerly.
  const bool useGraph = index.numInstances > 1 && !timingEnabled();
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graphExec = nullptr;
  while (st.ok() && numComponents > finalComponents) {
    if (useGraph && rounds > 0) {
      if (!graphExec) {
        CUHC_TRY(st, cudaStreamBeginCapture(stream, cudaStreamCaptureModeRelaxed));
        const int captured = enqueueRound(false, jumpsFor(n), false);
        const cudaError_t ended = cudaStreamEndCapture(stream, &graph);
        CUHC_TRY(st, captured);
        CUHC_TRY(st, ended);
        CUHC_TRY(st, cudaGraphInstantiate(&graphExec, graph, 0));
        if (!st.ok())
          break;
      }
      CUHC_TRY(st, cudaGraphLaunch(graphExec, stream));
    } else {
      CUHC_TRY(st, enqueueRound(rounds == 0, jumpsFor(numComponents), true));
    }
    CUHC_TRY(st, cudaMemcpyAsync(hostCounters, counters.get(), 4 * sizeof(int),
                                 cudaMemcpyDeviceToHost, stream));
    CUHC_TRY(st, cudaStreamSynchronize(stream));
    if (!st.ok())
      break;
    ++rounds;
    if (hostCounters[3] != 0) {
      st(hostCounters[3]);
      break;
    }
    const int added = hostCounters[0] - totalEdges;
    if (hostCounters[2] != 0) {
      st(kErrorTimeout);
      break;
    }
    if (added == 0) {
      st(kErrorDisconnected);
      break;
    }
    totalEdges = hostCounters[0];
    numComponents = hostCounters[1];
    if (totalEdges > n - 1) {
      st(kErrorNonFinite);
      break;
    }
  }
  if (useRadius) {
    unsigned long long counts[5] = {};
    cudaMemcpyAsync(counts, certified.get(), sizeof(counts), cudaMemcpyDeviceToHost, stream);
    cudaStreamSynchronize(stream);
    addRadiusStats(counts[4], counts[0], counts[2], counts[3]);
  }
  if (graphExec)
    cudaGraphExecDestroy(graphExec);
  if (graph)
    cudaGraphDestroy(graph);
  unsigned long long tileCount = 0;
  CUHC_TRY(st, cudaMemcpyAsync(&tileCount, tiles.get(), sizeof(tileCount),
                               cudaMemcpyDeviceToHost, stream));
  CUHC_TRY(st, cudaStreamSynchronize(stream));
  edges.count = totalEdges;
  if (stats) {
    stats->tilesComputed += tileCount;
    stats->tilesTotal += (unsigned long long)rounds * index.numTiles * index.numTiles;
    stats->passes += rounds;
    stats->rounds += rounds;
  }
  return st.code;
}

template <class Metric>
int coreDistances(SpatialIndex &index, const Metric &metric, int k, bool prune, float *core,
                  PassStats *stats, cudaStream_t stream, const int *coreRank,
                  KnnLists *lists, bool rounds) {
  StatusChain st;
  DeviceBuffer<unsigned long long> tiles;
  DeviceBuffer<int> error;
  CUHC_TRY(st, tiles.allocate(1, stream));
  CUHC_TRY(st, error.allocate(1, stream));
  CUHC_TRY(st, cudaMemsetAsync(tiles.get(), 0, sizeof(unsigned long long), stream));
  CUHC_TRY(st, cudaMemsetAsync(error.get(), 0, sizeof(int), stream));
  if (!st.ok())
    return st.code;
  PassParams p{};
  p.tiled = index.tiled.get();
  p.n = index.n;
  p.d = index.d;
  p.numChunks = index.numChunks;
  p.numTiles = index.numTiles;
  p.order = index.order.get();
  p.component = nullptr;
  p.nodeLeft = index.nodeLeft.get();
  p.nodeRight = index.nodeRight.get();
  p.nodeFirstTile = index.nodeFirstTile.get();
  p.leafOfTile = index.leafOfTile.get();
  p.nodePure = nullptr;
  p.nodeLow = index.nodeLow.get();
  p.nodeHigh = index.nodeHigh.get();
  p.nodeMinValue = nullptr;
  p.prune = prune;
  p.core = core;
  p.k = k;
  p.coreRank = coreRank;
  if (lists) {
    p.knnPos = lists->pos;
    p.knnVal = lists->val;
    p.knnTie = lists->tie;
  }
  if (index.orderMatters()) {
    CUHC_TRY(st, index.orderTiles(!index.tileWorkValid));
    p.tileOrder = index.tileOrder.get();
    p.tileWork = index.tileWork.get();
  }
  p.tilesComputed = tiles.get();
  p.error = error.get();
  p.screenStats = screenCounters();
  p.screenAudit = screenAuditWords();
  p.rootOfTile = index.numInstances > 1 ? index.rootOfTile.get() : nullptr;
  {
    const bool screened =
        useScreen<Metric>(index.d, k) && screenDataOk<Metric>(index);
    const ScreenShape shape = screened && !rounds
                                  ? tunedScreenShape<Metric>(index, metric, k, core, stream)
                                  : ScreenShape{};
    ScreenShapeScope shapeScope(shape);
    PassTimer timer(rounds ? (screened ? kTimerScreenPass : kTimerNearestPass)
                           : (screened ? kTimerScreenKnnPass : kTimerKnnPass),
                    stream);
    if (screened)
      CUHC_TRY(st, (launchScreen<Metric, PlainWeight, true>(p, metric, PlainWeight{}, index.kc,
                                                            stream)));
    else
      CUHC_TRY(st, (launchPass<Metric, PlainWeight, true>(p, metric, PlainWeight{}, index.kc,
                                                          stream)));
    if (timer.start) {
      unsigned long long tilesNow = 0;
      cudaMemcpyAsync(&tilesNow, tiles.get(), sizeof(tilesNow), cudaMemcpyDeviceToHost, stream);
      timer.finish(tilesNow);
    }
  }
  index.tileWorkValid = true;
  int err = 0;
  unsigned long long tileCount = 0;
  CUHC_TRY(st, cudaMemcpyAsync(&err, error.get(), sizeof(int), cudaMemcpyDeviceToHost, stream));
  CUHC_TRY(st, cudaMemcpyAsync(&tileCount, tiles.get(), sizeof(tileCount),
                               cudaMemcpyDeviceToHost, stream));
  CUHC_TRY(st, cudaStreamSynchronize(stream));
  if (err)
    st(err);
  if (lists)
    lists->tilesSearched = (double)tileCount;
  if (stats) {
    stats->tilesComputed += tileCount;
    stats->tilesTotal += (unsigned long long)index.numTiles * index.numTiles;
    stats->passes += 1;
  }
  return st.code;
}

// Device milliseconds of the k-NN pass restricted to the first sampleTiles
// row tiles, screened or plain (the batched path's autotuner); writes the
// core distances of those rows only.
template <class Metric>
float timeKnnSample(SpatialIndex &index, const Metric &metric, int k, bool screened,
                    int sampleTiles, float *core, cudaStream_t stream) {
  PassParams p{};
  p.tiled = index.tiled.get();
  p.n = index.n;
  p.d = index.d;
  p.numChunks = index.numChunks;
  p.numTiles = std::min(sampleTiles, index.numTiles);
  p.order = index.order.get();
  p.nodeLeft = index.nodeLeft.get();
  p.nodeRight = index.nodeRight.get();
  p.nodeFirstTile = index.nodeFirstTile.get();
  p.leafOfTile = index.leafOfTile.get();
  p.nodeLow = index.nodeLow.get();
  p.nodeHigh = index.nodeHigh.get();
  p.prune = true;
  p.core = core;
  p.k = k;
  p.rootOfTile = index.numInstances > 1 ? index.rootOfTile.get() : nullptr;
  cudaEvent_t start, stop;
  cudaEventCreate(&start);
  cudaEventCreate(&stop);
  cudaEventRecord(start, stream);
  const int status =
      screened ? launchScreen<Metric, PlainWeight, true>(p, metric, PlainWeight{}, index.kc, stream)
               : launchPass<Metric, PlainWeight, true>(p, metric, PlainWeight{}, index.kc, stream);
  cudaEventRecord(stop, stream);
  cudaEventSynchronize(stop);
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, start, stop);
  cudaEventDestroy(start);
  cudaEventDestroy(stop);
  return status == 0 ? ms : INFINITY;
}

template <class Metric> bool listsFit(int d, int k) {
  return listPassFits<Metric, PlainWeight>(d, k);
}

// Whether this index's passes can run screened (metric, width, shared
// memory, data extent), ignoring the screen mode's "off".
template <class Metric> bool screenable(SpatialIndex &index, int k) {
  return useScreen<Metric>(index.d, k) && screenDataOk<Metric>(index);
}

// Pipeline-shape tuner of the screened k-NN pass: times candidate (ring
// slots, copy lead) pairs -- the most slots that fit with leads 2-6, and the
// fewest slots with lead 3 -- on the first 2 x SMs row tiles of the index
// (twice each, the faster kept) and returns the fastest, cached per process
// by (metric, d, k, batched or not). A shape changes time only, never a
// result. `scratch` receives throw-away core distances (n floats).
template <class Metric>
ScreenShape tunedScreenShape(SpatialIndex &index, const Metric &m, int k, float *scratch,
                             cudaStream_t s) {
  static std::mutex mutex;
  static std::map<std::tuple<size_t, int, int, bool>, ScreenShape> tuned;
  const auto key = std::make_tuple(typeid(Metric).hash_code(), index.d, k, index.numInstances > 1);
  {
    std::lock_guard<std::mutex> lock(mutex);
    const auto it = tuned.find(key);
    if (it != tuned.end())
      return it->second;
  }
  const int maxStages = screenStagesFor(index.d, k);
  std::vector<ScreenShape> candidates;
  for (int lead = 2; lead <= 6; ++lead)
    if (lead <= maxStages - 1)
      candidates.push_back(ScreenShape{maxStages, lead});
  if (maxStages > kScreenMinStages)
    candidates.push_back(ScreenShape{kScreenMinStages, 3});
  int device = 0, sms = 148;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  ScreenShape best{};
  float bestMs = INFINITY;
  for (const ScreenShape shape : candidates) {
    ScreenShapeScope scope(shape);
    float ms = INFINITY;
    for (int rep = 0; rep < 2; ++rep)
      ms = std::min(ms, timeKnnSample(index, m, k, true, 2 * sms, scratch, s));
    if (ms < bestMs) {
      bestMs = ms;
      best = shape;
    }
  }
  std::lock_guard<std::mutex> lock(mutex);
  tuned[key] = best;
  return best;
}

} // namespace cuhc
