// Ward linkage by rounds of reciprocal nearest neighbours (RNN), on the
// shared pass engine.
//
// Each round: one all-pairs nearest pass over the active clusters' centroids
// with the Ward selection weight (every cluster its own component); every
// pair of clusters that are each other's nearest merges, all at once; the
// survivors are compacted for the next round. Same algorithm and formulas as
// the reference (rnn_ward.cuh:248-368), with its hand-over rule to a dense or
// chain tail when a round merges less than minProgress of the clusters.
//
// Clusters are stored in k-d order (for pruning) but every decision uses the
// cluster's representative, its smallest original point index: the packed
// keys carry it, ties go to the lower one, and the merged centroid is formed
// from the lower-representative cluster. Without pruning the reference keeps
// its slots in representative order (compaction preserves it), so this is
// the reference's arithmetic bit for bit, whatever the physical order.
//
// A round changes few clusters, so nearest neighbours are kept across rounds.
// Every cluster i holds a list of its kListK lightest partners (as of its last
// search) and a lower bound b_i of its exact weight W(i, c) to every cluster c
// that is not in the list. Ward's weight is reducible: for a merged pair (a, b)
// of reciprocal nearest neighbours and a third cluster, W(i, a u b) >=
// min(W(i, a), W(i, b)). So when clusters outside the list merge, b_i stays a
// bound; when a list member merges, the merged cluster takes its place with its
// new exact weight; and when i itself merges with j, the union of their lists
// and the smaller bound describe the merged row. Rounding costs the bound a
// little each round (updateLists). A row whose best list weight is below its
// bound has its answer: every other cluster is heavier. Only the other rows
// (15 % in the middle rounds of 200,000 x 32) search again, packed into row
// tiles of their own, capped near the heaviest partner they still know. Ward of
// 200,000 x 32: 690 -> 172 ms.
#include "profiling.cuh"
#include "rnn.cuh"

#include <algorithm>
#include <cmath>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <vector>

#include "metrics.cuh"
#include "passes.cuh"
#include "screen.cuh"

namespace cuhc {

int chainOnClusters(const float *centroids, const int *sizes, int m, int d, cudaStream_t s,
                    std::vector<int> &a, std::vector<int> &b, std::vector<float> &h);
int denseOnWardMatrix(const float *centroids, const int *sizes, const int *reps, int m, int d,
                      int numPoints, cudaStream_t s, std::vector<int> &u, std::vector<int> &v,
                      std::vector<float> &h);
int denseLinkageFromMatrix(float *distances, const int *initialSize, const int *initialId,
                           int firstNewId, int m, int linkageId, double *hostTree,
                           cudaStream_t s, int residentSlots);

namespace {

inline int blocks(long long work, int threads = 256) { return (int)((work + threads - 1) / threads); }

// Ward distance squared from the squared distance of two centroids, in the
// reference's operation order (rnn_ward.cuh:45-48).
__device__ __forceinline__ float wardFromSquared(float squared, float si, float sj) {
  return 2.0f * (si * sj) / (si + sj) * squared;
}

__global__ void initClusters(const int *__restrict__ order, int n, int *__restrict__ size,
                             float *__restrict__ sizeF, int *__restrict__ rep,
                             int *__restrict__ slotOfRep) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  size[i] = 1;
  sizeF[i] = 1.0f;
  rep[i] = order[i];
  slotOfRep[order[i]] = i;
}

// Positions -> row-major centroids in position order.
__global__ void gatherRows(const float *__restrict__ points, const int *__restrict__ order, int n,
                           int d, float *__restrict__ out) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)n * d)
    return;
  const int i = (int)(e / d), f = (int)(e % d);
  out[e] = points[(size_t)order[i] * d + f];
}

// partner[i]: the slot that i pairs with this round, or -1; survive[i] = 0
// if i is absorbed into a partner with a lower representative.
__global__ void rnnPartners(const unsigned long long *__restrict__ nearest,
                            const int *__restrict__ slotOfRep, const int *__restrict__ rep, int m,
                            int *__restrict__ partner, int *__restrict__ survive) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m)
    return;
  const unsigned long long key = nearest[i];
  int j = -1;
  if (key != kEmptyKey) {
    const int cand = slotOfRep[keyIndex(key)];
    const unsigned long long back = nearest[cand];
    if (back != kEmptyKey && (int)keyIndex(back) == rep[i])
      j = cand;
  }
  partner[i] = j;
  survive[i] = !(j >= 0 && rep[j] < rep[i]);
}

// Next round's clusters: slot i (not absorbed) goes to newIndex[i]; with a
// partner j its centroid is c_i + (c_j - c_i) * n_j / (n_i + n_j), the
// reference's incremental form (exact for equal centroids), and the merge is
// recorded with the exact height sqrt(ward(|c_i - c_j|^2)).
__global__ void rnnMerge(const float *__restrict__ cent, const int *__restrict__ size,
                         const int *__restrict__ rep, const int *__restrict__ partner,
                         const int *__restrict__ newIndex, int m, int d, float *__restrict__ nextCent,
                         int *__restrict__ nextSize, float *__restrict__ nextSizeF,
                         int *__restrict__ nextRep, int *__restrict__ slotOfRep,
                         unsigned char *__restrict__ nextChanged,
                         float *__restrict__ nextMergeWeight,
                         const unsigned long long *__restrict__ nearest, int *__restrict__ mergeU,
                         int *__restrict__ mergeV, float *__restrict__ mergeH,
                         int *__restrict__ mergeCount, int capacity) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)m * d)
    return;
  const int i = (int)(e / d), f = (int)(e % d);
  const int j = partner[i];
  if (j >= 0 && rep[j] < rep[i])
    return;
  const int to = newIndex[i];
  const float ci = cent[e];
  float c = ci;
  const float si = (float)size[i];
  if (j >= 0) {
    const float sj = (float)size[j];
    c = fmaf(cent[(size_t)j * d + f] - ci, sj / (si + sj), ci);
  }
  nextCent[(size_t)to * d + f] = c;
  if (f == 0) {
    const int merged = size[i] + (j >= 0 ? size[j] : 0);
    nextSize[to] = merged;
    nextSizeF[to] = (float)merged;
    nextRep[to] = rep[i];
    slotOfRep[rep[i]] = to;
    if (nextChanged)
      nextChanged[to] = j >= 0;
    if (j >= 0) {
      slotOfRep[rep[j]] = to; // where the lists that name j find it now
      if (nextMergeWeight)
        nextMergeWeight[to] = keyWeight(nearest[i]);
      const float *a = cent + (size_t)i * d, *b = cent + (size_t)j * d;
      float squared = 0.0f;
      for (int k = 0; k < d; ++k) {
        const float diff = a[k] - b[k];
        squared = fmaf(diff, diff, squared);
      }
      const int slot = atomicAdd(mergeCount, 1);
      if (slot < capacity) {
        mergeU[slot] = min(rep[i], rep[j]);
        mergeV[slot] = max(rep[i], rep[j]);
        mergeH[slot] = sqrtf(wardFromSquared(squared, si, (float)size[j]));
      }
    }
  }
}

// Entries of a cluster's list. Longer lists last more rounds but widen the
// search radius; odd, so that rows spread over the shared-memory banks. Whole
// calls of 200,000 x 32 in ms for 5 / 7 / 9 / 13 entries: 281 / 186 / 190 /
// 206 (5 measured before the size term of screen.cuh got its updates).
constexpr int kListK = 7;

// With this many clusters or fewer every round searches all of them for their
// nearest alone: the full pass is then cheaper than the launches that would
// spare part of it (passes of 200,000 x 32: a round at 4,000 clusters takes 0.2
// ms with lists and 0.5 without, below 800 about 0.15 either way; 3,916 x 8 in
// all, mostly such rounds: 10.1 ms with lists throughout, 9.35 without).
constexpr int kSearchAllBelow = 2048;

// Points from which lists are kept when the passes are plain: their list pass
// offers values one at a time, which the later rounds have to earn back. Whole
// calls in ms, with lists and without: 48 features blobs 10,000 24 / 20, 20,000
// 40 / 34, 30,000 52 / 48, 40,000 63 / 68; normal 10,000 32 / 30, 20,000 49 / 53,
// 40,000 85 / 126; 100 features blobs 20,000 59 / 58, 30,000 82 / 99.
constexpr int kPlainListsFrom = 30000;

// The lists of all clusters, entry-major ([entry][slot], `stride` slots):
// partners by representative and their exact weights, lightest first by (weight,
// representative), -1 / +inf past the last; the square root of the bound b.
struct WardLists {
  int *rep;
  float *weight;
  float *rootBound;
  size_t stride;
};

// Relative and absolute rounding of one round, for the bounds. eps bounds the
// relative error of a computed weight against the exact one (the squared
// distance's chain, the size products and the fast division: (d + 12) units of
// rounding, taken 1.5 times over). delta bounds the distance between a stored
// merged centroid and the exact mean: per feature at most 3.01 u |c_j - c_i| +
// u |c|, with the data's extent and largest magnitude.
struct WardRounding {
  float eps, delta;
};

// The weights' relative error model needs normal arithmetic: rows with lighter
// weights search every round, and no bound exceeds kBoundMax (a list may be
// short because the weights of the other clusters overflow).
constexpr float kWeightMin = 1e-30f, kBoundMax = 1e37f;

__device__ __forceinline__ float boundFromWeight(float w, const WardRounding &r) {
  return sqrtf(fminf(w, kBoundMax) * (1.0f - 2.0f * r.eps)) * (1.0f - 1e-6f);
}

// Adds (weight, rep) to a sorted list of kListK entries; returns the weight
// that does not fit (+inf: none did fall out).
__device__ __forceinline__ float keepLightest(float (&w)[kListK], int (&rep)[kListK], float nw,
                                              int nrep) {
#pragma unroll
  for (int e = 0; e < kListK; ++e) {
    const bool before = nw < w[e] || (nw == w[e] && (unsigned)nrep < (unsigned)rep[e]);
    const float tw = before ? w[e] : nw;
    const int tr = before ? rep[e] : nrep;
    w[e] = before ? nw : w[e];
    rep[e] = before ? nrep : rep[e];
    nw = tw;
    nrep = tr;
  }
  return nw;
}

__device__ __forceinline__ void storeList(const WardLists &out, int slot,
                                          const float (&w)[kListK], const int (&rep)[kListK]) {
#pragma unroll
  for (int e = 0; e < kListK; ++e) {
    out.rep[e * out.stride + slot] = rep[e];
    out.weight[e * out.stride + slot] = w[e];
  }
}

// After a round's merges: the lists, bounds and answers of the next round's
// clusters (one thread per old slot that is not absorbed). First, clusters
// outside a row's list may have merged: W(i, a u b) >= t (1 - 3 eps') with t =
// min(W(i, a), W(i, b)) by the Lance-Williams form, since the computed w(a, b)
// is at most the computed w(a, i); the stored centroid's offset takes at most
// sqrt(2 n_i) delta off its square root. Then the row itself may have merged
// with j at weight h: for c outside both lists the same form gives
//   W(i u j, c) = [n_i W(i, c) + n_j W(j, c) + n_c (W(i, c) + W(j, c) - h)] /
//                 (n_i + n_j + n_c),
// a mean of (n_i b_i + n_j b_j) / (n_i + n_j) and b_i + b_j - h or more; the
// second is the larger as a rule and weighs least for n_c = 1. flag <- whether
// the row must search, cap <- the weight up to which it does (a partner at most
// that heavy is known).
__global__ void updateLists(WardLists in, WardLists out, const int *__restrict__ partner,
                            const float *__restrict__ mergeWeight,
                            const int *__restrict__ newIndex, const int *__restrict__ rep,
                            const float *__restrict__ oldSize, int m,
                            const int *__restrict__ slotOfRep, const float *__restrict__ cent,
                            const float *__restrict__ size, const int *__restrict__ nextRep,
                            const unsigned char *__restrict__ changed, int d, WardRounding r,
                            unsigned long long *nearest, unsigned char *__restrict__ flag,
                            float *__restrict__ cap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m)
    return;
  const int j = partner[i];
  if (j >= 0 && rep[j] < rep[i])
    return;
  const int to = newIndex[i];
  const float si = size[to];
  const float *ci = cent + (size_t)to * d;
  float w[kListK];
  int reps[kListK];
#pragma unroll
  for (int e = 0; e < kListK; ++e) {
    w[e] = INFINITY;
    reps[e] = -1;
  }
  WardWeight weight;
  auto stepped = [&](float root, float points) {
    return root * (1.0f - 4.0f * r.eps) - 1.5f * sqrtf(2.0f * points) * r.delta;
  };
  float root = stepped(in.rootBound[i], j >= 0 ? oldSize[i] : si);
  if (j >= 0) {
    const float ni = oldSize[i], nj = oldSize[j];
    const float rj = stepped(in.rootBound[j], nj);
    const float bi = root > 0.0f ? root * root : 0.0f, bj = rj > 0.0f ? rj * rj : 0.0f;
    const float near = bi * (ni / (ni + nj)) + bj * (nj / (ni + nj)); // no overflow
    const float far = bi + bj - mergeWeight[to] * (1.0f + 2.0f * r.eps);
    const float both =
        far >= near ? near * (si / (si + 1.0f)) + far * (1.0f / (si + 1.0f)) : far;
    root = stepped(sqrtf(fminf(fmaxf(both, 0.0f), kBoundMax)) * (1.0f - 1e-6f), si);
  }
  for (int side = 0; side < (j >= 0 ? 2 : 1); ++side) {
    const int row = side ? j : i;
    for (int e = 0; e < kListK; ++e) {
      const int old = in.rep[e * in.stride + row];
      if (old < 0)
        break;
      const int slot = slotOfRep[old];
      if (slot == to)
        continue; // the partner
      const int now = nextRep[slot];
      bool known = false;
#pragma unroll
      for (int q = 0; q < kListK; ++q)
        known |= reps[q] == now;
      if (known)
        continue; // two members merged, or both rows list it
      float nw = in.weight[e * in.stride + row];
      if (j >= 0 || changed[slot]) {
        // The pass's arithmetic: squared distance in feature order, weight.
        const float *cj = cent + (size_t)slot * d;
        float squared = 0.0f;
        for (int k = 0; k < d; ++k) {
          const float diff = ci[k] - cj[k];
          squared = fmaf(diff, diff, squared);
        }
        nw = weight.weight(squared, si, size[slot]);
      }
      if (!(nw < INFINITY))
        continue; // no edge
      const float out = keepLightest(w, reps, nw > 0.0f ? nw : 0.0f, now);
      if (out < INFINITY) // a partner leaves the list: the bound must cover it
        root = fminf(root, boundFromWeight(out, r));
    }
  }
  storeList(out, to, w, reps);
  out.rootBound[to] = root;
  // Computed weights outside the list are at least b (1 - eps).
  const float bound = root * root * (1.0f - 2.0f * r.eps) * (1.0f - 1e-6f);
  const bool settled = root > 0.0f && reps[0] >= 0 && w[0] > kWeightMin && w[0] < bound;
  nearest[to] = reps[0] >= 0 ? packKey(w[0], (uint32_t)reps[0]) : kEmptyKey;
  flag[to] = !settled;
  float last = INFINITY;
#pragma unroll
  for (int e = 0; e < kListK; ++e)
    last = reps[e] >= 0 ? w[e] : last;
  // A list of one or two close partners would only be renewed as short.
  cap[to] = fmaxf(last, w[0] * 1.1f);
}

// The searched rows' lists from the blocks' parts (one block of 128 threads per
// row tile, thread = row): the kListK lightest of the parts' entries, the bound
// from the last, the answer from the first by (weight, representative).
// rowTiles: how many row tiles were searched (null: all of them, row tile I =
// positions from I * 128 on); cap: the searched rows' cap, beyond which nothing
// was evaluated (null: none). Every block of a searched row tile writes its
// part: a split leaves every block at least kSplitTiles / 2 column tiles.
__global__ void __launch_bounds__(kTile)
    collectLists(const unsigned long long *__restrict__ parts, const int *__restrict__ rowTiles,
                 const int *__restrict__ rowPos, int numBlocks, int numTiles, int m,
                 const float *__restrict__ cap, WardLists out, WardRounding r,
                 unsigned long long *__restrict__ nearest) {
  const int tile = blockIdx.x, tiles = rowTiles ? *rowTiles : numBlocks;
  if (tile >= tiles)
    return;
  const int pos = rowPos ? rowPos[(size_t)tile * kTile + threadIdx.x]
                         : tile * kTile + (int)threadIdx.x;
  if (pos < 0 || pos >= m)
    return;
  const int splits = rowTiles ? 1 << splitBitsFor(tiles, numBlocks, numTiles) : 1;
  float w[kListK];
  int reps[kListK];
#pragma unroll
  for (int e = 0; e < kListK; ++e) {
    w[e] = INFINITY;
    reps[e] = -1;
  }
  float least = cap ? fminf(cap[pos], kBoundMax) : kBoundMax; // of the weights left out
  for (int s = 0; s < splits; ++s) {
    const unsigned long long *part =
        parts + (size_t)(s * tiles + tile) * kListK * kTile + threadIdx.x;
    for (int e = 0; e < kListK; ++e) {
      const unsigned long long key = part[(size_t)e * kTile];
      const float v = listKeyValue(key);
      if (!(v < INFINITY))
        break;
      if (e == kListK - 1)
        least = fminf(least, v); // the block may have dropped others like it
      least = fminf(least, keepLightest(w, reps, v, (int)(uint32_t)key));
    }
  }
  storeList(out, pos, w, reps);
  out.rootBound[pos] = boundFromWeight(least, r);
  nearest[pos] = reps[0] >= 0 ? packKey(w[0], (uint32_t)reps[0]) : kEmptyKey;
}

__global__ void gatherClusters(const int *__restrict__ perm, const float *__restrict__ cent,
                               const int *__restrict__ size, int m, int d,
                               float *__restrict__ outCent, int *__restrict__ outSize) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)m * d)
    return;
  const int i = (int)(e / d), f = (int)(e % d);
  outCent[e] = cent[(size_t)perm[i] * d + f];
  if (f == 0)
    outSize[i] = size[perm[i]];
}

bool lessEdge(float wa, int ua, int va, float wb, int ub, int vb) {
  if (wa != wb)
    return wa < wb;
  if (ua != ub)
    return ua < ub;
  return va < vb;
}

struct Merge {
  int u, v;
  float w;
};

// Chain-order merges -> tree order: heights made non-decreasing up the tree
// (a merge at least as high as the merges below it), then a stable sort by
// height, as the reference's orderChainMerges (nn_chain.cuh:178-188).
void orderChainMerges(std::vector<Merge> &merges, int n) {
  std::vector<int> parent(n);
  std::vector<float> height(n, 0.0f);
  for (int i = 0; i < n; ++i)
    parent[i] = i;
  auto find = [&](int x) {
    while (parent[x] != x) {
      parent[x] = parent[parent[x]];
      x = parent[x];
    }
    return x;
  };
  for (Merge &mg : merges) {
    const int ru = find(mg.u), rv = find(mg.v);
    mg.w = std::max({mg.w, height[ru], height[rv]});
    parent[rv] = ru;
    height[ru] = mg.w;
  }
  std::stable_sort(merges.begin(), merges.end(),
                   [](const Merge &x, const Merge &y) { return x.w < y.w; });
}

bool wardMatrixFits(int m) {
  size_t freeBytes = 0, total = 0;
  if (cudaMemGetInfo(&freeBytes, &total) != cudaSuccess)
    return false;
  return 4.0 * m * m <= 0.9 * (double)freeBytes;
}

} // namespace

int rnnWard(const float *devPoints, int n, int d, const RnnOptions &options, double *hostTree,
            PassStats *stats, cudaStream_t s) {
  if (n < 2)
    return 0;
  StatusChain st;
  const int mode = currentPruneMode();
  const bool prune = mode != 2 && d <= 256 && numTilesFor(n) >= 2;
  SpatialIndex index;
  CUHC_TRY(st, index.build(devPoints, n, d, prune, s));
  DeviceBuffer<float> cent[2], sizeF[2];
  DeviceBuffer<int> size[2], rep[2];
  DeviceBuffer<int> slotOfRep, partner, survive, newIndex, counter, error, listRep[2];
  DeviceBuffer<float> listWeight[2], rootBound[2], cap, mergeWeight;
  DeviceBuffer<unsigned char> changed, searchFlag;
  DeviceBuffer<unsigned long long> parts;
  DeviceBuffer<int> mergeU, mergeV;
  DeviceBuffer<float> mergeH;
  DeviceBuffer<unsigned long long> nearest, tiles;
  for (int b = 0; b < 2; ++b) {
    CUHC_TRY(st, cent[b].allocate((size_t)n * d, s));
    CUHC_TRY(st, sizeF[b].allocate(paddedToTiles(n), s));
    CUHC_TRY(st, size[b].allocate(n, s));
    CUHC_TRY(st, rep[b].allocate(paddedToTiles(n), s));
  }
  CUHC_TRY(st, slotOfRep.allocate(n, s));
  CUHC_TRY(st, partner.allocate(n, s));
  CUHC_TRY(st, survive.allocate(n, s));
  CUHC_TRY(st, newIndex.allocate(n, s));
  CUHC_TRY(st, counter.allocate(1, s));
  CUHC_TRY(st, error.allocate(1, s));
  CUHC_TRY(st, mergeU.allocate(n - 1, s));
  CUHC_TRY(st, mergeV.allocate(n - 1, s));
  CUHC_TRY(st, mergeH.allocate(n - 1, s));
  CUHC_TRY(st, nearest.allocate(n, s));
  CUHC_TRY(st, tiles.allocate(1, s));
  size_t scanBytes = 0;
  CUHC_TRY(st, cub::DeviceScan::ExclusiveSum(nullptr, scanBytes, survive.get(), newIndex.get(),
                                             n, s));
  DeviceBuffer<unsigned char> scanTemp;
  CUHC_TRY(st, scanTemp.allocate(scanBytes, s));
  if (!st.ok())
    return st.code;
  CUHC_TRY(st, cudaMemsetAsync(counter.get(), 0, sizeof(int), s));
  CUHC_TRY(st, cudaMemsetAsync(error.get(), 0, sizeof(int), s));
  CUHC_TRY(st, cudaMemsetAsync(tiles.get(), 0, sizeof(unsigned long long), s));
  initClusters<<<blocks(n), 256, 0, s>>>(index.order.get(), n, size[0].get(), sizeF[0].get(),
                                         rep[0].get(), slotOfRep.get());
  noteLaunch();
  gatherRows<<<blocks((long long)n * d), 256, 0, s>>>(devPoints, index.order.get(), n, d,
                                                      cent[0].get());
  noteLaunch();
  CUHC_TRY(st, cudaGetLastError());

  auto listsOf = [&](int b) {
    return WardLists{listRep[b].get(), listWeight[b].get(), rootBound[b].get(), (size_t)n};
  };
  WardRounding rounding{};
  std::vector<float> boxLow(d), boxHigh(d);
  CUHC_TRY(st, index.rootBox(boxLow, boxHigh));
  if (st.ok()) {
    const double u = std::ldexp(1.0, -24);
    double square = 0.0;
    for (int f = 0; f < d; ++f) {
      const double extent = (double)boxHigh[f] - boxLow[f];
      const double magnitude = std::max(std::fabs((double)boxLow[f]), std::fabs((double)boxHigh[f]));
      const double e = u * (3.1 * extent + 1.1 * magnitude);
      square += e * e;
    }
    rounding.eps = (float)(1.5 * (d + 12) * u);
    rounding.delta = (float)(1.01 * std::sqrt(square));
  }
  // Merged centroids stay inside the points' box: the extent test holds for
  // every round.
  const bool screened =
      st.ok() && useScreen<SqEuclideanMetric>(d, kListK) && index.extentsWithin(kScreenMaxExtent);
  // Lists, where there is room for them.
  const int listsAbove = options.listsAbove >= 0               ? options.listsAbove
                         : screened || n >= kPlainListsFrom ? kSearchAllBelow
                                                              : n;
  bool canList =
      n > listsAbove && (screened || listPassFits<SqEuclideanMetric, WardWeight>(d, kListK));
  for (int b = 0; b < 2; ++b)
    canList = canList && allocateOptional(st, listRep[b], (size_t)n * kListK, s) &&
              allocateOptional(st, listWeight[b], (size_t)n * kListK, s) &&
              allocateOptional(st, rootBound[b], n, s);
  canList = canList && allocateOptional(st, cap, n, s) &&
            allocateOptional(st, mergeWeight, n, s) && allocateOptional(st, changed, n, s) &&
            allocateOptional(st, searchFlag, n, s) &&
            allocateOptional(st, parts, paddedToTiles(n) * kListK, s) && index.reserveRows(st);
  if (!canList) {
    for (int b = 0; b < 2; ++b) {
      listRep[b].release();
      listWeight[b].release();
    }
    changed.release();
    mergeWeight.release();
    parts.release();
  }
  std::vector<int> roundEnd;
  int m = n, merged = 0, cur = 0, rounds = 0, listedRounds = 0;
  enum { kNone, kDense, kChain } tail = kNone;
  unsigned long long tilesSoFar = 0;
  while (st.ok() && m > 1) {
    if (options.allowDense && m <= options.denseBelow && wardMatrixFits(m)) {
      tail = kDense;
      break;
    }
    if (rounds > 0)
      CUHC_TRY(st, index.retile(cent[cur].get(), m));
    CUHC_TRY(st, index.updateMinValues(sizeF[cur].get()));
    PassParams p{};
    p.tiled = index.tiled.get();
    p.n = m;
    p.d = d;
    p.numChunks = index.numChunks;
    p.numTiles = index.numTiles;
    p.order = rep[cur].get();
    p.component = nullptr;
    p.nodeLeft = index.nodeLeft.get();
    p.nodeRight = index.nodeRight.get();
    p.nodeFirstTile = index.nodeFirstTile.get();
    p.leafOfTile = index.leafOfTile.get();
    p.nodePure = nullptr;
    p.nodeLow = index.nodeLow.get();
    p.nodeHigh = index.nodeHigh.get();
    p.nodeMinValue = index.nodeMinValue.get();
    p.prune = prune;
    p.nearest = nearest.get();
    p.k = kListK;
    p.knnParts = parts.get();
    p.tilesComputed = tiles.get();
    p.error = error.get();
    p.screenStats = screenCounters();
    p.screenAudit = screenAuditWords();
    WardWeight w;
    w.value = sizeF[cur].get();
    const bool listed = canList && m > listsAbove;
    if (rounds > 0 && listed) {
      ++listedRounds;
      bool ordered = false;
      CUHC_TRY(st, index.selectRows(searchFlag.get(), nullptr, sizeF[cur].get(), &ordered));
      p.rowPos = index.rowPos.get();
      p.rowTiles = index.rowTiles.get();
      p.rowTiled = index.rowTiled.get();
      p.rowBoxLow = index.rowBoxLow.get();
      p.rowBoxHigh = index.rowBoxHigh.get();
      p.rowMinValue = index.rowMinValue.get();
      p.rowPure = index.rowPure.get();
      p.radius = cap.get();
    }
    {
      PassTimer timer(screened ? kTimerScreenPass : kTimerNearestPass, s);
      if (screened && !listed)
        CUHC_TRY(st, (launchScreen<SqEuclideanMetric, WardWeight, false>(
                         p, SqEuclideanMetric{}, w, index.kc, s)));
      else if (!listed)
        CUHC_TRY(st, (launchPass<SqEuclideanMetric, WardWeight, false>(p, SqEuclideanMetric{}, w,
                                                                       index.kc, s)));
      else if (screened)
        CUHC_TRY(st, (launchScreen<SqEuclideanMetric, WardWeight, true>(
                         p, SqEuclideanMetric{}, w, index.kc, s)));
      else
        CUHC_TRY(st, (launchPass<SqEuclideanMetric, WardWeight, true>(p, SqEuclideanMetric{}, w,
                                                                      index.kc, s)));
      if (timer.start) {
        unsigned long long now = 0;
        cudaMemcpyAsync(&now, tiles.get(), sizeof(now), cudaMemcpyDeviceToHost, s);
        timer.finish(now - tilesSoFar);
        tilesSoFar = now;
      }
    }
    if (listed) {
      collectLists<<<index.numTiles, kTile, 0, s>>>(parts.get(), p.rowTiles, p.rowPos,
                                                    index.numTiles, index.numTiles, m, p.radius,
                                                    listsOf(cur), rounding, nearest.get());
      noteLaunch();
    }
    rnnPartners<<<blocks(m), 256, 0, s>>>(nearest.get(), slotOfRep.get(), rep[cur].get(), m,
                                          partner.get(), survive.get());
    noteLaunch();
    CUHC_TRY(st, cub::DeviceScan::ExclusiveSum(scanTemp.get(), scanBytes, survive.get(),
                                               newIndex.get(), m, s));
    const int nxt = 1 - cur;
    rnnMerge<<<blocks((long long)m * d), 256, 0, s>>>(
        cent[cur].get(), size[cur].get(), rep[cur].get(), partner.get(), newIndex.get(), m, d,
        cent[nxt].get(), size[nxt].get(), sizeF[nxt].get(), rep[nxt].get(), slotOfRep.get(),
        changed.get(), mergeWeight.get(), nearest.get(), mergeU.get(), mergeV.get(),
        mergeH.get(), counter.get(), n - 1);
    noteLaunch();
    if (listed) {
      updateLists<<<blocks(m, 128), 128, 0, s>>>(
          listsOf(cur), listsOf(nxt), partner.get(), mergeWeight.get(), newIndex.get(),
          rep[cur].get(), sizeF[cur].get(), m, slotOfRep.get(), cent[nxt].get(),
          sizeF[nxt].get(), rep[nxt].get(), changed.get(), d, rounding, nearest.get(),
          searchFlag.get(), cap.get());
      noteLaunch();
    }
    CUHC_TRY(st, cudaGetLastError());
    int total = 0, passError = 0;
    CUHC_TRY(st, cudaMemcpyAsync(&total, counter.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    CUHC_TRY(st, cudaMemcpyAsync(&passError, error.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    CUHC_TRY(st, cudaStreamSynchronize(s));
    if (!st.ok())
      break;
    if (passError != 0) {
      st(passError);
      break;
    }
    ++rounds;
    const int roundMerges = total - merged;
    merged = total;
    roundEnd.push_back(total);
    cur = nxt;
    const int before = m;
    m -= roundMerges;
    if (merged > n - 1) {
      st(kErrorNonFinite);
      break;
    }
    if (m > 1 && (roundMerges == 0 || roundMerges < options.minProgress * before)) {
      tail = options.allowDense && wardMatrixFits(m) ? kDense : kChain;
      break;
    }
  }
  if (options.listedRounds)
    *options.listedRounds = listedRounds;
  int err = 0;
  CUHC_TRY(st, cudaMemcpyAsync(&err, error.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  unsigned long long tileCount = 0;
  CUHC_TRY(st, cudaMemcpyAsync(&tileCount, tiles.get(), sizeof(tileCount),
                               cudaMemcpyDeviceToHost, s));
  std::vector<int> hu(merged), hv(merged);
  std::vector<float> hh(merged);
  if (merged > 0) {
    CUHC_TRY(st, cudaMemcpyAsync(hu.data(), mergeU.get(), merged * sizeof(int),
                                 cudaMemcpyDeviceToHost, s));
    CUHC_TRY(st, cudaMemcpyAsync(hv.data(), mergeV.get(), merged * sizeof(int),
                                 cudaMemcpyDeviceToHost, s));
    CUHC_TRY(st, cudaMemcpyAsync(hh.data(), mergeH.get(), merged * sizeof(float),
                                 cudaMemcpyDeviceToHost, s));
  }
  CUHC_TRY(st, cudaStreamSynchronize(s));
  if (err)
    st(err);
  if (stats) {
    stats->tilesComputed += tileCount;
    stats->passes += rounds;
    for (int r = 0, mm = n; r < rounds; ++r) {
      const int t = numTilesFor(mm);
      stats->tilesTotal += (unsigned long long)t * t;
      mm -= roundEnd[r] - (r ? roundEnd[r - 1] : 0);
    }
  }
  if (!st.ok())
    return st.code;

  std::vector<Merge> merges(merged);
  for (int i = 0; i < merged; ++i)
    merges[i] = Merge{hu[i], hv[i], hh[i]};
  // Within a round merges arrive in atomic order; sorting each round by the
  // edge order makes the result independent of scheduling.
  for (size_t r = 0; r < roundEnd.size(); ++r)
    std::sort(merges.begin() + (r == 0 ? 0 : roundEnd[r - 1]), merges.begin() + roundEnd[r],
              [](const Merge &x, const Merge &y) { return lessEdge(x.w, x.u, x.v, y.w, y.u, y.v); });

  if (tail != kNone && m > 1) {
    // The remaining clusters in representative order (the reference's slot
    // order), so the tails see the same slots.
    DeviceBuffer<int> keysOut, perm, permOut, tSize, repSorted;
    DeviceBuffer<float> tCent;
    CUHC_TRY(st, keysOut.allocate(m, s));
    CUHC_TRY(st, perm.allocate(m, s));
    CUHC_TRY(st, permOut.allocate(m, s));
    CUHC_TRY(st, tSize.allocate(m, s));
    CUHC_TRY(st, tCent.allocate((size_t)m * d, s));
    std::vector<int> iota(m);
    for (int i = 0; i < m; ++i)
      iota[i] = i;
    CUHC_TRY(st, cudaMemcpyAsync(perm.get(), iota.data(), m * sizeof(int),
                                 cudaMemcpyHostToDevice, s));
    size_t sortBytes = 0;
    CUHC_TRY(st, cub::DeviceRadixSort::SortPairs(nullptr, sortBytes, rep[cur].get(),
                                                 keysOut.get(), perm.get(), permOut.get(), m, 0,
                                                 32, s));
    DeviceBuffer<unsigned char> sortTemp;
    CUHC_TRY(st, sortTemp.allocate(sortBytes, s));
    CUHC_TRY(st, cub::DeviceRadixSort::SortPairs(sortTemp.get(), sortBytes, rep[cur].get(),
                                                 keysOut.get(), perm.get(), permOut.get(), m, 0,
                                                 32, s));
    gatherClusters<<<blocks((long long)m * d), 256, 0, s>>>(permOut.get(), cent[cur].get(),
                                                            size[cur].get(), m, d, tCent.get(),
                                                            tSize.get());
    noteLaunch();
    CUHC_TRY(st, cudaGetLastError());
    std::vector<int> reps(m);
    CUHC_TRY(st, cudaMemcpyAsync(reps.data(), keysOut.get(), m * sizeof(int),
                                 cudaMemcpyDeviceToHost, s));
    CUHC_TRY(st, cudaStreamSynchronize(s));
    std::vector<int> tu, tv;
    std::vector<float> th;
    if (tail == kDense) {
      CUHC_TRY(st, denseOnWardMatrix(tCent.get(), tSize.get(), keysOut.get(), m, d, n, s, tu, tv,
                                     th));
      for (size_t i = 0; i < tu.size(); ++i)
        merges.push_back(Merge{std::min(tu[i], tv[i]), std::max(tu[i], tv[i]), th[i]});
    } else {
      CUHC_TRY(st, chainOnClusters(tCent.get(), tSize.get(), m, d, s, tu, tv, th));
      for (size_t i = 0; i < tu.size(); ++i) {
        const int a = reps[tu[i]], b = reps[tv[i]];
        merges.push_back(Merge{std::min(a, b), std::max(a, b), th[i]});
      }
    }
    if (!st.ok())
      return st.code;
  }
  std::vector<int> u(merges.size()), v(merges.size());
  std::vector<float> h(merges.size());
  for (size_t i = 0; i < merges.size(); ++i) {
    u[i] = merges[i].u;
    v[i] = merges[i].v;
    h[i] = merges[i].w;
  }
  if (!mergesFormTree(u, v, h, n))
    return kErrorNonFinite;
  orderChainMerges(merges, n);
  for (size_t i = 0; i < merges.size(); ++i) {
    u[i] = merges[i].u;
    v[i] = merges[i].v;
    h[i] = merges[i].w;
  }
  treeFromOrderedMerges(u, v, h, n, hostTree);
  return 0;
}

int nnChainWard(const float *devPoints, int n, int d, double *hostTree, cudaStream_t s) {
  if (n < 2)
    return 0;
  StatusChain st;
  DeviceBuffer<int> ones;
  CUHC_TRY(st, ones.allocate(n, s));
  std::vector<int> hostOnes(n, 1);
  CUHC_TRY(st, cudaMemcpyAsync(ones.get(), hostOnes.data(), n * sizeof(int),
                               cudaMemcpyHostToDevice, s));
  std::vector<int> a, b;
  std::vector<float> h;
  CUHC_TRY(st, chainOnClusters(devPoints, ones.get(), n, d, s, a, b, h));
  if (!st.ok())
    return st.code;
  std::vector<Merge> merges(a.size());
  std::vector<int> u(a.size()), v(a.size());
  for (size_t i = 0; i < a.size(); ++i) {
    merges[i] = Merge{std::min(a[i], b[i]), std::max(a[i], b[i]), h[i]};
    u[i] = merges[i].u;
    v[i] = merges[i].v;
  }
  if (!mergesFormTree(u, v, h, n))
    return kErrorNonFinite;
  orderChainMerges(merges, n);
  for (size_t i = 0; i < merges.size(); ++i) {
    u[i] = merges[i].u;
    v[i] = merges[i].v;
    h[i] = merges[i].w;
  }
  treeFromOrderedMerges(u, v, h, n, hostTree);
  return 0;
}

} // namespace cuhc
