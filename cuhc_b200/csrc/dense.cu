// Agglomerative clustering on the dense n x n float32 distance matrix
// (algorithm "dense": complete / average linkage, any linkage on request,
// and the dense tail of the RNN rounds).
//
// Clusters live in matrix slots; merging slots a < b keeps the cluster in a.
// Every active slot caches its nearest active slot, so one merge is: the
// argmin of the cache (ties to the lower slot), a Lance-Williams update of
// row / column a in double, and a rescan of the rows whose cached nearest
// was a or b and got farther. The reference does the same three steps per
// merge (linkage.cuh:86-268) with the same tie rules and formulas.
//
// B200 shape: a merge is a chain of short dependent steps. Up to a few thousand
// slots all merges run in one thread-block cluster that stays resident for the
// whole tree: the slots are dealt out over its blocks, whose shared memory holds
// their nearest neighbours and sizes; per merge the blocks exchange their minima
// through distributed shared memory around one cluster barrier, and read and
// write the matrix through L2. That is bound by the chain's latency (reduction,
// barrier, two row reads, the rescans). With more slots a merge is a captured
// graph of four kernels over the whole GPU (three launches' latency, and the
// bandwidth of all SMs for the rescans). Both take the same merges, bit for bit.
#include "profiling.cuh"
#include "rnn.cuh"

#include <algorithm>
#include <vector>

#include <cooperative_groups.h>

#include "metrics.cuh"
#include "pairwise.cuh"

namespace cg = cooperative_groups;

namespace cuhc {

int pairwiseIntoMatrix(const float *points, int n, int d, int metricId, float p, float *out,
                       cudaStream_t s);

namespace {

constexpr int kRescanThreads = 256;
// Blocks of the cluster (the portable limit) and their threads; a block takes
// fewer than kMinSlots slots only when it is alone.
constexpr int kClusterBlocks = 8, kMergeThreads = 512, kMinSlots = 128;
// Slots up to which the cluster makes the merges. Its eight blocks lose to the
// whole GPU where many rows lose their nearest slot per merge: some points are
// many others' nearest, the more so the more features there are. Average linkage
// of normal points in ms, cluster / whole GPU: 2 features 4,000 points 23 / 46,
// 8,000 70 / 121, 20,000 337 / 507; 64 features 4,000 35 / 48, 6,000 73 / 83, 8,000
// 121 / 125, 20,000 698 / 526; 128 features 4,096 37 / 47, 6,144 81 / 82, 7,168
// 113 / 103; 300 features 4,000 47 / 49, 5,000 72 / 65, 20,000 1,443 / 538; 1,000
// features 3,072 34 / 37, 4,096 55 / 49. Ward of 400-fold duplicates, 8 features:
// 6,000 75 / 85, 8,000 118 / 115.
inline int residentSlotsFor(int d) { return d <= 64 ? 7168 : d <= 128 ? 5120 : 3072; }
// The wide form: threads of the reducing block, merges per captured graph.
constexpr int kReduceThreads = 1024, kStepsPerGraph = 64;
enum LinkageKind : int { kSingleL = 0, kCompleteL = 1, kAverageL = 2, kWardL = 3 };

// One merge: slots a < b at `distance` into a cluster of `size` points.
struct MergeRecord {
  int a, b;
  float distance;
  int size;
};

// Distance from the merged cluster (a u b) to k from the old distances, in
// double (O(n) per merge; rounding would compound over thousands of merges).
__device__ double lanceWilliams(int linkage, double dak, double dbk, double dab, double na,
                                double nb, double nk) {
  switch (linkage) {
  case kSingleL:
    return fmin(dak, dbk);
  case kCompleteL:
    return fmax(dak, dbk);
  case kAverageL:
    return (na * dak + nb * dbk) / (na + nb);
  default: {
    // Ward on Euclidean (not squared) distances, as scipy and sklearn.
    const double t = na + nb + nk;
    const double sq = ((na + nk) * dak * dak + (nb + nk) * dbk * dbk - nk * dab * dab) / t;
    return sqrt(fmax(sq, 0.0));
  }
  }
}

__device__ __forceinline__ bool lessLoc(float da, int ia, float db, int ib) {
  return da < db || (da == db && ia < ib);
}

// The nearest other slot of a row, by one block of kRescanThreads.
__device__ __forceinline__ void nearestOfRow(const float *__restrict__ r, int n, int row,
                                             float *nearDist, int *nearSlot) {
  __shared__ float wd[kRescanThreads / 32];
  __shared__ int ws[kRescanThreads / 32];
  float best = INFINITY;
  int slot = 0x7fffffff;
#pragma unroll 4
  for (int c = threadIdx.x; c < n; c += kRescanThreads) {
    const float x = r[c]; // loaded whatever c is, so that the loads overlap
    if (c != row && lessLoc(x, c, best, slot)) {
      best = x;
      slot = c;
    }
  }
  for (int off = 16; off > 0; off /= 2) {
    const float od = __shfl_xor_sync(0xffffffffu, best, off);
    const int os = __shfl_xor_sync(0xffffffffu, slot, off);
    if (lessLoc(od, os, best, slot)) {
      best = od;
      slot = os;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    wd[threadIdx.x >> 5] = best;
    ws[threadIdx.x >> 5] = slot;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kRescanThreads / 32; ++w)
      if (lessLoc(wd[w], ws[w], best, slot)) {
        best = wd[w];
        slot = ws[w];
      }
    *nearDist = best;
    *nearSlot = slot;
  }
  __syncthreads();
}

// Nearest other slot of every row.
__global__ void __launch_bounds__(kRescanThreads)
    denseNearest(const float *__restrict__ dist, int n, float *__restrict__ nearDist,
                 int *__restrict__ nearSlot) {
  for (int row = blockIdx.x; row < n; row += gridDim.x)
    nearestOfRow(dist + (size_t)row * n, n, row, &nearDist[row], &nearSlot[row]);
}

// (distance, slot) as a key whose unsigned order is lessLoc's (-0 as +0).
__device__ __forceinline__ unsigned long long locKey(float d, int slot) {
  return ((unsigned long long)orderedBits(d + 0.0f) << 32) | (unsigned int)slot;
}

__device__ __forceinline__ unsigned long long minKey(unsigned long long x, unsigned long long y) {
  return y < x ? y : x;
}

__device__ __forceinline__ unsigned long long warpMinKey(unsigned long long key) {
#pragma unroll
  for (int off = 16; off > 0; off /= 2)
    key = minKey(key, __shfl_xor_sync(0xffffffffu, key, off));
  return key;
}

// What a block tells the others per merge: its closest slot with its nearest
// slot, and its part of the last merged row's nearest slot.
struct MergeNote {
  unsigned long long best, row;
  int other, unused;
};

// The nearest active slot of row `r`, over `lanes` threads of which this is
// number `lane`: the thread's part (the caller reduces).
__device__ __forceinline__ unsigned long long scanRow(const float *__restrict__ r, int n, int self,
                                                      const unsigned int *active, int lane,
                                                      int lanes) {
  unsigned long long best = kEmptyKey;
#pragma unroll 8
  for (int c = lane; c < n; c += lanes) {
    const float d = __ldcg(r + c);
    // Same as lessLoc from (+inf, INT_MAX): NaN never enters.
    if (c != self && ((active[c >> 5] >> (c & 31)) & 1u) && d <= INFINITY)
      best = minKey(best, locKey(d, c));
  }
  return best;
}

// All merges, in one cluster. Block c owns the slots [c * perBlock, ...): their
// nearest slots and sizes live in its shared memory, and only it rescans their
// rows; `active` is a copy of the live slots per block.
//
// Per merge: (1) every block reduces its closest slot and its part of the last
// merged row's nearest; (2) they go to every block's notes, and one cluster
// barrier later (notes alternate between two buffers) every block knows the
// closest pair a < b; (3) each thread updates its slots k: distance to the
// merged cluster into row a and column a, and k's nearest slot -- kept, taken,
// or lost, when it was a or b and got farther; (4) lost ones are rescanned. The
// barrier also publishes the matrix entries that a later merge reads in other
// blocks (loads bypass L1). A size changes only after the barrier that follows
// its merge; until then the readers know it as the last merge's.
__global__ void __launch_bounds__(kMergeThreads)
    denseMerges(float *__restrict__ dist, int n, int perBlock, int linkage,
                const float *__restrict__ nearDist0, const int *__restrict__ nearSlot0,
                const int *__restrict__ initialSize, MergeRecord *__restrict__ merges,
                int *__restrict__ mergeCount) {
  extern __shared__ __align__(16) unsigned char dense_shared[];
  __shared__ MergeNote notes[2][kClusterBlocks];
  __shared__ unsigned long long warpBest[kMergeThreads / 32], warpRow[kMergeThreads / 32];
  __shared__ int lostCount;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks();
  int *size = reinterpret_cast<int *>(dense_shared);
  unsigned int *active = reinterpret_cast<unsigned int *>(size + perBlock);
  float *nearDist = reinterpret_cast<float *>(active + (n + 31) / 32);
  int *nearSlot = reinterpret_cast<int *>(nearDist + perBlock);
  int *lost = nearSlot + perBlock;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kMergeThreads / 32;
  const int first = rank * perBlock, slots = max(0, min(perBlock, n - first));
  for (int i = tid; i < slots; i += kMergeThreads) {
    nearDist[i] = nearDist0[first + i];
    nearSlot[i] = nearSlot0[first + i];
    size[i] = initialSize ? initialSize[first + i] : 1;
  }
  for (int w = tid; w < (n + 31) / 32; w += kMergeThreads)
    active[w] = n - w * 32 >= 32 ? 0xffffffffu : (1u << (n - w * 32)) - 1;
  if (tid == 0)
    lostCount = 0;
  __syncthreads();

  unsigned long long rowPart = kEmptyKey; // this thread's part of the last merged row
  int lastA = -1, lastSize = 0, step = 0;
  for (; step < n - 1; ++step) {
    // (1) The block's closest slot (the last merged row's is not known yet).
    unsigned long long best = kEmptyKey;
    for (int i = tid; i < slots; i += kMergeThreads)
      if (first + i != lastA && nearDist[i] < INFINITY)
        best = minKey(best, locKey(nearDist[i], first + i));
    best = warpMinKey(best);
    rowPart = warpMinKey(rowPart);
    if (lane == 0) {
      warpBest[warp] = best;
      warpRow[warp] = rowPart;
    }
    __syncthreads();
    // (2) To every block.
    if (warp == 0) {
      best = warpMinKey(lane < kWarps ? warpBest[lane] : kEmptyKey);
      rowPart = warpMinKey(lane < kWarps ? warpRow[lane] : kEmptyKey);
      if (lane < blocks) {
        MergeNote note;
        note.best = best;
        note.row = rowPart;
        note.other = best == kEmptyKey ? -1 : nearSlot[(int)(uint32_t)best - first];
        note.unused = 0;
        *cluster.map_shared_rank(&notes[step & 1][rank], lane) = note;
      }
    }
    cluster.sync();
    MergeNote note;
    note.best = note.row = kEmptyKey;
    note.other = -1;
    if (lane < blocks)
      note = notes[step & 1][lane];
    const unsigned long long blockBest = note.best, row = warpMinKey(note.row);
    best = warpMinKey(blockBest);
    const unsigned from = __ballot_sync(0xffffffffu, blockBest == best);
    int other = __shfl_sync(0xffffffffu, note.other, __ffs(from) - 1);
    if (lastA >= 0) {
      const float d = row == kEmptyKey ? INFINITY : orderedFloat((uint32_t)(row >> 32));
      const int slot = row == kEmptyKey ? 0x7fffffff : (int)(uint32_t)row;
      if (d < INFINITY && locKey(d, lastA) < best) {
        best = locKey(d, lastA);
        other = slot;
      }
      if (lastA >= first && lastA < first + slots && tid == 0) {
        nearDist[lastA - first] = d;
        nearSlot[lastA - first] = slot;
        size[lastA - first] = lastSize;
      }
    }
    if (best == kEmptyKey)
      break; // no finite pair left
    const float distance = orderedFloat((uint32_t)(best >> 32));
    const int closest = (int)(uint32_t)best;
    const int a = min(closest, other), b = max(closest, other);
    auto sizeOf = [&](int slot) {
      return slot == lastA ? lastSize
                           : *cluster.map_shared_rank(&size[slot % perBlock], slot / perBlock);
    };
    const int sizeA = sizeOf(a), sizeB = sizeOf(b);
    if (rank == 0 && tid == 0)
      merges[step] = MergeRecord{a, b, distance, sizeA + sizeB};
    // Everyone has read the old nearest slots and the last row's is stored.
    __syncthreads();
    if (tid == 0) {
      active[b >> 5] &= ~(1u << (b & 31));
      lostCount = 0;
    }
    __syncthreads();
    // (3) The slots' distances to the merged cluster.
    rowPart = kEmptyKey;
    for (int i = tid; i < slots; i += kMergeThreads) {
      const int k = first + i;
      if (k == b)
        nearDist[i] = INFINITY;
      if (k == a || !((active[k >> 5] >> (k & 31)) & 1u))
        continue;
      const float nd = (float)lanceWilliams(
          linkage, __ldcg(dist + (size_t)a * n + k), __ldcg(dist + (size_t)b * n + k), distance,
          sizeA, sizeB, k == lastA ? lastSize : size[i]);
      dist[(size_t)a * n + k] = nd;
      dist[(size_t)k * n + a] = nd;
      if (nd <= INFINITY)
        rowPart = minKey(rowPart, locKey(nd, k));
      const int near = nearSlot[i];
      if (near == a || near == b) {
        if (nd <= nearDist[i]) {
          nearDist[i] = nd;
          nearSlot[i] = a;
        } else {
          lost[atomicAdd(&lostCount, 1)] = i;
        }
      } else if (nd < nearDist[i]) {
        nearDist[i] = nd;
        nearSlot[i] = a;
      }
    }
    __syncthreads();
    // (4) Rescans: the block's warps shared out over the lost rows (a warp per
    // row took 15 us per merge at 3,001 points).
    const int count = lostCount;
    int perRow = kWarps; // warps per row, a power of two
    while (perRow > 1 && perRow * count > kWarps)
      perRow /= 2;
    for (int base = 0; base < count; base += kWarps / perRow) {
      const int q = base + warp / perRow, part = warp % perRow;
      unsigned long long key = kEmptyKey;
      if (q < count) {
        const int row = first + lost[q];
        key = warpMinKey(scanRow(dist + (size_t)row * n, n, row, active, part * 32 + lane,
                                 perRow * 32));
      }
      if (lane == 0)
        warpBest[warp] = key;
      __syncthreads();
      if (q < count && part == 0 && lane == 0) {
        for (int w = 1; w < perRow; ++w)
          key = minKey(key, warpBest[warp + w]);
        nearDist[lost[q]] = key == kEmptyKey ? INFINITY : orderedFloat((uint32_t)(key >> 32));
        nearSlot[lost[q]] = key == kEmptyKey ? 0x7fffffff : (int)(uint32_t)key;
      }
      __syncthreads();
    }
    __syncthreads();
    lastA = a;
    lastSize = sizeA + sizeB;
  }
  if (rank == 0 && tid == 0)
    *mergeCount = step;
  cluster.sync(); // no block's shared memory goes while another may read it
}

// ---- the wide form: a merge as four kernels ----

struct WideState {
  float *dist, *nearDist;
  int *nearSlot, *size, *lost, *lostCount, *step;
  unsigned char *active;
  MergeRecord *merges;
  int n, linkage;
};

__global__ void wideStart(WideState s, const int *__restrict__ initialSize) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.n)
    return;
  s.dist[(size_t)i * s.n + i] = INFINITY;
  s.size[i] = initialSize ? initialSize[i] : 1;
  s.active[i] = 1;
  if (i == 0)
    *s.lostCount = *s.step = 0;
}

// One block: the closest pair, its record, the bookkeeping of its slots. Without
// a finite pair the step goes past the last merge, which ends the tree early.
__global__ void __launch_bounds__(kReduceThreads) wideClosest(WideState s) {
  const int step = *s.step, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (step >= s.n - 1)
    return;
  __shared__ unsigned long long warpBest[kReduceThreads / 32];
  unsigned long long best = kEmptyKey;
#pragma unroll 4
  for (int i = threadIdx.x; i < s.n; i += kReduceThreads) {
    const float d = s.nearDist[i];
    best = minKey(best, d < INFINITY ? locKey(d, i) : kEmptyKey);
  }
  best = warpMinKey(best);
  if (lane == 0)
    warpBest[warp] = best;
  __syncthreads();
  if (warp != 0)
    return;
  best = warpMinKey(warpBest[lane]);
  if (lane != 0)
    return;
  if (best == kEmptyKey) {
    *s.step = s.n;
    return;
  }
  const int slot = (int)(uint32_t)best, other = s.nearSlot[slot];
  const int a = min(slot, other), b = max(slot, other);
  const int merged = s.size[a] + s.size[b];
  s.merges[step] = MergeRecord{a, b, orderedFloat((uint32_t)(best >> 32)), merged};
  s.size[a] = merged;
  s.active[b] = 0;
  s.nearDist[b] = INFINITY;
  *s.lostCount = 0;
}

// One thread per slot k: its distance to the merged cluster, and its nearest
// slot kept, taken or lost. Retired columns hold +inf.
__global__ void wideMerge(WideState s) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x, step = *s.step;
  if (k >= s.n || step >= s.n - 1 || !s.active[k])
    return;
  const MergeRecord merge = s.merges[step];
  const int a = merge.a, b = merge.b, sizeB = s.size[b];
  const size_t n = s.n;
  if (k == a) {
    s.dist[(size_t)a * n + b] = INFINITY;
    s.lost[atomicAdd(s.lostCount, 1)] = a;
    return;
  }
  const float nd =
      (float)lanceWilliams(s.linkage, s.dist[(size_t)a * n + k], s.dist[(size_t)b * n + k],
                           merge.distance, merge.size - sizeB, sizeB, s.size[k]);
  s.dist[(size_t)a * n + k] = nd;
  s.dist[(size_t)k * n + a] = nd;
  s.dist[(size_t)k * n + b] = INFINITY;
  const int near = s.nearSlot[k];
  if (near == a || near == b) {
    if (nd <= s.nearDist[k]) {
      s.nearDist[k] = nd;
      s.nearSlot[k] = a;
    } else {
      s.lost[atomicAdd(s.lostCount, 1)] = k;
    }
  } else if (nd < s.nearDist[k]) {
    s.nearDist[k] = nd;
    s.nearSlot[k] = a;
  }
}

// The nearest slots of the rows that lost theirs, a block per row.
__global__ void __launch_bounds__(kRescanThreads) wideRescan(WideState s) {
  if (*s.step >= s.n - 1)
    return;
  const int count = *s.lostCount;
  for (int item = blockIdx.x; item < count; item += gridDim.x) {
    const int row = s.lost[item];
    nearestOfRow(s.dist + (size_t)row * s.n, s.n, row, &s.nearDist[row], &s.nearSlot[row]);
  }
}

__global__ void wideAdvance(WideState s) {
  if (*s.step < s.n - 1)
    ++*s.step;
}

__global__ void wardTransform(float *dist, const int *size, int m) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)m * m)
    return;
  const int i = (int)(e / m), j = (int)(e % m);
  const float si = (float)size[i], sj = (float)size[j];
  dist[e] = sqrtf(2.0f * (si * sj) / (si + sj) * dist[e]);
}

} // namespace

namespace {

// All merges by the resident cluster.
int mergeResident(float *distances, int m, int linkageId, const float *nearDist,
                  const int *nearSlot, const int *initialSize, MergeRecord *merges,
                  int *mergeCount, cudaStream_t s) {
  StatusChain st;
  int blocks = 1;
  while (blocks < kClusterBlocks && m > blocks * kMinSlots)
    blocks *= 2;
  const int perBlock = (m + blocks - 1) / blocks;
  const size_t shared = ((size_t)4 * perBlock + (m + 31) / 32) * sizeof(int);
  CUHC_TRY(st, allowDynamicShared(denseMerges, shared));
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(blocks);
  config.blockDim = dim3(kMergeThreads);
  config.dynamicSmemBytes = shared;
  config.stream = s;
  cudaLaunchAttribute attribute{};
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = blocks;
  attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  CUHC_TRY(st, cudaLaunchKernelEx(&config, denseMerges, distances, m, perBlock, linkageId,
                                  nearDist, nearSlot, initialSize, merges, mergeCount));
  noteLaunch();
  return st.code;
}

// All merges by replays of a graph of kStepsPerGraph of them: the step counter
// lives on the device, and surplus steps leave at once.
int mergeWide(float *distances, int m, int linkageId, float *nearDist, int *nearSlot,
              const int *initialSize, MergeRecord *merges, int *step, int sms, cudaStream_t s) {
  StatusChain st;
  DeviceBuffer<int> ints;
  DeviceBuffer<unsigned char> active;
  CUHC_TRY(st, ints.allocate((size_t)2 * m + 1, s));
  CUHC_TRY(st, active.allocate(m, s));
  if (!st.ok())
    return st.code;
  WideState state{};
  state.dist = distances;
  state.nearDist = nearDist;
  state.nearSlot = nearSlot;
  state.size = ints.get();
  state.lost = ints.get() + m;
  state.lostCount = ints.get() + 2 * (size_t)m;
  state.step = step;
  state.active = active.get();
  state.merges = merges;
  state.n = m;
  state.linkage = linkageId;
  const int perSlot = (m + 255) / 256;
  wideStart<<<perSlot, 256, 0, s>>>(state, initialSize);
  noteLaunch();
  CUHC_TRY(st, cudaGetLastError());
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  CUHC_TRY(st, cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  if (st.ok()) {
    for (int i = 0; i < kStepsPerGraph; ++i) {
      wideClosest<<<1, kReduceThreads, 0, s>>>(state);
      wideMerge<<<perSlot, 256, 0, s>>>(state);
      wideRescan<<<4 * sms, kRescanThreads, 0, s>>>(state);
      wideAdvance<<<1, 1, 0, s>>>(state);
    }
    CUHC_TRY(st, cudaStreamEndCapture(s, &graph));
  }
  CUHC_TRY(st, cudaGraphInstantiate(&exec, graph, 0));
  const int replays = (m - 1 + kStepsPerGraph - 1) / kStepsPerGraph;
  for (int r = 0; r < replays && st.ok(); ++r) {
    CUHC_TRY(st, cudaGraphLaunch(exec, s));
    noteLaunch(4 * kStepsPerGraph);
  }
  CUHC_TRY(st, cudaStreamSynchronize(s));
  if (exec)
    cudaGraphExecDestroy(exec);
  if (graph)
    cudaGraphDestroy(graph);
  return st.code;
}

} // namespace

int denseLinkageFromMatrix(float *distances, const int *initialSize, const int *initialId,
                           int firstNewId, int m, int linkageId, double *hostTree,
                           cudaStream_t s, int residentSlots) {
  if (m < 2)
    return 0;
  StatusChain st;
  DeviceBuffer<float> nearDist;
  DeviceBuffer<int> nearSlot, mergeCount;
  DeviceBuffer<MergeRecord> merges;
  CUHC_TRY(st, nearDist.allocate(m, s));
  CUHC_TRY(st, nearSlot.allocate(m, s));
  CUHC_TRY(st, mergeCount.allocate(1, s));
  CUHC_TRY(st, merges.allocate(m - 1, s));
  if (!st.ok())
    return st.code;
  int device = 0, sms = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  denseNearest<<<std::min(m, 8 * sms), kRescanThreads, 0, s>>>(distances, m, nearDist.get(),
                                                               nearSlot.get());
  noteLaunch();
  CUHC_TRY(st, cudaGetLastError());
  if (m <= residentSlots)
    CUHC_TRY(st, mergeResident(distances, m, linkageId, nearDist.get(), nearSlot.get(),
                               initialSize, merges.get(), mergeCount.get(), s));
  else
    CUHC_TRY(st, mergeWide(distances, m, linkageId, nearDist.get(), nearSlot.get(), initialSize,
                           merges.get(), mergeCount.get(), sms, s));
  std::vector<MergeRecord> host(m - 1);
  std::vector<int> id(m);
  int count = 0;
  CUHC_TRY(st, cudaMemcpyAsync(host.data(), merges.get(), merges.bytes(), cudaMemcpyDeviceToHost,
                               s));
  CUHC_TRY(st, cudaMemcpyAsync(&count, mergeCount.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  if (initialId)
    CUHC_TRY(st, cudaMemcpyAsync(id.data(), initialId, m * sizeof(int), cudaMemcpyDeviceToHost,
                                 s));
  else
    for (int i = 0; i < m; ++i)
      id[i] = i;
  CUHC_TRY(st, cudaStreamSynchronize(s));
  if (st.ok() && count != m - 1)
    st(kErrorNonFinite);
  if (!st.ok())
    return st.code;
  for (int step = 0; step < m - 1; ++step) {
    const MergeRecord &merge = host[step];
    double *row = hostTree + (size_t)step * 4;
    row[0] = std::min(id[merge.a], id[merge.b]);
    row[1] = std::max(id[merge.a], id[merge.b]);
    row[2] = merge.distance;
    row[3] = merge.size;
    id[merge.a] = firstNewId + step;
  }
  return 0;
}

int denseLinkage(const float *devPoints, int n, int d, int metricId, float p, int linkageId,
                 double *hostTree, cudaStream_t s, int residentSlots) {
  if (n < 2)
    return 0;
  StatusChain st;
  DeviceBuffer<float> dist;
  CUHC_TRY(st, dist.allocate((size_t)n * n, s));
  CUHC_TRY(st, pairwiseIntoMatrix(devPoints, n, d, metricId, p, dist.get(), s));
  CUHC_TRY(st, denseLinkageFromMatrix(dist.get(), nullptr, nullptr, n, n, linkageId, hostTree, s,
                                      residentSlots >= 0 ? residentSlots : residentSlotsFor(d)));
  return st.code;
}

int denseOnWardMatrix(const float *centroids, const int *sizes, const int *reps, int m, int d,
                      int numPoints, cudaStream_t s, std::vector<int> &u, std::vector<int> &v,
                      std::vector<float> &h) {
  StatusChain st;
  DeviceBuffer<float> dist;
  CUHC_TRY(st, dist.allocate((size_t)m * m, s));
  CUHC_TRY(st, pairwiseIntoMatrix(centroids, m, d, kSqEuclidean, 2.0f, dist.get(), s));
  wardTransform<<<(int)(((long long)m * m + 255) / 256), 256, 0, s>>>(dist.get(), sizes, m);
  noteLaunch();
  CUHC_TRY(st, cudaGetLastError());
  std::vector<double> host((size_t)(m - 1) * 4);
  CUHC_TRY(st, denseLinkageFromMatrix(dist.get(), sizes, reps, numPoints, m, kWardL, host.data(),
                                      s, residentSlotsFor(d)));
  if (!st.ok())
    return st.code;
  // Tree ids -> representative points: a new cluster is represented by the
  // representative of its first child.
  std::vector<int> repOfStep(m - 1, -1);
  auto repOf = [&](double id, int step) {
    const long long c = id >= 0 && id < (double)numPoints + step ? (long long)id : -1;
    return c < 0 ? -1 : c < numPoints ? (int)c : repOfStep[c - numPoints];
  };
  u.resize(m - 1);
  v.resize(m - 1);
  h.resize(m - 1);
  for (int step = 0; step < m - 1; ++step) {
    const double *row = &host[(size_t)step * 4];
    u[step] = repOf(row[0], step);
    v[step] = repOf(row[1], step);
    h[step] = (float)row[2];
    repOfStep[step] = u[step];
  }
  return 0;
}

} // namespace cuhc
