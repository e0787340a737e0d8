// Full distance matrix (cuhc_pairwise_distances): the engine's tile loop
// with a store epilogue, one block per 128 x 128 output tile. Same per-pair
// arithmetic as every pass, so the matrix equals the reference's
// pairwiseDistanceKernel (distance_matrix.cuh:177-200) bit for bit.
#pragma once

#include "profiling.cuh"
#include "engine.cuh"

namespace cuhc {

// A tiled copy of points in their original order (no spatial index).
int buildTiled(const float *points, int n, int d, DeviceBuffer<float> &tiled, cudaStream_t s);

__device__ __forceinline__ void copyAsync16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src));
}

// The 8 x 8 distances of a thread: one accumulator per pair, or for cosine a
// dot product per pair and the squared norms per row and column (every pair of
// a row folds the same features in the same order, so the bits are those of
// the metric's own three sums; 192 accumulators a thread would spill).
template <class Metric, int KC> struct PairBlock {
  typename Metric::Acc acc[8][8];
  __device__ __forceinline__ void init(const Metric &m) {
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 8; ++c)
        acc[r][c] = m.init();
  }
  __device__ __forceinline__ void fold(const float *sA, const float *sB, const Metric &m,
                                       const TileGeom &g) {
    accumulateChunk<Metric, KC>(sA, sB, m, acc, g);
  }
  __device__ __forceinline__ float distance(const Metric &m, int r, int c) const {
    return m.finalize(acc[r][c]);
  }
};

template <int KC> struct PairBlock<CosineMetric, KC> {
  float dot[8][8], rowNorm[8], colNorm[8];
  __device__ __forceinline__ void init(const CosineMetric &) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      rowNorm[r] = colNorm[r] = 0.0f;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        dot[r][c] = 0.0f;
    }
  }
  __device__ __forceinline__ void fold(const float *sA, const float *sB, const CosineMetric &,
                                       const TileGeom &g) {
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const float4 a0 = reinterpret_cast<const float4 *>(sA + k * kTile)[g.tr];
      const float4 a1 = reinterpret_cast<const float4 *>(sA + k * kTile + 64)[g.tr];
      const float4 b0 = reinterpret_cast<const float4 *>(sB + k * kTile)[g.tc];
      const float4 b1 = reinterpret_cast<const float4 *>(sB + k * kTile + 64)[g.tc];
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        rowNorm[r] = fmaf(a[r], a[r], rowNorm[r]);
        colNorm[r] = fmaf(b[r], b[r], colNorm[r]);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          dot[r][c] = fmaf(a[r], b[c], dot[r][c]);
      }
    }
  }
  __device__ __forceinline__ float distance(const CosineMetric &m, int r, int c) const {
    return m.finalize(make_float3(dot[r][c], rowNorm[r], colNorm[c]));
  }
};

// Bound by the FP32 pipes (a subtraction and a fused multiply-add per feature
// and pair for the Euclidean metrics). With several feature chunks the next
// one is copied into the other half of a double buffer while this one is
// folded in; a thread's runs of four columns are stored as one 16-byte word
// when every output row starts on such a boundary (`vector`). 16,384 x 16,384,
// whole calls in ms: euclidean 64 features 1.50 -> 1.33, 32 features 1.08 ->
// 0.84; cosine (PairBlock above) 64 features 22.1 -> 1.45.
template <class Metric, int KC>
__global__ void __launch_bounds__(kThreads, 2)
    pairwiseKernel(const float *__restrict__ tiledA, const float *__restrict__ tiledB, int nA,
                   int nB, int numChunks, bool vector, Metric m, float *__restrict__ out) {
  extern __shared__ __align__(128) float dyn[];
  constexpr int kChunk = KC * kTile;
  const TileGeom g;
  const int I = blockIdx.y, J = blockIdx.x;
  PairBlock<Metric, KC> pairs;
  pairs.init(m);
  const float *srcA = tiledA + (size_t)I * numChunks * kChunk;
  const float *srcB = tiledB + (size_t)J * numChunks * kChunk;
  auto stage = [&](int chunk) {
    float *buffer = dyn + (chunk & 1) * 2 * kChunk;
    for (int i = threadIdx.x * 4; i < kChunk; i += kThreads * 4) {
      copyAsync16(buffer + i, srcA + (size_t)chunk * kChunk + i);
      copyAsync16(buffer + kChunk + i, srcB + (size_t)chunk * kChunk + i);
    }
    asm volatile("cp.async.commit_group;");
  };
  stage(0);
  for (int chunk = 0; chunk < numChunks; ++chunk) {
    if (chunk + 1 < numChunks) {
      stage(chunk + 1);
      asm volatile("cp.async.wait_group 1;");
    } else {
      asm volatile("cp.async.wait_group 0;");
    }
    __syncthreads();
    const float *buffer = dyn + (chunk & 1) * 2 * kChunk;
    pairs.fold(buffer, buffer + kChunk, m, g);
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const long long row = (long long)I * kTile + g.row(r);
    if (row >= nA)
      continue;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      const int col = J * kTile + g.col(h);
      if (vector && col < nB) { // nB is a multiple of 4: all four columns exist
        *reinterpret_cast<float4 *>(out + row * nB + col) =
            make_float4(pairs.distance(m, r, h), pairs.distance(m, r, h + 1),
                        pairs.distance(m, r, h + 2), pairs.distance(m, r, h + 3));
        continue;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (col + c < nB)
          out[row * nB + col + c] = pairs.distance(m, r, h + c);
    }
  }
}

template <class Metric>
int launchPairwise(const float *tiledA, const float *tiledB, int nA, int nB, int d,
                   const Metric &m, float *out, cudaStream_t s) {
  const int kc = chunkWidthFor(d), numChunks = numChunksFor(d);
  const dim3 grid(numTilesFor(nB), numTilesFor(nA));
  // Two buffers of both operands' chunks; one when there is one chunk.
  const size_t dyn = (numChunks > 1 ? 4 : 2) * (size_t)kc * kTile * sizeof(float);
  const bool vector = nB % 4 == 0 && ((uintptr_t)out & 15) == 0;
  auto run = [&](auto kernel) {
    const int e = allowDynamicShared(kernel, dyn);
    if (e != 0)
      return e;
    kernel<<<grid, kThreads, dyn, s>>>(tiledA, tiledB, nA, nB, numChunks, vector, m, out);
    noteLaunch();
    return (int)cudaGetLastError();
  };
  switch (kc) {
  case 4:
    return run(pairwiseKernel<Metric, 4>);
  case 8:
    return run(pairwiseKernel<Metric, 8>);
  case 16:
    return run(pairwiseKernel<Metric, 16>);
  default:
    return run(pairwiseKernel<Metric, 32>);
  }
}

template <class Metric>
int pairwiseDistances(const float *A, int nA, const float *B, int nB, int d, const Metric &m,
                      float *out, cudaStream_t s);

} // namespace cuhc
