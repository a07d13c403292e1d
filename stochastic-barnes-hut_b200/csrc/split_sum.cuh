// All-pairs sums with the sources split over a warp's lanes (the plain sums,
// brute_force.cu, and the gradients, adjoint.cu).
//
// A warp carries Q queries, the same ones in every lane as packed FP32x2 pairs,
// and its lanes take every 32nd source of a range, so 1 to 8 queries are enough
// to keep a warp busy.  What is left of the parallelism goes over the sources:
// `sw` of a CTA's 8 warps take parts of the sources of the same queries (the
// others have queries of their own and read the same sources through L1), and a
// cluster of up to 16 CTAs splits them further.  Lanes, warps and CTAs (through
// distributed shared memory, in rank order) merge their compensated sums.  No scratch
// memory, one launch, and the result depends only on the call's shape.
#pragma once

#include <cooperative_groups.h>

#include <algorithm>

#include "lane_sum.cuh"

namespace sbh {
namespace {

constexpr int kSplitWarps = 8;
constexpr int kSplitThreads = 32 * kSplitWarps;
// Acc: a lane's state for Q queries (lane_sum.cuh); sum(j) is query j's
// compensated sum (Acc::Sum, with merge()), store() writes a query's result.
template <class Acc, int DIM>
__global__ void __launch_bounds__(kSplitThreads, Acc::kMinCtas)
    split_sum_kernel(DevTree t, const float* __restrict__ qsoa, long long nq, KParams kp, int sw,
                     float* __restrict__ out, float* __restrict__ grads,
                     int* __restrict__ contribs) {
  using Sum = typename Acc::Sum;
  constexpr int Q = Acc::Q;
  __shared__ Sum s_warp[kSplitWarps * Q];
  __shared__ Sum s_cta[kSplitWarps * Q];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tiles = kSplitWarps / sw;  // query tiles of this CTA
  const long long tile0 = (long long)(blockIdx.x / csize) * tiles;
  const int parts = csize * sw;
  const long long chunk = ((t.n + parts - 1) / parts + 31) / 32 * 32;
  const long long c0 = min((long long)(rank * sw + warp % sw) * chunk, t.n);
  const long long c1 = min(c0 + chunk, t.n);

  Acc acc;
  acc.load(qsoa, nq, (tile0 + warp / sw) * Q, kp);
  sum_range(acc, t.pt_pm, t.pt_nrm, c0, c1);

#pragma unroll
  for (int j = 0; j < Q; j++) {
    const Sum v = merge_lanes(acc.sum(j));
    if (lane == 0) s_warp[warp * Q + j] = v;
  }
  __syncthreads();
  const int mine = threadIdx.x;  // this thread's query of the CTA's, if it has one
  const bool has = mine < tiles * Q;
  Sum v;
  if (has) {
    v = s_warp[(mine / Q) * sw * Q + mine % Q];
    for (int p = 1; p < sw; p++) v.merge(s_warp[((mine / Q) * sw + p) * Q + mine % Q]);
    s_cta[mine] = v;
  }
  if (csize > 1) cluster.sync();
  if (rank == 0 && has) {
    for (int r = 1; r < csize; r++) v.merge(cluster.map_shared_rank(s_cta, r)[mine]);
    const long long qi = tile0 * Q + mine;
    if (qi < nq) {
      Acc::store(out, grads, nq, qi, v, kp);
      if (contribs) contribs[qi] = (int)t.n;
    }
  }
  // Peers keep their shared memory alive until rank 0 has read it.
  if (csize > 1) cluster.sync();
}

// How a call's warps and clusters split the sources.
struct SplitShape {
  int sw, csize;
  double cost;  // rounds of resident CTAs x share of the sources each takes
};

// Every warp does Q queries x n / (sw * csize) sources, and ending a warp's sum
// takes about as long as 250 sources, 250 more across a cluster.  Of the shapes
// that leave a lane a group of sources, the one with the least of rounds x
// (sources of a part + that); below one round of resident CTAs the time does not
// fall, above it half a round covers the last one's tail.  Measured (us, sw x
// csize, smooth distance): 1M sources x 997 queries 1x1 6,292, 8x1 720, 8x2 603,
// 8x8 570 (chosen), 8x16 649; 65,536 x 16,000 1x1 647, 8x1 515 (chosen), 8x2 541;
// 20,000 x 262,144 1x1 2,470 (chosen 2x1, 2,511), 8x1 2,627.
inline SplitShape split_shape(long long nq, long long n, int q_per_warp, int ctas_per_sm,
                              int sm_count) {
  SplitShape best = {1, 1, -1.0};
  for (int sw = 1; sw <= kSplitWarps; sw *= 2) {
    const long long per_cta = (long long)(kSplitWarps / sw) * q_per_warp;
    for (int c = 1; c <= 16; c *= 2) {
      const int parts = sw * c;
      if (parts > 1 && n < (long long)parts * 32 * kSplitGroup) break;
      // a cluster sits inside one GPC, and a GPC's last SMs may not hold another:
      // 284, 264 and 224 of 296 CTAs in clusters of 4, 8 and 16
      const double fit = c <= 2 ? 1.0 : c == 4 ? 0.96 : c == 8 ? 0.89 : 0.757;
      const double rounds =
          (double)((nq + per_cta - 1) / per_cta * c) / (sm_count * ctas_per_sm * fit);
      const double cost =
          std::max(1.0, rounds + 0.5) * ((double)n / parts + (c > 1 ? 500.0 : 250.0));
      if (best.cost < 0.0 || cost < best.cost * 0.999) best = {sw, c, cost};
    }
  }
  return best;
}

// A cluster of 16 is more than every context must be able to place (8 is not): where
// one cannot, the launch is refused and the call runs in clusters of 8.
template <class Acc, int DIM>
cudaError_t launch_split(const DevTree& t, const float* q, long long nq, const KParams& kp,
                         float* out, float* grads, int* contribs, cudaStream_t stream,
                         const SplitShape& shape) {
  const long long per_cta = (long long)(kSplitWarps / shape.sw) * Acc::Q;
  const long long tiles = (nq + per_cta - 1) / per_cta;
  auto launch = [&](int csize) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * csize), 1, 1);
    cfg.blockDim = dim3(kSplitThreads, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, split_sum_kernel<Acc, DIM>, t, q, nq, kp, shape.sw, out, grads,
                              contribs);
  };
  if (shape.csize <= 8) return launch(shape.csize);
  cudaError_t e = cudaFuncSetAttribute(split_sum_kernel<Acc, DIM>,
                                       cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = launch(shape.csize);
  if (e == cudaSuccess) return e;
  cudaGetLastError();
  return launch(8);
}

// Few sources and many queries: a lane per Acc::Q queries (sum_all), without the merging
// of lanes' sums, which takes as long as 250 sources.
template <class Acc, int DIM>
__global__ void __launch_bounds__(kSplitThreads, Acc::kMinCtas)
    lane_query_kernel(DevTree t, const float* __restrict__ qsoa, long long nq, KParams kp,
                      float* __restrict__ out, float* __restrict__ grads,
                      int* __restrict__ contribs) {
  const long long q0 = ((long long)blockIdx.x * kSplitThreads + threadIdx.x) * Acc::Q;
  if (q0 >= nq) return;
  Acc acc;
  acc.load(qsoa, nq, q0, kp);
  sum_all(acc, t.pt_pm, t.pt_nrm, t.n);
#pragma unroll
  for (int j = 0; j < Acc::Q; j++) {
    if (q0 + j >= nq) break;
    Acc::store(out, grads, nq, q0 + j, acc.sum(j), kp);
    if (contribs) contribs[q0 + j] = (int)t.n;
  }
}

// Where that is the faster form: the call lasts as long as one lane's sum over all
// sources, so the queries have to be many beside them, and beyond a few hundred sources
// (some thousands for gradients, whose merging is longer) a warp's shared loads win.
// Measured (us, split / lane per query, 3D): Plummer, 100 sources: 10,000 queries 7.5 /
// 11.0, 30,000 13.0 / 10.9, 400,000 68 / 22; 300: 60,000 17 / 24, 100,000 25 / 24; 600:
// 200,000 60 / 50; 1,000: 400,000 156 / 180, 2M 750 / 574; gradients of the smooth
// distance, 100: 10,000 27 / 17, 400,000 554 / 50; 1,000: 60,000 151 / 121; 4,000: 200,000
// 981 / 1,001, 400,000 1,931 / 1,471.
inline bool lane_per_query(long long nq, long long n, int sm_count, bool gradients) {
  if (gradients) return n <= 4096 && 2 * nq >= n * sm_count;
  return n <= (nq >= 8192LL * sm_count ? 2048 : 768) && nq >= 2 * n * sm_count;
}

template <class Acc, int DIM>
cudaError_t launch_lane_query(const DevTree& t, const float* q, long long nq, const KParams& kp,
                              float* out, float* grads, int* contribs, cudaStream_t stream) {
  const long long per_cta = (long long)kSplitThreads * Acc::Q;
  lane_query_kernel<Acc, DIM><<<(unsigned)((nq + per_cta - 1) / per_cta), kSplitThreads, 0,
                                stream>>>(t, q, nq, kp, out, grads, contribs);
  return cudaGetLastError();
}

}  // namespace
}  // namespace sbh
