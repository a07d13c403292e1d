// Host-side launchers of the summation kernels (internal to libsbh_b200.so).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "device_common.cuh"

namespace sbh {

cudaError_t launch_brute_force(const DevTree& t, int kernel, const float* q, long long nq,
                               const KParams& kp, float* out, cudaStream_t stream, int sm_count);

// Without neighbours sharing a warp the query order only helps the L1 cache; up
// to this many queries that is worth less than the ordering's seven launches
// (1M-point torus and 10,000-point Gaussian mixture: 16,000 queries 379 -> 384 and
// 122 -> 94 us without it; 65,536 1,015 -> 1,105 and 227 -> 220).
constexpr long long kBhUnorderedQueries = 16384;

// Barnes-Hut calls run a warp per query (bh_query_task) up to a number of queries, a
// lane per query (bh_warp_task) beyond.  A lane per query does a node test in fewer
// instructions, but a call lasts at least as long as its longest walk, one node after
// the other, and that grows with the tree.  Measured on B200 (us, lane / warp per query,
// theta 0.5): circle in 2D, 1,000 points: 20,000 queries 78 / 70, 40,000 104 / 101,
// 300,000 104 / 523; 150,000 points: 40,000 248 / 111, 150,000 363 / 284, 300,000 469 /
// 532; torus, 1,000 points: 40,000 431 / 197, 80,000 462 / 350, 300,000 429 / 1,185;
// 40,000 points: 150,000 1,498 / 1,004, 300,000 1,503 / 1,954; 1M points: 300,000 3,406 /
// 2,156; 500,000 (branching 64) 6,085 / 6,950.  Over 1,872 calls (2D and 3D, 100 to 1M
// points, leaves of 1 and 8, theta 0.2 to 0.8, gradients) this line costs 2% over the
// better of the two; 2,048 queries per SM whatever the tree cost 30%, and 5 times the
// lane walk's time on small trees.
inline bool bh_query_per_warp(long long nq, const DevTree& t, int sm_count) {
  const double per_sm = (t.dim == 3 ? 15.0 : 7.0) * std::sqrt((double)t.nn);
  return nq <= kBhUnorderedQueries || (double)nq <= std::min(per_sm, 2048.0) * sm_count;
}

// stage_leaves: accepted multi-point leaves are copied to shared memory by bulk
// asynchronous copies (SBH_FLAG_STAGE_LEAVES; not with vote).
cudaError_t launch_barnes_hut(const DevTree& t, int kernel, bool vote, const float* q,
                              long long nq, const int* order, float beta, const KParams& kp,
                              float* out, int* contribs, int* status, cudaStream_t stream,
                              int sm_count, bool stage_leaves = false);

// Queries a warp of the sampler takes at a time: a power of two up to 32 that
// leaves 64 to 128 units of work per SM (128 to 256 before 32 are taken; 32 warps
// of an SM run at once).  A warp's queries run one after the other, so a call lasts
// at least as long as one unit; sharing the first level among them is worth
// little by comparison.  Measured on B200 (us, 100,000-point Gaussian mixture, 256
// paths, groups of 1 / 4 / 8 / 16 / 32): 1,500 queries 131 / 350 / 619 / 1,177 / 2,202;
// 16,000 453 / 467 / 709 / 1,321 / 2,378; 100,000 2,488 / 2,208 / 2,241 / 2,622 /
// 3,003; 400,000 10,099 / 8,258 / 8,136 / 8,288 / 8,370.
int sampler_group(long long nq, int sm_count);

// self_mass (optional, indexed like the queries): subtract each query's own
// source term, as batched requests may ask.  query_base: index of q[0] within
// its whole request (keys the random streams of a request split into parts).
cudaError_t launch_stochastic(const DevTree& t, int kernel, const float* q, long long nq,
                              int samples, unsigned long long seed, const KParams& kp,
                              float* out, int* contribs, int* status, cudaStream_t stream,
                              int sm_count, const float* self_mass = nullptr, long long query_base = 0);

// Values and query-position gradients (adjoint.cu): method is SBH_METHOD_*,
// kernel gravity, Plummer or smooth distance; grads is SoA [dim][nq] or null.
cudaError_t launch_gradient(const DevTree& t, int method, int kernel, const float* q, long long nq,
                            const int* order, float beta, int samples, unsigned long long seed,
                            const KParams& kp, float* out, float* grads, int* contribs,
                            int* status, cudaStream_t stream, int sm_count);

// Spatial ordering of queries: order[i] is the i-th query in Morton-bucket
// order.  `ws` must hold query_sort_workspace_bytes(nq) bytes: the query box
// and the bucket scan's tile sums (1,280 B), 2^18 bucket counters, a key per
// query.
constexpr int kQuerySortBuckets = 1 << 18;
constexpr size_t kQuerySortHeadBytes = 256 + 1024;
constexpr size_t query_sort_workspace_bytes(long long nq) {
  return kQuerySortHeadBytes + (size_t)kQuerySortBuckets * 4 + (size_t)(nq > 0 ? nq : 1) * 4;
}
cudaError_t launch_query_sort(const float* q, long long nq, int dim, void* ws, int* order,
                              cudaStream_t stream);

cudaError_t launch_fill_int(int* p, long long n, int value, cudaStream_t stream);

}  // namespace sbh
