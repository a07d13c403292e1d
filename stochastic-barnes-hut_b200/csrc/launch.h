// Host-side launchers of the summation kernels (internal to libsbh_b200.so).
#pragma once

#include <cuda_runtime.h>

#include "device_common.cuh"

namespace sbh {

cudaError_t launch_brute_force(const DevTree& t, int kernel, const float* q, long long nq,
                               const KParams& kp, float* out, cudaStream_t stream, int sm_count);

// Barnes-Hut calls of up to 2,048 queries per SM run a warp per query
// (bh_query_task), larger ones a lane per query (bh_warp_task).  A lane per query
// does a node test in fewer instructions, but a call lasts at least as long as
// its longest walk, one node after the other.  Measured on B200 (us, lane / warp
// per query, theta 0.5): 1M-point torus, branching 64: 1,000 queries 2,910 / 170,
// 65,536 4,206 / 1,032, 200,000 5,207 / 2,833, 300,000 5,252 / 4,194, 500,000 6,085 /
// 6,950; 10,000-point Gaussian mixture, branching 8: 490 / 54, 603 / 236, 725 / 545,
// 689 / 799, 751 / 1,290; 65,536 points, leaf 8: 1,414 / 282, 2,009 / 576, 2,298 /
// 1,164, 2,370 / 1,635, 2,299 / 2,603.
inline bool bh_query_per_warp(long long nq, int sm_count) { return nq <= 2048LL * sm_count; }
// Without neighbours sharing a warp the query order only helps the L1 cache; up
// to this many queries that is worth less than the ordering's seven launches
// (16,000 queries on the same trees: 379 -> 384 and 122 -> 94 us without it;
// 65,536: 1,015 -> 1,105 and 227 -> 220).
constexpr long long kBhUnorderedQueries = 16384;

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
