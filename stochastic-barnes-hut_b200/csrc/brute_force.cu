// All-pairs summation (replaces bruteForceSummationGPU, reference
// include/brute_force_gpu.h:18-66, and its wrappers src/sbh_gpu.cu:39-77).
//
// Design (B200):
//   * A warp carries 8 queries (2 in calls of few) and its lanes split the sources;
//     warps of a CTA and CTAs of a cluster split them further as the call's shape
//     asks (split_sum.cuh).  With a query per thread instead -- the sources
//     staged in shared memory -- a call of up to 4,000 queries filled 16 of the
//     148 SMs with two warps each: 997 queries x 1,000,003 sources, smooth
//     distance, took 11,697 us, now 570.
//   * The queries are packed pairs and the pairwise arithmetic runs on Blackwell's
//     FP32x2 instructions (FADD2 / FMUL2 / FFMA2, two lanes of FP32 per issue): a
//     Plummer pair costs 3.5 FP32 issue slots plus one MUFU rsqrt.  Both pipes are
//     loaded: 65,536 x 65,536 Plummer pairs take 1,180 us (0.79 of the MUFU bound;
//     1,350 with a query per thread), smooth distance 1,980 (2,322), winding
//     number 2,348 (2,519), gravity 1,919 (2,309).
//   * Compensated accumulation in two levels: plain FP32 over 32 sources of a
//     lane, then a Knuth two-sum into a (sum, error) pair -- the reference's Kahan
//     loop (brute_force_gpu.h:52-60) at a fraction of its cost per pair.
#include "launch.h"
#include "pairs.cuh"
#include "split_sum.cuh"
#include "tasks.cuh"

namespace sbh {
namespace {

template <int DIM, int K>
cudaError_t launch_bf(const DevTree& t, const float* q, long long nq, const KParams& kp, float* out,
                      cudaStream_t stream, int sm_count) {
  // 8 queries a warp, or 2 where that spreads a call of few over more warps: per
  // source a warp of 2 takes 0.55 of the time of one of 8.  Measured (us, 8 / 2 a
  // warp, smooth distance, 1M sources): 1 query 65 / 40, 40 67 / 52, 200 151 / 156.
  using Eight = PlainAcc<DIM, K, 4>;
  using Two = PlainAcc<DIM, K, 1>;
  if (lane_per_query(nq, t.n, sm_count, false))
    return launch_lane_query<Two, DIM>(t, q, nq, kp, out, nullptr, nullptr, stream);
  const SplitShape s8 = split_shape(nq, t.n, Eight::Q, Eight::kMinCtas, sm_count);
  const SplitShape s2 = split_shape(nq, t.n, Two::Q, Two::kMinCtas, sm_count);
  if (0.55 * s2.cost < s8.cost)
    return launch_split<Two, DIM>(t, q, nq, kp, out, nullptr, nullptr, stream, s2);
  return launch_split<Eight, DIM>(t, q, nq, kp, out, nullptr, nullptr, stream, s8);
}

}  // namespace

cudaError_t launch_brute_force(const DevTree& t, int kernel, const float* q, long long nq,
                               const KParams& kp, float* out, cudaStream_t stream, int sm_count) {
  if (nq <= 0) return cudaSuccess;
#define SBH_BF_CASE(D, K) \
  if (t.dim == D && kernel == K) return launch_bf<D, K>(t, q, nq, kp, out, stream, sm_count);
  SBH_BF_CASE(3, kGravity)
  SBH_BF_CASE(3, kWindingNumber)
  SBH_BF_CASE(3, kSmoothDist)
  SBH_BF_CASE(3, kPlummer)
  SBH_BF_CASE(2, kGravity)
  SBH_BF_CASE(2, kWindingNumber)
  SBH_BF_CASE(2, kSmoothDist)
  SBH_BF_CASE(2, kPlummer)
#undef SBH_BF_CASE
  return cudaErrorInvalidValue;
}

}  // namespace sbh
