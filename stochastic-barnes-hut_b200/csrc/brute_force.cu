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
//     number 2,348 (2,519), gravity 2,105 (2,309).
//   * Compensated accumulation in two levels: plain FP32 over 32 sources of a
//     lane, then a Knuth two-sum into a (sum, error) pair -- the reference's Kahan
//     loop (brute_force_gpu.h:52-60) at a fraction of its cost per pair.
#include "launch.h"
#include "pairs.cuh"
#include "split_sum.cuh"
#include "tasks.cuh"

namespace sbh {
namespace {

// A lane's compensated sum of one query.
struct PlainSum {
  float hi, lo;
  __device__ __forceinline__ void merge(const PlainSum& b) {
    two_sum_add(hi, lo, b.hi);
    lo += b.lo;
  }
};

// A lane's NP query pairs (split_sum.cuh).
template <int DIM, int K, int NP>
struct PlainAcc {
  using Sum = PlainSum;
  static constexpr int Q = 2 * NP;
  static constexpr int kMinCtas = NP == 4 ? 2 : K == kWindingNumber ? 3 : 4;  // no spills
  static constexpr bool kNormals = K == kWindingNumber;
  float2 nqx[NP], nqy[NP], nqz[NP], part[NP];
  float hi[Q], lo[Q];
  KParams kp;

  __device__ __forceinline__ void load(const float* qsoa, long long nq, long long q0,
                                       const KParams& params) {
    kp = params;
#pragma unroll
    for (int p = 0; p < NP; p++) {
      float3 a = make_float3(0.f, 0.f, 0.f), b = a;
      if (q0 + 2 * p < nq) a = load_query<DIM>(qsoa, nq, q0 + 2 * p);
      if (q0 + 2 * p + 1 < nq) b = load_query<DIM>(qsoa, nq, q0 + 2 * p + 1);
      nqx[p] = make_float2(-a.x, -b.x);
      nqy[p] = make_float2(-a.y, -b.y);
      nqz[p] = make_float2(-a.z, -b.z);
      part[p] = make_float2(0.f, 0.f);
      hi[2 * p] = lo[2 * p] = hi[2 * p + 1] = lo[2 * p + 1] = 0.f;
    }
  }
  template <int MODE>
  __device__ __forceinline__ void add(float4 s, float4 n) {
    const SrcPair sp = {dup(s.x), dup(s.y), dup(s.z), dup(s.w)};
    const NrmPair np = {dup(n.x), dup(n.y), dup(n.z), dup(0.f)};
#pragma unroll
    for (int p = 0; p < NP; p++)
      part[p] = accumulate2<DIM, K, MODE>(part[p], sp, np, nqx[p], nqy[p], nqz[p], kp);
  }
  __device__ __forceinline__ bool scaled() const { return K == kSmoothDist && kp.alpha >= 0.f; }
  __device__ __forceinline__ void group(const float4 (&s)[kSplitGroup],
                                        const float4 (&n)[kSplitGroup]) {
    static_assert(kSplitGroup == kSdFmaEvery, "one source of a group on the FP32 pipe");
    if (scaled()) {
      add<2>(s[0], n[0]);
#pragma unroll
      for (int i = 1; i < kSplitGroup; i++) add<1>(s[i], n[i]);
    } else {
#pragma unroll
      for (int i = 0; i < kSplitGroup; i++) add<0>(s[i], n[i]);
    }
  }
  __device__ __forceinline__ void single(float4 s, float4 n) {
    if (scaled())
      add<1>(s, n);
    else
      add<0>(s, n);
  }
  __device__ __forceinline__ void flush() {
#pragma unroll
    for (int p = 0; p < NP; p++) {
      if (scaled()) part[p] = __fmul2_rn(part[p], dup(kExp2Unscale));
      two_sum_add(hi[2 * p], lo[2 * p], part[p].x);
      two_sum_add(hi[2 * p + 1], lo[2 * p + 1], part[p].y);
      part[p] = make_float2(0.f, 0.f);
    }
  }
  __device__ __forceinline__ Sum sum(int j) const { return Sum{hi[j], lo[j]}; }
  __device__ __forceinline__ static void store(float* out, float*, long long, long long qi,
                                               const Sum& s, const KParams&) {
    const float v = s.hi + s.lo;
    out[qi] = K == kGravity ? -v : v;
  }
};

template <int DIM, int K>
cudaError_t launch_bf(const DevTree& t, const float* q, long long nq, const KParams& kp, float* out,
                      cudaStream_t stream, int sm_count) {
  // 8 queries a warp, or 2 where that spreads a call of few over more warps: per
  // source a warp of 2 takes 0.55 of the time of one of 8.  Measured (us, 8 / 2 a
  // warp, smooth distance, 1M sources): 1 query 65 / 40, 40 67 / 52, 200 151 / 156.
  using Eight = PlainAcc<DIM, K, 4>;
  using Two = PlainAcc<DIM, K, 1>;
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
