// Adjoint evaluation: values and query-position gradients.
//
// The reference has no gradient path (its gravityGrad, include/kernel.h:61-66,
// is unused and is not the derivative of gravityPotential).  These kernels run
// the same three methods over the value-and-gradient policies of sums.cuh:
//   * gravity and Plummer: the potential and its analytic gradient, summed
//     term by term over exactly the terms the plain method sums;
//   * smooth distance: D = -log(sum_i exp(-alpha r_i)) / alpha and its gradient
//     sum_i w_i (q - p_i) / r_i / sum_i w_i (w_i = exp(-alpha r_i)), with the
//     sum kept max-shifted so it never underflows.
// Barnes-Hut opens the same nodes as the plain walk (bh_warp_task; the value of
// gravity and Plummer equals the plain result bit for bit) and differentiates
// each accepted term.  The stochastic method walks the same Philox paths as the
// plain sampler for the same seed (the paths depend only on tree, query and
// random stream) and differentiates every term of the estimator with the path
// weights held fixed: E[sum over paths of weight * grad(term)] = grad(sum) by
// the same argument that makes the value unbiased, so the gradient of gravity
// and Plummer, and the gradient of the sum behind the smooth distance, are
// unbiased.  The smooth distance's gradient is the ratio of the two unbiased
// estimates from the same paths (consistent, like D itself).
#include "../../include/sbh_b200.h"
#include "launch.h"
#include "split_sum.cuh"
#include "tasks.cuh"

namespace sbh {
namespace {

constexpr int AD_THREADS = 128;
constexpr int AD_WARPS = AD_THREADS / 32;

// ------------------------------------------------------------ Barnes-Hut ---

template <int DIM, int K, bool VOTE, class A>
__global__ void __launch_bounds__(AD_THREADS)
    bh_grad_kernel(DevTree t, const float* __restrict__ qsoa, long long nq,
                   const int* __restrict__ order, float beta, KParams kp,
                   float* __restrict__ out, float* __restrict__ grads,
                   int* __restrict__ contribs, int* status, int stack_cap) {
  extern __shared__ BhStackEntry s_stack[];
  const int warp = threadIdx.x >> 5;
  const long long slot0 = ((long long)blockIdx.x * AD_WARPS + warp) * 32;
  bh_warp_task<DIM, K, VOTE, A>(t, qsoa, nq, order, slot0, min(slot0 + 32, nq), beta, kp, out,
                                contribs, status, s_stack + warp * stack_cap, stack_cap, nullptr,
                                grads);
}

// A warp per query (bh_query_task): calls of up to bh_query_per_warp() queries.
template <int DIM, int K, class A>
__global__ void __launch_bounds__(AD_THREADS)
    bh_grad_query_kernel(DevTree t, const float* __restrict__ qsoa, long long nq,
                         const int* __restrict__ order, float beta, KParams kp,
                         float* __restrict__ out, float* __restrict__ grads,
                         int* __restrict__ contribs, int* status) {
  extern __shared__ float4 s_query[];
  const int warp = threadIdx.x >> 5;
  const long long slot = (long long)blockIdx.x * AD_WARPS + warp;
  if (slot >= nq) return;
  char* scratch = reinterpret_cast<char*>(s_query) + warp * bh_query_smem(t.depth);
  bh_query_task<DIM, K, A>(t, qsoa, nq, order ? (long long)__ldg(order + slot) : slot, beta, kp,
                           out, contribs, status, scratch, nullptr, grads);
}

// --------------------------------------------------------------- sampler ---

// Seven CTAs per SM, with a few spills, hide more of the path steps' loads than the
// five that the unbounded 96 registers allow (1M queries, 128 paths, us: 3D gravity
// 17,567 -> 14,949, smooth distance 18,966 -> 17,301, Plummer 17,838 -> 14,719; 2D
// 9,179 -> 8,925, 9,644 -> 9,709, 8,648 -> 8,625; eight: 2D Plummer 8,958).
template <int DIM, int K, class A, bool FEW>
__global__ void __launch_bounds__(AD_THREADS, 7)
    sbh_grad_kernel(DevTree t, const float* __restrict__ qsoa, long long nq,
                    int samples, unsigned long long seed, KParams kp, float* __restrict__ out, float* __restrict__ grads,
                    int* __restrict__ contribs, int* status, int group) {
  using V = typename A::V;
  extern __shared__ float s_mem[];
  const int warp = threadIdx.x >> 5;
  const SbhWarpSmem<V> ws = sbh_carve<V>(s_mem + (size_t)warp * sbh_warp_words<V>());
  const long long units = (nq + group - 1) / group;
  const long long stride = (long long)gridDim.x * AD_WARPS;
  for (long long u = (long long)blockIdx.x * AD_WARPS + warp; u < units; u += stride)
    sbh_warp_task<DIM, K, FEW, A>(t, qsoa, nq, u * group, min(nq, (u + 1) * group), 0, samples, seed,
                             kp, ws, status, out, contribs, nullptr, grads);
}

// ----------------------------------------------------------- brute force ---

// Compensated running sum of policy values: partial sums are merged
// with Knuth's two-sum on every component (after aligning the exponents of the
// max-shifted form).
template <class A>
struct CompSum;

template <int DIM, int K>
struct CompSum<SumGrad<DIM, K>> {
  GradValue hi{0.f, 0.f, 0.f, 0.f}, lo{0.f, 0.f, 0.f, 0.f};
  __device__ __forceinline__ void add(const GradValue& p) {
    two_sum_add(hi.v, lo.v, p.v);
    two_sum_add(hi.gx, lo.gx, p.gx);
    two_sum_add(hi.gy, lo.gy, p.gy);
    two_sum_add(hi.gz, lo.gz, p.gz);
  }
  __device__ __forceinline__ void merge(const CompSum& b) {
    add(b.hi);
    lo = GradValue{lo.v + b.lo.v, lo.gx + b.lo.gx, lo.gy + b.lo.gy, lo.gz + b.lo.gz};
  }
  __device__ __forceinline__ GradValue result() const {
    return GradValue{hi.v + lo.v, hi.gx + lo.gx, hi.gy + lo.gy, hi.gz + lo.gz};
  }
};

template <int DIM>
struct CompSum<SumLse<DIM>> {
  LseValue hi = SumLse<DIM>::zero(), lo{0.f, 0.f, 0.f, 0.f, 0.f};
  // A NaN exponent takes the first branch, here and at every later addition, and stays
  // NaN in s; a zero (m = -inf) adds nothing without a branch of its own.
  __device__ __forceinline__ void add(LseValue p) {
    if (!(p.m <= hi.m)) {
      const float f = hi.m == -__int_as_float(0x7f800000) ? 0.f : expf(hi.m - p.m);
      hi = LseValue{p.m, hi.s * f, hi.gx * f, hi.gy * f, hi.gz * f};
      lo = LseValue{p.m, lo.s * f, lo.gx * f, lo.gy * f, lo.gz * f};
    } else if (p.m < hi.m) {
      const float f = expf(p.m - hi.m);
      p = LseValue{hi.m, p.s * f, p.gx * f, p.gy * f, p.gz * f};
    }
    two_sum_add(hi.s, lo.s, p.s);
    two_sum_add(hi.gx, lo.gx, p.gx);
    two_sum_add(hi.gy, lo.gy, p.gy);
    two_sum_add(hi.gz, lo.gz, p.gz);
  }
  __device__ __forceinline__ void merge(const CompSum& b) {
    add(b.hi);
    const float f = b.hi.m == hi.m ? 1.f : expf(b.hi.m - hi.m);
    lo = LseValue{hi.m, lo.s + f * b.lo.s, lo.gx + f * b.lo.gx, lo.gy + f * b.lo.gy,
                  lo.gz + f * b.lo.gz};
  }
  __device__ __forceinline__ LseValue result() const {
    return LseValue{hi.m, hi.s + lo.s, hi.gx + lo.gx, hi.gy + lo.gy, hi.gz + lo.gz};
  }
};

// All pairs: the sources split over a warp's lanes (split_sum.cuh), NP query
// pairs per warp, the pair arithmetic packed (pairs.cuh).  Bound by the MUFU and
// FP32 pipes together (two MUFU and about 16 FP32 operations a pair).  Two pairs
// a warp; one measured 1.1 to 2.1 times the time.  Against a query per thread with
// IEEE roots and divisions (us): 4,001 queries x 262,144 sources in 2D, smooth
// distance 34,550 -> 867, gravity 47,130 -> 691, Plummer 42,081 -> 504; 30,000 x
// 65,536 in 3D 10,818 -> 2,207, 12,826 -> 1,608, 11,269 -> 1,216.  A group of sources is
// summed on its own first: a term outside the fast form's range (a source at the
// query, distances whose square leaves the FP32 normal range, NaN) makes the
// group's sum infinite or NaN, and that query's group is then evaluated term by
// term as the policies define it.
//
// The root r = r2 * rsqrt(r2) gets one Newton step, r + (r2 - r^2) rsqrt(r2) / 2:
// the MUFU's last bits would otherwise show in the smooth distance, which is r
// itself near a source.
template <int NP>
struct QueryPairs {
  float2 nx[NP], ny[NP], nz[NP];  // negated
  template <int DIM>
  __device__ __forceinline__ void load(const float* qsoa, long long nq, long long q0) {
#pragma unroll
    for (int p = 0; p < NP; p++) {
      float3 a = make_float3(0.f, 0.f, 0.f), b = a;
      if (q0 + 2 * p < nq) a = load_query<DIM>(qsoa, nq, q0 + 2 * p);
      if (q0 + 2 * p + 1 < nq) b = load_query<DIM>(qsoa, nq, q0 + 2 * p + 1);
      nx[p] = make_float2(-a.x, -b.x);
      ny[p] = make_float2(-a.y, -b.y);
      nz[p] = make_float2(-a.z, -b.z);
    }
  }
  __device__ __forceinline__ float3 query(int j) const {
    return j & 1 ? make_float3(-nx[j / 2].y, -ny[j / 2].y, -nz[j / 2].y)
                 : make_float3(-nx[j / 2].x, -ny[j / 2].x, -nz[j / 2].x);
  }
};

__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// r and its reciprocal y from r2.
__device__ __forceinline__ float2 root2(float2 r2, float2& y) {
  y = rsqrt2(r2);
  const float2 r0 = __fmul2_rn(r2, y);
  const float2 e = __ffma2_rn(neg2(r0), r0, r2);
  return __ffma2_rn(e, __fmul2_rn(dup(0.5f), y), r0);
}

__device__ __forceinline__ bool usable(float v) { return fabsf(v) <= 3.402823466e38f; }

// The group's sum for query q, term by term.
template <class A>
__device__ __noinline__ typename A::V slow_group(float4 s0, float4 s1, float4 s2, float4 s3,
                                                 float3 q, KParams kp) {
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  typename A::V v = A::add(A::zero(), A::point(s0, none, q, kp));
  v = A::add(v, A::point(s1, none, q, kp));
  v = A::add(v, A::point(s2, none, q, kp));
  return A::add(v, A::point(s3, none, q, kp));
}

// What the two forms of GradAcc share.
template <int DIM, class A, int NP>
struct GradBase {
  using Sum = CompSum<A>;
  static constexpr int Q = 2 * NP;
  static constexpr int kMinCtas = 2;
  static constexpr bool kNormals = false;
  QueryPairs<NP> q;
  Sum total[Q];
  KParams kp;
  // The policy's addition drops a term e^-inf, whose gradient may be NaN (0 times an
  // infinite distance); the compensated sum would keep it.
  __device__ __forceinline__ void single(float4 s, float4 n) {
#pragma unroll
    for (int j = 0; j < Q; j++) total[j].add(A::add(A::zero(), A::point(s, n, q.query(j), kp)));
  }
  __device__ __forceinline__ const Sum& sum(int j) const { return total[j]; }
  __device__ __forceinline__ static void store(float* out, float* grads, long long nq,
                                               long long qi, const Sum& s, const KParams& kp) {
    A::store(out, grads, nq, qi, s.result(), kp);
  }
};

// Gravity and Plummer (positive sums; gravity changes the sign when a run ends).
template <int DIM, int K, class A, int NP>
struct GradAcc : GradBase<DIM, A, NP> {
  using GradBase<DIM, A, NP>::q;
  using GradBase<DIM, A, NP>::total;
  using GradBase<DIM, A, NP>::kp;
  float2 v[NP], gx[NP], gy[NP], gz[NP];
  __device__ __forceinline__ void load(const float* qsoa, long long nq, long long q0,
                                       const KParams& params) {
    kp = params;
    q.template load<DIM>(qsoa, nq, q0);
#pragma unroll
    for (int p = 0; p < NP; p++) v[p] = gx[p] = gy[p] = gz[p] = dup(0.f);
  }
  __device__ __forceinline__ void group(const float4 (&s)[kSplitGroup],
                                        const float4 (&)[kSplitGroup]) {
#pragma unroll
    for (int p = 0; p < NP; p++) {
      float2 a = dup(0.f), ax = a, ay = a, az = a;
#pragma unroll
      for (int i = 0; i < kSplitGroup; i++) {
        const float2 dx = __fadd2_rn(dup(s[i].x), q.nx[p]), dy = __fadd2_rn(dup(s[i].y), q.ny[p]);
        const float2 dz = DIM == 3 ? __fadd2_rn(dup(s[i].z), q.nz[p]) : dup(0.f);
        float2 r2 = K == kPlummer ? __ffma2_rn(dx, dx, dup(kp.eps2)) : __fmul2_rn(dx, dx);
        r2 = __ffma2_rn(dy, dy, r2);
        if (DIM == 3) r2 = __ffma2_rn(dz, dz, r2);
        float2 y, t, c;
        if (K == kPlummer) {  // m / s^(1/2), m / s^(3/2)
          y = rsqrt2(r2);
          t = __fmul2_rn(dup(s[i].w), y);
          c = __fmul2_rn(__fmul2_rn(t, y), y);
        } else {  // m / (r + 0.1), m / (r (r + 0.1)^2)
          const float2 inv = rcp2(__fadd2_rn(root2(r2, y), dup(1e-1f)));
          t = __fmul2_rn(dup(s[i].w), inv);
          c = __fmul2_rn(__fmul2_rn(t, inv), y);
        }
        a = __fadd2_rn(a, t);
        ax = __ffma2_rn(c, dx, ax);
        ay = __ffma2_rn(c, dy, ay);
        if (DIM == 3) az = __ffma2_rn(c, dz, az);
      }
      if (!(usable(a.x) && usable(a.y))) {
        constexpr float sign = K == kGravity ? -1.f : 1.f;
        if (!usable(a.x)) {
          const GradValue w = slow_group<A>(s[0], s[1], s[2], s[3], q.query(2 * p), kp);
          a.x = sign * w.v, ax.x = sign * w.gx, ay.x = sign * w.gy, az.x = sign * w.gz;
        }
        if (!usable(a.y)) {
          const GradValue w = slow_group<A>(s[0], s[1], s[2], s[3], q.query(2 * p + 1), kp);
          a.y = sign * w.v, ax.y = sign * w.gx, ay.y = sign * w.gy, az.y = sign * w.gz;
        }
      }
      v[p] = __fadd2_rn(v[p], a);
      gx[p] = __fadd2_rn(gx[p], ax);
      gy[p] = __fadd2_rn(gy[p], ay);
      if (DIM == 3) gz[p] = __fadd2_rn(gz[p], az);
    }
  }
  __device__ __forceinline__ void flush() {
    constexpr float sign = K == kGravity ? -1.f : 1.f;
#pragma unroll
    for (int p = 0; p < NP; p++) {
      total[2 * p].add(GradValue{sign * v[p].x, sign * gx[p].x, sign * gy[p].x, sign * gz[p].x});
      total[2 * p + 1].add(
          GradValue{sign * v[p].y, sign * gx[p].y, sign * gy[p].y, sign * gz[p].y});
      v[p] = gx[p] = gy[p] = gz[p] = dup(0.f);
    }
  }
};

// Smooth distance: terms e^(t - m), t = -alpha r, against a query's own reference
// exponent m, raised when a group's largest t is kLag above it.  The MUFU's argument
// (t - m) log2 e is rounded at its own magnitude, so what m may lag behind the terms
// that count is a relative error of those terms.  Measured with the nearest sources 39
// above the first ones (median gradient error against FP64, 3D; 4,001 queries x 262,144
// sources in 2D, us): kLag 40 4.7e-7, 816; 8 6.7e-8, 839; 4 6.7e-8, 867; 2 6.7e-8,
// 907; 0 6.7e-8, 975; a running maximum with IEEE operations 7.1e-8.  What flushes to
// zero is below e^-83 of the largest term.
template <int DIM, class A, int NP>
struct GradAcc<DIM, kSmoothDist, A, NP> : GradBase<DIM, A, NP> {
  using GradBase<DIM, A, NP>::q;
  using GradBase<DIM, A, NP>::total;
  using GradBase<DIM, A, NP>::kp;
  float2 m[NP], s_[NP], gx[NP], gy[NP], gz[NP];
  __device__ __forceinline__ void load(const float* qsoa, long long nq, long long q0,
                                       const KParams& params) {
    kp = params;
    q.template load<DIM>(qsoa, nq, q0);
#pragma unroll
    for (int p = 0; p < NP; p++) {
      m[p] = dup(-__int_as_float(0x7f800000));
      s_[p] = gx[p] = gy[p] = gz[p] = dup(0.f);
    }
  }
  static constexpr float kLag = 4.f;
  // Factor that takes sums from reference exponent m to the higher one, tm.
  __device__ __forceinline__ static float raise(float& m, float tm) {
    if (!(tm > m + kLag) || !usable(tm)) return 1.f;
    const float f = expf(m - tm);
    m = tm;
    return f;
  }
  __device__ __forceinline__ void group(const float4 (&s)[kSplitGroup],
                                        const float4 (&)[kSplitGroup]) {
#pragma unroll
    for (int p = 0; p < NP; p++) {
      float2 t[kSplitGroup], y[kSplitGroup], dx[kSplitGroup], dy[kSplitGroup], dz[kSplitGroup];
#pragma unroll
      for (int i = 0; i < kSplitGroup; i++) {
        dx[i] = __fadd2_rn(dup(s[i].x), q.nx[p]);
        dy[i] = __fadd2_rn(dup(s[i].y), q.ny[p]);
        dz[i] = DIM == 3 ? __fadd2_rn(dup(s[i].z), q.nz[p]) : dup(0.f);
        float2 r2 = __ffma2_rn(dy[i], dy[i], __fmul2_rn(dx[i], dx[i]));
        if (DIM == 3) r2 = __ffma2_rn(dz[i], dz[i], r2);
        t[i] = __fmul2_rn(dup(-kp.alpha), root2(r2, y[i]));
      }
      const float tx = fmaxf(fmaxf(t[0].x, t[1].x), fmaxf(t[2].x, t[3].x));
      const float ty = fmaxf(fmaxf(t[0].y, t[1].y), fmaxf(t[2].y, t[3].y));
      if (tx > m[p].x + kLag || ty > m[p].y + kLag) {
        const float2 f = make_float2(raise(m[p].x, tx), raise(m[p].y, ty));
        s_[p] = __fmul2_rn(s_[p], f);
        gx[p] = __fmul2_rn(gx[p], f);
        gy[p] = __fmul2_rn(gy[p], f);
        gz[p] = __fmul2_rn(gz[p], f);
      }
      float2 a = dup(0.f), ax = a, ay = a, az = a;
#pragma unroll
      for (int i = 0; i < kSplitGroup; i++) {
        const float2 u = __fmul2_rn(__fadd2_rn(t[i], neg2(m[p])), dup(1.44269504088896341f));
        const float2 w = make_float2(mufu_ex2_ftz(u.x), mufu_ex2_ftz(u.y));
        a = __fadd2_rn(a, w);
        const float2 c = __fmul2_rn(w, y[i]);
        ax = __ffma2_rn(c, dx[i], ax);
        ay = __ffma2_rn(c, dy[i], ay);
        if (DIM == 3) az = __ffma2_rn(c, dz[i], az);
      }
      if (!(usable(a.x) && usable(a.y))) {
        if (!usable(a.x)) {
          total[2 * p].add(slow_group<A>(s[0], s[1], s[2], s[3], q.query(2 * p), kp));
          a.x = ax.x = ay.x = az.x = 0.f;
        }
        if (!usable(a.y)) {
          total[2 * p + 1].add(slow_group<A>(s[0], s[1], s[2], s[3], q.query(2 * p + 1), kp));
          a.y = ax.y = ay.y = az.y = 0.f;
        }
      }
      s_[p] = __fadd2_rn(s_[p], a);
      gx[p] = __fadd2_rn(gx[p], ax);
      gy[p] = __fadd2_rn(gy[p], ay);
      if (DIM == 3) gz[p] = __fadd2_rn(gz[p], az);
    }
  }
  __device__ __forceinline__ void flush() {
    const float al = kp.alpha;
#pragma unroll
    for (int p = 0; p < NP; p++) {
      total[2 * p].add(LseValue{m[p].x, s_[p].x, al * gx[p].x, al * gy[p].x, al * gz[p].x});
      total[2 * p + 1].add(LseValue{m[p].y, s_[p].y, al * gx[p].y, al * gy[p].y, al * gz[p].y});
      s_[p] = gx[p] = gy[p] = gz[p] = dup(0.f);
    }
  }
  // The value's logarithm and its addition in FP64, one per query: m lies below the
  // largest term, log s is larger for it, and its FP32 rounding showed (value errors up
  // to 1.1 times a running maximum's, now 0.4 to 0.8).
  __device__ __forceinline__ static void store(float* out, float* grads, long long nq,
                                               long long qi, const CompSum<A>& s,
                                               const KParams& kp) {
    A::store(out, grads, nq, qi, s.result(), kp);
    out[qi] = (float)(-(s.hi.m + log((double)s.hi.s + s.lo.s)) / kp.alpha);
  }
};

// --------------------------------------------------------------- launch ---

template <int DIM, int K, class A>
cudaError_t launch_policy(const DevTree& t, int method, const float* q, long long nq,
                          const int* order, float beta, int samples, unsigned long long seed,
                          const KParams& kp, float* out, float* grads, int* contribs,
                          int* status, cudaStream_t stream, int sm_count) {
  if (method == SBH_METHOD_BRUTE_FORCE) {
    if (lane_per_query(nq, t.n, sm_count, true))
      return launch_lane_query<GradAcc<DIM, K, A, 1>, DIM>(t, q, nq, kp, out, grads, contribs,
                                                           stream);
    using Acc = GradAcc<DIM, K, A, 2>;
    const SplitShape shape = split_shape(nq, t.n, Acc::Q, Acc::kMinCtas, sm_count);
    return launch_split<Acc, DIM>(t, q, nq, kp, out, grads, contribs, stream, shape);
  }
  if (method == SBH_METHOD_BARNES_HUT && bh_query_per_warp(nq, t, sm_count)) {
    const size_t smem = AD_WARPS * bh_query_smem(t.depth);
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(bh_grad_query_kernel<DIM, K, A>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    const long long blocks = (nq + AD_WARPS - 1) / AD_WARPS;
    bh_grad_query_kernel<DIM, K, A><<<(unsigned)blocks, AD_THREADS, smem, stream>>>(
        t, q, nq, order, beta, kp, out, grads, contribs, status);
    return cudaGetLastError();
  }
  if (method == SBH_METHOD_BARNES_HUT || method == SBH_METHOD_BARNES_HUT_VOTE) {
    const int stack_cap = t.depth + 2;
    const size_t smem = (size_t)AD_WARPS * stack_cap * sizeof(BhStackEntry);
    const long long blocks = (nq + AD_THREADS - 1) / AD_THREADS;
    const auto kernel = method == SBH_METHOD_BARNES_HUT_VOTE ? bh_grad_kernel<DIM, K, true, A>
                                                             : bh_grad_kernel<DIM, K, false, A>;
    if (smem > 48 * 1024) {  // trees deeper than 766
      cudaError_t e =
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    kernel<<<(unsigned)blocks, AD_THREADS, smem, stream>>>(t, q, nq, order, beta, kp, out, grads,
                                                           contribs, status, stack_cap);
    return cudaGetLastError();
  }
  using V = typename A::V;
  const size_t smem = (size_t)AD_WARPS * sbh_warp_words<V>() * sizeof(float);
  const int group = sampler_group(nq, sm_count);
  long long blocks = ((nq + group - 1) / group + AD_WARPS - 1) / AD_WARPS;
  const long long cap = (long long)sm_count * 256;
  if (blocks > cap) blocks = cap;
  const auto kernel = group <= FewQueries<A>::kMax ? sbh_grad_kernel<DIM, K, A, true>
                                                   : sbh_grad_kernel<DIM, K, A, false>;
  if (smem > 48 * 1024) {
    cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  kernel<<<(unsigned)blocks, AD_THREADS, smem, stream>>>(t, q, nq, samples, seed, kp, out, grads,
                                                         contribs, status, group);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_gradient(const DevTree& t, int method, int kernel, const float* q, long long nq,
                            const int* order, float beta, int samples, unsigned long long seed,
                            const KParams& kp, float* out, float* grads, int* contribs,
                            int* status, cudaStream_t stream, int sm_count) {
  if (nq <= 0) return cudaSuccess;
  using G3 = SumGrad<3, kGravity>;
  using P3 = SumGrad<3, kPlummer>;
  using G2 = SumGrad<2, kGravity>;
  using P2 = SumGrad<2, kPlummer>;
#define SBH_AD_CASE(D, KID, POLICY)                                                             \
  if (t.dim == D && kernel == KID)                                                              \
    return launch_policy<D, KID, POLICY>(t, method, q, nq, order, beta, samples, seed, kp, out, \
                                         grads, contribs, status, stream, sm_count);
  SBH_AD_CASE(3, kGravity, G3)
  SBH_AD_CASE(3, kPlummer, P3)
  SBH_AD_CASE(3, kSmoothDist, SumLse<3>)
  SBH_AD_CASE(2, kGravity, G2)
  SBH_AD_CASE(2, kPlummer, P2)
  SBH_AD_CASE(2, kSmoothDist, SumLse<2>)
#undef SBH_AD_CASE
  return cudaErrorInvalidValue;
}

}  // namespace sbh
