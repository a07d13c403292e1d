// Summation arithmetic of the evaluators.
//
// The routines that add kernel values -- the Barnes-Hut walk, the sampler's
// expansions and estimator (tasks.cuh) and brute force -- are written once over
// a policy that says what a "value" is and how two are added:
//
//   SumF<DIM, K>     an FP32 kernel value, one IEEE rounding per operation: the
//                    reference's sums bit for bit (include/kernel.h:31-59).
//   SumGrad<DIM, K>  gravity or Plummer value plus its query-position gradient.
//                    The value is rounded exactly as SumF rounds it, so it equals
//                    the plain evaluation bit for bit; the gradient is an
//                    ordinary FP32 sum of the terms' analytic gradients, each
//                    rounded before it is added and without contractions left
//                    to the compiler, so that sums of the same terms in the same
//                    order agree bit for bit whichever routine forms them.
//   SumLse<DIM>      smooth distance in max-shifted form.  (m, s, g) stands for
//                    the sum e^m * s of exp(-alpha r) terms and for its gradient
//                    e^m * g; adding two values rescales the one with the smaller
//                    exponent, so no term underflows however far the query is
//                    from every source.  The stored result is the smooth distance
//                    D = -(m + log s) / alpha and its gradient -(g / s) / alpha.
//
// Each policy provides: V (the value type), zero(), nan(), add, sub, scale by a
// float, div by a float, warp shuffles of a value (shfl, shfl_up),
// segment_scan() (the inclusive sum over a lane's segment of the warp: `head` its
// first lane, `later` the first lanes of the segments after it), point() and
// node() (the value of one source record or
// node aggregate at query q), and store() (writes the result and, when the
// caller asks, the gradient as structure-of-arrays [dim][nq]).  For sums whose
// terms are evaluated by several lanes: kOrdered says that ordered(), the part of
// a value whose additions must happen in the reference's order, exists; add_rest()
// adds the other parts, which lanes may group as they like, and join() puts an
// ordered sum and the rest together.
#pragma once

#include "device_common.cuh"

namespace sbh {

template <int DIM, int K>
struct SumF {
  using V = float;
  static constexpr bool kGrad = false;
  static constexpr bool kOrdered = true;
  __device__ __forceinline__ static float ordered(V a) { return a; }
  __device__ __forceinline__ static V add_rest(V a, V) { return a; }
  __device__ __forceinline__ static V join(float sum, V) { return sum; }
  __device__ __forceinline__ static V zero() { return 0.f; }
  __device__ __forceinline__ static V nan() { return __int_as_float(0x7fc00000); }
  __device__ __forceinline__ static V add(V a, V b) { return radd(a, b); }
  __device__ __forceinline__ static V sub(V a, V b) { return rsub(a, b); }
  __device__ __forceinline__ static V scale(float w, V a) { return rmul(w, a); }
  __device__ __forceinline__ static V div(V a, float d) { return rdiv(a, d); }
  __device__ __forceinline__ static V shfl(V a, int src) {
    return __shfl_sync(0xffffffffu, a, src);
  }
  __device__ __forceinline__ static V shfl_up(V a, int d) {
    return __shfl_up_sync(0xffffffffu, a, d);
  }
  __device__ __forceinline__ static V segment_scan(V x, int head, unsigned) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const V y = shfl_up(x, d);
      if (lane - d >= head) x = add(y, x);
    }
    return x;
  }
  __device__ __forceinline__ static V point(float4 pm, float4 nr, float3 q, const KParams& kp) {
    return kernel_exact<DIM, K>(pm, nr, q, kp);
  }
  __device__ __forceinline__ static V node(float4 cm, float4 agg, float3 q, const KParams& kp) {
    return kernel_node<DIM, K>(cm, agg, q, kp);
  }
  __device__ __forceinline__ static void store(float* out, float*, long long, long long qi, V v,
                                               const KParams&) {
    out[qi] = v;
  }
};

struct GradValue {
  float v, gx, gy, gz;
};

// Gravity -m / (r + 0.1): gradient -m (p - q) / (r (r + 0.1)^2), 0 at r = 0.
// Plummer m / sqrt(r^2 + eps^2): gradient m (p - q) / (r^2 + eps^2)^(3/2).
template <int DIM, int K>
struct SumGrad {
  static_assert(K == kGravity || K == kPlummer, "gradients of gravity and Plummer only");
  using V = GradValue;
  static constexpr bool kGrad = true;
  static constexpr bool kOrdered = true;
  __device__ __forceinline__ static float ordered(V a) { return a.v; }
  __device__ __forceinline__ static V add_rest(V a, V b) {
    return V{a.v, radd(a.gx, b.gx), radd(a.gy, b.gy), radd(a.gz, b.gz)};
  }
  __device__ __forceinline__ static V join(float sum, V rest) {
    return V{sum, rest.gx, rest.gy, rest.gz};
  }
  __device__ __forceinline__ static V zero() { return V{0.f, 0.f, 0.f, 0.f}; }
  __device__ __forceinline__ static V nan() {
    const float n = __int_as_float(0x7fc00000);
    return V{n, n, n, n};
  }
  __device__ __forceinline__ static V add(V a, V b) {
    return V{radd(a.v, b.v), radd(a.gx, b.gx), radd(a.gy, b.gy), radd(a.gz, b.gz)};
  }
  __device__ __forceinline__ static V sub(V a, V b) {
    return V{rsub(a.v, b.v), rsub(a.gx, b.gx), rsub(a.gy, b.gy), rsub(a.gz, b.gz)};
  }
  __device__ __forceinline__ static V scale(float w, V a) {
    return V{rmul(w, a.v), rmul(w, a.gx), rmul(w, a.gy), rmul(w, a.gz)};
  }
  __device__ __forceinline__ static V div(V a, float d) {
    return V{rdiv(a.v, d), a.gx / d, a.gy / d, a.gz / d};
  }
  __device__ __forceinline__ static V shfl(V a, int src) {
    const unsigned f = 0xffffffffu;
    return V{__shfl_sync(f, a.v, src), __shfl_sync(f, a.gx, src), __shfl_sync(f, a.gy, src),
             DIM == 3 ? __shfl_sync(f, a.gz, src) : 0.f};
  }
  __device__ __forceinline__ static V shfl_up(V a, int d) {
    const unsigned f = 0xffffffffu;
    return V{__shfl_up_sync(f, a.v, d), __shfl_up_sync(f, a.gx, d), __shfl_up_sync(f, a.gy, d),
             DIM == 3 ? __shfl_up_sync(f, a.gz, d) : 0.f};
  }
  __device__ __forceinline__ static V segment_scan(V x, int head, unsigned) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const V y = shfl_up(x, d);
      if (lane - d >= head) x = add(y, x);
    }
    return x;
  }
  __device__ __forceinline__ static V point(float4 pm, float4 nr, float3 q, const KParams& kp) {
    const float v = kernel_exact<DIM, K>(pm, nr, q, kp);
    const float dx = pm.x - q.x, dy = pm.y - q.y, dz = DIM == 3 ? pm.z - q.z : 0.f;
    const float r2 = fmaf(dz, dz, fmaf(dy, dy, rmul(dx, dx)));
    float c;
    if (K == kGravity) {
      const float r = sqrtf(r2), rs = r + 1e-1f;
      c = r > 0.f ? -pm.w / (r * rs * rs) : 0.f;
    } else {
      const float s = r2 + kp.eps2;
      c = pm.w / (s * sqrtf(s));
    }
    return V{v, rmul(c, dx), rmul(c, dy), rmul(c, dz)};
  }
  __device__ __forceinline__ static V node(float4 cm, float4 agg, float3 q, const KParams& kp) {
    return point(make_float4(cm.x, cm.y, cm.z, agg.x), make_float4(agg.y, agg.z, agg.w, 0.f), q,
                 kp);
  }
  __device__ __forceinline__ static void store(float* out, float* grads, long long nq,
                                               long long qi, V v, const KParams&) {
    out[qi] = v.v;
    if (grads) {
      grads[qi] = v.gx;
      grads[nq + qi] = v.gy;
      if (DIM == 3) grads[2 * nq + qi] = v.gz;
    }
  }
};

struct LseValue {
  float m, s, gx, gy, gz;
};

// The larger of two, NaN if either is.
__device__ __forceinline__ float max_or_nan(float a, float b) {
  float y;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}

// Smooth distance exp(-alpha r): exponent t = -alpha r, gradient of t
// alpha (p - q) / r (0 at r = 0); a term is (t, 1, grad t).
template <int DIM>
struct SumLse {
  using V = LseValue;
  static constexpr bool kGrad = true;
  static constexpr bool kOrdered = false;
  __device__ __forceinline__ static float ordered(V) { return 0.f; }
  __device__ __forceinline__ static V add_rest(V a, V b) { return add(a, b); }
  __device__ __forceinline__ static V join(float, V rest) { return rest; }
  __device__ __forceinline__ static V zero() {
    return V{-__int_as_float(0x7f800000), 0.f, 0.f, 0.f, 0.f};
  }
  __device__ __forceinline__ static V nan() {
    const float n = __int_as_float(0x7fc00000);
    return V{n, n, n, n, n};
  }
  // A NaN stays in m: a zero's m, -inf, would otherwise be taken for "nothing here".
  __device__ __forceinline__ static V add(V a, V b) {
    if (a.m < b.m || b.m != b.m) {
      const V t = a;
      a = b;
      b = t;
    }
    if (b.m == -__int_as_float(0x7f800000)) return a;  // b is zero (and so is a if equal)
    const float f = expf(b.m - a.m);
    return V{a.m, fmaf(f, b.s, a.s), fmaf(f, b.gx, a.gx), fmaf(f, b.gy, a.gy),
             fmaf(f, b.gz, a.gz)};
  }
  __device__ __forceinline__ static V sub(V a, V b) {
    return add(a, V{b.m, -b.s, -b.gx, -b.gy, -b.gz});
  }
  __device__ __forceinline__ static V scale(float w, V a) {
    return V{a.m, rmul(w, a.s), rmul(w, a.gx), rmul(w, a.gy), rmul(w, a.gz)};
  }
  __device__ __forceinline__ static V div(V a, float d) {
    return V{a.m, a.s / d, a.gx / d, a.gy / d, a.gz / d};
  }
  __device__ __forceinline__ static V shfl(V a, int src) {
    const unsigned f = 0xffffffffu;
    return V{__shfl_sync(f, a.m, src), __shfl_sync(f, a.s, src), __shfl_sync(f, a.gx, src),
             __shfl_sync(f, a.gy, src), DIM == 3 ? __shfl_sync(f, a.gz, src) : 0.f};
  }
  __device__ __forceinline__ static V shfl_up(V a, int d) {
    const unsigned f = 0xffffffffu;
    return V{__shfl_up_sync(f, a.m, d), __shfl_up_sync(f, a.s, d), __shfl_up_sync(f, a.gx, d),
             __shfl_up_sync(f, a.gy, d), DIM == 3 ? __shfl_up_sync(f, a.gz, d) : 0.f};
  }
  // The terms of a segment are brought to its largest exponent first: one
  // exponential a lane instead of one at each of the five steps of the scan.
  __device__ __forceinline__ static V segment_scan(V x, int head, unsigned later) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    float top = x.m;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float y = __shfl_up_sync(full, top, d);
      if (lane - d >= head) top = max_or_nan(top, y);
    }
    top = __shfl_sync(full, top, later ? __ffs(later) - 2 : 31);
    const float f = x.m == -__int_as_float(0x7f800000) ? 0.f : expf(x.m - top);
    x = V{top, f * x.s, f * x.gx, f * x.gy, f * x.gz};
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const V y = shfl_up(x, d);
      if (lane - d >= head) {
        x.s += y.s;
        x.gx += y.gx;
        x.gy += y.gy;
        if (DIM == 3) x.gz += y.gz;
      }
    }
    return x;
  }
  __device__ __forceinline__ static V point(float4 pm, float4, float3 q, const KParams& kp) {
    const float dx = rsub(pm.x, q.x), dy = rsub(pm.y, q.y), dz = DIM == 3 ? rsub(pm.z, q.z) : 0.f;
    // The exponent exactly as the plain kernel forms it (include/kernel.h:55-58).
    const float r = rsqrt_ieee(dot_exact<DIM>(dx, dy, dz, dx, dy, dz));
    const float c = r == 0.f ? 0.f : kp.alpha / r;
    return V{rmul(-kp.alpha, r), 1.f, rmul(c, dx), rmul(c, dy), rmul(c, dz)};
  }
  __device__ __forceinline__ static V node(float4 cm, float4 agg, float3 q, const KParams& kp) {
    return point(make_float4(cm.x, cm.y, cm.z, agg.x), make_float4(agg.y, agg.z, agg.w, 0.f), q,
                 kp);
  }
  __device__ __forceinline__ static void store(float* out, float* grads, long long nq,
                                               long long qi, V v, const KParams& kp) {
    // log of a negative estimate is NaN, as -log(w)/alpha is for the reference's
    // callers (python/example.py:79); a zero sum gives +inf.
    out[qi] = -(v.m + logf(v.s)) / kp.alpha;
    if (grads) {
      const float k = -1.f / (kp.alpha * v.s);
      grads[qi] = k * v.gx;
      grads[nq + qi] = k * v.gy;
      if (DIM == 3) grads[2 * nq + qi] = k * v.gz;
    }
  }
};

}  // namespace sbh
