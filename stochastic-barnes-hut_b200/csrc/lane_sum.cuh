// A warp's sum of a range of sources for a few queries: every lane carries the same
// queries as packed pairs and takes every 32nd source (the all-pairs kernels,
// brute_force.cu and adjoint.cu through split_sum.cuh, and the batched
// brute-force task, tasks.cuh).  Lanes sum plain FP32 runs of kSplitRun sources and merge
// each into a compensated sum.
#pragma once

#include "device_common.cuh"
#include "pairs.cuh"

namespace sbh {

constexpr int kSplitGroup = 4;  // sources a lane loads at a time
constexpr int kSplitRun = 32;   // sources of a plain FP32 sum

template <class T>
__device__ __forceinline__ T shfl_down_words(const T& v, int d) {
  static_assert(sizeof(T) % 4 == 0, "word-sized members");
  T r;
  const int* src = reinterpret_cast<const int*>(&v);
  int* dst = reinterpret_cast<int*>(&r);
#pragma unroll
  for (int w = 0; w < (int)(sizeof(T) / 4); w++) dst[w] = __shfl_down_sync(0xffffffffu, src[w], d);
  return r;
}

// Adds the sources [c0, c1) to the lanes' state Acc (load() has read its
// queries): group() takes kSplitGroup sources of a lane, loaded while the
// group before is summed (PREFETCH; a kernel short of registers leaves the
// latency to its other warps), single() one, flush() ends a run.
template <class Acc, bool PREFETCH = true>
__device__ __forceinline__ void sum_range(Acc& acc, const float4* __restrict__ pt_pm,
                                          const float4* __restrict__ pt_nrm, long long c0,
                                          long long c1) {
  const int lane = threadIdx.x & 31;
  const long long full_end = c0 + (c1 - c0) / (32 * kSplitGroup) * (32 * kSplitGroup);
  long long base = c0;
  float4 s[kSplitGroup], nr[kSplitGroup], s2[kSplitGroup], nr2[kSplitGroup];
  auto fetch = [&](long long at, float4 (&s)[kSplitGroup], float4 (&nr)[kSplitGroup]) {
#pragma unroll
    for (int i = 0; i < kSplitGroup; i++) {
      s[i] = __ldg(pt_pm + at + 32 * i + lane);
      nr[i] = Acc::kNormals ? __ldg(pt_nrm + at + 32 * i + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (PREFETCH && base < full_end) fetch(base, s, nr);
  int run = 0;
  for (; base < full_end; base += 32 * kSplitGroup) {
    if (!PREFETCH) fetch(base, s, nr);
    if (PREFETCH && base + 32 * kSplitGroup < full_end) fetch(base + 32 * kSplitGroup, s2, nr2);
    acc.group(s, nr);
    if ((++run & (kSplitRun / kSplitGroup - 1)) == 0) acc.flush();
#pragma unroll
    for (int i = 0; PREFETCH && i < kSplitGroup; i++) {
      s[i] = s2[i];
      nr[i] = nr2[i];
    }
  }
  for (base += lane; base < c1; base += 32)
    acc.single(__ldg(pt_pm + base),
               Acc::kNormals ? __ldg(pt_nrm + base) : make_float4(0.f, 0.f, 0.f, 0.f));
  acc.flush();
}

// Adds all of the n sources to a lane's state, the lane's own queries: every lane reads
// the same sources.
template <class Acc>
__device__ __forceinline__ void sum_all(Acc& acc, const float4* __restrict__ pt_pm,
                                        const float4* __restrict__ pt_nrm, long long n) {
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  long long base = 0;
  int run = 0;
  for (; base + kSplitGroup <= n; base += kSplitGroup) {
    float4 s[kSplitGroup], nr[kSplitGroup];
#pragma unroll
    for (int i = 0; i < kSplitGroup; i++) {
      s[i] = __ldg(pt_pm + base + i);
      nr[i] = Acc::kNormals ? __ldg(pt_nrm + base + i) : none;
    }
    acc.group(s, nr);
    if ((++run & (kSplitRun / kSplitGroup - 1)) == 0) acc.flush();
  }
  for (; base < n; base++)
    acc.single(__ldg(pt_pm + base), Acc::kNormals ? __ldg(pt_nrm + base) : none);
  acc.flush();
}

// The lanes' sums of one query, merged into lane 0's.
template <class Sum>
__device__ __forceinline__ Sum merge_lanes(Sum v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v.merge(shfl_down_words(v, o));
  return v;
}

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
  // Spills (bytes loaded): 12 at most, but 40 and 112 in the 3D gravity and winding-number
  // kernels of one pair.
  static constexpr int kMinCtas = NP == 4 ? 2 : K == kWindingNumber ? 3 : 4;
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
  // Gravity: two sources share a reciprocal, a / b + c / d = (a d + c b) / (b d), one
  // MUFU operation and two more FP32 ones in place of two MUFU ones (with the
  // root 1.5 a pair instead of 2; the MUFU bound this kernel).  The product of
  // two denominators stays in range up to distances of 1e9; a group beyond them,
  // or whose sum is infinite or NaN, is evaluated a source at a time.  65,536 x
  // 65,536: 2,105 -> 1,919 us in 3D, 2,110 -> 1,697 in 2D, errors against FP64 as
  // before.  (The 3D winding number, whose FP32 work is nearly as long as its MUFU
  // work, went from 2,348 to 2,675 us with it and keeps a reciprocal a source.)
  static constexpr bool kShared = K == kGravity;
  __device__ __forceinline__ void shared_group(const float4 (&s)[kSplitGroup]) {
    constexpr float kLargest = 3.402823466e38f;
#pragma unroll
    for (int p = 0; p < NP; p++) {
      float2 acc = dup(0.f);
      float top = 0.f;
#pragma unroll
      for (int i = 0; i < kSplitGroup; i += 2) {
        float2 den[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const float4 v = s[i + h];
          const float2 dx = __fadd2_rn(dup(v.x), nqx[p]), dy = __fadd2_rn(dup(v.y), nqy[p]);
          float2 r2 = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
          if (DIM == 3) {
            const float2 dz = __fadd2_rn(dup(v.z), nqz[p]);
            r2 = __ffma2_rn(dz, dz, r2);
          }
          top = fmaxf(top, fmaxf(r2.x, r2.y));
          den[h] = __fadd2_rn(norm_from_sq(r2), dup(1e-1f));
        }
        const float2 num = __ffma2_rn(dup(s[i + 1].w), den[0], __fmul2_rn(dup(s[i].w), den[1]));
        acc = __ffma2_rn(num, rcp2(__fmul2_rn(den[0], den[1])), acc);
      }
      if (!(top <= 1e18f && fabsf(acc.x) <= kLargest && fabsf(acc.y) <= kLargest)) {
        const NrmPair none = {};
        acc = dup(0.f);
#pragma unroll 1
        for (int i = 0; i < kSplitGroup; i++) {
          const float4 v = i == 0 ? s[0] : i == 1 ? s[1] : i == 2 ? s[2] : s[3];
          const SrcPair sp = {dup(v.x), dup(v.y), dup(v.z), dup(v.w)};
          acc = accumulate2<DIM, K>(acc, sp, none, nqx[p], nqy[p], nqz[p], kp);
        }
      }
      part[p] = __fadd2_rn(part[p], acc);
    }
  }
  __device__ __forceinline__ bool scaled() const { return K == kSmoothDist && kp.alpha >= 0.f; }
  __device__ __forceinline__ void group(const float4 (&s)[kSplitGroup],
                                        const float4 (&n)[kSplitGroup]) {
    static_assert(kSplitGroup == kSdFmaEvery, "one source of a group on the FP32 pipe");
    if constexpr (kShared) {
      shared_group(s);
    } else if (scaled()) {
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

}  // namespace sbh
