// Batched evaluation: a list of requests -- each its own tree, method, kernel,
// parameters and query count -- runs as one fixed pipeline, built once per launch
// shape as a CUDA graph:
//
//   (the first four only where some request's queries are ordered)
//   batch_bbox_kernel     the bounding box of every request's queries;
//   batch_keys_kernel     Morton bucket of every query of every request, inside
//                         its request's query box, with a per-request bucket
//                         count sized to the request (about 8 queries per
//                         bucket);
//   scan (scan.cuh)       one exclusive scan over all requests' buckets (each
//                         request's buckets follow the previous request's, so
//                         the scan also places every request at its offset);
//   batch_scatter_kernel  the sorted position of every query;
//   batch_eval_kernel<C>, batch_bf_kernel<D, K>
//                         a persistent kernel per class the batch has (Barnes-Hut,
//                         sampler, each kind of brute force), as parallel
//                         branches of the graph: warps take that class's work
//                         units from its atomic counter and run the same device
//                         routines as the single-call kernels (tasks.cuh,
//                         lane_sum.cuh), the traversals dispatching on kernel and
//                         dimension per unit.  Each is compiled for its own work
//                         alone, so none carries the registers of the others.
//
// Every launch parameter of the graph is fixed (grids are persistent; sizes and
// the request table live in device memory, refreshed by one host-to-device copy
// before each launch), so one instantiated graph serves every batch.  Results
// are per request identical to a single call: Barnes-Hut is exact per query and
// the sampler's random streams are keyed by (seed, query index in its request).
#include <algorithm>
#include <cstring>

#include "batch.h"
#include "launch.h"
#include "scan.cuh"
#include "tasks.cuh"

namespace sbh {
namespace {

constexpr int kEvalThreads = 128;
constexpr int kEvalWarps = kEvalThreads / 32;
constexpr int kAuxThreads = 256;

__device__ __forceinline__ int find_item_by(const BatchItem* items, int n, long long v,
                                            long long BatchItem::*field) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (items[mid].*field <= v) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ unsigned spread(unsigned v, int bits, int stride) {
  unsigned r = 0;
  for (int b = 0; b < bits; b++) r |= ((v >> b) & 1u) << (stride * b);
  return r;
}

// Order-preserving map of floats to unsigned ints (for atomicMax), and back.
__device__ __forceinline__ unsigned to_ordered(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Per request, the bounding box of its queries (NaN queries excluded):
// qbox[6 * item + d] = ~to_ordered(min_d) and qbox[6 * item + 3 + d] =
// to_ordered(max_d), both reduced with atomicMax from zero.  A warp takes 32
// consecutive queries; while they all belong to one request it reduces them
// in registers and flushes once per request it met.
__global__ void batch_bbox_kernel(const BatchHeader* __restrict__ hdr,
                                  const BatchItem* __restrict__ items, unsigned* qbox) {
  const int n = hdr->n_items;
  const long long total = hdr->total_queries;
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * blockDim.x / 32;
  const long long wid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  int cur = -1;
  unsigned acc[6] = {0u, 0u, 0u, 0u, 0u, 0u};
  auto flush = [&]() {
    if (cur >= 0 && lane == 0)
      for (int k = 0; k < 6; k++)
        if (acc[k]) atomicMax(qbox + 6 * (size_t)cur + k, acc[k]);
  };
  for (long long base = wid * 32; base < total; base += warps * 32) {
    const long long g = base + lane;
    int item = -1;
    unsigned v[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    if (g < total) {
      item = find_item_by(items, n, g, &BatchItem::sort_base);
      const BatchItem& it = items[item];
      if (it.sort_bits > 0) {
        const long long i = g - it.sort_base;
        for (int d = 0; d < it.dim; d++) {
          const float x = it.q[d * it.nq + i];
          if (x == x) {
            v[d] = ~to_ordered(x);
            v[3 + d] = to_ordered(x);
          }
        }
      }
    }
    const int first = __shfl_sync(0xffffffffu, item, 0);
    if (__all_sync(0xffffffffu, item == first)) {
      if (first != cur) {
        flush();
        cur = first;
        for (int k = 0; k < 6; k++) acc[k] = 0u;
      }
      for (int k = 0; k < 6; k++) acc[k] = max(acc[k], __reduce_max_sync(0xffffffffu, v[k]));
    } else if (item >= 0) {
      for (int k = 0; k < 6; k++)
        if (v[k]) atomicMax(qbox + 6 * (size_t)item + k, v[k]);
    }
  }
  flush();
}

// Morton bucket of every query inside its request's query box (as the
// single-call sort does), counted into the request's buckets.
__global__ void batch_keys_kernel(const BatchHeader* __restrict__ hdr,
                                  const BatchItem* __restrict__ items,
                                  const unsigned* __restrict__ qbox, unsigned* keys,
                                  unsigned* hist) {
  const int n = hdr->n_items;
  const long long total = hdr->total_queries;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int item = find_item_by(items, n, g, &BatchItem::sort_base);
    const BatchItem& it = items[item];
    const long long i = g - it.sort_base;
    unsigned key = 0;
    const int bits = it.sort_bits;
    if (bits > 0) {
      const float cells = (float)(1 << bits);
      const int dim = it.dim;
      const unsigned* box = qbox + 6 * (size_t)item;
      unsigned c[3] = {0u, 0u, 0u};
      for (int d = 0; d < dim; d++) {
        const float lo = from_ordered(~__ldg(box + d)), hi = from_ordered(__ldg(box + 3 + d));
        const float ext = hi - lo;
        float f = ext > 0.f ? (it.q[d * it.nq + i] - lo) * (cells / ext) : 0.f;
        f = f == f ? fminf(fmaxf(f, 0.f), cells - 1.f) : 0.f;
        c[d] = (unsigned)f;
      }
      key = dim == 3 ? (spread(c[0], bits, 3) | (spread(c[1], bits, 3) << 1) |
                        (spread(c[2], bits, 3) << 2))
                     : (spread(c[0], bits, 2) | (spread(c[1], bits, 2) << 1));
    }
    const unsigned bucket = (unsigned)(it.bucket_base + key);
    keys[g] = bucket;
    atomicAdd(hist + bucket, 1u);
  }
}

__global__ void batch_scatter_kernel(const BatchHeader* __restrict__ hdr,
                                     const BatchItem* __restrict__ items,
                                     const unsigned* __restrict__ keys, unsigned* hist,
                                     int* order) {
  const int n = hdr->n_items;
  const long long total = hdr->total_queries;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const BatchItem& it = items[find_item_by(items, n, g, &BatchItem::sort_base)];
    const unsigned pos = atomicAdd(hist + keys[g], 1u);
    order[pos] = (int)(g - it.sort_base);
  }
}

constexpr int kTreeWords = (int)((sizeof(DevTree) + 15) / 16 * 4);
constexpr int kItemWords = (int)((sizeof(BatchItem) + 15) / 16 * 4);

// One work unit of a request, by method class; inlined into that class's
// kernel.  `t` is a register copy of the request's tree record.
template <int DIM, int K>
__device__ __forceinline__ void run_bh(const DevTree& t, const BatchItem& it, long long u,
                                       const int* ord, float* scratch, int stack_cap,
                                       int* status) {
  const long long s0 = u * it.unit_queries;
  const long long s1 = min(it.nq, s0 + it.unit_queries);
  BhStackEntry* stk = reinterpret_cast<BhStackEntry*>(scratch);
  if (it.method == 2)
    bh_warp_task<DIM, K, true>(t, it.q, it.nq, ord, s0, s1, it.beta, it.kp, it.out, it.contribs,
                               status, stk, stack_cap, it.self_mass);
  else
    bh_warp_task<DIM, K, false>(t, it.q, it.nq, ord, s0, s1, it.beta, it.kp, it.out,
                                it.contribs, status, stk, stack_cap, it.self_mass);
}

template <int DIM, int K, bool FEW>
__device__ __noinline__ void run_sbh(const DevTree& t, const BatchItem& it, long long u,
                                     float* scratch, int* status) {
  const SbhWarpSmem<float> ws = sbh_carve<float>(scratch);
  const long long s0 = u * it.unit_queries;
  const long long s1 = min(it.nq, s0 + it.unit_queries);
  for (long long s = s0; s < s1; s += 32)
    sbh_warp_task<DIM, K, FEW>(t, it.q, it.nq, s, min(s1, s + 32), it.query_base, it.samples,
                          it.seed, it.kp, ws, status, it.out, it.contribs, it.self_mass);
}

template <int DIM, int K>
__device__ __noinline__ void run_bh_query(const DevTree& t, const BatchItem& it, long long u,
                                          const int* ord, char* scratch, int* status) {
  const long long s1 = min(it.nq, (u + 1) * it.unit_queries);
  for (long long s = u * it.unit_queries; s < s1; s++)
    bh_query_task<DIM, K>(t, it.q, it.nq, ord ? (long long)__ldg(ord + s) : s, it.beta, it.kp,
                          it.out, it.contribs, status, scratch, it.self_mass);
}

// Brute force: a tile of kBfTileQueries queries against all parts of the sources
// (bf_parts), or, of a split request, against one of them; one warp
// (lane_sum.cuh).  The sums of one part go to `partials` ([tile][part][query]) and
// the tile's last unit, by its counter (at zero when the batch starts), merges them
// in part order and stores.  `tot` is the warp's scratch of kBfTileQueries sums.  The request's fields are read where they are needed, not carried
// through the sums' registers.
template <int DIM, int K>
__device__ __forceinline__ void run_bf(const DevTree& t, const BatchItem& it, long long u,
                                       PlainSum* tot, PlainSum* partials, unsigned* counters) {
  using Acc = PlainAcc<DIM, K, kBfTileQueries / 2>;
  const int lane = threadIdx.x & 31;
  const int split = it.split;
  const int tile = split ? (int)(u / split) : (int)u;
  const int part = split ? (int)(u - (long long)tile * split) : -1;
  const int p1 = split ? part + 1 : bf_parts(t.n);
  for (int p = split ? part : 0; p < p1; p++) {
    Acc acc;
    acc.load(it.q, it.nq, (long long)tile * kBfTileQueries, it.kp);
    const long long len = bf_part_sources(t.n);
    sum_range<Acc, !Acc::kNormals>(acc, t.pt_pm, t.pt_nrm, min(p * len, t.n),
                                   min((p + 1) * len, t.n));
#pragma unroll
    for (int j = 0; j < kBfTileQueries; j++) {
      PlainSum v = merge_lanes(acc.sum(j));
      if (lane == 0) {
        if (it.split == 0 && p > 0) {
          const PlainSum part_sum = v;
          v = tot[j];
          v.merge(part_sum);
        }
        tot[j] = v;
      }
    }
  }
  __syncwarp();
  PlainSum v = tot[lane & (kBfTileQueries - 1)];
  if (it.split) {
    // [part][query] sums of the tile; a lane per query
    float2* sums = reinterpret_cast<float2*>(partials + it.partial_base +
                                             (long long)tile * it.split * kBfTileQueries);
    unsigned* counter = counters + it.counter_base + tile;
    if (lane < kBfTileQueries) {
      __stcg(sums + part * kBfTileQueries + lane, make_float2(v.hi, v.lo));
      __threadfence();  // this part's sums before the count that announces them
    }
    __syncwarp();
    unsigned before = 0;
    if (lane == 0) before = atomicAdd(counter, 1u);
    before = __shfl_sync(0xffffffffu, before, 0);
    if (before + 1 != (unsigned)it.split) return;
    __threadfence();
    for (int p = 0; p < it.split; p++) {
      const float2 x = __ldcg(sums + p * kBfTileQueries + (lane & (kBfTileQueries - 1)));
      const PlainSum y = {x.x, x.y};
      if (p == 0)
        v = y;
      else
        v.merge(y);
    }
  }
  const long long qi = (long long)tile * kBfTileQueries + lane;
  if (lane < kBfTileQueries && qi < it.nq) {
    float r = v.hi + v.lo;
    if (K == kGravity) r = -r;  // accumulate2 adds +m / (r + 0.1)
    if (it.self_mass)
      r -= self_term<DIM, K>(load_query<DIM>(it.q, it.nq, qi), __ldg(it.self_mass + qi), it.kp);
    it.out[qi] = r;
    if (it.contribs) it.contribs[qi] = (int)t.n;
  }
}

template <int CLASS, int DIM, int K>
__device__ __forceinline__ void run_unit(const DevTree& t, const BatchItem& it, long long u,
                                         const int* order, float* scratch, int stack_cap,
                                         int* status) {
  const int* ord = it.sort_bits > 0 ? order + it.sort_base : nullptr;
  if (CLASS == kClassBh) {
    if (it.per_query)
      run_bh_query<DIM, K>(t, it, u, ord, reinterpret_cast<char*>(scratch), status);
    else
      run_bh<DIM, K>(t, it, u, ord, scratch, stack_cap, status);
  }
  if (CLASS == kClassSbh) {
    if (it.unit_queries <= FewQueries<SumF<DIM, K>>::kMax)
      run_sbh<DIM, K, true>(t, it, u, scratch, status);
    else
      run_sbh<DIM, K, false>(t, it, u, scratch, status);
  }
}

template <int CLASS>
__device__ __forceinline__ void dispatch_unit(const DevTree& t, const BatchItem& it, long long u,
                                              const int* order, float* scratch, int stack_cap,
                                              int* status) {
  const int key = (t.dim == 3 ? 0 : 4) + it.kernel;
  switch (key) {
    case 0: run_unit<CLASS, 3, kGravity>(t, it, u, order, scratch, stack_cap, status); break;
    case 1: run_unit<CLASS, 3, kWindingNumber>(t, it, u, order, scratch, stack_cap, status); break;
    case 2: run_unit<CLASS, 3, kSmoothDist>(t, it, u, order, scratch, stack_cap, status); break;
    case 3: run_unit<CLASS, 3, kPlummer>(t, it, u, order, scratch, stack_cap, status); break;
    case 4: run_unit<CLASS, 2, kGravity>(t, it, u, order, scratch, stack_cap, status); break;
    case 5: run_unit<CLASS, 2, kWindingNumber>(t, it, u, order, scratch, stack_cap, status); break;
    case 6: run_unit<CLASS, 2, kSmoothDist>(t, it, u, order, scratch, stack_cap, status); break;
    default: run_unit<CLASS, 2, kPlummer>(t, it, u, order, scratch, stack_cap, status); break;
  }
}

// A warp's turn through a class's work units: takes them from the class's counter
// and calls run(tree, item, unit) with the unit's tree and request records, which
// it keeps in the warp's shared memory (`wbase`), where the walks read them
// instead of holding them in registers.
template <class Run>
__device__ __forceinline__ void for_each_unit(BatchHeader* hdr, const BatchItem* __restrict__ items,
                                              const DevTree* __restrict__ trees, int cls,
                                              float* wbase, const Run& run) {
  const int lane = threadIdx.x & 31;
  const DevTree& ts = *reinterpret_cast<const DevTree*>(wbase);
  const BatchItem& it = *reinterpret_cast<const BatchItem*>(wbase + kTreeWords);
  const int ib = hdr->item_begin[cls], ie = hdr->item_end[cls];
  const long long total = hdr->total_units[cls];
  int cached_tree = -1, cached_item = -1;
  for (;;) {
    unsigned long long unit = 0;
    if (lane == 0) unit = atomicAdd(&hdr->next_unit[cls], 1ull);
    unit = __shfl_sync(0xffffffffu, unit, 0);
    if ((long long)unit >= total) break;
    const int item = ib + find_item_by(items + ib, ie - ib, (long long)unit, &BatchItem::unit_base);
    if (item != cached_item) {
      __syncwarp();
      const int* src = reinterpret_cast<const int*>(items + item);
      int* dst = reinterpret_cast<int*>(wbase + kTreeWords);
      for (int w = lane; w < (int)(sizeof(BatchItem) / 4); w += 32) dst[w] = __ldg(src + w);
      cached_item = item;
      __syncwarp();
    }
    if (it.tree != cached_tree) {
      const int tree = it.tree;
      __syncwarp();
      const int* src = reinterpret_cast<const int*>(trees + tree);
      int* dst = reinterpret_cast<int*>(wbase);
      for (int w = lane; w < (int)(sizeof(DevTree) / 4); w += 32) dst[w] = __ldg(src + w);
      cached_tree = tree;
      __syncwarp();
    }
    run(ts, it, (long long)unit - it.unit_base);
    __syncwarp();
  }
}

// The persistent kernel of a traversal class.  Minimum CTAs per SM: the
// single-call kernels' occupancy (sampler 8 at 64 registers, Barnes-Hut 10 at 48).
template <int CLASS>
__global__ void __launch_bounds__(kEvalThreads, CLASS == kClassSbh ? 8 : 10)
    batch_eval_kernel(BatchHeader* hdr, const BatchItem* __restrict__ items,
                      const DevTree* __restrict__ trees, const int* __restrict__ order,
                      int* status, int warp_words, int stack_cap) {
  extern __shared__ float4 s_eval[];
  float* wbase = reinterpret_cast<float*>(s_eval) + (size_t)(threadIdx.x >> 5) * warp_words;
  float* scratch = wbase + kTreeWords + kItemWords;
  for_each_unit(hdr, items, trees, CLASS, wbase,
                [&](const DevTree& t, const BatchItem& it, long long u) {
                  dispatch_unit<CLASS>(t, it, u, order, scratch, stack_cap, status);
                });
}

// The persistent kernel of one kind of brute force, 16 warps per SM as the single
// call's: in one kernel for all eight kinds the sums spilled 1 KB a thread, and
// 200,000 queries x 1M sources took 125 ms (smooth distance) instead of 95.  With
// 64 queries a warp against all sources in turn (sources staged in shared memory)
// they took 111, and a batch of few lasted as long as its longest unit: 40
// requests of 1 to 100,000 queries on trees of 10,000 to 2M points 159 ms, now 38;
// one query on 1M points 35.6 ms, now 0.18.
template <int DIM, int K>
__global__ void __launch_bounds__(kEvalThreads, 4)
    batch_bf_kernel(BatchHeader* hdr, const BatchItem* __restrict__ items,
                    const DevTree* __restrict__ trees, int warp_words, PlainSum* partial,
                    unsigned* counters) {
  extern __shared__ float4 s_eval[];
  float* wbase = reinterpret_cast<float*>(s_eval) + (size_t)(threadIdx.x >> 5) * warp_words;
  PlainSum* tot = reinterpret_cast<PlainSum*>(wbase + kTreeWords + kItemWords);
  for_each_unit(hdr, items, trees, batch_class(0, DIM, K), wbase,
                [&](const DevTree& t, const BatchItem& it, long long u) {
                  run_bf<DIM, K>(t, it, u, tot, partial, counters);
                });
}

// Per-warp shared words of a class's kernel for a launch shape: the tree and
// request records, then the class's scratch (Barnes-Hut stack of `bh_stack`
// entries or bh_query_task's scratch, or the sampler's).
int class_warp_words(int cls, int bh_stack, bool bh_query) {
  int scratch = 0;
  if (cls == kClassBh) scratch = bh_stack * (int)sizeof(BhStackEntry) / 4;
  if (cls == kClassBh && bh_query)
    scratch = std::max(scratch, (int)(bh_query_smem(bh_stack) / 4));
  if (cls == kClassSbh) scratch = sbh_warp_words<float>();
  if (cls >= kClassBf) scratch = kBfTileQueries * (int)sizeof(PlainSum) / 4;
  return kTreeWords + kItemWords + (scratch + 3) / 4 * 4;
}

size_t class_smem(int cls, int bh_stack, bool bh_query) {
  return (size_t)kEvalWarps * class_warp_words(cls, bh_stack, bh_query) * sizeof(float);
}

using BfKernel = void (*)(BatchHeader*, const BatchItem*, const DevTree*, int, PlainSum*, unsigned*);
const BfKernel kBfKernels[8] = {
    batch_bf_kernel<3, kGravity>,    batch_bf_kernel<3, kWindingNumber>,
    batch_bf_kernel<3, kSmoothDist>, batch_bf_kernel<3, kPlummer>,
    batch_bf_kernel<2, kGravity>,    batch_bf_kernel<2, kWindingNumber>,
    batch_bf_kernel<2, kSmoothDist>, batch_bf_kernel<2, kPlummer>};

const void* class_kernel(int cls) {
  if (cls == kClassBh) return reinterpret_cast<const void*>(batch_eval_kernel<kClassBh>);
  if (cls == kClassSbh) return reinterpret_cast<const void*>(batch_eval_kernel<kClassSbh>);
  return reinterpret_cast<const void*>(kBfKernels[cls - kClassBf]);
}

void allow_smem(int cls, size_t smem) {
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(class_kernel(cls), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

int class_occupancy(int cls, size_t smem) {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, class_kernel(cls), kEvalThreads, smem);
  return std::max(1, n);
}

// Launch shapes are rounded so that few graphs serve every batch: the stack
// to a multiple of 32 entries.
// Shared memory sized to the batch (not to the engine's limits) leaves the
// rest of each SM's 228 KB to the L1 cache the traversals depend on.
int round_stack(int need, const BatchEngine::Limits& lim) {
  return std::min((need + 31) / 32 * 32, lim.max_tree_depth + 2);
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Tile parts a batch may split its brute force into (16 MiB of sums).
constexpr long long kMaxTileParts = 1LL << 18;

// Bucket capacity: at least 2 queries per bucket (the tuning's lower bound),
// plus a bucket per request for requests below a full bucket.
long long max_buckets(const BatchEngine::Limits& lim) {
  return lim.max_queries / 2 + 2LL * lim.max_items + 1024;
}

int sort_bits_for(long long nq, int dim, int bucket_queries) {
  // About bucket_queries queries per bucket; 6 bits per axis (3D) / 9 (2D) at most.
  if (nq < 64) return 0;
  int bits = 0;
  const int cap = dim == 3 ? 6 : 9;
  while (bits < cap && (1LL << (dim * (bits + 1))) * bucket_queries <= nq) bits++;
  return bits;
}

}  // namespace

BatchEngine::BatchEngine(const Limits& lim, int sm_count) : lim_(lim), sm_count_(sm_count) {
  const long long nb = max_buckets(lim_);
  const size_t o_hdr = 0;
  const size_t o_items = o_hdr + align256(sizeof(BatchHeader));
  const size_t o_keys = o_items + align256(sizeof(BatchItem) * lim_.max_items);
  const size_t o_hist = o_keys + align256(sizeof(unsigned) * lim_.max_queries);
  const size_t o_order = o_hist + align256(sizeof(unsigned) * nb);
  const size_t o_qbox = o_order + align256(sizeof(int) * lim_.max_queries);
  const size_t o_sums = o_qbox + align256(sizeof(unsigned) * 6 * lim_.max_items);
  const size_t o_partial = o_sums + align256(sizeof(unsigned) * scan_tiles_for(nb));
  const size_t o_counters = o_partial + align256(sizeof(PlainSum) * kBfTileQueries * kMaxTileParts);
  dev_bytes_ = o_counters + align256(sizeof(unsigned) * kMaxTileParts / 2);
  if (cudaMalloc(&dev_, dev_bytes_) != cudaSuccess) {
    dev_ = nullptr;
    return;
  }
  char* b = static_cast<char*>(dev_);
  d_header_ = reinterpret_cast<BatchHeader*>(b + o_hdr);
  d_items_ = reinterpret_cast<BatchItem*>(b + o_items);
  d_keys_ = reinterpret_cast<unsigned*>(b + o_keys);
  d_hist_ = reinterpret_cast<unsigned*>(b + o_hist);
  d_order_ = reinterpret_cast<int*>(b + o_order);
  d_qbox_ = reinterpret_cast<unsigned*>(b + o_qbox);
  d_sums_ = reinterpret_cast<unsigned*>(b + o_sums);
  d_partial_ = reinterpret_cast<PlainSum*>(b + o_partial);
  d_counters_ = reinterpret_cast<unsigned*>(b + o_counters);
  if (cudaMallocHost(&h_stage_, o_keys) != cudaSuccess) h_stage_ = nullptr;
  // Allow each class's kernel the shared memory of the engine's largest
  // shape; report occupancy at the smallest (the register bound).
  const int big_stack = lim_.max_tree_depth + 2, small_stack = round_stack(0, lim_);
  for (int c = 0; c < kClasses; c++) allow_smem(c, class_smem(c, big_stack, true));
  for (int c = 0; c < kClasses; c++)
    per_sm_[c] = class_occupancy(c, class_smem(c, small_stack, false));
}

BatchEngine::~BatchEngine() {
  release_all(graphs_);
  release_all(any_);
  if (h_stage_) cudaFreeHost(h_stage_);
  if (dev_) cudaFree(dev_);
}

std::string BatchEngine::plan(std::vector<BatchItem>& items,
                              const std::vector<DevTree>& host_trees,
                              const Tuning& tuning) const {
  if (!dev_ || !h_stage_) return "batch engine has no device or pinned memory";
  if (tuning.sampler_unit < 1 || tuning.sampler_unit > 64 || tuning.bucket_queries < 2 ||
      tuning.bucket_queries > 4096 || tuning.blocks_per_sm < 0 || tuning.bh_unit < 1 ||
      tuning.bh_unit > 32)
    return "batch tuning out of range";
  if ((int)items.size() > lim_.max_items) return "too many requests in one batch";
  for (const BatchItem& it : items)
    if (it.tree < 0 || it.tree >= (int)host_trees.size()) return "request names an unknown tree";
  // Grouped by class; within the brute-force and sampler classes, the requests
  // whose work units cost most come first (brute force: sources per query;
  // sampler: sampled paths per query), so that the class's warps take the long
  // units early and the short ones fill in at the end.  The order changes no
  // result: every unit is summed by one warp on its own.
  auto class_of = [&](const BatchItem& it) {
    return batch_class(it.method, host_trees[it.tree].dim, it.kernel);
  };
  auto unit_cost = [&](const BatchItem& it) -> double {
    const DevTree& t = host_trees[it.tree];
    if (it.method == 0) return (double)t.n;
    if (it.method == 3) return (double)it.samples * t.root_children;
    return 0.0;
  };
  std::stable_sort(items.begin(), items.end(), [&](const BatchItem& a, const BatchItem& b) {
    const int ca = class_of(a), cb = class_of(b);
    if (ca != cb) return ca < cb;
    return unit_cost(a) > unit_cost(b);
  });
  long long sampled = 0, walked = 0;
  double bf_work = 0.0;  // sources read by all brute-force tiles
  for (const BatchItem& it : items) {
    if (it.method == 3) sampled += it.nq;
    if (it.method == 1) walked += it.nq;
    if (it.method == 0)
      bf_work += (double)((it.nq + kBfTileQueries - 1) / kBfTileQueries) *
                 (double)host_trees[it.tree].n;
  }
  // Barnes-Hut walks: a warp per query under the same rule as a single call, here by
  // the batch's queries, and in larger batches for requests of up to
  // kBhUnorderedQueries whose queries lie too far apart for neighbours to share a walk:
  // a twelfth of the tree's nodes at most in 3D, a hundredth in 2D (us, lane / warp per
  // query, theta 0.5: 100 requests of 10,000 queries, 3D Gaussian mixtures of 10,000
  // points 1,955 / 2,515, of 100,000 5,085 / 3,046, 2D circles of 1,000 469 / 2,181, of
  // 100,000 834 / 2,204; 1,000 of 1,000, 3D of 1,000 1,743 / 2,828, 2D of 100,000 4,328 /
  // 3,464); units of a few queries where there are many.
  auto per_query = [&](const BatchItem& it, const DevTree& t) {
    return it.method == 1 &&
           (bh_query_per_warp(walked, t, sm_count_) ||
            (it.nq <= kBhUnorderedQueries && it.nq * (t.dim == 3 ? 12 : 100) <= t.nn));
  };
  int walk_unit = 1;
  while (walk_unit < 8 && walked > 64LL * walk_unit * sm_count_) walk_unit *= 2;
  // Brute force: a tile's sum over all sources is one unit while that is at most
  // an eighth of a warp's share of the batch; longer ones are split into their
  // parts (largest trees first, as far as the partial sums' room goes), since the
  // batch ends with its longest unit.
  const double bf_share = bf_work / ((double)per_sm_[kClassBf] * kEvalWarps * sm_count_);
  long long tile_parts = 0, split_tiles = 0;
  const int sampler_unit = std::min(tuning.sampler_unit, sampler_group(sampled, sm_count_));
  long long sort_base = 0, bucket_base = 0, unit_base[kClasses] = {};
  for (BatchItem& it : items) {
    if (it.tree < 0 || it.tree >= (int)host_trees.size()) return "request names an unknown tree";
    const DevTree& t = host_trees[it.tree];
    if (t.depth + 2 > lim_.max_tree_depth + 2) return "tree deeper than the engine supports";
    it.per_query = per_query(it, t);
    // vote and the sampler keep the caller's order, and so do few walks
    const bool sorted = it.method == 1 && !(it.per_query && it.nq <= kBhUnorderedQueries);
    it.sort_bits =
        (sorted && it.sort_bits >= 0) ? sort_bits_for(it.nq, t.dim, tuning.bucket_queries) : 0;
    it.dim = t.dim;
    it.depth = t.depth;
    it.sort_base = sort_base;
    it.bucket_base = bucket_base;
    it.buckets = it.sort_bits > 0 ? (1LL << (t.dim * it.sort_bits)) : 1;
    it.unit_base = unit_base[class_of(it)];
    // Work unit: sampler queries per warp (tuned; fewer in batches of few, as in
    // a single call); Barnes-Hut queries per warp
    // walk (tuned; vote keeps 32, its acceptance is defined over 32 queries);
    // brute force kBfTileQueries per warp against all sources or a part of them.
    it.unit_queries = it.method == 3   ? sampler_unit
                      : it.method == 1 ? (it.per_query ? walk_unit : tuning.bh_unit)
                      : it.method == 0 ? kBfTileQueries
                                       : kUnitQueriesWarp;
    it.units = (it.nq + it.unit_queries - 1) / it.unit_queries;
    it.split = 0;
    if (it.method == 0) {
      const int parts = bf_parts(t.n);
      if (parts > 1 && (double)t.n > bf_share / 8 &&
          tile_parts + it.units * parts <= kMaxTileParts) {
        it.split = parts;
        it.partial_base = tile_parts * kBfTileQueries;
        it.counter_base = split_tiles;
        tile_parts += it.units * parts;
        split_tiles += it.units;
        it.units *= parts;
      }
    }
    sort_base += it.nq;
    bucket_base += it.buckets;
    unit_base[class_of(it)] += it.units;
  }
  if (sort_base > lim_.max_queries) return "batch exceeds the engine's query capacity";
  if (bucket_base > max_buckets(lim_)) return "batch exceeds the engine's bucket capacity";
  return "";
}

void BatchEngine::release(Graph& g) {
  if (g.exec) cudaGraphExecDestroy(g.exec);
  if (g.graph) cudaGraphDestroy(g.graph);
  g = Graph();
}

void BatchEngine::release_all(std::vector<Graph>& graphs) {
  for (Graph& g : graphs) release(g);
  graphs.clear();
}

// Builds the pipeline's graph of g's shape node by node.  (Capturing it
// from streams cost a stream and an event per branch, 0.5 ms each, and any other
// thread's device synchronisation -- a tree being destroyed -- invalidates a capture
// in progress.)
cudaError_t BatchEngine::build_graph(const DevTree* d_trees, int* d_status, Graph& g) {
  const Shape& shape = g.shape;
  cudaError_t e = cudaGraphCreate(&g.graph, 0);
  if (e != cudaSuccess) return e;
  cudaGraph_t graph = g.graph;
  using Nodes = std::vector<cudaGraphNode_t>;
  auto clear = [&](void* p, size_t words) {
    cudaGraphNode_t node = nullptr;
    cudaMemsetParams m = {};
    m.dst = p;
    m.elementSize = 4;
    m.width = words;
    m.height = 1;
    if (e == cudaSuccess) e = cudaGraphAddMemsetNode(&node, graph, nullptr, 0, &m);
    return node;
  };
  // Arguments are copied into the node.
  auto kernel = [&](const void* fn, unsigned grid, unsigned block, size_t smem, const Nodes& after,
                    auto... args) {
    cudaGraphNode_t node = nullptr;
    void* ptrs[] = {&args...};
    cudaKernelNodeParams k = {};
    k.func = const_cast<void*>(fn);
    k.gridDim = dim3(grid);
    k.blockDim = dim3(block);
    k.sharedMemBytes = (unsigned)smem;
    k.kernelParams = ptrs;
    if (e == cudaSuccess) e = cudaGraphAddKernelNode(&node, graph, after.data(), after.size(), &k);
    return node;
  };
  auto fn = [](auto* f) { return reinterpret_cast<const void*>(f); };
  const unsigned aux = sm_count_ * 4;
  const BatchHeader* hdr = d_header_;
  const BatchItem* items = d_items_;
  const unsigned *qbox = d_qbox_, *keys = d_keys_;
  Nodes ordered;
  if (shape.sorted) {
    const cudaGraphNode_t hist0 = clear(d_hist_, max_buckets(lim_));
    const cudaGraphNode_t box0 = clear(d_qbox_, 6 * (size_t)lim_.max_items);
    cudaGraphNode_t n =
        kernel(fn(batch_bbox_kernel), aux, kAuxThreads, 0, {box0}, hdr, items, d_qbox_);
    n = kernel(fn(batch_keys_kernel), aux, kAuxThreads, 0, {n, hist0}, hdr, items, qbox, d_keys_,
               d_hist_);
    // the scan of the buckets (launch_scan's three kernels)
    const long long* buckets = &d_header_->total_buckets;
    const long long fixed = 0;
    const unsigned tiles = (unsigned)scan_tiles_for(max_buckets(lim_));
    const unsigned *hist = d_hist_, *sums = d_sums_;
    n = kernel(fn(scan_tile_sums), tiles, kScanThreads, 0, {n}, hist, buckets, fixed, d_sums_);
    n = kernel(fn(scan_tile_offsets), 1, kScanThreads, 0, {n}, d_sums_, buckets, fixed);
    n = kernel(fn(scan_tiles), tiles, kScanThreads, 0, {n}, d_hist_, buckets, fixed, sums);
    n = kernel(fn(batch_scatter_kernel), aux, kAuxThreads, 0, {n}, hdr, items, keys, d_hist_,
               d_order_);
    ordered.push_back(n);
  }
  // The classes' kernels, parallel branches: they share no state but the item
  // table.  Only Barnes-Hut reads the ordering, but all start after it, Barnes-Hut
  // first: its walks end one by one and brute force fills in behind them (the
  // other way round the batch ends on the walks).
  for (int c = 0; c < kClasses; c++) {
    if (!((shape.classes >> c) & 1u)) continue;
    const size_t smem = class_smem(c, shape.bh_stack, shape.bh_query);
    const int fit = class_occupancy(c, smem);
    const unsigned blocks =
        (unsigned)((shape.per_sm_cap > 0 ? std::min(shape.per_sm_cap, fit) : fit) * sm_count_);
    const int words = class_warp_words(c, shape.bh_stack, shape.bh_query);
    if (c < kClassBf)
      g.node[c] = kernel(class_kernel(c), blocks, kEvalThreads, smem, ordered, d_header_, items,
                         d_trees, (const int*)d_order_, d_status, words, shape.bh_stack);
    else
      g.node[c] = kernel(class_kernel(c), blocks, kEvalThreads, smem, ordered, d_header_, items,
                         d_trees, words, d_partial_, d_counters_);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&g.exec, graph, 0);
  g.enabled = shape.classes;
  if (e != cudaSuccess) release(g);
  return e;
}

// A graph of the batch's own classes is the fastest to launch (with nodes switched from
// batch to batch the serving stream at twice the plain capacity fell from 22.3 to 20.6 M
// queries/s), and building one takes 0.1 to 2 ms, 0.1 a kernel.  So the first shapes
// get their own, and later ones when they come a second time; until then a graph of
// all classes serves them with the others' nodes switched off (45 us more).
cudaError_t BatchEngine::find_graph(const DevTree* d_trees, int* d_status, const Shape& shape,
                                    cudaGraphExec_t* out) {
  constexpr size_t kFirst = 8, kMost = 32;
  for (size_t i = 0; i < graphs_.size(); i++) {
    if (!(graphs_[i].shape == shape)) continue;
    std::rotate(graphs_.begin() + i, graphs_.begin() + i + 1, graphs_.end());
    *out = graphs_.back().exec;
    return cudaSuccess;
  }
  const auto again = std::find(seen_.begin(), seen_.end(), shape);
  if (graphs_.size() < kFirst || again != seen_.end()) {
    Graph g;
    g.shape = shape;
    cudaError_t e = build_graph(d_trees, d_status, g);
    if (e != cudaSuccess) return e;
    if (again != seen_.end()) seen_.erase(again);
    if (graphs_.size() >= kMost) {  // the one not used for longest
      release(graphs_.front());
      graphs_.erase(graphs_.begin());
    }
    graphs_.push_back(g);
    *out = g.exec;
    return cudaSuccess;
  }
  if (seen_.size() >= 64) seen_.erase(seen_.begin());
  seen_.push_back(shape);
  // One of all classes serves the batch if their other parameters agree (Barnes-Hut's
  // matter to a batch that has it, and not to a graph without it).
  constexpr unsigned kBh = 1u << kClassBh, kAll = (1u << kClasses) - 1u;
  size_t at = 0;
  for (; at < any_.size(); at++) {
    Shape s = any_[at].shape;
    if (shape.bh_stack == 0) s.bh_stack = 0, s.bh_query = false;
    s.classes = shape.classes;
    if (s == shape) break;
  }
  if (at == any_.size()) {
    Graph g;
    g.shape = shape;
    g.shape.classes = shape.bh_stack ? kAll : kAll & ~kBh;
    cudaError_t e = build_graph(d_trees, d_status, g);
    if (e != cudaSuccess) return e;
    if (any_.size() >= 4) {
      release(any_.front());
      any_.erase(any_.begin());
    }
    any_.push_back(g);
    at = any_.size() - 1;
  }
  Graph& g = any_[at];
  for (int c = 0; c < kClasses; c++) {
    const unsigned bit = 1u << c;
    if (((shape.classes ^ g.enabled) & bit) == 0) continue;
    cudaError_t e = cudaGraphNodeSetEnabled(g.exec, g.node[c], (shape.classes & bit) != 0);
    if (e != cudaSuccess) return e;
    g.enabled ^= bit;
  }
  *out = g.exec;
  return cudaSuccess;
}

cudaError_t BatchEngine::launch(const std::vector<BatchItem>& items, const DevTree* d_trees,
                                int* d_status, cudaStream_t stream, const Tuning& tuning) {
  if (!dev_ || !h_stage_) return cudaErrorMemoryAllocation;
  if (captured_trees_ != d_trees || captured_status_ != d_status) {
    release_all(graphs_);
    release_all(any_);
    seen_.clear();
    captured_trees_ = d_trees;
    captured_status_ = d_status;
  }
  int need_depth = -1;
  Shape shape;
  shape.per_sm_cap = std::max(0, tuning.blocks_per_sm);
  for (const BatchItem& it : items) {
    const int c = batch_class(it.method, it.dim, it.kernel);
    if (c == kClassBh) need_depth = std::max(need_depth, it.depth);
    shape.bh_query = shape.bh_query || it.per_query;
    shape.sorted = shape.sorted || it.sort_bits > 0;
    shape.classes |= 1u << c;
  }
  if (need_depth >= 0) shape.bh_stack = round_stack(need_depth + 2, lim_);
  cudaGraphExec_t exec = nullptr;
  cudaError_t e = find_graph(d_trees, d_status, shape, &exec);
  if (e != cudaSuccess) return e;
  BatchHeader h = {};
  long long split_tiles = 0;
  h.n_items = (int)items.size();
  for (int c = 0; c < kClasses; c++) h.item_begin[c] = h.item_end[c] = 0;
  int prev = -1;
  for (int i = 0; i < (int)items.size(); i++) {
    const BatchItem& it = items[i];
    const int c = batch_class(it.method, it.dim, it.kernel);
    if (c != prev) {
      h.item_begin[c] = i;
      prev = c;
    }
    h.item_end[c] = i + 1;
    h.total_queries += it.nq;
    h.total_buckets += it.buckets;
    h.total_units[c] += it.units;
    if (it.split) split_tiles += it.units / it.split;
  }
  char* st = static_cast<char*>(h_stage_);
  std::memcpy(st, &h, sizeof(h));
  const size_t o_items = align256(sizeof(BatchHeader));
  if (!items.empty()) std::memcpy(st + o_items, items.data(), sizeof(BatchItem) * items.size());
  e = cudaMemcpyAsync(d_header_, st, o_items + sizeof(BatchItem) * items.size(),
                      cudaMemcpyHostToDevice, stream);
  // The counters of this batch's split tiles, on the stream that runs it: nothing
  // else orders a clearing before a batch (the default stream's work does not come
  // before a non-blocking stream's).
  if (e == cudaSuccess && split_tiles > 0)
    e = cudaMemsetAsync(d_counters_, 0, sizeof(unsigned) * split_tiles, stream);
  if (e != cudaSuccess) return e;
  return cudaGraphLaunch(exec, stream);
}

}  // namespace sbh
