// Batched evaluation: many requests (trees, kernels, methods, query counts) in
// one pipeline of persistent kernels, a CUDA graph.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "device_common.cuh"

namespace sbh {

struct PlainSum;  // a compensated sum (lane_sum.cuh)

// One request of a batch, as the device reads it.
struct BatchItem {
  int tree;                  // index into the engine's tree table
  int dim;                   // the tree's dimension
  int method;                // SBH_METHOD_*
  int kernel;                // SBH_KERNEL_*
  int samples;               // stochastic method
  float beta;                // Barnes-Hut
  int sort_bits;             // Morton bits per axis of the query bucketing (0: keep order)
  int unit_queries;          // queries per work unit
  int depth;                 // the tree's depth (sizes the launch's shared memory)
  KParams kp;
  unsigned long long seed;   // stochastic method
  const float* q;            // device SoA [dim][nq]
  float* out;                // device [nq]
  int* contribs;             // device [nq] or null
  const float* self_mass;    // device [nq] or null: subtract each query's own source term
  long long nq;
  long long query_base;      // index of q[0] within its whole request (keys the sampler's
                             // random streams when a request is split across batches)
  long long sort_base;       // first position of this request in the batch order array
  long long bucket_base;     // first bucket of this request
  long long buckets;         // buckets of this request
  long long unit_base;       // first work unit of this request within its class
  long long units;           // work units of this request
  int per_query;             // Barnes-Hut: a warp per query (bh_query_task)
  int split;                 // brute force: parts per tile that are units of their own
                             // (0: a unit sums all parts)
  long long partial_base;    // first tile sum of a split request's parts
  long long counter_base;    // first tile counter of a split request
};

// Requests are evaluated by one persistent kernel per class, each compiled for
// its own work alone, so none pays for another's registers: Barnes-Hut, the
// sampler, and brute force by dimension and kernel function.
enum BatchClass : int { kClassBh = 0, kClassSbh = 1, kClassBf = 2, kClasses = 2 + 8 };

__host__ __device__ inline int batch_class(int method, int dim, int kernel) {
  return method == 3 ? kClassSbh
         : (method == 1 || method == 2) ? kClassBh
                                        : kClassBf + (dim == 3 ? 0 : 4) + kernel;
}

struct BatchHeader {
  int n_items;
  int pad;
  long long total_queries;
  long long total_buckets;
  int item_begin[kClasses], item_end[kClasses];  // each class's items are contiguous
  long long total_units[kClasses];
  unsigned long long next_unit[kClasses];  // work counters of the persistent kernels
};

// Queries per work unit (one warp task) of warp-vote Barnes-Hut: 32, a lane
// each (brute force takes kBfTileQueries).  The sampler's and Barnes-Hut's unit
// sizes (queries per warp task) are tuned.
constexpr int kUnitQueriesWarp = 32;

class BatchEngine {
 public:
  // Schedule knobs (the autotuner's search space); results never depend on them.
  struct Tuning {
    int sampler_unit = 32;    // sampler queries per work unit (the first-level
                              // sum runs a lane per query of a unit)
    int bucket_queries = 8;   // target queries per Morton bucket
    int blocks_per_sm = 0;    // persistent CTAs per SM (0: as many as fit)
    int bh_unit = 32;         // Barnes-Hut queries per warp walk (1..32)
    // Stochastic requests of at least this many queries leave the batch and
    // run as single-call launches (0: never); read by the batch's caller.
    int direct_queries = 65536;
  };

  struct Limits {
    int max_items = 4096;
    long long max_queries = 1 << 20;   // sorted positions (sum of request sizes)
    int max_tree_depth = 128;          // deepest tree the engine will see
  };

  // Creates the engine on the current device; `trees` is a device table of
  // `n_trees` trees that batches index.
  BatchEngine(const Limits& lim, int sm_count);
  ~BatchEngine();
  BatchEngine(const BatchEngine&) = delete;
  BatchEngine& operator=(const BatchEngine&) = delete;

  // Orders `items` by method class (stably) and fills their bookkeeping
  // (sort/bucket/unit ranges, sort bits) in place; checks limits.  Returns an
  // error string or "".
  std::string plan(std::vector<BatchItem>& items, const std::vector<DevTree>& host_trees,
                   const Tuning& tuning) const;
  // Enqueues the batch on `stream` (items already planned with `tuning`):
  // copies the item table and header from pinned staging, then launches the
  // graph of the batch's launch shape.
  cudaError_t launch(const std::vector<BatchItem>& items, const DevTree* d_trees,
                     int* d_status, cudaStream_t stream, const Tuning& tuning);

  const Limits& limits() const { return lim_; }
  size_t device_bytes() const { return dev_bytes_; }
  // CTAs per SM of the evaluation kernels at full occupancy (the largest, at
  // the smallest launch shape).
  int max_blocks_per_sm() const {
    return *std::max_element(per_sm_, per_sm_ + kClasses);
  }

 private:
  // What a pipeline's graph is specialised for.
  struct Shape {
    int per_sm_cap = 0;  // the tuning's CTAs-per-SM cap (0: none)
    bool sorted = false;  // whether some request's queries are ordered
    int bh_stack = 0;    // Barnes-Hut stack entries per warp (0: no Barnes-Hut class)
    bool bh_query = false;  // whether the scratch holds bh_query_task's
    unsigned classes = 0;  // bit c: a kernel node for class c
    bool operator==(const Shape& o) const {
      return per_sm_cap == o.per_sm_cap && sorted == o.sorted && bh_stack == o.bh_stack &&
             bh_query == o.bh_query && classes == o.classes;
    }
  };
  struct Graph {
    Shape shape;
    unsigned enabled = 0;  // bit c: class c's kernel node runs
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaGraphNode_t node[kClasses] = {};
  };
  cudaError_t build_graph(const DevTree* d_trees, int* d_status, Graph& g);
  // The graph for a batch of this shape (built if need be).
  cudaError_t find_graph(const DevTree* d_trees, int* d_status, const Shape& shape,
                         cudaGraphExec_t* out);
  static void release(Graph& g);
  static void release_all(std::vector<Graph>& graphs);

  Limits lim_;
  int sm_count_;
  int per_sm_[kClasses] = {};  // at the smallest launch shape
  // device buffers
  void* dev_ = nullptr;
  size_t dev_bytes_ = 0;
  BatchHeader* d_header_ = nullptr;
  BatchItem* d_items_ = nullptr;
  unsigned* d_keys_ = nullptr;
  unsigned* d_hist_ = nullptr;
  int* d_order_ = nullptr;
  unsigned* d_qbox_ = nullptr;  // per request: its queries' bounding box
  unsigned* d_sums_ = nullptr;  // tile sums of the bucket scan
  PlainSum* d_partial_ = nullptr;  // split brute force: the tiles' sums, part by part ...
  unsigned* d_counters_ = nullptr;  // ... and how many of a tile's parts are done
  // pinned staging of header + items
  void* h_stage_ = nullptr;
  // instantiated pipelines of recurring shapes, the last used at the end; some with all
  // classes for shapes met once, and those shapes
  std::vector<Graph> graphs_, any_;
  std::vector<Shape> seen_;
  const DevTree* captured_trees_ = nullptr;
  int* captured_status_ = nullptr;
};

}  // namespace sbh
