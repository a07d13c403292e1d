// GPU tree build (sbh_gpu_tree_build): the reference's tree (Tree2D/Tree3D,
// include/tree3d.h:238-371) built level by level on the device, producing the
// same node numbering, child order, bounds, diameters, aggregates, point
// order and device image as building on the host (host_tree.cpp) and
// uploading.
//
// Why the result is the reference's, for leaf size 1:
//   * a node's children are its non-empty cells in cell order, numbered level
//     by level in node order then cell order (the reference's breadth-first
//     numbering, tree3d.h:291-301): the mask of a node's non-empty cells and a
//     scan of the masks' population counts give exactly those indices;
//   * cells, child bounds and diameters use the reference's FP32 formulas with
//     one IEEE rounding per operation (quantize, min + i*inc, |max - min|);
//   * the reference permutes points with std::partition, whose order inside a
//     cell differs from ours, but with one point per leaf the final order is
//     fixed by the leaves' order alone: position i holds the point of the leaf
//     whose range starts at i;
//   * aggregates are summed per node over its children in cell order (leaves:
//     its single point), as tree3d.h:310-327 does.
// What a build costs: 1,048,576 torus points, branching 64, take 4.0 ms, of which
// the pageable host-to-device copy of 28 MB is 1.5 and the kernels 1.1.
// The driver's calls were most of the 42 ms it took before -- about fifty
// cudaMalloc/cudaFree pairs at 0.65 ms, a device property query at 2.5, a stream at
// 0.5 -- so the scratch and the tree are two allocations from the library's pool.
// On the device, per-node histograms of all cells (217 MB at the widest level)
// became cell masks and per-child counts, and levels of few nodes count in shared
// memory first.
//
// For a leaf size above 1, or when the depth cap leaves several points in one
// leaf, the order of the points inside a leaf is std::partition's and this
// build cannot reproduce it: sbh_gpu_tree_build then builds on the host and
// uploads (same result).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "gpu_internal.h"
#include "scan.cuh"

namespace {

using sbh::DevTree;

constexpr int kThreads = 256;

int blocks_for(long long n) { return (int)std::max<long long>(1, (n + kThreads - 1) / kThreads); }

// Device arrays of the nodes (parts of the build's workspace).  A node is a leaf
// when it has no children.
struct Nodes {
  int mw = 1;
  int *start = nullptr, *cnt = nullptr, *first = nullptr, *nch = nullptr;
  float4 *bmin = nullptr, *bmax = nullptr;
  unsigned long long* mask = nullptr;
  float4 *acm = nullptr, *anm = nullptr;  // aggregates: centroid, normal and mass
};

// Per point, at its current position: index in the input, node, path code (see
// compute_path_codes in host_tree.cpp).
struct Points {
  int *perm, *node;
  unsigned long long* code;
};

constexpr unsigned short kOutside = 0x8000;  // cell flag: the node's AABB check fails

// ---------------------------------------------------------------- kernels ---

__global__ void k_root(Nodes nd, int n, float4 lo, float4 hi) {
  nd.start[0] = 0;
  nd.cnt[0] = n;
  nd.bmin[0] = lo;
  nd.bmax[0] = hi;
}

__global__ void k_init_points(int n, Points p) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    p.perm[i] = (int)i;
    p.node[i] = 0;
    p.code[i] = 0ull;
  }
}

// Whether node v of the level is split (tree3d.h:245-246: more than leaf_size
// points, above the depth cap).
__device__ __forceinline__ bool is_split(const Nodes& nd, int v, int leaf_size, bool capped) {
  return !capped && nd.cnt[v] > leaf_size;
}

// Cell of every point in a node of the level that is split, into the node's mask
// of non-empty cells.
template <int DIM>
__global__ void k_cells(Nodes nd, int lb, int n, const float* __restrict__ pts, Points p,
                        unsigned short* cellv, int dsl, int leaf_size) {
  const int ds = 1 << dsl;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int v = p.node[i];
    if (v < lb || !is_split(nd, v, leaf_size, false)) continue;
    const float* s = pts + (long long)p.perm[i] * DIM;
    const float4 lo = nd.bmin[v], hi = nd.bmax[v];
    const float3 x = make_float3(s[0], s[1], DIM == 3 ? s[2] : 0.f);
    const int cx = sbh::quantize1(x.x, lo.x, hi.x, ds);
    const int cy = sbh::quantize1(x.y, lo.y, hi.y, ds);
    const int cz = DIM == 3 ? sbh::quantize1(x.z, lo.z, hi.z, ds) : 0;
    const int cell = (((cz << dsl) + cy) << dsl) + cx;
    // a path code is void where an ancestor's AABB check fails (include/aabb.h:28-32)
    const bool inside = v == 0 || sbh::aabb_contains<DIM>(lo, hi, x);
    cellv[i] = (unsigned short)cell | (inside ? 0 : kOutside);
    unsigned long long* w = nd.mask + (long long)v * nd.mw + (cell >> 6);
    const unsigned long long bit = 1ull << (cell & 63);
    if (!(__ldcg(w) & bit)) atomicOr(w, bit);  // once a cell is marked, only a read
  }
}

// Children per node of the level (nch_out gets a zero after the last for the
// scan's total); a capped node with several points needs the host build.
__global__ void k_count_children(Nodes nd, int lb, int le, int leaf_size, bool capped,
                                 unsigned* nch_out, int* info) {
  const int v = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (v == le) nch_out[v - lb] = 0u;
  if (v >= le) return;
  int k = 0;
  if (is_split(nd, v, leaf_size, capped))
    for (int w = 0; w < nd.mw; w++) k += __popcll(nd.mask[(long long)v * nd.mw + w]);
  if (capped && nd.cnt[v] > 1) info[1] = 1;
  nd.nch[v] = k;
  nch_out[v - lb] = (unsigned)k;
}

// First children from the scanned counts; info[0] = the level's children.
__global__ void k_first(Nodes nd, int lb, int le, const unsigned* __restrict__ offs, int* info) {
  const int v = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (v == le) info[0] = (int)offs[v - lb];
  if (v < le) nd.first[v] = nd.nch[v] ? le + (int)offs[v - lb] : 0;
}

// Index among v's children of the one in `cell`.
__device__ __forceinline__ int child_rank(const Nodes& nd, int v, int cell) {
  const unsigned long long* m = nd.mask + (long long)v * nd.mw;
  const int w = cell >> 6;
  int r = __popcll(__ldg(m + w) & ((1ull << (cell & 63)) - 1ull));
  for (int k = 0; k < w; k++) r += __popcll(__ldg(m + k));
  return r;
}

constexpr int kAssignPerThread = 8;
constexpr int kLocalChildren = 4096;  // children counted in shared memory (16 KB)

// Child of every point of the level's split nodes, and the point's place among
// the child's points in no particular order (which the leaves do not keep).
// LOCAL (levels of few children, where a million points meet on a few
// counters): a block counts its points in shared memory and takes the places of
// all of a child's points with one global addition.
template <bool LOCAL>
__global__ void __launch_bounds__(kThreads)
    k_assign(Nodes nd, int lb, int first_new, int children, int n, Points p,
             const unsigned short* __restrict__ cellv, int* child, int* place, int leaf_size) {
  extern __shared__ int s_cnt[];
  if (LOCAL) {
    for (int c = threadIdx.x; c < children; c += kThreads) s_cnt[c] = 0;
    __syncthreads();
  }
  const long long base = (long long)blockIdx.x * kThreads * kAssignPerThread + threadIdx.x;
  int u[kAssignPerThread], o[kAssignPerThread];
#pragma unroll
  for (int k = 0; k < kAssignPerThread; k++) {
    const long long i = base + k * kThreads;
    u[k] = -1;
    if (i >= n) continue;
    const int v = p.node[i];
    if (v < lb || !is_split(nd, v, leaf_size, false)) continue;
    u[k] = nd.first[v] + child_rank(nd, v, cellv[i] & ~kOutside);
    o[k] = LOCAL ? atomicAdd(s_cnt + (u[k] - first_new), 1) : atomicAdd(nd.cnt + u[k], 1);
  }
  if (LOCAL) {
    __syncthreads();
    for (int c = threadIdx.x; c < children; c += kThreads)
      if (s_cnt[c]) s_cnt[c] = atomicAdd(nd.cnt + first_new + c, s_cnt[c]);
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < kAssignPerThread; k++) {
    const long long i = base + k * kThreads;
    if (i >= n) continue;
    child[i] = u[k];
    if (u[k] >= 0) place[i] = LOCAL ? s_cnt[u[k] - first_new] + o[k] : o[k];
  }
}

// The k-th set bit of v's mask.
__device__ __forceinline__ int nth_cell(const Nodes& nd, int v, int k) {
  const unsigned long long* m = nd.mask + (long long)v * nd.mw;
  int w = 0;
  unsigned long long x = __ldg(m);
  for (int c = __popcll(x); k >= c; c = __popcll(x)) {
    k -= c;
    x = __ldg(m + ++w);
  }
  int b = 0;
#pragma unroll
  for (int h = 32; h > 0; h >>= 1) {
    const int c = __popcll((x >> b) & ((1ull << h) - 1ull));
    if (k >= c) {
      k -= c;
      b += h;
    }
  }
  return w * 64 + b;
}

// The node of its level that a thread of k_children works on, eight lanes a node: a
// level of 2^29 nodes has as many threads as 32 bits can number.
__host__ __device__ constexpr long long child_thread_node(unsigned block, unsigned thread) {
  return ((long long)block * kThreads + thread) / 8;
}
static_assert(child_thread_node(1u << 24, 8) == (1LL << 29) + 1, "thread numbers beyond 32 bits");

// Child nodes of the level's split nodes (tree3d.h:291-301): ranges, bounds
// min + i*inc (include/aabb.h).  Eight lanes per node, a child each at a time.
template <int DIM>
__global__ void k_children(Nodes nd, int lb, int le, int dsl) {
  const long long at = lb + child_thread_node(blockIdx.x, threadIdx.x);
  const int l = threadIdx.x & 7;
  const int nch = at < le ? nd.nch[at] : 0;
  if (nch == 0) return;  // the same for the node's eight lanes
  const int v = (int)at;
  const unsigned group = 0xffu << (threadIdx.x & 24);
  const int ds = 1 << dsl;
  const float4 lo = nd.bmin[v], hi = nd.bmax[v];
  const float fds = (float)ds;
  const float incx = sbh::rdiv(sbh::rsub(hi.x, lo.x), fds);
  const float incy = sbh::rdiv(sbh::rsub(hi.y, lo.y), fds);
  const float incz = DIM == 3 ? sbh::rdiv(sbh::rsub(hi.z, lo.z), fds) : 0.f;
  int off = nd.start[v];
  for (int k0 = 0; k0 < nch; k0 += 8) {
    const int k = k0 + l, u = nd.first[v] + k;
    const int cnt = k < nch ? nd.cnt[u] : 0;
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int y = __shfl_up_sync(group, incl, o, 8);
      if (l >= o) incl += y;
    }
    if (k < nch) {
      const int c = nth_cell(nd, v, k);
      const int x = c & (ds - 1), y = (c >> dsl) & (ds - 1), z = c >> (2 * dsl);
      float4 clo, chi;
      clo.x = sbh::radd(lo.x, sbh::rmul((float)x, incx));
      clo.y = sbh::radd(lo.y, sbh::rmul((float)y, incy));
      clo.z = DIM == 3 ? sbh::radd(lo.z, sbh::rmul((float)z, incz)) : 0.f;
      chi.x = sbh::radd(clo.x, incx);
      chi.y = sbh::radd(clo.y, incy);
      chi.z = DIM == 3 ? sbh::radd(clo.z, incz) : 0.f;
      clo.w = chi.w = 0.f;
      nd.start[u] = off + incl - cnt;
      nd.bmin[u] = clo;
      nd.bmax[u] = chi;
    }
    off += __shfl_sync(group, incl, 7, 8);
  }
}

// Points of the level's split nodes move to their child's range, their codes take
// the level's cell; the rest keep their place.
__global__ void k_scatter(Nodes nd, int n, Points p, const unsigned short* __restrict__ cellv,
                          const int* __restrict__ child, const int* __restrict__ place,
                          int code_shift, Points p2) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int u = child[i];
    unsigned long long code = p.code[i];
    long long pos = i;
    int node = p.node[i];
    if (u >= 0) {
      pos = nd.start[u] + place[i];
      node = u;
      const unsigned c = cellv[i];
      if (code_shift >= 0) code |= (unsigned long long)(c & ~(unsigned)kOutside) << code_shift;
      if (c & kOutside) code |= 1ull << 63;
    }
    p2.perm[pos] = p.perm[i];
    p2.node[pos] = node;
    p2.code[pos] = code;
  }
}

// Points in build order.
template <int DIM>
__global__ void k_points(int n, Points p, const float* __restrict__ pts,
                         const float* __restrict__ nrm, const float* __restrict__ mass,
                         float4* pt_pm, float4* pt_nrm, unsigned long long* pt_code) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long s = p.perm[i];
    const float px = pts[s * DIM], py = pts[s * DIM + 1], pz = DIM == 3 ? pts[s * DIM + 2] : 0.f;
    const float nx = nrm[s * DIM], ny = nrm[s * DIM + 1], nz = DIM == 3 ? nrm[s * DIM + 2] : 0.f;
    pt_pm[i] = make_float4(px, py, pz, mass[s]);
    pt_nrm[i] = make_float4(nx, ny, nz, 0.f);
    pt_code[i] = p.code[i];
  }
}

// Aggregates of one level (tree3d.h:255-265 for leaves, 310-327 for internal
// nodes): mass, mass-weighted centroid and normal, in point / cell order.
template <int DIM>
__global__ void k_aggregate(Nodes nd, int lb, int le, const float4* __restrict__ pt_pm,
                            const float4* __restrict__ pt_nrm) {
  const int v = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= le) return;
  float m = 0.f, p[3] = {0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f};
  auto add = [&](float mass, float4 x, float4 r) {
    m = sbh::radd(m, mass);
    const float xv[3] = {x.x, x.y, x.z}, rv[3] = {r.x, r.y, r.z};
#pragma unroll
    for (int k = 0; k < DIM; k++) {
      p[k] = sbh::radd(p[k], sbh::rmul(mass, xv[k]));
      q[k] = sbh::radd(q[k], sbh::rmul(mass, rv[k]));
    }
  };
  const int nch = nd.nch[v];
  if (nch == 0) {
    const int s = nd.start[v], e = s + nd.cnt[v];
    for (int i = s; i < e; i++) add(pt_pm[i].w, pt_pm[i], pt_nrm[i]);
  } else {
    const int c0 = nd.first[v];
#pragma unroll 4
    for (int c = c0; c < c0 + nch; c++) add(nd.anm[c].w, nd.acm[c], nd.anm[c]);
  }
  float ap[3] = {0.f, 0.f, 0.f}, an[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int k = 0; k < DIM; k++) {
    ap[k] = sbh::rdiv(p[k], m);
    an[k] = sbh::rdiv(q[k], m);
    // An empty node (the root of an empty tree) divides 0 by 0: x86's SSE
    // gives the "indefinite" NaN 0xffc00000, the GPU its own NaN; keep x86's.
    if (m == 0.f && p[k] == 0.f) ap[k] = __int_as_float(0xffc00000);
    if (m == 0.f && q[k] == 0.f) an[k] = __int_as_float(0xffc00000);
  }
  nd.acm[v] = make_float4(ap[0], ap[1], ap[2], 0.f);
  nd.anm[v] = make_float4(an[0], an[1], an[2], m);
}

// Device image of the nodes (as the upload in gpu_tree.cu writes it).
template <int DIM>
__global__ void k_node_image(Nodes nd, int nn, const float4* __restrict__ pt_pm,
                             const float4* __restrict__ pt_nrm, float4* cm, float4* agg,
                             int4* topo, float4* bmin, float4* bmax,
                             unsigned long long* mask_out) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nn) return;
  const float4 lo = nd.bmin[v], hi = nd.bmax[v];
  const float dx = sbh::rsub(hi.x, lo.x), dy = sbh::rsub(hi.y, lo.y),
              dz = DIM == 3 ? sbh::rsub(hi.z, lo.z) : 0.f;
  const float diam = sbh::rsqrt_ieee(sbh::dot_exact<DIM>(dx, dy, dz, dx, dy, dz));
  const bool leaf = nd.nch[v] == 0;
  const int s = nd.start[v], e = s + nd.cnt[v];
  if (leaf && e - s == 1) {
    const float4 p = pt_pm[s], r = pt_nrm[s];
    cm[v] = make_float4(p.x, p.y, p.z, diam);
    agg[v] = make_float4(p.w, r.x, r.y, r.z);
  } else {
    const float4 a = nd.acm[v], b = nd.anm[v];
    cm[v] = make_float4(a.x, a.y, a.z, leaf ? -1.0f : diam);
    agg[v] = make_float4(b.w, b.x, b.y, b.z);
  }
  topo[v] = make_int4(leaf ? 0 : nd.first[v], leaf ? 0 : nd.nch[v], s, e);
  bmin[v] = lo;
  bmax[v] = hi;
  for (int w = 0; w < nd.mw; w++) mask_out[(long long)v * nd.mw + w] = nd.mask[(long long)v * nd.mw + w];
}

// Carves a workspace: with a null base it only counts the bytes.
struct Carver {
  char* base;
  size_t off = 0;
  template <class T>
  T* take(size_t count) {
    T* p = reinterpret_cast<T*>(base + off);
    off += (count * sizeof(T) + 255) & ~size_t(255);
    return p;
  }
};

struct Workspace {
  Nodes nd;
  Points p[2];
  float *pts, *nrm, *mass;
  unsigned short* cellv;
  int *child, *place, *info;
  unsigned *offs, *sums;
  size_t zero_begin, zero_end, bytes;  // node masks and counts start at zero
};

Workspace carve(char* base, int dim, size_t n, size_t cap, int mw) {
  Workspace w;
  Carver c{base};
  w.pts = c.take<float>(n * dim);
  w.nrm = c.take<float>(n * dim);
  w.mass = c.take<float>(n);
  for (Points& p : w.p) {
    p.perm = c.take<int>(n);
    p.node = c.take<int>(n);
    p.code = c.take<unsigned long long>(n);
  }
  w.cellv = c.take<unsigned short>(n);
  w.child = c.take<int>(n);
  w.place = c.take<int>(n);
  w.offs = c.take<unsigned>(cap + 1);
  w.sums = c.take<unsigned>((size_t)sbh::scan_tiles_for((long long)cap + 1));
  Nodes& nd = w.nd;
  nd.mw = mw;
  nd.start = c.take<int>(cap);
  nd.first = c.take<int>(cap);
  nd.nch = c.take<int>(cap);
  nd.bmin = c.take<float4>(cap);
  nd.bmax = c.take<float4>(cap);
  nd.acm = c.take<float4>(cap);
  nd.anm = c.take<float4>(cap);
  w.zero_begin = c.off;
  nd.mask = c.take<unsigned long long>(cap * mw);
  nd.cnt = c.take<int>(cap);
  w.info = c.take<int>(2);  // children of the level; whether the build needs the host
  w.zero_end = w.bytes = c.off;
  return w;
}

// Streams of past builds, kept for the next (creating one takes 0.5 ms): at most
// four per device, each used by one build at a time.
struct StreamCache {
  std::mutex mu;
  std::vector<cudaStream_t> idle[64];
  cudaStream_t take(int device) {
    {
      std::lock_guard<std::mutex> lock(mu);
      if (!idle[device].empty()) {
        cudaStream_t s = idle[device].back();
        idle[device].pop_back();
        return s;
      }
    }
    cudaStream_t s = nullptr;
    return cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess ? s : nullptr;
  }
  void give(int device, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu);
    if (idle[device].size() < 4)
      idle[device].push_back(s);
    else
      cudaStreamDestroy(s);
  }
};
StreamCache g_streams;

// Builds on the device with room for `cap` nodes; SBH_ERR_UNSUPPORTED (nothing
// kept) when the build needs the host (see the file comment) or the tree does not
// fit beside the workspace, kMoreNodes when cap was too small.
constexpr int kMoreNodes = -1;

template <int DIM>
int build_with(Workspace& w, cudaStream_t s, size_t cap, int dsl, int leaf_size, int max_depth,
               const float* points, const float* normals, const float* masses, int n,
               const float* lo, const float* hi, float alpha, int device, int sm_count,
               sbh_gpu_tree** out) {
  cudaError_t e = cudaSuccess;
  const char* what = "tree build";
  auto ck = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
    return e == cudaSuccess;
  };
  const int bits = DIM * dsl, bf = 1 << bits, mw = w.nd.mw, levels = 63 / bits;
  if (n > 0) {
    ck(cudaMemcpyAsync(w.pts, points, (size_t)n * DIM * sizeof(float), cudaMemcpyHostToDevice, s));
    ck(cudaMemcpyAsync(w.nrm, normals, (size_t)n * DIM * sizeof(float), cudaMemcpyHostToDevice, s));
    ck(cudaMemcpyAsync(w.mass, masses, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, s));
  }
  ck(cudaMemsetAsync(reinterpret_cast<char*>(w.nd.mask), 0, w.zero_end - w.zero_begin, s));
  std::vector<long long> level_begin = {0};
  int cur = 0, info[2] = {0, 0};
  long long nn = 1;
  const float4 flo = make_float4(lo[0], lo[1], DIM == 3 ? lo[2] : 0.f, 0.f);
  const float4 fhi = make_float4(hi[0], hi[1], DIM == 3 ? hi[2] : 0.f, 0.f);
  k_root<<<1, 1, 0, s>>>(w.nd, n, flo, fhi);
  k_init_points<<<blocks_for(n), kThreads, 0, s>>>(n, w.p[0]);
  const int pgrid = std::min(blocks_for(n), sm_count * 8);
  for (int level = 0; e == cudaSuccess; level++) {
    const long long lb = level_begin.back(), le = nn, m = le - lb;
    const bool capped = level >= max_depth;
    if (!capped)
      k_cells<DIM><<<pgrid, kThreads, 0, s>>>(w.nd, (int)lb, n, w.pts, w.p[cur], w.cellv, dsl,
                                              leaf_size);
    k_count_children<<<blocks_for(m + 1), kThreads, 0, s>>>(w.nd, (int)lb, (int)le, leaf_size,
                                                            capped, w.offs, w.info);
    sbh::launch_scan(w.offs, nullptr, m + 1, m + 1, w.sums, s);
    k_first<<<blocks_for(m + 1), kThreads, 0, s>>>(w.nd, (int)lb, (int)le, w.offs, w.info);
    ck(cudaMemcpyAsync(info, w.info, sizeof(info), cudaMemcpyDeviceToHost, s));
    if (!ck(cudaStreamSynchronize(s))) break;
    if (info[1]) return SBH_ERR_UNSUPPORTED;
    level_begin.push_back(le);
    const long long children = info[0];
    if (children == 0) break;
    if (nn + children > (long long)INT32_MAX) return SBH_ERR_UNSUPPORTED;
    if (nn + children > (long long)cap) return kMoreNodes;
    const int ablocks = (n + kThreads * kAssignPerThread - 1) / (kThreads * kAssignPerThread);
    if (children <= kLocalChildren)
      k_assign<true><<<ablocks, kThreads, children * sizeof(int), s>>>(
          w.nd, (int)lb, (int)le, (int)children, n, w.p[cur], w.cellv, w.child, w.place, leaf_size);
    else
      k_assign<false><<<ablocks, kThreads, 0, s>>>(w.nd, (int)lb, (int)le, (int)children, n,
                                                   w.p[cur], w.cellv, w.child, w.place, leaf_size);
    k_children<DIM><<<blocks_for(m * 8), kThreads, 0, s>>>(w.nd, (int)lb, (int)le, dsl);
    k_scatter<<<pgrid, kThreads, 0, s>>>(w.nd, n, w.p[cur], w.cellv, w.child, w.place,
                                         level < levels ? bits * level : -1, w.p[cur ^ 1]);
    cur ^= 1;
    nn += children;
  }
  if (e != cudaSuccess) return sbh::cuda_fail(e, what);

  // The tree's device image.
  const sbh::TreeLayout L = sbh::tree_layout(n, nn, mw);
  sbh_gpu_tree* g = new (std::nothrow) sbh_gpu_tree();
  if (!g) return sbh::fail(SBH_ERR_OUT_OF_MEMORY, "host allocation failed");
  g->device = device;
  g->sm_count = sm_count;
  g->bytes = L.bytes;
  if (!ck(sbh::alloc_tree_memory(device, L.bytes, s, &g->mem))) what = "tree memory";
  if (e == cudaErrorMemoryAllocation) {  // it may fit without the workspace
    cudaGetLastError();
    delete g;
    return SBH_ERR_UNSUPPORTED;
  }
  if (e == cudaSuccess) {
    sbh::bind_tree(g, L);
    char* base = static_cast<char*>(g->mem);
    float4* pt_pm = reinterpret_cast<float4*>(base + L.pm);
    float4* pt_nrm = reinterpret_cast<float4*>(base + L.nrm);
    ck(cudaMemsetAsync(base + L.status, 0, sizeof(int), s));
    k_points<DIM><<<blocks_for(n), kThreads, 0, s>>>(
        n, w.p[cur], w.pts, w.nrm, w.mass, pt_pm, pt_nrm,
        reinterpret_cast<unsigned long long*>(base + L.code));
    for (int l = (int)level_begin.size() - 2; l >= 0; l--) {
      const long long lb = level_begin[l], le = level_begin[l + 1];
      k_aggregate<DIM><<<blocks_for(le - lb), kThreads, 0, s>>>(w.nd, (int)lb, (int)le, pt_pm,
                                                                pt_nrm);
    }
    k_node_image<DIM><<<blocks_for(nn), kThreads, 0, s>>>(
        w.nd, (int)nn, pt_pm, pt_nrm, reinterpret_cast<float4*>(base + L.cm),
        reinterpret_cast<float4*>(base + L.agg), reinterpret_cast<int4*>(base + L.topo),
        reinterpret_cast<float4*>(base + L.bmin), reinterpret_cast<float4*>(base + L.bmax),
        reinterpret_cast<unsigned long long*>(base + L.mask));
    ck(cudaGetLastError());
    int root_nch = 0;
    ck(cudaMemcpyAsync(&root_nch, w.nd.nch, sizeof(int), cudaMemcpyDeviceToHost, s));
    ck(cudaStreamSynchronize(s));
    if (e == cudaSuccess) e = cudaEventCreate(&g->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&g->ev1);
    DevTree& t = g->dev;
    t.code_bits = bits;
    t.code_levels = levels;
    t.n = n;
    t.nn = nn;
    t.dim = DIM;
    t.dsl = dsl;
    t.ds = 1 << dsl;
    t.bf = bf;
    t.mw = mw;
    t.depth = (int)level_begin.size() - 2;
    t.root_children = root_nch;
    t.alpha = alpha;
    for (int k = 0; k < DIM; k++) {
      g->box_lo[k] = lo[k];
      g->box_hi[k] = hi[k];
    }
    sbh_tree_info& info = g->info;
    info = sbh_tree_info();
    info.dim = DIM;
    info.dim_split_log = dsl;
    info.leaf_size = leaf_size;
    info.max_depth = max_depth;
    info.num_points = n;
    info.num_nodes = nn;
    info.depth = t.depth;
    info.root_children = t.root_children;
    info.alpha = alpha;
    info.device_bytes = L.bytes;
  }
  if (e != cudaSuccess) {
    if (g->ev0) cudaEventDestroy(g->ev0);
    if (g->ev1) cudaEventDestroy(g->ev1);
    cudaStreamSynchronize(s);
    sbh::free_tree_memory(device, g->mem);
    delete g;
    return sbh::cuda_fail(e, what);
  }
  *out = g;
  return SBH_OK;
}

// Builds with a workspace of the library's pool, with room for two nodes per
// point at first (a leaf per point and the nodes above them; 1.3 to 1.6 on the
// generators' clouds), four times as many when chains of single children need it.
template <int DIM>
int build_on_device(int dsl, int leaf_size, int max_depth, const float* points,
                    const float* normals, const float* masses, int n, const float* lo,
                    const float* hi, float alpha, int device, int sm_count, sbh_gpu_tree** out) {
  const int bf = 1 << (DIM * dsl), mw = bf >= 64 ? bf / 64 : 1;
  cudaMemPool_t pool = nullptr;
  int st = sbh::scratch_pool(device, &pool);
  if (st != SBH_OK) return st;
  cudaStream_t s = g_streams.take(device);
  if (!s) return sbh::cuda_fail(cudaGetLastError(), "cudaStreamCreate");
  size_t cap = std::min<size_t>(2 * (size_t)n + 4096, (size_t)INT32_MAX);
  do {
    const size_t bytes = carve(nullptr, DIM, n, cap, mw).bytes;
    void* mem = nullptr;
    cudaError_t e = cudaMallocFromPoolAsync(&mem, bytes, pool, s);
    if (e == cudaErrorMemoryAllocation) {  // the host build needs the tree's memory alone
      cudaGetLastError();
      st = SBH_ERR_UNSUPPORTED;
      break;
    }
    if (e != cudaSuccess) {
      st = sbh::cuda_fail(e, "cudaMallocFromPoolAsync(tree build)");
      break;
    }
    Workspace w = carve(static_cast<char*>(mem), DIM, n, cap, mw);
    st = build_with<DIM>(w, s, cap, dsl, leaf_size, max_depth, points, normals, masses, n, lo, hi,
                         alpha, device, sm_count, out);
    cudaFreeAsync(mem, s);
    // nothing of a failed build may still read the caller's arrays
    cudaStreamSynchronize(s);
    sbh::trim_pool(pool);
    cap = std::min<size_t>(cap * 4, (size_t)INT32_MAX);
  } while (st == kMoreNodes);
  g_streams.give(device, s);
  return st;
}

}  // namespace

SBH_API int sbh_gpu_tree_build(int dim, int dim_split_log, int leaf_size, int max_depth,
                               const float* points, const float* normals, const float* masses,
                               int64_t n, const float* min_corner, const float* max_corner,
                               float alpha, int device, sbh_gpu_tree** out, int32_t* on_device) {
  if (!out) return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "out must be non-null");
  *out = nullptr;
  if (on_device) *on_device = 0;
  if (dim != 2 && dim != 3) return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "dim must be 2 or 3");
  if (dim_split_log < 1 || dim_split_log > 3)
    return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "dim_split_log must be 1, 2 or 3");
  if (leaf_size < 1) return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "leaf_size must be >= 1");
  if (max_depth < 0 || max_depth > 1000)
    return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "max_depth must be in [0, 1000]");
  if (n < 0 || n > (int64_t)INT32_MAX)
    return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "point count must be in [0, 2^31)");
  if (n > 0 && (!points || !normals || !masses))
    return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "points, normals and masses must be non-null");
  if (!min_corner || !max_corner)
    return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "min_corner and max_corner must be non-null");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
    cudaGetLastError();
    return sbh::fail(SBH_ERR_NO_DEVICE, "no such CUDA device");
  }
  int sm_count = 0;
  int st = sbh::check_device(device, &sm_count);
  if (st != SBH_OK) return st;
  st = SBH_ERR_UNSUPPORTED;
  if (leaf_size == 1) {
    sbh::DeviceGuard guard(device);
    st = dim == 3 ? build_on_device<3>(dim_split_log, leaf_size, max_depth, points, normals, masses,
                                       (int)n, min_corner, max_corner, alpha, device, sm_count, out)
                  : build_on_device<2>(dim_split_log, leaf_size, max_depth, points, normals, masses,
                                       (int)n, min_corner, max_corner, alpha, device, sm_count, out);
    if (st == SBH_OK) {
      if (on_device) *on_device = 1;
      return sbh::ok();
    }
    if (st != SBH_ERR_UNSUPPORTED) return st;
  }
  // The host build reproduces std::partition's order inside multi-point leaves.
  sbh_host_tree* h = nullptr;
  st = sbh_host_tree_create(dim, dim_split_log, leaf_size, max_depth, points, normals, masses, n,
                            min_corner, max_corner, alpha, &h);
  if (st != SBH_OK) return st;
  st = sbh_gpu_tree_create(h, device, out);
  sbh_host_tree_destroy(h);
  return st;
}

SBH_API int sbh_gpu_tree_export(const sbh_gpu_tree* tree, float* pt_pm, float* pt_nrm, float* nd_cm,
                                float* nd_agg, int32_t* nd_topo, float* nd_bmin, float* nd_bmax,
                                uint64_t* nd_mask, uint64_t* pt_code) {
  if (!tree) return sbh::fail(SBH_ERR_INVALID_ARGUMENT, "null tree");
  sbh::DeviceGuard guard(tree->device);
  const DevTree& t = tree->dev;
  const size_t n = (size_t)t.n, nn = (size_t)t.nn;
  struct Out {
    void* dst;
    const void* src;
    size_t bytes;
  } outs[] = {{pt_pm, t.pt_pm, n * sizeof(float4)},       {pt_nrm, t.pt_nrm, n * sizeof(float4)},
              {nd_cm, t.nd_cm, nn * sizeof(float4)},      {nd_agg, t.nd_agg, nn * sizeof(float4)},
              {nd_topo, t.nd_topo, nn * sizeof(int4)},    {nd_bmin, t.nd_bmin, nn * sizeof(float4)},
              {nd_bmax, t.nd_bmax, nn * sizeof(float4)},
              {nd_mask, t.nd_mask, nn * t.mw * sizeof(uint64_t)},
              {pt_code, t.pt_code, n * sizeof(uint64_t)}};
  for (const Out& o : outs) {
    if (!o.dst || o.bytes == 0) continue;
    cudaError_t e = cudaMemcpy(o.dst, o.src, o.bytes, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return sbh::cuda_fail(e, "copy tree out");
  }
  return sbh::ok();
}
