// Training's starting Gaussians from a point cloud (src/loadDataset.ts:93-149):
// for each point the mean squared distance to its 3 nearest other points, then
// one Gaussian per point sized by it.
//
// The reference finds the neighbours by brute force (src/shaders/nearestNeighbors.wgsl:13-44),
// N² distances. Here the points are sorted along a Morton (Z-order) curve of 21
// bits per axis, and each 32 consecutive ones (a leaf) get their bounding box, each
// 32 leaves theirs, and so on up to at most 32 boxes. A warp then answers the 32
// queries of one leaf together:
//   1. every lane offers its point the leaf's other points and the two leaves beside
//      it on the curve: a first bound on each third-smallest distance;
//   2. the warp descends the tree, of a node's children (a lane each) the nearest to
//      any of its points first, leaving out those no point is near enough to;
//   3. a leaf it reaches is read once and offered to all 32 points (or, when few
//      of them are near enough, to those).
// One thread per point descending an octree by binary searches of the curve (27
// cells a point) took 1,519 us for a clustered cloud of 180,000 points where this
// takes 195: its threads waited for the warp's longest search and for one dependent
// load after another; here 32 points share every box and every point that is read.
// (The whole call: 1,448 -> 315 us.) What bounds
// it: instructions at 1.1M points (16 a distance, 512 a leaf, about 28 leaves a
// warp); at 180,000, whose warps all run at once, the longest walks.
//
// The search is exact: it finds the same three smallest squared distances, each
// computed as the reference computes it (d = q - p, then d.x² + d.y² + d.z²
// rounded in that order; this file is compiled without contraction), so every
// result is the brute force's bit for bit. A box's distance is computed by the same
// rounded operations from its nearest faces; each of them is monotone, so no point
// in the box has a smaller computed distance, and a box at or past the third
// distance so far cannot hold a smaller one. The visiting order does not matter:
// the three smallest values of a set do not depend on the order they are met in.
//
// The curve spans the points' bounds trimmed to the mean ± 3 standard deviations
// per axis (so that a few far outliers do not coarsen it); points outside are
// clamped onto its border. Points with a non-finite coordinate are no point's
// neighbours (their distances are infinite or NaN, never below the starting 3.4e38),
// so the boxes leave them out, and they get the reference's result for a point
// without neighbours.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "dg_common.cuh"
#include "dg_scan.cuh"

namespace dg {
namespace {

constexpr uint32_t KNN_THREADS = 256;
constexpr uint32_t BITS = 21;  // per axis: 63-bit Morton codes
constexpr uint32_t LEVELS = 6;  // of boxes: 32^6 points
constexpr uint32_t QUERY_WARPS = 4;
constexpr int FEW = 16;  // queries that a leaf is offered to one by one (10 and 22 measured the same)
constexpr float FAR = 3.4e38f;        // nearestNeighbors.wgsl:19, the starting "distance"

struct Octree {
  float lo[3];
  float scale;  // finest cells per unit length
};

// The finite points' bounds and moments.
struct Moments {
  float lo[3], hi[3];
  double sum[3], sum2[3];  // in 64 bits: squares of float32 coordinates may exceed float32
  uint32_t finite;         // points with three finite coordinates
};

__device__ __forceinline__ bool finite3(float4 p) { return isfinite(p.x) && isfinite(p.y) && isfinite(p.z); }

__device__ __forceinline__ Moments no_moments() {
  Moments m;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    m.lo[k] = INFINITY;
    m.hi[k] = -INFINITY;
    m.sum[k] = m.sum2[k] = 0.0;
  }
  m.finite = 0;
  return m;
}

__device__ __forceinline__ void add_moments(Moments& m, const Moments& o) {
  m.finite += o.finite;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    m.lo[k] = fminf(m.lo[k], o.lo[k]);
    m.hi[k] = fmaxf(m.hi[k], o.hi[k]);
    m.sum[k] += o.sum[k];
    m.sum2[k] += o.sum2[k];
  }
}

// Sums m over `lanes` lanes of the warp, lane ^ 1 last.
__device__ __forceinline__ void reduce_lanes(Moments& m, int lanes) {
  for (int off = lanes / 2; off > 0; off >>= 1) {
    Moments o;
    o.finite = __shfl_xor_sync(0xffffffffu, m.finite, off);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      o.lo[k] = __shfl_xor_sync(0xffffffffu, m.lo[k], off);
      o.hi[k] = __shfl_xor_sync(0xffffffffu, m.hi[k], off);
      o.sum[k] = __shfl_xor_sync(0xffffffffu, m.sum[k], off);
      o.sum2[k] = __shfl_xor_sync(0xffffffffu, m.sum2[k], off);
    }
    add_moments(m, o);
  }
}

// Sums m over the CTA; the first warp's first 8 lanes get the whole.
__device__ __forceinline__ void reduce_moments(Moments& m, Moments* s_warp) {
  constexpr uint32_t WARPS = KNN_THREADS / 32;
  const uint32_t lane = threadIdx.x & 31u;
  reduce_lanes(m, 32);
  if (lane == 0) s_warp[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  m = s_warp[lane % WARPS];
  reduce_lanes(m, WARPS);
}

// Each CTA's share of the moments (4,900 warps adding to one global record took
// 70 us at 180,000 points). Bound by the FP64 sums: with a thread's points summed in
// float32 12.3 us instead of 15.4 at 180,000 points and 16 instead of 37 at 1.1M, but
// coordinates past 2^64 then gave no trimmed span and took 14 times as long to search.
__global__ void __launch_bounds__(KNN_THREADS) bounds_kernel(const float4* __restrict__ points, uint32_t n,
                                                             Moments* __restrict__ shares) {
  __shared__ Moments s_warp[KNN_THREADS / 32];
  Moments m = no_moments();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 p = points[i];
    if (!finite3(p)) continue;
    const float c[3] = {p.x, p.y, p.z};
    m.finite++;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      m.lo[k] = fminf(m.lo[k], c[k]);
      m.hi[k] = fmaxf(m.hi[k], c[k]);
      m.sum[k] += (double)c[k];
      m.sum2[k] += (double)c[k] * (double)c[k];
    }
  }
  reduce_moments(m, s_warp);
  if (threadIdx.x == 0) shares[blockIdx.x] = m;
}

// The octree for the shares' bounds and moments. One CTA.
__global__ void __launch_bounds__(KNN_THREADS) octree_kernel(const Moments* __restrict__ shares, uint32_t count,
                                                             Octree* __restrict__ out) {
  __shared__ Moments s_warp[KNN_THREADS / 32];
  Moments m = no_moments();
  for (uint32_t k = threadIdx.x; k < count; k += KNN_THREADS) add_moments(m, shares[k]);
  reduce_moments(m, s_warp);
  if (threadIdx.x >= 32) return;
  // Lane k: axis k.
  const uint32_t k = threadIdx.x % 3;
  const double finite = m.finite ? (double)m.finite : 1.0;
  auto axis = [&](const auto (&v)[3]) { return k == 0 ? v[0] : k == 1 ? v[1] : v[2]; };
  double lo = axis(m.lo), hi = axis(m.hi);
  if (!(lo <= hi)) lo = hi = 0.0;  // no finite points
  const double mean = axis(m.sum) / finite;
  const double reach = 3.0 * sqrt(fmax(0.0, axis(m.sum2) / finite - mean * mean));
  lo = fmax(lo, mean - reach);
  hi = fmin(hi, mean + reach);
  if (!(lo <= hi)) lo = hi = mean;
  if (threadIdx.x < 3) out->lo[k] = (float)lo;
  double extent = hi - lo;
  for (int other = 1; other < 3; other++) extent = fmax(extent, __shfl_sync(0xffffffffu, hi - lo, (k + other) % 3));
  if (!(extent > 0.0) || !isfinite(extent)) extent = 1.0;
  if (threadIdx.x == 0) out->scale = (float)((double)(1u << BITS) / extent);
}

// Finest-level cell coordinate of a position, clamped into the octree (NaN
// coordinates land at 0).
__device__ __forceinline__ void quantize(const Octree& o, float x, float y, float z, uint32_t q[3]) {
  const float p[3] = {x, y, z};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float t = floorf((p[k] - o.lo[k]) * o.scale);
    q[k] = (uint32_t)fminf(fmaxf(t, 0.0f), (float)((1u << BITS) - 1u));
  }
}

// The bits of v (up to 21) spread to every third bit.
__device__ __forceinline__ uint64_t spread3(uint32_t v) {
  uint64_t x = v & 0x1fffffu;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}

__device__ __forceinline__ uint64_t morton(uint32_t x, uint32_t y, uint32_t z) {
  return spread3(x) | spread3(y) << 1 | spread3(z) << 2;
}

// Each point's Morton code (the sort key, as (low, high) words) and index.
__global__ void morton_kernel(const float4* __restrict__ points, uint32_t n, const Octree* __restrict__ octree,
                              uint2* __restrict__ keys, uint32_t* __restrict__ values) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Octree o = *octree;
  const float4 p = points[i];
  uint32_t q[3];
  quantize(o, p.x, p.y, p.z, q);
  const uint64_t code = morton(q[0], q[1], q[2]);
  keys[i] = make_uint2((uint32_t)code, (uint32_t)(code >> 32));
  values[i] = i;
}

// A box of finite points (lo above hi when it holds none).
struct Box {
  float4 lo, hi;
};

// The union of the warp's 32 boxes, on every lane.
__device__ __forceinline__ Box warp_box(Box b) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    b.lo.x = fminf(b.lo.x, __shfl_xor_sync(0xffffffffu, b.lo.x, off));
    b.lo.y = fminf(b.lo.y, __shfl_xor_sync(0xffffffffu, b.lo.y, off));
    b.lo.z = fminf(b.lo.z, __shfl_xor_sync(0xffffffffu, b.lo.z, off));
    b.hi.x = fmaxf(b.hi.x, __shfl_xor_sync(0xffffffffu, b.hi.x, off));
    b.hi.y = fmaxf(b.hi.y, __shfl_xor_sync(0xffffffffu, b.hi.y, off));
    b.hi.z = fmaxf(b.hi.z, __shfl_xor_sync(0xffffffffu, b.hi.z, off));
  }
  return b;
}

__device__ __forceinline__ Box no_box() {
  return Box{make_float4(INFINITY, INFINITY, INFINITY, 0.0f), make_float4(-INFINITY, -INFINITY, -INFINITY, 0.0f)};
}

// The points in curve order, each carrying its original index in w, and the box of
// each 32.
__global__ void __launch_bounds__(KNN_THREADS) gather_points_kernel(const float4* __restrict__ points, uint32_t n,
                                                                    const uint32_t* __restrict__ order,
                                                                    float4* __restrict__ sorted,
                                                                    Box* __restrict__ leaves) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  Box b = no_box();
  if (s < n) {
    const uint32_t i = order[s];
    const float4 p = points[i];
    sorted[s] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
    if (finite3(p)) b = Box{p, p};
  }
  b = warp_box(b);
  if ((s & 31u) == 0 && s < n) leaves[s >> 5] = b;
}

// The boxes of each 32 of `count` boxes.
__global__ void __launch_bounds__(KNN_THREADS) parents_kernel(const Box* __restrict__ boxes, uint32_t count,
                                                              Box* __restrict__ parents) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  Box b = no_box();
  if (i < count) b = boxes[i];
  b = warp_box(b);
  if ((i & 31u) == 0 && i < count) parents[i >> 5] = b;
}

struct Tree {
  const Box* boxes[LEVELS];  // level 0: the leaves
  uint32_t count[LEVELS];
  uint32_t top;  // the first level of at most 32 boxes
};

struct Best {
  float x = FAR, y = FAR, z = FAR;  // the three smallest squared distances, smallest first

  // nearestNeighbors.wgsl:26-41, without branches: a distance that is not below the
  // third (or is NaN) is taken as FAR, which changes nothing.
  __device__ __forceinline__ void offer(float d2) {
    const float d = d2 < z ? d2 : FAR;
    const float a = fmaxf(x, d);
    x = fminf(x, d);
    const float b = fmaxf(y, a);
    y = fminf(y, a);
    z = fminf(z, b);
  }
};

__device__ __forceinline__ float distance2(float4 q, float px, float py, float pz) {
  const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
  return dx * dx + dy * dy + dz * dz;
}

// No point of box b has a smaller distance2 from any point of [lo, hi] than this.
__device__ __forceinline__ float gap2(const Box& b, float4 lo, float4 hi) {
  const float dx = fmaxf(fmaxf(b.lo.x - hi.x, lo.x - b.hi.x), 0.0f);
  const float dy = fmaxf(fmaxf(b.lo.y - hi.y, lo.y - b.hi.y), 0.0f);
  const float dz = fmaxf(fmaxf(b.lo.z - hi.z, lo.z - b.hi.z), 0.0f);
  return dx * dx + dy * dy + dz * dz;
}

// A warp per leaf. (Two or four lanes per query, so two or four warps per leaf, were
// no faster from 10,000 points on, and half as fast at 1.1M.)
__global__ void __launch_bounds__(QUERY_WARPS * 32) knn_query_kernel(const float4* __restrict__ sorted, uint32_t n,
                                                                     const Tree tree,
                                                                     float* __restrict__ distance2_out) {
  __shared__ float4 s_points[QUERY_WARPS][32];
  __shared__ Box s_boxes[QUERY_WARPS][32];
  __shared__ uint32_t s_key[QUERY_WARPS][LEVELS][32];
  __shared__ uint32_t s_base[QUERY_WARPS][LEVELS];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t leaf = blockIdx.x * QUERY_WARPS + warp;
  if (leaf >= tree.count[0]) return;
  const uint32_t s = leaf * 32 + lane;
  const float4 me = s < n ? sorted[s] : make_float4(NAN, NAN, NAN, 0.0f);
  const bool query = finite3(me);
  const Box own = tree.boxes[0][leaf];
  float4* points = s_points[warp];
  Box* boxes = s_boxes[warp];
  uint32_t(*keys)[32] = s_key[warp];
  uint32_t* base = s_base[warp];
  Best best;
  // The largest third distance of the queries (of non-negative floats the bits compare alike).
  auto worst = [&]() { return __uint_as_float(__reduce_max_sync(0xffffffffu, query ? __float_as_uint(best.z) : 0u)); };
  // Offers the 32 points of leaf f to every query (its own point is not its neighbour;
  // past the end NaN).
  auto offer_leaf = [&](uint32_t f, bool mine) {
    __syncwarp();
    points[lane] = f * 32 + lane < n ? sorted[f * 32 + lane] : make_float4(NAN, NAN, NAN, 0.0f);
    __syncwarp();
#pragma unroll 8
    for (uint32_t j = 0; j < 32; j++) {
      const float d = distance2(points[j], me.x, me.y, me.z);
      best.offer(mine && j == lane ? FAR : d);
    }
  };
  offer_leaf(leaf, true);
  if (leaf > 0) offer_leaf(leaf - 1, false);
  if (leaf + 1 < tree.count[0]) offer_leaf(leaf + 1, false);
  float bound = worst();
  // A lane's child of the node at hand: the distance of the query nearest to it, with
  // the lane in the low bits (rounded down: still a lower bound), or all ones when it
  // is out of reach of all. The queries' own box sorts out most children at once; the
  // rest are held against the queries one after another, independently. (Scattered
  // outliers have a box that reaches everywhere, while they need about 30 leaves like
  // the others.)
  auto expand = [&](uint32_t level, uint32_t first) {
    Box b = no_box();
    if (first + lane < tree.count[level]) b = tree.boxes[level][first + lane];
    __syncwarp();
    boxes[lane] = b;
    uint32_t left = __ballot_sync(0xffffffffu, gap2(b, own.lo, own.hi) < bound);
    __syncwarp();
    uint32_t key = ~0u;
    while (left) {  // four at a time
      uint32_t child[4], nearest[4];
#pragma unroll
      for (uint32_t u = 0; u < 4; u++) {
        child[u] = left ? __ffs(left) - 1 : child[0];
        left &= left - 1;
      }
#pragma unroll
      for (uint32_t u = 0; u < 4; u++) {
        const float g = gap2(boxes[child[u]], me, me);
        nearest[u] = __reduce_min_sync(0xffffffffu, query && g < best.z ? __float_as_uint(g) : ~0u);
      }
#pragma unroll
      for (uint32_t u = 0; u < 4; u++)
        if (lane == child[u] && nearest[u] != ~0u) key = (nearest[u] & ~31u) | lane;
    }
    keys[level][lane] = key;
    if (lane == 0) base[level] = first;
    __syncwarp();
  };
  uint32_t level = tree.top;
  expand(level, 0);
  while (true) {
    const uint32_t next = __reduce_min_sync(0xffffffffu, keys[level][lane]);
    if (next == ~0u || __uint_as_float(next & ~31u) >= bound) {
      if (level == tree.top) break;
      level++;
      continue;
    }
    const uint32_t child = next & 31u, node = base[level] + child;
    __syncwarp();
    if (lane == child) keys[level][lane] = ~0u;
    __syncwarp();
    if (level > 0) {
      expand(--level, node * 32);
      continue;
    }
    if (node + 1 >= leaf && node <= leaf + 1) continue;  // offered above
    uint32_t near = __ballot_sync(0xffffffffu, query && gap2(tree.boxes[0][node], me, me) < best.z);
    if (near == 0) continue;
    if (__popc(near) > FEW) {
      offer_leaf(node, false);
    } else {
      // For few queries, a lane per point of the leaf: each query's points below its
      // third distance (mostly none) are offered to its lane.
      const uint32_t at = node * 32 + lane;
      const float4 p = at < n ? sorted[at] : make_float4(NAN, NAN, NAN, 0.0f);
      for (; near; near &= near - 1) {
        const int q = __ffs(near) - 1;
        const float d = distance2(p, __shfl_sync(0xffffffffu, me.x, q), __shfl_sync(0xffffffffu, me.y, q),
                                  __shfl_sync(0xffffffffu, me.z, q));
        const float third = __shfl_sync(0xffffffffu, best.z, q);
        for (uint32_t hits = __ballot_sync(0xffffffffu, d < third); hits; hits &= hits - 1) {
          const float found = __shfl_sync(0xffffffffu, d, __ffs(hits) - 1);
          if ((int)lane == q) best.offer(found);
        }
      }
    }
    bound = worst();
  }
  // nearestNeighbors.wgsl:43; a point that is not finite has no neighbours.
  if (s < n)
    distance2_out[__float_as_uint(me.w)] = query ? (best.x + best.y + best.z) / 3.0f : (FAR + FAR + FAR) / 3.0f;
}

__global__ void pad_points_kernel(const float* __restrict__ positions, uint32_t n, float4* __restrict__ points) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  points[i] = make_float4(positions[3 * i], positions[3 * i + 1], positions[3 * i + 2], 0.0f);
}

// src/loadDataset.ts:99-121 for point i: the host arithmetic is float64 there, so
// it is float64 here, rounded to float32 on the store as a Float32Array store rounds.
__global__ void initial_gaussians_kernel(const float4* __restrict__ points, const uint8_t* __restrict__ colors,
                                         const float* __restrict__ distance2, uint32_t n, float opacity_logit,
                                         float* __restrict__ params) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 p = points[i];
  const double log_scale = 0.5 * log(fmax((double)distance2[i], 1e-7));
  float out[16];
  const float pos[3] = {p.x, p.y, p.z};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    out[k] = pos[k];
    out[4 + k] = (float)log_scale;
    out[12 + k] = (float)(((double)colors[3 * i + k] / 255.0 - 0.5) / 0.28209479177387814);
  }
  out[3] = opacity_logit;
  out[7] = 0.0f;
  out[8] = 1.0f;  // the quaternion (1, 0, 0, 0)
  out[9] = out[10] = out[11] = 0.0f;
  out[15] = 0.0f;
  float4* dst = reinterpret_cast<float4*>(params + (size_t)i * FLOATS_PER_GAUSSIAN);
#pragma unroll
  for (int q = 0; q < 4; q++) dst[q] = make_float4(out[4 * q], out[4 * q + 1], out[4 * q + 2], out[4 * q + 3]);
}

// A stream-ordered allocation freed when it goes out of scope (after the work
// already enqueued on the stream).
struct Scratch {
  cudaStream_t stream;
  void* ptr = nullptr;
  explicit Scratch(cudaStream_t s) : stream(s) {}
  ~Scratch() {
    if (ptr) cudaFreeAsync(ptr, stream);
  }
  template <typename T>
  T* at(size_t offset) const {
    return reinterpret_cast<T*>(static_cast<char*>(ptr) + offset);
  }
};

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Mean neighbour distances of n points (float4, xyz + padding) into distance2.
dg_status neighbor_distance2(dg_context* ctx, const float4* points, uint32_t n, float* distance2) {
  if (n == 0) return DG_OK;
  cudaStream_t st = ctx->stream;
  // 63-bit keys: all 32 low-word bits and 31 high-word bits, 8 even passes.
  const SortPlan plan = sort_plan_digits(n, 2, 3 * BITS - 32);
  const uint32_t shares = std::min(ceil_div(n, KNN_THREADS), (uint32_t)ctx->sm_count * 2u);
  Tree tree{};
  size_t boxes = 0;
  for (uint32_t count = ceil_div(n, 32);; count = ceil_div(count, 32)) {
    tree.count[tree.top] = count;
    boxes += count;
    if (count <= 32) break;
    tree.top++;
  }
  const size_t off_values = align256((size_t)n * 8);
  const size_t off_keys_alt = align256(off_values + (size_t)n * 4);
  const size_t off_values_alt = align256(off_keys_alt + (size_t)n * 8);
  const size_t off_sort = align256(off_values_alt + (size_t)n * 4);
  const size_t off_sorted = align256(off_sort + sort_scratch_bytes(plan));
  const size_t off_boxes = align256(off_sorted + (size_t)n * 16);
  const size_t off_shares = align256(off_boxes + boxes * sizeof(Box));
  const size_t off_octree = align256(off_shares + shares * sizeof(Moments));
  Scratch scratch(st);
  DG_CUDA(cudaMallocAsync(&scratch.ptr, off_octree + sizeof(Octree), st));
  uint2* keys = scratch.at<uint2>(0);
  uint32_t* values = scratch.at<uint32_t>(off_values);
  float4* sorted = scratch.at<float4>(off_sorted);
  Box* level = scratch.at<Box>(off_boxes);
  Octree* octree = scratch.at<Octree>(off_octree);
  DG_LAUNCH(ctx, "knn_bounds", bounds_kernel<<<shares, KNN_THREADS, 0, st>>>(points, n, scratch.at<Moments>(off_shares)));
  DG_LAUNCH(ctx, "knn_octree", octree_kernel<<<1, KNN_THREADS, 0, st>>>(scratch.at<Moments>(off_shares), shares, octree));
  const uint32_t grid = ceil_div(n, KNN_THREADS);
  DG_LAUNCH(ctx, "knn_morton", morton_kernel<<<grid, KNN_THREADS, 0, st>>>(points, n, octree, keys, values));
  DG_TRY(sort_launch(ctx, plan, keys, values, scratch.at<void>(off_keys_alt), scratch.at<uint32_t>(off_values_alt),
                     nullptr, scratch.at<void>(off_sort)));
  DG_LAUNCH(ctx, "knn_gather", gather_points_kernel<<<grid, KNN_THREADS, 0, st>>>(points, n, values, sorted, level));
  tree.boxes[0] = level;
  for (uint32_t l = 1; l <= tree.top; l++) {
    Box* parents = level + tree.count[l - 1];
    DG_LAUNCH(ctx, "knn_parents",
              parents_kernel<<<ceil_div(tree.count[l - 1], KNN_THREADS), KNN_THREADS, 0, st>>>(level, tree.count[l - 1],
                                                                                               parents));
    tree.boxes[l] = level = parents;
  }
  DG_LAUNCH(ctx, "knn_query",
            knn_query_kernel<<<ceil_div(tree.count[0], QUERY_WARPS), QUERY_WARPS * 32, 0, st>>>(sorted, n, tree,
                                                                                                distance2));
  return DG_OK;
}

}  // namespace
}  // namespace dg

using namespace dg;

dg_status dg_mean_neighbor_distance2_buffers(dg_context* ctx, dg_buffer* points, uint32_t count,
                                             dg_buffer* distance2) {
  DG_REQUIRE(ctx && points && distance2, "NULL argument");
  DG_REQUIRE((uint64_t)count * 16 <= points->bytes, "points buffer smaller than count × 16 bytes");
  DG_REQUIRE((uint64_t)count * 4 <= distance2->bytes, "distance2 buffer smaller than count × 4 bytes");
  return neighbor_distance2(ctx, typed<float4>(points), count, typed<float>(distance2));
}

dg_status dg_mean_neighbor_distance2(dg_context* ctx, const float* positions, uint32_t count, float* distance2) {
  DG_REQUIRE(ctx && (count == 0 || (positions && distance2)), "NULL argument");
  if (count == 0) return DG_OK;
  cudaStream_t st = ctx->stream;
  // positions (12 B per point), points (16 B, 16-byte aligned), distance2 (4 B)
  const size_t off_points = align256((size_t)count * 12);
  const size_t off_out = off_points + (size_t)count * 16;
  Scratch dev(st);
  DG_CUDA(cudaMallocAsync(&dev.ptr, off_out + (size_t)count * 4, st));
  float4* points = dev.at<float4>(off_points);
  float* out = dev.at<float>(off_out);
  DG_CUDA(cudaMemcpyAsync(dev.ptr, positions, (size_t)count * 12, cudaMemcpyHostToDevice, st));
  DG_LAUNCH(ctx, "knn_pad_points",
            pad_points_kernel<<<ceil_div(count, KNN_THREADS), KNN_THREADS, 0, st>>>(dev.at<float>(0), count, points));
  DG_TRY(neighbor_distance2(ctx, points, count, out));
  DG_CUDA(cudaMemcpyAsync(distance2, out, (size_t)count * 4, cudaMemcpyDeviceToHost, st));
  DG_CUDA(cudaStreamSynchronize(st));
  return DG_OK;
}

dg_status dg_initial_gaussians(dg_context* ctx, const float* positions, const uint8_t* colors, uint32_t count,
                               float* params, float* sh) {
  DG_REQUIRE(ctx && (count == 0 || (positions && colors && params && sh)), "NULL argument");
  if (count == 0) return DG_OK;
  cudaStream_t st = ctx->stream;
  // positions (12 B), points (16 B), distance2 (4 B), params (64 B), colors (3 B)
  const size_t off_points = align256((size_t)count * 12);
  const size_t off_dist = off_points + (size_t)count * 16;
  const size_t off_params = align256(off_dist + (size_t)count * 4);
  const size_t off_colors = off_params + (size_t)count * 64;
  Scratch dev(st);
  DG_CUDA(cudaMallocAsync(&dev.ptr, off_colors + (size_t)count * 3, st));
  float4* points = dev.at<float4>(off_points);
  float* dist = dev.at<float>(off_dist);
  float* dparams = dev.at<float>(off_params);
  uint8_t* dcolors = dev.at<uint8_t>(off_colors);
  DG_CUDA(cudaMemcpyAsync(dev.ptr, positions, (size_t)count * 12, cudaMemcpyHostToDevice, st));
  DG_CUDA(cudaMemcpyAsync(dcolors, colors, (size_t)count * 3, cudaMemcpyHostToDevice, st));
  const uint32_t grid = ceil_div(count, KNN_THREADS);
  DG_LAUNCH(ctx, "knn_pad_points", pad_points_kernel<<<grid, KNN_THREADS, 0, st>>>(dev.at<float>(0), count, points));
  DG_TRY(neighbor_distance2(ctx, points, count, dist));
  // Math.log(0.1 / 0.9) (src/loadDataset.ts:102), rounded to float32.
  const float opacity_logit = (float)std::log(0.1 / 0.9);
  DG_LAUNCH(ctx, "initial_gaussians", initial_gaussians_kernel<<<grid, KNN_THREADS, 0, st>>>(
                                          points, dcolors, dist, count, opacity_logit, dparams));
  DG_CUDA(cudaMemcpyAsync(params, dparams, (size_t)count * 64, cudaMemcpyDeviceToHost, st));
  DG_CUDA(cudaStreamSynchronize(st));
  std::memset(sh, 0, (size_t)count * SH_REST_FLOATS * 4);  // new Float32Array: zeros
  return DG_OK;
}
