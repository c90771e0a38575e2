// The tile lists of a frame (src/shaders/tiles.wgsl:37-84, src/radixSort.ts) from
// splats already sorted by depth: a counting sort of the (splat, tile) pairs by
// tile, without ever writing the pairs' keys.
//
// A splat covers a rectangle of tiles, so its pairs need not be emitted to be
// counted or placed. The depth order is cut into chunks of 256 to 2048 splats and
// the grid of tiles into bins of 16 x 16. For a (chunk, bin):
//   1. the CTA keeps the chunk's splats that touch the bin, in order, and turns
//      each 32 of them into 32 words by a bit transpose across the warp: word c
//      (below 16) has bit i set when splat i covers column c, word 16 + r when it
//      covers row r. The splats of a tile are then one AND of two words.
//   2. The CTA writes the bin's entries to their places in the tiles' lists
//      (bin_scatter_kernel).
// Before that, bin_count_kernel counts each chunk's splats per tile, bin_scan_kernel
// turns the counts into the chunk's place within each tile's list, and
// bin_ranges_kernel scans the tiles and writes their ranges. Within a tile the splats come out nearest first, ties by index: the order
// of the reference's stable sort of (tile, depth) keys.
//
// A stable two-pass radix sort of emitted pairs moves 16 bytes a pair and pass,
// after writing 8 bytes a pair and reading 4 for the digit histograms; here a pair
// costs the 4 bytes of its list entry and a few instructions. Emission also gave
// each warp the pairs of 32 neighbours in depth order, and the nearest splats are
// the largest: the first warps wrote up to 8000 pairs a splat while the rest of
// the GPU was done.
// Measured against it (duplicate + digit histogram + 2 passes + ranges + plan, and
// the scan of the tile counts): 1.1M splats and 28.6M pairs in 8487 tiles, 852 ->
// 243 us; 1.1M and 5.5M in 2170 tiles, 213 -> 109; 100,000 and 468,000, 78 -> 47;
// 5,003 and 13,000 in 192 tiles, 48 -> 35 (event-timed, a launch's 2 us each).
// What bounds it: instructions (issue 56-64%), about 4.5 a pair at 26 pairs a
// splat, and the barriers of CTAs whose bins hold few splats. MAX_CHUNK 4096 gave
// 200 and 82 us for the scatter of the first two against 193 and 68.
#include "dg_bin.cuh"

#include <algorithm>

#include "dg_render_kernels.cuh"  // the plan's layout (no kernels here)

namespace dg {
namespace {

constexpr uint32_t BIN_THREADS = 256, BIN_WARPS = BIN_THREADS / 32;
constexpr uint32_t BIN_SIDE = 16;  // tiles per side of a bin: a thread per tile
constexpr uint32_t MIN_CHUNK = BIN_THREADS, MAX_CHUNK = 2048;
constexpr uint32_t SCATTER_ROOM = 6144;  // entries of one (chunk, bin) that go through shared memory
constexpr uint32_t DENSE = 48;  // tiles of a bin that its splats cover on average, from which it is dense
constexpr uint32_t ROUNDS = MAX_CHUNK / 1024;  // words of 32 splats a lane holds of a chunk at most
constexpr uint32_t SCAN_THREADS = 1024, SCAN_ROWS = 24;
constexpr uint32_t RANGE_THREADS = 1024;

// Where a frame that needs more pairs than there is room for stops: the first
// `kept` pairs of the splat `index` of chunk `chunk` are the last ones listed.
struct Limit {
  uint32_t chunk, index, kept, pad;
};
struct State {
  Limit limit;
};

struct Bins {
  BinShape s;
  uint32_t tiles;          // per view
  uint32_t chunk, chunks;  // splats per chunk, chunks per view
  uint32_t bins_x, bins;
  uint32_t* counts;        // [view][chunk][tile]: splats, then their place in the tile's list
  uint32_t* totals;        // [view][tile]
  uint32_t* chunk_pairs;   // [view][chunk]
  uint32_t* sorted;        // [view][splat]: the rectangles in depth order
  uint32_t* hits;          // [view][chunk][32 splats][bin]: which of them touch the bin
  State* state;
};

// Chunks small enough that a small scene still gives every SM work, and large
// enough that the counts (4 bytes per chunk and tile, read and written twice) stay
// small beside the pairs.
uint32_t chunk_of(uint32_t per_view) {
  uint32_t c = MIN_CHUNK;
  while (c < MAX_CHUNK && (uint64_t)c * 256 < per_view) c *= 2;
  return c;
}

Bins bins_of(const BinShape& s, void* scratch) {
  Bins b{};
  b.s = s;
  b.tiles = s.grid_x * s.grid_y;
  b.chunk = chunk_of(s.per_view);
  b.chunks = std::max(1u, ceil_div(s.per_view, b.chunk));
  b.bins_x = ceil_div(s.grid_x, BIN_SIDE);
  b.bins = b.bins_x * ceil_div(s.grid_y, BIN_SIDE);
  b.state = static_cast<State*>(scratch);
  b.chunk_pairs = reinterpret_cast<uint32_t*>(b.state + 1);
  b.totals = b.chunk_pairs + (size_t)s.views * b.chunks;
  b.sorted = b.totals + (size_t)s.views * b.tiles;
  b.hits = b.sorted + (size_t)s.views * s.per_view;
  b.counts = b.hits + (size_t)s.views * b.chunks * (b.chunk / 32) * b.bins;
  return b;
}

// Words per row of the count's difference array: past the last column, and odd.
__host__ __device__ __forceinline__ uint32_t count_pitch(uint32_t width) { return (width + 1) | 1u; }
size_t count_bytes(const Bins& b) { return (size_t)count_pitch(b.s.grid_x) * (b.s.grid_y + 1) * 4; }

__device__ __forceinline__ uint32_t rect_area(uint32_t r) {
  return ((r >> 16 & 0xffu) - (r & 0xffu)) * ((r >> 24) - (r >> 8 & 0xffu));
}

__device__ __forceinline__ bool rect_covers(uint32_t r, uint32_t x, uint32_t y) {
  return x >= (r & 0xffu) && x < (r >> 16 & 0xffu) && y >= (r >> 8 & 0xffu) && y < r >> 24;
}

// Bits [lo - origin, hi - origin) of a bin's 16 columns or rows.
__device__ __forceinline__ uint32_t span_bits(uint32_t lo, uint32_t hi, uint32_t origin) {
  const int32_t a = max((int32_t)(lo - origin), 0), b = min((int32_t)(hi - origin), (int32_t)BIN_SIDE);
  return ((1u << b) - 1u) & ~((1u << a) - 1u);
}

// The 32 x 32 bit matrix whose row l is lane l's word, transposed.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, uint32_t lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (uint32_t j = 16; j > 0; j >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = lane & j ? (x & ~m) | (y >> j & m) : (x & m) | (y & m) << j;
    m ^= m << (j >> 1);
  }
  return x;
}

// Bit b set for each of the grid's (at most 64) bins, row by row, that a rectangle touches.
__device__ __forceinline__ uint64_t rect_bins(uint32_t r, uint32_t bins_x) {
  const uint32_t x0 = r & 0xffu, y0 = r >> 8 & 0xffu, x1 = r >> 16 & 0xffu, y1 = r >> 24;
  if (x1 <= x0 || y1 <= y0) return 0;
  const uint64_t columns = (1ull << ((x1 + BIN_SIDE - 1) / BIN_SIDE)) - (1ull << (x0 / BIN_SIDE));
  uint64_t bins = 0;
  for (uint32_t y = y0 / BIN_SIDE; y <= (y1 - 1) / BIN_SIDE; y++) bins |= columns << (y * bins_x);
  return bins;
}

// counts[view][chunk][tile] = the chunk's splats covering the tile, chunk_pairs =
// its pairs, sorted = its rectangles in depth order. A rectangle adds 1 at its
// first corner and takes it off past its sides, in a difference array of the whole
// grid in shared memory; prefix sums along the rows, then down the columns, give
// the counts: four shared-memory additions a splat whatever it covers. (Counting
// bits of the bins' words like the scatter took 52 us instead of 15 at 1.1M
// splats and 8487 tiles.) Grid: (chunks, views).
__global__ void __launch_bounds__(BIN_THREADS) bin_count_kernel(const Bins b, const uint32_t* rects,
                                                                const uint32_t* order) {
  chain_begin();
  extern __shared__ uint32_t smem[];
  __shared__ uint32_t s_sum[BIN_WARPS];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const uint32_t chunk = blockIdx.x, view = blockIdx.y, row = view * b.chunks + chunk;
  const uint32_t width = b.s.grid_x, height = b.s.grid_y, pitch = count_pitch(width);
  for (uint32_t k = t; k < pitch * (height + 1); k += BIN_THREADS) smem[k] = 0;
  const uint32_t first = chunk * b.chunk, n = min(b.chunk, b.s.per_view - min(first, b.s.per_view));
  const size_t at0 = (size_t)view * b.s.per_view + first;
  uint32_t r[MAX_CHUNK / BIN_THREADS];
#pragma unroll
  for (uint32_t u = 0; u < MAX_CHUNK / BIN_THREADS; u++) {
    const uint32_t i = u * BIN_THREADS + t;
    r[u] = i < n ? order[at0 + i] : ~0u;
  }
#pragma unroll
  for (uint32_t u = 0; u < MAX_CHUNK / BIN_THREADS; u++) r[u] = r[u] != ~0u ? rects[r[u]] : 0u;
  uint32_t area = 0;
#pragma unroll
  for (uint32_t u = 0; u < MAX_CHUNK / BIN_THREADS; u++) {
    const uint32_t i = u * BIN_THREADS + t;
    if (i < n) b.sorted[at0 + i] = r[u];
    area += rect_area(r[u]);
  }
  area = __reduce_add_sync(0xffffffffu, area);
  if (lane == 0) s_sum[warp] = area;
  // Which bins each 32 splats touch, bin by bin.
#pragma unroll
  for (uint32_t u = 0; u < MAX_CHUNK / BIN_THREADS; u++) {
    if (u * BIN_THREADS >= b.chunk) break;
    const uint64_t bins = rect_bins(r[u], b.bins_x);
    uint32_t* hits = b.hits + ((size_t)row * (b.chunk / 32) + u * BIN_WARPS + warp) * b.bins;
    const uint32_t lo = transpose32((uint32_t)bins, lane);
    if (lane < b.bins) hits[lane] = lo;
    if (b.bins > 32) {
      const uint32_t hi = transpose32((uint32_t)(bins >> 32), lane);
      if (lane + 32 < b.bins) hits[lane + 32] = hi;
    }
  }
  __syncthreads();
  if (t == 0) {
    uint32_t pairs = 0;
#pragma unroll
    for (uint32_t w = 0; w < BIN_WARPS; w++) pairs += s_sum[w];
    b.chunk_pairs[row] = pairs;
  }
#pragma unroll
  for (uint32_t u = 0; u < MAX_CHUNK / BIN_THREADS; u++) {
    if (rect_area(r[u]) == 0) continue;
    const uint32_t x0 = r[u] & 0xffu, x1 = r[u] >> 16 & 0xffu;
    uint32_t* top = smem + (r[u] >> 8 & 0xffu) * pitch;
    uint32_t* end = smem + (r[u] >> 24) * pitch;
    atomicAdd(top + x0, 1u);
    atomicAdd(top + x1, ~0u);
    atomicAdd(end + x0, ~0u);
    atomicAdd(end + x1, 1u);
  }
  __syncthreads();
  for (uint32_t y = t; y < height; y += BIN_THREADS) {  // the odd pitch keeps the rows in different banks
    uint32_t sum = 0;
#pragma unroll 8
    for (uint32_t x = 0; x < width; x++) {
      sum += smem[y * pitch + x];
      smem[y * pitch + x] = sum;
    }
  }
  __syncthreads();
  uint32_t* out = b.counts + (size_t)row * b.tiles;
  for (uint32_t x = t; x < width; x += BIN_THREADS) {
    uint32_t sum = 0;
#pragma unroll 8
    for (uint32_t y = 0; y < height; y++) {
      sum += smem[y * pitch + x];
      out[y * width + x] = sum;
    }
  }
}

// Shared memory of the scatter: the chunk's splats that touch the bin, in order, and
// their transposed words; then the entries on their way to the lists (the splat's
// place in the chunk, and its tile) or the listed splats' numbers.
struct ChunkStage {
  uint32_t* words;  // [chunk]: 32 words per 32 listed splats
  uint16_t* list;   // [chunk]

  // Which of the 32 listed splats from k on cover tile t (x + 16 y) of the bin.
  __device__ __forceinline__ uint32_t covering(uint32_t k, uint32_t t) const {
    return words[k + (t & 15u)] & words[k + BIN_SIDE + (t >> 4)];
  }
};
static_assert(SCATTER_ROOM * 3 >= MAX_CHUNK * 4, "the room also holds the listed splats' numbers");
size_t scatter_bytes(uint32_t chunk) { return (size_t)chunk * 6 + SCATTER_ROOM * 3; }

// Exclusive scan of one value per thread over the CTA's 256 threads; `total` gets the sum.
__device__ __forceinline__ uint32_t bin_exclusive(uint32_t v, uint32_t* s_warp, uint32_t& total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += u;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t before = 0;
  total = 0;
#pragma unroll
  for (uint32_t w = 0; w < BIN_WARPS; w++) {
    before += w < warp ? s_warp[w] : 0u;
    total += s_warp[w];
  }
  return before + incl - v;
}

// Writes the splats of the (chunk, bin)s to their places in the tiles' lists
// (counts holds each chunk's place in each list). Thread t owns tile t (x + 16 y) of
// a bin. Two ways to write a bin's splats:
// - dense (their rectangles cover DENSE tiles of the bin each, or more): a thread
//   walks the bits of its tile's words and writes its own list, four entries
//   together. The tiles' lists are then about as long as each other.
// - else a warp takes 32 of the splats at a time; pair p of their clipped
//   rectangles in turn goes to lane p % 32, which finds its splat by a binary search
//   over the rectangles' prefix and its place in the tile's list by counting the
//   bits of the tile's word before the splat's. (On a captured scene, whose densest
//   tile holds 30,000 splats and its neighbours few, a warp of threads with a tile
//   each would wait for its fullest tile: the whole pass took 1.7 times as long.)
//   The entries go through shared memory when they fit there, grouped by tile, so
//   that a tile's run is written together; a 4-byte store into a list of its own
//   costs a 32-byte sector.
// Grid: (bins x chunks, views): the nearest chunks, which cover the most tiles, first.
__global__ void __launch_bounds__(BIN_THREADS) bin_scatter_kernel(const Bins b,
                                                                  const uint32_t* order,
                                                                  const uint2* ranges,
                                                                  uint32_t* values) {
  chain_begin();
  extern __shared__ uint32_t smem[];
  constexpr uint32_t TILES = BIN_SIDE * BIN_SIDE;
  static_assert(TILES == BIN_THREADS, "a thread per tile of the bin");
  __shared__ uint32_t s_sum[BIN_WARPS];
  __shared__ uint32_t s_at[BIN_WARPS][TILES];  // where a warp's next entry of a tile goes
  __shared__ uint32_t s_delta[TILES];          // a tile's place in the lists less its place in the buffer
  __shared__ uint32_t s_excl[BIN_WARPS][32];   // of a warp's 32 splats: the pairs before each,
  __shared__ uint2 s_hit[BIN_WARPS][32];       // and its rectangle
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, below = (1u << lane) - 1u;
  const uint32_t bin = blockIdx.x % b.bins, chunk = blockIdx.x / b.bins, view = blockIdx.y, row = view * b.chunks + chunk;
  const uint32_t rounds = b.chunk / 32;  // 32 splats each
  const ChunkStage st{smem, reinterpret_cast<uint16_t*>(smem + b.chunk)};
  uint16_t* const buffer = st.list + b.chunk;                                      // [SCATTER_ROOM]
  uint8_t* const buffer_tile = reinterpret_cast<uint8_t*>(buffer + SCATTER_ROOM);  // [SCATTER_ROOM]
  uint32_t* const listed_splat = reinterpret_cast<uint32_t*>(buffer);              // [chunk]
  const Limit limit = b.state->limit;
  if (row > limit.chunk) return;
  const uint32_t first = chunk * b.chunk;
  const size_t at0 = (size_t)view * b.s.per_view + first;
  const uint32_t* splats = order + at0;
  const uint32_t* rects = b.sorted + at0;
  const uint32_t bx = bin % b.bins_x * BIN_SIDE, by = bin / b.bins_x * BIN_SIDE;
  const uint32_t x = bx + (t & 15u), y = by + (t >> 4), tile = y * b.s.grid_x + x;
  const bool inside = x < b.s.grid_x && y < b.s.grid_y;
  // The bin's splats of each round (lane l: rounds l, l + 32, ...), and before it.
  const uint32_t* hits = b.hits + (size_t)row * rounds * b.bins + bin;
  uint32_t word[ROUNDS], before[ROUNDS], kept = 0;
#pragma unroll
  for (uint32_t u = 0; u < ROUNDS; u++) {
    const uint32_t j = u * 32 + lane;
    word[u] = j < rounds ? hits[(size_t)j * b.bins] : 0u;
    // Past the limit nothing is listed; the last splat goes in at the end, as far as
    // there is room.
    if (row == limit.chunk && j * 32 + 32 > limit.index)
      word[u] &= j * 32 >= limit.index ? 0u : (1u << (limit.index - j * 32)) - 1u;
  }
  // The tile's entries of this chunk, and where they go.
  uint32_t start = 0, mine = 0;
  if (inside) {
    const uint32_t* place = b.counts + (size_t)row * b.tiles + tile;
    start = place[0];
    mine = (chunk + 1 < b.chunks ? place[b.tiles] : b.totals[(size_t)view * b.tiles + tile]) - start;
    start += ranges[(size_t)view * b.tiles + tile].x;
    if (row == limit.chunk) {
      const uint32_t cut = rects[limit.index], width = (cut >> 16 & 0xffu) - (cut & 0xffu);
      if (rect_covers(cut, x, y) && (y - (cut >> 8 & 0xffu)) * width + x - (cut & 0xffu) < limit.kept)
        values[start + --mine] = splats[limit.index];
    }
  }
#pragma unroll
  for (uint32_t u = 0; u < ROUNDS; u++) {
    before[u] = __popc(word[u]);
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, before[u], d);
      if (lane >= d) before[u] += v;
    }
    const uint32_t sum = __shfl_sync(0xffffffffu, before[u], 31);
    before[u] += kept - __popc(word[u]);
    kept += sum;
  }
  if (kept == 0) return;  // the same on every thread
  // Warp w lists rounds w, w + 8, ...
#pragma unroll
  for (uint32_t u = 0; u < ROUNDS; u++) {
#pragma unroll
    for (uint32_t v = 0; v < 32 / BIN_WARPS; v++) {
      const uint32_t from = v * BIN_WARPS + warp, j = u * 32 + from;
      const uint32_t bits = __shfl_sync(0xffffffffu, word[u], from);
      if (bits == 0) continue;
      const uint32_t base = __shfl_sync(0xffffffffu, before[u], from);
      if (bits >> lane & 1u) st.list[base + __popc(bits & below)] = (uint16_t)(j * 32 + lane);
    }
  }
  uint32_t entries;
  const uint32_t local = bin_exclusive(mine, s_sum, entries);  // and a barrier: the list is complete
  // 32 listed splats at a time, consecutive ones to a warp.
  const uint32_t per_warp = (kept + 32 * BIN_WARPS - 1) / (32 * BIN_WARPS) * 32;
  const uint32_t from = min(warp * per_warp, kept), to = min(from + per_warp, kept);
  for (uint32_t k = from; k < to; k += 32) {
    uint32_t w = 0;
    if (k + lane < to) {
      const uint32_t r = rects[st.list[k + lane]];
      w = span_bits(r & 0xffu, r >> 16 & 0xffu, bx) | span_bits(r >> 8 & 0xffu, r >> 24, by) << BIN_SIDE;
    }
    st.words[k + lane] = transpose32(w, lane);
  }
  if (entries >= kept * DENSE) {
    for (uint32_t k = t; k < kept; k += BIN_THREADS) listed_splat[k] = splats[st.list[k]];
    __syncthreads();
    uint32_t* out = values + start;
    const uint32_t head = (4u - (start & 3u)) & 3u;  // entries before the first 16-byte boundary
    uint32_t done = 0, p0 = 0, p1 = 0, p2 = 0;       // the last three entries
    for (uint32_t k = 0; k < kept; k += 32) {
      uint32_t bits = st.covering(k, t);
      while (bits) {
        const uint32_t splat = listed_splat[k + __ffs(bits) - 1];
        bits &= bits - 1;
        if (done < head) {
          out[done] = splat;
        } else if (((done - head) & 3u) == 3u) {
          *reinterpret_cast<uint4*>(out + done - 3) = make_uint4(p0, p1, p2, splat);
        }
        p0 = p1;
        p1 = p2;
        p2 = splat;
        done++;
      }
    }
    const uint32_t tail = done > head ? (done - head) & 3u : 0u;
    if (tail > 2) out[done - 3] = p0;
    if (tail > 1) out[done - 2] = p1;
    if (tail > 0) out[done - 1] = p2;
    return;
  }
  __syncthreads();
  const bool buffered = entries <= SCATTER_ROOM;
  s_delta[t] = start - local;
  mine = buffered ? local : start;
  for (uint32_t w = 0, k = 0; k < kept; w++) {
    s_at[w][t] = mine;
    for (const uint32_t end = min(k + per_warp, kept); k < end; k += 32) mine += __popc(st.covering(k, t));
  }
  __syncthreads();
  uint32_t* at = s_at[warp];
  for (uint32_t k = from; k < to; k += 32) {
    // The lane's splat: its rectangle within the bin and the pairs before its own.
    uint32_t pairs = 0, x0 = 0, y0 = 0, width = 1;
    if (k + lane < to) {
      const uint32_t r = rects[st.list[k + lane]];
      x0 = max(r & 0xffu, bx) - bx;
      y0 = max(r >> 8 & 0xffu, by) - by;
      width = min((r >> 16 & 0xffu) - bx, BIN_SIDE) - x0;
      pairs = width * (min((r >> 24) - by, BIN_SIDE) - y0);
    }
    uint32_t incl = pairs;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    // The tile of pair p of a rectangle: p + q (16 - width) past its first tile, with
    // q = p / width, which for p < 256 is p * (65536 / width + 1) / 65536, exactly.
    uint32_t* excl = s_excl[warp];
    excl[lane] = incl - pairs;
    s_hit[warp][lane] = make_uint2((y0 * BIN_SIDE + x0) | (BIN_SIDE - width) << 16, 65536u / width + 1u);
    __syncwarp();
    for (uint32_t p = lane; p < total; p += 32) {
      uint32_t i = 0;
#pragma unroll
      for (uint32_t step = 16; step > 0; step >>= 1)
        if (excl[i + step] <= p) i += step;
      const uint2 hit = s_hit[warp][i];
      const uint32_t in_rect = p - excl[i];
      const uint32_t c = (hit.x & 0xffffu) + in_rect + (in_rect * hit.y >> 16) * (hit.x >> 16);
      const uint32_t slot = at[c] + __popc(st.covering(k, c) & ((1u << i) - 1u));
      const uint32_t which = st.list[k + i];
      if (buffered) {
        buffer[slot] = (uint16_t)which;
        buffer_tile[slot] = (uint8_t)c;
      } else {
        values[slot] = splats[which];
      }
    }
    __syncwarp();
    if (k + 32 < to) {  // the tiles' places after these splats
#pragma unroll
      for (uint32_t c = lane; c < TILES; c += 32) at[c] += __popc(st.covering(k, c));
      __syncwarp();
    }
  }
  __syncthreads();
  if (buffered) {
    for (uint32_t k = t; k < entries; k += BIN_THREADS) values[s_delta[buffer_tile[k]] + k] = splats[buffer[k]];
  }
}

// Of `n` counts, consecutive ones per thread, the first whose running sum passes `left`
// (their whole sum does): its place, and what of `left` remains before it. All threads get
// it. count(i) is called once or twice per i.
struct Passed {
  uint32_t at, left;
};
template <class Count>
__device__ __forceinline__ Passed first_past(uint32_t n, uint32_t left, Count count) {
  __shared__ unsigned long long s_warp[SCAN_THREADS / 32];
  __shared__ Passed s_passed;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t each = (n + SCAN_THREADS - 1) / SCAN_THREADS;
  const uint32_t from = min(threadIdx.x * each, n), to = min(from + each, n);
  unsigned long long mine = 0;
  for (uint32_t i = from; i < to; i++) mine += count(i);
  unsigned long long before = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, before, d);
    if (lane >= d) before += v;
  }
  if (lane == 31) s_warp[warp] = before;
  before -= mine;
  __syncthreads();
  for (uint32_t w = 0; w < warp; w++) before += s_warp[w];
  if (before <= left && left < before + mine) {  // one thread
    Passed p{from, left - (uint32_t)before};
    for (uint32_t c = count(p.at); c <= p.left; c = count(++p.at)) p.left -= c;
    s_passed = p;
  }
  __syncthreads();
  const Passed p = s_passed;
  __syncthreads();
  return p;
}

// The chunk and splat at which the pairs reach `capacity` (there are more than
// that). One call per CTA.
__device__ __forceinline__ Limit find_limit(const Bins& b, uint32_t capacity) {
  const Passed row = first_past(b.s.views * b.chunks, capacity, [&](uint32_t c) { return b.chunk_pairs[c]; });
  const uint32_t first = row.at % b.chunks * b.chunk, n = min(b.chunk, b.s.per_view - first);
  const uint32_t* sorted = b.sorted + (size_t)(row.at / b.chunks) * b.s.per_view + first;
  const Passed splat = first_past(n, row.left, [&](uint32_t i) { return rect_area(sorted[i]); });
  return Limit{row.at, splat.at, splat.left, 0u};
}

// Each tile's counts over the chunks become exclusive prefixes, its total goes to
// totals. A CTA takes 32 tiles, a lane each;
// its 32 warps take consecutive runs of chunks, in registers up to SCAN_ROWS each
// (1.5M splats a view), so the counts are read once and all at the same time.
// (8 warps reading them twice took 55 us instead of 14 at 538 chunks x 8487 tiles.)
// Grid: (tiles / 32, views).
__global__ void __launch_bounds__(SCAN_THREADS) bin_scan_kernel(const Bins b, uint32_t capacity,
                                                                uint32_t* pair_total) {
  chain_begin();
  constexpr uint32_t WARPS = SCAN_THREADS / 32;
  __shared__ uint32_t s_sum[WARPS][32];
  __shared__ unsigned long long s_pairs[WARPS];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, view = blockIdx.y;
  const uint32_t tile = blockIdx.x * 32u + lane;
  const bool inside = tile < b.tiles;
  const uint32_t per_warp = (b.chunks + WARPS - 1) / WARPS;
  const uint32_t r0 = min(warp * per_warp, b.chunks), r1 = min(r0 + per_warp, b.chunks);
  uint32_t* column = b.counts + (size_t)view * b.chunks * b.tiles + tile;
  uint32_t v[SCAN_ROWS];
#pragma unroll
  for (uint32_t k = 0; k < SCAN_ROWS; k++) v[k] = inside && r0 + k < r1 ? column[(size_t)(r0 + k) * b.tiles] : 0u;
  // The pairs of the whole frame.
  unsigned long long pairs = 0;
  for (uint32_t k = threadIdx.x; k < b.s.views * b.chunks; k += SCAN_THREADS) pairs += b.chunk_pairs[k];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, d);
  if (lane == 0) s_pairs[warp] = pairs;
  __syncthreads();
  pairs = 0;
#pragma unroll
  for (uint32_t w = 0; w < WARPS; w++) pairs += s_pairs[w];
  const bool first_cta = blockIdx.x == 0 && view == 0 && threadIdx.x == 0;
  if (first_cta) *pair_total = (uint32_t)pairs;
  if (pairs > capacity) {
    // Nothing past the limit counts.
    const Limit limit = find_limit(b, capacity);
    if (first_cta) b.state->limit = limit;
    const uint32_t row0 = view * b.chunks;
    if (inside) {
      for (uint32_t r = r0; r < r1; r++) {
        if (row0 + r < limit.chunk) continue;
        uint32_t c = 0;
        if (row0 + r == limit.chunk) {
          const uint32_t* sorted = b.sorted + (size_t)view * b.s.per_view + r * b.chunk;
          const uint32_t x = tile % b.s.grid_x, y = tile / b.s.grid_x;
          for (uint32_t i = 0; i < limit.index; i++) c += rect_covers(sorted[i], x, y);
          const uint32_t cut = sorted[limit.index];
          const uint32_t x0 = cut & 0xffu, y0 = cut >> 8 & 0xffu, w = (cut >> 16 & 0xffu) - x0;
          if (rect_covers(cut, x, y) && (y - y0) * w + x - x0 < limit.kept) c++;
        }
        column[(size_t)r * b.tiles] = c;
      }
#pragma unroll
      for (uint32_t k = 0; k < SCAN_ROWS; k++) v[k] = r0 + k < r1 ? column[(size_t)(r0 + k) * b.tiles] : 0u;
    }
  } else if (first_cta) {
    b.state->limit = Limit{~0u, 0u, 0u, 0u};
  }
  uint32_t sum = 0;
#pragma unroll
  for (uint32_t k = 0; k < SCAN_ROWS; k++) sum += v[k];
  if (inside)
    for (uint32_t r = r0 + SCAN_ROWS; r < r1; r++) sum += column[(size_t)r * b.tiles];
  s_sum[warp][lane] = sum;
  __syncthreads();
  uint32_t before = 0;
#pragma unroll
  for (uint32_t w = 0; w < WARPS; w++) before += w < warp ? s_sum[w][lane] : 0u;
  if (inside) {
#pragma unroll
    for (uint32_t k = 0; k < SCAN_ROWS; k++) {
      if (r0 + k < r1) column[(size_t)(r0 + k) * b.tiles] = before;
      before += v[k];
    }
    for (uint32_t r = r0 + SCAN_ROWS; r < r1; r++) {
      const uint32_t c = column[(size_t)r * b.tiles];
      column[(size_t)r * b.tiles] = before;
      before += c;
    }
  }
  // The last warp has its tiles' lengths.
  if (warp == WARPS - 1 && inside) b.totals[(size_t)view * b.tiles + tile] = before;
}

// A thread per tile: the tile's run of the pair list. Each CTA adds up the tiles
// before its own (a few L2 reads a thread). The first clears what the blend's plan
// counts into.
__global__ void __launch_bounds__(RANGE_THREADS) bin_ranges_kernel(const Bins b, uint2* ranges,
                                                                   uint32_t* plan,
                                                                   uint32_t* work) {
  chain_begin();
  constexpr uint32_t WARPS = RANGE_THREADS / 32;
  static_assert(WARPS == 32, "a warp's lanes read one word per warp");
  __shared__ uint32_t s_before[WARPS], s_sum[WARPS];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t tiles = b.s.views * b.tiles, t = blockIdx.x * RANGE_THREADS + tid;
  if (blockIdx.x == 0) {
    if (tid < PLAN_HEADER) plan[tid] = 0;
    if (tid < 4) work[tid] = 0;
  }
  uint32_t before = 0;
  for (uint32_t k = tid; k < blockIdx.x * RANGE_THREADS; k += RANGE_THREADS) before += b.totals[k];
  const uint32_t len = t < tiles ? b.totals[t] : 0u;
  uint32_t incl = len;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += u;
  }
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 31) {
    s_before[warp] = before;
    s_sum[warp] = incl;
  }
  __syncthreads();
  const uint32_t start =
      __reduce_add_sync(0xffffffffu, s_before[lane] + (lane < warp ? s_sum[lane] : 0u)) + incl - len;
  if (t < tiles) ranges[t] = len ? make_uint2(start, start + len) : make_uint2(0u, 0u);
}

// A warp per tile.
__global__ void __launch_bounds__(BIN_THREADS) bin_keys_kernel(uint32_t tiles, const uint2* __restrict__ ranges,
                                                               const uint32_t* __restrict__ values,
                                                               const float* __restrict__ splats,
                                                               uint64_t* __restrict__ keys) {
  const uint32_t tile = (blockIdx.x * BIN_THREADS + threadIdx.x) >> 5;
  if (tile >= tiles) return;
  const uint2 run = ranges[tile];
  for (uint32_t k = run.x + (threadIdx.x & 31u); k < run.y; k += 32)
    keys[k] = (uint64_t)tile << 32 | __float_as_uint(splats[(size_t)values[k] * FLOATS_PER_SPLAT + 2]);
}

}  // namespace

bool bin_fits(uint32_t grid_x, uint32_t grid_y) {
  // A rectangle's four coordinates take a byte each. Every bin tests every splat,
  // so the work grows with the grid: past 64 bins the sort's, which grows with the
  // pairs, may be the smaller.
  return grid_x >= 1 && grid_x <= 255 && grid_y >= 1 && grid_y <= 255 &&
         ceil_div(grid_x, BIN_SIDE) * ceil_div(grid_y, BIN_SIDE) <= 64;
}

size_t bin_scratch_bytes(const BinShape& s) {
  const Bins b = bins_of(s, nullptr);
  return sizeof(State) + (size_t)s.views *
                             (s.per_view + b.tiles +
                              (size_t)b.chunks * (1 + b.tiles + (size_t)(b.chunk / 32) * b.bins)) * 4;
}

dg_status bin_init() {
  // A grid of at most 64 bins: at most 255 x 64 tiles (or 64 x 255), and a row and a
  // column past them.
  DG_CUDA(cudaFuncSetAttribute(bin_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 257 * 66 * 4));
  DG_CUDA(cudaFuncSetAttribute(bin_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)scatter_bytes(MAX_CHUNK)));
  return DG_OK;
}

dg_status bin_launch(dg_context* ctx, const BinShape& s, const BinLaunch& l) {
  const Bins b = bins_of(s, l.scratch);
  DG_CHAIN(ctx, "bin_count", (bin_count_kernel), dim3(b.chunks, s.views), BIN_THREADS, count_bytes(b),
           b, l.rects, l.order);
  DG_CHAIN(ctx, "bin_scan", (bin_scan_kernel), dim3(ceil_div(b.tiles, 32), s.views), SCAN_THREADS, 0,
           b, l.capacity, l.pair_total);
  DG_CHAIN(ctx, "bin_ranges", (bin_ranges_kernel), ceil_div((uint64_t)s.views * b.tiles, RANGE_THREADS), RANGE_THREADS, 0,
           b, l.ranges, l.plan, l.work);
  DG_CHAIN(ctx, "bin_scatter", (bin_scatter_kernel), dim3(b.bins * b.chunks, s.views), BIN_THREADS, scatter_bytes(b.chunk),
           b, l.order, l.ranges, l.values);
  return DG_OK;
}

dg_status bin_keys_launch(dg_context* ctx, uint32_t tiles, const uint2* ranges, const uint32_t* values,
                          const float* splats, uint64_t* keys) {
  DG_LAUNCH(ctx, "bin_keys",
            bin_keys_kernel<<<std::max(1u, ceil_div(tiles, BIN_WARPS)), BIN_THREADS, 0, ctx->stream>>>(
                tiles, ranges, values, splats, keys));
  return DG_OK;
}

}  // namespace dg
