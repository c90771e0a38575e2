// RadixSort (src/radixSort.ts:27-142, src/shaders/radixSort.wgsl:45-120): a
// stable LSD radix sort of u32 keys, or u64 keys stored as (low, high) of which
// the high word contributes `high_bits` bits, each key carrying a u32 value.
//
// The pass plan is the reference's: 8-bit digits, four passes over the low word,
// then 2·ceil(high_bits/16) over the high word, ping-ponging so the result lands
// back in keys/values. Any stable LSD sort over the same digits yields the same
// permutation, so the result is bit-identical to the reference's.
//
// The reference runs count_digits, a multi-level scan and scatter per pass (three
// or more dispatches and four barriers per 256-key chunk). Here it is onesweep
// (Adinets & Merrill 2022): one upfront kernel reads every key once and builds
// the digit histograms of all passes, then each pass is ONE kernel. A CTA takes
// the next tile of 3840 keys (2816 while they are few) by ticket, ranks each key within its warp
// (stable: warp-striped loads are ranked round by round), publishes its
// per-digit counts, looks back over earlier tiles' counts (bounded waits), and
// scatters through shared memory so each digit's run is written contiguously. Up to
// 65,536 u32 keys (43,000 u64) the passes run in one kernel instead (sort_cluster_kernel).
#include "dg_common.cuh"
#include "dg_scan.cuh"

#include <cuda/atomic>

namespace dg {

namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORT_WARPS = SORT_THREADS / 32;
#ifndef DG_SORT_MIN_BLOCKS
#define DG_SORT_MIN_BLOCKS 3  // resident CTAs per SM the pass kernel's registers allow
#endif
// Keys per thread: 15 at 3 CTAs per SM measured fastest for many keys (26M keys 1,319
// us) against 8 and 11 (smaller tiles, longer look-backs) and 19 and 23 at 2 CTAs per
// SM. While the tiles are few, a pass is one tile's chain of 15 rounds, and 11 are
// faster: four passes over 100,000 u32 keys 46.8 and 40.9 us, 201,000 48.5 and 40.7,
// 400,000 48.5 and 48.4, 700,000 62.6 and 56.8, 1.1M 65.0 and 71.8; six over 201,000 u64
// keys 73.7 and 63.6, 700,000 97.7 and 88.7, 1.1M 109.6 and 111.8 (8 keys: as 11 up to
// 201,000, slower beyond).
constexpr int SORT_ITEMS = 15, SORT_ITEMS_FEW = 11;
constexpr uint32_t FEW_KEYS = 800'000;
template <int ITEMS>
constexpr uint32_t SORT_TILE = SORT_THREADS * ITEMS;  // 3840 and 2816
constexpr uint32_t RADIX = 256;
constexpr uint32_t FLAG_AGGREGATE = 1u << 30;
constexpr uint32_t FLAG_PREFIX = 2u << 30;
constexpr uint32_t FLAG_MASK = 3u << 30;
constexpr uint32_t VALUE_MASK = (1u << 30) - 1;
constexpr int HIST_THREADS = 256;
constexpr int MAX_PASSES = 8;
#ifndef DG_SORT_LOOK_WIDTH
#define DG_SORT_LOOK_WIDTH 4
#endif
constexpr int LOOK_WIDTH = DG_SORT_LOOK_WIDTH;  // predecessors read per look-back step (4-32 measured: 4-8 best)

template <int KW>
struct KeyOf;
template <>
struct KeyOf<1> {
  using type = uint32_t;
};
template <>
struct KeyOf<2> {
  using type = uint64_t;
};

__device__ __forceinline__ uint32_t load_status(uint32_t* p) {
  cuda::atomic_ref<uint32_t, cuda::thread_scope_device> ref(*p);
  return ref.load(cuda::memory_order_relaxed);
}
__device__ __forceinline__ void store_status(uint32_t* p, uint32_t v) {
  cuda::atomic_ref<uint32_t, cuda::thread_scope_device> ref(*p);
  ref.store(v, cuda::memory_order_relaxed);
}

struct PassShifts {
  uint32_t shift[MAX_PASSES];
};
// Words from one segment's digit histograms, and states, to the next one's.
struct SegmentStates {
  uint32_t hist, status;
};

// Digit histograms of every pass from one read of the keys. Each thread takes
// HIST_ITEMS consecutive keys and counts runs of equal digits in a register,
// adding a run to the CTA's shared histogram when the digit changes: a splat's
// pairs sit next to each other with the same depth and nearby tiles, so runs are
// common, and the lanes of a warp rarely land on one bin in the same instant.
constexpr uint32_t HIST_ITEMS = 8;
#ifndef DG_HIST_ROUNDS
// HIST_ITEMS-key rounds per thread the grid is sized for (at most 8 CTAs per SM):
// 1, 2 and 4 measured 16.7, 16.0 and 17.0 us per in-step histogram.
#define DG_HIST_ROUNDS 2
#endif

template <int KW>
__global__ void __launch_bounds__(HIST_THREADS) sort_histogram_kernel(const typename KeyOf<KW>::type* keys,
                                                                      uint32_t capacity, const uint32_t* count,
                                                                      uint32_t passes, PassShifts shifts,
                                                                      uint32_t* hist) {
  chain_begin();
  using K = typename KeyOf<KW>::type;
  __shared__ uint32_t s_hist[MAX_PASSES][RADIX];
  keys += (size_t)blockIdx.y * capacity;  // the segment's
  hist += (size_t)blockIdx.y * passes * RADIX;
  for (uint32_t i = threadIdx.x; i < passes * RADIX; i += HIST_THREADS) s_hist[i / RADIX][i % RADIX] = 0;
  __syncthreads();
  const uint32_t n = count ? min(*count, capacity) : capacity;
  const uint64_t stride = (uint64_t)gridDim.x * HIST_THREADS * HIST_ITEMS;
  for (uint64_t base = ((uint64_t)blockIdx.x * HIST_THREADS + threadIdx.x) * HIST_ITEMS; base < n; base += stride) {
    K k[HIST_ITEMS];
    const uint64_t left = (uint64_t)n - base;
    const uint32_t m = left < HIST_ITEMS ? (uint32_t)left : HIST_ITEMS;
    if (m == HIST_ITEMS && (reinterpret_cast<uintptr_t>(keys + base) & 15) == 0) {
      // 16-byte loads (base is a multiple of 8 keys: 32 or 64 bytes in).
      const uint4* src = reinterpret_cast<const uint4*>(keys + base);
#pragma unroll
      for (uint32_t q = 0; q < HIST_ITEMS * sizeof(K) / 16; q++)
        reinterpret_cast<uint4*>(k)[q] = src[q];
    } else {
#pragma unroll
      for (uint32_t j = 0; j < HIST_ITEMS; j++) k[j] = j < m ? keys[base + j] : K(0);
    }
    for (uint32_t p = 0; p < passes; p++) {
      uint32_t run_digit = (uint32_t)((uint64_t)k[0] >> shifts.shift[p]) & 0xffu, run = 1;
#pragma unroll
      for (uint32_t j = 1; j < HIST_ITEMS; j++) {
        if (j >= m) break;
        const uint32_t d = (uint32_t)((uint64_t)k[j] >> shifts.shift[p]) & 0xffu;
        if (d == run_digit) {
          run++;
        } else {
          atomicAdd(&s_hist[p][run_digit], run);
          run_digit = d;
          run = 1;
        }
      }
      atomicAdd(&s_hist[p][run_digit], run);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < passes * RADIX; i += HIST_THREADS) {
    uint32_t c = s_hist[i / RADIX][i % RADIX];
    if (c) atomicAdd(&hist[i], c);
  }
}

// Exclusive scan of one value per thread over the CTA's 256 threads.
__device__ __forceinline__ uint32_t block_exclusive_256(uint32_t v, uint32_t* s_tmp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t n = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += n;
  }
  if (lane == 31) s_tmp[warp] = incl;
  __syncthreads();
  uint32_t before = 0;
#pragma unroll
  for (int w = 0; w < SORT_WARPS; w++) before += w < warp ? s_tmp[w] : 0u;
  __syncthreads();
  return before + incl - v;
}

// One pass over digits of DBITS bits (8, or 4 for a last pass whose key bits
// above it are all zero): fewer ballots per key, and with 16 digits the per-tile
// prefix work and look-back run on 16 threads instead of 256.
template <int KW, int DBITS, int ITEMS>
__global__ void __launch_bounds__(SORT_THREADS, DG_SORT_MIN_BLOCKS)
    sort_pass_kernel(const typename KeyOf<KW>::type* keys_in, const uint32_t* vals_in,
                     typename KeyOf<KW>::type* keys_out, uint32_t* vals_out,
                     uint32_t capacity, const uint32_t* count, uint32_t shift,
                     const uint32_t* pass_hist, uint32_t* status,
                     uint32_t* ticket, SegmentStates states, uint32_t* error) {
  chain_begin();
  using K = typename KeyOf<KW>::type;
  constexpr uint32_t TILE = SORT_TILE<ITEMS>;
  static_assert(TILE * 8 >= SORT_WARPS * 2 * RADIX * 4, "the bits lie where the keys and values are placed");
  extern __shared__ __align__(16) unsigned char smem[];
  K* s_keys = reinterpret_cast<K*>(smem);
  uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys + TILE);
  uint32_t* s_whist = s_vals + TILE;          // [warp][digit]
  uint32_t* s_block_start = s_whist + SORT_WARPS * RADIX;
  uint32_t* s_base = s_block_start + RADIX;
  uint32_t* s_tmp = s_base + RADIX;
  uint32_t* s_match = reinterpret_cast<uint32_t*>(smem);  // [warp][2][digit], until the keys are placed
  __shared__ uint32_t s_tile;

  // The segment's keys and states.
  const size_t segment = (size_t)blockIdx.y * capacity;
  keys_in += segment;
  vals_in += segment;
  keys_out += segment;
  vals_out += segment;
  pass_hist += (size_t)blockIdx.y * states.hist;
  status += (size_t)blockIdx.y * states.status;
  ticket += blockIdx.y * MAX_PASSES;

  constexpr uint32_t DIGITS = 1u << DBITS, DMASK = DIGITS - 1u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t n = count ? min(*count, capacity) : capacity;
  const uint32_t tiles = (n + TILE - 1) / TILE;
  // The grid covers the capacity; CTAs past the tiles of this call's keys leave at
  // once. The first `tiles` CTAs take the tickets 0..tiles-1, in arrival order.
  if (blockIdx.x >= tiles) return;
  if (tid == 0) s_tile = atomicAdd(ticket, 1u);
  for (int i = tid; i < SORT_WARPS * RADIX; i += SORT_THREADS) s_whist[i] = 0;
  for (int i = tid; i < SORT_WARPS * 2 * RADIX; i += SORT_THREADS) s_match[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  if (tile >= tiles) return;
  const uint32_t digit_total = tid < DIGITS ? pass_hist[tid] : 0u;  // on its way while the keys are ranked

  // Load, warp-striped: warp w owns 32 * ITEMS consecutive keys of the tile, round j
  // reads 32 consecutive ones, so order within the tile is (warp, round, lane).
  const uint32_t base = tile * TILE + warp * 32 * ITEMS + lane;
  K key[ITEMS];
  uint32_t val[ITEMS];
  uint32_t rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    uint32_t idx = base + j * 32;
    bool valid = idx < n;
    key[j] = valid ? keys_in[idx] : K(0);
    val[j] = valid ? vals_in[idx] : 0u;
  }
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t* my_hist = s_whist + warp * DIGITS;
  // The lanes that hold the same digit, from a word per digit in which each lane sets
  // its bit: two sets of words in turn, so that a round's bits need not wait for the
  // round before to be cleared. Against eight ballots and their selects per round (the
  // ALU pipe's, 45 cycles of an SM a round): 4.2M u64 keys 285 -> 261 us in six passes,
  // 1.1M u32 keys 73 -> 65 in four, 100k 49 -> 44. __match_any_sync took 90 for 1.1M.
  uint32_t* my_match = s_match + warp * 2 * DIGITS;
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const bool valid = base + j * 32 < n;
    const uint32_t d = (uint32_t)(key[j] >> shift) & DMASK;
    uint32_t* match = my_match + (j & 1) * DIGITS;
    if (valid) atomicOr(&match[d], 1u << lane);
    __syncwarp();
    const uint32_t peers = match[d], old = my_hist[d], before = __popc(peers & lt_mask);
    __syncwarp();
    if (valid && before == 0) {  // the first of them counts them all
      my_hist[d] = old + __popc(peers);
      match[d] = 0;
    }
    rank[j] = old + before;
    __syncwarp();
  }
  __syncthreads();

  // Per digit (thread = digit, threads past the digits idle): offsets of each
  // warp's run, and the tile's count.
  const uint32_t d = tid;
  const bool digit = d < DIGITS;
  uint32_t running = 0;
  if (digit) {
#pragma unroll
    for (int w = 0; w < SORT_WARPS; w++) {
      uint32_t c = s_whist[w * DIGITS + d];
      s_whist[w * DIGITS + d] = running;
      running += c;
    }
    store_status(&status[tile * RADIX + d], (tile == 0 ? FLAG_PREFIX : FLAG_AGGREGATE) | running);
  }
  const uint32_t tile_count = running;
  const uint32_t block_start = block_exclusive_256(tile_count, s_tmp);
  const uint32_t global_start = block_exclusive_256(digit_total, s_tmp);
  if (digit) s_block_start[d] = block_start;

  // Decoupled look-back over earlier tiles, for this thread's digit: the states
  // of LOOK_WIDTH predecessors are read together (one round trip instead of
  // LOOK_WIDTH), then taken in order back to the first inclusive prefix.
  uint32_t prefix = 0;
  if (digit && tile > 0) {
    int32_t look = (int32_t)tile - 1;
    uint32_t spins = 0;
    bool found = false;
    while (look >= 0 && !found) {
      uint32_t st[LOOK_WIDTH];
#pragma unroll
      for (int k = 0; k < LOOK_WIDTH; k++)
        st[k] = look - k >= 0 ? load_status(&status[(look - k) * RADIX + d]) : FLAG_PREFIX;
#pragma unroll
      for (int k = 0; k < LOOK_WIDTH; k++) {
        if (found || look - k < 0) break;
        uint32_t s = st[k];
        while ((s & FLAG_MASK) == 0) {
          if (++spins > SPIN_LIMIT) {
            atomicOr(error, DEVICE_ERROR_SORT_WAIT);
            s = FLAG_PREFIX;  // give up: the order is wrong, but nothing hangs
            break;
          }
          s = load_status(&status[(look - k) * RADIX + d]);
        }
        prefix += s & VALUE_MASK;
        found = (s & FLAG_MASK) == FLAG_PREFIX;
      }
      look -= LOOK_WIDTH;
    }
    store_status(&status[tile * RADIX + d], FLAG_PREFIX | ((prefix + tile_count) & VALUE_MASK));
  }
  if (digit) s_base[d] = global_start + prefix - block_start;
  __syncthreads();

  // Place each key at its rank within the tile, grouped by digit.
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    if (base + j * 32 < n) {
      uint32_t dj = (uint32_t)(key[j] >> shift) & DMASK;
      uint32_t pos = s_block_start[dj] + s_whist[warp * DIGITS + dj] + rank[j];
      s_keys[pos] = key[j];
      s_vals[pos] = val[j];
    }
  }
  __syncthreads();
  const uint32_t here = min(TILE, n - tile * TILE);
  for (uint32_t k = tid; k < here; k += SORT_THREADS) {
    K kk = s_keys[k];
    uint32_t dk = (uint32_t)(kk >> shift) & DMASK;
    uint32_t out = s_base[dk] + k;
    // Only a look-back that gave up (error bit already set) can place a key
    // outside the output; drop it rather than write out of bounds.
    if (out >= n) continue;
    keys_out[out] = kk;
    vals_out[out] = s_vals[k];
  }
}

// ---------------------------------------------------------------- one cluster
// Few keys: the whole sort is one kernel on one cluster of 16 CTAs, which hold the
// keys in their shared memory (CTA c has positions [c seg, (c + 1) seg)) from the
// first pass to the last. A pass reads its keys into registers, ranks them within the
// warp, exchanges the CTAs' digit counts over distributed shared memory, and stores
// each key straight into its new place, in whichever CTA that lies: two cluster
// barriers instead of a launch, a ticket, a look-back and a trip through L2 each.
// What bounds it: at a few thousand keys the barriers (12 us for 300 keys), beyond that
// 16 SMs' shared memory and ranking (0.3 us per 1,000 keys).
// Passes (clear and histogram with them) against one cluster, in us, of sorts in a row of
// keys in random order: u32 keys in four passes, 300 21 and 12; 5,000 27 and 13; 16,384 29
// and 17; 32,768 31 and 22; 50,000 33 and 26; 65,536 33 and 30. u64 keys in six, 5,000 39
// and 20; 16,384 43 and 29; 32,768 45 and 40; 40,000 47 and 44; 45,000 47 and 46; 50,000
// 47 and 48; 65,536 49 and 62. In eight, 5,000 52 and 26; 16,384 57 and 38; 32,768 60 and
// 54; 40,000 61 and 59; 45,000 62 and 63; 65,536 65 and 85. So u32 keys go to one cluster
// up to its room, u64 keys up to 43,000.
// 256 threads with the same room take as long, 1024 more (their bookkeeping); 8 CTAs 48
// us where 16 take 38 (50,000 keys); putting a CTA's keys in digit order first, so that
// its stores come in runs, changed nothing.
constexpr uint32_t CLUSTER = 16;
constexpr uint32_t CLUSTER_THREADS = 512, CLUSTER_WARPS = CLUSTER_THREADS / 32;
constexpr uint32_t CLUSTER_PARTS = CLUSTER_THREADS / RADIX;  // 2 threads share a digit's sums
constexpr int CLUSTER_ITEMS = 8;
constexpr uint32_t CLUSTER_ROOM = CLUSTER * CLUSTER_THREADS * CLUSTER_ITEMS;  // 65,536
template <int KW>
constexpr uint32_t CLUSTER_KEYS = KW == 1 ? CLUSTER_ROOM : 43'000;

template <int KW>
struct ClusterShared {
  static constexpr uint32_t ROOM = CLUSTER_THREADS * CLUSTER_ITEMS;
  // u32 keys: a key and its value in one word, which one store brings to its place.
  uint64_t keys[ROOM];
  uint32_t vals[KW == 2 ? ROOM : 4];
  alignas(16) uint16_t whist[CLUSTER_WARPS][RADIX];  // a warp's counts, then where its run of a digit begins in the CTA's
  uint16_t counts[CLUSTER][RADIX];           // every CTA's counts
  uint32_t match[CLUSTER_WARPS][2][RADIX];           // the lanes that have a digit; zero between rounds
  uint32_t part[2][CLUSTER_PARTS][RADIX];
  uint32_t base[RADIX];                      // the CTA's first place for a digit
  uint32_t tmp[RADIX / 32];
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// The address of this CTA's shared variable in CTA `cta` of the cluster.
__device__ __forceinline__ uint32_t remote(const void* p, uint32_t cta) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
  return a;
}
__device__ __forceinline__ void store_remote(uint32_t addr, uint16_t v) {
  asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t addr, uint64_t v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

template <int KW>
__global__ void __launch_bounds__(CLUSTER_THREADS, 1)
    sort_cluster_kernel(const typename KeyOf<KW>::type* keys_in, const uint32_t* vals_in,
                        typename KeyOf<KW>::type* keys_out, uint32_t* vals_out, uint32_t capacity,
                        const uint32_t* count, uint32_t passes, PassShifts shifts) {
  chain_begin();
  using K = typename KeyOf<KW>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  auto& s = *reinterpret_cast<ClusterShared<KW>*>(smem);
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = cluster_rank();
  const uint32_t n = count ? min(*count, capacity) : capacity;
  if (n == 0) return;  // in every CTA of the cluster
  const size_t segment = (size_t)(blockIdx.x / CLUSTER) * capacity;  // the cluster's
  keys_in += segment;
  vals_in += segment;
  keys_out += segment;
  vals_out += segment;
  cluster_arrive();    // nothing is stored in a CTA that has not started
  const uint32_t seg = ((n + CLUSTER - 1) / CLUSTER + 31) & ~31u;
  // pos / seg = pos * magic >> 32: magic is off by less than seg <= 2^12 parts in 2^32,
  // and pos < 2^16.
  const uint32_t magic = 0xffffffffu / seg + 1u;
  const uint32_t begin = cta * seg, mine = begin < n ? min(seg, n - begin) : 0u;
  // Warp w has keys [w * rounds * 32, (w + 1) * rounds * 32) of the segment, round j
  // reads 32 consecutive ones: order within the CTA is (warp, round, lane).
  const uint32_t rounds = (seg + CLUSTER_THREADS - 1) / CLUSTER_THREADS;
  const uint32_t first = warp * rounds * 32 + lane;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t digit = tid % RADIX, part = tid / RADIX;
  uint16_t* my_hist = s.whist[warp];

  for (uint32_t k = lane; k < 2 * RADIX; k += 32) s.match[warp][k / RADIX][k % RADIX] = 0;

  for (uint32_t p = 0; p < passes; p++) {
    const uint32_t shift = shifts.shift[p];
    K key[CLUSTER_ITEMS];
    uint32_t val[CLUSTER_ITEMS], rank[(CLUSTER_ITEMS + 1) / 2];
    reinterpret_cast<uint4*>(my_hist)[lane] = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < CLUSTER_ITEMS; j++) {
      const uint32_t at = first + j * 32;
      if (j < rounds && at < mine) {
        if (p == 0) {
          key[j] = keys_in[begin + at];
          val[j] = vals_in[begin + at];
        } else {
          key[j] = (K)s.keys[at];
          val[j] = KW == 1 ? (uint32_t)(s.keys[at] >> 32) : s.vals[at];
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < CLUSTER_ITEMS; j++) {
      if (j >= rounds) break;
      const bool valid = first + j * 32 < mine;
      const uint32_t d = valid ? (uint32_t)(key[j] >> shift) & (RADIX - 1) : 0u;
      uint32_t* m = s.match[warp][j & 1];
      if (valid) atomicOr(&m[d], 1u << lane);
      __syncwarp();
      const uint32_t peers = m[d], old = my_hist[d], before = __popc(peers & lt_mask);
      __syncwarp();
      if (valid && before == 0) {
        my_hist[d] = (uint16_t)(old + __popc(peers));
        m[d] = 0;
      }
      rank[j / 2] = j & 1 ? rank[j / 2] | (old + before) << 16 : old + before;
      __syncwarp();
    }
    __syncthreads();

    // Where each warp's run of a digit begins; the CTA's counts, sent to every CTA.
    // Thread (part, digit) has a share of the warps and of the CTAs.
    constexpr uint32_t PARTS = CLUSTER_PARTS, WP = CLUSTER_WARPS / PARTS, CP = CLUSTER / PARTS;
    uint32_t c[WP], sum = 0;
#pragma unroll
    for (uint32_t w = 0; w < WP; w++) {
      c[w] = s.whist[part * WP + w][digit];
      sum += c[w];
    }
    s.part[0][part][digit] = sum;
    __syncthreads();
    uint32_t running = 0, total = 0;
#pragma unroll
    for (uint32_t q = 0; q < PARTS; q++) {
      const uint32_t v = s.part[0][q][digit];
      running += q < part ? v : 0u;
      total += v;
    }
#pragma unroll
    for (uint32_t w = 0; w < WP; w++) {
      s.whist[part * WP + w][digit] = (uint16_t)running;
      running += c[w];
    }
    if (p == 0) cluster_wait();
#pragma unroll
    for (uint32_t k = 0; k < CP; k++)
      store_remote(remote(&s.counts[cta][digit], part * CP + k), (uint16_t)total);
    cluster_arrive();
    cluster_wait();

    // The first place of each digit of this CTA's: the keys of smaller digits, and
    // those of the same digit in CTAs before.
    uint32_t all = 0, before = 0;
#pragma unroll
    for (uint32_t k = 0; k < CP; k++) {
      const uint32_t v = s.counts[part * CP + k][digit];
      all += v;
      before += part * CP + k < cta ? v : 0u;
    }
    s.part[0][part][digit] = all;
    s.part[1][part][digit] = before;
    __syncthreads();
    uint32_t incl = 0;
    if (tid < RADIX) {
#pragma unroll
      for (uint32_t q = 1; q < PARTS; q++) {
        all += s.part[0][q][digit];
        before += s.part[1][q][digit];
      }
      incl = all;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
      }
      if (lane == 31) s.tmp[warp] = incl;
    }
    __syncthreads();
    if (tid < RADIX) {
#pragma unroll
      for (uint32_t w = 0; w < RADIX / 32; w++) before += w < warp ? s.tmp[w] : 0u;
      s.base[digit] = incl - all + before;
    }
    __syncthreads();

#pragma unroll
    for (int j = 0; j < CLUSTER_ITEMS; j++) {
      if (j >= rounds) break;
      if (first + j * 32 < mine) {
        const uint32_t d = (uint32_t)(key[j] >> shift) & (RADIX - 1);
        const uint32_t r = j & 1 ? rank[j / 2] >> 16 : rank[j / 2] & 0xffffu;
        const uint32_t pos = s.base[d] + my_hist[d] + r;
        const uint32_t to = __umulhi(pos, magic), at = pos - to * seg;
        if constexpr (KW == 1) {
          store_remote(remote(&s.keys[at], to), (uint64_t)val[j] << 32 | key[j]);
        } else {
          store_remote(remote(&s.keys[at], to), key[j]);
          store_remote(remote(&s.vals[at], to), val[j]);
        }
      }
    }
    cluster_arrive();
    cluster_wait();
  }
  for (uint32_t k = tid; k < mine; k += CLUSTER_THREADS) {
    keys_out[begin + k] = (K)s.keys[k];
    vals_out[begin + k] = KW == 1 ? (uint32_t)(s.keys[k] >> 32) : s.vals[k];
  }
}

template <int KW>
cudaLaunchConfig_t cluster_config(uint32_t clusters, cudaStream_t stream, cudaLaunchAttribute (&attrs)[2]) {
  attrs[0] = attrs[1] = {};
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = CLUSTER;
  attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as DG_CHAIN's
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = CLUSTER * clusters;
  config.blockDim = CLUSTER_THREADS;
  config.dynamicSmemBytes = sizeof(ClusterShared<KW>);
  config.stream = stream;
  config.attrs = attrs;
  config.numAttrs = 2;
  return config;
}

// The clusters that the device runs at once; 0 where it cannot run one.
template <int KW>
int cluster_init() {
  const auto kernel = sort_cluster_kernel<KW>;
  cudaLaunchAttribute attrs[2];
  const cudaLaunchConfig_t config = cluster_config<KW>(1, nullptr, attrs);
  int clusters = 0;
  const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)config.dynamicSmemBytes) == cudaSuccess &&
                  cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) == cudaSuccess;
  if (ok) return clusters;
  cudaGetLastError();
  return 0;
}

template <int KW>
dg_status cluster_launch(dg_context* ctx, const SortPlan& plan, void* keys, uint32_t* values, void* keys_alt,
                         uint32_t* values_alt, const uint32_t* count) {
  using K = typename KeyOf<KW>::type;
  PassShifts shifts{};
  for (uint32_t p = 0; p < plan.passes; p++) shifts.shift[p] = plan.shift[p];
  const bool odd = plan.passes & 1;
  cudaLaunchAttribute attrs[2];
  const cudaLaunchConfig_t config = cluster_config<KW>(plan.segments, ctx->stream, attrs);
  cudaError_t err = cudaSuccess;
  DG_LAUNCH(ctx, "sort_cluster",
            err = cudaLaunchKernelEx(&config, sort_cluster_kernel<KW>, static_cast<const K*>(keys),
                                     static_cast<const uint32_t*>(values), static_cast<K*>(odd ? keys_alt : keys),
                                     odd ? values_alt : values, plan.capacity, count, plan.passes, shifts));
  DG_CUDA(err);
  return DG_OK;
}

template <int KW, int ITEMS>
size_t pass_smem_bytes() {
  return SORT_TILE<ITEMS> * (sizeof(typename KeyOf<KW>::type) + 4) + (SORT_WARPS * RADIX + 2 * RADIX + 32) * 4;
}

template <int KW, int ITEMS>
dg_status pass_init() {
  DG_CUDA(cudaFuncSetAttribute(sort_pass_kernel<KW, 8, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)pass_smem_bytes<KW, ITEMS>()));
  DG_CUDA(cudaFuncSetAttribute(sort_pass_kernel<KW, 4, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)pass_smem_bytes<KW, ITEMS>()));
  return DG_OK;
}

struct ScratchLayout {
  size_t tickets, hist, status, total;
  uint32_t tile, max_tiles;  // keys per tile, tiles per segment
};

ScratchLayout layout_of(const SortPlan& plan) {
  ScratchLayout l;
  const bool few = (uint64_t)plan.capacity * plan.segments <= FEW_KEYS;
  l.tile = few ? SORT_TILE<SORT_ITEMS_FEW> : SORT_TILE<SORT_ITEMS>;
  l.max_tiles = std::max(1u, ceil_div(plan.capacity, l.tile));
  l.tickets = 0;
  l.hist = ((size_t)plan.segments * MAX_PASSES * 4 + 255) & ~(size_t)255;
  l.status = l.hist + (size_t)plan.segments * plan.passes * RADIX * 4;
  l.total = l.status + (size_t)plan.segments * plan.passes * l.max_tiles * RADIX * 4;
  return l;
}

template <int KW>
dg_status launch_typed(dg_context* ctx, const SortPlan& plan, void* keys, uint32_t* values, void* keys_alt,
                       uint32_t* values_alt, const uint32_t* count, void* scratch) {
  using K = typename KeyOf<KW>::type;
  // One cluster up to the sizes at which it still beats the passes (figures above
  // sort_cluster_kernel).
  if (plan.segments <= (uint32_t)ctx->sort_clusters && plan.capacity <= CLUSTER_KEYS<KW>)
    return cluster_launch<KW>(ctx, plan, keys, values, keys_alt, values_alt, count);
  ScratchLayout l = layout_of(plan);
  char* s = static_cast<char*>(scratch);
  auto* tickets = reinterpret_cast<uint32_t*>(s + l.tickets);
  auto* hist = reinterpret_cast<uint32_t*>(s + l.hist);
  auto* status = reinterpret_cast<uint32_t*>(s + l.status);
  DG_CUDA(cudaMemsetAsync(scratch, 0, l.total, ctx->stream));
  PassShifts shifts{};
  for (uint32_t p = 0; p < plan.passes; p++) shifts.shift[p] = plan.shift[p];
  uint32_t hist_blocks =
      std::min<uint32_t>(ceil_div(plan.capacity, HIST_THREADS * HIST_ITEMS * DG_HIST_ROUNDS), (uint32_t)ctx->sm_count * 8);
  hist_blocks = std::max(1u, std::min(hist_blocks, ceil_div((uint32_t)ctx->sm_count * 8, plan.segments)));
  const SegmentStates states{plan.passes * RADIX, plan.passes * l.max_tiles * RADIX};
  DG_CHAIN(ctx, "sort_histogram", (sort_histogram_kernel<KW>), dim3(hist_blocks, plan.segments), HIST_THREADS, 0,
           static_cast<const K*>(keys), plan.capacity, count, plan.passes, shifts, hist);
  const bool few = l.tile == SORT_TILE<SORT_ITEMS_FEW>;
  const size_t smem = few ? pass_smem_bytes<KW, SORT_ITEMS_FEW>() : pass_smem_bytes<KW, SORT_ITEMS>();
  K* in_k = static_cast<K*>(keys);
  uint32_t* in_v = values;
  K* out_k = static_cast<K*>(keys_alt);
  uint32_t* out_v = values_alt;
  for (uint32_t p = 0; p < plan.passes; p++) {
    const bool narrow = plan.narrow_last && p + 1 == plan.passes;
    const auto kernel = few ? (narrow ? sort_pass_kernel<KW, 4, SORT_ITEMS_FEW> : sort_pass_kernel<KW, 8, SORT_ITEMS_FEW>)
                            : (narrow ? sort_pass_kernel<KW, 4, SORT_ITEMS> : sort_pass_kernel<KW, 8, SORT_ITEMS>);
    DG_CHAIN(ctx, "sort_pass", (kernel), dim3(l.max_tiles, plan.segments), SORT_THREADS, smem,
             in_k, in_v, out_k, out_v, plan.capacity, count, shifts.shift[p], hist + p * RADIX,
             status + (size_t)p * l.max_tiles * RADIX, tickets + p, states, ctx->device_error);
    std::swap(in_k, out_k);
    std::swap(in_v, out_v);
  }
  return DG_OK;
}

}  // namespace

dg_status sort_init(dg_context* ctx) {
  // A device without 16 SMs in one GPC (a partition of one) sorts by passes.
  ctx->sort_clusters = std::min(cluster_init<1>(), cluster_init<2>());
  // The pass kernels use more than the default 48 KB of dynamic shared memory.
  DG_TRY((pass_init<1, SORT_ITEMS>()));
  DG_TRY((pass_init<2, SORT_ITEMS>()));
  DG_TRY((pass_init<1, SORT_ITEMS_FEW>()));
  DG_TRY((pass_init<2, SORT_ITEMS_FEW>()));
  return DG_OK;
}

SortPlan sort_plan(uint32_t capacity, uint32_t high_bits) {
  SortPlan p{};
  p.capacity = capacity;
  p.key_words = high_bits > 0 ? 2 : 1;
  p.high_bits = high_bits;
  p.passes = 4 + 2 * ((high_bits + 15) / 16);
  for (uint32_t k = 0; k < p.passes; k++) p.shift[k] = k < 4 ? k * 8 : 32 + (k - 4) * 8;
  return p;
}

SortPlan sort_plan_low_bits(uint32_t capacity, uint32_t bits) {
  SortPlan p{};
  p.capacity = capacity;
  p.key_words = 1;
  p.high_bits = 0;
  p.passes = 2 * ((bits + 15) / 16);
  for (uint32_t k = 0; k < p.passes; k++) p.shift[k] = k * 8;
  return p;
}

SortPlan sort_plan_digits(uint32_t capacity, uint32_t key_words, uint32_t bits) {
  SortPlan p{};
  p.capacity = capacity;
  p.key_words = key_words;
  p.high_bits = key_words == 2 ? bits : 0;
  p.passes = key_words == 2 ? 4 + (bits + 7) / 8 : std::max(1u, (bits + 7) / 8);
  for (uint32_t k = 0; k < p.passes; k++) p.shift[k] = k * 8;
  sort_plan_key_bits(p, key_words == 2 ? 32 + bits : bits);
  return p;
}

void sort_plan_key_bits(SortPlan& p, uint32_t bits) {
  // The last pass's digit: bits [shift, shift + 8) of the key; only `bits` vary.
  const uint32_t last = p.shift[p.passes - 1];
  p.narrow_last = bits <= last + 4;
}

size_t sort_scratch_bytes(const SortPlan& plan) { return layout_of(plan).total; }

dg_status sort_launch(dg_context* ctx, const SortPlan& plan, void* keys, uint32_t* values, void* keys_alt,
                      uint32_t* values_alt, const uint32_t* count, void* scratch) {
  if (plan.key_words == 2)
    return launch_typed<2>(ctx, plan, keys, values, keys_alt, values_alt, count, scratch);
  return launch_typed<1>(ctx, plan, keys, values, keys_alt, values_alt, count, scratch);
}

}  // namespace dg

using namespace dg;

struct dg_radix_sort {
  dg_context* ctx;
  SortPlan plan;
  dg_buffer* keys;
  dg_buffer* values;
  dg_buffer* keys_alt;
  dg_buffer* values_alt;
  dg_buffer* scratch;
  dg_buffer* count;  // borrowed, may be NULL
};

extern "C" {

dg_status dg_radix_sort_create(dg_context* ctx, uint32_t capacity, uint32_t high_bits, dg_buffer* count,
                               dg_radix_sort** out) {
  DG_REQUIRE(ctx && out, "NULL argument");
  DG_REQUIRE(high_bits <= 32, "high_bits is at most 32");
  DG_REQUIRE(capacity < (1u << 30), "capacity must be below 2^30 keys");
  DG_REQUIRE(!count || count->bytes >= 4, "count buffer too small");
  auto* s = new dg_radix_sort{ctx, sort_plan(capacity, high_bits), nullptr, nullptr, nullptr, nullptr, nullptr, count};
  size_t kb = (size_t)capacity * (high_bits > 0 ? 8 : 4);
  dg_status st = alloc_buffer(ctx, kb, &s->keys);
  if (st == DG_OK) st = alloc_buffer(ctx, (size_t)capacity * 4, &s->values);
  if (st == DG_OK) st = alloc_buffer(ctx, kb, &s->keys_alt);
  if (st == DG_OK) st = alloc_buffer(ctx, (size_t)capacity * 4, &s->values_alt);
  if (st == DG_OK) st = alloc_buffer(ctx, sort_scratch_bytes(s->plan), &s->scratch);
  if (st != DG_OK) {
    dg_radix_sort_destroy(s);
    return st;
  }
  *out = s;
  return DG_OK;
}

dg_buffer* dg_radix_sort_keys(dg_radix_sort* s) { return s ? s->keys : nullptr; }
dg_buffer* dg_radix_sort_values(dg_radix_sort* s) { return s ? s->values : nullptr; }
uint32_t dg_radix_sort_capacity(const dg_radix_sort* s) { return s ? s->plan.capacity : 0; }

dg_status dg_radix_sort_encode(dg_radix_sort* s) {
  DG_REQUIRE(s, "NULL argument");
  return sort_launch(s->ctx, s->plan, s->keys->ptr, typed<uint32_t>(s->values), s->keys_alt->ptr,
                     typed<uint32_t>(s->values_alt), s->count ? typed<uint32_t>(s->count) : nullptr, s->scratch->ptr);
}

dg_status dg_radix_sort_destroy(dg_radix_sort* s) {
  if (!s) return DG_OK;
  free_buffer(s->keys);
  free_buffer(s->values);
  free_buffer(s->keys_alt);
  free_buffer(s->values_alt);
  free_buffer(s->scratch);
  delete s;
  return DG_OK;
}

}  // extern "C"
