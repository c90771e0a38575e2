// The renderer's backward passes: the blend's (src/shaders/rasterizeBackward.wgsl)
// and the preprocess's (src/shaders/preprocessBackward.wgsl).
//
// Compiled with the default --fmad=true: gradients only need to agree to rounding
// (their tile sums meet through float atomics anyway). The arithmetic that decides
// which splats a pixel blended (blend_power_negated, exp_blend_negated, the alpha product and its
// thresholds) is written with non-fusing intrinsics or explicit fmaf, so it makes
// exactly the forward pass's decisions.
#include "dg_adam.cuh"
#include "dg_render.cuh"
#include "dg_render_kernels.cuh"

#include <algorithm>
#include <type_traits>

namespace dg {
namespace {

__device__ __forceinline__ void load_camera(Camera& dst, const Camera* src) {
  const float* s = reinterpret_cast<const float*>(src);
  float* d = reinterpret_cast<float*>(&dst);
  for (int k = threadIdx.x; k < 36; k += blockDim.x) d[k] = s[k];
}

// A pixel's state on its back-to-front walk: the transmittance in front of the
// current splat, the colour composited behind it and the last splat passed.
struct PixelBackward {
  float T, pgx, pgy, pgz, tf_bg;  // tf_bg: the final T times (background . pixel gradient)
  float bhx, bhy, bhz;  // colour of everything behind
  float na, ncx, ncy, ncz;

  // Starts the walk at a point where the transmittance is T0 and the colour
  // composited behind, relative to T0, is `behind`.
  __device__ __forceinline__ void begin(float final_T, float T0, float3 behind, float gx, float gy, float gz,
                                        float4 bg) {
    T = T0;
    pgx = gx;
    pgy = gy;
    pgz = gz;
    tf_bg = final_T * (bg.x * gx + bg.y * gy + bg.z * gz);
    bhx = behind.x;
    bhy = behind.y;
    bhz = behind.z;
    na = ncx = ncy = ncz = 0.0f;
  }

  // Steps in front of a splat of this alpha and colour (alpha 0 and a finite colour: one
  // that the pixel did not blend, which changes nothing) and returns the gradient of its alpha.
  __device__ __forceinline__ float step(float alpha, float4 c) {
    // 1 / (1 - alpha), used twice; the approximate reciprocal (~1 ulp) is plenty:
    // a chunk's chain of divisions is at most CHUNK entries long.
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(1.0f - alpha));
    T = T * inv;
    // The colour behind, na nc + (1 - na) bh, as bh + na (nc - bh).
    bhx = fmaf(na, ncx - bhx, bhx);
    bhy = fmaf(na, ncy - bhy, bhy);
    bhz = fmaf(na, ncz - bhz, bhz);
    na = alpha;
    ncx = c.x;
    ncy = c.y;
    ncz = c.z;
    const float dotv = (c.x - bhx) * pgx + (c.y - bhy) * pgy + (c.z - bhz) * pgz;
    return T * dotv - inv * tf_bg;
  }
};

// Per-warp shared memory of the backward blend.
constexpr uint32_t BATCH = 32, HALF_BATCH = BATCH / 2;
constexpr uint32_t SHARE_ROW = 34;  // 32 pixels, and rows that begin two banks apart
struct BackStage {
  BlendPair pair[BATCH / 2];
  float4 color[BATCH];
  uint32_t pos[BATCH];    // position in the tile's list
  uint32_t index[BATCH];  // splat
  // Per pixel (pixel p at place 2 (p % 16) + p / 16: p and p + 16 side by side, as
  // packed instructions take them): its gradients, and half a batch's shares: the
  // gradients of the powers and of the opacities, and alpha T.
  float grad[3][32];
  float share[3][HALF_BATCH][SHARE_ROW];
  uint16_t list[CHUNK];  // the chunk's entries some pixel of the block blended, back to front
};

// The 9 gradients of half a batch's splats from the shares: lane l sums splat l % 16
// over the pixels p with p % 2 = l / 16, both lanes' sums meet, and they go to the
// splat's global gradients, one atomic add each. The sums run in the order of a
// butterfly over the block's pixels (p + 16 first, p + 1 last). Pixel p is at
// (corner_x + p % 8, corner_y + p / 8).
__device__ __forceinline__ void add_gradients(const BackStage& st, uint32_t first, uint32_t n, uint32_t lane,
                                              float corner_x, float corner_y, float* splat_grads) {
  const uint32_t s = lane & 15u, h = lane >> 4, e = first + s;
  const float* f = reinterpret_cast<const float*>(&st.pair[e / 2]) + (e & 1u);
  const float nx = f[0], ny = f[2], a = 2.0f * f[4], b = f[6], c = 2.0f * f[8];  // conic (a, b, c)
  const F2 a2 = f2(a, a), b2 = f2(b, b), c2 = f2(c, c);
  constexpr int N = SPLAT_GRADS;
  // Pixels p = 2 k + h and p + 16.
  auto leaf = [&](uint32_t k, float (&out)[N]) {
    const uint32_t at = 2u * (2u * k + h);
    auto two = [&](const float* row) { return f2_load(reinterpret_cast<const float2*>(row + at)); };
    const F2 pg = two(st.share[0][s]), og = two(st.share[1][s]), wt = two(st.share[2][s]);
    const float dx = (corner_x + (float)(2u * k % 8u + h)) + nx, y = corner_y + (float)(2u * k / 8u);
    const F2 dx2 = f2(dx, dx), dy2 = f2(y + ny, (y + 2.0f) + ny);
    const F2 pdx = f2_mul(pg, dx2), pdy = f2_mul(pg, dy2);
    // The power's gradient is -(a dx + b dy, b dx + c dy) for the pixel's offset and
    // (-dx^2 / 2, -dx dy, -dy^2 / 2) for the conic (factors without a rounding later).
    const F2 v[N] = {f2_fma(b2, pdy, f2_mul(a2, pdx)),
                     f2_fma(b2, pdx, f2_mul(c2, pdy)),
                     f2_mul(pdx, dx2),
                     f2_mul(pdx, dy2),
                     f2_mul(pdy, dy2),
                     og,
                     f2_mul(wt, two(st.grad[0])),
                     f2_mul(wt, two(st.grad[1])),
                     f2_mul(wt, two(st.grad[2]))};
#pragma unroll
    for (int i = 0; i < N; i++) out[i] = __fadd_rn(f2_lo(v[i]), f2_hi(v[i]));
  };
  auto add = [](float (&x)[N], const float (&y)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++) x[i] = __fadd_rn(x[i], y[i]);
  };
  float sum[N], odd[N], l[N], m[N];
  leaf(0, sum), leaf(4, l), add(sum, l);
  leaf(2, m), leaf(6, l), add(m, l), add(sum, m);
  leaf(1, odd), leaf(5, l), add(odd, l);
  leaf(3, m), leaf(7, l), add(m, l), add(odd, m);
  add(sum, odd);
#pragma unroll
  for (int i = 0; i < N; i++) sum[i] = __fadd_rn(sum[i], __shfl_xor_sync(0xffffffffu, sum[i], 16));
  if (s >= n) return;
  sum[2] *= -0.5f;
  sum[3] = -sum[3];
  sum[4] *= -0.5f;
  float* out = splat_grads + (size_t)st.index[e] * SPLAT_GRADS;
#pragma unroll
  for (int i = 0; i < N; i++)
    if ((i < 5) == (h == 0) && sum[i] != 0.0f) atomicAdd(out + i, sum[i]);
}

// The items of rasterize_backward_kernel, and the splats' gradients cleared for it: for
// each tile the chunks that some block of it walked, chunk by chunk with the blocks of one
// beside each other, tiles of several chunks before those of one. The order decides nothing
// but in which one the blocks' sums of a splat meet, and so the last bits of its gradients;
// the blocks of a chunk run together. (With the chunks listed block by block as the forward
// pass ended, the longest first, the blend took 149 us for 1.1M splats at 980x545 and 79
// for 100k, this way 159 and 84. But where a gradient is 0 but for rounding, a first step
// of Adam turns its sign into a whole step, and the sums that met in another order changed
// more of those: of 1.6M gradients of a step of 100k splats 57 differ by over a thousandth
// between a run of that order and one of this, 50 between two runs of this.) A warp per
// tile, one atomic per CTA and class.
constexpr uint32_t LIST_THREADS = 256, LIST_WARPS = LIST_THREADS / 32;

__global__ void __launch_bounds__(LIST_THREADS) list_items_kernel(const uint2* ranges, const uint32_t* walked,
                                                                  uint32_t* plan, uint2* items, uint32_t item_room,
                                                                  float* splat_grads, size_t floats) {
  chain_begin();
  const size_t i = (size_t)blockIdx.x * LIST_THREADS + threadIdx.x, step = (size_t)gridDim.x * LIST_THREADS;
  const size_t vecs = (reinterpret_cast<uintptr_t>(splat_grads) & 15) == 0 ? floats / 4 : 0;
  for (size_t k = i; k < vecs; k += step) reinterpret_cast<float4*>(splat_grads)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (size_t k = 4 * vecs + i; k < floats; k += step) splat_grads[k] = 0.0f;
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u, block = lane & 7u;
  const uint32_t tiles = plan[PLAN_TILES];
  __shared__ uint32_t s_total[LIST_WARPS], s_at[LIST_WARPS];
  const uint32_t warp = threadIdx.x >> 5;
  for (uint32_t first = blockIdx.x * LIST_WARPS; first < tiles; first += gridDim.x * LIST_WARPS) {
    const uint32_t tile = first + warp;
    uint32_t chunks = 0, total = 0, several = 0;
    if (tile < tiles) {
      const uint2 run = ranges[tile];
      chunks = (walked[tile * 8u + block] + CHUNK - 1u) / CHUNK;
      total = __reduce_add_sync(0xffffffffu, lane < 8u ? chunks : 0u);
      several = run.y - run.x > CHUNK;
    }
    // One atomic per class for the CTA's tiles.
    if (lane == 0) s_total[warp] = total << 1 | several;
    __syncthreads();
    if (warp < ITEM_CLASSES) {
      const uint32_t has = lane < LIST_WARPS ? s_total[lane] : 0u, n = (has & 1u) != warp ? has >> 1 : 0u;
      uint32_t incl = n;
#pragma unroll
      for (uint32_t d = 1; d < LIST_WARPS; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
      }
      uint32_t base = 0;
      if (lane == LIST_WARPS - 1u && incl) base = atomicAdd(plan + PLAN_ITEMS + warp, incl);
      base = __shfl_sync(0xffffffffu, base, LIST_WARPS - 1);
      if (n) s_at[lane] = base + incl - n;
    }
    __syncthreads();
    uint32_t at = s_at[warp];
    uint2* out = items + (several ? 0 : (size_t)item_room);
    const uint32_t most = __reduce_max_sync(0xffffffffu, chunks);
    for (uint32_t k0 = 0; k0 < most; k0 += 4u) {  // lane (k, block): chunk k0 + k
      const uint32_t k = k0 + (lane >> 3);
      const uint32_t listed = __ballot_sync(0xffffffffu, k < chunks), to = at + __popc(listed & below);
      if (k < chunks && to < item_room) out[to] = make_uint2(tile * 8u + block, k);
      at += __popc(listed);
    }
  }
}

// src/shaders/rasterizeBackward.wgsl:50-163. The work is split into independent
// items, one per (tile, CHUNK-entry chunk of its list, 8x4 pixel block), taken by
// persistent warps from a counter in list_items_kernel's order, so no warp waits for
// another and a long list is spread over many warps. For an item, the warp lists the
// chunk's entries that some pixel of its block blended in the forward pass (the
// forward's blend mask), back to front, and takes 32 of them at a time; the records of
// the next 32 are loaded meanwhile. Each pixel
// starts from its state behind the chunk: the transmittance the forward pass saved
// at the chunk's end, and the colour behind it, (final colour - colour saved) /
// that transmittance; behind its last splat (the whole list for most tiles) these
// are the final transmittance and nothing. The alphas of four splats are computed
// together, then each pixel recovers the transmittance in front of each splat by
// dividing by (1 - alpha), in list order, and leaves three numbers per splat in shared
// memory; after 16 splats the lanes change over from pixels to splats and sum them
// (add_gradients).
//
// What bounds it: on large frames instructions and shared memory, on small ones the
// longest items (512 entries, 20 us and more for one warp) and an item's first loads (a
// chain of eight, 3 us). Summing 9 shares over the pixels took most of it: with a
// reduce-scatter over the warp per two splats (18 shares, 20 shuffles and as many
// selects and adds) 280 us for 1.1M splats at 980x545, 147 for 100k, 122 for 201k at
// 489x273, 38 for 5k at 251x187; this way, in the same order of additions, 179 | 92 |
// 65 | 21. Items only for what the forward pass walked: 159 | 84 | 62 | 21.5. With the
// longest items first, 5 and 6 CTAs per SM took 155 | 83 | 65 and 167 | 88 | 66 against
// 152 | 80 | 61 with 4; the groups of 4 unrolled
// 2 or 4 times the same. Chunks of 256 entries 140 | 75 | 45 | 18, and the shares' sums
// as moments about the block's center 20% less, but both round otherwise, and a first
// step of Adam turns a gradient's last bits into the sign of a whole step where it is 0
// but for rounding.
__global__ void __launch_bounds__(BWD_THREADS, 4) rasterize_backward_kernel(
    const Camera* camera, const float4* raster_params, const float* splats,
    const uint32_t* pair_splats, const uint2* ranges, uint32_t* plan,
    const uint2* item_list, uint32_t item_room, const float4* pixel_color, const uint32_t* pixel_last,
    const float4* checkpoints, const uint32_t* blend_mask,
    const float4* pixel_grads, float* splat_grads, uint32_t* work_counter,
    bool cut_in_record) {
  chain_begin();
  __shared__ BackStage stages[BWD_WARPS];
  const uint32_t lane = threadIdx.x & 31u;
  BackStage& st = stages[threadIdx.x >> 5];
  const float vpx = camera->viewport[0], vpy = camera->viewport[1];
  const uint32_t tiles_x = ((uint32_t)vpx + TILE - 1u) / TILE;
  const uint32_t tiles = plan[PLAN_TILES];
  uint32_t up_to[ITEM_CLASSES], items = 0;  // the items up to each class
#pragma unroll
  for (uint32_t k = 0; k < ITEM_CLASSES; k++) up_to[k] = items += min(plan[PLAN_ITEMS + k], item_room);
  const float4 bg = raster_params[0];
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(work_counter, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= items) break;
    size_t at = item;
#pragma unroll
    for (uint32_t k = 1; k < ITEM_CLASSES; k++)
      if (item >= up_to[k - 1]) at = (size_t)k * item_room + item - up_to[k - 1];
    const uint2 it = item_list[at];
    const uint32_t tile = it.x >> 3, block = it.x & 7u, chunk = it.y;
    const uint32_t bx = (tile % tiles_x) * TILE + (block & 1u) * 8u, by = (tile / tiles_x) * TILE + (block >> 1) * 4u;
    const uint32_t px = bx + (lane & 7u), py = by + (lane >> 3);
    const bool inside = (float)px < vpx && (float)py < vpy;
    const uint2 run = ranges[tile];
    const uint32_t chunk_lo = run.x + chunk * CHUNK, chunk_hi = min(chunk_lo + CHUNK, run.y);
    const uint32_t boundary = (chunk + 1u) * CHUNK;  // the chunk's end, relative to run.x
    // Lane k's mask word, of window k of the chunk; those past the walk hold anything.
    static_assert(CHUNK / 32 <= 32, "a chunk's mask words fit in the warp's lanes");
    uint32_t word = 0;
    if (chunk_lo + lane * 32u < chunk_hi)
      word = blend_mask[mask_at(tile, tiles, run.x, chunk * (CHUNK / 32u) + lane, block)];
    float4 color = make_float4(0.f, 0.f, 0.f, 0.f), pg = color;
    uint32_t last = 0;
    if (inside) {
      const uint32_t p = py * (uint32_t)vpx + px;
      color = pixel_color[p];
      last = pixel_last[p];
      pg = pixel_grads[p];
    }
    // Splats at or past the warp's largest `last` contribute nothing to it.
    const uint32_t end_all = min(chunk_hi, run.x + __reduce_max_sync(0xffffffffu, last));
    if (end_all <= chunk_lo) continue;
    // The chunk's blended entries: lane k has those of window k, and counts those behind it.
    const uint32_t windows = (end_all - chunk_lo + 31u) / 32u;
    if (lane >= windows) word = 0;
    const uint32_t left = end_all - chunk_lo - lane * 32u;
    if (lane < windows && left < 32u) word &= (1u << left) - 1u;
    uint32_t behind_it = __popc(word);
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_down_sync(0xffffffffu, behind_it, d);
      if (lane + d < 32u) behind_it += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, behind_it, 0);
    if (total == 0) continue;
    behind_it -= __popc(word);
    for (uint32_t k = 0; k < windows; k++) {
      const uint32_t bits = __shfl_sync(0xffffffffu, word, k), at = __shfl_sync(0xffffffffu, behind_it, k);
      if ((bits >> lane) & 1u) st.list[at + __popc(bits >> lane) - 1u] = (uint16_t)(k * 32u + lane);
    }
    const uint32_t place = 2u * (lane & 15u) + (lane >> 4);
    st.grad[0][place] = pg.x;
    st.grad[1][place] = pg.y;
    st.grad[2][place] = pg.z;
    __syncwarp();
    float T0 = color.w;
    float3 behind = make_float3(0.f, 0.f, 0.f);
    if (last > boundary) {  // the pixel blends splats behind this chunk
      const float4 ck = checkpoints[checkpoint_at(run.x, chunk + 1u, block, lane)];
      const float inv = 1.0f / ck.x;
      T0 = ck.x;
      behind = make_float3((color.x - color.w * bg.x - ck.y) * inv, (color.y - color.w * bg.y - ck.z) * inv,
                           (color.z - color.w * bg.z - ck.w) * inv);
    }
    PixelBackward pb;
    pb.begin(color.w, T0, behind, pg.x, pg.y, pg.z, bg);
    const F2 cx = f2((float)px + 0.5f, (float)px + 0.5f), cy = f2((float)py + 0.5f, (float)py + 0.5f);
    // This lane's entry of the next batch, and the splat of the one after.
    auto entry = [&](uint32_t k) { return k < total ? (uint32_t)st.list[k] : 0u; };
    SplatRecord raw;
    uint32_t index = lane < total ? pair_splats[chunk_lo + entry(lane)] : 0u;
    raw.load(splats, index, lane < total);
    uint32_t next_index = BATCH + lane < total ? pair_splats[chunk_lo + entry(BATCH + lane)] : 0u;
    for (uint32_t first = 0; first < total; first += BATCH) {
      const uint32_t staged = min(BATCH, total - first);
      float* e = reinterpret_cast<float*>(&st.pair[lane / 2]) + (lane & 1u);
      if (lane < staged) {
        stage_entry(e, raw, cut_in_record ? raw.s1.w : blend_cutoff(raw.s2.w));
        st.color[lane] = raw.s2;
        st.pos[lane] = chunk * CHUNK + entry(first + lane);
        st.index[lane] = index;
      } else {
        e[10] = 0.0f;  // nothing is below it
      }
      // A colour that is not finite must not reach a pixel that does not blend its splat,
      // where step() would multiply it by 0. Batches with one have a loop of their own (1%
      // of the pass; as a select in the one loop 2.4%).
      const bool endless = __any_sync(
          0xffffffffu, lane < staged && !(fabsf(raw.s2.x) + fabsf(raw.s2.y) + fabsf(raw.s2.z) < INFINITY));
      __syncwarp();
      index = next_index;
      raw.load(splats, index, first + BATCH + lane < total);
      const uint32_t ahead = first + 2 * BATCH + lane;
      next_index = ahead < total ? pair_splats[chunk_lo + entry(ahead)] : 0u;
#pragma unroll 1
      for (uint32_t half = 0; half < staged; half += HALF_BATCH) {
        const uint32_t n = min(HALF_BATCH, staged - half);
        auto walk = [&](auto endless_batch) {
          constexpr bool ENDLESS = decltype(endless_batch)::value;
#pragma unroll 1
          for (uint32_t j = 0; j < n; j += 4) {
            const uint4 pos = *reinterpret_cast<const uint4*>(&st.pos[half + j]);
            bool has[4] = {pos.x < last, pos.y < last, pos.z < last, pos.w < last};
            float alpha[4], G[4];
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {
              const BlendPair& pr = st.pair[(half + j) / 2 + h];
              F2 limit;
              const F2 q = blend_power_negated(pr, cx, cy, limit);
              has[2 * h] = has[2 * h] && __float_as_uint(f2_lo(q)) < __float_as_uint(f2_lo(limit));
              has[2 * h + 1] = has[2 * h + 1] && __float_as_uint(f2_hi(q)) < __float_as_uint(f2_hi(limit));
              // Any value may come out where the limit was not kept.
              const F2 ex = exp_blend_negated(q), al = f2_mul(F2{pr.opacity}, ex);
              G[2 * h] = f2_lo(ex);
              G[2 * h + 1] = f2_hi(ex);
              alpha[2 * h] = fminf(0.99f, f2_lo(al));
              alpha[2 * h + 1] = fminf(0.99f, f2_hi(al));
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
              has[u] = has[u] && alpha[u] >= 1.0f / 255.0f;
              const float al = has[u] ? alpha[u] : 0.0f;
              float4 c = st.color[half + j + u];
              if (ENDLESS && !has[u]) c.x = c.y = c.z = 0.0f;
              const float alpha_grad = pb.step(al, c);
              st.share[0][j + u][place] = has[u] ? alpha_grad * c.w * G[u] : 0.0f;
              st.share[1][j + u][place] = has[u] ? alpha_grad * G[u] : 0.0f;
              st.share[2][j + u][place] = al * pb.T;
            }
          }
        };
        if (endless)
          walk(std::true_type{});
        else
          walk(std::false_type{});
        __syncwarp();
        add_gradients(st, half, n, lane, (float)bx + 0.5f, (float)by + 0.5f, splat_grads);
        __syncwarp();
      }
    }
    __syncwarp();
  }
  // The last warp leaves the counters as it found them, for the next pass.
  if (lane == 0 && atomicAdd(work_counter + 1, 1u) == gridDim.x * BWD_WARPS - 1u) {
    work_counter[0] = 0;
    work_counter[1] = 0;
#pragma unroll
    for (uint32_t k = 0; k < ITEM_CLASSES; k++) plan[PLAN_ITEMS + k] = 0;
  }
}

#ifndef DG_PBWD_THREADS
#define DG_PBWD_THREADS 128
#endif
constexpr uint32_t PBWD_THREADS = DG_PBWD_THREADS;  // a multiple of 32

// Copies n floats between global and shared memory, 16 bytes at a time where both
// ends allow it; all threads of the CTA take part.
__device__ __forceinline__ void copy_floats(float* dst, const float* src, uint32_t n) {
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
    const uint32_t vecs = n / 4;
    for (uint32_t k = threadIdx.x; k < vecs; k += blockDim.x)
      reinterpret_cast<float4*>(dst)[k] = reinterpret_cast<const float4*>(src)[k];
    for (uint32_t k = vecs * 4 + threadIdx.x; k < n; k += blockDim.x) dst[k] = src[k];
  } else {
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) dst[k] = src[k];
  }
}

// src/shaders/preprocessBackward.wgsl:28-181 for one Gaussian: the 16-float
// Gaussian gradient (slots 7 and 15 zero) to out, and the 45 SH gradients over
// its 45 SH coefficients in shv (shared memory).
// gaussian: the Gaussian's 16 activated floats (16-byte aligned); radius: its
// splat's radius (0 when it was not drawn); grads: its 9 splat gradients. shv
// holds its SH coefficients and receives their gradients.
__device__ __forceinline__ void preprocess_backward_one(const Camera& cam, const float* gaussian,
                                                        float* shv, uint32_t basis_count, float radius,
                                                        const float* grads, float (&out)[16]) {
#pragma unroll
  for (int k = 0; k < 16; k++) out[k] = 0.0f;
  if (radius == 0.0f) {
    for (uint32_t k = 0; k < SH_REST_FLOATS; k++) shv[k] = 0.0f;
    return;
  }
  float grad[9];
#pragma unroll
  for (int k = 0; k < 9; k++) grad[k] = grads[k];
  float g[16];
  {
    const float4* gp = reinterpret_cast<const float4*>(gaussian);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      float4 q = gp[k];
      g[4 * k] = q.x; g[4 * k + 1] = q.y; g[4 * k + 2] = q.z; g[4 * k + 3] = q.w;
    }
  }
  Projection p;
  project(cam, g, p);
  const float depth = p.depth;
  const float ratio0 = p.t[0] / depth, ratio1 = p.t[1] / depth;
  const float free0 = fabsf(ratio0) > p.limit[0] ? 0.0f : 1.0f;
  const float free1 = fabsf(ratio1) > p.limit[1] ? 0.0f : 1.0f;
  const float depth2 = depth * depth, depth3 = depth2 * depth;
  const float a = p.a, b = p.b, c = p.c, det = p.det;
  // 1. conic -> 2D covariance
  const float det2 = det * det;
  const float a_grad = (-c * c * grad[2] + b * c * grad[3] - b * b * grad[4]) / det2;
  const float b_grad = (2.0f * b * c * grad[2] - (det + 2.0f * b * b) * grad[3] + 2.0f * a * b * grad[4]) / det2;
  const float c_grad = (-b * b * grad[2] + a * b * grad[3] - a * a * grad[4]) / det2;
  const float G2[2][2] = {{a_grad, 0.5f * b_grad}, {0.5f * b_grad, c_grad}};
  // 2. Σ' = T Σ Tᵀ with T = J W
  float Gjw[3][2];
#pragma unroll
  for (int col = 0; col < 3; col++)
#pragma unroll
    for (int row = 0; row < 2; row++) {
      float v = G2[0][row] * p.jw[col][0];
      v = v + G2[1][row] * p.jw[col][1];
      Gjw[col][row] = v;
    }
  float cov3d_grad[3][3];
#pragma unroll
  for (int col = 0; col < 3; col++)
#pragma unroll
    for (int row = 0; row < 3; row++) {
      float v = p.jw[row][0] * Gjw[col][0];
      v = v + p.jw[row][1] * Gjw[col][1];
      cov3d_grad[col][row] = v;
    }
  float t3[3][2];
#pragma unroll
  for (int col = 0; col < 3; col++)
#pragma unroll
    for (int row = 0; row < 2; row++) {
      float v = (2.0f * Gjw[0][row]) * p.cov3d[col][0];
      v = v + (2.0f * Gjw[1][row]) * p.cov3d[col][1];
      v = v + (2.0f * Gjw[2][row]) * p.cov3d[col][2];
      t3[col][row] = v;
    }
  float jg[3][2];
#pragma unroll
  for (int col = 0; col < 3; col++)
#pragma unroll
    for (int row = 0; row < 2; row++) {
      float v = t3[0][row] * p.w[0][col];
      v = v + t3[1][row] * p.w[1][col];
      v = v + t3[2][row] * p.w[2][col];
      jg[col][row] = v;
    }
  // 3. J moves with t
  float tg[3];
  tg[0] = jg[2][0] * free0 * p.focal[0] / depth2;
  tg[1] = jg[2][1] * free1 * -p.focal[1] / depth2;
  tg[2] = 0.0f;
  const float depth_grad = jg[0][0] * (-p.focal[0] / depth2) + jg[1][1] * (p.focal[1] / depth2) +
                           jg[2][0] * (-(1.0f + free0) * p.focal[0] * p.tx / depth3) +
                           jg[2][1] * ((1.0f + free1) * p.focal[1] * p.ty / depth3);
  tg[2] = tg[2] - depth_grad;
  // 4. the 2D center
  float clip[4];
#pragma unroll
  for (int row = 0; row < 4; row++) {
    float v = cam.proj[0 * 4 + row] * p.t[0];
    v = v + cam.proj[1 * 4 + row] * p.t[1];
    v = v + cam.proj[2 * 4 + row] * p.t[2];
    v = v + cam.proj[3 * 4 + row] * 1.0f;
    clip[row] = v;
  }
  const float ng0 = grad[0] * 0.5f * cam.viewport[0], ng1 = grad[1] * -0.5f * cam.viewport[1];
  float ndc_dot = ng0 * clip[0];
  ndc_dot = ndc_dot + ng1 * clip[1];
  const float clip_grad[4] = {ng0 / clip[3], ng1 / clip[3], 0.0f, -ndc_dot / (clip[3] * clip[3])};
#pragma unroll
  for (int col = 0; col < 3; col++) {
    float v = cam.proj[col * 4 + 0] * clip_grad[0];
    v = v + cam.proj[col * 4 + 1] * clip_grad[1];
    v = v + cam.proj[col * 4 + 2] * clip_grad[2];
    v = v + cam.proj[col * 4 + 3] * clip_grad[3];
    tg[col] = tg[col] + v;
  }
  // 5. colour
  float campos[3], off[3], dir[3], basis[15];
  camera_position(cam, campos);
  off[0] = g[0] - campos[0];
  off[1] = g[1] - campos[1];
  off[2] = g[2] - campos[2];
  const float dist = normalize3(off, dir);
  sh_basis(dir, basis);
  const float* coef = shv;
  float raw_color[3] = {g[12], g[13], g[14]};
  // These SH loops stay rolled: unrolled (basis and bgrad in registers) the
  // fused backward + Adam kernel takes 112 registers, 4 CTAs per SM instead of
  // 5, and runs slower (435 vs 408 us at 1.1M Gaussians).
  for (uint32_t k = 0; k < basis_count; k++)
#pragma unroll
    for (int ch = 0; ch < 3; ch++) raw_color[ch] = raw_color[ch] + basis[k] * coef[k * 3 + ch];
  float raw_grad[3];
#pragma unroll
  for (int ch = 0; ch < 3; ch++) raw_grad[ch] = raw_color[ch] < 0.0f ? 0.0f : grad[6 + ch];
  float dgrad[3] = {0.0f, 0.0f, 0.0f};
  {
    float bgrad[15][3];
    sh_basis_gradient(dir, bgrad);
    // Each coefficient is read before its slot of shv takes the gradient.
    for (uint32_t k = 0; k < SH_REST_FLOATS / 3; k++) {
      if (k < basis_count) {
        float d = coef[k * 3] * raw_grad[0];
        d = d + coef[k * 3 + 1] * raw_grad[1];
        d = d + coef[k * 3 + 2] * raw_grad[2];
#pragma unroll
        for (int ch = 0; ch < 3; ch++) shv[k * 3 + ch] = basis[k] * raw_grad[ch];
#pragma unroll
        for (int ax = 0; ax < 3; ax++) dgrad[ax] = dgrad[ax] + bgrad[k][ax] * d;
      } else {
#pragma unroll
        for (int ch = 0; ch < 3; ch++) shv[k * 3 + ch] = 0.0f;
      }
    }
  }
  float dd = dir[0] * dgrad[0];
  dd = dd + dir[1] * dgrad[1];
  dd = dd + dir[2] * dgrad[2];
  // 6. position
#pragma unroll
  for (int col = 0; col < 3; col++) {
    float v = p.w[col][0] * tg[0];
    v = v + p.w[col][1] * tg[1];
    v = v + p.w[col][2] * tg[2];
    out[col] = v + (dgrad[col] - dir[col] * dd) / dist;
  }
  // 7. scale and rotation
  float mg[3][3];
#pragma unroll
  for (int col = 0; col < 3; col++)
#pragma unroll
    for (int row = 0; row < 3; row++) {
      float v = 2.0f * cov3d_grad[0][row] * p.m[col][0];
      v = v + 2.0f * cov3d_grad[1][row] * p.m[col][1];
      v = v + 2.0f * cov3d_grad[2][row] * p.m[col][2];
      mg[col][row] = v;
    }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float v = mg[k][0] * p.r[k][0];
    v = v + mg[k][1] * p.r[k][1];
    v = v + mg[k][2] * p.r[k][2];
    out[4 + k] = v;
  }
  float rg[3][3];
#pragma unroll
  for (int col = 0; col < 3; col++)
#pragma unroll
    for (int row = 0; row < 3; row++) rg[col][row] = mg[col][row] * g[4 + col];
  const float qw = p.q[0], qx = p.q[1], qy = p.q[2], qz = p.q[3];
  const float g00 = rg[0][0], g01 = rg[1][0], g02 = rg[2][0];
  const float g10 = rg[0][1], g11 = rg[1][1], g12 = rg[2][1];
  const float g20 = rg[0][2], g21 = rg[1][2], g22 = rg[2][2];
  float qg[4];
  qg[0] = 2.0f * (-qz * g01 + qy * g02 + qz * g10 - qx * g12 - qy * g20 + qx * g21);
  qg[1] = 2.0f * (qy * g01 + qz * g02 + qy * g10 - 2.0f * qx * g11 - qw * g12 + qz * g20 + qw * g21 - 2.0f * qx * g22);
  qg[2] = 2.0f * (-2.0f * qy * g00 + qx * g01 + qw * g02 + qx * g10 + qz * g12 - qw * g20 + qz * g21 - 2.0f * qy * g22);
  qg[3] = 2.0f * (-2.0f * qz * g00 - qw * g01 + qx * g02 + qw * g10 - 2.0f * qz * g11 + qy * g12 + qx * g20 + qy * g21);
  float qd = p.q[0] * qg[0];
  qd = qd + p.q[1] * qg[1];
  qd = qd + p.q[2] * qg[2];
  qd = qd + p.q[3] * qg[3];
  out[3] = grad[5];
#pragma unroll
  for (int k = 0; k < 4; k++) out[8 + k] = (qg[k] - p.q[k] * qd) / p.qlen;
  out[12] = raw_grad[0];
  out[13] = raw_grad[1];
  out[14] = raw_grad[2];
}

__device__ __forceinline__ void store16(float* dst, const float (&v)[16]) {
#pragma unroll
  for (int k = 0; k < 4; k++)
    reinterpret_cast<float4*>(dst)[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
}

// One thread per Gaussian. The CTA's SH coefficients are staged in shared memory
// and its SH gradients written back from there, both as contiguous copies (a
// thread's own 45 floats would otherwise be 180 bytes apart from its neighbour's).
__global__ void __launch_bounds__(PBWD_THREADS) preprocess_backward_kernel(
    const Camera* camera, const float* gaussians, const float* sh,
    uint32_t count, const uint32_t* scene_params, const float* splats,
    const float* splat_grads, float* gaussian_grads, float* sh_grads) {
  chain_begin();
  __shared__ Camera s_cam;
  __shared__ __align__(16) float s_sh[PBWD_THREADS * SH_REST_FLOATS];
  load_camera(s_cam, camera);
  const uint32_t block_start = blockIdx.x * PBWD_THREADS;
  const uint32_t here = min(PBWD_THREADS, count - block_start);
  stage_floats_async(s_sh, sh + (size_t)block_start * SH_REST_FLOATS, here * SH_REST_FLOATS);
  cp_async_wait_all();
  __syncthreads();
  const uint32_t degree = scene_params[0];
  const uint32_t basis_count = (degree + 1u) * (degree + 1u) - 1u;
  const uint32_t i = block_start + threadIdx.x;
  if (i < count) {
    float out[16];
    preprocess_backward_one(s_cam, gaussians + (size_t)i * FLOATS_PER_GAUSSIAN, s_sh + threadIdx.x * SH_REST_FLOATS,
                            basis_count, splats[(size_t)i * FLOATS_PER_SPLAT + 3],
                            splat_grads + (size_t)i * SPLAT_GRADS, out);
    store16(gaussian_grads + (size_t)i * FLOATS_PER_GAUSSIAN, out);
  }
  __syncthreads();
  copy_floats(sh_grads + (size_t)block_start * SH_REST_FLOATS, s_sh, here * SH_REST_FLOATS);
}

// The fused kernel's tuning: the 16-byte groups of slots (four slots each) a
// thread loads before stepping them in the Adam passes.
#ifndef DG_ADAM_SH_QUADS
#define DG_ADAM_SH_QUADS 3
#endif
#ifndef DG_ADAM_P_QUADS
#define DG_ADAM_P_QUADS 4
#endif
// A minimum of resident CTAs per SM caps the registers (without one ptxas
// settles at 96 a thread, 5 CTAs of 128 per SM; an explicit minimum of 1 lets it
// take 141).
#ifdef DG_PBWD_MIN_BLOCKS
#define DG_PBWD_BOUNDS __launch_bounds__(PBWD_THREADS, DG_PBWD_MIN_BLOCKS)
#else
#define DG_PBWD_BOUNDS __launch_bounds__(PBWD_THREADS)
#endif

__device__ __forceinline__ float4 f4_load(const float* p) { return *reinterpret_cast<const float4*>(p); }

// The training step's preprocess backward with Adam applied at once
// (src/shaders/preprocessBackward.wgsl:28-181, then src/shaders/adam.wgsl:80-107).
// A CTA takes 128 consecutive Gaussians:
// 1. one bulk copy (TMA) brings their SH coefficients, a contiguous 23 KB, into
//    shared memory, completed on an mbarrier;
// 2. each thread computes one Gaussian's gradients into shared memory (the SH
//    coefficients staged there turn into their gradients; the 16 parameter
//    gradients go to a row of pitch 17) and adds its densification statistics
//    (src/shaders/adam.wgsl:126-134);
// 3. Adam steps the CTA's SH slots: their coefficients, SH moments (the second
//    plane of the moment buffer) and gradients share one index, so each thread
//    takes 16-byte groups of four slots;
// 4. Adam steps the raw parameter slots a quarter record (four slots) at a time:
//    raw values, parameter moments (the first plane) and activated values move
//    as 16-byte groups. Slots 7 and 15 (pads: a densified Gaussian's kind and
//    step) keep their raw value and moments; their activated value is 0, as the
//    reference leaves it (src/shaders/adam.wgsl:60-71 does not write them).
// The 244 bytes of gradients per Gaussian never go to memory and back;
// gaussian_grads and sh_grads (may be NULL) also receive them. The host checks
// that every buffer starts 16-byte aligned. A copy that does not complete within
// the wait limit sets DEVICE_ERROR_COPY_WAIT and the CTA returns.
__global__ void DG_PBWD_BOUNDS preprocess_backward_adam_kernel(
    const Camera* camera, float* gaussians, float* sh, uint32_t count,
    const uint32_t* scene_params, const float* radii, const float* splat_grads,
    const AdamParams* adam, float* params, float2* moments,
    float4* stats, float2* aux, float* gaussian_grads,
    float* sh_grads, uint32_t* error) {
  chain_begin();
  constexpr uint32_t GP = FLOATS_PER_GAUSSIAN + 1;  // a row pitch prime to 32
  __shared__ Camera s_cam;
  __shared__ __align__(16) float s_sh[PBWD_THREADS * SH_REST_FLOATS];  // coefficients, then their gradients
  __shared__ float s_pg[PBWD_THREADS * GP];                            // parameter gradients
  __shared__ AdamParams s_ap;
  __shared__ __align__(8) uint64_t s_bar;
  const uint32_t block_start = blockIdx.x * PBWD_THREADS;
  const uint32_t here = min(PBWD_THREADS, count - block_start);
  const uint32_t sh_total = here * SH_REST_FLOATS;
  float* sh_block = sh + (size_t)block_start * SH_REST_FLOATS;
  const uint32_t quads = sh_total / 4;  // the 16-byte groups (all of a full CTA's 5,760 floats)
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    mbar_arrive_expect_tx(&s_bar, quads * 16);
    // Kept in L2 for the Adam pass, which reads the coefficients again.
    bulk_copy_to_shared(s_sh, sh_block, quads * 16, &s_bar, l2_policy_evict_last());
    s_ap = *adam;
  }
  __syncthreads();  // the barrier is initialized before anyone waits on it
  load_camera(s_cam, camera);
  for (uint32_t e = quads * 4 + threadIdx.x; e < sh_total; e += PBWD_THREADS) s_sh[e] = sh_block[e];
  const bool copied = mbar_wait_bounded(&s_bar, 0);
  if (__syncthreads_or(!copied)) {
    if (threadIdx.x == 0) atomicOr(error, DEVICE_ERROR_COPY_WAIT);
    mbar_wait_bounded(&s_bar, 0);  // the copy may still be writing this CTA's shared memory
    return;
  }
  const uint32_t degree = scene_params[0];
  const uint32_t basis_count = (degree + 1u) * (degree + 1u) - 1u;
  const uint32_t i = block_start + threadIdx.x;
  if (i < count) {
    float out[16];
    const float radius = radii[i];
    const float* grads = splat_grads + (size_t)i * SPLAT_GRADS;
    preprocess_backward_one(s_cam, gaussians + (size_t)i * FLOATS_PER_GAUSSIAN, s_sh + threadIdx.x * SH_REST_FLOATS,
                            basis_count, radius, grads, out);
#pragma unroll
    for (int k = 0; k < 16; k++) s_pg[threadIdx.x * GP + k] = out[k];
    if (gaussian_grads) store16(gaussian_grads + (size_t)i * FLOATS_PER_GAUSSIAN, out);
    accumulate_stats_values(s_ap.viewport, radius, grads[0], grads[1], stats, aux, i);
  }
  __syncthreads();
  if (sh_grads) copy_floats(sh_grads + (size_t)block_start * SH_REST_FLOATS, s_sh, sh_total);
  const AdamParams& ap = s_ap;
  const float inv_bc1 = ap.inv_bias_correction1, inv_sqrt_bc2 = ap.inv_sqrt_bias_correction2;
  // The streams below are read and written once: evict them first, so the
  // coefficients staged with evict-last stay in L2 until step 3 reads them again.
  const uint64_t stream = l2_policy_evict_first();

  // 3. The SH slots, four at a time; a thread loads a batch of groups before
  // stepping them, so that enough reads are in flight.
  {
    constexpr uint32_t B = DG_ADAM_SH_QUADS;
    float4* m_block = reinterpret_cast<float4*>(moments + sh_moment_at(count, block_start, 0));
    const float lr = ap.sh_lr;
    for (uint32_t base = threadIdx.x; base < quads; base += PBWD_THREADS * B) {
      float4 v[B], m0[B], m1[B];
#pragma unroll
      for (uint32_t u = 0; u < B; u++) {
        const uint32_t q = base + u * PBWD_THREADS;
        if (q < quads) {
          v[u] = ld_hinted(sh_block + 4 * q, stream);
          m0[u] = ld_hinted(m_block + 2 * q, stream);
          m1[u] = ld_hinted(m_block + 2 * q + 1, stream);
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < B; u++) {
        const uint32_t q = base + u * PBWD_THREADS;
        if (q < quads) {
          const float4 g = f4_load(s_sh + 4 * q);
          float2 a = make_float2(m0[u].x, m0[u].y), b = make_float2(m0[u].z, m0[u].w);
          float2 c = make_float2(m1[u].x, m1[u].y), d = make_float2(m1[u].z, m1[u].w);
          float4 out;
          out.x = adam_step_fast(v[u].x, g.x, a, lr, inv_bc1, inv_sqrt_bc2);
          out.y = adam_step_fast(v[u].y, g.y, b, lr, inv_bc1, inv_sqrt_bc2);
          out.z = adam_step_fast(v[u].z, g.z, c, lr, inv_bc1, inv_sqrt_bc2);
          out.w = adam_step_fast(v[u].w, g.w, d, lr, inv_bc1, inv_sqrt_bc2);
          st_hinted(sh_block + 4 * q, out, stream);
          st_hinted(m_block + 2 * q, make_float4(a.x, a.y, b.x, b.y), stream);
          st_hinted(m_block + 2 * q + 1, make_float4(c.x, c.y, d.x, d.y), stream);
        }
      }
    }
    // The last floats of a partial CTA, one slot at a time.
    float2* m_slots = moments + sh_moment_at(count, block_start, 0);
    for (uint32_t e = quads * 4 + threadIdx.x; e < sh_total; e += PBWD_THREADS) {
      float2 m = m_slots[e];
      sh_block[e] = adam_step_fast(sh_block[e], s_sh[e], m, lr, inv_bc1, inv_sqrt_bc2);
      m_slots[e] = m;
    }
  }

  // 4. The raw parameter slots, a quarter record at a time (PBWD_THREADS is a
  // multiple of 4, so a thread always takes the same quarter of its records).
  {
    constexpr uint32_t B = DG_ADAM_P_QUADS;
    float* p_block = params + (size_t)block_start * FLOATS_PER_GAUSSIAN;
    float* a_block = gaussians + (size_t)block_start * FLOATS_PER_GAUSSIAN;
    float4* m_block = reinterpret_cast<float4*>(moments + param_moment_at(block_start, 0));
    const uint32_t p_quads = here * 4;
    const uint32_t k0 = 4 * (threadIdx.x & 3u);
    for (uint32_t base = threadIdx.x; base < p_quads; base += PBWD_THREADS * B) {
      float4 x[B], m0[B], m1[B];
#pragma unroll
      for (uint32_t u = 0; u < B; u++) {
        const uint32_t q = base + u * PBWD_THREADS;
        if (q < p_quads) {
          x[u] = ld_hinted(p_block + 4 * q, stream);
          m0[u] = ld_hinted(m_block + 2 * q, stream);
          m1[u] = ld_hinted(m_block + 2 * q + 1, stream);
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < B; u++) {
        const uint32_t q = base + u * PBWD_THREADS;
        if (q < p_quads) {
          const float* grad = s_pg + (q >> 2) * GP + k0;
          float xs[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
          float2 ms[4] = {make_float2(m0[u].x, m0[u].y), make_float2(m0[u].z, m0[u].w),
                          make_float2(m1[u].x, m1[u].y), make_float2(m1[u].z, m1[u].w)};
          float act[4];
#pragma unroll
          for (uint32_t j = 0; j < 4; j++) {
            const uint32_t k = k0 + j;
            if (j == 3 && (k == 7 || k == 15)) {
              act[j] = 0.0f;  // a pad: raw value and moments stay as they are
            } else {
              xs[j] = adam_param_slot(ap, k, xs[j], grad[j], ms[j], act[j]);
            }
          }
          st_hinted(p_block + 4 * q, make_float4(xs[0], xs[1], xs[2], xs[3]), stream);
          st_hinted(m_block + 2 * q, make_float4(ms[0].x, ms[0].y, ms[1].x, ms[1].y), stream);
          st_hinted(m_block + 2 * q + 1, make_float4(ms[2].x, ms[2].y, ms[3].x, ms[3].y), stream);
          st_hinted(a_block + 4 * q, make_float4(act[0], act[1], act[2], act[3]), stream);
        }
      }
    }
  }
}


}  // namespace

dg_status launch_rasterize_backward(dg_tile_rasterizer* tr, dg_buffer* pixel_grads, dg_buffer* splat_grads) {
  dg_context* ctx = tr->ctx;
  uint32_t* counter = typed<uint32_t>(tr->work) + 2;
  const uint32_t item_room = (uint32_t)(tr->items->bytes / sizeof(uint2) / ITEM_CLASSES);
  const size_t floats = (size_t)tr->count * SPLAT_GRADS;
  const uint32_t tiles = tr->tiles_x * tr->tiles_y;
  const uint64_t ctas = std::max<uint64_t>(ceil_div(tiles, LIST_WARPS), ceil_div(floats, 4 * LIST_THREADS));
  DG_CHAIN(ctx, "list_items", (list_items_kernel),
           (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(ctas, (uint64_t)ctx->sm_count * 8)), LIST_THREADS, 0,
           typed<uint2>(tr->ranges), typed<uint32_t>(tr->walked), typed<uint32_t>(tr->work_plan),
           typed<uint2>(tr->items), item_room, typed<float>(splat_grads), floats);
  DG_LAUNCH(ctx, "rasterize_backward",
            rasterize_backward_kernel<<<blend_grid(ctx, (const void*)rasterize_backward_kernel, BWD_THREADS,
                                                    tr->tiles_x * tr->tiles_y * 8u),
                                        BWD_THREADS, 0, ctx->stream>>>(
                typed<const Camera>(tr->camera), typed<float4>(tr->raster_params), typed<float>(tr->splats),
                typed<uint32_t>(tr->values), typed<uint2>(tr->ranges), typed<uint32_t>(tr->work_plan),
                typed<uint2>(tr->items), item_room, typed<float4>(tr->pixel_color), typed<uint32_t>(tr->pixel_last),
                typed<float4>(tr->checkpoints), typed<uint32_t>(tr->blend_mask), typed<float4>(pixel_grads),
                typed<float>(splat_grads), counter, tr->splat_cutoffs));
  return DG_OK;
}

dg_status launch_preprocess_backward_adam(dg_renderer* r, const AdamParams* adam, float* params, float2* moments,
                                         float4* stats, float2* aux, bool keep_gradients) {
  // Every stream of the kernel moves 16-byte groups from the start of each buffer.
  const void* starts[] = {params, moments, ptr_of(r->gaussians), ptr_of(r->sh)};
  for (const void* p : starts)
    DG_REQUIRE((reinterpret_cast<uintptr_t>(p) & 15) == 0, "the training buffers must start 16-byte aligned");
  DG_CHAIN(r->ctx, "preprocess_backward_adam", (preprocess_backward_adam_kernel), ceil_div(r->count, PBWD_THREADS), PBWD_THREADS, 0,
           typed<const Camera>(r->camera), typed<float>(r->gaussians), typed<float>(r->sh), r->count,
           typed<uint32_t>(r->scene_params), typed<float>(r->radii), typed<float>(r->grad_splats), adam, params,
           moments, stats, aux, keep_gradients ? typed<float>(r->grad_gaussians) : nullptr,
           keep_gradients ? typed<float>(r->grad_sh) : nullptr, r->ctx->device_error);
  return DG_OK;
}

dg_status launch_preprocess_backward(dg_renderer* r) {
  DG_CHAIN(r->ctx, "preprocess_backward", (preprocess_backward_kernel), ceil_div(r->count, PBWD_THREADS), PBWD_THREADS, 0,
           typed<const Camera>(r->camera), typed<float>(r->gaussians), typed<float>(r->sh), r->count,
           typed<uint32_t>(r->scene_params), typed<float>(r->splats), typed<float>(r->grad_splats),
           typed<float>(r->grad_gaussians), typed<float>(r->grad_sh));
  return DG_OK;
}

}  // namespace dg
