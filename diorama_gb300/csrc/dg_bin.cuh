// Tile binning of depth-ordered splats, shared by the renderer (dg_render.cu) and
// the batches of views (dg_views.cu).
#pragma once
#include "dg_common.cuh"

namespace dg {

// The splats of one frame, or of each view of a batch (per_view consecutive ones
// of the depth order each), and the grid of tiles they are listed in.
struct BinShape {
  uint32_t per_view, views, grid_x, grid_y;
};
// Whether bin_launch takes this grid (the caller sorts the pairs otherwise).
bool bin_fits(uint32_t grid_x, uint32_t grid_y);
// Per-device kernel attributes; called once when a context is created.
dg_status bin_init();
size_t bin_scratch_bytes(const BinShape& s);

struct BinLaunch {
  const uint32_t* rects;  // per splat, its rectangle of tiles (pack_rect)
  const uint32_t* order;  // splat numbers, view by view, nearest first
  uint32_t capacity;      // pairs that `values` holds
  void* scratch;
  uint32_t* pair_total;  // element 0: the pairs the frame needs
  uint32_t* values;      // out: each tile's splats, nearest first, tile after tile
  uint2* ranges;         // out: each tile's run of values (0, 0 when it has none)
  uint32_t* plan;        // out: the blend's work plan, its header cleared (dg_render_kernels.cuh)
  uint32_t* work;        // out: the blend kernels' 4 item counters, cleared
};
// Lists every tile's splats. Of a frame that needs more than
// `capacity` pairs, the ones that come first in depth order (then row by row of
// the splat's rectangle) are kept.
dg_status bin_launch(dg_context* ctx, const BinShape& s, const BinLaunch& l);
// The 64-bit (tile << 32 | depth bits) key of every listed pair.
dg_status bin_keys_launch(dg_context* ctx, uint32_t tiles, const uint2* ranges, const uint32_t* values,
                          const float* splats, uint64_t* keys);

// A rectangle of tiles [x, z) x [y, w) of a grid that bin_fits, in 4 bytes.
__device__ __forceinline__ uint32_t pack_rect(uint4 r) { return r.x | r.y << 8 | r.z << 16 | r.w << 24; }

}  // namespace dg
