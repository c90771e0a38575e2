// TrainingLoss (src/trainingLoss.ts:16-130, src/shaders/loss.wgsl:53-121):
// 0.8 L1 + 0.2 (1 - SSIM) between a render and a photo, with an 11x11 Gaussian
// window (sigma 1.5, zero padding), and its gradient with respect to every
// rendered pixel.
//
// The reference makes 7 dispatches over 5-map and 3-map vec4 buffers (moments,
// blur h, blur v, ssim, blur h, blur v, gradient: ~900 B/pixel of traffic). Here
// it is 2 kernels:
//   ssim_kernel:     moments -> blur h -> blur v -> SSIM, its three partials and the
//                    pixel loss
//   gradient_kernel: partials -> blur h -> blur v -> dL/dpixel
// An ssim_kernel CTA owns a 16x16 block of pixels, loads its 26x26 halo once, and does
// the separable blurs in shared memory. A gradient_kernel CTA walks down a strip of 32
// columns instead: each row is staged and blurred along the row once, and the blur
// down the columns stays in registers (the sums of the 11 output rows that a row
// belongs to move up one place each as its tap is added, acc[k] = w[k] v + acc[k - 1]),
// so no blurred row is stored or read back and a strip costs 10 extra rows, not a halo
// around every 16x16 pixels.
// Sums run over the taps -5..5 in order, one fused multiply-add per tap (in ssim_kernel
// two sums per packed FP32 instruction where they pair up); taps past the image add
// exactly 0 (zeros are staged there), the same as the WGSL's skipping them.
//
// Both are bound by instructions, not by memory (1957x1091: 132 bytes per pixel in
// 167 us are 1.7 TB/s). Blocks against strips, in us, at 96x96 | 251x187 | 489x273 |
// 980x545 | 1957x1091: gradient 8.3 | 10.1 | 14.2 | 33.0 | 127 with blocks, 10.2 | 10.6 |
// 14.5 | 24.8 | 62 with strips. The SSIM pass has five maps to keep sums of, not three,
// and spills: 12.2 | 13.2 | 17.4 | 36 | 110 with blocks, 22 | 22 | 25 | 45 | 132 with
// strips (blocks of 16x32 pixels with two rows per thread: 15 | 17 | 17 | 35 | 109; of
// 16x16 with two rows and half the threads 13.5 | 17 | 18 | 34 | 119). Without bank
// conflicts in its horizontal pass, and the halo's loads ahead of the table of bytes, it
// takes 11 | 13 | 17.4 | 34 | 105.
// The partials lie in planes of their own, which a strip's warp reads in whole lines.
//
// The same ssim_kernel also measures held-out renders (PSNR and SSIM of the
// 8-bit-quantized image, src/trainer.ts:371-386 and src/metrics.ts) on the GPU.
#include "dg_common.cuh"
#include "dg_loss.cuh"

namespace dg {
namespace {

constexpr int HALO = 5;
constexpr int TAPS = 2 * HALO + 1;
// ssim_kernel: a CTA's block of pixels and its halo.
constexpr int LT = 16;
constexpr int LS = LT + 2 * HALO;  // 26
constexpr int SSIM_THREADS = LT * LT;
// gradient_kernel: a strip's columns (a lane each) and its halo; a warp per channel.
constexpr int COLS = 32;
constexpr int SPAN = COLS + 2 * HALO;  // 42
constexpr int STRIP_THREADS = 3 * 32;
constexpr uint32_t STRIPS_PER_SM = 6;
constexpr int MIN_ROWS = 6;
constexpr float LAMBDA = 0.2f;
constexpr float C1 = 0.0001f;
constexpr float C2 = 0.0009f;

struct Window {
  float w[6];
};

// src/trainer.ts:381: round(min(1, max(0, v)) * 255) / 255, in double as the
// TypeScript does, then stored as float32.
__device__ __forceinline__ float3 quantized(float4 v) {
  auto q = [](float c) {
    double d = rint((double)fminf(1.0f, fmaxf(0.0f, c)) * 255.0);
    return __double2float_rn(d / 255.0);
  };
  return make_float3(q(v.x), q(v.y), q(v.z));
}

// A byte's value as float, v / 255: the loss's float quotient, or for metrics
// (exact_quotient) Float32Array.from(bytes, v => v / 255), the double quotient
// rounded to float.
__device__ __forceinline__ float unorm8(uint32_t v, bool exact_quotient) {
  return exact_quotient ? __double2float_rn(v / 255.0) : (float)v / 255.0f;
}

// The 256 values of unorm8 in shared memory, so a pixel's three channels take three
// loads, not divisions.
__device__ __forceinline__ void fill_unorm8(float* table, bool exact_quotient, uint32_t threads) {
  for (uint32_t k = threadIdx.x; k < 256; k += threads) table[k] = unorm8(k, exact_quotient);
}

// The weight of tap k - 5.
__device__ __forceinline__ int tap_weight(int k) { return k < HALO ? HALO - k : k - HALO; }

// Moments, both blurs and the SSIM partials for one 16x16 block. mode 0 (loss):
// writes each channel's partials, (dS/dmu_x, dS/dE[x^2]) and dS/dE[xy], in planes of
// their own (`partials`: 3 planes of float2, then 3 of float, one value per pixel),
// and the pixel loss. mode 1 (metrics): the render is quantized first, and each CTA
// adds its Σ S and Σ squared error to `sums`.
//
// The x and y sums of each blur, and the x^2 and y^2 ones, run as pairs through
// packed FP32 fused multiply-adds (F2): each lane is the scalar fmaf sum.
__global__ void __launch_bounds__(SSIM_THREADS, 5) ssim_kernel(const float4* __restrict__ rendered,
                                                   const uchar4* const* __restrict__ target_slot, int w, int h,
                                                   Window win, float* __restrict__ partials,
                                                   float* __restrict__ pixel_loss, int mode,
                                                   double* __restrict__ sums) {
  // Rows of odd length: the lanes of the horizontal pass read and write two rows or
  // channels at once, eight pairs of columns each, without bank conflicts.
  __shared__ float2 s_xy[LS][LS * 3 + 1];   // (x, y) per halo pixel and channel
  __shared__ float2 s_h01[LS][LT * 3 + 1];  // horizontal blurs of x and y
  __shared__ float2 s_h23[LS][LT * 3 + 1];  // of x^2 and y^2
  __shared__ float s_h4[LS][LT * 3 + 1];    // of xy
  __shared__ double s_red[2][SSIM_THREADS / 32];
  __shared__ float s_unorm[256];
  const uchar4* target = *target_slot;
  const int x0 = blockIdx.x * LT - HALO, y0 = blockIdx.y * LT - HALO;
  const bool metrics = mode == 1;
  // The halo's pixels are on their way while the table is filled.
  constexpr int EACH = (LS * LS + SSIM_THREADS - 1) / SSIM_THREADS;
  float4 px[EACH];
  uchar4 py[EACH];
#pragma unroll
  for (int u = 0; u < EACH; u++) {
    const int k = threadIdx.x + u * SSIM_THREADS, x = x0 + k % LS, y = y0 + k / LS;
    const bool in = k < LS * LS && x >= 0 && y >= 0 && x < w && y < h;
    px[u] = in ? rendered[(size_t)y * w + x] : make_float4(0.f, 0.f, 0.f, 0.f);
    py[u] = in ? target[(size_t)y * w + x] : make_uchar4(0, 0, 0, 0);
  }
  fill_unorm8(s_unorm, metrics, SSIM_THREADS);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < EACH; u++) {
    const int k = threadIdx.x + u * SSIM_THREADS;
    if (k >= LS * LS) break;
    // Past the image both are 0, as the table's entry for 0 is.
    const float3 xv = metrics ? quantized(px[u]) : make_float3(px[u].x, px[u].y, px[u].z);
    float2* to = &s_xy[k / LS][3 * (k % LS)];
    to[0] = make_float2(xv.x, s_unorm[py[u].x]);
    to[1] = make_float2(xv.y, s_unorm[py[u].y]);
    to[2] = make_float2(xv.z, s_unorm[py[u].z]);
  }
  F2 wp[6];
#pragma unroll
  for (int k = 0; k < 6; k++) wp[k] = f2(win.w[k], win.w[k]);
  __syncthreads();
  // Horizontal pass over every halo row, for the 16 output columns, two adjacent
  // columns per item: their 11-tap windows share 10 halo values, read (and
  // squared) once. Each column's sums still run over its taps -5..5 in order.
  for (int k = threadIdx.x; k < LS * (LT / 2) * 3; k += SSIM_THREADS) {
    const int col = 2 * (k % (LT / 2)), ch = k / (LT / 2) % 3, row = k / (3 * (LT / 2));
    F2 a01 = f2(0.f, 0.f), a23 = f2(0.f, 0.f), b01 = a01, b23 = a01;
    float a4 = 0.f, b4 = 0.f;
    // Taps past the image read the halo's zeros and add exactly 0: the same sums
    // as skipping them, without a branch per tap.
#pragma unroll
    for (int t = -HALO; t <= HALO + 1; t++) {  // halo column col + HALO + t
      const F2 xy = f2_load(&s_xy[row][3 * (col + HALO + t) + ch]);
      const F2 sq = f2_mul(xy, xy);
      const float pr = f2_lo(xy) * f2_hi(xy);
      if (t <= HALO) {  // column col, tap t
        const int at = t < 0 ? -t : t;
        a01 = f2_fma(wp[at], xy, a01);  // x, y
        a23 = f2_fma(wp[at], sq, a23);  // x^2, y^2
        a4 = fmaf(win.w[at], pr, a4);   // xy
      }
      if (t > -HALO) {  // column col + 1, tap t - 1
        const int at = t - 1 < 0 ? 1 - t : t - 1;
        b01 = f2_fma(wp[at], xy, b01);
        b23 = f2_fma(wp[at], sq, b23);
        b4 = fmaf(win.w[at], pr, b4);
      }
    }
    f2_store(&s_h01[row][3 * col + ch], a01);
    f2_store(&s_h23[row][3 * col + ch], a23);
    s_h4[row][3 * col + ch] = a4;
    f2_store(&s_h01[row][3 * col + 3 + ch], b01);
    f2_store(&s_h23[row][3 * col + 3 + ch], b23);
    s_h4[row][3 * col + 3 + ch] = b4;
  }
  __syncthreads();
  const int lx = threadIdx.x % LT, ly = threadIdx.x / LT;
  const int gx = blockIdx.x * LT + lx, gy = blockIdx.y * LT + ly;
  double s_sum = 0.0, se_sum = 0.0;
  if (gx < w && gy < h) {
    const size_t pixels = (size_t)w * h, p = (size_t)gy * w + gx;
    float lsum = 0.0f;
#pragma unroll
    for (int ch = 0; ch < 3; ch++) {
      F2 m01 = f2(0.f, 0.f), m23 = f2(0.f, 0.f);
      float m4 = 0.f;
#pragma unroll
      for (int k = 0; k < TAPS; k++) {  // rows past the image were blurred to 0
        const int at = tap_weight(k);
        m01 = f2_fma(wp[at], f2_load(&s_h01[ly + k][3 * lx + ch]), m01);
        m23 = f2_fma(wp[at], f2_load(&s_h23[ly + k][3 * lx + ch]), m23);
        m4 = fmaf(win.w[at], s_h4[ly + k][3 * lx + ch], m4);
      }
      const float mx = f2_lo(m01), my = f2_hi(m01);
      const float vx = f2_lo(m23) - mx * mx, vy = f2_hi(m23) - my * my, cxy = m4 - mx * my;
      const float a1 = 2.0f * mx * my + C1, a2 = 2.0f * cxy + C2;
      const float b1 = mx * mx + my * my + C1, b2 = vx + vy + C2;
      const float s = a1 * a2 / (b1 * b2);
      const float2 xy = s_xy[ly + HALO][3 * (lx + HALO) + ch];
      if (metrics) {
        s_sum += (double)s;
        const double d = (double)xy.x - (double)xy.y;
        se_sum += d * d;
      } else {
        reinterpret_cast<float2*>(partials)[ch * pixels + p] =
            make_float2(s * (2.0f * my / a1 - 2.0f * my / a2 - 2.0f * mx / b1 + 2.0f * mx / b2), -s / b2);
        partials[(6 + ch) * pixels + p] = 2.0f * s / a2;
        lsum = lsum + ((1.0f - LAMBDA) * fabsf(xy.x - xy.y) - LAMBDA * s);
      }
    }
    if (!metrics) pixel_loss[p] = lsum * (1.0f / (float)(3u * (uint32_t)(w * h)));
  }
  if (metrics) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      s_sum += __shfl_xor_sync(0xffffffffu, s_sum, d);
      se_sum += __shfl_xor_sync(0xffffffffu, se_sum, d);
    }
    if ((threadIdx.x & 31) == 0) {
      s_red[0][threadIdx.x >> 5] = s_sum;
      s_red[1][threadIdx.x >> 5] = se_sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0, b = 0;
      for (int k = 0; k < SSIM_THREADS / 32; k++) {
        a += s_red[0][k];
        b += s_red[1][k];
      }
      atomicAdd(&sums[0], a);
      atomicAdd(&sums[1], b);
    }
  }
}

// Blurs the three partials and forms dL/dpixel (src/shaders/loss.wgsl:108-121) for
// one strip's rows [y_begin, y_end): a warp per channel, a lane per column.
__global__ void __launch_bounds__(STRIP_THREADS, STRIPS_PER_SM) gradient_kernel(
    const float4* __restrict__ rendered, const uchar4* const* __restrict__ target_slot, int w, int h, int rows,
    Window win, const float* __restrict__ partials, float4* __restrict__ pixel_grads) {
  __shared__ float2 s_p01[4][3][SPAN];
  __shared__ float s_p2[4][3][SPAN];
  __shared__ float s_grad[2][2][3][COLS];
  __shared__ float s_unorm[256];
  const uchar4* target = *target_slot;
  const int lane = threadIdx.x & 31, ch = threadIdx.x >> 5;
  const int x0 = blockIdx.x * COLS - HALO, gx = blockIdx.x * COLS + lane;
  const int y_begin = blockIdx.y * rows, y_end = min(y_begin + rows, h);
  const size_t pixels = (size_t)w * h;
  const float2* p01 = reinterpret_cast<const float2*>(partials) + ch * pixels;
  const float* p2 = partials + (6 + ch) * pixels;
  // The warp's channel of rows y and y + 1 (zeros past the image): lane l brings
  // columns x0 + l and x0 + 32 + l (the first 10 lanes), loaded while the rows before
  // are blurred.
  float2 next01[2][2];
  float next2[2][2];
  auto fetch = [&](int y) {
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int c = 32 * u + lane, col = x0 + c;
        const bool in = c < SPAN && col >= 0 && col < w && y + r >= 0 && y + r < h;
        next01[r][u] = in ? p01[(size_t)(y + r) * w + col] : make_float2(0.f, 0.f);
        next2[r][u] = in ? p2[(size_t)(y + r) * w + col] : 0.f;
      }
  };
  auto stage = [&](int y) {
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int u = 0; u < 2; u++) {
        if (32 * u + lane >= SPAN) continue;
        s_p01[(y + r) & 3][ch][32 * u + lane] = next01[r][u];
        s_p2[(y + r) & 3][ch][32 * u + lane] = next2[r][u];
      }
  };
  // acc[m][k]: map m's sum over taps -5..k - 5 of the output row 5 - k rows below.
  float acc[3][TAPS - 1];
#pragma unroll
  for (int m = 0; m < 3; m++)
#pragma unroll
    for (int k = 0; k < TAPS - 1; k++) acc[m][k] = 0.f;
  const float scale = 1.0f / (float)(3u * (uint32_t)(w * h));
  fetch(y_begin - HALO);
  fill_unorm8(s_unorm, false, STRIP_THREADS);
  stage(y_begin - HALO);
  fetch(y_begin - HALO + 2);
  __syncthreads();
  // Two rows at a time: twice the independent work per barrier.
  for (int y = y_begin - HALO; y < y_end + HALO; y += 2) {
    stage(y + 2);
    fetch(y + 4);
    // The output rows' own pixels.
    float x[2];
    uint32_t byte[2];
    bool wanted[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int out = y + u - HALO;
      const size_t p = (size_t)out * w + gx;
      wanted[u] = out >= y_begin && out < y_end && gx < w;
      x[u] = wanted[u] ? reinterpret_cast<const float*>(rendered + p)[ch] : 0.f;
      byte[u] = wanted[u] ? reinterpret_cast<const unsigned char*>(target + p)[ch] : 0u;
    }
    float b[2][3];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const float2* row01 = s_p01[(y + u) & 3][ch] + lane;
      const float* row2 = s_p2[(y + u) & 3][ch] + lane;
      b[u][0] = b[u][1] = b[u][2] = 0.f;
#pragma unroll
      for (int k = 0; k < TAPS; k++) {
        const float2 v = row01[k];
        const float wk = win.w[tap_weight(k)];
        b[u][0] = fmaf(wk, v.x, b[u][0]);
        b[u][1] = fmaf(wk, v.y, b[u][1]);
        b[u][2] = fmaf(wk, row2[k], b[u][2]);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
      float sum[3];
#pragma unroll
      for (int m = 0; m < 3; m++) {
        sum[m] = fmaf(win.w[HALO], b[u][m], acc[m][TAPS - 2]);
#pragma unroll
        for (int k = TAPS - 2; k > 0; k--) acc[m][k] = fmaf(win.w[tap_weight(k)], b[u][m], acc[m][k - 1]);
        acc[m][0] = fmaf(win.w[HALO], b[u][m], 0.f);
      }
      if (wanted[u]) {
        const float yv = s_unorm[byte[u]];
        const float sg = sum[0] + 2.0f * x[u] * sum[1] + yv * sum[2];
        const float diff = x[u] - yv;
        const float sign = diff > 0.0f ? 1.0f : (diff < 0.0f ? -1.0f : 0.0f);
        s_grad[(y >> 1) & 1][u][ch][lane] = ((1.0f - LAMBDA) * sign - LAMBDA * sg) * scale;
      }
    }
    __syncthreads();
    if (ch < 2 && (ch == 0 ? wanted[0] : wanted[1])) {  // warps 0 and 1: a row each
      const float(*g)[COLS] = s_grad[(y >> 1) & 1][ch];
      pixel_grads[(size_t)(y + ch - HALO) * w + gx] = make_float4(g[0][lane], g[1][lane], g[2][lane], 0.0f);
    }
  }
}

// Σ pixel_loss in double, in a fixed order (per-CTA partial sums, then one CTA).
__global__ void __launch_bounds__(256) loss_sum_kernel(const float* __restrict__ pixel_loss, uint32_t n,
                                                       double* __restrict__ partial, uint32_t per_block) {
  __shared__ double s[8];
  const uint32_t begin = blockIdx.x * per_block, end = min(n, begin + per_block);
  double acc = 0.0;
  for (uint32_t i = begin + threadIdx.x; i < end; i += 256) acc += (double)pixel_loss[i];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int k = 0; k < 8; k++) t += s[k];
    partial[blockIdx.x] = t;
  }
}

__global__ void loss_total_kernel(const double* __restrict__ partial, uint32_t blocks, double* __restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double t = 0;
    for (uint32_t k = 0; k < blocks; k++) t += partial[k];
    out[0] = t + (double)LAMBDA;
  }
}

Window window_weights() {
  double raw[6], total;
  for (int k = 0; k < 6; k++) raw[k] = std::exp(-(double)(k * k) / (2 * 1.5 * 1.5));
  total = raw[0] + 2 * (raw[1] + raw[2] + raw[3] + raw[4] + raw[5]);
  Window win;
  for (int k = 0; k < 6; k++) win.w[k] = (float)(raw[k] / total);
  return win;
}

}  // namespace

// Rows per strip of gradient_kernel (even): as few as still fit on the GPU at once, so
// that no strip waits for another's end; each strip costs 10 rows more. Six strips per
// SM: 5 take 65 us at 1957x1091, 6 take 62, 7 take 68, 8 take 60; at 489x273 14 us for 6,
// 15 for 7 and 8. At least 6 rows: at 251x187 10.6 us, 8 rows 11.5, 12 rows 12.3, 4 rows
// no faster and at 489x273 1 us slower. But 2 or 4 rows while there are no more than 2
// strips per SM, where a strip's own chain of rows is all there is: the whole loss at 96x96
// 22.2 us with 6 rows, 18.3 with 2 (21.5 with blocks); at 200x150 22.7 and 21.7 with 4
// (21.6); with up to 3 strips per SM so, 160x120 takes 21.5 instead of 20.2.
static int strip_rows(const dg_context* ctx, uint32_t width, uint32_t height) {
  const uint32_t across = ceil_div(width, COLS), room = (uint32_t)ctx->sm_count * STRIPS_PER_SM;
  for (int rows = 2; rows < MIN_ROWS; rows += 2)
    if (across * ceil_div(height, rows) <= 2 * (uint32_t)ctx->sm_count) return rows;
  const uint32_t down = std::max(1u, room / across);
  return std::max(MIN_ROWS, (int)(ceil_div(ceil_div(height, down), 2) * 2));
}

dg_status loss_launch(dg_training_loss* l, dg_buffer* rendered) {
  dg_context* ctx = l->ctx;
  const Window win = window_weights();
  const int w = (int)l->width, h = (int)l->height, rows = strip_rows(ctx, l->width, l->height);
  const auto* target = typed<const uchar4* const>(l->target_slot);
  DG_LAUNCH(ctx, "loss_ssim",
            ssim_kernel<<<dim3(ceil_div(w, LT), ceil_div(h, LT)), SSIM_THREADS, 0, ctx->stream>>>(
                typed<float4>(rendered), target, w, h, win, typed<float>(l->partials), typed<float>(l->pixel_loss), 0,
                nullptr));
  DG_LAUNCH(ctx, "loss_gradient",
            gradient_kernel<<<dim3(ceil_div(w, COLS), ceil_div(h, rows)), STRIP_THREADS, 0, ctx->stream>>>(
                typed<float4>(rendered), target, w, h, rows, win, typed<float>(l->partials),
                typed<float4>(l->pixel_grads)));
  return DG_OK;
}

dg_status loss_sum_launch(dg_training_loss* l) {
  dg_context* ctx = l->ctx;
  const uint32_t n = l->width * l->height;
  const uint32_t per_block = 4096;
  const uint32_t blocks = std::max(1u, ceil_div(n, per_block));
  DG_LAUNCH(ctx, "loss_sum",
            loss_sum_kernel<<<blocks, 256, 0, ctx->stream>>>(typed<float>(l->pixel_loss), n,
                                                             typed<double>(l->sum_scratch), per_block));
  DG_LAUNCH(ctx, "loss_total",
            loss_total_kernel<<<1, 32, 0, ctx->stream>>>(typed<double>(l->sum_scratch), blocks,
                                                          typed<double>(l->sum_scratch) + l->sum_blocks));
  return DG_OK;
}

dg_status metrics_launch(dg_context* ctx, dg_buffer* rendered, dg_buffer* target_slot, uint32_t width, uint32_t height,
                         double* sums_device) {
  const Window win = window_weights();
  dim3 grid(ceil_div(width, LT), ceil_div(height, LT));
  DG_LAUNCH(ctx, "metrics_ssim",
            ssim_kernel<<<grid, SSIM_THREADS, 0, ctx->stream>>>(typed<float4>(rendered),
                                                       typed<const uchar4* const>(target_slot), (int)width,
                                                       (int)height, win, nullptr, nullptr, 1, sums_device));
  return DG_OK;
}

}  // namespace dg

using namespace dg;

extern "C" {

dg_status dg_training_loss_create(dg_context* ctx, uint32_t width, uint32_t height, dg_training_loss** out) {
  DG_REQUIRE(ctx && out, "NULL argument");
  DG_REQUIRE(width > 0 && height > 0, "empty image");
  auto* l = new dg_training_loss();
  l->ctx = ctx;
  l->width = width;
  l->height = height;
  const size_t pixels = (size_t)width * height;
  l->sum_blocks = std::max(1u, ceil_div(pixels, 4096));
  dg_status st = alloc_buffer(ctx, pixels * 16, &l->pixel_grads);
  if (st == DG_OK) st = alloc_buffer(ctx, pixels * 4, &l->pixel_loss);
  if (st == DG_OK) st = alloc_buffer(ctx, pixels * 9 * 4, &l->partials);
  if (st == DG_OK) st = alloc_buffer(ctx, 8, &l->target_slot);
  if (st == DG_OK) st = alloc_buffer(ctx, (l->sum_blocks + 1) * 8, &l->sum_scratch);
  if (st != DG_OK) {
    dg_training_loss_destroy(l);
    return st;
  }
  *out = l;
  return DG_OK;
}

dg_status dg_training_loss_encode(dg_training_loss* l, dg_buffer* rendered, dg_buffer* target) {
  DG_REQUIRE(l && rendered && target, "NULL argument");
  const uint64_t pixels = (uint64_t)l->width * l->height;
  DG_REQUIRE(rendered->bytes >= pixels * 16, "rendered buffer smaller than the image");
  DG_REQUIRE(target->bytes >= pixels * 4, "target smaller than the image");
  const void* ptr = target->ptr;
  DG_TRY(write_async(l->ctx, l->target_slot->ptr, &ptr, sizeof(ptr)));
  return loss_launch(l, rendered);
}

dg_buffer* dg_training_loss_pixel_grads(dg_training_loss* l) { return l ? l->pixel_grads : nullptr; }
dg_buffer* dg_training_loss_pixel_loss(dg_training_loss* l) { return l ? l->pixel_loss : nullptr; }

dg_status dg_training_loss_read(dg_training_loss* l, double* out) {
  DG_REQUIRE(l && out, "NULL argument");
  const size_t pixels = (size_t)l->width * l->height;
  std::vector<float> shares(pixels);
  DG_CUDA(cudaMemcpyAsync(shares.data(), l->pixel_loss->ptr, pixels * 4, cudaMemcpyDeviceToHost, l->ctx->stream));
  DG_CUDA(cudaStreamSynchronize(l->ctx->stream));
  double sum = 0;
  for (float s : shares) sum += s;
  *out = sum + (double)LAMBDA;
  return DG_OK;
}

dg_status dg_training_loss_destroy(dg_training_loss* l) {
  if (!l) return DG_OK;
  for (dg_buffer* b : {l->pixel_grads, l->pixel_loss, l->partials, l->target_slot, l->sum_scratch}) free_buffer(b);
  delete l;
  return DG_OK;
}

}  // extern "C"
