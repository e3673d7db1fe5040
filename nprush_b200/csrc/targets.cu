// targets.cu — target preprocessing passes on device images: the separable
// Gaussian blur (src/lib/gpu/blur.wgsl:23-48, GpuBlurPipelineManager), the
// depth-aware bilateral blur (depth_aware_blur.wgsl:12-53,
// GpuDepthAwareBlurPipelineManager) and the Sobel depth-edge pass
// (splat_edge.wgsl:13-44), which feed the Bezier layers' targets.
//
// Images are H x W float4 RGBA in device memory (a depth image uses .x).  The
// reference stores into rgba8unorm textures; `quantize` applies that
// conversion (clamp to [0, 1], round to the nearest of 256 levels) so the
// outputs equal what the reference's textures hold, and without it the kernels
// return the stored float values.  The blurs work on shared-memory tiles; for
// directions off the axes and halos too wide for a tile, and for the edge
// pass, one thread per output pixel reads its neighbourhood through the
// read-only cache.
#include <cuda_runtime.h>

#include <cmath>

#include "common.cuh"
#include "context.h"

namespace nps {
namespace tgt {

__device__ __forceinline__ float unorm8(float x) { return rintf(fminf(fmaxf(x, 0.0f), 1.0f) * 255.0f) / 255.0f; }

__device__ __forceinline__ float4 finish(float r, float g, float b, int quantize) {
  if (quantize) return make_float4(unorm8(r), unorm8(g), unorm8(b), 1.0f);
  return make_float4(r, g, b, 1.0f);
}

__device__ __forceinline__ float srgb_to_linear(float c) {
  return c > 0.04045f ? powf((c + 0.055f) / 1.055f, 2.4f) : c / 12.92f;
}
__device__ __forceinline__ float linear_to_srgb(float c) {
  const float s = fmaxf(c, 0.0f);
  return s > 0.0031308f ? 1.055f * powf(s, 1.0f / 2.4f) - 0.055f : s * 12.92f;
}

// blur.wgsl:23-48: taps along `dir`, edge-clamped, weights exp(-i^2 / 2 sigma^2)
__global__ void k_blur(const float4* __restrict__ src, float4* __restrict__ dst, int w, int h, int dx, int dy,
                       int radius, uint32_t flags, float sigma, int quantize) {
  const int x = blockIdx.x * 16 + threadIdx.x, y = blockIdx.y * 16 + threadIdx.y;
  if (x >= w || y >= h) return;
  const bool in_srgb = flags & 1u, out_srgb = flags & 2u;
  float sr = 0.0f, sg = 0.0f, sb = 0.0f, ws = 0.0f;
  for (int i = -radius; i <= radius; ++i) {
    const int cx = min(max(x + dx * i, 0), w - 1), cy = min(max(y + dy * i, 0), h - 1);
    const float4 c = __ldg(src + (size_t)cy * w + cx);
    float r = c.x, g = c.y, b = c.z;
    if (in_srgb) r = srgb_to_linear(r), g = srgb_to_linear(g), b = srgb_to_linear(b);
    const float wt = expf(-(float)(i * i) / (2.0f * sigma * sigma));
    sr += r * wt;
    sg += g * wt;
    sb += b * wt;
    ws += wt;
  }
  float r = sr / ws, g = sg / ws, b = sb / ws;
  if (out_srgb) r = linear_to_srgb(r), g = linear_to_srgb(g), b = linear_to_srgb(b);
  dst[(size_t)y * w + x] = finish(r, g, b, quantize);
}

// The axis-aligned passes of the separable blur, k_blur's sums in its order.  A
// block stages its tile and halo in shared memory, decoded once, where k_blur
// decodes (powf three times) and reads every tap again, and takes the weights
// from a table.  kVert: 32 x 32 pixels, taps along y; else 128 x 8, along x;
// four pixels per thread.  1024 x 768, radius 8, sRGB in and out: the two
// passes 155 -> 40 us (floor: 50 MB, 7.7 us).
template <bool kVert>
__global__ void __launch_bounds__(256, 6) k_blur_axis(const float4* __restrict__ src, float4* __restrict__ dst, int w,
                                                   int h, int radius, uint32_t flags, float sigma, int quantize) {
  constexpr int kTW = kVert ? 32 : 128, kTH = kVert ? 32 : 8;
  extern __shared__ float4 sm_tile[];
  const int sw = kVert ? kTW : kTW + 2 * radius, sh = kVert ? kTH + 2 * radius : kTH;
  float* wts = reinterpret_cast<float*>(sm_tile + sw * sh);
  const int x0 = blockIdx.x * kTW, y0 = blockIdx.y * kTH, tid = threadIdx.x;
  const bool in_srgb = flags & 1u, out_srgb = flags & 2u;
  for (int i = tid; i <= 2 * radius; i += 256) {
    const int t = i - radius;
    wts[i] = expf(-(float)(t * t) / (2.0f * sigma * sigma));
  }
  for (int e = tid; e < sw * sh; e += 256) {
    const int ly = e / sw, lx = e - ly * sw;
    const int gx = min(max(x0 + lx - (kVert ? 0 : radius), 0), w - 1);
    const int gy = min(max(y0 + ly - (kVert ? radius : 0), 0), h - 1);
    float4 c = __ldg(src + (size_t)gy * w + gx);
    if (in_srgb) c.x = srgb_to_linear(c.x), c.y = srgb_to_linear(c.y), c.z = srgb_to_linear(c.z);
    sm_tile[e] = c;
  }
  __syncthreads();
  constexpr int kPer = kTW * kTH / 256;
  float sr[kPer], sg[kPer], sb[kPer], ws = 0.0f;
  int at[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    sr[k] = sg[k] = sb[k] = 0.0f;
    const int o = tid + k * 256;
    at[k] = (o / kTW) * sw + o % kTW;
  }
  const int step = kVert ? sw : 1;
  for (int i = 0, off = 0; i <= 2 * radius; ++i, off += step) {
    const float wt = wts[i];
    ws += wt;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const float4 c = sm_tile[at[k] + off];
      sr[k] = fmaf(c.x, wt, sr[k]);
      sg[k] = fmaf(c.y, wt, sg[k]);
      sb[k] = fmaf(c.z, wt, sb[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int o = tid + k * 256, x = x0 + o % kTW, y = y0 + o / kTW;
    if (x >= w || y >= h) continue;
    float r = sr[k] / ws, g = sg[k] / ws, b = sb[k] / ws;
    if (out_srgb) r = linear_to_srgb(r), g = linear_to_srgb(g), b = linear_to_srgb(b);
    dst[(size_t)y * w + x] = finish(r, g, b, quantize);
  }
}
constexpr size_t kMaxTileBytes = 96 << 10;  // two blocks per SM; wider halos keep the kernel without a tile
constexpr size_t blur_axis_smem(bool vert, int radius) {
  return (size_t)(vert ? 32 * (32 + 2 * radius) : 8 * (128 + 2 * radius)) * 16 + (2 * (size_t)radius + 1) * 4;
}

// depth_aware_blur.wgsl:12-53: (2r+1)^2 window, spatial / colour / depth
// Gaussian weights (sigmas 10, 0.5, 0.5), out-of-image neighbours weigh 0
__global__ void k_depth_blur(const float4* __restrict__ color, const float4* __restrict__ depth,
                             float4* __restrict__ dst, int w, int h, int radius, int quantize) {
  const int x = blockIdx.x * 16 + threadIdx.x, y = blockIdx.y * 16 + threadIdx.y;
  if (x >= w || y >= h) return;
  const float4 cc = __ldg(color + (size_t)y * w + x);
  const float cd = __ldg(depth + (size_t)y * w + x).x;
  const float ss = 10.0f, sc = 0.5f, sd = 0.5f;
  float sr = 0.0f, sg = 0.0f, sb = 0.0f, sw = 0.0f;
  for (int dy = -radius; dy <= radius; ++dy)
    for (int dx = -radius; dx <= radius; ++dx) {
      const int nx = x + dx, ny = y + dy;
      const bool in = nx >= 0 && nx < w && ny >= 0 && ny < h;
      const int sx = min(max(nx, 0), w - 1), sy = min(max(ny, 0), h - 1);
      const float4 nc = __ldg(color + (size_t)sy * w + sx);
      const float nd = __ldg(depth + (size_t)sy * w + sx).x;
      const float d2 = (float)(dx * dx + dy * dy);
      const float er = nc.x - cc.x, eg = nc.y - cc.y, eb = nc.z - cc.z;
      const float dc2 = er * er + eg * eg + eb * eb;
      const float dd2 = (nd - cd) * (nd - cd);
      const float wr = expf(-d2 / (2.0f * ss * ss)) * expf(-dc2 / (2.0f * sc * sc)) * expf(-dd2 / (2.0f * sd * sd));
      const float wt = in ? wr : 0.0f;
      sr += nc.x * wt;
      sg += nc.y * wt;
      sb += nc.z * wt;
      sw += wt;
    }
  const float inv = fmaxf(sw, 1e-5f);
  dst[(size_t)y * w + x] = finish(sr / inv, sg / inv, sb / inv, quantize);
}

// k_depth_blur's sums in its order from a shared-memory tile: 32 x 16 pixels
// and halo with the depth beside the colour (one 16-byte load per tap), two
// vertically adjacent pixels per thread (a tap's load serves both, at two
// values of dy), the spatial weights from a table.  Two exponentials per tap
// remain and bound it (packed arithmetic for the two pixels gained nothing).
// kEdge: the halo leaves the image, so taps are tested.  1024 x 768, radius 4: 167
// -> 89 us.
template <bool kEdge>
__device__ __forceinline__ void depth_blur_tile(const float4* tile, const float* spatial, int radius, int sw, int lx,
                                                int ly, int x, int y, int w, int h, float4* __restrict__ dst,
                                                int quantize) {
  const float sc = 0.5f, sd = 0.5f;
  const float4 c0 = tile[(ly + radius) * sw + lx + radius], c1 = tile[(ly + 1 + radius) * sw + lx + radius];
  float s0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  auto tap = [&](const float4& n, const float4& c, float es, bool in, float (&s)[4]) {
    const float er = n.x - c.x, eg = n.y - c.y, eb = n.z - c.z;
    const float dc2 = er * er + eg * eg + eb * eb;
    const float dd2 = (n.w - c.w) * (n.w - c.w);
    const float wr = es * expf(-dc2 / (2.0f * sc * sc)) * expf(-dd2 / (2.0f * sd * sd));
    const float wt = !kEdge || in ? wr : 0.0f;
    s[0] = fmaf(n.x, wt, s[0]);
    s[1] = fmaf(n.y, wt, s[1]);
    s[2] = fmaf(n.z, wt, s[2]);
    s[3] += wt;
  };
  // rows y - radius + r: dy = r - radius for the upper pixel, one less for the lower
  const int d = 2 * radius + 1;
  auto row_taps = [&](int r, bool up, bool down) {
    const float4* row = tile + (ly + r) * sw + lx;
    const float* es = spatial + r * d;
    const int ny = y + r - radius;
    const bool in_y = ny >= 0 && ny < h;
#pragma unroll 3
    for (int i = 0; i < d; ++i) {
      const float4 n = row[i];
      const int nx = x + i - radius;
      const bool in = in_y && nx >= 0 && nx < w;
      if (up) tap(n, c0, es[i], in, s0);
      if (down) tap(n, c1, es[i - d], in, s1);
    }
  };
  row_taps(0, true, false);
  for (int r = 1; r < d; ++r) row_taps(r, true, true);
  row_taps(d, false, true);
  auto put = [&](int yy, const float (&s)[4]) {
    if (x >= w || yy >= h) return;
    const float inv = fmaxf(s[3], 1e-5f);
    dst[(size_t)yy * w + x] = finish(s[0] / inv, s[1] / inv, s[2] / inv, quantize);
  };
  put(y, s0);
  put(y + 1, s1);
}
__global__ void __launch_bounds__(256) k_depth_blur_tiled(const float4* __restrict__ color,
                                                          const float4* __restrict__ depth, float4* __restrict__ dst,
                                                          int w, int h, int radius, int quantize) {
  extern __shared__ float4 sm_tile[];
  const int sw = 32 + 2 * radius, sh = 16 + 2 * radius, d = 2 * radius + 1;
  float* spatial = reinterpret_cast<float*>(sm_tile + sw * sh);
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 16, tid = threadIdx.x;
  const float ss = 10.0f;
  for (int i = tid; i < d * d; i += 256) {
    const int dy = i / d - radius, dx = i % d - radius;
    spatial[i] = expf(-(float)(dx * dx + dy * dy) / (2.0f * ss * ss));
  }
  for (int e = tid; e < sw * sh; e += 256) {
    const int ly = e / sw, lx = e - ly * sw;
    const size_t g = (size_t)min(max(y0 + ly - radius, 0), h - 1) * w + min(max(x0 + lx - radius, 0), w - 1);
    float4 c = __ldg(color + g);
    c.w = __ldg(&depth[g].x);
    sm_tile[e] = c;
  }
  __syncthreads();
  const int lx = tid & 31, ly = 2 * (tid >> 5);
  const bool edge = x0 < radius || y0 < radius || x0 + 32 + radius > w || y0 + 16 + radius > h;
  if (edge) depth_blur_tile<true>(sm_tile, spatial, radius, sw, lx, ly, x0 + lx, y0 + ly, w, h, dst, quantize);
  else depth_blur_tile<false>(sm_tile, spatial, radius, sw, lx, ly, x0 + lx, y0 + ly, w, h, dst, quantize);
}
constexpr size_t depth_blur_smem(int radius) {
  return (size_t)(32 + 2 * radius) * (16 + 2 * radius) * 16 + (2 * (size_t)radius + 1) * (2 * radius + 1) * 4;
}

// splat_edge.wgsl:13-44: Sobel magnitude of the depth, edge-clamped, through
// smoothstep(thr_min, thr_max, .)
__global__ void k_edge(const float4* __restrict__ depth, float4* __restrict__ dst, int w, int h, float tmin,
                       float tmax, int quantize) {
  const int x = blockIdx.x * 16 + threadIdx.x, y = blockIdx.y * 16 + threadIdx.y;
  if (x >= w || y >= h) return;
  auto at = [&](int ox, int oy) {
    const int cx = min(max(x + ox, 0), w - 1), cy = min(max(y + oy, 0), h - 1);
    return __ldg(depth + (size_t)cy * w + cx).x;
  };
  const float tl = at(-1, -1), tc = at(0, -1), tr = at(1, -1), ml = at(-1, 0), mr = at(1, 0);
  const float bl = at(-1, 1), bc = at(0, 1), br = at(1, 1);
  const float gx = -tl - 2.0f * ml - bl + tr + 2.0f * mr + br;
  const float gy = -tl - 2.0f * tc - tr + bl + 2.0f * bc + br;
  const float e = sqrtf(gx * gx + gy * gy);
  const float t = fminf(fmaxf((e - tmin) / (tmax - tmin), 0.0f), 1.0f);
  const float v = t * t * (3.0f - 2.0f * t);
  dst[(size_t)y * w + x] = finish(v, v, v, quantize);
}

}  // namespace tgt
}  // namespace nps

using namespace nps;

namespace {
int check_image(nps_ctx* ctx, const void* a, const void* b, const void* out, uint32_t w, uint32_t h) {
  if (!ctx || !a || !b || !out || w == 0 || h == 0 || w > 65536 || h > 65536) {
    set_error("target pass: bad arguments");
    return NPS_ERR_INVALID;
  }
  if ((((uintptr_t)a | (uintptr_t)b | (uintptr_t)out) & 15) != 0) {
    set_error("target pass: images must be 16-byte aligned float4 arrays");
    return NPS_ERR_INVALID;
  }
  return bind_device(ctx);
}
}  // namespace

extern "C" {

int nps_blur(nps_ctx* ctx, const float* src_rgba, float* dst_rgba, uint32_t w, uint32_t h, int32_t dir_x,
             int32_t dir_y, int32_t radius, uint32_t flags, float sigma, int quantize) {
  NPS_TRY(check_image(ctx, src_rgba, src_rgba, dst_rgba, w, h));
  if (radius < 0 || radius > 1024 || !(sigma > 0.0f) || src_rgba == dst_rgba) {
    set_error("nps_blur: radius in [0, 1024], sigma > 0, distinct source and destination");
    return NPS_ERR_INVALID;
  }
  // one of the two passes of the separable blur, with a halo that fits in a tile?
  const bool vert = dir_x == 0;
  const size_t smem = tgt::blur_axis_smem(vert, radius);
  if ((vert ? dir_y == 1 : dir_x == 1 && dir_y == 0) && smem <= tgt::kMaxTileBytes) {
    if (vert) {
      NPS_CUDA(cudaFuncSetAttribute(tgt::k_blur_axis<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tgt::kMaxTileBytes));
      tgt::k_blur_axis<true><<<dim3(div_up(w, 32), div_up(h, 32)), 256, smem, ctx->stream>>>(
          (const float4*)src_rgba, (float4*)dst_rgba, (int)w, (int)h, radius, flags, sigma, quantize);
    } else {
      NPS_CUDA(cudaFuncSetAttribute(tgt::k_blur_axis<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tgt::kMaxTileBytes));
      tgt::k_blur_axis<false><<<dim3(div_up(w, 128), div_up(h, 8)), 256, smem, ctx->stream>>>(
          (const float4*)src_rgba, (float4*)dst_rgba, (int)w, (int)h, radius, flags, sigma, quantize);
    }
    NPS_CHECK_LAUNCH();
    return NPS_OK;
  }
  const dim3 grid(div_up(w, 16), div_up(h, 16));
  tgt::k_blur<<<grid, dim3(16, 16), 0, ctx->stream>>>((const float4*)src_rgba, (float4*)dst_rgba, (int)w, (int)h,
                                                      dir_x, dir_y, radius, flags, sigma, quantize);
  NPS_CHECK_LAUNCH();
  return NPS_OK;
}

int nps_depth_aware_blur(nps_ctx* ctx, const float* color_rgba, const float* depth_rgba, float* dst_rgba, uint32_t w,
                         uint32_t h, int32_t radius, int quantize) {
  NPS_TRY(check_image(ctx, color_rgba, depth_rgba, dst_rgba, w, h));
  if (radius < 0 || radius > 64 || color_rgba == dst_rgba) {
    set_error("nps_depth_aware_blur: radius in [0, 64], distinct source and destination");
    return NPS_ERR_INVALID;
  }
  const size_t smem = tgt::depth_blur_smem(radius);
  if (smem <= tgt::kMaxTileBytes) {  // radius up to 25
    NPS_CUDA(cudaFuncSetAttribute(tgt::k_depth_blur_tiled, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)tgt::kMaxTileBytes));
    tgt::k_depth_blur_tiled<<<dim3(div_up(w, 32), div_up(h, 16)), 256, smem, ctx->stream>>>(
        (const float4*)color_rgba, (const float4*)depth_rgba, (float4*)dst_rgba, (int)w, (int)h, radius, quantize);
    NPS_CHECK_LAUNCH();
    return NPS_OK;
  }
  const dim3 grid(div_up(w, 16), div_up(h, 16));
  tgt::k_depth_blur<<<grid, dim3(16, 16), 0, ctx->stream>>>((const float4*)color_rgba, (const float4*)depth_rgba,
                                                            (float4*)dst_rgba, (int)w, (int)h, radius, quantize);
  NPS_CHECK_LAUNCH();
  return NPS_OK;
}

int nps_splat_edge(nps_ctx* ctx, const float* depth_rgba, float* dst_rgba, uint32_t w, uint32_t h, float thr_min,
                   float thr_max, int quantize) {
  NPS_TRY(check_image(ctx, depth_rgba, depth_rgba, dst_rgba, w, h));
  if (depth_rgba == dst_rgba) {
    set_error("nps_splat_edge: distinct source and destination");
    return NPS_ERR_INVALID;
  }
  const dim3 grid(div_up(w, 16), div_up(h, 16));
  tgt::k_edge<<<grid, dim3(16, 16), 0, ctx->stream>>>((const float4*)depth_rgba, (float4*)dst_rgba, (int)w, (int)h,
                                                      thr_min, thr_max, quantize);
  NPS_CHECK_LAUNCH();
  return NPS_OK;
}

}  // extern "C"
