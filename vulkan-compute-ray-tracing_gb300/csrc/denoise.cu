// smartDeNoise as a CUDA pass over an RGBA32F image: the filter the
// reference's post-process shader defines (post-process-shader.frag:26-68,
// after BrutPitt's glslSmartDeNoise) and leaves switched off in main()
// (frag:73 blends it 50/50 with the unfiltered pixel in the commented line).
//
// Per pixel: a circular kernel of radius round(kSigma * sigma); for each
// column x in [-radius, radius] the rows run y = -pt, -pt + 1, ... <= pt with
// pt = sqrt(radius^2 - x^2), so most taps fall between two texel rows. Each
// tap is weighted by a spatial Gaussian exp(-|d|^2 / (2 sigma^2)) / (pi 2
// sigma^2) and a range Gaussian of its RGBA distance to the centre pixel,
// exp(-|dC|^2 / (2 threshold^2)) / (sqrt(2 pi) threshold); the result is the
// weighted mean. Taps are fetched the way the reference's sampler does
// (linear filter, REPEAT wrap: src/memory/Image.cpp:353-357), here in texel
// space: position (px + x, py + y), bilinear between the four texels around
// it, indices wrapped modulo the image size. Every operation is a separately
// rounded fp32 step in shader order, as in the oracle's restatement; only
// expf/sqrtf come from CUDA's library.
#include <cuda_runtime.h>

#include <cmath>

#include "rt_internal.h"
#include "rt_math.cuh"

namespace rtgb {
namespace {

struct DenoiseParams {
  float radius, rad_q, inv_sigma_q2, inv_sigma_q2pi, inv_thr_q2, inv_thr_sqrt2pi, mix;
};

__device__ __forceinline__ float4 texel(const float4 *__restrict__ img, int x, int y, int W, int H) {
  x %= W;
  y %= H;
  if (x < 0) x += W;
  if (y < 0) y += H;
  return __ldg(img + (size_t)y * W + x);
}

__device__ __forceinline__ float lerp_rn(float a, float b, float w) {
  return __fadd_rn(__fmul_rn(__fsub_rn(1.0f, w), a), __fmul_rn(w, b));
}

__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float w) {
  return make_float4(lerp_rn(a.x, b.x, w), lerp_rn(a.y, b.y, w), lerp_rn(a.z, b.z, w), lerp_rn(a.w, b.w, w));
}

// One pixel, every tap fetched from the image.
__device__ __forceinline__ void denoise_pixel(const float4 *__restrict__ in, int W, int H, const DenoiseParams &p,
                                              int px, int py, float4 *__restrict__ out) {
  const float4 c = in[(size_t)py * W + px];
  float z = 0.0f;
  float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (float x = -p.radius; x <= p.radius; x = __fadd_rn(x, 1.0f)) {
    const float pt = __fsqrt_rn(__fsub_rn(p.rad_q, __fmul_rn(x, x)));
    for (float y = -pt; y <= pt; y = __fadd_rn(y, 1.0f)) {
      const float dd = __fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y));
      const float blur = __fmul_rn(expf(__fmul_rn(-dd, p.inv_sigma_q2)), p.inv_sigma_q2pi);
      // Bilinear tap at texel-space position (px + x, py + y).
      const float s = __fadd_rn((float)px, x), t = __fadd_rn((float)py, y);
      const float fs = floorf(s), ft = floorf(t);
      const float al = __fsub_rn(s, fs), be = __fsub_rn(t, ft);
      const int i0 = (int)fs, j0 = (int)ft;
      const float4 w = lerp4(lerp4(texel(in, i0, j0, W, H), texel(in, i0 + 1, j0, W, H), al),
                             lerp4(texel(in, i0, j0 + 1, W, H), texel(in, i0 + 1, j0 + 1, W, H), al), be);
      const float dx = __fsub_rn(w.x, c.x), dy = __fsub_rn(w.y, c.y), dz = __fsub_rn(w.z, c.z),
                  dw = __fsub_rn(w.w, c.w);
      const float dc2 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)),
                                  __fmul_rn(dw, dw));
      const float delta =
          __fmul_rn(__fmul_rn(expf(__fmul_rn(-dc2, p.inv_thr_q2)), p.inv_thr_sqrt2pi), blur);
      z = __fadd_rn(z, delta);
      a.x = __fadd_rn(a.x, __fmul_rn(delta, w.x));
      a.y = __fadd_rn(a.y, __fmul_rn(delta, w.y));
      a.z = __fadd_rn(a.z, __fmul_rn(delta, w.z));
      a.w = __fadd_rn(a.w, __fmul_rn(delta, w.w));
    }
  }
  const float4 f = make_float4(__fdiv_rn(a.x, z), __fdiv_rn(a.y, z), __fdiv_rn(a.z, z), __fdiv_rn(a.w, z));
  out[(size_t)py * W + px] = lerp4(c, f, p.mix);
}

// As a call, for the tile kernel: its own loop keeps its registers.
__device__ __noinline__ void denoise_pixel_call(const float4 *__restrict__ in, int W, int H, const DenoiseParams &p,
                                                int px, int py, float4 *__restrict__ out) {
  denoise_pixel(in, W, H, p, px, py, out);
}

// Radii above kTileRadius, and small images.
__global__ void k_denoise(const float4 *__restrict__ in, int W, int H, DenoiseParams p, float4 *__restrict__ out) {
  const int px = blockIdx.x * blockDim.x + threadIdx.x, py = blockIdx.y * blockDim.y + threadIdx.y;
  if (px < W && py < H) denoise_pixel(in, W, H, p, px, py, out);
}

// The same from shared memory, for radii up to kTileRadius: a CTA takes 64 x
// kTileRows pixels, a warp a row, a lane two pixels of it. The texels a CTA
// needs are loaded once, with the wrap; a tap's spatial weight depends only on
// the tap, and its two texel rows and their weights only on the tap and the
// pixel row, so a table holds them; taps down a column share a texel row. The
// columns' positions are whole texels (their linear weight is 0): the second
// texel of that direction only counts where 0 * texel is not 0, so a CTA that
// sees a texel that is not finite takes denoise_pixel. Four channels are two
// packed pairs, each operation rounded as in denoise_pixel: the results are
// its, bit for bit. Issue-bound (about 40 instructions a tap): 1920 x 1080 at
// radius 4 in 219 us, 627 us with every tap fetched and weighted by itself
// (four wrapped loads and two exponentials).
constexpr int kTileRadius = 8, kTileRows = 16, kTileCols = 64, kMaxTaps = 205;  // taps at kTileRadius

struct Tap {
  float upper, lower;  // weights of the two texel rows
  float blur;          // spatial weight
  int row;             // first texel row in the tile, times the pitch
};

__host__ __device__ __forceinline__ int tile_pitch(int radius) { return kTileCols + 2 * radius + 1; }
__host__ __device__ __forceinline__ size_t tile_smem(int radius, int taps) {
  return sizeof(float4) * (size_t)tile_pitch(radius) * (kTileRows + 2 * radius + 2) +
         sizeof(Tap) * (size_t)taps * kTileRows + 2 * sizeof(float) * taps;
}

// One pixel's running sums.
struct TapSum {
  f2 cxy, czw;  // the pixel itself
  f2 uxy, uzw;  // the tap's upper texel row
  f2 axy, azw;
  float z;
};
__device__ __forceinline__ void upper_row(TapSum &s, float4 u) {
  s.uxy = pk2(u.x, u.y);
  s.uzw = pk2(u.z, u.w);
}
__device__ __forceinline__ void add_tap(TapSum &s, const Tap &q, float4 l, const DenoiseParams &p) {
  const f2 lxy = pk2(l.x, l.y), lzw = pk2(l.z, l.w);
  const f2 up = pk2(q.upper, q.upper), low = pk2(q.lower, q.lower);
  const f2 wxy = add2(mul2_add(up, s.uxy), mul2_add(low, lxy)), wzw = add2(mul2_add(up, s.uzw), mul2_add(low, lzw));
  s.uxy = lxy;
  s.uzw = lzw;
  const f2 dxy = sub2(wxy, s.cxy), dzw = sub2(wzw, s.czw);
  const f2 sxy = mul2(dxy, dxy), szw = mul2(dzw, dzw);
  const float dc2 = __fadd_rn(__fadd_rn(__fadd_rn(lo2(sxy), hi2(sxy)), lo2(szw)), hi2(szw));
  const float delta = __fmul_rn(__fmul_rn(expf(__fmul_rn(-dc2, p.inv_thr_q2)), p.inv_thr_sqrt2pi), q.blur);
  const f2 dd = pk2(delta, delta);
  s.z = __fadd_rn(s.z, delta);
  s.axy = add2(s.axy, mul2_add(dd, wxy));
  s.azw = add2(s.azw, mul2_add(dd, wzw));
}

__global__ void __launch_bounds__(32 * kTileRows, 2) k_denoise_tile(const float4 *__restrict__ in, int W, int H,
                                                                    DenoiseParams p, int radius, int taps,
                                                                    float4 *__restrict__ out) {
  extern __shared__ __align__(16) unsigned char s_mem[];
  __shared__ int s_beg[2 * kTileRadius + 2];
  const int lane = threadIdx.x, warp = threadIdx.y, tid = warp * 32 + lane;
  const int pitch = tile_pitch(radius), rows = kTileRows + 2 * radius + 2, columns = 2 * radius + 1;
  float4 *s_tex = reinterpret_cast<float4 *>(s_mem);
  Tap *s_tap = reinterpret_cast<Tap *>(s_tex + pitch * rows);
  float *s_y = reinterpret_cast<float *>(s_tap + taps * kTileRows), *s_blur = s_y + taps;
  const int x0 = blockIdx.x * kTileCols, y0 = blockIdx.y * kTileRows;
  bool finite = true;
  for (int r = warp; r < rows; r += kTileRows) {
    for (int c = lane; c < pitch; c += 32) {
      const float4 t = texel(in, x0 - radius + c, y0 - radius + r, W, H);
      s_tex[r * pitch + c] = t;
      finite = finite && fabsf(t.x) < 1e37f && fabsf(t.y) < 1e37f && fabsf(t.z) < 1e37f && fabsf(t.w) < 1e37f;
    }
  }
  // Columns, one a thread: y = -pt, -pt + 1, ... as the loop adds them up.
  if (tid <= columns) {
    int k = 0;
    for (int c = 0; c < tid; c++) {
      const float x = (float)(c - radius), pt = __fsqrt_rn(__fsub_rn(p.rad_q, __fmul_rn(x, x)));
      for (float y = -pt; y <= pt; y = __fadd_rn(y, 1.0f)) {
        if (c == tid - 1 && k < taps) {
          const float dd = __fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y));
          s_y[k] = y;
          s_blur[k] = __fmul_rn(expf(__fmul_rn(-dd, p.inv_sigma_q2)), p.inv_sigma_q2pi);
        }
        k++;
      }
    }
    s_beg[tid] = min(k, taps);
  }
  const int py = y0 + warp;
  if (!__syncthreads_and(finite)) {
    for (int px = x0 + lane; px < min(W, x0 + kTileCols); px += 32)
      if (py < H) denoise_pixel_call(in, W, H, p, px, py, out);
    return;
  }
  // This warp's row of the table.
  Tap *tap = s_tap + taps * warp;
  for (int k = lane; k < taps; k += 32) {
    const float t = __fadd_rn((float)py, s_y[k]), ft = floorf(t), be = __fsub_rn(t, ft);
    tap[k] = Tap{__fsub_rn(1.0f, be), be, s_blur[k], ((int)ft - (y0 - radius)) * pitch};
  }
  __syncwarp();
  if (py >= H) return;
  TapSum s[2];
  float4 c[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    c[i] = s_tex[(warp + radius) * pitch + radius + lane + 32 * i];
    s[i].cxy = pk2(c[i].x, c[i].y);
    s[i].czw = pk2(c[i].z, c[i].w);
    s[i].axy = s[i].azw = s[i].uxy = s[i].uzw = pk2(0.0f, 0.0f);
    s[i].z = 0.0f;
  }
  for (int col = 0; col < columns; col++) {
    const float4 *tex = s_tex + lane + col;
    int next = -1;
    const int end = s_beg[col + 1];
    for (int k = s_beg[col]; k < end; k++) {
      const Tap q = tap[k];
      if (q.row != next) {
        upper_row(s[0], tex[q.row]);
        upper_row(s[1], tex[q.row + 32]);
      }
      next = q.row + pitch;
      add_tap(s[0], q, tex[next], p);
      add_tap(s[1], q, tex[next + 32], p);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int px = x0 + lane + 32 * i;
    if (px >= W) continue;
    const float4 f = make_float4(__fdiv_rn(lo2(s[i].axy), s[i].z), __fdiv_rn(hi2(s[i].axy), s[i].z),
                                 __fdiv_rn(lo2(s[i].azw), s[i].z), __fdiv_rn(hi2(s[i].azw), s[i].z));
    out[(size_t)py * W + px] = lerp4(c[i], f, p.mix);
  }
}

int g_sms = 0;

}  // namespace

cudaError_t launch_denoise(const float *in, uint32_t W, uint32_t H, float sigma, float ksigma, float threshold,
                           float mix, float *out, cudaStream_t st) {
  if (W == 0 || H == 0) return cudaSuccess;
  // frag:29-36, each constant as one fp32 expression.
  const float kInvPi = 0.31830988618379067154f, kInvSqrt2Pi = 0.39894228040143267794f;
  DenoiseParams p;
  p.radius = roundf(ksigma * sigma);
  p.rad_q = p.radius * p.radius;
  p.inv_sigma_q2 = 0.5f / (sigma * sigma);
  p.inv_sigma_q2pi = kInvPi * p.inv_sigma_q2;
  p.inv_thr_q2 = 0.5f / (threshold * threshold);
  p.inv_thr_sqrt2pi = kInvSqrt2Pi / threshold;
  p.mix = mix;
  const bool tile_radius = p.radius <= (float)kTileRadius;  // not one that is NaN (kSigma 0, sigma infinite)
  const int radius = tile_radius ? (int)p.radius : kTileRadius + 1;
  const dim3 pixels(16, 16), pixel_grid((W + 15) / 16, (H + 15) / 16);
  // An image of at most a 16 x 16 block an SM (two, where a block has few taps)
  // takes as long as one block, and the tile kernel's is longer. us, per pixel /
  // tile: 200 x 150 (130 blocks) radius 2 10.3 / 12.3, 4 20.6 / 24.6, 8 65.8 /
  // 71.8; 33 x 1080 (204) 12.3 / 12.2, 30.6 / 23.6, 98.4 / 71.7; radius 1 256 x
  // 256 (256) 6.2 / 8.3, 384 x 256 (384) 8.2 / 8.3, 640 x 480 16.4 / 10.3.
  if (g_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const uint64_t small = (uint64_t)g_sms * (radius <= 1 ? 2 : 1);
  if (tile_radius && (uint64_t)pixel_grid.x * pixel_grid.y > small) {
    int taps = 0;
    for (float x = -p.radius; x <= p.radius; x += 1.0f) {
      const float pt = std::sqrt(p.rad_q - x * x);
      for (float y = -pt; y <= pt; y += 1.0f) taps++;
    }
    const size_t smem = tile_smem(radius, taps);
    // One limit for every radius: calls from several threads set the same.
    const cudaError_t e = cudaFuncSetAttribute(k_denoise_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)tile_smem(kTileRadius, kMaxTaps));
    if (e != cudaSuccess) return e;
    const dim3 block(32, kTileRows), grid((W + kTileCols - 1) / kTileCols, (H + kTileRows - 1) / kTileRows);
    k_denoise_tile<<<grid, block, smem, st>>>(reinterpret_cast<const float4 *>(in), (int)W, (int)H, p, radius, taps,
                                              reinterpret_cast<float4 *>(out));
    return cudaGetLastError();
  }
  k_denoise<<<pixel_grid, pixels, 0, st>>>(reinterpret_cast<const float4 *>(in), (int)W, (int)H, p,
                                     reinterpret_cast<float4 *>(out));
  return cudaGetLastError();
}

}  // namespace rtgb
