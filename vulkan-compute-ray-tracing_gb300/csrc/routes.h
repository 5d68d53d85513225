// Which kernels take a call, by its sizes alone. Host code without CUDA, so
// that the rules are tested on a CPU; results are the same on every route.
#pragma once
#include <stdint.h>

#include <algorithm>

#include "rtgb/rt_api.h"

namespace rtgb {

// Batches of fewer than this many rays, and of fewer than 3/2 of the triangles,
// are cast as they are, in input order: sorting them and tracing packets pays
// where many camera rays meet each triangle. us, cast as they are / sorted and
// in packets, camera rays into an icosphere: 1,280 triangles 1.05M rays 207 /
// 231, 2.1M 381 / 374; 5,120 triangles 0.79M 203 / 200, 1.05M 257 / 237; 82K
// 0.79M 362 / 300, 1.05M 456 / 336; 328K 1.05M 773 / 788; 1.31M triangles 1.05M
// 1523 / 2478, 1.9M 2585 / 2923, 2.1M 2835 / 3016, 3M 3947 / 3852; into a grid
// mesh of 2.05M triangles 3.1M 915 / 1013. Random rays are cast as they are on
// either side, above the line after the 0.05 ms that finding out takes, so the
// line is drawn at 7/8 only where casts in packets on the reference's tree were
// clearly quicker (82K triangles 0.79M 356, 0.92M 382, 20K 1.05M 290; 5,120 1.05M
// 250): between 10,000 and 100,000 triangles. Beside another batch packets' fewer
// instructions count for more: two of 1.05M into 1.31M triangles 2848 / 3249, of
// 1.9M 4992 / 4574. The chunks of a host batch always run so (2 x 4.19M through
// host arrays from two threads, chunks of 2.1M: 767 / 950 Mrays/s) and keep the
// plain line.
constexpr uint32_t kPacketMinRays = 1u << 20;
inline bool direct_rays(uint32_t ntris, uint32_t n, uint32_t packet_min_rays, bool overlapped) {
  uint64_t line = packet_min_rays;
  if (ntris >= 10000 && ntris < 100000)
    line = line * 7 / 8;
  else if (!overlapped)
    line = std::max(line, line * 3 * ntris / (2 * kPacketMinRays));
  return n < line;
}

// Renders of fewer pixels can fall back from a form that takes scratch to the
// megakernel in one launch: a fixed size, whatever the tuning. From here up the
// wavefront is the faster form of every call by so much that its scratch is a
// condition (1024 x 1024, 12K triangles, 4 samples: 546 / 837 Mrays/s).
constexpr uint64_t kOneLaunchPixels = 1u << 18;

// Calls of several samples below that size run as a wavefront from this many
// samples up (~0: never), else as the megakernel. A wavefront runs the samples
// side by side, where the megakernel's threads run them one after the other,
// but pays three launches a bounce (about 15 us) whether paths are left or not:
// it wants triangles enough to make a path's steps dear, or samples enough, the
// more the longer the paths may be and the fewer triangles there are. us,
// megakernel / wavefront, 256 x 256, 8 bounces: Cornell box of 12 triangles, 2
// samples 119 / 219, 16 (128 x 128) 655 / 257; of 312, 2 samples 292 / 346, 8
// and 4 bounces with 4 samples 587 / 423 and 304 / 246; of 1K, 2 samples 495 /
// 456; of 12K 1488 / 912; an icosphere in the open of 320, 2 samples 93 / 193, 4
// (4 bounces) 109 / 128, 8 (128 x 128) 213 / 197; of 5120, 2 samples 284 / 288.
// One bounce, 2 samples: 1K 32 / 44, 16 x 16 91 / 35, 12K 84 / 90. Of images of
// few pixels, or narrower than a tile of 8 x 4, most lanes are idle: 4096 x 1, 2
// samples, 12K 24 / 139, 100K 375 / 232.
inline uint64_t wave_min_samples(uint32_t ntris, const rt_render_params &p) {
  const uint64_t pixels = (uint64_t)p.width * p.height, bounces = p.max_bounces, never = ~0ull;
  if (pixels < 64 || (p.height < 4 && ntris < 50000) || (p.width < 8 && (ntris < 1000 || bounces <= 1))) return never;
  if (bounces <= 1) return ntris >= 10000 || (ntris >= 1000 && pixels <= 1024) ? 2 : 16;
  if (ntris >= 1000) return 2;
  return ntris >= 100 ? std::max<uint64_t>(4, bounces) : 4 * bounces;
}

// Calls of one sample run in paths.cu up to this many pixels (tile positions,
// of an image narrower than a tile), else in the megakernel: a warp's pools
// shorten a path's chain of steps, which few triangles make short anyway, and
// cost more the fuller the GPU is. us, megakernel / paths.cu, 8 bounces: Cornell
// box of 12 triangles 64 x 64 57 / 59, 256 x 256 70 / 150; of 32, 32 x 32 67 /
// 55; of 112, 96 x 96 92 / 86, 180 x 180 98 / 129; of 1K, 180 x 180 223 / 198,
// 256 x 256 266 / 325 and with 3 bounces 106 / 180 (the megakernel on the
// reference's tree 406 and 153: the line keeps clear of what was slower than
// that); of 3K, 96 x 96 361 / 140, 256 x 256 433 / 463; of 12K, 256 x 256 740 /
// 714. One bounce: of 312, 32 x 32 28 / 18, 128 x 128 20 / 30; of 1K, 128 x 128 30
// / 35, 180 x 180 28 / 41. Wide images, whose side rays leave the scene sooner,
// take less: 443 x 110, 3K, 2 bounces 102 / 74 (221 x 221 101 / 126); 1024 x 48, 1K,
// 8 bounces 216 / 129, 1 bounce 41 / 28. One pixel, 5120 triangles: 8 / 10.
constexpr uint64_t kPathsMinPixels = 8;
inline uint64_t paths_max_pixels(uint32_t ntris, const rt_render_params &p) {
  const uint32_t bounces = p.max_bounces;
  const bool wide = p.width >= 4ull * p.height;
  if (ntris < 30) return 0;
  if (ntris < 100) return 1u << 10;
  if (ntris < 1000) return bounces <= 1 ? 1u << 11 : 10000;
  if (ntris >= 10000 || wide || bounces >= (ntris < 3000 ? 5 : 4)) return 1u << 16;
  return bounces <= 1 && ntris < 3000 ? 1u << 14 : 1u << 15;
}
inline bool paths_fit(uint32_t ntris, const rt_render_params &p) {
  const uint64_t pixels = (uint64_t)p.width * p.height;
  const bool thin = p.width < 8 || p.height < 4;
  const uint64_t extent = thin ? (uint64_t)((p.width + 7) / 8) * ((p.height + 3) / 4) * 32 : pixels;
  return pixels >= kPathsMinPixels && extent <= paths_max_pixels(ntris, p);
}

constexpr uint64_t kWavefrontPixels = 1u << 17;
constexpr uint32_t kWavefrontTris = 1000;

// Render launch-shape knobs (rtSetTuning "render.mode").
struct RenderOpts {
  int mode = 2;  // 0 megakernel, 1 wavefront, 2 choose by sizes, 3 choose, without the wavefront
  // mode 2, at this value: every call is a wavefront from kOneLaunchPixels up;
  // below, those of several samples by wave_min_samples, those of one from this
  // many pixels up in scenes of kWavefrontTris, the rest in paths.cu (paths_fit)
  // or the megakernel. One sample, 8 bounces, us, megakernel / wavefront: 380 x
  // 380, Cornell box of 112 triangles 210 / 299, 312 294 / 356, 1K 480 / 466,
  // 12K 1264 / 939, an icosphere of 320 86 / 200; 511 x 512, 100K 3920 / 2238, a
  // mesh of 512K 1300 / 806.
  // Any other value is the caller's own line, for calls of any number of
  // samples (2^31: never).
  uint64_t wavefront_pixels = kWavefrontPixels;
  int batch_streams = 16;                // side streams a batch spreads its wavefront jobs over (1..16)
  // Batches and the render server: jobs from this many pixels up run as
  // wavefronts on side streams (the rest in the persistent tile launch).
  // Jobs that run side by side keep the GPU busy at any size, and queued
  // bounce rays in the 8-wide caster beat the megakernel's diverged lanes,
  // so all of them do by default; a render alone keeps wavefront_pixels.
  uint64_t batch_wavefront_pixels = 1;
  // Wavefront renders: reorder each bounce's rays by Morton key of origin and
  // direction before casting them (1) or cast them in queue order (0). The
  // queue keeps the shading warps' order, which is close to the camera
  // tiles' order, and the 8-wide caster takes them faster unsorted; the
  // closest-hit entry points keep trace.sort.
  int sort = 0;
};
// True when a render of a scene of ntris triangles goes to the wavefront kernels.
inline bool use_wavefront(const RenderOpts &o, uint32_t ntris, const rt_render_params &p) {
  if (p.flags & RT_COMPAT_STACK16) return false;  // the literal 16-entry traversal is megakernel-only
  const uint64_t pixels = (uint64_t)p.width * p.height;
  if (pixels >= (1ull << 31)) return false;
  if (o.mode != 2) return o.mode == 1;
  if (o.wavefront_pixels != kWavefrontPixels) return pixels >= o.wavefront_pixels;
  if (pixels >= kOneLaunchPixels) return true;
  return p.spp > 1 ? p.spp >= wave_min_samples(ntris, p) : pixels >= kWavefrontPixels && ntris >= kWavefrontTris;
}
// True when a job of a batch or a server step goes to the wavefront kernels.
inline bool use_wavefront_batched(const RenderOpts &o, const rt_render_params &p) {
  if (p.flags & RT_COMPAT_STACK16) return false;
  const uint64_t pixels = (uint64_t)p.width * p.height;
  return pixels < (1ull << 31) && (o.mode == 1 || (o.mode == 2 && pixels >= o.batch_wavefront_pixels));
}
// True when a render that cannot have scratch runs as the megakernel instead.
inline bool one_launch_fallback(const RenderOpts &o, const rt_render_params &p) {
  return o.mode >= 2 && (uint64_t)p.width * p.height < std::max(kOneLaunchPixels, o.wavefront_pixels);
}

}  // namespace rtgb
