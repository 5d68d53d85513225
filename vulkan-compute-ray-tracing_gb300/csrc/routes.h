// Which kernels take a call, by its sizes alone. Host code without CUDA, so
// that the rules are tested on a CPU; results are the same on every route.
#pragma once
#include <stdint.h>

#include <algorithm>

#include "rtgb/rt_api.h"

namespace rtgb {

// Renders of fewer pixels can fall back from a form that takes scratch to the
// megakernel in one launch: a fixed size, whatever the tuning. From here up the
// wavefront is the faster form of every call by so much that its scratch is a
// condition (1024 x 1024, 12K triangles, 4 samples: 546 / 837 Mrays/s).
constexpr uint64_t kOneLaunchPixels = 1u << 18;

constexpr uint64_t kWavefrontPixels = 1u << 17;

// Render launch-shape knobs (rtSetTuning "render.mode").
struct RenderOpts {
  int mode = 2;  // 0 megakernel, 1 wavefront, 2 choose by image size, 3 choose, without the wavefront
  // mode 2, at this value: calls of one sample run as a wavefront from 2^17 pixels up
  // (below, paths.cu up to 65,536 and the megakernel between), calls of
  // several samples always: the samples share a wave, where the megakernel's
  // threads run them one after the other. Megakernel / wavefront, Cornell box
  // of 1K, 12K, 100K triangles, mesh of 512K, 8 bounces, 1 sample, us: 288 x
  // 288 386 / 409, 1005 / 843, 1752 / 1497, 800 / 589; 352 x 352 459 / 458,
  // 1256 / 950, 2367 / 1664, 967 / 677; 511 x 512 842 / 573, 2285 / 1334, 3920
  // / 2238, 1300 / 806. 4 samples, 12K: 48 x 48 2354 / 983, 512 x 512 8897 /
  // 4344.
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
// True when a render of these params goes to the wavefront kernels.
inline bool use_wavefront(const RenderOpts &o, const rt_render_params &p) {
  if (p.flags & RT_COMPAT_STACK16) return false;  // the literal 16-entry traversal is megakernel-only
  const uint64_t pixels = (uint64_t)p.width * p.height;
  if (pixels >= (1ull << 31)) return false;
  if (o.mode != 2) return o.mode == 1;
  return pixels >= o.wavefront_pixels || (o.wavefront_pixels == kWavefrontPixels && p.spp > 1);
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
