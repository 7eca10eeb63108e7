// mega.h -- the persistent render kernel (mega.cu), launched by render.cu.
#pragma once

#include <cuda_runtime.h>

#include "render_common.cuh"

namespace trg {

// Material kinds (bit per MAT_* kind) and features one instantiation of the
// persistent kernel handles; the host picks the smallest that covers a set.
enum : unsigned {
  MK_PHONG = 1u << MAT_PHONG,
  MK_DISNEY12 = 1u << MAT_DISNEY12,
  MK_GLASS = 1u << MAT_GLASS,
  MK_METAL = 1u << MAT_METAL,
  MK_DISNEY15 = 1u << MAT_DISNEY15,
  MK_ENV = 1u << 8,   // an environment light
  MK_MAPS = 1u << 9,  // Phong image maps
};
// Lights of one scene the persistent kernel keeps per-thread state for (the
// remembered occluders); sets with more render with the wavefront.
constexpr int kMegaLights = 16;

struct MegaLaunch {
  DScene sc;
  const JobDev* jobs;
  int njobs, nslots;
  int lanes;             // lanes of a warp that own pixels (1 .. 32)
  DMat* mt;              // sets with image maps: one material set-up per thread of the launch
  int occluder_cache;    // remember each (slot, light)'s last occluder (tr_tuning.occluder_cache)
  unsigned int* fetch;   // next unclaimed path slot (zeroed by the host)
  int* err;              // bit 0: traversal stack overflow; bit 1: a slot ran past its vertex bound
  unsigned long long* stats;  // samples, extend rays, shadow rays, vertices, 4-7 unused, occluder hits (8)
};

// The smallest instantiation covering a scene set (MK_* bits).
unsigned mega_kernel_mask(const DScene& sc, bool has_disney12);
// Threads of a block, of which one is resident per SM: of the usual
// instantiations (128 registers a thread) and of those for few pixels (255).
constexpr int kMegaThreads = 512, kMegaFewThreads = 256;
struct MegaShape {
  int threads, lanes, grid;
};
// Launches the persistent kernel of instantiation `mask` and of the shape's
// block size on `st`.
cudaError_t launch_mega(const MegaLaunch& P, unsigned mask, const MegaShape& shape, cudaStream_t st);

}  // namespace trg
