// pf_superres.cuh - the upscale kernel's launch interface (pf_superres.cu),
// shared with the chain on super-resolved frames (pf_api.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "goav1pf.h"

namespace pf {

// One frame to upscale: device planes of the coded frame, and either the
// upscaled planes or the restoration boundary lines (`boundaries` slots a
// plane, 0 where there are none) they are resampled into.
struct SrFrame {
  const pf_frame* coded;
  int up_width;
  const uint8_t* src[3];
  int64_t sstride[3];
  uint8_t* dst[3];
  int64_t dstride[3];
  int boundaries[3];
};

cudaError_t superres_upload_tables();
// Upscales n frames (lines: their boundary lines), several frames a launch.
cudaError_t launch_superres(const SrFrame* frames, int n, bool lines, cudaStream_t st);

}  // namespace pf
