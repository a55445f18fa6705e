// The start of the grayscale hole fill (fillstart.cu).
#pragma once

#include <cuda_runtime.h>

#include "batch.cuh"
#include "ccl.cuh"

namespace nsgb {

// Writes the start of the erosion reconstruction that fills the holes of `I` (one image, its labelling
// fields set; dtype u8, u16, i32 or f32) into `out` (rows `I.one.pitch` bytes apart).  `f` and `bits`
// (one bit per pixel, bits_bytes) are a labelling's scratch, `ctl` at least kFillCtlBytes, all device
// memory that the caller does not otherwise use.  Enqueues only.
constexpr size_t kFillCtlBytes = 1024;
cudaError_t fill_start_launch(int dtype, const Imgs& I, int c_tiles, const ccl::Forest& f, unsigned* bits,
                              size_t bits_bytes, void* ctl, void* out, int conn, cudaStream_t s);

}  // namespace nsgb
