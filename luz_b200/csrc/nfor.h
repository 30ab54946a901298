// NFOR denoiser entry shared by the render path (integrator.cu) and nfor.cu.
#pragma once
#include <cuda_runtime.h>


#include <cstdint>
#include <string>

#include "luz_gpu.h"

// Denoise::applyNFOR (src/core/Denoise/NFOR.cpp:977-1102) on device-resident
// NFOR buffers laid out as LuzNforBuffers; writes width*height*3 doubles to
// d_out in `stream`'s order. settings NULL = NFORSettings defaults.
// Returns LUZ_OK, or a LUZ_E_* code with its message in msg.
int luz_nfor_on_device(const double* color_a, const double* color_b, const double* color_variance,
                       const double* features_a, const double* features_b, const double* feature_variance,
                       int32_t width, int32_t height, const LuzNforSettings* settings, double* d_out, void* stream,
                       std::string& msg);

// Device scratch of single calls (ray batches, NFOR and adaptive buffers, gradients, cache
// rows) comes from one stream-ordered pool per device instead of cudaMalloc: an allocation
// and its release cost 0.6 ms there, and these calls make 3 to 45 of them. The pool keeps at
// most kScratchKeep bytes between calls (what lies above goes back to the device at the next
// synchronisation) and gives all of it back when the last user of the device goes (a scene or
// cache handle, or a denoise under way without one) and when the device refuses this library
// an allocation, which is then tried again. Reuse between streams and threads is ordered by the
// streams' own dependencies.
constexpr unsigned long long kScratchKeep = 3ull << 30;

// `bytes` from the current device's scratch pool in the order of `st`; cudaFreeAsync gives them
// back. What a stream has given back can be trimmed only after a wait for that stream, which
// costs a short call 13 us: the trim waits, for every stream alive that took from the pool.
// `own_wait`: the caller waits itself after giving back (its stream may be capturing when
// another thread trims).
cudaError_t luz_scratch_alloc(void** p, size_t bytes, cudaStream_t st, bool own_wait = false);
// Waits for `st`, which is about to be destroyed, and forgets it.
void luz_scratch_forget(int device, cudaStream_t st);
// A user of the pool of `device` comes and goes; the last one's leaving empties the pool.
void luz_scratch_open(int device);
void luz_scratch_close(int device);
// Gives what the pool of `device` holds idle back to the device.
void luz_scratch_trim(int device);
