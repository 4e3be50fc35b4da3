// Device staging memory of the calls that take host buffers and keep nothing between calls.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace lvbgs {

// Stream-ordered allocation on `device` from a memory pool of this library; give it back with cudaFreeAsync on
// the same stream. The device's default pool returns its memory to the driver at every synchronisation, so that
// each call paid for a new mapping (100 us and more); this one keeps at most kStagingKeep bytes a device and
// returns the rest at the next synchronisation. Safe from several threads and streams, as the pool is.
constexpr size_t kStagingKeep = (size_t)32 << 20;
cudaError_t staging_alloc(int device, void** out, size_t bytes, cudaStream_t st);

}  // namespace lvbgs
