// Device staging memory of the calls that take host buffers and keep nothing between calls.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace lvbgs {

// Stream-ordered allocation on `device` from a memory pool of this library; give it back with cudaFreeAsync on
// the same stream. The device's default pool returns its memory to the driver at every synchronisation, so that
// each call paid for a new mapping (100 us and more); this one keeps at most kStagingKeep bytes a device and
// returns the rest at the next synchronisation. Safe from several threads and streams, as the pool is.
constexpr size_t kStagingKeep = (size_t)32 << 20;
cudaError_t staging_alloc(int device, void** out, size_t bytes, cudaStream_t st);

// Whether a kernel on `device` may use the buffer p (with the attributes a) where it is: managed memory or this
// device's own, at a multiple of `align`. Another device's memory would need peer access, which nothing here enables.
inline bool usable_in_place(const cudaPointerAttributes& a, int device, const void* p, size_t align) {
    const bool here = a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeDevice && a.device == device);
    return here && (uintptr_t)p % align == 0;
}
inline bool ranges_overlap(const void* a, size_t na, const void* b, size_t nb) {
    return (uintptr_t)a < (uintptr_t)b + nb && (uintptr_t)b < (uintptr_t)a + na;
}

}  // namespace lvbgs
