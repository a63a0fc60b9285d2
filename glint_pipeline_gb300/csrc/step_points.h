/*
 * step_points.h -- which of a step's points the kernels read where they lie.
 * Host code only.
 */
#ifndef GLINT_STEP_POINTS_H_
#define GLINT_STEP_POINTS_H_

#include <cuda_runtime_api.h>
#include <stdint.h>

namespace glint {

/* Device memory of the context's own GPU, on the 16-byte boundary that a point
 * is loaded with.  Everything else is copied into the context's buffer first:
 * another GPU's memory, which the copy engine reaches where a kernel would need
 * peer access, managed memory, and points on other boundaries. */
inline bool points_in_place(const cudaPointerAttributes &at, int device, const void *points) {
    return at.type == cudaMemoryTypeDevice && at.device == device && ((uintptr_t)points & 15) == 0;
}

} // namespace glint

#endif
