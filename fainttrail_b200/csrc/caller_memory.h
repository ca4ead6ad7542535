// Whose memory a caller's device pointer is.
#pragma once

#include <cuda_runtime_api.h>

namespace ftb {

// Whether kernels on `device` may read and write a caller's buffer in place: that GPU's own
// memory, or managed memory. What else unified addressing reaches (another GPU's memory,
// which needs peer access in a kernel, or page-locked host memory) goes through copies.
inline bool in_place(const cudaPointerAttributes& a, int device) {
    return a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeDevice && a.device == device);
}

}  // namespace ftb
