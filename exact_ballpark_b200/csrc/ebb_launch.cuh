// SPDX-License-Identifier: MIT
// Launches whose shared memory is sized by the call.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace ebb {

// A block gets 48 KB of shared memory unless its kernel has opted in to more, its static arrays (the torque tables, a
// tile's counters) among them. So a launch opts in whenever its dynamic bytes leave less than STATIC_ROOM of the 48 KB: more
// than any such kernel's static arrays (416 bytes at most), and opting in early costs nothing.
constexpr size_t DEFAULT_SHARED = 48 * 1024, STATIC_ROOM = 1024;

template <class K>
cudaError_t allow_shared(K kernel, size_t dynamic) {
    if (dynamic + STATIC_ROOM <= DEFAULT_SHARED) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dynamic);
}

}  // namespace ebb
