// launch_table.h — resident blocks of the persistent kernels (host code, no
// CUDA calls of its own).
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>

namespace solrt {

// Threads of the largest resident grid per SM, and the stack entries of each
// kept in Context::deep_stack: those from the smallest number of shared slots
// up.
constexpr uint32_t kMaxThreadsPerSm = 1536;
constexpr uint32_t kMinStackSlots = 12;

// Blocks of `block` threads per SM of a persistent launch of which `fits` are
// resident: no more than deep_stack has entries for.
inline int resident_blocks(int fits, uint32_t block) {
    return std::min(std::max(fits, 1), (int)(kMaxThreadsPerSm / block));
}

}  // namespace solrt
