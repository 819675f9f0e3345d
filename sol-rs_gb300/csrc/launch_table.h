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

// Resident blocks per SM of one kernel, looked up once for each device and
// launch shape: occupancy is a property of the compiled kernel and the device,
// and an attribute that the lookup sets on the kernel holds on that device only.
class LaunchTable {
public:
    static constexpr int kDevices = 64, kShapes = 6;
    // `*blocks` receives the shape's entry for the device; query(int* fits)
    // finds it where it is not known yet. Its status, 0 when known.
    template <class Query>
    auto blocks(int device, int shape, uint32_t block, Query query, int* blocks) -> decltype(query(blocks)) {
        std::atomic<int>* const entry = device >= 0 && device < kDevices ? &table_[device][shape] : nullptr;
        *blocks = entry ? entry->load(std::memory_order_relaxed) : 0;
        if (*blocks) return {};
        int fits = 0;
        const auto s = query(&fits);
        if (s != decltype(s){}) return s;
        *blocks = resident_blocks(fits, block);
        if (entry) entry->store(*blocks, std::memory_order_relaxed);
        return s;
    }

private:
    std::atomic<int> table_[kDevices][kShapes] = {};
};

}  // namespace solrt
