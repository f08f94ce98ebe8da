// attention_ring.h -- what the slots of the prompt kernel's ring hold, and which are filled again (attention_prefill_mma.cu;
// no CUDA needed).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LUX_HOST_DEVICE __host__ __device__
#else
#define LUX_HOST_DEVICE
#endif

namespace luxcuda {

struct RingEntry {
    uint32_t tile;
    bool is_v;
};

// Entry i of 2 tiles: K0, K1, V0, K2, V1, ..., the order in which the products read them.
LUX_HOST_DEVICE constexpr RingEntry ring_entry(uint32_t i, uint32_t tiles) {
    if (i == 0) return {0u, false};
    if (i + 1u == 2u * tiles) return {tiles - 1u, true};
    return i & 1u ? RingEntry{(i + 1u) / 2u, false} : RingEntry{i / 2u - 1u, true};
}
// Whether the slot of entry i is filled again after it.
LUX_HOST_DEVICE constexpr bool ring_refilled(uint32_t i, uint32_t entries, uint32_t slots) { return i + slots < entries; }

}  // namespace luxcuda
