// Bounded waits on shared-memory mbarriers, of the kernels on the tcgen05 tensor cores: a wait that runs out says so, and its kernel ends with a poisoned result.
#pragma once

#include <cstdint>

namespace b200kv {

constexpr uint32_t kSpin = 1u << 20;

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: false if the phase did not complete within the spin limit.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t spin = 0; spin < kSpin; ++spin)
        if (mbar_try(bar, parity)) return true;
    return false;
}
// Bounded wait of a whole warp for two phases, asked for together: all lanes go on or none.
__device__ __forceinline__ bool mbar_wait_both(uint32_t bar_a, uint32_t parity_a, uint32_t bar_b, uint32_t parity_b) {
    bool ok = false;
    for (uint32_t spin = 0; spin < kSpin && !ok; ++spin) {
        const bool a = mbar_try(bar_a, parity_a), b = mbar_try(bar_b, parity_b);
        ok = a && b;
    }
    return __all_sync(0xffffffffu, ok);
}
// The same of single lanes.
__device__ __forceinline__ bool mbar_wait_both_lane(uint32_t bar_a, uint32_t parity_a, uint32_t bar_b, uint32_t parity_b) {
    for (uint32_t spin = 0; spin < kSpin; ++spin) {
        const bool a = mbar_try(bar_a, parity_a), b = mbar_try(bar_b, parity_b);
        if (a && b) return true;
    }
    return false;
}

}  // namespace b200kv
