// lanes.cuh - lane-level work distribution of the persistent kernels.
#pragma once

#include <cstdint>

namespace shiro_gpu {

constexpr uint32_t kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// A warp claims kChunk queue entries with one atomicAdd and hands them to its
// lanes; once `refillIdle` lanes have finished their entries they take the
// next ones, so a warp is not held back by its slowest entry.
struct LaneFeed {
    uint32_t next = 0, end = 0;  // the warp's claimed entries [next, end)
    bool exhausted = false;
};

// Assigns queue entries to idle lanes (`has` false); warp-uniform call.
// Returns the entry index this lane received, or 0xffffffff.
template <uint32_t kChunk>
__device__ __forceinline__ uint32_t feed_lanes(LaneFeed& f, uint32_t* counter, uint32_t count, bool has, int refillIdle) {
    const uint32_t lane = lane_id();
    uint32_t got = 0xffffffffu;
    uint32_t idle = __ballot_sync(kFull, !has);
    if (f.exhausted || __popc(idle) < refillIdle) return got;
    while (idle != 0u) {
        if (f.next >= f.end) {
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(counter, kChunk);
            b = __shfl_sync(kFull, b, 0);
            if (b >= count) {
                f.exhausted = true;
                break;
            }
            f.next = b;
            f.end = min(b + kChunk, count);
        }
        const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
        const uint32_t take = min(f.end - f.next, static_cast<uint32_t>(__popc(idle)));
        if (((idle >> lane) & 1u) && rank < take) got = f.next + rank;
        f.next += take;
        idle = __ballot_sync(kFull, !has && got == 0xffffffffu);
    }
    return got;
}

}  // namespace shiro_gpu
