// lanes.cuh - lane-level work distribution of the persistent kernels.
#pragma once

#include <cstdint>

namespace shiro_gpu {

constexpr uint32_t kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// How a resident grid's warps share a queue of `count` entries: the lanes of a
// warp that take entries, and how many it claims at a time.  A queue shorter
// than the grid's lanes spreads over all warps, a few lanes of each (one ray
// traced alone ends sooner than 32 that wait for one another's branches), and
// chunks stay small until a warp has several to claim.  With 64 entries a claim
// for any queue, half of the warps of a 65536-ray launch had nothing to do and
// the others two rays a lane: previews of 64x64, 130x127 and 256x256 pixels
// took 0.295, 0.333 and 0.358 ms on the device, now 0.214, 0.245 and 0.295; a
// 256x256 16-spp frame, whose last bounces are short queues, 1.35, now 1.12;
// the 1080p field frame 92.2, now 90.7.  At least 4, 8 or 16 lanes a warp: 0.234,
// 0.253 and 0.252 ms for 64x64.  Claims of 32 throughout: field 91.7 ms.
struct WarpShare {
    uint32_t lanes, chunk;
};

__device__ __forceinline__ WarpShare warp_share(uint32_t count) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), per = (count + warps - 1u) / warps;
    const uint32_t lanes = min(max(per, 1u), 32u);
    return WarpShare{lanes, per >= 512u ? 64u : lanes};
}

// A warp claims `chunk` queue entries with one atomicAdd and hands them to its
// lanes; once `refillIdle` lanes have finished their entries they take the
// next ones, so a warp is not held back by its slowest entry.
struct LaneFeed {
    uint32_t next = 0, end = 0;  // the warp's claimed entries [next, end)
    bool exhausted = false;
};

// Assigns queue entries to idle lanes (`has` false); warp-uniform call.
// Returns the entry index this lane received, or 0xffffffff.
__device__ __forceinline__ uint32_t feed_lanes(LaneFeed& f, uint32_t* counter, uint32_t count, uint32_t chunk, bool has, int refillIdle) {
    const uint32_t lane = lane_id();
    uint32_t got = 0xffffffffu;
    uint32_t idle = __ballot_sync(kFull, !has);
    if (f.exhausted || __popc(idle) < refillIdle) return got;
    while (idle != 0u) {
        if (f.next >= f.end) {
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(counter, chunk);
            b = __shfl_sync(kFull, b, 0);
            if (b >= count) {
                f.exhausted = true;
                break;
            }
            f.next = b;
            f.end = min(b + chunk, count);
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
