// resolve.cuh - path records averaged into the AOV planes.
//
// A pixel's records are summed in sample order, with the additions of
// CpuPathTracer::RenderSampleBatch (src/backend/cpu/CpuPathTracer.cpp:
// 2093-2137).
#pragma once

#include <cmath>

#include "common.cuh"
#include "kernels.h"
#include "lanes.cuh"

namespace shiro_gpu {

// The records of `paths` paths in one block: the (albedo, 0), (normal, 0) pairs
// of all, then the (radiance, depth) of all.  Most paths write the two parts in
// different stages, and averaging reads the second alone of paths that hit
// nothing: as three float4 a path, each end of a path wrote half a sector.
// (1080p x64 field frame 90.7 -> 89.7 ms, 24 uneven frames 30.6 -> 30.1, the
// plain form's 961x541 15-spp frame 13.1 -> 12.95.)
struct PathRecords {
    F4Pair* first;
    float4* radiance;
    __device__ __forceinline__ PathRecords(float4* base, uint64_t paths)
        : first(reinterpret_cast<F4Pair*>(base)), radiance(base + 2 * paths) {}
};

struct PixelAov {
    float4 beauty;
    V3 albedo, normal;
    float depth;
};

struct PixelSum {
    float b0 = 0.0f, b1 = 0.0f, b2 = 0.0f, b3 = 0.0f, depth = HUGE_VALF;  // +inf
    V3 alb{0.0f, 0.0f, 0.0f}, nrm{0.0f, 0.0f, 0.0f};

    __device__ __forceinline__ static bool hit(const float4& a) { return a.w < __int_as_float(0x7f800000); }

    // Albedo and normal (b, c) of a path whose first ray missed are zero
    // (adding them changes nothing) and not in the record.
    __device__ __forceinline__ void add(const float4& a, const float4& b, const float4& c) {
        b0 = b0 + a.x;
        b1 = b1 + a.y;
        b2 = b2 + a.z;
        b3 = b3 + (hit(a) ? 1.0f : 0.0f);
        if (hit(a)) {
            alb = alb + V3{b.x, b.y, b.z};
            nrm = nrm + V3{c.x, c.y, c.z};
        }
        if (a.w < depth) depth = a.w;
    }
};

// The average of a pixel's n records, the loads of kResolveBatch records in
// flight at a time (measured with records of three float4: one at a time 304
// and 399 us where four took 297 and 379, a 1279x719 4-spp frame and a wave of
// uneven frames; eight 288 and 369, but 25 instead of 17 us for two samples a
// pixel).
constexpr uint32_t kResolveBatch = 4;

__device__ __forceinline__ PixelAov resolve_pixel(const PathRecords& r, uint64_t path, uint32_t n) {
    const float4* __restrict__ rad = r.radiance + path;
    const F4Pair* first = r.first + path;
    PixelSum s;
    uint32_t k = 0;
    for (; k + kResolveBatch <= n; k += kResolveBatch) {
        float4 a[kResolveBatch];
        F4Pair f[kResolveBatch];
#pragma unroll
        for (uint32_t j = 0; j < kResolveBatch; ++j) a[j] = rad[k + j];
#pragma unroll
        for (uint32_t j = 0; j < kResolveBatch; ++j) {
            if (PixelSum::hit(a[j])) f[j] = ld_pair(first + k + j);
        }
#pragma unroll
        for (uint32_t j = 0; j < kResolveBatch; ++j) s.add(a[j], f[j].a, f[j].b);
    }
    for (; k < n; ++k) {
        const float4 a = rad[k];
        F4Pair f{};
        if (PixelSum::hit(a)) f = ld_pair(first + k);
        s.add(a, f.a, f.b);
    }
    const float cnt = static_cast<float>(n);
    const float inv = 1.0f / cnt;
    return PixelAov{make_float4(s.b0 / cnt, s.b1 / cnt, s.b2 / cnt, s.b3 / cnt), s.alb * inv, s.nrm * inv, s.depth};
}

// One float3 plane's part of store_pixels: the lanes' 96 floats in order, as
// three stores of 32 consecutive ones.
__device__ __forceinline__ void store_plane3(float* __restrict__ plane, size_t firstPx, float* stage, const V3& x) {
    const uint32_t lane = lane_id();
    __syncwarp();
    stage[3 * lane + 0] = x.x;
    stage[3 * lane + 1] = x.y;
    stage[3 * lane + 2] = x.z;
    __syncwarp();
    float* o = plane + 3 * firstPx;
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i) o[32 * i + lane] = stage[32 * i + lane];
}

// Writes the pixels of the lanes with `on` (px: the lane's pixel) to the
// planes; all 32 lanes call, `stage` is 96 floats of the warp's own.  Where a
// warp's pixels follow one another, the three-float planes are written through
// it, 32 consecutive floats a store: the planes may lie in page-locked host
// memory, and a lane's three floats at a stride of twelve bytes crossed the
// link as three partial lines (the 40 MB of a 1279x719 frame: 571 us, now 291;
// a device-to-host copy of as many bytes takes 208).
__device__ __forceinline__ void store_pixels(const AovPtrs& aov, bool together, bool on, size_t px, const PixelAov& r,
                                             float* stage) {
    if (on) {
        if ((reinterpret_cast<uintptr_t>(aov.beauty) & 15u) == 0u) {
            reinterpret_cast<float4*>(aov.beauty)[px] = r.beauty;
        } else {
            aov.beauty[4 * px + 0] = r.beauty.x;
            aov.beauty[4 * px + 1] = r.beauty.y;
            aov.beauty[4 * px + 2] = r.beauty.z;
            aov.beauty[4 * px + 3] = r.beauty.w;
        }
        aov.depth[px] = r.depth;
    }
    if (together) {  // 32 consecutive pixels of one frame
        const size_t first = px - lane_id();
        store_plane3(aov.albedo, first, stage, r.albedo);
        store_plane3(aov.normal, first, stage, r.normal);
    } else if (on) {
        aov.albedo[3 * px + 0] = r.albedo.x;
        aov.albedo[3 * px + 1] = r.albedo.y;
        aov.albedo[3 * px + 2] = r.albedo.z;
        aov.normal[3 * px + 0] = r.normal.x;
        aov.normal[3 * px + 1] = r.normal.y;
        aov.normal[3 * px + 2] = r.normal.z;
    }
}

}  // namespace shiro_gpu
