// render_plain.cu - the plain GPU form: one launch follows every path to its end.
//
// CpuPathTracer::RenderSampleBatch (src/backend/cpu/CpuPathTracer.cpp:
// 2043-2170) loops pixels on host threads and samples inside each pixel; here
// a lane runs the whole estimator of a (pixel, sample) path (camera ray,
// traversal, shading, next-event estimation, Russian roulette), writes a
// 48-byte record and takes the next path.  A second kernel sums each
// pixel's records in sample order, so the batch average is formed with the
// same additions, in the same order, as the reference.
#include <algorithm>

#include "integrator.cuh"
#include "kernels.h"
#include "lanes.cuh"
#include "resolve.cuh"

namespace shiro_gpu {

namespace {

// A warp's lanes pass the steps of a bounce together: the lanes with a path
// trace it to its next vertex, each light sample's shadow rays are traced side
// by side (warp_closest, warp_occluded), and lanes whose path has ended take
// the next path once kPlainRefill of them are idle.  With a thread per path
// that ran on its own, warps came apart at the first branch and stayed apart
// (7.3 of 32 lanes active on the 961x541 15-spp field frame, now 11.8); bound
// by the latency of the tree's loads, the kernel then wants warps in flight
// rather than registers: at 128, 80, 64, 48 and 40 registers a thread (4, 6, 8,
// 10, 12 blocks of 128 per SM) that frame takes 18.6, 16.6, 14.9, 13.6 and 13.0
// ms (19.5 with a thread per path).  Lanes 1, 4, 8 idle: no difference; a warp
// that waits for all its paths takes 15.0 instead of 13.8 ms.  Paths in any
// phase side by side were three times slower: the light samples then run a few
// lanes at a time.
//
// The next limit was instruction fetch (8.4 stall cycles per issue, 7.4 for
// loads): 48 warps at 48 places of a long program.  So the warps of larger
// blocks meet at the starts of a bounce, of its shading and of its
// continuation, and - where the program is longest, with every lobe in - of
// each light sample.  Field frame, 1280x720 2-spp field frame, 640x480 8-spp
// frame with every lobe, 512x512 4-spp sphere: 12.96, 2.08, 10.55 and 1.09 ms
// without; 12.4, 2.00, 8.7 and 0.87 in 5 blocks of 256; 12.7, 2.13, 7.5 and 0.87
// in 3 of 512; there with the light samples 13.3, 2.22, 6.3 and 0.88.
//
// A launch too small to fill kPlainSmall has no use for more warps and keeps
// its registers (256x256 pixels of a sphere: 303 us, 353 with 48 registers); its
// paths spread over all of those blocks' warps, a few lanes of each (96x64
// pixels: 134 us, with 32 a warp 199; 160x120 of every lobe 614 and 738).  How
// far past its resident lanes (77 824 on 152 SMs) that shape stays the better
// one is small_paths below.
enum { kSyncBounce = 1, kSyncHit = 2, kSyncContinue = 4, kSyncLight = 8 };
struct PlainShape {
    uint32_t threads;
    int blocks, sync;
};
constexpr PlainShape kPlainLean{256, 5, kSyncBounce | kSyncHit | kSyncContinue};
constexpr PlainShape kPlainExt{512, 3, kSyncBounce | kSyncHit | kSyncContinue | kSyncLight};
constexpr PlainShape kPlainSmall{128, 4, 0};
constexpr int kPlainRefill = 4;
constexpr uint32_t kPlainChunk = 32;

template <bool kExt, uint32_t kThreads, int kBlocks, int kSync>
__global__ void __launch_bounds__(kThreads, kBlocks) k_plain_paths(const __grid_constant__ DevScene s,
                                                                        const __grid_constant__ DevRequest q,
                                                                        uint64_t pixelBase, uint32_t count,
                                                                        uint32_t perWarp, uint32_t* __restrict__ next,
                                                                        float4* records) {
    NullCounter ctr;
    PathState ps;
    Sampler smp{0u, 0u, 0u, s.radical};
    bool alive = false;
    uint32_t path = 0, depth = 0;
    float depth0 = 0.0f;
    const PathRecords rec(records, count);
    const uint32_t nls = light_sample_count<kExt>(s, q), domeEnd = s.distantCount + s.domeCount * q.domeSamples;
    const float domeDiv = static_cast<float>(q.domeSamples);
    // the first perWarp paths of a warp have its own indices, the rest come from the queue
    const uint32_t warp = (blockIdx.x * kThreads + threadIdx.x) >> 5;
    const uint32_t first = gridDim.x * (kThreads >> 5) * perWarp, queued = count > first ? count - first : 0u;
    uint32_t got = warp * perWarp + lane_id();
    if (lane_id() >= perWarp || got >= count) got = 0xffffffffu;
    LaneFeed feed;
    for (;;) {
        if (got != 0xffffffffu) {
            path = got;
            const uint32_t local = path / q.sampleCount;
            const uint64_t pixel = pixelBase + local;
            const uint64_t y = pixel / q.width;
            smp.px = static_cast<uint32_t>(pixel - y * q.width);
            smp.py = static_cast<uint32_t>(y);
            smp.index = q.sampleStart + (path - local * q.sampleCount);
            init_path(q, smp, ps);
            depth = 0;
            depth0 = __int_as_float(0x7f800000);
            alive = true;
        }
        if constexpr (kSync & kSyncBounce) {
            if (!__syncthreads_or(alive)) break;
        } else {
            if (__ballot_sync(kFull, alive) == 0u) break;
        }
        bool on = alive && q.maxDepth != 0u;
        HitRec h;
        const bool found = warp_closest(s, on, ps.ro, ps.rd, &h);
        if constexpr (kSync & kSyncHit) __syncthreads();
        else __syncwarp();
        bool shaded = false;
        Vertex v;
        if (on) {
            if (!found) {
                add_miss(s, q, ps, depth, ctr);
                on = false;
            } else {
                v = make_vertex(s, ps.ro, ps.rd, h);
                shaded = true;
                if constexpr (kExt) shaded = enter_hit(s, smp, depth, v, h.t, ps);
                if (shaded) {
                    if (depth == 0) {
                        const float4 dc = __ldg(bsdf_rec(s, v.hit.material) + 3);  // DiffuseColor
                        const V3 nn = v.n * 0.5f + V3{0.5f, 0.5f, 0.5f};
                        st_pair(rec.first + path, make_float4(dc.x, dc.y, dc.z, 0.0f), make_float4(nn.x, nn.y, nn.z, 0.0f));
                        depth0 = h.t;
                    }
                    if constexpr (kExt) add_emission(s, v, depth, ps);
                }
            }
        }
        // sum_direct, its shadow rays a sample at a time for the whole warp
        V3 out{0.0f, 0.0f, 0.0f}, acc{0.0f, 0.0f, 0.0f};
        for (uint32_t k = 0;; ++k) {
            if (k > s.distantCount && k <= domeEnd && (k - s.distantCount) % q.domeSamples == 0u) {
                out = out + acc / domeDiv;
                acc = V3{0.0f, 0.0f, 0.0f};
            }
            if (k >= nls) break;
            V3 dir, c;
            float reach = 0.0f;
            if constexpr (kSync & kSyncLight) __syncthreads();
            const bool lit = shaded && light_sample<kExt>(s, q, v, smp, depth, k, &dir, &c, &reach, ctr);
            __syncwarp();
            const bool blocked = warp_occluded(s, lit, shadow_origin(v), dir, reach);
            if (lit && !blocked) {
                if (k >= s.distantCount && k < domeEnd) acc = acc + c;
                else out = out + c;
            }
        }
        if constexpr (kSync & kSyncContinue) __syncthreads();
        else __syncwarp();
        if (shaded) {
            ps.radiance = ps.radiance + ps.T * out;
            on = continue_path<kExt>(s, q, v, smp, depth, ps, ctr);
        }
        if (on) on = ++depth < q.maxDepth;
        if (alive && !on)
            rec.radiance[path] = make_float4(ps.radiance.x, ps.radiance.y, ps.radiance.z, depth0);
        alive = on;
        got = feed_lanes(feed, next, queued, kPlainChunk, alive, kPlainRefill);
        if (got != 0xffffffffu) got += first;
    }
}

__global__ void __launch_bounds__(128) k_resolve(const DevRequest q, uint64_t pixelBase, uint32_t count,
                                                 float4* records, AovPtrs aov) {
    __shared__ float stage[4][96];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = i < count;
    PixelAov px;
    if (on) px = resolve_pixel(PathRecords(records, static_cast<uint64_t>(count) * q.sampleCount),
                               static_cast<uint64_t>(i) * q.sampleCount, q.sampleCount);
    store_pixels(aov, __all_sync(kFull, on) != 0, on, static_cast<size_t>(pixelBase + i), px, stage[threadIdx.x >> 5]);
}

__global__ void k_primary_hits(const DevScene s, const DevRequest q, uint32_t* __restrict__ prim, float* __restrict__ tout) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.width * q.height) return;
    const uint32_t y = i / q.width, x = i - y * q.width;
    const Sampler smp{x, y, q.sampleStart, s.radical};
    V3 o, d;
    camera_ray(q, x, y, smp.next2d(0u), &o, &d);
    HitRec h;
    NullCounter ctr;
    const bool hit = trace_closest(s, o, d, &h, ctr);
    prim[i] = hit ? h.gid : 0xffffffffu;
    tout[i] = hit ? h.t : FLT_MAX;
}

// The closest hit (blockIdx.y 0) and the occlusion of listed rays, perWarp rays a
// warp: fewer than 32 where the rays would leave SMs without a warp.  Bound by
// the latency of each ray's chain of node loads: with both queries one after
// the other in a thread, 32 rays a warp and 89 registers, 1003, 10007, 200003
// and a million rays at a sphere took 50, 58, 141 and 493 us; as two halves of
// the grid, spread, at 48 registers 19, 30, 112 and 449 (at 59 registers, 8
// blocks per SM, 18, 31, 115 and 488; at 40, 12 blocks, 20, 34, 113 and 458).
// Traced warp by warp (warp_closest) they were slower: 164 for 200003.
//
// The tree is the one the caller's width selects, by default the binary one for
// any scene and any number of rays.  Kernel us, binary and wide tree, 1003,
// 10007, 100003 and 1000003 rays: sphere of 4 thousand triangles 20 and 24, 29 and
// 43, 69 and 69, 446 and 507; field of 1.3 million 49 and 52, 74 and 77, 171 and
// 133, 1074 and 958: many rays at a large scene would gain from the wide one.
constexpr int kRayBlocks = 10;
constexpr uint32_t kRayWarpsPerSm = 16;

__global__ void __launch_bounds__(128, kRayBlocks) k_trace_rays(const DevScene s, const float* __restrict__ o,
                                                                const float* __restrict__ d,
                                                                const float* __restrict__ tmax, uint32_t n,
                                                                uint32_t perWarp, uint32_t* __restrict__ prim,
                                                                float* __restrict__ tout, uint32_t* __restrict__ occ) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, i = warp * perWarp + lane_id();
    if (lane_id() >= perWarp || i >= n) return;
    const V3 ro{o[3 * i], o[3 * i + 1], o[3 * i + 2]};
    const V3 rd{d[3 * i], d[3 * i + 1], d[3 * i + 2]};
    NullCounter ctr;
    if (blockIdx.y == 0) {
        HitRec h;
        const bool hit = trace_closest(s, ro, rd, &h, ctr);
        prim[i] = hit ? h.gid : 0xffffffffu;
        tout[i] = hit ? h.t : FLT_MAX;
    } else {
        occ[i] = trace_occluded(s, ro, rd, tmax[i], ctr) ? 1u : 0u;
    }
}

// Work-counting variant: every `stride`-th path of the request, same
// decisions as k_plain_paths; totals accumulated with one atomic per field
// per warp.
__global__ void __launch_bounds__(128) k_count_paths(const DevScene s, const DevRequest q, uint64_t totalPaths,
                                                     uint32_t stride, unsigned long long* __restrict__ totals) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t path = i * stride;
    LocalCounter c;
    uint32_t traced = 0;
    if (path < totalPaths) {
        const uint64_t pixel = path / q.sampleCount;
        const uint32_t smp = static_cast<uint32_t>(path - pixel * q.sampleCount);
        const uint32_t y = static_cast<uint32_t>(pixel / q.width);
        const uint32_t x = static_cast<uint32_t>(pixel - static_cast<uint64_t>(y) * q.width);
        trace_path<true>(s, q, x, y, q.sampleStart + smp, c);
        traced = 1;
    }
    const uint32_t v[12] = {traced,  c.closestRays, c.occlusionRays, c.nodes + c.onodes, c.tris + c.otris, c.hits,
                            c.envEvals, c.envSamples, c.bsdfEvals, c.bsdfPdfs, c.onodes, c.otris};
    for (int k = 0; k < 12; ++k) {
        unsigned long long x = v[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(&totals[k], x);
    }
}

__global__ void k_qmc_table(float* __restrict__ table) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < 24u * kQmcTable) table[e] = qmc_radical_dim(e / kQmcTable, e % kQmcTable);
}

// The sampler of the kernels on explicit tuples (diagnostic).
__global__ void k_sample_probe(const uint4* __restrict__ tuples, uint32_t n, const float* __restrict__ table,
                               float* __restrict__ out) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint4 t = tuples[k];
    const V2 v = Sampler{t.x, t.y, t.z, table}.next2d(t.w);
    out[2 * static_cast<size_t>(k)] = v.x;
    out[2 * static_cast<size_t>(k) + 1] = v.y;
}

// Listed paths of the plain form (diagnostic): out[10 i ..] = radiance,
// albedo, normal, depth of path (pixels[i], sample index sampleIdx[i]).
template <bool kExt>
__global__ void __launch_bounds__(128) k_render_paths(const DevScene s, const DevRequest q, const uint32_t* __restrict__ pixels,
                                                      const uint32_t* __restrict__ sampleIdx, uint32_t n,
                                                      float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t y = pixels[i] / q.width, x = pixels[i] - y * q.width;
    NullCounter ctr;
    const PathResult r = trace_path<kExt>(s, q, x, y, sampleIdx[i], ctr);
    float* o = out + 10 * static_cast<size_t>(i);
    o[0] = r.radiance.x;
    o[1] = r.radiance.y;
    o[2] = r.radiance.z;
    o[3] = r.albedo.x;
    o[4] = r.albedo.y;
    o[5] = r.albedo.z;
    o[6] = r.normal.x;
    o[7] = r.normal.y;
    o[8] = r.normal.z;
    o[9] = r.depth;
}

// Texel picks of a dome texture for explicit 2-D points (diagnostic).
__global__ void k_env_pick(const DevEnv e, const float2* __restrict__ u, uint32_t n, uint32_t useCdf,
                           uint32_t* __restrict__ texel, float* __restrict__ pdf) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 v = u[i];
    const size_t t = env_pick(e, V2{v.x, v.y}, useCdf != 0u);
    texel[i] = static_cast<uint32_t>(t);
    pdf[i] = e.samples[2 * t].w;
}

inline unsigned grid(uint64_t n, unsigned b) { return static_cast<unsigned>((n + b - 1) / b); }

}  // namespace

void launch_sample_probe(const uint4* tuples, uint32_t n, const float* table, float* out, cudaStream_t stream) {
    if (n == 0) return;
    k_sample_probe<<<grid(n, 256), 256, 0, stream>>>(tuples, n, table, out);
}

void launch_qmc_table(float* table, cudaStream_t stream) {
    k_qmc_table<<<grid(24u * kQmcTable, 256), 256, 0, stream>>>(table);
}

template <bool kExt, const PlainShape& kShape>
static void launch_plain(const DevScene& s, const DevRequest& q, uint64_t pixelBase, uint32_t count, uint32_t perWarp,
                         unsigned maxBlocks, float4* records, cudaStream_t stream) {
    const unsigned blocks = grid(count, kShape.threads / 32u * perWarp), resident = std::min(blocks, maxBlocks);
    uint32_t* next = s.error + 1;  // the path queue's counter
    if (resident < blocks) cudaMemsetAsync(next, 0, sizeof(uint32_t), stream);
    k_plain_paths<kExt, kShape.threads, kShape.blocks, kShape.sync>
        <<<resident, kShape.threads, 0, stream>>>(s, q, pixelBase, count, perWarp, next, records);
}

// Launches of at most this many paths take kPlainSmall, a path per lane and as
// many blocks as that makes; `lanes` are its resident ones.  With few paths per
// resident lane the larger shapes have no queue to refill lanes from, and what
// is left is each path's own latency, which fewer registers and the meetings of
// a block lengthen, the more the deeper the paths and the less of their time is
// the traversal of a large tree.  Kernel us, kPlainSmall and
// the larger shape, four samples a pixel: field of 256 objects, depth 3, 100
// thousand paths 507 and 603, 140 thousand 701 and 673, 180 thousand 794 and 745;
// field of 16, depth 4, 140 thousand 315 and 361, 180 thousand 345 and 417;
// sphere, depth 4, 140 thousand 256 and 291, 200 thousand 295 and 310; depth 12,
// field of 256, 200 thousand 1042 and 1077, 230 thousand 1064 and 964; field of
// 16, 200 thousand 434 and 522; sphere, 200 thousand 379 and 430.
// With the extended lobes in, the larger shape pays early where shading is most
// of the work (every lobe in 36 thousand triangles, depth 4: of the time of a
// thread per path, 100 thousand paths 0.70 and 0.79, 135 thousand 0.66 and 0.66,
// 175 thousand 0.70 and 0.61; depth 12: 0.87 and 1.07, 0.74 and 0.88, 0.77 and
// 0.78) and late in larger scenes (a field of 64 objects, one of them emitting:
// 100 thousand 0.95 and 1.46, 195 thousand 0.95 and 1.17, 270 thousand 0.93 and
// 1.06; a transmitting one in a field of 256: 100 thousand 0.91 and 1.23, 195
// thousand 0.88 and 0.85).
static uint64_t small_paths(const DevScene& s, const DevRequest& q, uint64_t lanes) {
    const bool large = s.triCount >= (s.extended ? 1u << 16 : 1u << 18), deep = q.maxDepth > (!s.extended && !large ? 4u : 6u);
    if (s.extended) return large ? lanes * 3u : lanes * (deep ? 4u : 3u) / 2u;
    return deep ? lanes * 3u : large ? lanes * 2u : lanes * 5u / 2u;
}

void launch_plain_paths(const DevScene& s, const DevRequest& q, uint64_t pathBase, uint32_t count, float4* records,
                        cudaStream_t stream) {
    if (count == 0) return;
    int device = 0, sms = 1;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const uint64_t pixelBase = pathBase / q.sampleCount;
    const auto resident = [&](const PlainShape& p) { return static_cast<unsigned>(p.blocks * sms); };
    const uint32_t smallWarps = resident(kPlainSmall) * kPlainSmall.threads / 32u;
    if (count <= small_paths(s, q, 32ull * smallWarps)) {
        const uint32_t perWarp = std::min(32u, (count + smallWarps - 1u) / smallWarps);
        if (s.extended) launch_plain<true, kPlainSmall>(s, q, pixelBase, count, perWarp, ~0u, records, stream);
        else launch_plain<false, kPlainSmall>(s, q, pixelBase, count, perWarp, ~0u, records, stream);
    } else {
        if (s.extended) launch_plain<true, kPlainExt>(s, q, pixelBase, count, 32u, resident(kPlainExt), records, stream);
        else launch_plain<false, kPlainLean>(s, q, pixelBase, count, 32u, resident(kPlainLean), records, stream);
    }
}

void launch_render_paths(const DevScene& s, const DevRequest& q, const uint32_t* pixels, const uint32_t* sampleIdx,
                         uint32_t n, float* out, cudaStream_t stream) {
    if (n == 0) return;
    if (s.extended)
        k_render_paths<true><<<grid(n, 128), 128, 0, stream>>>(s, q, pixels, sampleIdx, n, out);
    else
        k_render_paths<false><<<grid(n, 128), 128, 0, stream>>>(s, q, pixels, sampleIdx, n, out);
}

void launch_env_pick(const DevEnv& e, const float2* u, uint32_t n, bool useCdf, uint32_t* texel, float* pdf,
                     cudaStream_t stream) {
    if (n == 0) return;
    k_env_pick<<<grid(n, 256), 256, 0, stream>>>(e, u, n, useCdf ? 1u : 0u, texel, pdf);
}

// Loads an instance and launches it over no paths (it reads no scene then), so
// that the driver has sized its thread-local memory for it.
template <bool kExt, const PlainShape& kShape>
static cudaError_t preload_plain(cudaStream_t stream) {
    k_plain_paths<kExt, kShape.threads, kShape.blocks, kShape.sync>
        <<<1, kShape.threads, 0, stream>>>(DevScene{}, DevRequest{}, 0, 0u, 32u, nullptr, nullptr);
    return cudaGetLastError();
}

// The shapes keep 960 to 1440 bytes a thread (their registers differ), and the
// size of a launch chooses one: without this the first large frame after a
// small one took 65 (lean) to 120 MB (extended) of device memory more.
cudaError_t preload_plain_kernels(cudaStream_t stream) {
    cudaFuncAttributes a;
    cudaError_t e = preload_plain<false, kPlainLean>(stream);
    if (e == cudaSuccess) e = preload_plain<true, kPlainExt>(stream);
    if (e == cudaSuccess) e = preload_plain<false, kPlainSmall>(stream);
    if (e == cudaSuccess) e = preload_plain<true, kPlainSmall>(stream);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_resolve);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e;
}

void launch_resolve_pixels(const DevRequest& q, uint64_t pixelBase, uint32_t count, float4* records, AovPtrs aov,
                           cudaStream_t stream) {
    if (count == 0) return;
    k_resolve<<<grid(count, 128), 128, 0, stream>>>(q, pixelBase, count, records, aov);
}

void launch_primary_hits(const DevScene& s, const DevRequest& q, uint32_t* prim, float* t, cudaStream_t stream) {
    const uint64_t n = static_cast<uint64_t>(q.width) * q.height;
    if (n == 0) return;
    k_primary_hits<<<grid(n, 128), 128, 0, stream>>>(s, q, prim, t);
}

void launch_count_paths(const DevScene& s, const DevRequest& q, uint32_t stride, unsigned long long* totals,
                        cudaStream_t stream) {
    const uint64_t total = static_cast<uint64_t>(q.width) * q.height * q.sampleCount;
    const uint64_t n = (total + stride - 1) / stride;
    if (n == 0) return;
    k_count_paths<<<grid(n, 128), 128, 0, stream>>>(s, q, total, stride, totals);
}

void launch_trace_rays(const DevScene& s, const float* o, const float* d, const float* tmax, uint32_t n, uint32_t* prim,
                       float* t, uint32_t* occ, cudaStream_t stream) {
    if (n == 0) return;
    int device = 0, sms = 1;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const uint32_t warps = static_cast<uint32_t>(sms) * kRayWarpsPerSm;
    const uint32_t perWarp = std::min(32u, n / warps + 1u);
    k_trace_rays<<<dim3(grid(n, 4 * perWarp), 2), 128, 0, stream>>>(s, o, d, tmax, n, perWarp, prim, t, occ);
}

}  // namespace shiro_gpu
