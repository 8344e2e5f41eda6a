// pool.h - device blocks kept by a context between uploads.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <map>
#include <unordered_map>

namespace shiro_gpu {

// Scene uploads and importance-table builds take and give back up to 140
// device blocks each (an upload of 327 k triangles spent 9 ms in cudaMalloc
// and cudaFree).  A context keeps the blocks given back, up to kMaxIdle bytes,
// and hands them out again; they return to the driver past that bound, when an
// allocation of the context fails, at shiro_gpu_trim, and with the context.
// Within a call a block is used on the context's stream alone, whose order
// makes the next use follow the last one.  Between calls, which the caller serialises, the
// stream may become another one (shiro_gpu_set_stream): so every call that
// takes blocks or gives some back, or reads the scene's, has waited for its
// stream when it returns, also when it failed, and no block that is idle or
// replaced by the next upload is still in use.
class DevicePool {
  public:
    static constexpr size_t kMaxIdle = size_t(1) << 30;

    DevicePool() = default;
    DevicePool(const DevicePool&) = delete;
    DevicePool& operator=(const DevicePool&) = delete;
    ~DevicePool() { trim(0); }

    cudaError_t get(void** out, size_t bytes) {
        const size_t exact = steps(bytes, 512);
        size_t size = exact > kMaxIdle ? exact : round(bytes);  // what is never kept needs no common size
        auto it = idle_.lower_bound(size);
        if (it != idle_.end() && it->first <= size + size / 4) {
            *out = it->second;
            live_[it->second] = it->first;
            liveBytes_ += it->first;
            idleBytes_ -= it->first;
            idle_.erase(it);
            return cudaSuccess;
        }
        cudaError_t e = cudaMalloc(out, size);
        if (e != cudaSuccess) {
            cudaGetLastError();
            trim(0);
            size = exact;
            e = cudaMalloc(out, size);
        }
        if (e == cudaSuccess) {
            live_[*out] = size;
            liveBytes_ += size;
        } else {
            cudaGetLastError();  // reported by the return value alone: a later launch's check must not find it
            *out = nullptr;
        }
        return e;
    }

    void put(void* p) {
        if (!p) return;
        const auto it = live_.find(p);
        if (it == live_.end()) return;
        idle_.emplace(it->second, p);
        idleBytes_ += it->second;
        liveBytes_ -= it->second;
        live_.erase(it);
        trim(kMaxIdle);
    }

    // Returns idle blocks, largest first, until at most `keep` bytes are idle.
    void trim(size_t keep) {
        while (idleBytes_ > keep) {
            const auto it = std::prev(idle_.end());
            idleBytes_ -= it->first;
            cudaFree(it->second);
            idle_.erase(it);
        }
    }

    // Device bytes of the blocks handed out and of the idle ones.
    size_t bytes() const { return liveBytes_ + idleBytes_; }

  private:
    static size_t steps(size_t bytes, size_t step) { return (std::max<size_t>(bytes, 16) + step - 1) / step * step; }
    // 512-byte steps, then an eighth of the power of two below: blocks of
    // similar size are interchangeable
    static size_t round(size_t bytes) {
        size_t step = 512;
        while (step * 16 < bytes) step <<= 1;
        return steps(bytes, step);
    }
    std::multimap<size_t, void*> idle_;
    std::unordered_map<void*, size_t> live_;
    size_t idleBytes_ = 0, liveBytes_ = 0;
};

}  // namespace shiro_gpu
