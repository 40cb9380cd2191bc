// Device allocations, and the memory of states that are gone.  Only cudaMalloc, cudaFree and cudaGetDevice are called, so that it can be checked on
// the CPU with stand-ins for them.
#pragma once
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstddef>
#include <initializer_list>
#include <mutex>
#include <utility>
#include <vector>

namespace rsv {

// Allocations of states that are gone, for the next ones of the same model (mapping device memory costs up to 4 ms): the last kMost of
// at most kMostBytes each, so a gigabyte per model at most.  Shared by the model, which empties and closes it when it goes, and its states, which may outlive
// it.  All work on a state goes through the model's stream, so the next user's clearing is ordered behind it.  When any allocation of
// this library finds the device full, the pools of all models on that device are emptied first (device_malloc).
class StatePool {
  public:
    static constexpr size_t kMost = 2, kMostBytes = 512u << 20;
    const int device;
    explicit StatePool(int device_) : device(device_) {
        std::lock_guard<std::mutex> lock(registry().mu);
        registry().pools.push_back(this);
    }
    ~StatePool() {
        {
            std::lock_guard<std::mutex> lock(registry().mu);
            auto& p = registry().pools;
            p.erase(std::find(p.begin(), p.end(), this));
        }
        release(true);
    }
    StatePool(const StatePool&) = delete;
    StatePool& operator=(const StatePool&) = delete;
    float* take(size_t bytes) {
        std::lock_guard<std::mutex> lock(mu);
        for (size_t i = 0; i < kept.size(); ++i)
            if (kept[i].first == bytes) {
                float* p = kept[i].second;
                kept.erase(kept.begin() + (long)i);
                return p;
            }
        return nullptr;
    }
    void give(size_t bytes, float* p) {
        std::lock_guard<std::mutex> lock(mu);
        if (open && bytes <= kMostBytes) {
            kept.emplace_back(bytes, p);
            if (kept.size() <= kMost) return;
            p = kept.front().second;
            kept.erase(kept.begin());
        }
        cudaFree(p);
    }
    // Frees what is kept, and with `close` keeps nothing from now on; whether there was anything.
    bool release(bool close) {
        std::lock_guard<std::mutex> lock(mu);
        const bool any = !kept.empty();
        for (auto& k : kept) cudaFree(k.second);
        kept.clear();
        if (close) open = false;
        return any;
    }
    static bool release_device(int device) {
        std::lock_guard<std::mutex> lock(registry().mu);
        bool any = false;
        for (StatePool* p : registry().pools)
            if (p->device == device) any = p->release(false) || any;
        return any;
    }

  private:
    struct Registry {
        std::mutex mu;
        std::vector<StatePool*> pools;
    };
    static Registry& registry() {
        static Registry* r = new Registry;  // (never destroyed: a state may go after the program's static objects)
        return *r;
    }
    std::mutex mu;
    std::vector<std::pair<size_t, float*>> kept;  // newest last
    bool open = true;
};

// cudaMalloc on the current device; where that is full, once more with what the pools of the device have kept.
template <typename T>
cudaError_t device_malloc(T** p, size_t bytes) {
    cudaError_t e = cudaMalloc((void**)p, bytes);
    int device = 0;
    if (e == cudaErrorMemoryAllocation && cudaGetDevice(&device) == cudaSuccess && StatePool::release_device(device)) {
        cudaGetLastError();
        e = cudaMalloc((void**)p, bytes);
    }
    return e;
}

// A work area that grows and that its user can do without: where the device is full, reserve() says so instead of throwing.
class SpareArea {
  public:
    // At least `bytes`, with a quarter on top where there is room for it, so that needs that creep up reallocate a few times only.  `idle` waits for the work
    // on the memory that the area has.  Its contents are lost when it grows.
    template <typename Idle>
    bool reserve(size_t bytes, Idle&& idle) {
        if (bytes <= size) return true;
        if (p) idle();
        release();
        for (size_t want : {bytes + bytes / 4, bytes}) {
            const cudaError_t e = device_malloc(&p, want);
            if (e == cudaSuccess) {
                size = want;
                return true;
            }
            p = nullptr;
            if (e != cudaErrorMemoryAllocation) return false;  // (an earlier failure of the device: the next call that checks reports it)
            cudaGetLastError();
        }
        return false;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        size = 0;
    }
    template <typename T>
    T* as() const {
        return static_cast<T*>(p);
    }
    size_t bytes() const { return size; }

  private:
    void* p = nullptr;
    size_t size = 0;
};

}  // namespace rsv
