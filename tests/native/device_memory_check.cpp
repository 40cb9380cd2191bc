// CPU check of csrc/device_memory.hpp with stand-ins for cudaMalloc, cudaFree, cudaGetDevice and cudaGetLastError: two devices of limited memory.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <memory>
#include <thread>

#include "device_memory.hpp"

static std::mutex g_mu;
static size_t g_free[2];
static std::map<void*, std::pair<int, size_t>> g_live;
static thread_local int g_device = 0;
static int bad = 0;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes) {
    std::lock_guard<std::mutex> lock(g_mu);
    if (bytes > g_free[g_device]) return cudaErrorMemoryAllocation;
    g_free[g_device] -= bytes;
    *p = std::malloc(1);
    g_live[*p] = {g_device, bytes};
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lock(g_mu);
    auto it = g_live.find(p);
    if (it == g_live.end()) {
        std::printf("freed something that is not allocated\n");
        ++bad;
        return cudaErrorInvalidValue;
    }
    g_free[it->second.first] += it->second.second;
    std::free(p);
    g_live.erase(it);
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = g_device;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}
#define CHECK(cond, ...)             \
    do {                             \
        if (!(cond)) {               \
            std::printf(__VA_ARGS__); \
            std::printf("\n");       \
            ++bad;                   \
        }                            \
    } while (0)

using namespace rsv;
constexpr size_t MB = 1 << 20;

int main() {
    g_free[0] = g_free[1] = 1000 * MB;
    {
        auto pool = std::make_shared<StatePool>(0), other = std::make_shared<StatePool>(0), far = std::make_shared<StatePool>(1);
        auto fill = [&](StatePool& p, size_t bytes) {
            float* q = nullptr;
            CHECK(device_malloc(&q, bytes) == cudaSuccess, "no memory for a state");
            p.give(bytes, q);
        };
        // an allocation of another kind that needs what two models' pools hold
        fill(*pool, 400 * MB);
        fill(*other, 300 * MB);
        g_device = 1;
        fill(*far, 400 * MB);
        g_device = 0;
        void* weights = nullptr;
        CHECK(device_malloc(&weights, 900 * MB) == cudaSuccess, "an allocation failed while freed states held the memory");
        CHECK(g_free[0] == 100 * MB && g_free[1] == 600 * MB, "pools of another device were emptied, or something was left");
        CHECK(far->take(400 * MB) != nullptr, "the other device's pool lost its state");
        float* q = nullptr;
        CHECK(device_malloc(&q, 200 * MB) == cudaErrorMemoryAllocation, "an allocation larger than the device succeeded");
        cudaFree(weights);
        // bounds: two states, none of more than 512 MB; the oldest goes first; a taken one is gone from the pool
        fill(*pool, 10 * MB);
        fill(*pool, 20 * MB);
        fill(*pool, 30 * MB);
        CHECK(g_free[0] == 950 * MB, "more than two states kept");
        CHECK(pool->take(10 * MB) == nullptr, "the oldest state was kept");
        float* a = pool->take(20 * MB);
        CHECK(a != nullptr && pool->take(20 * MB) == nullptr, "a state was not handed out once");
        fill(*pool, 600 * MB);
        CHECK(g_free[0] == 950 * MB, "a state of 600 MB was kept");
        // a state that outlives its model
        pool->release(true);
        pool->give(20 * MB, a);
        CHECK(g_free[0] == 1000 * MB, "a closed pool kept a state");
        // threads: states come and go while another thread is short of memory
        std::thread t[3];
        for (int k = 0; k < 3; ++k)
            t[k] = std::thread([&, k] {
                for (int i = 0; i < 2000; ++i) {
                    auto mine = std::make_shared<StatePool>(0);
                    float* p = other->take(100 * MB);
                    if (!p && device_malloc(&p, 100 * MB) != cudaSuccess) continue;
                    (k ? *other : *mine).give(100 * MB, p);
                    float* big = nullptr;
                    if (k == 2 && device_malloc(&big, 700 * MB) == cudaSuccess) cudaFree(big);
                }
            });
        for (auto& x : t) x.join();
        g_device = 1;
    }
    g_device = 0;
    {
        // a work area: slack, no reallocation below its size, the exact size where the slack does not fit, and a refusal instead of an error
        SpareArea area;
        int waits = 0;
        auto idle = [&] { ++waits; };
        CHECK(area.reserve(100 * MB, idle) && area.bytes() == 125 * MB && waits == 0, "first growth");
        void* first = area.as<void>();
        CHECK(area.reserve(125 * MB, idle) && area.as<void>() == first && waits == 0, "an area that was large enough moved");
        CHECK(area.reserve(900 * MB, idle) && area.bytes() == 900 * MB && waits == 1 && g_free[0] == 100 * MB, "the exact size was not taken where the slack does not fit");
        CHECK(!area.reserve(1100 * MB, idle) && area.bytes() == 0 && !area.as<void>() && waits == 2 && g_free[0] == 1000 * MB, "refused, and the old memory kept");
        CHECK(area.reserve(200 * MB, idle) && area.bytes() == 250 * MB, "no use after a refusal");
        area.release();
        area.release();
        auto pool = std::make_shared<StatePool>(0);
        float* q = nullptr;
        CHECK(device_malloc(&q, 500 * MB) == cudaSuccess, "no memory for a state");
        pool->give(500 * MB, q);
        CHECK(area.reserve(600 * MB, idle) && area.bytes() == 750 * MB, "the memory of freed states was not given back for it");
        area.release();
    }
    CHECK(g_free[0] == 1000 * MB, "%zu bytes of device 0 lost", 1000 * MB - g_free[0]);
    if (!bad) std::printf("device memory ok\n");
    return bad != 0;
}
