// An array that arrives in parts, moved on by a few threads.  No CUDA call: checked on the CPU.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <functional>
#include <system_error>
#include <thread>
#include <vector>

namespace rsv {

class PartsToHost {
  public:
    ~PartsToHost() { join(); }
    // first element of part i when `count` elements come in `parts` parts (i == parts: the end)
    static size_t part_begin(size_t count, int parts, int i) { return std::min(count, (size_t)i * ((count + parts - 1) / parts)); }
    // Copies `count` elements from `src` to `dst`, part by part behind `arrived(i)`, which blocks until part i is in `src` and says whether it
    // came; returns while that is under way.  An earlier call's copies are complete when this one begins.
    void start(float* dst, const float* src, size_t count, int parts, int workers, std::function<bool(int)> arrived) {
        join();
        threads.reserve((size_t)workers);
        for (int w = 0; w < workers; ++w) {
            auto work = [this, dst, src, count, parts, workers, w, arrived] {
                for (int i = w; i < parts; i += workers) {
                    if (!arrived(i)) {
                        failed = true;
                        return;
                    }
                    const size_t at = part_begin(count, parts, i);
                    memcpy(dst + at, src + at, (part_begin(count, parts, i + 1) - at) * sizeof(float));
                }
            };
            try {
                threads.emplace_back(work);
            } catch (const std::system_error&) {  // no more threads to be had: this one does the work
                work();
            }
        }
    }
    // Waits for the copies; whether every part of every call since the last `finish` came.
    bool finish() {
        join();
        return !failed.exchange(false);
    }
    void join() {
        for (auto& t : threads) t.join();
        threads.clear();
    }

  private:
    std::vector<std::thread> threads;
    std::atomic<bool> failed{false};
};

}  // namespace rsv
