// CPU check of csrc/parts_to_host.hpp: what arrives is copied, every element once, and a part that does not come is reported however many
// calls follow before anybody asks.
#include <chrono>
#include <cstdio>

#include "parts_to_host.hpp"

using rsv::PartsToHost;
static int bad = 0;
#define CHECK(cond, ...)             \
    do {                             \
        if (!(cond)) {               \
            std::printf(__VA_ARGS__); \
            std::printf("\n");       \
            ++bad;                   \
        }                            \
    } while (0)

int main() {
    for (size_t count : {(size_t)1, (size_t)31, (size_t)32, (size_t)33, (size_t)1000, (size_t)100003})
        for (int workers : {1, 3, 8, 40}) {
            std::vector<float> src(count), dst(count + 2, -1.f);
            PartsToHost m;
            // the source is filled as the parts "arrive", each in its own time
            m.start(dst.data() + 1, src.data(), count, 32, workers, [&](int i) {
                std::this_thread::sleep_for(std::chrono::microseconds((i * 37) % 11));
                for (size_t k = PartsToHost::part_begin(count, 32, i); k < PartsToHost::part_begin(count, 32, i + 1); ++k) src[k] = (float)(k % 9973 + 1);
                return true;
            });
            CHECK(m.finish(), "%zu elements, %d workers: a failure out of nowhere", count, workers);
            bool same = dst.front() == -1.f && dst.back() == -1.f;
            for (size_t k = 0; k < count; ++k) same = same && dst[k + 1] == (float)(k % 9973 + 1);
            CHECK(same, "%zu elements, %d workers: wrong data", count, workers);
        }
    // a part of one chunk fails, the chunks after it come whole
    for (int which = 0; which < 3; ++which) {
        std::vector<float> src(4096, 1.f), dst(4096);
        PartsToHost m;
        for (int chunk = 0; chunk < 3; ++chunk) m.start(dst.data(), src.data(), src.size(), 32, 4, [=](int i) { return !(chunk == which && i == 7); });
        CHECK(!m.finish(), "the failure in chunk %d was not reported", which);
        m.start(dst.data(), src.data(), src.size(), 32, 4, [](int) { return true; });
        CHECK(m.finish(), "a failure was reported twice");
    }
    if (!bad) std::printf("parts ok\n");
    return bad != 0;
}
