// CPU check of csrc/cuda_error.hpp with stand-ins for the CUDA calls it makes: errors as exceptions, and passes that get shorter where memory is short.
#include <cstdio>
#include <vector>

#include "cuda_error.hpp"

static int bad = 0, cleared = 0;
extern "C" {
const char* cudaGetErrorString(cudaError_t) { return "an error"; }
cudaError_t cudaGetLastError(void) {
    ++cleared;
    return cudaSuccess;
}
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

// What a text of n rows does on a device with room for `room` rows a pass (`late`: for the passes from row `late` on), or one whose allocation fails in the middle of a pass.
struct Run {
    std::vector<int64_t> at, rows;
    bool failed = false;
};
static Run run(int64_t n, int64_t most, int64_t fewer, int64_t room, int64_t late = 0, bool in_the_middle = false) {
    Run r;
    long launches = 0;
    try {
        in_passes(n, most, fewer, [&] { return launches; }, [&](int64_t at, int64_t rows) {
            if (in_the_middle) ++launches;
            if (at >= late) RSV_CUDA(rows > room ? cudaErrorMemoryAllocation : cudaSuccess);
            ++launches;
            r.at.push_back(at);
            r.rows.push_back(rows);
        });
    } catch (const OutOfMemory&) {
        r.failed = true;
    }
    return r;
}

int main() {
    for (int64_t n : {1, 127, 128, 129, 255, 256, 257, 384, 600, 1000})
        for (int64_t room : {0, 60, 128, 200, 256, 1000})
            for (int64_t late : {0, 256, 512}) {
                const Run r = run(n, 256, 128, room, late);
                int64_t next = 0;
                bool whole = true;
                for (size_t i = 0; i < r.at.size(); ++i) {
                    whole = whole && r.at[i] == next && r.rows[i] >= 1 && (next < late || r.rows[i] <= room);
                    next += r.rows[i];
                }
                CHECK(whole, "%ld rows, room for %ld: rows left out, twice or out of order", (long)n, (long)room);
                if (room >= 128) CHECK(!r.failed && next == n, "%ld rows, room for %ld: a text that fits in passes of 128 failed", (long)n, (long)room);
                if (room >= 256 || n <= room) CHECK(r.at.size() == (size_t)((n + 255) / 256), "%ld rows, room for %ld: short passes without need", (long)n, (long)room);
                if (room == 0 && late == 0) CHECK(r.failed && next == 0, "a failure was swallowed");
            }
    CHECK(run(256, 256, 256, 128).failed, "shorter passes where they were not asked for");
    const Run half = run(512, 256, 128, 128, 0, true);
    CHECK(half.failed && half.at.empty(), "a pass that had launched something was run again");
    cleared = 0;
    run(256, 256, 128, 128);
    CHECK(cleared == 1, "the error was left for a later check to find");
    try {
        RSV_CUDA(cudaErrorInvalidValue);
        CHECK(false, "no exception");
    } catch (const OutOfMemory&) {
        CHECK(false, "another error taken for a lack of memory");
    } catch (const CudaError&) {
    }
    if (!bad) std::printf("passes ok\n");
    return bad != 0;
}
