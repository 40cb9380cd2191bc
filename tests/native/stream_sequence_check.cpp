// CPU check of csrc/stream_sequence.hpp against a model of the device: the numbers a launch is given must be the ones the launches that ran
// left behind, whatever launches failed in between.
#include <cstdio>
#include <stdexcept>

#include "stream_sequence.hpp"

int main() {
    rsv::StreamSequence seq;
    uint32_t tag = 1;      // device: tag the next layer to run has
    unsigned counter = 0;  // device: the grid barrier's counter
    int bad = 0;
    unsigned rnd = 12345;
    for (int i = 0; i < 1000; ++i) {
        rnd = rnd * 1664525u + 1013904223u;
        const uint32_t tokens = 1 + (rnd >> 24) % 7, layers = tokens * 31;
        const unsigned arrivals = 148 * (tokens - (rnd >> 20 & 1));
        const bool fails = (rnd >> 16 & 3) == 0;
        try {
            seq.run(layers, arrivals, [&](uint32_t epoch, unsigned base) {
                if (epoch != tag || base != counter) ++bad;
                if (fails) throw std::runtime_error("launch failed");
                tag += layers;
                counter += arrivals;
            });
            if (fails) ++bad;
        } catch (const std::runtime_error&) {
            if (!fails) ++bad;
        }
    }
    std::printf(bad ? "%d launches were given wrong numbers\n" : "sequence ok\n", bad);
    return bad != 0;
}
