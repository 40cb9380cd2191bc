// What consecutive launches of the single-session decode kernel hand on to one another.  No CUDA call: checked on the CPU.
#pragma once
#include <cstdint>

namespace rsv {

// Exchanged values carry the number of their layer, counted over all launches (decode_stream.cuh), and the grid barrier's counter only grows.  Both
// numbers move on by what a launch does, so they may move only if it was accepted: after a launch that failed the device holds the values of
// the one before it, and a base ahead of them would make every later barrier wait for arrivals that never come (and, ahead by an odd
// number of layers, let stale hidden values pass, whose tag is a parity).
struct StreamSequence {
    uint32_t epoch = 1;     // tag of the next launch's first layer (0: no launch's)
    unsigned bar_base = 0;  // value of the grid barrier's counter when the next launch begins
    // `launch(epoch, bar_base)` throws if the launch was not accepted
    template <class Launch>
    void run(uint32_t layers, unsigned arrivals, Launch&& launch) {
        launch(epoch, bar_base);
        epoch += layers;
        bar_base += arrivals;
    }
};

}  // namespace rsv
