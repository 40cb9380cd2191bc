// Shared definitions for the sm_100a RWKV-7 forward-step library.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>

#include "cuda_error.hpp"

namespace rsv {

// Numerical constants of the reference's CPU path (src/model.rs:6-8, :438).
constexpr float kLnEps = 1.0e-5f;
constexpr float kGnEps = 64.0e-5f;
constexpr float kL2Eps = 1.0e-12f;
constexpr float kDecayScale = -0.60653065971263342f;  // -1/sqrt(e)
constexpr int kHeadSize = 64;                         // the only head size RWKV-7 checkpoints use

enum WType : int { W_F16 = 0, W_INT8 = 1 };

// Epilogues of the linear layers.  `acc` is the dot product for (row r, output m).
enum Epi : int {
    EPI_STORE = 0,         // y = acc
    EPI_RELU2 = 1,         // y = max(acc,0)^2                           (ffn.key)
    EPI_TANH = 2,          // y = tanh(acc)                              (decay adapter, rank space)
    EPI_SIGMOID = 3,       // y = sigmoid(acc)                           (gate adapter, rank space)
    EPI_DECAY = 4,         // y = exp(-sigmoid(acc + bias[m]) / sqrt(e)) (w)
    EPI_SIGMOID_BIAS = 5,  // y = sigmoid(acc + bias[m])                 (a, v gate)
};

// Row r of a packed step: which session slot it belongs to and how it chains to its neighbours.
struct RowMeta {
    int slot;      // state slot of the session this row belongs to
    int has_prev;  // 1: row r-1 is the previous token of the same session; 0: previous token lives in the slot state
    int is_last;   // 1: last row of its session in this step -> writes the shift state
    int seg;       // index of the row's segment
};
// A segment = consecutive rows of one session (1 row for decode, up to the chunk length for prefill).
struct SegMeta {
    int start, len, slot;
    int chunk0;  // chunks of sixteen tokens (wkv_chunk.cuh) in the segments before: filled in when a plan is uploaded
};

// Programmatic dependent launch.  A kernel launched with the programmatic-stream-serialization attribute may start
// while its predecessor in the stream still runs; pdl_wait() blocks until that predecessor has completed and its
// memory is visible, pdl_launch_dependents() allows the successor to be scheduled.  Both are no-ops for a normal
// launch.  Rule used here: a kernel reads or writes nothing but its parameters and the model's weights (and state that
// only an earlier step wrote) before pdl_wait().
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A pointer to data the predecessor produces, as seen after pdl_wait().  `const __restrict__` parameters promise the compiler
// that nobody writes the data while the kernel runs, so it may move their loads above the wait; passing the pointer through
// this (empty) asm after the wait makes every later load depend on it.
template <typename T>
__device__ __forceinline__ T* pdl_fresh(T* p) {
    asm volatile("" : "+l"(p)::"memory");
    return p;
}
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace rsv
