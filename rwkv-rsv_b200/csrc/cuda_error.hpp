// Errors of CUDA calls as exceptions.
#pragma once
#include <cuda_runtime_api.h>

#include <cstdint>
#include <stdexcept>
#include <string>

namespace rsv {

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct OutOfMemory : CudaError {  // an allocation on the device, or of pinned memory
    using CudaError::CudaError;
};

#define RSV_CUDA(expr)                                                                                                                            \
    do {                                                                                                                                          \
        cudaError_t _e = (expr);                                                                                                                  \
        if (_e != cudaSuccess) {                                                                                                                  \
            const std::string _m = std::string(#expr) + " failed: " + cudaGetErrorString(_e) + " (" __FILE__ ":" + std::to_string(__LINE__) + ")"; \
            if (_e == cudaErrorMemoryAllocation) throw ::rsv::OutOfMemory(_m);                                                                    \
            throw ::rsv::CudaError(_m);                                                                                                           \
        }                                                                                                                                         \
    } while (0)

// n rows in passes of up to `most`.  Where memory is short for that many, which a pass finds out (OutOfMemory) before it has launched anything, up to `fewer` from there
// on; `launches` counts what has been launched.
template <class Launches, class Pass>
void in_passes(int64_t n, int64_t most, int64_t fewer, Launches&& launches, Pass&& pass) {
    for (int64_t at = 0; at < n;) {
        const int64_t rows = n - at < most ? n - at : most;
        const auto before = launches();
        try {
            pass(at, rows);
        } catch (const OutOfMemory&) {
            if (rows <= fewer || launches() != before) throw;
            cudaGetLastError();
            most = fewer;
            continue;
        }
        at += rows;
    }
}

}  // namespace rsv
