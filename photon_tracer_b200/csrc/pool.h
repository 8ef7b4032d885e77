// Memory that renders borrow while they run (pool.cpp).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace pt {

// A scene joins its device's pool when it is made and leaves it when it is
// destroyed, with none of its work in flight; the pool's memory goes with the
// last one.
void pool_join(int device);
void pool_leave(int device);

// Device memory for the stream's work from pool_borrow to pool_return, both of
// which return at once. Null, with no error state set, when there is none.
struct PoolBlock {
    void* ptr = nullptr;
    size_t bytes = 0;
    cudaEvent_t used = nullptr;     // the end of its last borrower's work
    unsigned long long stream = 0;  // and the id of the stream of that work
    bool lent = false;
};
PoolBlock* pool_borrow(int device, size_t bytes, cudaStream_t stream);
void pool_return(PoolBlock* block, cudaStream_t stream);

// Allocations and event queries while this lives do not disturb a capture on
// another stream.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace pt
