// Memory that renders borrow while they run (pool.cpp).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace pt {

// A scene or batch joins its device's pool when it is made and leaves it when
// it is destroyed; the pool goes with the last one.
void pool_join(int device);
void pool_leave(int device);
// Device memory from the stream's next work on, until pool_return in the
// stream's order. Returns an error, and sets no error state, when there is none.
cudaError_t pool_borrow(int device, void** ptr, size_t bytes, cudaStream_t stream);
void pool_return(void* ptr, cudaStream_t stream);

}  // namespace pt
