// A memory pool per device for what renders need only while they run: work
// counters and samples, borrowed and given back in the order of a stream. So
// renders of one scene on several streams share nothing, no call waits for the
// device (cudaFree would), and an object that is not rendering holds none:
// a hundred scenes that rendered hold what the pool keeps, not a buffer each.
#include "pool.h"

#include <map>
#include <mutex>

namespace pt {

namespace {

// What the pool keeps of given-back memory for the next borrower: two streams'
// largest usual buffers of samples.
constexpr unsigned long long kPoolKeep = 512ull << 20;

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    int users = 0;  // scenes and batches
};
std::mutex g_lock;
std::map<int, DevicePool> g_pools;  // by device

cudaMemPool_t device_pool(int device) {
    std::lock_guard<std::mutex> lock(g_lock);
    DevicePool& d = g_pools[device];
    if (!d.pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        unsigned long long keep = kPoolKeep;
        if (cudaMemPoolCreate(&d.pool, &props) == cudaSuccess)
            cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        else
            d.pool = nullptr;
    }
    return d.pool;
}

// The pool's own work must not disturb a capture on another stream.
struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace

void pool_join(int device) {
    std::lock_guard<std::mutex> lock(g_lock);
    ++g_pools[device].users;
}

void pool_leave(int device) {
    std::lock_guard<std::mutex> lock(g_lock);
    const auto it = g_pools.find(device);
    if (it == g_pools.end() || --it->second.users > 0) return;
    // Memory that a stream has yet to give back goes when it has.
    if (it->second.pool) cudaMemPoolDestroy(it->second.pool);
    g_pools.erase(it);
}

cudaError_t pool_borrow(int device, void** ptr, size_t bytes, cudaStream_t stream) {
    Relaxed relaxed;
    *ptr = nullptr;
    const cudaMemPool_t pool = device_pool(device);
    const cudaError_t e = pool ? cudaMallocFromPoolAsync(ptr, bytes, pool, stream) : cudaErrorMemoryAllocation;
    if (e) {
        cudaGetLastError();
        *ptr = nullptr;
    }
    return e;
}

void pool_return(void* ptr, cudaStream_t stream) {
    if (!ptr) return;
    Relaxed relaxed;
    if (cudaFreeAsync(ptr, stream) != cudaSuccess) cudaGetLastError();
}

}  // namespace pt
