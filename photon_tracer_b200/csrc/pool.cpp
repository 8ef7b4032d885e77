// A memory pool per device for what renders need only while they run: work
// counters and samples. Renders of one scene on several streams share nothing
// that way, and a scene that is not rendering holds none: a hundred scenes that
// rendered hold what the pool keeps, not a buffer each.
//
// Neither borrowing nor giving back waits for the device: a block is taken
// again by work that its last borrower's stream orders behind it, or once the
// event at that work's end has passed; else a new one is allocated (cudaMalloc
// returns in 0.4 ms beside running kernels, cudaFree only when they are done, so
// blocks are freed with the device's last scene). At the pool's bound the
// borrower's stream waits for a block. CUDA's own stream-ordered pools do the
// same, but 256 MB took them 1.4 to 30 ms to map, and to unmap, against 0.35.
#include "pool.h"

#include <map>
#include <memory>
#include <mutex>
#include <vector>

namespace pt {

namespace {

constexpr size_t kMiB = size_t(1) << 20;
// All blocks of a device: one of a sample per pixel of the largest streamed
// frame (1 GiB), or four streams' usual largest ones.
constexpr size_t kPoolMost = 1280 * kMiB;

struct DevicePool {
    std::vector<std::unique_ptr<PoolBlock>> blocks;
    size_t bytes = 0;
    int users = 0;
};
std::mutex g_lock;
std::map<int, DevicePool> g_pools;  // by device

// Sizes are rounded up by at most two, so that frames of similar sizes share.
size_t block_size(size_t bytes) {
    size_t b = kMiB;
    while (b < bytes && b < 256 * kMiB) b *= 2;
    if (b < bytes) b = bytes <= 257 * kMiB ? 257 * kMiB : (bytes + kMiB - 1) / kMiB * kMiB;
    return b;
}

void clear_last_error() { cudaGetLastError(); }

PoolBlock* new_block(DevicePool& d, size_t bytes) {
    if (d.bytes + bytes > kPoolMost) return nullptr;
    auto b = std::make_unique<PoolBlock>();
    if (cudaMalloc(&b->ptr, bytes) != cudaSuccess) {
        clear_last_error();
        return nullptr;
    }
    if (cudaEventCreateWithFlags(&b->used, cudaEventDisableTiming) != cudaSuccess) {
        clear_last_error();
        cudaFree(b->ptr);
        return nullptr;
    }
    b->bytes = bytes;
    d.bytes += bytes;
    d.blocks.push_back(std::move(b));
    return d.blocks.back().get();
}

}  // namespace

void pool_join(int device) {
    std::lock_guard<std::mutex> lock(g_lock);
    ++g_pools[device].users;
}

void pool_leave(int device) {
    std::lock_guard<std::mutex> lock(g_lock);
    const auto it = g_pools.find(device);
    if (it == g_pools.end() || --it->second.users > 0) return;
    for (const auto& b : it->second.blocks) {
        cudaEventDestroy(b->used);
        cudaFree(b->ptr);
    }
    g_pools.erase(it);
}

PoolBlock* pool_borrow(int device, size_t bytes, cudaStream_t stream) {
    RelaxedCapture relaxed;
    std::lock_guard<std::mutex> lock(g_lock);
    DevicePool& d = g_pools[device];
    unsigned long long id = 0;
    if (cudaStreamGetId(stream, &id) != cudaSuccess) {
        clear_last_error();
        return nullptr;
    }
    PoolBlock *best = nullptr, *busy = nullptr;  // the smallest that is free at once, and that is not
    for (const auto& b : d.blocks) {
        if (b->lent || b->bytes < bytes) continue;
        PoolBlock*& slot = b->stream == id || cudaEventQuery(b->used) == cudaSuccess ? best : busy;
        if (!slot || b->bytes < slot->bytes) slot = b.get();
    }
    if (busy && cudaPeekAtLastError() == cudaErrorNotReady) clear_last_error();
    if (!best) {
        try {
            best = new_block(d, block_size(bytes));
        } catch (const std::bad_alloc&) {
            best = nullptr;
        }
    }
    if (!best && busy) {
        if (cudaStreamWaitEvent(stream, busy->used, 0) != cudaSuccess) {
            clear_last_error();
            return nullptr;
        }
        best = busy;
    }
    if (best) best->lent = true;
    return best;
}

void pool_return(PoolBlock* block, cudaStream_t stream) {
    if (!block) return;
    RelaxedCapture relaxed;
    std::lock_guard<std::mutex> lock(g_lock);
    block->stream = 0;
    if (cudaStreamGetId(stream, &block->stream) != cudaSuccess || cudaEventRecord(block->used, stream) != cudaSuccess) {
        // what its work is doing is not known any more: not lent again
        clear_last_error();
        return;
    }
    block->lent = false;
}

}  // namespace pt
