// Device memory and streams reused from call to call (pool.h).
#include "pool.h"

#include <algorithm>
#include <list>
#include <map>
#include <mutex>
#include <vector>

namespace b200sa {
namespace host {

thread_local bool IdleScope::idle_ = false;

namespace {

// What pool_free and pool_stream_free keep, per device.  Never destroyed: the
// driver takes everything back when the process ends.
struct Block {
    void *ptr;
    size_t size;
};
struct DevicePool {
    std::list<Block> blocks;  // oldest first
    size_t bytes = 0;
    std::vector<cudaStream_t> streams;
};
std::mutex g_pool_mutex;
std::map<int, DevicePool> &device_pools() {
    static auto *pools = new std::map<int, DevicePool>();
    return *pools;
}

size_t pool_size(size_t bytes) {
    if (bytes > kPoolSmall) return (bytes + 511) & ~size_t(511);
    size_t c = 512;
    while (c < bytes) c <<= 1;
    return c;
}

}  // namespace

cudaError_t pool_alloc(void **ptr, size_t bytes, size_t *size) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const size_t exact = (bytes + 511) & ~size_t(511);
    bytes = pool_size(bytes);
    if (bytes <= kPoolBlock) {
        const size_t most = bytes + bytes / 8;
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool &pool = device_pools()[device];
        auto best = pool.blocks.end();
        for (auto it = pool.blocks.begin(); it != pool.blocks.end(); ++it)
            if (it->size >= bytes && it->size <= most &&
                (best == pool.blocks.end() || it->size < best->size))
                best = it;
        if (best != pool.blocks.end()) {
            *ptr = best->ptr;
            *size = best->size;
            pool.bytes -= best->size;
            pool.blocks.erase(best);
            return cudaSuccess;
        }
    }
    *size = bytes;
    e = cudaMalloc(ptr, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    std::list<Block> back;  // give everything back and try once more
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool &pool = device_pools()[device];
        back.swap(pool.blocks);
        pool.bytes = 0;
    }
    for (const Block &b : back) cudaFree(b.ptr);
    *size = exact;
    return cudaMalloc(ptr, exact);
}

void pool_free(void *ptr, size_t size, int device) {
    std::list<Block> back;
    if (size <= kPoolBlock && IdleScope::idle()) {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool &pool = device_pools()[device];
        pool.blocks.push_back({ptr, size});
        pool.bytes += size;
        while (pool.bytes > kPoolBytes) {
            pool.bytes -= pool.blocks.front().size;
            back.splice(back.end(), pool.blocks, pool.blocks.begin());
        }
    } else {
        back.push_back({ptr, size});
    }
    if (back.empty()) return;
    int current = 0;
    if (cudaGetDevice(&current) != cudaSuccess) current = device;
    if (current != device) cudaSetDevice(device);
    for (const Block &b : back) cudaFree(b.ptr);
    if (current != device) cudaSetDevice(current);
}

cudaError_t pool_stream(cudaStream_t *stream) {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        std::vector<cudaStream_t> &free = device_pools()[device].streams;
        if (!free.empty()) {
            *stream = free.back();
            free.pop_back();
            return cudaSuccess;
        }
    }
    return cudaStreamCreateWithFlags(stream, cudaStreamNonBlocking);
}

void pool_stream_free(cudaStream_t stream, int device) {
    if (cudaStreamSynchronize(stream) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        std::vector<cudaStream_t> &free = device_pools()[device].streams;
        if (free.size() < kPoolStreams) {
            free.push_back(stream);
            return;
        }
    }
    cudaStreamDestroy(stream);
}

}  // namespace host
}  // namespace b200sa
