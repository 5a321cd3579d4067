// Device memory and streams reused from call to call (pool.h).
#include "pool.h"

#include <map>
#include <mutex>
#include <vector>

namespace b200sa {
namespace host {

thread_local bool IdleScope::idle_ = false;

namespace {

// What pool_free and pool_stream_free keep, per device.  Never destroyed: the
// driver takes everything back when the process ends.
struct DevicePool {
    std::map<size_t, std::vector<void *>> blocks;  // by size class
    size_t bytes = 0;
    std::vector<cudaStream_t> streams;
};
std::mutex g_pool_mutex;
std::map<int, DevicePool> &device_pools() {
    static auto *pools = new std::map<int, DevicePool>();
    return *pools;
}

size_t pool_class(size_t bytes) {
    size_t c = 512;
    while (c < bytes) c <<= 1;
    return c;
}

}  // namespace

cudaError_t pool_alloc(void **ptr, size_t bytes) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const size_t size = bytes <= kPoolBlock ? pool_class(bytes) : bytes;
    if (bytes <= kPoolBlock) {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool &pool = device_pools()[device];
        auto it = pool.blocks.find(size);
        if (it != pool.blocks.end() && !it->second.empty()) {
            *ptr = it->second.back();
            it->second.pop_back();
            pool.bytes -= size;
            return cudaSuccess;
        }
    }
    e = cudaMalloc(ptr, size);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    std::vector<void *> back;  // give everything back and try once more
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool &pool = device_pools()[device];
        for (auto &b : pool.blocks) back.insert(back.end(), b.second.begin(), b.second.end());
        pool.blocks.clear();
        pool.bytes = 0;
    }
    for (void *b : back) cudaFree(b);
    return cudaMalloc(ptr, bytes <= kPoolBlock ? size : bytes);
}

void pool_free(void *ptr, size_t bytes, int device) {
    const size_t size = bytes <= kPoolBlock ? pool_class(bytes) : 0;
    if (size && IdleScope::idle()) {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool &pool = device_pools()[device];
        if (pool.bytes + size <= kPoolBytes) {
            pool.blocks[size].push_back(ptr);
            pool.bytes += size;
            return;
        }
    }
    int current = 0;
    if (cudaGetDevice(&current) != cudaSuccess) current = device;
    if (current != device) cudaSetDevice(device);
    cudaFree(ptr);
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
