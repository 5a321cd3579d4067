// Device memory and streams reused from call to call.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace b200sa {
namespace host {

// Device memory and non-blocking streams of the current device, reused from
// call to call: a call's buffers and stream otherwise cost it about 20
// microseconds each to make and as many to free (0.7 ms for 8 MB, 0.15 to 0.2
// ms for a stream).  Freed blocks of at most kPoolBlock bytes are kept, up to
// kPoolBytes in all per device (the oldest ones go first), and go back to the
// driver when an allocation fails; streams likewise up to kPoolStreams.  Every
// function may be called from any thread.
//
// A new block above kPoolSmall is as large as what was asked for: rounded up to
// a power of two, a 33 MB buffer needed 64 MB of free memory.  Smaller ones are
// rounded up, so that calls of other sizes find them, but not when memory is
// short.  A kept block serves requests up to an eighth smaller.
constexpr size_t kPoolBlock = size_t(64) << 20;
constexpr size_t kPoolBytes = size_t(256) << 20;
constexpr size_t kPoolSmall = size_t(16) << 20;
constexpr size_t kPoolStreams = 16;
cudaError_t pool_alloc(void **ptr, size_t bytes, size_t *size);  // size: of the block
// Inside an IdleScope whose work is done the block is kept; otherwise it is
// freed, which waits for the device.
void pool_free(void *ptr, size_t size, int device);
cudaError_t pool_stream(cudaStream_t *stream);
void pool_stream_free(cudaStream_t stream, int device);  // with no work in flight

// Declared before a call's buffers.  Once the call has waited for its own work
// it says so (done), and what this thread frees from then on, to the end of the
// scope, may be kept: nothing on the device uses it any more.  The pool itself
// waits for nothing: to wait for the device is an error while any thread
// captures one of its streams, and ends that capture.
class IdleScope {
  public:
    IdleScope() : outer_(idle_) { idle_ = false; }
    ~IdleScope() { idle_ = outer_; }
    IdleScope(const IdleScope &) = delete;
    IdleScope &operator=(const IdleScope &) = delete;
    static void done() { idle_ = true; }
    static bool idle() { return idle_; }

  private:
    static thread_local bool idle_;
    const bool outer_;
};

}  // namespace host
}  // namespace b200sa
