// stream_guard.h — host memory behind asynchronous copies.
#pragma once
#include <cuda_runtime.h>

namespace ptx_host {

// Waits for a stream at the end of its scope.  Declared after host memory that copies on the
// stream read or write, it keeps every way out of the scope, an error's too, from giving the
// memory back while a copy may still be at it.
class StreamGuard {
public:
    explicit StreamGuard(cudaStream_t stream) : stream_(stream) {}
    ~StreamGuard() { if (pending_) cudaStreamSynchronize(stream_); }
    StreamGuard(const StreamGuard&) = delete;
    StreamGuard& operator=(const StreamGuard&) = delete;
    void waited() { pending_ = false; }   // the stream was waited for and takes no such copy any more

private:
    cudaStream_t stream_;
    bool pending_ = true;
};

}  // namespace ptx_host
