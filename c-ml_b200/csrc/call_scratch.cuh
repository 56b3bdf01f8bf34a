// Device scratch of one call, in stream order and under capture.
#pragma once
#include <mutex>
#include "common.cuh"

// Outside a capture the memory comes from a pool of the library (cudaMallocFromPoolAsync) and goes back in stream order when the
// object goes, so calls in any number of streams and threads never share it. In a capture (any capture mode) it belongs to the
// graph: one buffer per capture and stream, kept until the last graph and executable made from that capture are gone. The object
// lives until the call's last kernel is launched.
class CallScratch {
public:
    CallScratch() {}
    ~CallScratch();
    CallScratch(const CallScratch&) = delete;
    CallScratch& operator=(const CallScratch&) = delete;
    int get(cudaStream_t stream, size_t bytes, void** out);

private:
    void* ptr_ = nullptr;                       // what goes back with the object
    cudaStream_t stream_ = nullptr;
    std::unique_lock<std::mutex> captured_;     // captured calls of all threads one at a time: their launches share the buffer
};
