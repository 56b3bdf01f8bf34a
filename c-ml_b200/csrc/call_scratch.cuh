// Device scratch of one call, in stream order and under capture.
#pragma once
#include <mutex>
#include "common.cuh"

// Outside a capture a stream keeps its buffer from call to call (kScratchStreams streams of a device; it goes with
// cmlb200_stream_destroy), further streams get one for each call from a pool, in stream order. In a capture (any capture mode) the
// buffer belongs to the graph: one per capture and stream, kept until the last graph and executable made from that capture are gone.
// Nobody else ever gets a buffer that a stream or a graph has. The object lives until the call's last kernel is launched.
constexpr int kScratchStreams = 16;

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
    std::unique_lock<std::mutex> lock_;         // calls that share a buffer launch their kernels one call after another
};

// The stream is about to be destroyed.
void cmlb_scratch_release(cudaStream_t stream);
