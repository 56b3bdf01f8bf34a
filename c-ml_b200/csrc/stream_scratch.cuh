// Device scratch that belongs to a stream: launches of one stream use it one after another, launches of different streams never
// share it. A stream's scratch keeps its address (captured graphs hold it) until the stream is destroyed through
// cmlb200_stream_destroy; at most kScratchStreams streams of a device have one at a time, a further stream takes over the least
// recently used one's after waiting for the device.
#pragma once
#include "common.cuh"

constexpr int kScratchStreams = 16;

// `bytes` (the same in every call) of device memory for `stream` on the current device
int cmlb_stream_scratch(cudaStream_t stream, size_t bytes, void** out);
void cmlb_stream_scratch_release(cudaStream_t stream);
