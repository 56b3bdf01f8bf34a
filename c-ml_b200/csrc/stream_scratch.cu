// See stream_scratch.cuh.
#include <mutex>
#include "stream_scratch.cuh"

namespace {
struct Entry { unsigned long long stream, used; void* ptr; };
Entry g_entries[kMaxDevices][kScratchStreams] = {};
unsigned long long g_clock = 0;
std::mutex g_mutex;
}  // namespace

int cmlb_stream_scratch(cudaStream_t stream, size_t bytes, void** out) {
    unsigned long long id = 0;
    CMLB_CUDA(cudaStreamGetId(stream, &id));                 // unique in the process, unlike the handle
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* table = g_entries[cmlb_device_index()];
    Entry* e = table;
    for (int i = 0; i < kScratchStreams; i++) {
        if (table[i].ptr && table[i].stream == id) { e = &table[i]; break; }
        if (table[i].used < e->used) e = &table[i];
    }
    if (!e->ptr) {                                           // (allowed while the stream is being captured, too)
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        CMLB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        const cudaError_t rc = cudaMalloc(&e->ptr, bytes);
        CMLB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        if (rc != cudaSuccess) e->ptr = nullptr;
        CMLB_CUDA(rc);
    }
    else if (e->stream != id) CMLB_CUDA(cudaDeviceSynchronize());
    e->stream = id;
    e->used = ++g_clock;
    *out = e->ptr;
    return CMLB200_OK;
}

void cmlb_stream_scratch_release(cudaStream_t stream) {
    unsigned long long id = 0;
    if (cudaStreamGetId(stream, &id) != cudaSuccess) { cudaGetLastError(); return; }
    std::lock_guard<std::mutex> lock(g_mutex);
    for (int d = 0; d < kMaxDevices; d++)
        for (int i = 0; i < kScratchStreams; i++) {
            Entry& e = g_entries[d][i];
            if (!e.ptr || e.stream != id) continue;
            cudaFree(e.ptr);                                 // waits for the launches that use it
            e = Entry();
        }
}
