// See call_scratch.cuh. A call costs about 0.5 us of host time for the memory (two launches: 4.1 us), and launches before and behind
// it still overlap programmatically.
#include <atomic>
#include <vector>
#include "call_scratch.cuh"

namespace {

constexpr unsigned long long kPoolKeeps = 32ull << 20;      // bytes that stay with a device's pool while nobody uses them

// What the calls below may do while this or another thread captures in one of the stricter modes
class Relaxed {
public:
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode_); }

private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// A buffer that captured launches use. `gone` is set when the last graph that holds them is (CUDA may not be called there).
struct Held {
    unsigned long long capture;
    cudaStream_t stream;
    int device;
    size_t bytes;
    void* ptr;
    std::atomic<bool> gone;
};

struct Device {
    cudaMemPool_t pool;
    cudaStream_t side;                                      // allocations that belong to no stream of a caller
};

struct Library {
    std::mutex mutex, captured;
    Device devices[kMaxDevices] = {};
    std::vector<Held*> held;
    std::atomic<int> gone{0};
};
Library& library() {
    static Library* l = new Library;                        // graphs may go after the library's statics have
    return *l;
}

int device_of(Library& l, int index, Device** out) {
    std::lock_guard<std::mutex> lock(l.mutex);
    Device& d = l.devices[index];
    if (!d.side) {
        if (!d.pool) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = index;
            cudaMemPool_t pool = nullptr;
            unsigned long long keep = kPoolKeeps;
            CMLB_CUDA(cudaMemPoolCreate(&pool, &props));
            CMLB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
            d.pool = pool;
        }
        CMLB_CUDA(cudaStreamCreateWithFlags(&d.side, cudaStreamNonBlocking));
    }
    *out = &d;
    return CMLB200_OK;
}

void CUDART_CB graphs_are_gone(void* held) {
    static_cast<Held*>(held)->gone.store(true, std::memory_order_release);
    library().gone.fetch_add(1, std::memory_order_release);
}

// Buffers whose graphs are gone return to the pool.
void collect(Library& l) {
    if (l.gone.load(std::memory_order_acquire) == 0) return;
    std::lock_guard<std::mutex> lock(l.mutex);
    for (size_t i = 0; i < l.held.size();) {
        Held* h = l.held[i];
        if (!h->gone.load(std::memory_order_acquire)) { i++; continue; }
        cudaFreeAsync(h->ptr, l.devices[h->device].side);
        l.gone.fetch_sub(1, std::memory_order_relaxed);
        delete h;
        l.held[i] = l.held.back();
        l.held.pop_back();
    }
}

int held_by(Library& l, Device* d, int index, cudaStream_t stream, unsigned long long capture, cudaGraph_t graph, size_t bytes, void** out) {
    {
        std::lock_guard<std::mutex> lock(l.mutex);
        for (Held* h : l.held)
            if (h->capture == capture && h->stream == stream && h->device == index && h->bytes >= bytes && !h->gone.load(std::memory_order_acquire)) {
                *out = h->ptr;
                return CMLB200_OK;
            }
    }
    void* ptr = nullptr;
    CMLB_CUDA(cudaMallocFromPoolAsync(&ptr, bytes, d->pool, d->side));
    cudaError_t rc = cudaStreamSynchronize(d->side);
    Held* h = new Held{capture, stream, index, bytes, ptr, {false}};
    cudaUserObject_t object = nullptr;
    if (rc == cudaSuccess) rc = cudaUserObjectCreate(&object, h, graphs_are_gone, 1, cudaUserObjectNoDestructorSync);
    if (rc == cudaSuccess) {
        {
            std::lock_guard<std::mutex> lock(l.mutex);
            l.held.push_back(h);
        }
        rc = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
        if (rc != cudaSuccess) cudaUserObjectRelease(object);              // (collected like any other)
    } else {
        cudaFreeAsync(ptr, d->side);
        delete h;
    }
    CMLB_CUDA(rc);
    *out = ptr;
    return CMLB200_OK;
}

}  // namespace

int CallScratch::get(cudaStream_t stream, size_t bytes, void** out) {
    Library& l = library();
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    cudaGraph_t graph = nullptr;
    CMLB_CUDA(cudaStreamGetCaptureInfo(stream, &status, &capture, &graph));
    if (status == cudaStreamCaptureStatusActive) captured_ = std::unique_lock<std::mutex>(l.captured);
    const Relaxed relaxed;
    const int index = cmlb_device_index();
    Device* d = nullptr;
    const int rc = device_of(l, index, &d);
    if (rc) return rc;
    collect(l);
    if (status == cudaStreamCaptureStatusActive) return held_by(l, d, index, stream, capture, graph, bytes, out);
    CMLB_CUDA(cudaMallocFromPoolAsync(&ptr_, bytes, d->pool, stream));
    stream_ = stream;
    *out = ptr_;
    return CMLB200_OK;
}

CallScratch::~CallScratch() {
    if (!ptr_) return;
    const Relaxed relaxed;
    cudaFreeAsync(ptr_, stream_);
}
