// See call_scratch.cuh. Memory from the pool and back costs 0.9 us of host time a call (8 rows through Q8_0 512x1024: 6.3 us a call,
// launches included, 5.4 with a buffer that the stream keeps), and launches before and behind it still overlap programmatically.
#include <atomic>
#include <vector>
#include "call_scratch.cuh"

namespace {

// Whole 2 MB, so that buffers start on such a boundary: 32 rows through Q4_0 1536x8960 take 20.95 us a call, 22.2 with a buffer that
// starts 512 bytes off one (Q8_0 1024x4096, 17 rows: 10.55 and 11.2)
constexpr size_t kWhole = (size_t)2 << 20;
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

// A stream's buffer. The stream is known by its id: handles come again.
struct Owned {
    std::mutex busy;
    unsigned long long stream = 0;
    size_t bytes = 0;
    void* ptr = nullptr;
};

struct Device {
    cudaMemPool_t pool = nullptr;
    cudaStream_t side = nullptr;                            // allocations that belong to no stream of a caller
    Owned owned[kScratchStreams];
};

struct Library {
    std::mutex mutex, captured;
    Device devices[kMaxDevices];
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
        const Relaxed relaxed;
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
    const Relaxed relaxed;
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

// A stream's place in the table; nullptr where as many streams as may have one do
Owned* owned_by(Library& l, Device* d, unsigned long long id) {
    std::lock_guard<std::mutex> lock(l.mutex);
    Owned* free = nullptr;
    for (Owned& o : d->owned) {
        if (o.stream == id) return &o;
        if (!o.stream && !free) free = &o;
    }
    if (free) free->stream = id;
    return free;
}

int stream_id(cudaStream_t stream, unsigned long long* id) {
    CMLB_CUDA(cudaStreamGetId(stream, id));
    *id += 1;                                               // 0 stands for none
    return CMLB200_OK;
}

}  // namespace

int CallScratch::get(cudaStream_t stream, size_t bytes, void** out) {
    Library& l = library();
    bytes = (bytes + kWhole - 1) / kWhole * kWhole;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    cudaGraph_t graph = nullptr;
    CMLB_CUDA(cudaStreamGetCaptureInfo(stream, &status, &id, &graph));
    const int index = cmlb_device_index();
    Device* d = nullptr;
    int rc = device_of(l, index, &d);
    if (rc) return rc;
    collect(l);
    if (status == cudaStreamCaptureStatusActive) {
        lock_ = std::unique_lock<std::mutex>(l.captured);
        const Relaxed relaxed;
        return held_by(l, d, index, stream, id, graph, bytes, out);
    }
    if ((rc = stream_id(stream, &id))) return rc;
    Owned* o = owned_by(l, d, id);
    if (!o) {
        const Relaxed relaxed;
        CMLB_CUDA(cudaMallocFromPoolAsync(&ptr_, bytes, d->pool, stream));
        stream_ = stream;
        *out = ptr_;
        return CMLB200_OK;
    }
    lock_ = std::unique_lock<std::mutex>(o->busy);
    if (o->bytes < bytes) {
        const Relaxed relaxed;
        void* more = nullptr;
        CMLB_CUDA(cudaMallocFromPoolAsync(&more, bytes, d->pool, stream));
        if (o->ptr) cudaFreeAsync(o->ptr, stream);          // (behind the launches that use it)
        o->ptr = more;
        o->bytes = bytes;
    }
    *out = o->ptr;
    return CMLB200_OK;
}

CallScratch::~CallScratch() {
    if (!ptr_) return;
    const Relaxed relaxed;
    cudaFreeAsync(ptr_, stream_);
}

void cmlb_scratch_release(cudaStream_t stream) {
    Library& l = library();
    unsigned long long id = 0;
    if (cudaStreamGetId(stream, &id) != cudaSuccess) { cudaGetLastError(); return; }
    std::lock_guard<std::mutex> lock(l.mutex);
    const Relaxed relaxed;
    for (Device& d : l.devices)
        for (Owned& o : d.owned) {
            if (o.stream != id + 1) continue;
            if (o.ptr) cudaFreeAsync(o.ptr, stream);
            o.stream = 0;
            o.bytes = 0;
            o.ptr = nullptr;
        }
}
