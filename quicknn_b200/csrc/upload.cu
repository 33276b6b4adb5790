// Small host arrays to the device without stalling the host: a ring of pinned buffers, an event per buffer.
//
// A copy from ordinary host memory makes the caller wait until the stream has drained; a copy from pinned memory does not, but
// reads the pinned bytes when the stream gets to it, by which time the host may have written the next step's values.  So every
// array goes into the next buffer of the ring and is sent from there; a buffer is written again only after the copy that read
// it has run.  The same over torch tensors and events took about 18 us of host time a copy, this 4.
//
// Several threads may send through one ring (a call from Python gives the interpreter away): a lock holds the choice of a buffer, the
// bytes and the copy together.  An event belongs to the device it was made on; a buffer that goes to another one next gets another.
#include <mutex>
#include <new>
#include <string.h>

#include "common.cuh"

namespace {

struct Buffer {
    void* bytes;
    size_t size;
    cudaEvent_t sent;
    int device;                  // of the event
    bool own;                    // allocated here: an array that was larger than the caller's pieces
};
struct Ring {
    int n, next;
    Buffer* buffers;
    std::mutex lock;
};

// the device that is current while this lives
struct OnDevice {
    int before = -1;
    cudaError_t rc;
    explicit OnDevice(int device) {
        rc = cudaGetDevice(&before);
        if (rc == cudaSuccess && before != device) rc = cudaSetDevice(device);
        else before = -1;
    }
    ~OnDevice() {
        if (before >= 0) (void)cudaSetDevice(before);
    }
};

int fill(Buffer& b, size_t n, int device) {
    if (b.sent != nullptr) {
        const cudaError_t e = cudaEventSynchronize(b.sent);
        if (e != cudaSuccess) return (int)e;
        if (b.device != device) {
            (void)cudaEventDestroy(b.sent);
            b.sent = nullptr;
        }
    }
    if (b.sent == nullptr) {
        const cudaError_t e = cudaEventCreateWithFlags(&b.sent, cudaEventDisableTiming);
        if (e != cudaSuccess) {
            b.sent = nullptr;
            return (int)e;
        }
        b.device = device;
    }
    if (b.size < n) {
        void* p = nullptr;
        const cudaError_t e = cudaHostAlloc(&p, n, cudaHostAllocDefault);
        if (e != cudaSuccess) return (int)e;
        if (b.own) (void)cudaFreeHost(b.bytes);
        b.bytes = p;
        b.size = n;
        b.own = true;
    }
    return 0;
}

}  // namespace

// A ring of `entries` buffers of `each` bytes, pieces of the pinned memory at `slab` (the caller's, kept until the ring is free: an
// allocation of pinned memory takes about 1 ms, so the pieces come from one that a caching allocator may have at hand); a larger array
// gets a buffer of its own.  Events are made as buffers are first used.
QNN_API int qnn_upload_ring(int entries, long long each, void* slab, void** ring) {
    if (entries < 1 || each < 1 || slab == nullptr || ring == nullptr) return QNN_ERR_ARGUMENT;
    Ring* r = new (std::nothrow) Ring();
    if (r == nullptr) return (int)cudaErrorMemoryAllocation;
    r->n = entries;
    r->buffers = new (std::nothrow) Buffer[entries]();
    if (r->buffers == nullptr) {
        delete r;
        return (int)cudaErrorMemoryAllocation;
    }
    for (int i = 0; i < entries; ++i) {
        r->buffers[i].bytes = (char*)slab + (size_t)i * (size_t)each;
        r->buffers[i].size = (size_t)each;
    }
    *ring = r;
    return 0;
}

// dst (on `device`) = the n bytes at src, ordered on the stream, one of that device's; src may change as soon as this returns.
QNN_API int qnn_upload(void* ring, void* dst, const void* src, long long n, int device, cudaStream_t st) {
    if (ring == nullptr || n < 0 || device < 0 || (n > 0 && (dst == nullptr || src == nullptr))) return QNN_ERR_ARGUMENT;
    if (n == 0) return 0;
    Ring* r = (Ring*)ring;
    const OnDevice there(device);
    if (there.rc != cudaSuccess) return (int)there.rc;
    const std::lock_guard<std::mutex> held(r->lock);
    Buffer& b = r->buffers[r->next];
    const int rc = fill(b, (size_t)n, device);
    if (rc != 0) return rc;
    r->next = (r->next + 1) % r->n;
    memcpy(b.bytes, src, (size_t)n);
    const cudaError_t e = cudaMemcpyAsync(dst, b.bytes, (size_t)n, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaEventRecord(b.sent, st);
}

// Gives the ring back; waits for the copies that still read it.
QNN_API int qnn_upload_ring_free(void* ring) {
    if (ring == nullptr) return 0;
    Ring* r = (Ring*)ring;
    for (int i = 0; i < r->n; ++i) {
        Buffer& b = r->buffers[i];
        if (b.sent != nullptr) {
            (void)cudaEventSynchronize(b.sent);
            (void)cudaEventDestroy(b.sent);
        }
        if (b.own) (void)cudaFreeHost(b.bytes);
    }
    delete[] r->buffers;
    delete r;
    return 0;
}
