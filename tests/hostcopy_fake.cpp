// A stand-in for the parts of the CUDA runtime that hostcopy.cu calls, for the CPU
// tests: device memory is host memory, a stream is a queue of operations that run
// when something waits for them, and cudaStreamPerThread names another queue in
// every thread.
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <thread>
#include <utility>
#include <vector>

#include "rgs_internal.cuh"

namespace {

using Key = std::pair<cudaStream_t, std::thread::id>;
struct Queue {
    std::deque<std::function<void()>> ops;
    size_t queued = 0, run = 0;
};
struct Event {
    Queue* q;
    size_t at;
};
std::recursive_mutex mu;
std::map<Key, Queue> queues;
std::map<char*, size_t> registered;
int fail_after = -1;  // the copies that still succeed (-1: all)
bool capturing = false;       // another thread captures a graph in the global mode
bool no_unregister = false;  // cudaHostUnregister fails whatever the mode
thread_local cudaStreamCaptureMode capture_mode = cudaStreamCaptureModeGlobal;

Queue& queue_of(cudaStream_t st) {
    return queues[{st, st == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id()}];
}
void run_to(Queue& q, size_t at) {
    while (q.run < at) {
        q.ops.front()();
        q.ops.pop_front();
        ++q.run;
    }
}
void put(cudaStream_t st, std::function<void()> op) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    Queue& q = queue_of(st);
    q.ops.push_back(std::move(op));
    ++q.queued;
}
bool locked(const void* p) {
    for (auto& r : registered)
        if ((char*)p >= r.first && (char*)p < r.first + r.second) return true;
    return false;
}

}  // namespace

extern "C" {

cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* mode) {
    std::swap(capture_mode, *mode);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    std::memset(a, 0, sizeof *a);
    a->type = locked(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    if (capturing && capture_mode != cudaStreamCaptureModeRelaxed) return cudaErrorStreamCaptureUnsupported;
    registered[(char*)p] = n;
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void* p) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    if (no_unregister) return cudaErrorUnknown;
    if (capturing && capture_mode != cudaStreamCaptureModeRelaxed) return cudaErrorStreamCaptureUnsupported;
    registered.erase((char*)p);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t) new Event{nullptr, 0}, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete (Event*)e, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    Queue& q = queue_of(st);
    *(Event*)e = {&q, q.queued};
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    if (((Event*)e)->q) run_to(*((Event*)e)->q, ((Event*)e)->at);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    run_to(queue_of(st), queue_of(st).queued);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    if (fail_after == 0) return cudaErrorUnknown;
    if (fail_after > 0) --fail_after;
    put(st, [=] { std::memcpy(d, s, n); });
    // pageable memory: done when the call returns
    if (!locked(kind == cudaMemcpyHostToDevice ? s : d)) cudaStreamSynchronize(st);
    return cudaSuccess;
}

// ---- what the tests call: 0, or the step that went wrong --------------------

void fake_user(int add) { rgs::host_copy_user(add); }

// A read after a queued kernel that fills the buffer, and a write after one that
// still reads it, on `stream`.
int fake_ordered(size_t bytes, int per_thread) {
    cudaStream_t st = per_thread ? cudaStreamPerThread : (cudaStream_t)0x1000;
    std::vector<char> dev(bytes), host(bytes), seen(bytes), want(bytes);
    for (size_t i = 0; i < bytes; ++i) want[i] = (char)(i * 2654435761u >> 13);
    put(st, [&] { dev = want; });
    if (rgs::copy_to_host(host.data(), dev.data(), bytes, st) != cudaSuccess) return 1;
    cudaStreamSynchronize(st);
    if (host != want) return 2;
    for (size_t i = 0; i < bytes; ++i) host[i] = (char)(i * 40503u >> 7);
    put(st, [&] { seen = dev; });
    if (rgs::copy_from_host(dev.data(), host.data(), bytes, st) != cudaSuccess) return 3;
    std::vector<char> sent = host;
    std::fill(host.begin(), host.end(), 0);  // the caller may reuse its array
    cudaStreamSynchronize(st);
    if (seen != want) return 4;
    return dev == sent ? 0 : 5;
}

// A copy whose transfers fail after `good` of them: an error, and no slab lost.
int fake_failing(size_t bytes, int good, int to_host) {
    std::vector<char> dev(bytes), host(bytes);
    fail_after = good;
    const cudaError_t e = to_host ? rgs::copy_to_host(host.data(), dev.data(), bytes, (cudaStream_t)0x1000)
                                  : rgs::copy_from_host(dev.data(), host.data(), bytes, (cudaStream_t)0x1000);
    fail_after = -1;
    return e == cudaErrorUnknown ? 0 : 1;
}

int fake_registered() { return (int)registered.size(); }
void fake_capturing(int on) { capturing = on != 0; }
void fake_no_unregister(int on) { no_unregister = on != 0; }

// Registered ranges that are no longer mapped, which no program may leave behind.
int fake_dangling() {
    int bad = 0;
    for (auto& r : registered) {
        const size_t page = (size_t)sysconf(_SC_PAGESIZE);
        std::vector<unsigned char> in((r.second + page - 1) / page);
        bad += mincore((void*)((uintptr_t)r.first & ~(page - 1)), r.second, in.data()) != 0;
    }
    return bad;
}
}
