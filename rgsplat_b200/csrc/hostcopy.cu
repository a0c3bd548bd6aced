// hostcopy.cu -- large copies between device memory and the caller's pageable
// host arrays (Gaussians, gradients, moments, images).
//
// cudaMemcpyAsync on pageable memory goes through the driver's staging buffers
// on the calling thread, which also takes every page fault of a fresh
// destination: 4.9 GB/s into a newly allocated array. Here several threads claim
// chunks in turn; each copies its chunk between the caller's array and one of
// its two page-locked slabs while the other slab is on the bus, so both the
// memory copies and the page faults run in parallel. Measured on a 16-core host,
// before and after: reading a scene of 47 MB 9.9 -> 2.9 ms, 236 MB 48 -> 11.7 ms
// (20 GB/s); writing one 2.6 -> 1.5, 21 -> 5.8 ms. HOST_COPY_MIN lies where the
// threads' start is paid back: 6.1 MB read 0.84 -> 0.78 ms but written 0.38 ->
// 0.47, 8.4 MB 1.1 -> 1.2 and 0.51 -> 0.54, 9.4 MB 1.23 -> 0.86 and 0.60 -> 0.48.
//
// The slabs belong to the process, not to a context: one block of HC_SLABS, handed
// out under a mutex and given back when the last context is destroyed. It is
// huge-page memory registered as a whole (16 MiB: 2.1 ms, and 0.7 to give back;
// sixteen cudaHostAlloc of 1 MiB took 10 to 22; slabs of 512 KiB wrote 236 MB in 8.0
// ms instead of 5.9). The block is made once HC_FIRST bytes have gone by in large
// copies, when the plain copies have lost about what it costs: 32 MiB read in arrays
// of 9 to 24 MB lose 1 to 1.5 ms, in one array of 47 MB 7 ms, written 0.4 to 1. A
// program that copies less and ends never pays; one that goes on pays 2.8 ms for what
// each such call then saves (a drop-in call of 50k Gaussians, 24 MB, 3.7 -> 2.7).
// A copy that finds no slab free, or that is on a stream its threads cannot name
// (cudaStreamPerThread), is the plain copy.
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

#include "rgs_internal.cuh"

namespace rgs {

namespace {

constexpr size_t HC_CHUNK = 1 << 20;
constexpr int HC_THREADS = 8;
constexpr int HC_SLABS = 2 * HC_THREADS;
constexpr size_t HC_BLOCK = HC_SLABS * HC_CHUNK;
constexpr size_t HC_HUGE = 2 << 20;
constexpr size_t HC_FIRST = 32 << 20;

struct Pool {
    std::mutex mu;
    void* map = nullptr;  // the block's mapping, HC_BLOCK + HC_HUGE bytes
    char* block = nullptr;
    void* idle[HC_SLABS];
    int idle_n = 0, users = 0;
    size_t seen = 0;  // bytes of large copies while there was no block
};
Pool& pool() {
    static Pool* p = new Pool;  // outlives static destruction: contexts may too
    return *p;
}

// Another thread of the program may be capturing a graph in a mode that would refuse
// this thread's call outside the relaxed mode.
template <class Call>
cudaError_t relaxed(const Call& call) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const cudaError_t e = call();
    cudaThreadExchangeStreamCaptureMode(&mode);
    return e;
}

void make_block(Pool& p) {
    void* m = mmap(nullptr, HC_BLOCK + HC_HUGE, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == MAP_FAILED) return;
    char* q = (char*)(((uintptr_t)m + HC_HUGE - 1) & ~(uintptr_t)(HC_HUGE - 1));
    madvise(q, HC_BLOCK, MADV_HUGEPAGE);  // a hint: small pages do the same, slower
    const cudaError_t e = relaxed([&] { return cudaHostRegister(q, HC_BLOCK, cudaHostRegisterPortable); });
    if (e != cudaSuccess) {
        cudaGetLastError();
        munmap(m, HC_BLOCK + HC_HUGE);
        return;
    }
    p.map = m;
    p.block = q;
    for (int k = 0; k < HC_SLABS; ++k) p.idle[k] = q + (size_t)k * HC_CHUNK;
    p.idle_n = HC_SLABS;
}

// With no context left and every slab back. A block that the driver does not let go
// stays mapped, for the next context: its addresses must not become another array's
// while they are taken for page-locked.
void free_block(Pool& p) {
    if (p.users != 0 || p.idle_n != (p.block ? HC_SLABS : 0)) return;
    if (p.block) {
        if (relaxed([&] { return cudaHostUnregister(p.block); }) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        munmap(p.map, HC_BLOCK + HC_HUGE);
    }
    p.map = nullptr;
    p.block = nullptr;
    p.idle_n = 0;
    p.seen = 0;
}

// Up to n slabs (an even number) for a copy of `bytes`.
int take(int n, size_t bytes, void** got) {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    if (!p.block) {
        p.seen += bytes;
        if (p.seen >= HC_FIRST) make_block(p);
    }
    n = std::min(n, p.idle_n) & ~1;
    for (int k = 0; k < n; ++k) got[k] = p.idle[--p.idle_n];
    return n;
}

void give(int n, void* const* slabs) {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    for (int k = 0; k < n; ++k) p.idle[p.idle_n++] = slabs[k];
    free_block(p);
}

struct Job {
    char* host;
    char* dev;
    size_t bytes;
    bool to_host;
    cudaStream_t st;
    int device;
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};

    void failed(cudaError_t e) {
        int ok = (int)cudaSuccess;
        if (e != cudaSuccess) err.compare_exchange_strong(ok, (int)e);
    }
    // Claims a chunk; false when none is left or a thread failed.
    bool claim(size_t& off, size_t& len) {
        off = next.fetch_add(1) * HC_CHUNK;
        if (off >= bytes || err.load() != (int)cudaSuccess) return false;
        len = std::min(HC_CHUNK, bytes - off);
        return true;
    }
    void run(void* slab0, void* slab1) {
        void* slab[2] = {slab0, slab1};
        cudaEvent_t ev[2] = {nullptr, nullptr};
        cudaError_t e = cudaSetDevice(device);
        for (int b = 0; b < 2 && e == cudaSuccess; ++b) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
        failed(e);
        if (e == cudaSuccess) {
            if (to_host) receive(slab, ev);
            else send(slab, ev);
        }
        for (cudaEvent_t v : ev)
            if (v) cudaEventDestroy(v);
    }
    void receive(void* const slab[2], const cudaEvent_t ev[2]) {
        size_t off[2] = {0, 0}, len[2] = {0, 0};
        bool live[2] = {false, false};
        auto issue = [&](int b) {
            live[b] = claim(off[b], len[b]);
            if (!live[b]) return;
            cudaError_t e = cudaMemcpyAsync(slab[b], dev + off[b], len[b], cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaEventRecord(ev[b], st);
            failed(e);
            live[b] = e == cudaSuccess;
        };
        issue(0);
        for (int b = 0; live[b]; b ^= 1) {
            issue(b ^ 1);
            const cudaError_t e = cudaEventSynchronize(ev[b]);
            failed(e);
            if (e == cudaSuccess) std::memcpy(host + off[b], slab[b], len[b]);
        }
    }
    void send(void* const slab[2], const cudaEvent_t ev[2]) {
        bool used[2] = {false, false};
        size_t off, len;
        for (int b = 0; claim(off, len); b ^= 1) {
            cudaError_t e = used[b] ? cudaEventSynchronize(ev[b]) : cudaSuccess;
            if (e == cudaSuccess) {
                std::memcpy(slab[b], host + off, len);
                e = cudaMemcpyAsync(dev + off, slab[b], len, cudaMemcpyHostToDevice, st);
            }
            if (e == cudaSuccess) e = cudaEventRecord(ev[b], st);
            used[b] = e == cudaSuccess;
            failed(e);
        }
        // the slabs go back to the pool: wait for what is still on the bus
        for (int b = 0; b < 2; ++b)
            if (used[b]) failed(cudaEventSynchronize(ev[b]));
    }
};

cudaError_t host_copy(void* host, void* dev, size_t bytes, bool to_host, cudaStream_t st) {
    const auto plain = [&] {
        return to_host ? cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st)
                       : cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    };
    // the workers issue on the caller's stream; cudaStreamPerThread would be another
    // stream in each of them, ordered after nothing the caller queued. (One thread
    // issuing every transfer for workers that only copy takes any handle, but its
    // hand-overs made writes of 9.4 and 24 MB 0.46 -> 0.75 and 0.91 -> 1.6 ms.)
    if (bytes < HOST_COPY_MIN || st == cudaStreamPerThread) return plain();
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        cudaGetLastError();
        return plain();
    }
    if (at.type != cudaMemoryTypeUnregistered) return plain();  // page-locked already
    const int cores = (int)std::max(1u, std::thread::hardware_concurrency());
    const int want = std::min({HC_THREADS, cores, (int)(bytes >> 21)});
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    void* slabs[HC_SLABS];
    const int got = take(2 * want, bytes, slabs);
    if (got == 0) return plain();
    std::thread threads[HC_THREADS];
    Job job;
    job.host = (char*)host;
    job.dev = (char*)dev;
    job.bytes = bytes;
    job.to_host = to_host;
    job.st = st;
    job.device = device;
    try {
        for (int k = 2; k < got; k += 2) threads[k / 2] = std::thread(&Job::run, &job, slabs[k], slabs[k + 1]);
    } catch (...) {  // fewer threads than asked for do the same work
    }
    job.run(slabs[0], slabs[1]);
    for (std::thread& t : threads)
        if (t.joinable()) t.join();
    e = (cudaError_t)job.err.load();
    if (e != cudaSuccess) cudaStreamSynchronize(st);  // no slab goes back with a copy in flight
    give(got, slabs);
    return e;
}

}  // namespace

cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    return host_copy(dst, const_cast<void*>(src), bytes, true, st);
}
cudaError_t copy_from_host(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    return host_copy(const_cast<void*>(src), dst, bytes, false, st);
}

void host_copy_user(int add) {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    p.users += add;
    free_block(p);
}

}  // namespace rgs
