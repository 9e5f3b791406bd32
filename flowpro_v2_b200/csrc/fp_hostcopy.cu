// Large copies between device memory and pageable host memory.
//
// A pageable copy goes through the driver's staging buffer on one thread, which also takes the page
// faults of a fresh destination: 38 MB (200,568 triangles of 24 unknowns) took 8.2 to 17 ms down,
// where the link needs 0.8.  Here the chunks go through pinned staging slots while several threads copy
// between the slots and the caller's memory, each its slice of every chunk: 2.5 ms.  Copies below
// kLeastDown and kLeastUp, pinned host memory and calls that find the staging memory in use by another thread take
// the plain cudaMemcpyAsync.
//
// Smaller slots were measured: 38 MB down / up, ms, 6 slots of 2 MB 2.5 / 2.3, 6 of 1 MB 2.45 / 2.1, 4 of 1 MB
// 2.65 / 1.85, 6 of 512 KB 2.8 / 1.8; but with 1 MB (slices of 128 KB) the threads' page faults meet in the same
// 2 MB of the destination, and 27 to 33 MB take 0.4 ms longer.  Pinning the 12 MB (5.0 to 8.4 ms, once while
// there are contexts) is part of the first copy that is large enough.  The threads exist only while the
// link is at work: the stream's earlier work is waited for first.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "fp_ctx.h"

namespace fp {

namespace {

constexpr size_t kSlotBytes = (size_t)2 << 20;
constexpr int kSlots = 6;
// Smallest copies that gain.  Below, starting the threads and their page faults in one address space cost
// more than they save.  Five explicit steps with the state read into a new array, ms, plain and staged: 2.7
// MB 1.10 and 1.67, 4.6 MB 1.57 and 2.35, 7.4 MB 2.05 and 2.9, 11.4 MB 2.97 and 3.6, 15.3 MB 3.7 and 4.0, 22.8 MB
// 5.2 and 5.0, 29.2 MB 6.6 and 5.8; the copy alone from 32.5 MB, where such an array is always fresh
// memory, 8.0 and 2.65.  Up: 16 MB 0.96 and 1.48, 27 MB 1.69 and 1.72, 32.5 MB 2.4 and 1.92, 65 MB 5.9 and 3.2.
constexpr size_t kLeastDown = (size_t)20 << 20, kLeastUp = (size_t)32 << 20;
constexpr unsigned kMostThreads = 8;

// One staging buffer per process, held by one copy at a time, freed with the last context.
struct Staging {
    std::mutex use, life;
    char* buf = nullptr;
    int contexts = 0;
};
Staging& staging() {
    static Staging s;
    return s;
}

bool pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// the threads that copy slices between the host memory and the slots
struct Copiers {
    char* host;
    char* slots;
    size_t bytes;
    bool down;
    int chunks, threads = 0;
    std::atomic<int> open{0};      // chunks a thread may copy
    std::atomic<bool> stop{false};
    std::unique_ptr<std::atomic<int>[]> done;  // threads that have copied a chunk
    std::vector<std::thread> pool;

    Copiers(char* h, char* s, size_t n, bool d)
        : host(h), slots(s), bytes(n), down(d), chunks((int)((n + kSlotBytes - 1) / kSlotBytes)),
          done(new std::atomic<int>[chunks]) {
        for (int k = 0; k < chunks; k++) done[k].store(0);
    }
    size_t size(int k) const { return std::min(kSlotBytes, bytes - (size_t)k * kSlotBytes); }
    void slice(int t, int k) {
        const size_t n = size(k), part = ((n + threads - 1) / threads + 4095) / 4096 * 4096;
        const size_t a = std::min(n, t * part), b = std::min(n, a + part);
        char *h = host + (size_t)k * kSlotBytes + a, *s = slots + (size_t)(k % kSlots) * kSlotBytes + a;
        if (b > a) std::memcpy(down ? h : s, down ? s : h, b - a);
        done[k].fetch_add(1, std::memory_order_release);
    }
    bool start(int n) {
        threads = n;
        try {
            for (int t = 0; t < n; t++)
                pool.emplace_back([this, t] {
                    for (int k = 0; k < chunks; k++) {
                        while (open.load(std::memory_order_acquire) <= k) {
                            if (stop.load(std::memory_order_acquire)) return;
                            std::this_thread::yield();
                        }
                        slice(t, k);
                    }
                });
        } catch (...) {  // no threads to be had: nothing has been opened, they all end
            stop.store(true, std::memory_order_release);
            return false;
        }
        return true;
    }
    bool finished(int k) const { return done[k].load(std::memory_order_acquire) == threads; }
    void await(int k) const {
        while (!finished(k)) std::this_thread::yield();
    }
    ~Copiers() {
        stop.store(true, std::memory_order_release);
        for (auto& t : pool) t.join();
    }
};

// the copy through the staging slots; *taken false: not applicable here, nothing has been copied
int staged_copy(fp_ctx* c, void* host, void* dev, size_t bytes, bool down, bool* taken) {
    *taken = false;
    if (bytes < (down ? kLeastDown : kLeastUp) || !pageable(host)) return FP_OK;
    Staging& S = staging();
    std::unique_lock<std::mutex> lock(S.use, std::try_to_lock);
    if (!lock.owns_lock()) return FP_OK;
    if (!S.buf && cudaHostAlloc((void**)&S.buf, kSlots * kSlotBytes, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        S.buf = nullptr;
        return FP_OK;
    }
    // before any thread waits for a chunk: on the caller's stream the work ahead may be long
    int rc = cuda_check(c, cudaStreamSynchronize(c->stream), "sync");
    if (rc) return rc;
    Copiers C((char*)host, S.buf, bytes, down);
    cudaEvent_t ev[kSlots] = {};
    for (auto& e : ev)
        if (!rc) rc = cuda_check(c, cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
    auto slot = [&](int k) { return S.buf + (size_t)(k % kSlots) * kSlotBytes; };
    auto at = [&](int k) { return (char*)dev + (size_t)k * kSlotBytes; };
    auto transfer = [&](int k) {  // chunk k between its slot and the device
        void *to = down ? slot(k) : at(k), *from = down ? at(k) : slot(k);
        rc = cuda_check(c, cudaMemcpyAsync(to, from, C.size(k), down ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, c->stream),
                        down ? "download" : "upload");
        if (!rc) rc = cuda_check(c, cudaEventRecord(ev[k % kSlots], c->stream), "event");
    };
    int issued = 0;
    if (down)  // on their way while the threads start
        for (; issued < std::min(C.chunks, kSlots) && !rc; issued++) transfer(issued);
    const unsigned hw = std::thread::hardware_concurrency();
    if (!rc && C.start((int)std::max(1u, std::min(kMostThreads, hw / 2)))) {
        *taken = true;
        if (down) {
            for (int k = 0; k < C.chunks && !rc; k++) {
                while (issued < C.chunks && issued < k + kSlots && !rc) {
                    if (issued > k && !C.finished(issued - kSlots)) break;  // later: chunk k is on its way
                    C.await(issued - kSlots);
                    transfer(issued++);
                }
                if (!rc) rc = cuda_check(c, cudaEventSynchronize(ev[k % kSlots]), "sync");
                if (!rc) C.open.store(k + 1, std::memory_order_release);
            }
            for (int k = std::max(0, C.chunks - kSlots); k < C.chunks && !rc; k++) C.await(k);
        } else {
            C.open.store(std::min(C.chunks, kSlots), std::memory_order_release);
            for (int k = 0; k < C.chunks && !rc; k++) {
                C.await(k);
                transfer(k);
                if (!rc && k >= 1) {  // the slot of chunk k - 1 takes chunk k - 1 + kSlots
                    rc = cuda_check(c, cudaEventSynchronize(ev[(k - 1) % kSlots]), "sync");
                    C.open.store(std::min(C.chunks, k + kSlots), std::memory_order_release);
                }
            }
            // the slots are free again when the last copies have left them
            if (!rc) rc = cuda_check(c, cudaEventSynchronize(ev[(C.chunks - 1) % kSlots]), "sync");
        }
    }
    if (rc || !*taken) cudaStreamSynchronize(c->stream);  // no copy may use the slots after this
    for (auto& e : ev)
        if (e) cudaEventDestroy(e);
    return rc;
}

// the same without exceptions: what can throw (host memory for the bookkeeping, the lock) does so before the
// first transfer
int staged(fp_ctx* c, void* host, void* dev, size_t bytes, bool down, bool* taken) {
    try {
        return staged_copy(c, host, dev, bytes, down, taken);
    } catch (...) {
        *taken = false;
        return FP_OK;
    }
}

}  // namespace

void staging_retain() {
    Staging& S = staging();
    std::lock_guard<std::mutex> l(S.life);
    S.contexts++;
}

void staging_release() {
    Staging& S = staging();
    std::lock_guard<std::mutex> l(S.life);
    if (--S.contexts == 0) {
        std::lock_guard<std::mutex> u(S.use);
        if (S.buf) cudaFreeHost(S.buf);
        S.buf = nullptr;
    }
}

int copy_to_host(fp_ctx* c, void* host, const void* dev, size_t bytes) {
    bool taken = false;
    int rc = staged(c, host, const_cast<void*>(dev), bytes, true, &taken);
    if (rc || taken) return rc;
    if ((rc = cuda_check(c, cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, c->stream), "download"))) return rc;
    return cuda_check(c, cudaStreamSynchronize(c->stream), "sync");
}

int copy_to_device(fp_ctx* c, void* dev, const void* host, size_t bytes) {
    bool taken = false;
    int rc = staged(c, const_cast<void*>(host), dev, bytes, false, &taken);
    if (rc || taken) return rc;
    return cuda_check(c, cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, c->stream), "upload");
}

}  // namespace fp
