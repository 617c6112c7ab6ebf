// A stand-in for the part of the CUDA runtime that stager.h calls, for tests on the CPU:
// a stream is a thread that does its operations in order, while its gate is open.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <thread>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2, cudaErrorNotReady = 600 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1 };
enum { cudaHostAllocDefault = 0, cudaEventDisableTiming = 2 };
struct cudaPointerAttributes { cudaMemoryType type; };

struct FakeStream {
    std::mutex m;
    std::condition_variable cv;
    std::deque<std::function<void()>> ops;
    bool open = true, quit = false, busy = false;
    std::thread worker{[this] {
        std::unique_lock<std::mutex> lock(m);
        for (;;) {
            cv.wait(lock, [&] { return quit || (open && !ops.empty()); });
            if (quit && ops.empty()) return;
            auto op = std::move(ops.front());
            ops.pop_front();
            busy = true;
            lock.unlock();
            op();
            lock.lock();
            busy = false;
            cv.notify_all();
        }
    }};
    void push(std::function<void()> op) {
        std::lock_guard<std::mutex> lock(m);
        ops.push_back(std::move(op));
        cv.notify_all();
    }
    void gate(bool is_open) {
        std::lock_guard<std::mutex> lock(m);
        open = is_open;
        cv.notify_all();
    }
    void drain() {
        std::unique_lock<std::mutex> lock(m);
        cv.wait(lock, [&] { return ops.empty() && !busy; });
    }
    ~FakeStream() {
        drain();
        {
            std::lock_guard<std::mutex> lock(m);
            quit = true;
            cv.notify_all();
        }
        worker.join();
    }
};
using cudaStream_t = FakeStream*;

struct FakeEvent {
    std::mutex m;
    std::condition_variable cv;
    uint64_t recorded = 0, done = 0;
};
using cudaEvent_t = FakeEvent*;

struct FakeState {
    std::atomic<int> host_allocs{0}, ring_copies{0}, plain_copies{0};
    std::atomic<int> fail_copy{-1};  // the ring copy that fails, counted from 0
    std::atomic<bool> fail_alloc{false};
    std::atomic<uint8_t*> pinned{nullptr};
    std::atomic<size_t> pinned_bytes{0};
};
inline FakeState fake;

inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void*) {
    at->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    ++fake.host_allocs;
    if (fake.fail_alloc) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    fake.pinned = static_cast<uint8_t*>(*p);
    fake.pinned_bytes = n;
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = new FakeEvent;
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete e;
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    uint64_t mark;
    {
        std::lock_guard<std::mutex> lock(e->m);
        mark = ++e->recorded;
    }
    st->push([e, mark] {
        std::lock_guard<std::mutex> lock(e->m);
        e->done = mark;
        e->cv.notify_all();
    });
    return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::unique_lock<std::mutex> lock(e->m);
    e->cv.wait(lock, [&] { return e->done == e->recorded; });
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    st->drain();
    return cudaSuccess;
}
// From the ring: done in its turn. From elsewhere (pageable memory): done on return.
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t st) {
    const uint8_t *s = static_cast<const uint8_t*>(src), *p = fake.pinned;
    if (p && s >= p && s < p + fake.pinned_bytes) {
        if (fake.ring_copies++ == fake.fail_copy) return cudaErrorInvalidValue;
        st->push([=] { std::memcpy(dst, src, n); });
    } else {
        ++fake.plain_copies;
        st->drain();
        std::memcpy(dst, src, n);
    }
    return cudaSuccess;
}
