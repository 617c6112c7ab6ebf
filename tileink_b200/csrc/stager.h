// Uploads of large pageable host arrays: several threads copy them into a ring
// of pinned chunks while the copy engine drains it.
#pragma once
#include <cuda_runtime.h>
#include <pthread.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace tk {

// A copy from pageable memory goes through the driver's own pinned buffer, one host
// thread filling it: 11 GB/s, or 20 where the source is in the CPU's caches, against 49
// from pinned memory. With the ring a page of 20,000 glyph outlines (77 MB of elements)
// takes 7.0 ms from record to image, without it 10.5.
// Two threads beside the caller's fill it: with six, and chunks of 256 KB, waking them and
// their turns at the chunks cost 0.3 ms a copy, and 16 MB from the caches took 1.09 ms,
// through the driver 0.84; now 0.85 (24 MB 1.08 against 1.25; not cached 16 MB 1.00 against
// 1.53, 128 MB 5.6 against 11.9). Below kLarge the driver is as fast, except on arrays that
// several threads have just written: they lie in those cores' caches, from which one thread
// reads 5.5 GB/s (the 5.6 MB of weights of a differentiable step: 1.0 ms; from kWritten
// on they take the ring, 6.2 -> 5.9 ms a step's forward).
// The ring and its threads are shared by the contexts of a device: made for a
// context whose large uploads come to kPays, given back with the last context
// that used them. 4 MB take about 2.7 ms to make, which 64 MB through them win back. One
// copy runs at a time; a second one does not wait, and goes the driver's way.
class Stager {
  public:
    static constexpr size_t kChunk = 512u << 10, kRing = 8, kLarge = 16u << 20, kWritten = 4u << 20, kPays = 64u << 20;
    static constexpr std::chrono::microseconds kPatience{100};

    // The ring of `device` (the current one); null when another device has it, or when it
    // cannot be made (`failed`).
    static std::shared_ptr<Stager> of(int device, bool& failed) {
        static std::mutex m;
        static std::weak_ptr<Stager> shared;
        std::lock_guard<std::mutex> lock(m);
        std::shared_ptr<Stager> s = shared.lock();
        if (!s) {
            s = std::shared_ptr<Stager>(new Stager(device));
            if (!s->start()) {
                failed = true;
                return nullptr;
            }
            shared = s;
        }
        return s->device_ == device ? s : nullptr;
    }
    ~Stager() { stop(); }

    // Whether src should go through a ring: `least` bytes or more, and not pinned already.
    static bool wants(const void* src, size_t bytes, size_t least) {
        if (bytes < least) return false;
        cudaPointerAttributes at{};
        if (cudaPointerGetAttributes(&at, src) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return at.type == cudaMemoryTypeUnregistered;
    }

    // dst[0, bytes) = src on `st`; done when it returns. An error of a copy is
    // returned, and cudaErrorNotReady when the ring is in use (nothing was copied
    // then).
    cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        std::unique_lock<std::mutex> use(use_, std::try_to_lock);
        if (!use) return cudaErrorNotReady;
        const size_t n = (bytes + kChunk - 1) / kChunk;
        for (size_t k = 0; k < kRing; ++k) filled_[k].store(0, std::memory_order_relaxed);
        src_ = static_cast<const uint8_t*>(src);
        bytes_ = bytes;
        limit_.store(kRing, std::memory_order_relaxed);
        next_.store(0, std::memory_order_relaxed);
        {
            std::lock_guard<std::mutex> lock(m_);
            chunks_ = n;
            ++job_;
        }
        wake_.notify_all();
        cudaError_t e = cudaSuccess;
        for (size_t k = 0; k < n && e == cudaSuccess; ++k) {
            // until chunk k is in its slot this thread fills chunks too
            while (filled_[k % kRing].load(std::memory_order_acquire) != k + 1)
                if (!fill_one(n)) std::this_thread::yield();
            const size_t at = k * kChunk, len = bytes - at < kChunk ? bytes - at : kChunk, slot = k % kRing;
            e = cudaMemcpyAsync(static_cast<uint8_t*>(dst) + at, ring_ + slot * kChunk, len, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(done_[slot], st);
            // the slot half a ring back is refilled once its copy is done
            if (e == cudaSuccess && k + 1 >= kRing / 2 && k + kRing / 2 < n) {
                const size_t back = k + 1 - kRing / 2;
                e = cudaEventSynchronize(done_[back % kRing]);
                if (e != cudaSuccess) break;
                limit_.store(back + 1 + kRing);
                if (waiting_.load()) wake_fillers();
            }
        }
        next_.store(n);  // after an error no chunk is taken any more: the slots may still be read
        {
            std::unique_lock<std::mutex> lock(m_);
            chunks_ = 0;  // a thread that wakes from now on finds nothing
            room_.notify_all();
            idle_.wait(lock, [&] { return active_ == 0; });
        }
        if (e != cudaSuccess) {
            cudaStreamSynchronize(st);  // the copies that were issued, out of slots that the next one fills
            return e;
        }
        // the last copy out of the ring ends after the others (one stream)
        return cudaEventSynchronize(done_[(n - 1) % kRing]);
    }

  private:
    explicit Stager(int device) : device_(device) {}
    Stager(const Stager&) = delete;
    Stager& operator=(const Stager&) = delete;

    bool start() {
        const unsigned cores = std::thread::hardware_concurrency();
        const size_t want = cores >= 4 ? 2 : 1;
        bool ok = cudaHostAlloc(reinterpret_cast<void**>(&ring_), kRing * kChunk, cudaHostAllocDefault) == cudaSuccess;
        if (!ok) ring_ = nullptr;
        for (size_t k = 0; ok && k < kRing; ++k)
            ok = cudaEventCreateWithFlags(&done_[k], cudaEventDisableTiming) == cudaSuccess;
        try {
            while (ok && threads_.size() < want) threads_.emplace_back([this] { work(); });
        } catch (...) {  // no thread to be had: as many as there are, and the caller's
        }
        if (!ok) cudaGetLastError();
        return ok;
    }

    void stop() {
        {
            std::lock_guard<std::mutex> lock(m_);
            quit_ = true;
        }
        wake_.notify_all();
        for (std::thread& t : threads_) t.join();
        for (cudaEvent_t e : done_)
            if (e) cudaEventDestroy(e);
        if (ring_) cudaFreeHost(ring_);
    }

    // Fills the next chunk that has a free slot; false when there is none now.
    bool fill_one(size_t n) {
        size_t k = next_.load(std::memory_order_relaxed);
        do {
            if (k >= n || limit_.load() <= k) return false;
        } while (!next_.compare_exchange_weak(k, k + 1, std::memory_order_relaxed));
        const size_t at = k * kChunk, len = bytes_ - at < kChunk ? bytes_ - at : kChunk;
        std::memcpy(ring_ + (k % kRing) * kChunk, src_ + at, len);
        filled_[k % kRing].store(k + 1, std::memory_order_release);
        return true;
    }

    // (limit_ is stored before waiting_ is read, and a thread counts itself in waiting_
    // before it looks at limit_, both in one order for all: one of them sees the other)
    void wake_fillers() {
        { std::lock_guard<std::mutex> lock(m_); }
        room_.notify_all();
    }

    // While the ring is full a thread yields for kPatience (the copy engine frees a slot every
    // 10 us) and then sleeps: the stream may have a long frame to do before the copies.
    void work() {
        pthread_setname_np(pthread_self(), "tileink-upload");
        uint64_t seen = 0;
        std::unique_lock<std::mutex> lock(m_);
        for (;;) {
            wake_.wait(lock, [&] { return quit_ || job_ != seen; });
            if (quit_) return;
            seen = job_;
            const size_t n = chunks_;
            if (!n) continue;  // done without this thread
            ++active_;
            lock.unlock();
            auto since = std::chrono::steady_clock::now();
            while (next_.load(std::memory_order_relaxed) < n) {
                if (fill_one(n)) {
                    since = std::chrono::steady_clock::now();
                } else if (std::chrono::steady_clock::now() - since < kPatience) {
                    std::this_thread::yield();
                } else {
                    lock.lock();
                    ++waiting_;
                    room_.wait(lock, [&] { return !chunks_ || next_.load() >= n || limit_.load() > next_.load(); });
                    --waiting_;
                    lock.unlock();
                    since = std::chrono::steady_clock::now();
                }
            }
            lock.lock();
            if (--active_ == 0) idle_.notify_one();
        }
    }

    const int device_;
    std::mutex use_;  // held by the copy that has the ring
    uint8_t* ring_ = nullptr;
    cudaEvent_t done_[kRing] = {};
    std::vector<std::thread> threads_;
    // the copy in progress
    std::mutex m_;
    std::condition_variable wake_, room_, idle_;
    uint64_t job_ = 0;
    size_t active_ = 0;  // threads in it
    std::atomic<size_t> waiting_{0};  // of them, those that sleep until a slot is free
    size_t chunks_ = 0;
    bool quit_ = false;
    const uint8_t* src_ = nullptr;
    size_t bytes_ = 0;
    std::atomic<size_t> next_{0}, limit_{0};  // chunks taken; chunks whose slots are free
    std::atomic<size_t> filled_[kRing] = {};  // per slot, 1 + the chunk it holds
};

// The uploads of one context from the caller's memory.
class Uploads {
  public:
    // dst[0, bytes) = src on `st`: through the device's ring (the current one's) where that
    // pays, and as cudaMemcpyAsync does it otherwise. written: by several threads, just now.
    cudaError_t copy(int device, void* dst, const void* src, size_t bytes, cudaStream_t st, bool written = false) {
        if (Stager::wants(src, bytes, written ? Stager::kWritten : Stager::kLarge)) {
            large_ += bytes;
            if (!ring_ && !failed_ && large_ >= Stager::kPays) ring_ = Stager::of(device, failed_);
            const cudaError_t e = ring_ ? ring_->copy(dst, src, bytes, st) : cudaErrorNotReady;
            if (e != cudaErrorNotReady) return e;
        }
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    }

  private:
    std::shared_ptr<Stager> ring_;
    uint64_t large_ = 0;   // bytes of large uploads so far
    bool failed_ = false;  // no ring could be made: not tried again
};

}  // namespace tk
