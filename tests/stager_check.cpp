// The upload ring on the CPU (tests/test_stager.py): stager_check MODE, 0 when it holds.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <ctime>
#include <string>

#include "stager.h"

using tk::Stager;
using tk::Uploads;

static bool no_ring = false;

static std::vector<uint8_t> bytes(size_t n, uint32_t seed) {
    std::vector<uint8_t> v(n);
    uint32_t x = seed * 2654435761u + 1u;
    for (size_t i = 0; i < n; ++i) {
        x = x * 1664525u + 1013904223u;
        v[i] = uint8_t(x >> 24);
    }
    return v;
}

static void rest(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }

// Uploads of the sizes from several threads through one ring, as the library makes them.
static int data() {
    auto ring = Stager::of(0, no_ring);
    std::atomic<int> wrong{0};
    auto round = [&](uint32_t seed) {
        FakeStream st;
        for (size_t n : {size_t(1), Stager::kChunk, Stager::kChunk * Stager::kRing + 1, Stager::kLarge,
                         Stager::kLarge + Stager::kChunk / 2 + 3}) {
            const auto src = bytes(n, seed + uint32_t(n));
            std::vector<uint8_t> dst(n, 0);
            cudaError_t e = ring->copy(dst.data(), src.data(), n, &st);
            if (e == cudaErrorNotReady) e = cudaMemcpyAsync(dst.data(), src.data(), n, cudaMemcpyHostToDevice, &st);
            st.drain();
            if (e != cudaSuccess || dst != src) ++wrong;
        }
    };
    round(1);
    if (fake.plain_copies) return 2;  // nobody else had the ring
    std::vector<std::thread> ts;
    for (uint32_t k = 0; k < 3; ++k) ts.emplace_back(round, 10 * k);
    for (auto& t : ts) t.join();
    return wrong ? 1 : 0;
}

// An upload behind a stream that is busy: the CPU time of 400 ms of waiting, in per cent of one core.
static int busy() {
    auto ring = Stager::of(0, no_ring);
    FakeStream st;
    const size_t n = Stager::kChunk * Stager::kRing * 4;
    const auto src = bytes(n, 5);
    std::vector<uint8_t> dst(n, 0);
    st.gate(false);
    std::thread t([&] { ring->copy(dst.data(), src.data(), n, &st); });
    rest(300);  // the ring is full
    const std::clock_t c0 = std::clock();
    rest(400);
    const double used = double(std::clock() - c0) / CLOCKS_PER_SEC / 0.4;
    st.gate(true);
    t.join();
    std::printf("%.1f%% of a core\n", 100.0 * used);
    return dst != src ? 1 : used > 0.25 ? 2 : 0;
}

// A copy out of the ring that fails, behind a busy stream: the error comes back, and the
// chunks that were issued before arrive as they were, whatever the ring does next.
static int fail() {
    auto ring = Stager::of(0, no_ring);
    FakeStream st;
    const size_t n = Stager::kChunk * Stager::kRing * 4;
    const auto src = bytes(n, 6), other = bytes(n, 7);
    std::vector<uint8_t> dst(n, 0), dst2(n, 0);
    for (int at : {0, 2, int(Stager::kRing) + 1}) {
        std::fill(dst.begin(), dst.end(), uint8_t(0));
        fake.ring_copies = 0;
        fake.fail_copy = at;
        // up to the half of the ring after which the copy itself waits for the stream
        const bool closed = at < int(Stager::kRing) / 2;
        if (closed) st.gate(false);
        cudaError_t e = cudaSuccess;
        std::thread t([&] { e = ring->copy(dst.data(), src.data(), n, &st); });
        if (closed) {
            rest(200);
            st.gate(true);
        }
        t.join();
        st.drain();
        fake.fail_copy = -1;
        const size_t sent = size_t(at) * Stager::kChunk;
        if (e != cudaErrorInvalidValue) return 1;
        if (std::memcmp(dst.data(), src.data(), sent)) return 2;
        for (size_t i = sent; i < n; ++i)
            if (dst[i]) return 3;
        if (ring->copy(dst2.data(), other.data(), n, &st) != cudaSuccess) return 4;
        st.drain();
        if (dst2 != other) return 5;
    }
    return 0;
}

// A context's uploads: which of them take the ring, and that a ring that cannot be made is
// asked for once.
static int context() {
    FakeStream st;
    const size_t n = Stager::kLarge, enough = Stager::kPays / n;
    const auto src = bytes(n + 7, 8);
    std::vector<uint8_t> dst(n + 7);
    auto put = [&](Uploads& u, size_t len) {
        std::fill(dst.begin(), dst.end(), uint8_t(0));
        if (u.copy(0, dst.data(), src.data(), len, &st) != cudaSuccess) return false;
        st.drain();
        return std::equal(dst.begin(), dst.begin() + len, src.begin());
    };
    {
        Uploads u;
        fake.fail_alloc = true;
        for (size_t k = 0; k < 3 * enough; ++k)
            if (!put(u, n)) return 1;
        if (fake.host_allocs != 1 || fake.ring_copies != 0) return 2;
        fake.fail_alloc = false;
    }
    Uploads u;
    fake.host_allocs = 0;
    for (size_t k = 0; k + 1 < enough; ++k)
        if (!put(u, n)) return 3;
    if (!put(u, n - 1) || fake.host_allocs != 0) return 4;  // not large, and not yet enough
    if (!put(u, n) || fake.host_allocs != 1 || fake.ring_copies != int(n / Stager::kChunk)) return 5;
    if (!put(u, n + 7) || fake.ring_copies != int(2 * (n / Stager::kChunk) + 1)) return 6;
    const int before = fake.ring_copies;
    if (!put(u, n - 1) || fake.ring_copies != before) return 7;
    // arrays that several threads have just written, from kWritten on
    for (size_t len : {Stager::kWritten - 1, Stager::kWritten}) {
        if (u.copy(0, dst.data(), src.data(), len, &st, true) != cudaSuccess) return 8;
        st.drain();
        if (fake.ring_copies != before + int(len / Stager::kWritten * (Stager::kWritten / Stager::kChunk))) return 9;
    }
    return 0;
}

int main(int argc, char** argv) {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "data") return data();
    if (mode == "busy") return busy();
    if (mode == "fail") return fail();
    if (mode == "context") return context();
    return 100;
}
