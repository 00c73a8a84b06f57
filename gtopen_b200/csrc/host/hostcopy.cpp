#include "hostcopy.hpp"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "core.hpp"

namespace gtob {
namespace {

constexpr size_t kSmall = size_t(1) << 20;  // below: one plain copy

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw Error(std::string("cuda: ") + cudaGetErrorString(e) + " at " + what);
}
struct Events {
    cudaEvent_t ev[2] = {nullptr, nullptr};
    Events() {
        for (auto& e : ev) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    }
    ~Events() {
        for (auto& e : ev)
            if (e) {
                cudaEventSynchronize(e);  // an error path: the chunk may still be in flight
                cudaEventDestroy(e);
            }
    }
};
// Chunk j's bytes are moved by `nt` threads, slice by slice (fewer where the
// system starts no more); `turn` lets them start on a chunk, `done` counts the
// slices of each.
struct Crew {
    int nt;
    std::atomic<size_t> turn{0};
    std::atomic<bool> stop{false};
    std::vector<std::atomic<int>> done;
    std::vector<std::thread> ts;
    Crew(int n, size_t chunks) : nt(n), done(chunks) {
        for (auto& d : done) d = 0;
    }
    template <class F>
    void start(F move) {
        auto work = [this, move](int w) {
            for (size_t j = 0; j < done.size(); j++) {
                while (turn.load(std::memory_order_acquire) <= j) {
                    if (stop.load()) return;
                    std::this_thread::yield();
                }
                move(j, w, nt);
                done[j].fetch_add(1, std::memory_order_release);
            }
        };
        ts.reserve((size_t)nt);
        for (int w = 1; w < nt; w++) {
            try {
                ts.emplace_back(work, w);
            } catch (const std::system_error&) {
                nt = w;  // before the first turn: nobody has read it
            }
        }
    }
    void wait(size_t j) const {
        while (done[j].load(std::memory_order_acquire) < nt) std::this_thread::yield();
    }
    ~Crew() {
        stop = true;
        for (auto& t : ts) t.join();
    }
};

}  // namespace

void copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t s, unsigned char* pin) {
    if (bytes < kSmall || !pin) {
        if (bytes) ck(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
        ck(cudaStreamSynchronize(s), "cudaStreamSynchronize");
        return;
    }
    const size_t nc = (bytes + kPinChunk - 1) / kPinChunk;
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const int threads = (int)std::min<size_t>(std::min(8u, hw), std::max<size_t>(1, bytes / (kSmall / 2)));
    Events E;
    Crew crew(threads, nc);
    auto count = [=](size_t j) { return std::min(kPinChunk, bytes - j * kPinChunk); };
    auto move = [=](size_t j, int w, int nt) {
        const size_t n = count(j), pages = (n + 4095) / 4096, per = (pages + nt - 1) / nt * 4096;
        const size_t a = std::min(n, w * per), e = std::min(n, (w + 1) * per);
        std::memcpy((unsigned char*)dst + j * kPinChunk + a, pin + (j & 1) * kPinChunk + a, e - a);
    };
    auto issue = [&](size_t j) {
        ck(cudaMemcpyAsync(pin + (j & 1) * kPinChunk, (const unsigned char*)src + j * kPinChunk, count(j),
                           cudaMemcpyDeviceToHost, s),
           "cudaMemcpyAsync");
        ck(cudaEventRecord(E.ev[j & 1], s), "cudaEventRecord");
    };
    issue(0);
    crew.start(move);
    for (size_t j = 0; j < nc; j++) {
        if (j + 1 < nc) {
            if (j > 0) crew.wait(j - 1);  // its buffer is the next one's
            issue(j + 1);
        }
        ck(cudaEventSynchronize(E.ev[j & 1]), "cudaEventSynchronize");
        crew.turn.store(j + 1, std::memory_order_release);
        move(j, 0, crew.nt);
        crew.done[j].fetch_add(1, std::memory_order_release);
    }
    for (size_t j = nc > 2 ? nc - 2 : 0; j < nc; j++) crew.wait(j);
}

}  // namespace gtob
