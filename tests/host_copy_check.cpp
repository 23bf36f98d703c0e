// Runs csrc/host_copy.cpp on a CUDA runtime made of host memory: streams that do their copies only when somebody waits for
// them, and allocations that can be made to fail.  One check per run, named by the first argument; exit code 0 if it holds.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <chrono>
#include <functional>
#include <string>
#include <thread>
#include <vector>

#include "host_copy.h"

namespace {
thread_local int t_device = 0;
struct FakeStream {
    const int device = t_device;
    std::mutex mu;
    std::vector<std::function<void()>> ops;
    size_t done = 0;
    void drain(size_t upto) {
        std::lock_guard<std::mutex> lock(mu);
        for (; done < upto && done < ops.size(); ++done) {
            std::this_thread::sleep_for(std::chrono::milliseconds(2));      // the copy engine takes its time
            ops[done]();
        }
    }
};
struct FakeEvent { FakeStream* stream = nullptr; size_t upto = 0; };
std::atomic<int> g_pinned_left(1 << 20), g_streams_left(1 << 20), g_pinned_live(0), g_plain_copies(0), g_away(0);
int g_home = 0;                          // the device whose memory is copied
}  // namespace

extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    if (g_streams_left.fetch_sub(1) <= 0) { *s = nullptr; return cudaErrorMemoryAllocation; }
    *s = reinterpret_cast<cudaStream_t>(new FakeStream);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete reinterpret_cast<FakeStream*>(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { reinterpret_cast<FakeStream*>(s)->drain(~size_t(0)); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(new FakeEvent); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<FakeEvent*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    FakeEvent* ev = reinterpret_cast<FakeEvent*>(e);
    ev->stream = reinterpret_cast<FakeStream*>(s);
    std::lock_guard<std::mutex> lock(ev->stream->mu);
    ev->upto = ev->stream->ops.size();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    FakeEvent* ev = reinterpret_cast<FakeEvent*>(e);
    if (ev->stream) ev->stream->drain(ev->upto);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    if (!dst || !src) return cudaErrorInvalidValue;
    FakeStream* st = reinterpret_cast<FakeStream*>(s);
    if (st->device != g_home) ++g_away;
    std::lock_guard<std::mutex> lock(st->mu);
    st->ops.push_back([=] { memcpy(dst, src, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind) { ++g_plain_copies; memcpy(dst, src, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (g_pinned_left.fetch_sub(1) <= 0) { *p = nullptr; return cudaErrorMemoryAllocation; }
    ++g_pinned_live;
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { --g_pinned_live; free(p); return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}

namespace {

std::vector<unsigned char> pattern(size_t n, unsigned seed) {
    std::vector<unsigned char> v(n);
    unsigned s = seed * 2654435761u + 1;
    for (auto& b : v) { s = s * 1664525u + 1013904223u; b = static_cast<unsigned char>(s >> 24); }
    return v;
}

// One copy in each direction; true if every byte arrived.
bool round_trip(vdnn::HostCopy& copy, size_t bytes, unsigned seed) {
    const std::vector<unsigned char> want = pattern(bytes, seed);
    std::vector<unsigned char> got(bytes, 0), there(bytes, 0);
    if (copy.to_host(got.data(), want.data(), bytes, g_home) != cudaSuccess || got != want) return false;
    return copy.to_device(there.data(), want.data(), bytes, g_home) == cudaSuccess && there == want;
}

// Several threads use one object at once: small copies, which share a staging buffer, and large ones, which share the threads.
int concurrent() {
    vdnn::HostCopy copy;
    std::atomic<int> bad(0);
    std::vector<std::thread> threads;
    for (unsigned t = 0; t < 6; ++t)
        threads.emplace_back([&, t] {
            for (unsigned i = 0; i < 6; ++i)
                if (!round_trip(copy, t % 2 ? (400u << 10) + t : (5u << 20) + 3 * t, 10 * t + i)) ++bad;
        });
    for (auto& t : threads) t.join();
    return bad == 0 ? 0 : 1;
}

// Pinned memory or streams run out: before the first worker, in the middle of the second, or after it.  Copies go on with what
// there is, nothing half-made is kept, and what comes free later is used.
int scarce(int pinned, int streams) {
    {
        vdnn::HostCopy copy;
        g_pinned_left = pinned;
        g_streams_left = streams;
        for (unsigned i = 0; i < 2; ++i)
            if (!round_trip(copy, 300u << 10, i) || !round_trip(copy, (9u << 20) + 5, i + 2)) return 1;
        if (g_pinned_live % 2 != 0 || g_pinned_live > pinned) return 3;                 // two buffers to a worker
        if ((pinned < 2 || streams < 1) && g_plain_copies == 0) return 4;
        g_pinned_left = g_streams_left = 1 << 20;
        const int before = g_pinned_live;
        if (!round_trip(copy, (9u << 20) + 5, 7)) return 1;
        if (g_pinned_live < 2 || g_pinned_live < before) return 5;
    }
    return g_pinned_live == 0 ? 0 : 6;
}

// A thread whose current device is another one reads and writes: its device stays as it was, and the work is done on the
// memory's own device, whichever copy comes first.
int device() {
    g_home = 3;
    t_device = 1;
    for (int first = 0; first < 2; ++first) {
        vdnn::HostCopy copy;
        for (unsigned i = 0; i < 2; ++i) {
            if (!round_trip(copy, static_cast<int>(i) == first ? 300u << 10 : 9u << 20, i)) return 1;
            if (t_device != 1) return 3;
        }
    }
    return g_away == 0 ? 0 : 4;
}

}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "concurrent") return concurrent();
    if (what == "device") return device();
    if (what == "scarce" && argc == 4) return scarce(atoi(argv[2]), atoi(argv[3]));
    return 2;
}
