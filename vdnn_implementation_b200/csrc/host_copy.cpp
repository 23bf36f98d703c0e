// See host_copy.h.
#include "host_copy.h"

#include <stdint.h>
#include <string.h>

#include <atomic>
#include <functional>
#include <system_error>
#include <thread>

namespace vdnn {

namespace {
constexpr size_t kChunk = 2u << 20;         // a huge page of the host
constexpr size_t kDirect = 256u << 10;      // below this one cudaMemcpy is the faster way
constexpr unsigned kMaxWorkers = 8;
}  // namespace

HostCopy::~HostCopy() {
    for (Worker& w : workers_) {
        for (int i = 0; i < 2; ++i) {
            if (w.pinned[i]) cudaFreeHost(w.pinned[i]);
            if (w.done[i]) cudaEventDestroy(w.done[i]);
        }
        if (w.stream) cudaStreamDestroy(w.stream);
    }
}

cudaError_t HostCopy::make_workers(size_t want) {
    while (workers_.size() < want) {
        Worker w = {};
        cudaError_t e = cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking);
        for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
            e = cudaEventCreateWithFlags(&w.done[i], cudaEventDisableTiming);
            if (e == cudaSuccess) e = cudaHostAlloc(reinterpret_cast<void**>(&w.pinned[i]), kChunk, cudaHostAllocDefault);
        }
        workers_.push_back(w);              // a half-made worker is released with the rest
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t HostCopy::run(void* host, void* dev, size_t bytes, int device, bool to_host) {
    if (bytes <= kDirect)
        return to_host ? cudaMemcpy(host, dev, bytes, cudaMemcpyDeviceToHost) : cudaMemcpy(dev, host, bytes, cudaMemcpyHostToDevice);
    char* const h = static_cast<char*>(host);
    char* const d = static_cast<char*>(dev);
    // chunk 0 ends at the first 2 MB boundary of the host address
    size_t head = kChunk - (reinterpret_cast<uintptr_t>(h) & (kChunk - 1));
    if (head > bytes) head = bytes;
    const size_t chunks = 1 + (bytes - head + kChunk - 1) / kChunk;
    unsigned cores = std::thread::hardware_concurrency();
    size_t workers = cores > 2 ? cores / 2 : 1;
    if (workers > kMaxWorkers) workers = kMaxWorkers;
    if (workers > chunks) workers = chunks;
    cudaError_t e = make_workers(workers);
    if (e != cudaSuccess) return e;

    std::atomic<size_t> next(0);
    std::atomic<int> failed(static_cast<int>(cudaSuccess));
    auto span = [&](size_t c, size_t* off, size_t* len) {
        *off = c == 0 ? 0 : head + (c - 1) * kChunk;
        const size_t end = c == 0 ? head : *off + kChunk;
        *len = (end < bytes ? end : bytes) - *off;
    };
    auto work = [&](const Worker& w) {
        cudaError_t err = cudaSetDevice(device);
        size_t c[2] = {chunks, chunks}, off, len;
        // slot i holds chunk c[i] in flight; the other slot is being moved by this thread meanwhile
        for (int i = 0; err == cudaSuccess && failed.load() == static_cast<int>(cudaSuccess); i ^= 1) {
            if (to_host) {
                const size_t got = next.fetch_add(1);
                if (got < chunks) {
                    span(got, &off, &len);
                    err = cudaMemcpyAsync(w.pinned[i], d + off, len, cudaMemcpyDeviceToHost, w.stream);
                    if (err == cudaSuccess) err = cudaEventRecord(w.done[i], w.stream);
                }
                c[i] = got;
                const int o = i ^ 1;
                if (err == cudaSuccess && c[o] < chunks) {
                    err = cudaEventSynchronize(w.done[o]);
                    span(c[o], &off, &len);
                    if (err == cudaSuccess) memcpy(h + off, w.pinned[o], len);
                    c[o] = chunks;
                }
                if (got >= chunks) break;
            } else {
                if (c[i] < chunks) err = cudaEventSynchronize(w.done[i]);          // this slot's last copy has left it
                c[i] = next.fetch_add(1);
                if (err != cudaSuccess || c[i] >= chunks) break;
                span(c[i], &off, &len);
                memcpy(w.pinned[i], h + off, len);
                err = cudaMemcpyAsync(d + off, w.pinned[i], len, cudaMemcpyHostToDevice, w.stream);
                if (err == cudaSuccess) err = cudaEventRecord(w.done[i], w.stream);
            }
        }
        const cudaError_t last = cudaStreamSynchronize(w.stream);
        if (err == cudaSuccess) err = last;
        if (err != cudaSuccess) failed.store(static_cast<int>(err));
    };
    std::vector<std::thread> threads;
    try {
        for (size_t i = 1; i < workers; ++i) threads.emplace_back(work, std::cref(workers_[i]));
    } catch (const std::system_error&) {
        // the threads that could be started, or this one alone, take all chunks
    }
    work(workers_[0]);
    for (std::thread& t : threads) t.join();
    return static_cast<cudaError_t>(failed.load());
}

}  // namespace vdnn
