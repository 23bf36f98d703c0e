// See host_copy.h.
#include "host_copy.h"

#include <stdint.h>
#include <string.h>

#include <atomic>
#include <exception>

namespace vdnn {

namespace {
constexpr size_t kChunk = 2u << 20;         // a huge page of the host
// Up to these sizes one thread is the faster way.  Measured with the other way beside it (us, B200 host, fresh destinations):
//   reads   64 KB 25 alone, 31 by threads; 512 KB 48 and 55; 1 MB 106 and 103; 2 MB 184 and 135
//   writes  1 MB 61 by cudaMemcpy, 104 by threads; 2 MB 120 and 156; 4 MB 226 and 235; 6 MB 332 and 313; 8 MB 477 and 379
// A write takes longer to be worth it: its source has been touched.
constexpr size_t kDirectRead = 512u << 10, kDirectWrite = 4u << 20;
// From this size on a thread takes whole huge pages.  Below, the page faults of the destination are what takes long, and smaller
// pieces let more threads share them: 4 MB 179 us in quarters, 213 whole; 8 MB 308 and 331; 12 MB 452 and 424; 16 MB 613 and 530;
// 32 MB 1520 and 1240.
constexpr size_t kWholePages = 16u << 20;

// Makes a device current for as long as it lives; the thread gets its own device back.
struct OnDevice {
    int before;
    bool changed;
    cudaError_t status;
    explicit OnDevice(int device) : before(device), changed(false), status(cudaGetDevice(&before)) {
        if (status != cudaSuccess || before == device) return;
        status = cudaSetDevice(device);
        changed = status == cudaSuccess;
    }
    ~OnDevice() { if (changed) cudaSetDevice(before); }
};
}  // namespace

HostCopy::~HostCopy() {
    {
        std::lock_guard<std::mutex> lock(mu_);
        stop_ = true;
    }
    wake_.notify_all();
    for (std::thread& t : threads_) t.join();
    for (size_t i = 0; i < made_; ++i) release(&workers_[i]);
}

void HostCopy::release(Worker* w) {
    for (int i = 0; i < 2; ++i) {
        if (w->pinned[i]) cudaFreeHost(w->pinned[i]);
        if (w->done[i]) cudaEventDestroy(w->done[i]);
    }
    if (w->stream) cudaStreamDestroy(w->stream);
    *w = Worker();
}

cudaError_t HostCopy::make(Worker* w) {
    cudaError_t e = cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking);
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
        e = cudaEventCreateWithFlags(&w->done[i], cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaHostAlloc(reinterpret_cast<void**>(&w->pinned[i]), kChunk, cudaHostAllocDefault);
    }
    return e;
}

size_t HostCopy::make_workers(size_t want) {
    while (made_ < want) {
        if (make(&workers_[made_]) != cudaSuccess) {
            release(&workers_[made_]);
            (void)cudaGetLastError();
            break;
        }
        ++made_;
    }
    return made_ < want ? made_ : want;
}

void HostCopy::serve(size_t index) {
    unsigned long long seen = 0;
    std::unique_lock<std::mutex> lock(mu_);
    for (;;) {
        wake_.wait(lock, [&] { return stop_ || round_ != seen; });
        if (stop_) return;
        seen = round_;
        if (index >= wanted_) continue;
        lock.unlock();
        job_(workers_[index]);
        lock.lock();
        if (--busy_ == 0) done_.notify_one();
    }
}

cudaError_t HostCopy::run(void* host, void* dev, size_t bytes, int device, bool to_host) {
    if (!to_host && bytes <= kDirectWrite) return cudaMemcpy(dev, host, bytes, cudaMemcpyHostToDevice);
    std::lock_guard<std::mutex> turn(turn_);
    const OnDevice on(device);          // streams, events and staging buffers belong to the device of the memory
    if (on.status != cudaSuccess) return on.status;
    if (to_host && bytes <= kDirectRead && make_workers(1) == 1) {
        // through pinned memory: the driver's way into pageable memory takes 5 us longer
        const Worker& w = workers_[0];
        cudaError_t e = cudaMemcpyAsync(w.pinned[0], dev, bytes, cudaMemcpyDeviceToHost, w.stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(w.stream);
        if (e == cudaSuccess) memcpy(host, w.pinned[0], bytes);
        return e;
    }
    char* const h = static_cast<char*>(host);
    char* const d = static_cast<char*>(dev);
    // chunk 0 ends at the first 2 MB boundary of the host address
    size_t head = kChunk - (reinterpret_cast<uintptr_t>(h) & (kChunk - 1));
    if (head > bytes) head = bytes;
    const size_t piece = bytes >= kWholePages ? kChunk : kChunk / 4;
    if (piece < kChunk && head > piece) head = piece;
    const size_t chunks = 1 + (bytes - head + piece - 1) / piece;
    unsigned cores = std::thread::hardware_concurrency();
    size_t workers = cores > 2 ? cores / 2 : 1;
    if (workers > kMaxWorkers) workers = kMaxWorkers;
    if (workers > chunks) workers = chunks;
    workers = make_workers(workers);
    if (workers == 0) return cudaMemcpy(to_host ? host : dev, to_host ? dev : host, bytes, to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice);

    std::atomic<size_t> next(0);
    std::atomic<int> failed(static_cast<int>(cudaSuccess));
    auto span = [&](size_t c, size_t* off, size_t* len) {
        *off = c == 0 ? 0 : head + (c - 1) * piece;
        const size_t end = c == 0 ? head : *off + piece;
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
    {
        std::lock_guard<std::mutex> lock(mu_);
        try {
            job_ = work;
            while (threads_.size() + 1 < workers) { const size_t index = threads_.size() + 1; threads_.emplace_back([this, index] { serve(index); }); }
        } catch (const std::exception&) {
            // the threads that could be started, or this one alone, take all chunks
        }
        if (!job_) workers = 1;
        if (workers > threads_.size() + 1) workers = threads_.size() + 1;
        wanted_ = workers;
        busy_ = workers - 1;
        ++round_;
    }
    if (workers > 1) wake_.notify_all();
    work(workers_[0]);
    {
        std::unique_lock<std::mutex> lock(mu_);
        done_.wait(lock, [&] { return busy_ == 0; });
        job_ = nullptr;
    }
    return static_cast<cudaError_t>(failed.load());
}

}  // namespace vdnn
